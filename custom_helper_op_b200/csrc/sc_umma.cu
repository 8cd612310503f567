// Manifold 3-D convolution as an implicit GEMM on the 5th-generation tensor cores (tcgen05), for the
// case the depth-band networks actually run: 3x3x3 filter, stride 1, dilation 1, bfloat16 storage,
// float32 accumulation, 8, 16 or 32 channels.
//
//   D[m][n] = sum_k A[m][k] * B[n][k]     m: 128 output voxels of a tile (one per thread)
//                                          n: output channels (16 / 32)
//                                          k: tap * CIN + input channel  (27 taps)
// A is never materialised in global memory: every thread gathers, for its voxel and each tap, the CIN
// contiguous bf16 channels of the neighbour voxel - resolving the per-pixel depth shift
// d + base_plane[out] - base_plane[nbr] (custom_helper_op/cc/kernels/
// sparse_conv3d_fast_fixed_param_op_gpu.cu.cc:78-113), padding with default_value - and writes them into
// shared memory in the tensor core's canonical K-major layout (8-row x 16-byte core matrices, no
// swizzle).  The filter (27*CIN*COUT bf16) is laid out once per CTA in the same form.  One elected thread
// issues tcgen05.mma (M=128, N=COUT, K=16) per tap and 16 input channels, accumulating in tensor memory;
// tcgen05.commit signals an mbarrier; the four warps then read their 32 accumulator rows back with
// tcgen05.ld, round to bf16 and store 2*COUT contiguous bytes per voxel.
//
// A tile is processed in three rounds of nine taps (one filter row each) so that the A staging buffer is
// 9*128*CIN*2 bytes and several CTAs fit on an SM: while one CTA waits for its MMAs another gathers.
// The image gradient is the same kernel run over out_grad with the filter flipped in all three
// dimensions, channels swapped and zero padding (sparse_conv3d_fast_op.cc:298-323).
//
// Every wait on the mbarrier is bounded; if it ever gives up the kernel raises a device-side flag
// (readable through sc_umma_timeouts()), stops issuing work, frees its tensor memory and returns.
#include <cuda_bf16.h>

#include <atomic>
#include <mutex>

#include "sc_common.cuh"
#include "sc_entry.h"
#include "sc_umma_common.cuh"
#include "smem_grant.h"

namespace chop {
namespace {

__global__ void note_timeout_kernel() { note_timeout(); }
std::atomic<int> g_umma_rows{1};   // tuning knob "umma_rows": 0 = always the per-tap gather, 2 = never sc_band.cu and sc_up.cu

// ---- tap geometry (3x3x3, dilation 1) -----------------------------------------------------------------------
// The tile's voxels are OUTPUT voxels of the (strided) convolution, grid [B,oH,oW,oD]; a tap reads the input grid
// [B,H,W,D] (sc_tap in sc_common.cuh).  At stride 1 the same geometry serves the image gradient and the transposed
// convolution (S1: no multiplications by strides); with strides those run in sc_umma_class_kernel below.
struct VoxPos {
  int b, r, c;      // batch, row and column in the fine grid (of the voxel's centre tap)
  int depth_abs;    // absolute fine depth plane of the voxel
};

template <bool S1>
__device__ __forceinline__ VoxPos vox_pos(const ScArgs& a, long long v) {
  VoxPos p;
  const int d1 = S1 ? a.D : a.oD, d2 = S1 ? a.W : a.oW, d3 = S1 ? a.H : a.oH;
  int dz, cc, rr;
  if (v <= 0x7fffffffLL) {   // 64-bit divisions cost several times the rest of this function
    unsigned u = (unsigned)v;
    dz = (int)(u % (unsigned)d1); u /= (unsigned)d1;
    cc = (int)(u % (unsigned)d2); u /= (unsigned)d2;
    rr = (int)(u % (unsigned)d3);
    p.b = (int)(u / (unsigned)d3);
  } else {
    dz = (int)(v % d1); v /= d1;
    cc = (int)(v % d2); v /= d2;
    rr = (int)(v % d3);
    p.b = (int)(v / d3);
  }
  p.r = S1 ? rr : rr * a.sr;
  p.c = S1 ? cc : cc * a.sc;
  const int bp = __ldg(a.base_plane + (p.b * a.H + p.r) * a.W + p.c);
  p.depth_abs = S1 ? dz + bp : (dz + (bp + a.sd - 1) / a.sd) * a.sd;
  return p;
}

// One (fr, fc) column of taps: false if the whole column is padding; otherwise base = index of the source
// pixel's first voxel and shift = what to subtract from the tap's absolute depth.
__device__ __forceinline__ bool tap_column(const ScArgs& a, const VoxPos& p, int fr, int fc, long long& base, int& shift) {
  const int orow = p.r - 1 + fr, ocol = p.c - 1 + fc;
  if (oob(orow, a.H) || oob(ocol, a.W)) return false;
  shift = __ldg(a.base_plane + (p.b * a.H + orow) * a.W + ocol);
  base = ((long long)(p.b * a.H + orow) * a.W + ocol) * a.D;
  return true;
}

// Source voxel of tap fz in a column, or -1.
__device__ __forceinline__ long long tap_voxel(const ScArgs& a, const VoxPos& p, long long base, int shift, int fz) {
  const int ind = p.depth_abs - 1 + fz - shift;
  return oob(ind, a.D) ? -1 : base + ind;
}

// CR: channels of the gathered tensor (K per tap), NR: channels produced (N).
template <int CR, int NR, bool DGRAD, bool S1>
__global__ void __launch_bounds__(128) sc_umma_kernel(const ScArgs a, const long long nvox, const int ntiles) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) uint64_t mbar_s;
  __shared__ uint32_t tmem_base_s;
  constexpr int CIN = pad16(CR), COUT = pad16(NR);
  constexpr int KC = CIN / 8, KR = CR / 8;        // 16-byte k-chunks per tap, those that are channels
  constexpr uint32_t LBO = 128, SBO = KC * 128;   // core-matrix strides in K and in M/N
  constexpr int A_TAP_BYTES = 128 * CIN * 2;
  constexpr int B_TAP_BYTES = COUT * CIN * 2;
  unsigned char* sB = smem;                       // 27 taps
  unsigned char* sA = smem + 27 * B_TAP_BYTES;    // 9 taps (one filter row)
  const int tid = threadIdx.x, warp = tid >> 5;

  const __nv_bfloat16* src = static_cast<const __nv_bfloat16*>(DGRAD ? a.out_grad : a.images);
  __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(DGRAD ? a.images_grad : a.output);

  // ---- filter -> canonical K-major B tiles: B[n][k] of tap t at sB + t*B_TAP_BYTES -----------------------
  {
    stage_filter_tiles<CR, NR, DGRAD>(static_cast<const unsigned short*>(a.filters), sB, tid, LBO, SBO, B_TAP_BYTES);
    if (KR < KC)   // the padding channels of the staging rows stay zero
      for (int e = tid; e < 9 * 128; e += 128)
        *reinterpret_cast<uint4*>(sA + e / 128 * A_TAP_BYTES + (e % 128 / 8) * SBO + e % 8 * 16 + LBO) = make_uint4(0, 0, 0, 0);
  }
  if (warp == 0) {
    uint32_t slot = smem_u32(&tmem_base_s), ncols = 32;
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&mbar_s)), "r"(1) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base_s;
  const uint32_t mbar = smem_u32(&mbar_s);
  // instruction descriptor: D f32, A/B bf16, both K-major, N = COUT, M = 128
  constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(COUT >> 3) << 17) | ((128u >> 4) << 24);

  // padding value of the gathered tensor, replicated over 8 bf16 (zero for gradients with respect to images)
  uint4 padv = make_uint4(0, 0, 0, 0);
  if (!a.pad_zero) {
    const unsigned d16 = __ldg(static_cast<const unsigned short*>(a.default_value));
    const unsigned d32 = d16 | (d16 << 16);
    padv = make_uint4(d32, d32, d32, d32);
  }

  uint32_t phase = 0;
  bool alive = true;
  for (int tile = blockIdx.x; tile < ntiles && alive; tile += gridDim.x) {
    const long long v = (long long)tile * 128 + tid;
    const bool vvalid = v < nvox;
    VoxPos pos = {0, 0, 0, 0};
    if (vvalid) pos = vox_pos<S1>(a, v);
    unsigned char* a_row = sA + (tid / 8) * SBO + (tid % 8) * 16;

    for (int fr = 0; fr < 3; ++fr) {
      // ---- gather nine taps (filter row fr) into the staging buffer ---------------------------------------
#pragma unroll
      for (int fc = 0; fc < 3; ++fc) {
        long long base = 0;
        int shift = 0;
        const bool inb = vvalid && tap_column(a, pos, fr, fc, base, shift);
#pragma unroll
        for (int fz = 0; fz < 3; ++fz) {
          const long long sv = inb ? tap_voxel(a, pos, base, shift, fz) : -1;
          const bool ok = sv >= 0;
          const uint4* p = reinterpret_cast<const uint4*>(src + (size_t)(ok ? sv : 0) * CR);
          unsigned char* dstA = a_row + (fc * 3 + fz) * A_TAP_BYTES;
#pragma unroll
          for (int kc = 0; kc < KR; ++kc) {
            uint4 x = vvalid ? padv : make_uint4(0, 0, 0, 0);
            if (ok) x = __ldg(p + kc);
            *reinterpret_cast<uint4*>(dstA + kc * LBO) = x;
          }
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncthreads();
      // ---- one thread issues the round's MMAs ----------------------------------------------------------------
      if (tid == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int tt = 0; tt < 9; ++tt) {
#pragma unroll
          for (int k16 = 0; k16 < CIN / 16; ++k16) {
            const uint64_t da = umma_desc(smem_u32(sA + tt * A_TAP_BYTES + k16 * 2 * LBO), LBO, SBO);
            const uint64_t db = umma_desc(smem_u32(sB + (fr * 9 + tt) * B_TAP_BYTES + k16 * 2 * LBO), LBO, SBO);
            umma_bf16(tmem, da, db, IDESC, (fr | tt | k16) != 0 ? 1u : 0u);
          }
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
      }
      // ---- everyone waits until the tensor core has consumed the staging buffer ------------------------------
      // one warp polls the mbarrier (every poll is a shared-memory access); the others wait at the hardware barrier
      bool done = true;
      if (warp == 0) done = mbar_wait(mbar, phase);
      phase ^= 1;
      if (!__syncthreads_and(done)) {
        if (tid == 0) note_timeout();
        alive = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }
    if (!alive) break;

    // ---- epilogue: accumulator rows -> bf16 -> global ------------------------------------------------------------
    uint32_t acc[COUT];
    tmem_ld<COUT>(tmem + ((uint32_t)(warp * 32) << 16), acc);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    if (vvalid) {
      uint4* o = reinterpret_cast<uint4*>(dst + (size_t)v * NR);
#pragma unroll
      for (int q = 0; q < NR / 8; ++q) {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(acc[q * 8 + 2 * i]), __uint_as_float(acc[q * 8 + 2 * i + 1]));
          w[i] = *reinterpret_cast<const uint32_t*>(&h);
        }
        o[q] = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    uint32_t ncols = 32;
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols) : "memory");
  }
}


// ---------------------------------------------------------------------------------------------------------
// Strided image gradient and transposed convolution: every FINE voxel [B,H,W,D] sums the coarse voxels that lie under
// its taps.  A tap exists only where row, column and absolute depth are multiples of the strides - at strides (2,2,2)
// 3.4 of the 27 on average - and which filter columns exist depends on (row mod sr, column mod sc) alone.  So a tile
// takes 128 voxels of pixels of ONE such class: all its rows share the class's columns (1, 2 or 4 of the nine at
// stride 2) and only those are gathered and multiplied.
// Depth is not classed (its parity depends on the base planes): a depth tap that is not aligned is a row of zeros.
//
// Padded taps read default_value.  The op's own layer fixes it to zero, then they contribute nothing.  For any other value
// the padding rows of the class's columns are filled in, and the columns that do not exist in the class add the same
// constant to every voxel: default * (sum of their weights), added in the epilogue.  256x320x9, 16 -> 16 channels, strides
// (2,2,2), default 0.5: 47 us (88 with the absent columns staged and multiplied like the others).
// ---------------------------------------------------------------------------------------------------------
constexpr int CLS_COLS = 2;   // filter columns staged per round

// CTAs that shared memory lets reside on an SM; the register bound keeps it so.
constexpr size_t class_smem(int cr, int nr) {
  return (size_t)27 * pad16(nr) * pad16(cr) * 2 + (size_t)CLS_COLS * 3 * 128 * pad16(cr) * 2 + 1024;
}
constexpr int class_ctas(int cr, int nr) { return (int)((size_t)220 * 1024 / (class_smem(cr, nr) + 2048)); }

// The tiles of a CTA.  PAD: the default value is not zero (d16: its bits; wcol: per filter column and produced channel,
// default * sum of the weights; padsum: a buffer).
template <int CR, int NR, bool PAD>
__device__ __forceinline__ void class_walk(const ScArgs& a, const int ntiles, unsigned char* sA, const unsigned char* sB,
                                           const uint32_t tmem, const uint32_t mbar, const unsigned d16, const float* wcol,
                                           float (*padsum)[NR]) {
  constexpr int CIN = pad16(CR), COUT = pad16(NR), KC = CIN / 8, KR = CR / 8;
  constexpr uint32_t LBO = 128, SBO = KC * 128;
  constexpr int A_TAP_BYTES = 128 * CIN * 2;
  constexpr int B_TAP_BYTES = COUT * CIN * 2;
  constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(COUT >> 3) << 17) | ((128u >> 4) << 24);
  const int tid = threadIdx.x, warp = tid >> 5;
  const __nv_bfloat16* src = static_cast<const __nv_bfloat16*>(a.out_grad);
  __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(a.images_grad);
  const unsigned d32 = PAD ? d16 | (d16 << 16) : 0u;
  const uint4 padv = make_uint4(d32, d32, d32, d32);

  unsigned char* const a_row = sA + (tid / 8) * SBO + (tid % 8) * 16;

  // the round that is being loaded: this thread's voxel, the class's filter columns still to do
  int tile = blockIdx.x;
  TileClass cl;
  cl.k = 0;
  cl.begin = 0;
  class_open(a, cl, 128);
  unsigned todo = 0;                              // bit fr*3 + fc: filter column still to do
  bool vvalid = false;
  int b = 0, r = 0, c = 0, cr = 0, cc = 0;
  int cdz[3];                                     // absolute coarse plane under depth tap fz
  unsigned dok = 0;                               // bit fz: the depth tap is aligned
  long long out_vox = -1;                         // fine voxel of this thread, -1: none
  auto open_tile = [&]() {
    while (tile >= cl.end) {
      ++cl.k;
      cl.begin = cl.end;
      class_open(a, cl, 128);
    }
    todo = cl.real;
    const unsigned v = (unsigned)(tile - cl.begin) * 128u + tid;
    vvalid = v < (unsigned)a.B * cl.hc * cl.wc * a.D;
    out_vox = -1;
    dok = 0;
    if (vvalid) {
      unsigned u = v;
      const int dz = (int)(u % (unsigned)a.D); u /= (unsigned)a.D;
      cc = (int)(u % (unsigned)cl.wc); u /= (unsigned)cl.wc;
      cr = (int)(u % (unsigned)cl.hc);
      b = (int)(u / (unsigned)cl.hc);
      r = cr * a.sr + cl.pr;
      c = cc * a.sc + cl.pc;
      const int pix = (b * a.H + r) * a.W + c;
      out_vox = (long long)pix * a.D + dz;
      const int d = dz + __ldg(a.base_plane + pix);
      int q = d / a.sd, rem = d - q * a.sd;       // floor division: one for the three depth taps
      if (rem < 0) { rem += a.sd; --q; }
      cdz[0] = a.sd == 1 ? q - 1 : q;
      cdz[1] = q;
      cdz[2] = q + 1;
      dok = (a.sd == 1 || rem == 1 ? 1u : 0u) | (rem == 0 ? 2u : 0u) | (rem + 1 == a.sd ? 4u : 0u);
    }
  };
  int cols[CLS_COLS], ncols = 0;
  uint4 pre[CLS_COLS * 3 * KR];
  auto request = [&]() {   // the next CLS_COLS filter columns of the open tile into registers
    ncols = 0;
#pragma unroll
    for (int i = 0; i < CLS_COLS; ++i) {
      cols[i] = todo ? __ffs(todo) - 1 : 0;
      if (todo) {
        ++ncols;
        todo &= todo - 1;
      }
    }
    int base[CLS_COLS], shift[CLS_COLS];
    bool ok[CLS_COLS];
#pragma unroll
    for (int i = 0; i < CLS_COLS; ++i) {
      const int fr = cols[i] / 3, fc = cols[i] - fr * 3;
      const int orow = r - 1 + fr, ocol = c - 1 + fc;
      ok[i] = i < ncols && vvalid && !oob(orow, a.H) && !oob(ocol, a.W);
      base[i] = shift[i] = 0;
      if (ok[i]) {
        // (pr - 1 + fr) / sr of an aligned tap: -1, 0 or 1
        const int er = cl.pr - 1 + fr, ec = cl.pc - 1 + fc;
        base[i] = ((b * a.oH + cr + (er > 0) - (er < 0)) * a.oW + cc + (ec > 0) - (ec < 0)) * a.oD;
        shift[i] = (__ldg(a.base_plane + (b * a.H + orow) * a.W + ocol) + a.sd - 1) / a.sd;   // as in sc_tap_t
      }
    }
#pragma unroll
    for (int i = 0; i < CLS_COLS; ++i) {
#pragma unroll
      for (int fz = 0; fz < 3; ++fz) {
        const int cd = cdz[fz] - shift[i];
        const bool in = ok[i] && ((dok >> fz) & 1u) && !oob(cd, a.oD);
        const uint4* p = reinterpret_cast<const uint4*>(src + (size_t)(in ? base[i] + cd : 0) * CR);
#pragma unroll
        for (int kc = 0; kc < KR; ++kc) {
          uint4 x = PAD && vvalid ? padv : make_uint4(0, 0, 0, 0);
          if (in) x = __ldg(p + kc);
          pre[(i * 3 + fz) * KR + kc] = x;
        }
      }
    }
  };
  cdz[0] = cdz[1] = cdz[2] = 0;
  open_tile();
  request();

  uint32_t phase = 0;
  bool started = false;                           // the tile in the tensor core has accumulated something
  while (true) {
    // ---- the requested rows -> staging buffer; MMAs ------------------------------------------------------------
    const int n_now = ncols;
    int cols_now[CLS_COLS];
#pragma unroll
    for (int i = 0; i < CLS_COLS; ++i) cols_now[i] = cols[i];
    const bool last = todo == 0;                  // last round of its tile
    const long long out_now = out_vox;
    if (PAD && tid < NR) {                        // what the columns that the tile's class does not have add
      float sum = 0.f;
      for (unsigned m = 0x1ffu & ~cl.real; m; m &= m - 1) sum += wcol[(__ffs(m) - 1) * NR + tid];
      padsum[phase ^ 1][tid] = sum;               // read in this round's epilogue, where phase has changed
    }
    const int KT = CLS_COLS * 3;
#pragma unroll
    for (int q = 0; q < KT; ++q) {
      if (q < n_now * 3) {
#pragma unroll
        for (int kc = 0; kc < KR; ++kc) *reinterpret_cast<uint4*>(a_row + q * A_TAP_BYTES + kc * LBO) = pre[q * KR + kc];
      }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      for (int i = 0; i < n_now; ++i) {
#pragma unroll
        for (int fz = 0; fz < 3; ++fz) {
#pragma unroll
          for (int k16 = 0; k16 < CIN / 16; ++k16) {
            const uint64_t da = umma_desc(smem_u32(sA + (i * 3 + fz) * A_TAP_BYTES + k16 * 2 * LBO), LBO, SBO);
            const uint64_t db = umma_desc(smem_u32(sB + (cols_now[i] * 3 + fz) * B_TAP_BYTES + k16 * 2 * LBO), LBO, SBO);
            umma_bf16(tmem, da, db, IDESC, (started || i > 0 || fz > 0 || k16 > 0) ? 1u : 0u);
          }
        }
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
    }
    started = started || n_now > 0;

    // ---- while they run: the next round's lookups and rows -------------------------------------------------------
    bool more = true;
    if (last) {
      tile += gridDim.x;
      more = tile < ntiles;
      if (more) open_tile();
    }
    if (more) request();

    bool done = true;
    if (warp == 0) done = mbar_wait(mbar, phase);
    phase ^= 1;
    if (!__syncthreads_and(done)) {
      if (tid == 0) note_timeout();
      break;
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

    if (last) {
      // ---- epilogue: accumulator rows -> bf16 -> global; a class without taps (strides above 3) is zero --------
      uint32_t acc[COUT];
      if (started) {
        tmem_ld<COUT>(tmem + ((uint32_t)(warp * 32) << 16), acc);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      } else {
#pragma unroll
        for (int n = 0; n < COUT; ++n) acc[n] = 0u;
      }
      if (PAD) {
#pragma unroll
        for (int n = 0; n < NR; ++n) acc[n] = __float_as_uint(__uint_as_float(acc[n]) + padsum[phase][n]);
      }
      if (out_now >= 0) {
        uint4* o = reinterpret_cast<uint4*>(dst + (size_t)out_now * NR);
#pragma unroll
        for (int q = 0; q < NR / 8; ++q) {
          uint32_t w[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(acc[q * 8 + 2 * i]), __uint_as_float(acc[q * 8 + 2 * i + 1]));
            w[i] = *reinterpret_cast<const uint32_t*>(&h);
          }
          o[q] = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      started = false;
    }
    if (!more) break;
  }
}

template <int CR, int NR>
__global__ void __launch_bounds__(128, class_ctas(CR, NR)) sc_umma_class_kernel(const ScArgs a, const int ntiles) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) uint64_t mbar_s;
  __shared__ uint32_t tmem_base_s;
  __shared__ float wcol_s[9 * NR];
  __shared__ float padsum_s[2][NR];               // two: a round's is written while the last one's may still be read
  constexpr int CIN = pad16(CR), COUT = pad16(NR), KC = CIN / 8, KR = CR / 8;
  constexpr uint32_t LBO = 128, SBO = KC * 128;
  constexpr int A_TAP_BYTES = 128 * CIN * 2;
  constexpr int B_TAP_BYTES = COUT * CIN * 2;
  unsigned char* sB = smem;                       // 27 taps
  unsigned char* sA = smem + 27 * B_TAP_BYTES;    // CLS_COLS columns of three depth taps
  const int tid = threadIdx.x, warp = tid >> 5;

  stage_filter_tiles<CR, NR, true>(static_cast<const unsigned short*>(a.filters), sB, tid, LBO, SBO, B_TAP_BYTES);
  if (KR < KC)   // the padding channels of the staging rows stay zero
    for (int e = tid; e < CLS_COLS * 3 * 128; e += 128)
      *reinterpret_cast<uint4*>(sA + e / 128 * A_TAP_BYTES + (e % 128 / 8) * SBO + e % 8 * 16 + LBO) = make_uint4(0, 0, 0, 0);
  if (warp == 0) {
    uint32_t slot = smem_u32(&tmem_base_s), ncols = 32;
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&mbar_s)), "r"(1) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base_s;
  const uint32_t mbar = smem_u32(&mbar_s);
  unsigned d16 = 0;
  if (!a.pad_zero) d16 = __ldg(static_cast<const unsigned short*>(a.default_value));
  if ((d16 & 0x7fffu) != 0) {                     // a non-zero default: every tap of every voxel contributes
    for (int e = tid; e < 9 * NR; e += 128) {
      const int col = e / NR, n = e % NR;
      float sum = 0.f;
      for (int q = 0; q < 3 * KR; ++q) {          // sB holds eight weights of one (tap, n) in 16 bytes
        const uint4 x = *reinterpret_cast<const uint4*>(sB + (col * 3 + q / KR) * B_TAP_BYTES + (n / 8) * SBO + (q % KR) * LBO + (n % 8) * 16);
        const unsigned w4[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) sum += __uint_as_float(w4[i] << 16) + __uint_as_float(w4[i] & 0xffff0000u);
      }
      wcol_s[e] = __uint_as_float(d16 << 16) * sum;
    }
    __syncthreads();
    class_walk<CR, NR, true>(a, ntiles, sA, sB, tmem, mbar, d16, wcol_s, padsum_s);
  } else {
    class_walk<CR, NR, false>(a, ntiles, sA, sB, tmem, mbar, 0u, wcol_s, padsum_s);
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    uint32_t ncols = 32;
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols) : "memory");
  }
}


// ---- per-tile table of filter columns for the shifted-row kernels -------------------------------------------
// Entry (pixel q of the tile, filter column col) = {first voxel of the neighbour pixel (-1: outside the image,
// -2: the tile has no such pixel), base_plane[pixel] - base_plane[neighbour]}.  The D + 2 rows of a pixel share
// these nine entries, so the CTA computes each once (one entry per thread) instead of once per row.
constexpr int ROWS_TAB = 42 * 9;   // a tile has at most 128 / 3 pixels
__device__ __forceinline__ void rows_tab_write(const ScArgs& a, int2* tab, int tile, int ntiles, int PT, long long npix, int tid) {
  for (int e = tid; e < PT * 9; e += 128) {
    const int q = e / 9, col = e - q * 9;
    const long long pix = (long long)tile * PT + q;
    int2 ent = make_int2(-2, 0);
    if (tile < ntiles && pix < npix) {
      const unsigned p32 = (unsigned)pix;   // pixel counts are validated to fit 31 bits
      const int c = (int)(p32 % (unsigned)a.W);
      const unsigned t = p32 / (unsigned)a.W;
      const int r = (int)(t % (unsigned)a.H), b = (int)(t / (unsigned)a.H);
      const int orow = r - 1 + col / 3, ocol = c - 1 + col % 3;
      ent.x = -1;
      if (!oob(orow, a.H) && !oob(ocol, a.W)) {
        const int np = (b * a.H + orow) * a.W + ocol;
        ent.x = np * a.D;                   // voxel indices fit 31 bits (checked on the host)
        ent.y = __ldg(a.base_plane + pix) - __ldg(a.base_plane + np);
      }
    }
    tab[e] = ent;
  }
}
// Source voxel of row j of pixel q in each column: >= 0, -1 = padding (default_value), -2 = not part of the tile.
__device__ __forceinline__ void rows_tab_read(const int2* tab, int q, int j, int D, bool row_used, int* sv) {
#pragma unroll
  for (int col = 0; col < 9; ++col) {
    int v = -2;
    if (row_used) {
      const int2 e = tab[q * 9 + col];
      const int plane = j - 1 + e.y;
      v = e.x >= 0 ? (oob(plane, D) ? -1 : e.x + plane) : e.x;
    }
    sv[col] = v;
  }
}

// ---------------------------------------------------------------------------------------------------------
// Stride-1 variant with ONE staged copy per neighbour pixel instead of one per tap.
//
// The three depth taps of a filter column (fr, fc) read the same neighbour pixel at consecutive planes, so
// their A operands are the same rows shifted by one.  With SBO = 128 bytes the canonical K-major layout
// stores row r of a 16-byte K-chunk at r*16 bytes, i.e. rows are linear, and a tap's operand is simply the
// column buffer's address plus fz*16 bytes.  A tile therefore holds PT = 128 / (D + 2) pixels, every pixel
// owning D + 2 rows: row (p, j) of column (fr, fc) holds plane j - 1 + base_plane[p] - base_plane[nbr] of
// the neighbour pixel (default_value outside its band or outside the image), and MMA row m = p*(D+2) + d,
// d < D, is output voxel (p, d); the two remaining rows per pixel produce values that are discarded.
// Against the per-tap gather this stages 9 instead of 27 rows per voxel, issues all 27 taps of a tile
// behind one barrier (one commit, one wait) and reads every neighbour plane once.
// ---------------------------------------------------------------------------------------------------------
template <int CR, int NR, bool DGRAD>
__global__ void __launch_bounds__(128, CR <= 16 ? 4 : 2) sc_umma_rows_kernel(const ScArgs a, const int ntiles, const int PT) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) uint64_t mbar_s;
  __shared__ uint32_t tmem_base_s;
  __shared__ int2 tab_s[ROWS_TAB];
  constexpr int CIN = pad16(CR), COUT = pad16(NR), KC = CIN / 8, KR = CR / 8;
  // rows per column buffer: 128 + the two shifted reads; 132 rows make the K-chunk stride 64 bytes off a multiple
  // of 128, so the KC lanes that store the chunks of one row hit different banks
  constexpr int NRB = 132;
  constexpr uint32_t B_LBO = 128, B_SBO = KC * 128;     // filter tiles: K-chunks adjacent, then 8-row groups
  constexpr uint32_t A_LBO = NRB * 16, A_SBO = 128;     // column buffers: rows linear, K-chunks NRB rows apart
  constexpr int B_TAP_BYTES = COUT * CIN * 2;
  constexpr int COL_BYTES = KC * NRB * 16;
  unsigned char* sB = smem;                             // 27 taps
  unsigned char* sX = smem + 27 * B_TAP_BYTES;          // 9 filter columns
  const int tid = threadIdx.x, warp = tid >> 5;

  const __nv_bfloat16* src = static_cast<const __nv_bfloat16*>(DGRAD ? a.out_grad : a.images);
  __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(DGRAD ? a.images_grad : a.output);

  {
    stage_filter_tiles<CR, NR, DGRAD>(static_cast<const unsigned short*>(a.filters), sB, tid, B_LBO, B_SBO, B_TAP_BYTES);
    // rows 128..135 of every column buffer are only ever read into discarded output rows; keep them defined
    for (int e = tid; e < 9 * KC * (NRB - 128); e += 128) {
      const int rr = e % (NRB - 128), kc = (e / (NRB - 128)) % KC, col = e / ((NRB - 128) * KC);
      *reinterpret_cast<uint4*>(sX + col * COL_BYTES + kc * A_LBO + (128 + rr) * 16) = make_uint4(0, 0, 0, 0);
    }
    if (KR < KC)   // the padding channels stay zero
      for (int e = tid; e < 9 * 128; e += 128)
        *reinterpret_cast<uint4*>(sX + e / 128 * COL_BYTES + A_LBO + e % 128 * 16) = make_uint4(0, 0, 0, 0);
  }
  if (warp == 0) {
    uint32_t slot = smem_u32(&tmem_base_s), ncols = 32;
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&mbar_s)), "r"(1) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  rows_tab_write(a, tab_s, blockIdx.x, ntiles, PT, (long long)a.B * a.H * a.W, tid);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base_s;
  const uint32_t mbar = smem_u32(&mbar_s);
  constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(COUT >> 3) << 17) | ((128u >> 4) << 24);

  uint4 padv = make_uint4(0, 0, 0, 0);
  if (!a.pad_zero) {
    const unsigned d16 = __ldg(static_cast<const unsigned short*>(a.default_value));
    const unsigned d32 = d16 | (d16 << 16);
    padv = make_uint4(d32, d32, d32, d32);
  }

  const int H = a.H, W = a.W, D = a.D, RP = D + 2;
  const long long npix = (long long)a.B * H * W;
  const int p_in_tile = tid / RP, j = tid - p_in_tile * RP;   // this thread's row: pixel of the tile, row of the pixel
  const bool row_used = p_in_tile < PT;
  uint32_t phase = 0;
  bool alive = true;
  // Source voxel of this thread's row in each of the nine filter columns of a tile; -1 = padding (default_value),
  // -2 = the row is not part of the tile (zeros).  Voxel indices fit 31 bits (checked on the host).
  long long pix = 0;
  bool rvalid = false;
  int sv[9];
  auto locate = [&](int tile) {   // from the table that rows_tab_write(tile) left in shared memory
    pix = (long long)tile * PT + p_in_tile;
    rvalid = row_used && tile < ntiles && pix < npix;
    rows_tab_read(tab_s, p_in_tile, j, D, row_used, sv);
  };
  // The KR 16-byte chunks of a row are fetched by KR neighbouring lanes (the row's owner hands its source voxel
  // over by shuffle), so a warp-wide load covers whole rows - contiguous 32*16 bytes where the rows are
  // consecutive planes of one pixel - instead of every other 16 bytes of twice the span: half the L1 wavefronts.
  // Pass i of lane l: row 32*warp + l/KR + i*(32/KR), chunk l%KR.
  uint4 val[9][KR];
  const int lane = tid & 31, chunk = lane % KR, lrow = lane / KR;
  auto request = [&]() {
#pragma unroll
    for (int col = 0; col < 9; ++col) {
#pragma unroll
      for (int i = 0; i < KR; ++i) {
        const int sr = KR == 1 ? sv[col] : __shfl_sync(0xffffffffu, sv[col], lrow + i * (32 / KR));
        val[col][i] = sr == -2 ? make_uint4(0, 0, 0, 0) : padv;
        if (sr >= 0) val[col][i] = __ldg(reinterpret_cast<const uint4*>(src + (size_t)sr * CR) + chunk);
      }
    }
  };
  locate(blockIdx.x);
  request();
  __syncthreads();   // everybody has read the first tile's table before the loop writes the next one
  const uint64_t da0 = umma_desc(smem_u32(sX), A_LBO, A_SBO);
  const uint64_t db0 = umma_desc(smem_u32(sB), B_LBO, B_SBO);
  for (int tile = blockIdx.x; tile < ntiles && alive; tile += gridDim.x) {
    // ---- stage the nine filter columns: this tile's rows were requested a tile ago and waited in registers
    // while the previous tile's MMAs and epilogue ran (the gather latency is the longest step of a tile) --------
    const long long pix_out = pix;
    const bool rvalid_out = rvalid;
    // the next tile's column table (everybody has read the current one: it was consumed before the barrier that
    // closed the previous tile)
    rows_tab_write(a, tab_s, tile + gridDim.x, ntiles, PT, npix, tid);
#pragma unroll
    for (int col = 0; col < 9; ++col) {
      unsigned char* dx = sX + col * COL_BYTES + chunk * A_LBO + (warp * 32 + lrow) * 16;
#pragma unroll
      for (int i = 0; i < KR; ++i) *reinterpret_cast<uint4*>(dx + i * (32 / KR) * 16) = val[col][i];
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int col = 0; col < 9; ++col) {
#pragma unroll
        for (int fz = 0; fz < 3; ++fz) {
#pragma unroll
          for (int k16 = 0; k16 < CIN / 16; ++k16) {
            const uint64_t da = umma_desc_advance(da0, col * COL_BYTES + k16 * 2 * A_LBO + fz * 16);
            const uint64_t db = umma_desc_advance(db0, (col * 3 + fz) * B_TAP_BYTES + k16 * 2 * B_LBO);
            umma_bf16(tmem, da, db, IDESC, (col | fz | k16) != 0 ? 1u : 0u);
          }
        }
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
    }
    locate(tile + gridDim.x);   // table written before the barrier above; read here, before the barrier below
    request();                  // in flight during this tile's MMAs and epilogue
    // one warp polls the mbarrier (every poll is a shared-memory access); the others wait at the hardware barrier
    bool done = true;
    if (warp == 0) done = mbar_wait(mbar, phase);
    phase ^= 1;
    if (!__syncthreads_and(done)) {
      if (tid == 0) note_timeout();
      alive = false;
      break;
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

    // ---- epilogue: MMA row m = this thread's row; it is output voxel (pixel, j) when j < D -----------------------
    uint32_t acc[COUT];
    tmem_ld<COUT>(tmem + ((uint32_t)(warp * 32) << 16), acc);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    if (rvalid_out && j < D) {
      uint4* o = reinterpret_cast<uint4*>(dst + ((size_t)pix_out * D + j) * NR);
#pragma unroll
      for (int q = 0; q < NR / 8; ++q) {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(acc[q * 8 + 2 * i]), __uint_as_float(acc[q * 8 + 2 * i + 1]));
          w[i] = *reinterpret_cast<const uint32_t*>(&h);
        }
        o[q] = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    uint32_t ncols = 32;
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols) : "memory");
  }
}


// ---------------------------------------------------------------------------------------------------------
// Filter gradient on the tensor cores:  dW[k][n] = sum over voxels m of A[m][k] * G[m][n]
// (k = tap*CIN + input channel, n = output channel, A = the same gathered tile as in the forward pass,
// G = out_grad).  The reduction runs over voxels, so both operands are used "MN-major": the staging
// buffers hold [8 voxels][8 channels] core matrices, 16 voxels per MMA step, and the M dimension of
// the MMA is a group of 128 consecutive k (128/CIN taps).  ceil(27*CIN/128) such groups each own COUT
// tensor-memory columns, and the accumulators stay in tensor memory across ALL voxel tiles of the CTA;
// they are read once at the end and written as this CTA's partial [27*CIN][COUT] slab, which the same
// fixed-order reduction kernel as the generic path sums over the CTAs.
// d(default_value) (dynamic_default only) is accumulated on the CUDA cores while gathering.
// ---------------------------------------------------------------------------------------------------------
// TS = true is the filter gradient of the TRANSPOSED convolution with the roles swapped: a coarse voxel lies under tap t
// of exactly one fine voxel, which is the voxel that tap 26 - t of the STRIDED convolution reads.  So the same kernel runs
// over the coarse voxels with a.images = the fine upstream gradient and a.out_grad = the op's coarse input, padding
// nothing - instead of walking the fine grid (8x the voxels at strides (2,2,2)) whose taps are mostly empty: 133 -> 27 us
// at the c4 band, 16 -> 16 channels.
// What a non-zero default_value adds at the empty taps is linear: default * (sum of the fine gradient over all voxels -
// over the voxels with a coarse voxel under the tap).  The second sum comes out of the same MMAs: a column of ones beside
// the coarse input (the gathered rows are zero wherever a tap sees nothing).  Whether that column is there is decided in
// the kernel, since the default lives on the device; it widens N by 16 (nothing for 8 channels, which are padded to 16).
// Whole gradient at that band, default 0 / 0.5: 16 -> 16 channels 81 / 82 us, 32 -> 32 231 / 270, 32 -> 32 at stride 1
// 578 / 621 (the taps looked up again voxel by voxel for the second sum: 632, 1990 and 10100).
template <bool TS>
__host__ __device__ constexpr int wgrad_width(int cout) { return TS && cout >= 16 ? cout + 16 : pad16(cout); }
__device__ __forceinline__ constexpr uint32_t tmem_cols(uint32_t n) {   // an allocation is a power of two from 32 on
  return n <= 32 ? 32 : n <= 64 ? 64 : n <= 128 ? 128 : n <= 256 ? 256 : 512;
}
template <int CIN, int COUT, bool TS, bool S1>
__global__ void __launch_bounds__(128) sc_umma_wgrad_kernel(const ScArgs a, const long long nvox, const int ntiles) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) uint64_t mbar_s;
  __shared__ uint32_t tmem_base_s;
  __shared__ float red_s[128];
  constexpr int KC = CIN / 8;            // 16-byte channel chunks per tap
  constexpr int NP = pad16(COUT);        // N of an MMA; what the padding columns hold is not used
  constexpr int NX = wgrad_width<TS>(COUT);   // with the column of ones
  constexpr int TPR = 128 / CIN;         // taps per round (one 128-row M group)
  constexpr int NT = (27 + TPR - 1) / TPR;
  constexpr uint32_t SBO = 128;                    // between 8-channel groups (M / N direction)
  constexpr uint32_t LBO_A = 16 * 128;             // between 8-voxel groups of the A staging tile
  constexpr uint32_t LBO_G = (NX / 8) * 128;       // between 8-voxel groups of the G tile
  unsigned char* sA = smem;                        // 16 voxel groups x 2048 B
  unsigned char* sG = smem + 16 * LBO_A;           // 16 voxel groups x LBO_G
  float* wsum = reinterpret_cast<float*>(sG + 16 * LBO_G);  // [27][COUT], dynamic_default only
  const int tid = threadIdx.x, warp = tid >> 5;
  const __nv_bfloat16* img = static_cast<const __nv_bfloat16*>(a.images);
  const __nv_bfloat16* og = static_cast<const __nv_bfloat16*>(a.out_grad);

  const unsigned d16 = __ldg(static_cast<const unsigned short*>(a.default_value));
  const bool ones = TS && (d16 & 0x7fffu) != 0;
  const uint32_t np = ones ? NX : NP;              // tensor-memory columns of an M group

  const bool dyn = !TS && a.dynamic_default;
  if (dyn) {
    const __nv_bfloat16* flt = static_cast<const __nv_bfloat16*>(a.filters);
    for (int e = tid; e < 27 * COUT; e += 128) {
      const int t = e / COUT, n = e % COUT;
      float s = 0.f;
      for (int ci = 0; ci < CIN; ++ci) s += __bfloat162float(flt[((size_t)t * CIN + ci) * COUT + n]);
      wsum[e] = s;
    }
  }
  if (warp == 0) {
    uint32_t slot = smem_u32(&tmem_base_s), ncols = tmem_cols(NT * np);
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&mbar_s)), "r"(1) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base_s;
  const uint32_t mbar = smem_u32(&mbar_s);
  // D f32, A/B bf16, both operands MN-major (bits 15, 16), N = np, M = 128
  const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((np >> 3) << 17) | ((128u >> 4) << 24);
  const unsigned d32 = d16 | (d16 << 16);
  const uint4 padv = TS ? make_uint4(0, 0, 0, 0) : make_uint4(d32, d32, d32, d32);
  const uint4 zero4 = make_uint4(0, 0, 0, 0);

  uint32_t phase = 0;
  bool alive = true;
  bool first = true;
  float dacc = 0.f;
  unsigned char* a_row = sA + (tid / 8) * LBO_A + (tid % 8) * 16;
  unsigned char* g_row = sG + (tid / 8) * LBO_G + (tid % 8) * 16;
  if constexpr (TS) {   // the column of ones (bfloat16 1.0) behind the channels, zeros up to the width
#pragma unroll
    for (int nc = COUT / 8; nc < NX / 8; ++nc)
      *reinterpret_cast<uint4*>(g_row + nc * SBO) = make_uint4(nc == COUT / 8 ? 0x3f80u : 0u, 0u, 0u, 0u);
  }

  for (int tile = blockIdx.x; tile < ntiles && alive; tile += gridDim.x) {
    const long long v = (long long)tile * 128 + tid;
    const bool vvalid = v < nvox;
    VoxPos pos = {0, 0, 0, 0};
    float gf[COUT];
#pragma unroll
    for (int n = 0; n < COUT; ++n) gf[n] = 0.f;
    if (vvalid) pos = vox_pos<S1>(a, v);
    // out_grad row of this voxel -> G tile (previous tile's MMAs have completed: every round waits)
#pragma unroll
    for (int nc = 0; nc < COUT / 8; ++nc) {
      uint4 x = zero4;
      if (vvalid) x = __ldg(reinterpret_cast<const uint4*>(og + (size_t)v * COUT) + nc);
      *reinterpret_cast<uint4*>(g_row + nc * SBO) = x;
      if (dyn) {
        const unsigned w4[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          gf[nc * 8 + 2 * i] = __uint_as_float(w4[i] << 16);
          gf[nc * 8 + 2 * i + 1] = __uint_as_float(w4[i] & 0xffff0000u);
        }
      }
    }

    // the nine filter columns' source pixels, their base-plane lookups all in flight at once
    int cbase[9], cshift[9];
#pragma unroll
    for (int col = 0; col < 9; ++col) {
      long long base = 0;
      int shift = 0;
      cbase[col] = vvalid && tap_column(a, pos, col / 3, col % 3, base, shift) ? (int)base : -1;
      cshift[col] = pos.depth_abs - 1 - shift;
    }
    // rows of M group rd: requested while the previous group's MMAs run, so only the first group's latency is exposed
    uint4 pre[TPR * KC];
    auto request = [&](int rd) {
#pragma unroll
      for (int tt = 0; tt < TPR; ++tt) {
        const int t = rd * TPR + tt;
        const bool real_tap = t < 27;
        bool ok = false;
        size_t off = 0;
        if (real_tap) {
          const int col = t / 3, ind = cshift[t < 27 ? col : 0] + t % 3;
          ok = cbase[t < 27 ? col : 0] >= 0 && !oob(ind, a.D);
          if (ok) off = (size_t)(cbase[t < 27 ? col : 0] + ind) * CIN;
          if (!ok && dyn && vvalid) {
            // fixed_param_op_gpu.cu.cc:273-277: d(default) += sum_n (sum_ci filter[t][ci][n]) * out_grad[m][n]
            const float* ws = wsum + t * COUT;
#pragma unroll
            for (int n = 0; n < COUT; ++n) dacc = fmaf(ws[n], gf[n], dacc);
          }
        }
#pragma unroll
        for (int kc = 0; kc < KC; ++kc) {
          uint4 x = (real_tap && vvalid) ? padv : zero4;
          if (ok) x = __ldg(reinterpret_cast<const uint4*>(img + off) + kc);
          pre[tt * KC + kc] = x;
        }
      }
    };
    request(0);
#pragma unroll
    for (int rd = 0; rd < NT; ++rd) {
#pragma unroll
      for (int q = 0; q < TPR * KC; ++q) *reinterpret_cast<uint4*>(a_row + q * SBO) = pre[q];
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncthreads();
      if (tid == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {  // 16 voxels (two 8-voxel groups) per MMA
          const uint64_t da = umma_desc(smem_u32(sA + ks * 2 * LBO_A), LBO_A, SBO);
          const uint64_t db = umma_desc(smem_u32(sG + ks * 2 * LBO_G), LBO_G, SBO);
          umma_bf16(tmem + rd * np, da, db, idesc, (first && ks == 0) ? 0u : 1u);
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
      }
      if (rd + 1 < NT) request(rd + 1);
      // one warp polls the mbarrier (every poll is a shared-memory access); the others wait at the hardware barrier
      bool done = true;
      if (warp == 0) done = mbar_wait(mbar, phase);
      phase ^= 1;
      if (!__syncthreads_and(done)) {
        if (tid == 0) note_timeout();
        alive = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }
    first = false;
  }

  // ---- accumulators -> this CTA's partial slab -----------------------------------------------------------------
  constexpr int K = 27 * CIN;
  float* part = static_cast<float*>(a.workspace) + (size_t)blockIdx.x * ((size_t)K * COUT + 1);
  if constexpr (TS) {
    if (ones) {   // this CTA's share of the channel sums of the fine gradient, in a fixed order
      float fs[CIN];
#pragma unroll
      for (int ci = 0; ci < CIN; ++ci) fs[ci] = 0.f;
      for (long long v = (long long)blockIdx.x * 128 + tid; v < a.nvox_in; v += (long long)gridDim.x * 128) {
#pragma unroll
        for (int kc = 0; kc < KC; ++kc) {
          const uint4 x = __ldg(reinterpret_cast<const uint4*>(img + (size_t)v * CIN) + kc);
          const unsigned w4[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            fs[kc * 8 + 2 * i] += __uint_as_float(w4[i] << 16);
            fs[kc * 8 + 2 * i + 1] += __uint_as_float(w4[i] & 0xffff0000u);
          }
        }
      }
#pragma unroll
      for (int ci = 0; ci < CIN; ++ci) {
        for (int o = 16; o > 0; o >>= 1) fs[ci] += __shfl_xor_sync(0xffffffffu, fs[ci], o);
        if ((tid & 31) == 0) red_s[warp * CIN + ci] = fs[ci];
      }
    }
    __syncthreads();
  }
  if (alive) {
#pragma unroll
    for (int rd = 0; rd < NT; ++rd) {
      uint32_t acc[NP];
      if (!first) {
        tmem_ld<NP>(tmem + ((uint32_t)(warp * 32) << 16) + rd * np, acc);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      }
      float add = 0.f;
      if constexpr (TS) {
        if (ones) {
          float seen = 0.f;
          if (!first) {
            uint32_t s8[8];
            tmem_ld<8>(tmem + ((uint32_t)(warp * 32) << 16) + rd * np + COUT, s8);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            seen = __uint_as_float(s8[0]);
          }
          const int ci = (rd * 128 + tid) % CIN;
          add = __uint_as_float(d16 << 16) * ((((red_s[ci] + red_s[CIN + ci]) + red_s[2 * CIN + ci]) + red_s[3 * CIN + ci]) - seen);
        }
      }
      // through shared memory, so that the stores are consecutive (the staging buffer is free; rows of COUT + 1 floats)
      float* rows = reinterpret_cast<float*>(sA);
      __syncthreads();
#pragma unroll
      for (int n = 0; n < COUT; ++n) rows[tid * (COUT + 1) + n] = (first ? 0.f : __uint_as_float(acc[n])) + add;
      __syncthreads();
      for (int e = tid; e < 128 * COUT; e += 128)
        if (rd * 128 + e / COUT < K) part[(size_t)rd * 128 * COUT + e] = rows[(e / COUT) * (COUT + 1) + e % COUT];
    }
  }
  __syncthreads();
  red_s[tid] = dacc;
  __syncthreads();
  for (int o = 64; o > 0; o >>= 1) {
    if (tid < o) red_s[tid] += red_s[tid + o];
    __syncthreads();
  }
  if (tid == 0) part[(size_t)K * COUT] = red_s[0];

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    uint32_t ncols = tmem_cols(NT * np);
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols) : "memory");
  }
}

// ---------------------------------------------------------------------------------------------------------
// Stride-1 filter gradient with the column buffers of sc_umma_rows_kernel (16 gathered channels).
//
// The buffers hold, per 16-byte chunk q = (filter column, channel chunk), the rows of a tile at 16 bytes each -
// which is also the MN-major layout with the voxels as the reduction dimension (LBO = 128: eight voxels per core
// matrix, linear beyond; SBO = the chunk stride).  For a depth tap fz the operand is again the buffer address plus
// fz*16 bytes; out_grad (the other operand) is not shifted and carries zeros in the rows that are not voxels.
// One MMA block of M = 128 covers chunks 0..15 = filter columns 0..7; the ninth column is taken from a second
// block that starts at chunk 2 (columns 1..8, only its last 16 rows are kept) - the tensor pipe is idle anyway
// and no dummy shared memory is needed.  3 depth taps x 2 blocks x COUT tensor-memory columns accumulate over
// all tiles of the CTA.  One barrier per tile instead of four, 9 staged rows per voxel instead of 27.
// TG (transposed convolution) only changes the operand roles, exactly as in sc_umma_wgrad_kernel.
// ---------------------------------------------------------------------------------------------------------
template <int CIN, int COUT, bool TG>
__global__ void __launch_bounds__(128, 4) sc_umma_wgrad_rows_kernel(const ScArgs a, const int ntiles, const int PT) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) uint64_t mbar_s;
  __shared__ uint32_t tmem_base_s;
  __shared__ float red_s[128];
  constexpr int KC = CIN / 8;                      // 1 or 2
  constexpr int NBLK = KC;                         // eight channels: one block holds all nine columns
  constexpr int NRB = 132;                         // as in sc_umma_rows_kernel
  constexpr uint32_t X_SBO = NRB * 16;             // chunk stride (M direction)
  constexpr uint32_t X_LBO = 128;                  // eight voxels further (reduction direction): rows are linear
  // out_grad tile with the three depth taps side by side in N: chunk fz*(COUT/8) + nc of voxel group m'/8 holds
  // channels nc*8.. of out_grad row m' - fz, so ONE MMA with N = 3*COUT per 16 tile rows serves the three taps
  // (an N = 16 MMA costs the issuing thread as much as an N = 48 one, and that thread is the tile's critical path)
  constexpr int NCH = (3 * (COUT / 8) + 1) / 2 * 2;   // 16-byte chunks per row of the widened tile (N a multiple of 16)
  constexpr int NP = NCH * 8;                      // tensor-memory columns of a block
  constexpr uint32_t G_SBO = 128, G_LBO = NCH * 128;
  constexpr int TMEM_COLS = NBLK * NP <= 32 ? 32 : (NBLK * NP <= 64 ? 64 : (NBLK * NP <= 128 ? 128 : 256));
  unsigned char* sX = smem;                        // 18 chunks x NRB rows x 16 B
  unsigned char* sG = smem + 18 * X_SBO;           // 16 voxel groups x G_LBO
  float* wsum = reinterpret_cast<float*>(sG + 16 * G_LBO);   // [27][COUT], dynamic_default only
  const int tid = threadIdx.x, warp = tid >> 5;
  const __nv_bfloat16* img = static_cast<const __nv_bfloat16*>(a.images);
  const __nv_bfloat16* og = static_cast<const __nv_bfloat16*>(a.out_grad);

  const bool dyn = !TG && a.dynamic_default;
  if (dyn) {
    const __nv_bfloat16* flt = static_cast<const __nv_bfloat16*>(a.filters);
    for (int e = tid; e < 27 * COUT; e += 128) {
      const int t = e / COUT, n = e % COUT;
      float sum = 0.f;
      for (int ci = 0; ci < CIN; ++ci) sum += __bfloat162float(flt[((size_t)t * CIN + ci) * COUT + n]);
      wsum[e] = sum;
    }
  }
  // rows 0 (tap 1) and 0, 1 (tap 2) of the widened out_grad tile have no source row: zero, once
  if (tid < 3 * (COUT / 8)) {
    const int which = tid / (COUT / 8), nc = tid % (COUT / 8);          // (tap 1,row 0), (tap 2,row 0), (tap 2,row 1)
    const int fz = which == 0 ? 1 : 2, row = which == 2 ? 1 : 0;
    *reinterpret_cast<uint4*>(sG + (fz * (COUT / 8) + nc) * G_SBO + row * 16) = make_uint4(0, 0, 0, 0);
  }
  for (int e = tid; e < 18 * (NRB - 128); e += 128)   // rows 128..135: only multiplied by zero rows of out_grad, but
    *reinterpret_cast<uint4*>(sX + (e / (NRB - 128)) * X_SBO + (128 + e % (NRB - 128)) * 16) = make_uint4(0, 0, 0, 0);  // must be finite
  if (warp == 0) {
    uint32_t slot = smem_u32(&tmem_base_s), ncols = TMEM_COLS;
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&mbar_s)), "r"(1) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base_s;
  const uint32_t mbar = smem_u32(&mbar_s);
  // D f32, A/B bf16, both operands MN-major (bits 15, 16), N = COUT, M = 128
  constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((uint32_t)NCH << 17) |
                             ((128u >> 4) << 24);
  const unsigned d16 = __ldg(static_cast<const unsigned short*>(a.default_value));
  const unsigned d32 = d16 | (d16 << 16);
  const uint4 padv = make_uint4(d32, d32, d32, d32);
  const uint4 zero4 = make_uint4(0, 0, 0, 0);

  const int H = a.H, W = a.W, D = a.D, RP = D + 2;
  const long long npix = (long long)a.B * H * W;
  const int p_in_tile = tid / RP, j = tid - p_in_tile * RP;
  const bool row_used = p_in_tile < PT;
  uint32_t phase = 0;
  bool alive = true, first = true;
  float dacc = 0.f;

  // This thread's row of a tile: its pixel, its out_grad row (zeros for rows that are not voxels) and its source
  // voxel (or -1) in each of the nine filter columns (as in sc_umma_rows_kernel).
  bool rvalid = false;
  int sv[9];                                         // -1 = padding, -2 = row not in the tile
  unsigned padmask = 0;                              // bit col: this row of column col is padding
  uint4 gx[COUT / 8];
  auto locate = [&](int tile) {
    const long long pix = (long long)tile * PT + p_in_tile;
    rvalid = row_used && tile < ntiles && pix < npix;
    const bool is_voxel = rvalid && j < D;          // rows j = D, D+1 of a pixel are halo rows, not output voxels
    int b = 0, r = 0, c = 0, bp_out = 0;
    if (rvalid) {
      const unsigned p32 = (unsigned)pix;   // pixel counts are validated to fit 31 bits
      c = (int)(p32 % (unsigned)W);
      const unsigned t = p32 / (unsigned)W;
      r = (int)(t % (unsigned)H);
      b = (int)(t / (unsigned)H);
      bp_out = __ldg(a.base_plane + pix);
    }
#pragma unroll
    for (int nc = 0; nc < COUT / 8; ++nc) {
      gx[nc] = zero4;
      if (is_voxel) gx[nc] = __ldg(reinterpret_cast<const uint4*>(og + ((size_t)pix * D + j) * COUT) + nc);
    }
    padmask = 0;
#pragma unroll
    for (int col = 0; col < 9; ++col) {
      const int orow = r - 1 + col / 3, ocol = c - 1 + col % 3;
      const bool inb = rvalid && !oob(orow, H) && !oob(ocol, W);
      const int np = inb ? (b * H + orow) * W + ocol : 0;
      const int plane = j - 1 + bp_out - __ldg(a.base_plane + np);
      const bool ok = inb && !oob(plane, D);
      sv[col] = ok ? np * D + plane : (rvalid ? -1 : -2);
      if (!ok) padmask |= 1u << col;
    }
  };
  locate(blockIdx.x);
  const uint64_t da0 = umma_desc(smem_u32(sX), X_LBO, X_SBO);
  const uint64_t db0 = umma_desc(smem_u32(sG), G_LBO, G_SBO);

  for (int tile = blockIdx.x; tile < ntiles && alive; tile += gridDim.x) {
    // this thread's out_grad row m goes to row m + fz of tap block fz (rows 126, 127 are never voxels)
#pragma unroll
    for (int fz = 0; fz < 3; ++fz) {
      const int m = tid + fz;
      if (m < 128) {
        unsigned char* g_row = sG + (m / 8) * G_LBO + (m % 8) * 16 + fz * (COUT / 8) * G_SBO;
#pragma unroll
        for (int nc = 0; nc < COUT / 8; ++nc) *reinterpret_cast<uint4*>(g_row + nc * G_SBO) = gx[nc];
      }
    }
    const bool rvalid_cur = rvalid;
    const unsigned padmask_cur = padmask;
    // the two 16-byte chunks of a row are fetched by neighbouring lanes (see sc_umma_rows_kernel)
    uint4 val[9][KC];
    const int lane = tid & 31, chunk = lane % KC, lrow = lane / KC;
#pragma unroll
    for (int col = 0; col < 9; ++col) {
#pragma unroll
      for (int i = 0; i < KC; ++i) {
        const int sr = KC == 1 ? sv[col] : __shfl_sync(0xffffffffu, sv[col], lrow + i * (32 / KC));
        val[col][i] = sr == -2 ? zero4 : padv;
        if (sr >= 0) val[col][i] = __ldg(reinterpret_cast<const uint4*>(img + (size_t)sr * CIN) + chunk);
      }
    }
    locate(tile + gridDim.x);   // the next tile's lookups and out_grad row run while this tile's rows are in flight
#pragma unroll
    for (int col = 0; col < 9; ++col) {
      unsigned char* dx = sX + (col * KC + chunk) * X_SBO + (warp * 32 + lrow) * 16;
#pragma unroll
      for (int i = 0; i < KC; ++i) *reinterpret_cast<uint4*>(dx + i * (32 / KC) * 16) = val[col][i];
    }

    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int blk = 0; blk < NBLK; ++blk) {
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {   // 16 tile rows (two 8-row groups) per MMA
          const uint64_t da = umma_desc_advance(da0, blk * 2 * X_SBO + ks * 2 * X_LBO);
          const uint64_t db = umma_desc_advance(db0, ks * 2 * G_LBO);
          umma_bf16(tmem + blk * NP, da, db, IDESC, (first && ks == 0) ? 0u : 1u);
        }
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
    }
    if (dyn) {
      // fixed_param_op_gpu.cu.cc:273-277: d(default) += sum_n (sum_ci filter[tap][ci][n]) * out_grad[voxel][n] over the
      // padded taps.  This thread's row j of column col is tap (col, fz) of voxel d = j - fz of the same pixel; the
      // G tile (read here, behind the barrier above) holds that voxel's out_grad row at tile row tid - fz.
      for (int fz = 0; fz < 3; ++fz) {
        const int dv = j - fz;
        if (!rvalid_cur || dv < 0 || dv >= D || padmask_cur == 0) continue;
        const unsigned char* grow = sG + ((tid - fz) / 8) * G_LBO + ((tid - fz) % 8) * 16;
        float gf[COUT];
#pragma unroll
        for (int nc = 0; nc < COUT / 8; ++nc) {
          const uint4 x = *reinterpret_cast<const uint4*>(grow + nc * G_SBO);
          const unsigned w4[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            gf[nc * 8 + 2 * i] = __uint_as_float(w4[i] << 16);
            gf[nc * 8 + 2 * i + 1] = __uint_as_float(w4[i] & 0xffff0000u);
          }
        }
        for (int col = 0; col < 9; ++col) {
          if (!((padmask_cur >> col) & 1u)) continue;
          const float* ws = wsum + (col * 3 + fz) * COUT;
#pragma unroll
          for (int n = 0; n < COUT; ++n) dacc = fmaf(ws[n], gf[n], dacc);
        }
      }
    }
    // one warp polls the mbarrier (every poll is a shared-memory access); the others wait at the hardware barrier
    bool done = true;
    if (warp == 0) done = mbar_wait(mbar, phase);
    phase ^= 1;
    if (!__syncthreads_and(done)) {
      if (tid == 0) note_timeout();
      alive = false;
      break;
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    first = false;
  }

  // ---- accumulators -> this CTA's partial slab [27*CIN][COUT] (+ default-value gradient) -------------------
  constexpr int K = 27 * CIN;
  float* part = static_cast<float*>(a.workspace) + (size_t)blockIdx.x * ((size_t)K * COUT + 1);
  if (alive) {
#pragma unroll
    for (int fz = 0; fz < 3; ++fz) {
#pragma unroll
      for (int blk = 0; blk < NBLK; ++blk) {
        uint32_t acc[COUT];
        if (!first) {
          tmem_ld<COUT>(tmem + ((uint32_t)(warp * 32) << 16) + blk * NP + fz * COUT, acc);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        }
        // MMA row tid of block blk is chunk q = 2*blk + tid/8, element tid%8: column q/2, channel (q%2)*8 + tid%8.
        // Block 0 supplies columns 0..7, block 1 only column 8 (its rows 112..127); with eight channels block 0 holds all nine.
        const int q = 2 * blk + tid / 8;
        const int col = q / KC, ci = (q % KC) * 8 + (tid % 8);
        // Through shared memory (the column buffers are free), so that the stores are consecutive: the CIN rows of
        // (column, tap) are one stretch of the slab.
        float* rows = reinterpret_cast<float*>(sX);
        __syncthreads();
#pragma unroll
        for (int n = 0; n < COUT; ++n)
          if (col < 9) rows[(col * CIN + ci) * (COUT + 1) + n] = first ? 0.f : __uint_as_float(acc[n]);
        __syncthreads();
        for (int e = tid; e < (blk == 0 ? 10 - NBLK : 1) * CIN * COUT; e += 128) {
          const int cc = (blk == 0 ? 0 : 8) + e / (CIN * COUT), w = e % (CIN * COUT);
          part[(size_t)(cc * 3 + fz) * CIN * COUT + w] = rows[(cc * CIN + w / COUT) * (COUT + 1) + w % COUT];
        }
      }
    }
  }
  red_s[tid] = dacc;
  __syncthreads();
  for (int o = 64; o > 0; o >>= 1) {
    if (tid < o) red_s[tid] += red_s[tid + o];
    __syncthreads();
  }
  if (tid == 0) part[(size_t)K * COUT] = red_s[0];

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    uint32_t ncols = TMEM_COLS;
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols) : "memory");
  }
}

template <int CIN, int COUT, bool TG>
int launch_wgrad_rows(const ScArgs& a, int nparts, cudaStream_t st) {
  auto k = sc_umma_wgrad_rows_kernel<CIN, COUT, TG>;
  const size_t smem = (size_t)18 * 132 * 16 + (size_t)16 * ((3 * (COUT / 8) + 1) / 2 * 2) * 128 + (size_t)27 * COUT * 4 + 1024;
  if (int e = grant_smem(k, smem)) return e;
  const int PT = 128 / (a.D + 2);
  const long long npix = (long long)a.B * a.H * a.W;
  const long long ntiles = (npix + PT - 1) / PT;
  if (nparts > ntiles) nparts = (int)ntiles;
  k<<<nparts, 128, smem, st>>>(a, (int)ntiles, PT);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return (int)e;
  return sc_slab_reduce(static_cast<const float*>(a.workspace), nparts, 27, CIN, COUT, TG, static_cast<float*>(a.filter_grad),
                        TG ? nullptr : static_cast<float*>(a.default_grad), st);
}

template <int CIN, int COUT, bool TS>
int launch_wgrad(const ScArgs& a, int nparts, cudaStream_t st) {
  const bool s1 = a.sr == 1 && a.sc == 1 && a.sd == 1;
  if constexpr (CIN <= 16 && !TS) {
    if (s1 && a.D + 2 <= 128 && g_umma_rows.load()) return launch_wgrad_rows<CIN, COUT, false>(a, nparts, st);
  }
  auto k = s1 ? sc_umma_wgrad_kernel<CIN, COUT, TS, true> : sc_umma_wgrad_kernel<CIN, COUT, TS, false>;
  const size_t smem = (size_t)16 * 2048 + (size_t)16 * (wgrad_width<TS>(COUT) / 8) * 128 + (TS ? 0 : (size_t)27 * COUT * 4) + 1024;
  if (int e = grant_smem(k, smem)) return e;
  const int ntiles = (int)((a.nvox_out + 127) / 128);
  if (nparts > ntiles) nparts = ntiles;  // a persistent CTA per slab: more CTAs than tiles would leave slabs unwritten
  k<<<nparts, 128, smem, st>>>(a, a.nvox_out, ntiles);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return (int)e;
  return sc_slab_reduce(static_cast<const float*>(a.workspace), nparts, 27, CIN, COUT, false, static_cast<float*>(a.filter_grad),
                        TS ? nullptr : static_cast<float*>(a.default_grad), st);
}

template <int CIN, int COUT, bool DGRAD>
int launch_rows(const ScArgs& a, cudaStream_t st) {
  auto k = sc_umma_rows_kernel<CIN, COUT, DGRAD>;
  const size_t smem = (size_t)27 * pad16(COUT) * pad16(CIN) * 2 + (size_t)9 * (pad16(CIN) / 8) * 132 * 16 + 1024;
  if (int e = grant_smem(k, smem)) return e;
  const int PT = 128 / (a.D + 2);
  const long long npix = (long long)a.B * a.H * a.W;
  const long long ntiles = (npix + PT - 1) / PT;
  int per_sm = (int)((size_t)220 * 1024 / (smem + 2048));
  if (per_sm > 8) per_sm = 8;
  if (per_sm < 1) per_sm = 1;
  long long grid = 148LL * per_sm;
  if (grid > ntiles) grid = ntiles;
  k<<<(unsigned)grid, 128, smem, st>>>(a, (int)ntiles, PT);
  return (int)cudaGetLastError();
}


// Strided image gradient / transposed convolution (c4 band 256x320x9, 16 -> 16, strides (2,2,2): 38 us,
// against 75 us with all 27 taps gathered per voxel; bound by the index arithmetic of the gather).
template <int CIN, int COUT>
int launch_class(const ScArgs& a, cudaStream_t st) {
  auto k = sc_umma_class_kernel<CIN, COUT>;
  constexpr size_t smem = class_smem(CIN, COUT);
  if (int e = grant_smem(k, smem)) return e;
  const long long ntiles = class_tiles(a, 128);
  constexpr long long slots = 148LL * class_ctas(CIN, COUT);
  const long long grid = ntiles < slots ? ntiles : slots;
  k<<<(unsigned)grid, 128, smem, st>>>(a, (int)ntiles);
  return (int)cudaGetLastError();
}

template <int CIN, int COUT, bool DGRAD>
int launch(const ScArgs& a, long long nvox, cudaStream_t st) {
  const bool s1 = a.sr == 1 && a.sc == 1 && a.sd == 1;
  if (s1 && g_umma_rows.load() == 1 && sc_band_better(a, CIN, COUT)) return sc_band_launch(a, DGRAD, st);
  // otherwise at stride 1, for bands of at most 126 planes: the shifted-row kernel
  if (s1 && a.D + 2 <= 128 && g_umma_rows.load()) return launch_rows<CIN, COUT, DGRAD>(a, st);
  if constexpr (DGRAD) {
    if (!s1 && g_umma_rows.load() == 1 && sc_up_supported(2, a)) return sc_up_launch(a, st);   // 256x320x9: 37 -> 26 us, see there
    if (!s1) return launch_class<CIN, COUT>(a, st);
  }
  auto k = s1 ? sc_umma_kernel<CIN, COUT, DGRAD, true> : sc_umma_kernel<CIN, COUT, DGRAD, DGRAD>;
  const size_t smem = (size_t)27 * pad16(COUT) * pad16(CIN) * 2 + (size_t)9 * 128 * pad16(CIN) * 2 + 1024;
  if (int e = grant_smem(k, smem)) return e;
  const int ntiles = (int)((nvox + 127) / 128);
  int per_sm = (int)((size_t)220 * 1024 / (smem + 2048));
  if (per_sm > 8) per_sm = 8;
  if (per_sm < 1) per_sm = 1;
  int grid = 148 * per_sm;
  if (grid > ntiles) grid = ntiles;
  k<<<grid, 128, smem, st>>>(a, nvox, ntiles);
  return (int)cudaGetLastError();
}

}  // namespace

bool sc_umma_supported(int dtype, const ScArgs& a) {
  return dtype == 2 && a.fh == 3 && a.fw == 3 && a.fd == 3 && a.dr == 1 && a.dc == 1 && a.dd == 1 &&
         (a.Cin == 8 || a.Cin == 16 || a.Cin == 32) && (a.Cout == 8 || a.Cout == 16 || a.Cout == 32) && a.nvox_in < ((long long)1 << 31) - 128;
}

#define CHOP_UMMA_PAIRS(CASE) \
  CASE(8, 8) CASE(8, 16) CASE(8, 32) CASE(16, 8) CASE(16, 16) CASE(16, 32) CASE(32, 8) CASE(32, 16) CASE(32, 32)

int sc_umma_fwd_launch(const ScArgs& a, cudaStream_t st) {
#define CHOP_CASE(I, O) if (a.Cin == I && a.Cout == O) return launch<I, O, false>(a, a.nvox_out, st);
  CHOP_UMMA_PAIRS(CHOP_CASE)
#undef CHOP_CASE
  return -4;
}

// gathers out_grad (Cout channels) and produces images_grad (Cin channels)
int sc_umma_dgrad_launch(const ScArgs& a, cudaStream_t st) {
#define CHOP_CASE(I, O) if (a.Cin == I && a.Cout == O) return launch<O, I, true>(a, a.nvox_in, st);
  CHOP_UMMA_PAIRS(CHOP_CASE)
#undef CHOP_CASE
  return -4;
}

// nparts partial slabs of (27*Cin*Cout + 1) floats must fit in the workspace; every CTA writes one.
int sc_umma_wgrad_launch(const ScArgs& a, int nparts, cudaStream_t st) {
#define CHOP_CASE(I, O) if (a.Cin == I && a.Cout == O) return launch_wgrad<I, O, false>(a, nparts, st);
  CHOP_UMMA_PAIRS(CHOP_CASE)
#undef CHOP_CASE
  return -4;
}

// Filter gradient of the transposed convolution; a.images = its coarse input (Cout channels), a.out_grad = the fine
// upstream gradient (Cin channels), nparts slabs of 27*Cin*Cout + 1 floats in the workspace.  Stride 1 with 8 or 16 coarse
// channels: the shifted-row kernel over the fine grid; otherwise the swapped roles (see sc_umma_wgrad_kernel).
int sc_umma_twgrad_launch(const ScArgs& a, int nparts, cudaStream_t st) {
  if (a.Cout <= 16 && a.sr == 1 && a.sc == 1 && a.sd == 1 && a.D + 2 <= 128 && g_umma_rows.load()) {
#define CHOP_CASE(I, O) if (a.Cin == I && a.Cout == O) return launch_wgrad_rows<O, I, true>(a, nparts, st);
    CHOP_CASE(8, 8) CHOP_CASE(16, 8) CHOP_CASE(32, 8) CHOP_CASE(8, 16) CHOP_CASE(16, 16) CHOP_CASE(32, 16)
#undef CHOP_CASE
  }
  ScArgs w = a;
  w.images = a.out_grad;
  w.out_grad = a.images;
#define CHOP_CASE(I, O) if (a.Cin == I && a.Cout == O) return launch_wgrad<I, O, true>(w, nparts, st);
  CHOP_UMMA_PAIRS(CHOP_CASE)
#undef CHOP_CASE
  return -4;
}

void sc_umma_set_rows(int on) { g_umma_rows = on; }

int sc_umma_timeouts() {
  const int here = timeouts_here(), band = sc_band_timeouts(), up = sc_up_timeouts();
  return here < 0 || band < 0 || up < 0 ? -1 : here + band + up;
}

namespace {
std::mutex g_watch_mu;
int* g_watch_host = nullptr;          // mapped pinned int, shared by all devices of the process
unsigned long long g_watch_devs = 0;  // devices that know its address (bit = device ordinal, < 64)
}  // namespace

// Number of abandoned waits seen through the host-visible mirror; -1 if it cannot be set up.  The first call per
// device allocates (once per process) and publishes the mirror, on a stream of its own and with this thread's capture mode
// relaxed: a program may make its first call while a stream is being captured.  Later calls read host memory.
int sc_umma_watch() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -1;
  std::lock_guard<std::mutex> lk(g_watch_mu);
  if (g_watch_host && ((g_watch_devs >> dev) & 1ull)) return *const_cast<volatile int*>(g_watch_host);
  struct Relaxed {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
  } relaxed;
  if (!g_watch_host) {
    int* h = nullptr;
    if (cudaHostAlloc(reinterpret_cast<void**>(&h), sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) {
      cudaGetLastError();
      return -1;
    }
    *h = 0;
    g_watch_host = h;
  }
  int* dptr = nullptr;
  cudaStream_t st = nullptr;
  bool ok = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) == cudaSuccess;
  ok = ok && cudaHostGetDevicePointer(reinterpret_cast<void**>(&dptr), g_watch_host, 0) == cudaSuccess &&
       publish_mirror_here(dptr, st) == cudaSuccess && sc_band_publish_mirror(dptr, st) == 0 && sc_up_publish_mirror(dptr, st) == 0;
  if (st) cudaStreamDestroy(st);
  if (!ok) {
    cudaGetLastError();
    return -1;
  }
  g_watch_devs |= 1ull << dev;
  return *const_cast<volatile int*>(g_watch_host);
}

// Test facility (behind the tuning opt-in): on != 0 runs the give-up bookkeeping once (default stream), without any wait;
// on == 0 clears the device counter of the current device and the mirror.
int sc_umma_note_timeout_for_test(int on) {
  if (on) {
    note_timeout_kernel<<<1, 1>>>();
    return (int)cudaGetLastError();
  }
  if (clear_timeouts_here() != cudaSuccess || sc_band_clear_timeouts() != 0 || sc_up_clear_timeouts() != 0) return (int)cudaGetLastError();
  std::lock_guard<std::mutex> lk(g_watch_mu);
  if (g_watch_host) *const_cast<volatile int*>(g_watch_host) = 0;
  return 0;
}

}  // namespace chop
