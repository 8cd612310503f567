// Strided gather form on the tensor cores with every coarse voxel staged once: the transposed convolution and the image gradient
// of the strided one, 3x3x3, strides 2 along rows and columns and 1 or 2 along depth, bfloat16 and float32 (in three pieces, as in
// sc_band.cu), float32 accumulation, 8 or 16 produced channels.
//
// Row r and column c of a fine voxel decide which filter columns exist there: (fr, fc) belongs to class (fr != 1, fc != 1) of
// (r mod 2, c mod 2) and reads the coarse pixel (r/2 + (fr == 2), c/2 + (fc == 2)).  So the four fine pixels over one coarse pixel
// read the 2x2 coarse pixels from there on, and the nine columns are spread over the four.  A tile is PT coarse pixels of a row;
// the 2 x (PT+1) around them are staged once, as windows of RP absolute coarse planes (as in sc_band.cu), and each of the four
// offsets is ONE operand for all classes that use it: the accumulators of the classes (1,0), (1,1), (0,1), (0,0) lie side by side, so the
// offsets (0,0), (1,0), (0,1) and (1,1) are MMAs over four, two, two and one of them, each three depth taps wide.
// Depth: accumulator row zc holds, per tap fz, the product with coarse plane zc.  At depth stride 2 the fine plane 2*zc is tap 1 of
// row zc, 2*zc + 1 is tap 0 of row zc plus tap 2 of row zc + 1; at depth stride 1 rows z-1, z, z+1 add up.
// What a tap reads that does not exist (default_value, zero in gradients) is a constant per class and parity, added at the end.
// Base planes that do not fit the window take further passes, with the window moved.  A tile that would need a fifth is "rough" (no depth
// map) and left for the end: there the operand of each of its nine (offset, class) pairs - filter columns - is staged by itself, every
// fine pixel's rows from the first coarse plane that its own taps read, SL columns at a time.
// Bound: a tile's chain of staging, MMAs and epilogue (48 accumulator columns per class and row) at two CTAs of eight warps an SM: no pipe
// is above half (bfloat16 16 <- 16: load-store data 43 %, issue 44 %, operands 7 %; float32 43, 40, 22), the largest stall is the barrier
// (2.1 and 3.6 of 8 and 9 cycles an instruction).  Transposed forward, 256x320x9, bfloat16, strides (2,2,2), us with a gather
// per tap and class (sc_umma_class_kernel) and here, replayed from a graph: 16 <- 16 channels 37, 26; 16 <- 32 71, 30; 8 <- 8 32, 21; at 17
// planes 60, 29; strides (2,2,1) 39, 31; 60x75x12 11, 7.  With 32 produced channels the accumulators do not fit twice: those stay there.
// Base planes that vary: smooth / smooth with up to eight planes of noise on it / random, us of the gather | here with one pass more for
// every pixel that does not fit | with rough tiles.  256x320x9, bfloat16: (2,2,2) 16 <- 16 40 / 40 / 38 | 34 / 36 / 387 | 35 / 37 / 55, 16 <- 32
// 74 / 67 / 65 | 33 / 38 / 496 | 33 / 38 / 84; (2,2,1) 16 <- 16 41 / 40 / 38 | 31 / 63 / 439 | 32 / 64 / 51; float32 (sc_tile.cu, which leaves out
// taps that no voxel of a warp has) (2,2,2) 16 <- 16 155 / 153 / 100 | 76 / 79 / 766 | 77 / 80 / 163.  Two passes and no more: noise
// (2,2,1) 53, but objects with sharp edges in front of a background 40 instead of 37 (36 before, 41 the gather).
#include "sc_entry.h"
#include "sc_umma_common.cuh"
#include "smem_grant.h"

namespace chop {
namespace {

// T: bfloat16, all four classes in one CTA; float32, in three bfloat16 pieces as in sc_band.cu, two of the classes (blockIdx.y), each
// with an accumulator for x1*w1 and one for the five small products.
template <typename T, int CR, int NR, int RP> struct UpGeo {
  static constexpr int P = sizeof(T) == 2 ? 1 : 3, NCLS = P == 1 ? 4 : 2;
  static constexpr int PT = 128 / RP;                 // coarse pixels of a tile
  static constexpr int PW = PT + 1, NPIX = 2 * PW;    // staged coarse pixels
  static constexpr int ROWS = NPIX * RP;
  // filter columns that a rough tile stages at once, of nine; float32 has six (classes 0 and 1) or three
  static constexpr int SL = P == 1 ? (CR <= 16 ? 9 : 5) : 3;
  static constexpr int SROWS = ROWS > SL * 128 ? ROWS : SL * 128, NRB = (SROWS + 7) / 8 * 8 + 4;
  static constexpr int N3 = 3 * pad16(NR), COLS = 4 * N3;
  static constexpr int PIECE = 27 * pad16(NR) * pad16(CR) * 2;   // bytes of the filter's tiles
  static constexpr size_t SMEM = (size_t)P * PIECE + (size_t)P * (pad16(CR) / 8) * NRB * 16 + 1024;
  static constexpr int CTAS = SMEM > 110 * 1024 ? 1 : 2;   // tensor memory: 256 columns each
  static_assert(COLS <= 256 && 4 * PT <= 32, "tile");
};

// The columns of classes 2*half and 2*half + 1 by slot (half < 0: of all); the class of a slot and the coarse pixel that it reads.
__device__ __forceinline__ int up_column(int half, int i) {
  if (half < 0) return i;
  if (half > 0) return i < 2 ? 2 + i : 7;
  return i < 2 ? i : i < 5 ? 2 + i : 8;
}
__device__ __forceinline__ int up_class(int slot) { return slot < 4 ? slot : slot == 4 ? 0 : slot == 7 ? 2 : 1; }
__device__ __forceinline__ int up_below(int slot) { return slot == 4 || slot == 5 || slot == 8; }
__device__ __forceinline__ int up_right(int slot) { return slot >= 6; }
// Tiles of the flipped, channel-swapped filter (stage_filter_tiles) in the order in which the operands use them: per offset
// (di, dj) the classes side by side, three depth taps each.  Slot of filter column (fr, fc):
//   (0,0): classes (1,0) fr 0 fc 1 | (1,1) 0 0 | (0,1) 1 0 | (0,0) 1 1;  (1,0): 2 1 | 2 0;  (0,1): 0 2 | 1 2;  (1,1): 2 2
__device__ __forceinline__ int up_slot(int fr, int fc) {
  const int at[9] = {1, 0, 6, 2, 3, 7, 5, 4, 8};      // [fr*3 + fc]
  return at[fr * 3 + fc];
}

// The sums of the fine pixels `todo` (coarse pixel*4 + class) of a tile by plain multiply-adds: values that are not for the pieces.
// coarse, fine: the tile's tables; skip: as in band_plain.
template <int CR, int NR, int SD, int PW>
__device__ __noinline__ void up_plain(const ScArgs& a, const int2* coarse, const int2* fine, unsigned todo, float pad, bool skip) {
  const float* src = static_cast<const float*>(a.out_grad);
  const float* flt = static_cast<const float*>(a.filters);
  const bool aligned = (reinterpret_cast<size_t>(flt) & 15) == 0;
  const float4 pad4 = make_float4(pad, pad, pad, pad);
  constexpr int N4 = NR / 4;
  for (int e = threadIdx.x; e < 4 * (PW - 1) * a.D * N4; e += 256) {
    const int n = e % N4 * 4, d = e / N4 % a.D, f = e / N4 / a.D;
    if (!((todo >> f) & 1u)) continue;
    const int2 o = fine[f];
    const bool pr = f % 4 < 2, pc = f % 4 == 1 || f % 4 == 2;
    float s[4] = {0.f, 0.f, 0.f, 0.f};
    for (int t = 0; t < 27; ++t) {
      const int fr = t / 9, fc = t / 3 % 3, od = d + o.y - 1 + t % 3;
      const int2 c = coarse[(fr == 2 ? PW : 0) + f / 4 + (fc == 2)];
      const int plane = (SD == 1 ? od : od >> 1) - c.y;
      const bool in = (fr != 1) == pr && (fc != 1) == pc && (SD == 1 || (od & 1) == 0) && c.x >= 0 && !oob(plane, a.oD);
      if (!in && skip) continue;
      const float4* x = reinterpret_cast<const float4*>(src + (size_t)(in ? c.x + plane : 0) * CR);
      const float* w = flt + ((size_t)(26 - t) * NR + n) * CR;
#pragma unroll 1
      for (int k = 0; k < CR; k += 4) plain_fma<false>(s, in ? __ldg(x + k / 4) : pad4, w + k, CR, aligned);
    }
    *reinterpret_cast<float4*>(static_cast<float*>(a.images_grad) + ((size_t)o.x + d) * NR + n) = make_float4(s[0], s[1], s[2], s[3]);
  }
}

template <typename T, int CR, int NR, int RP, int SD>
__global__ void __launch_bounds__(256, (UpGeo<T, CR, NR, RP>::CTAS)) sc_up_kernel(const ScArgs a, const int ntiles, const int tiles_w) {
  extern __shared__ __align__(1024) unsigned char smem[];
  typedef UpGeo<T, CR, NR, RP> G;
  constexpr int PT = G::PT, PW = G::PW, NPIX = G::NPIX, NRB = G::NRB, N3 = G::N3, P = G::P, NCLS = G::NCLS;
  constexpr int CIN = pad16(CR), COUT = pad16(NR), KC = CIN / 8, KR = CR / 8;
  __shared__ __align__(8) uint64_t mbar_s;
  __shared__ uint32_t tmem_base_s;
  __shared__ int2 coarse_s[3][NPIX];                    // first voxel (-1: outside the image), first absolute coarse plane
  __shared__ int2 fine_s[3][4 * PT];                    // per fine pixel [coarse pixel][class]: first voxel (-1: none), base plane
  __shared__ unsigned top_s[4];                         // float32: largest magnitude of a step, three steps in turn; the filter's
  __shared__ unsigned rough_s[2];                       // rough tiles: a bit each, the last for all from the 64th on
  __shared__ float pad_s[4][2][NR];                     // class, parity: what the taps that do not exist add
  constexpr uint32_t B_LBO = 128, B_SBO = KC * 128;
  constexpr uint32_t A_LBO = NRB * 16, A_SBO = 128;
  constexpr int B_TAP_BYTES = COUT * CIN * 2;
  unsigned char* sB = smem;
  unsigned char* sX = smem + P * G::PIECE;              // [piece][K-chunk][row]
  const int half = P == 1 ? 0 : blockIdx.y;             // float32: classes 2*half, 2*half + 1
  const int tid = threadIdx.x, lane = tid & 31;
  const T* src = static_cast<const T*>(a.out_grad);
  T* dst = static_cast<T*>(a.images_grad);
  const int H = a.H, W = a.W, D = a.D, oD = a.oD;

  if (KR < KC)   // the padding channels stay zero
    for (int e = tid; e < P * G::SROWS; e += 256)
      *reinterpret_cast<uint4*>(sX + (e / G::SROWS * KC + 1) * A_LBO + e % G::SROWS * 16) = make_uint4(0, 0, 0, 0);
  if (tid < 32) {
    uint32_t slot = smem_u32(&tmem_base_s), ncols = 256;
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&mbar_s)), "r"(1) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  float padf = 0.f;
  uint4 padv = make_uint4(0, 0, 0, 0);                  // 16 bytes of padding values
  if (!a.pad_zero) {
    unsigned d32;
    if constexpr (P == 1) {
      const unsigned d16 = __ldg(static_cast<const unsigned short*>(a.default_value));
      padf = __uint_as_float(d16 << 16);
      d32 = d16 | (d16 << 16);
    } else {
      padf = __ldg(static_cast<const float*>(a.default_value));
      d32 = __float_as_uint(padf);
    }
    padv = make_uint4(d32, d32, d32, d32);
  }
  const bool padded = padf != 0.f;                      // also where it is not a number

  // this thread's entry of a tile's tables: a coarse pixel (tid < NPIX) or a fine one (tid - 64 < 4*PT)
  auto entry = [&](int tile) {
    int2 e = make_int2(-1, 0);
    if (tile >= ntiles) return e;
    const int tw = tile % tiles_w, t = tile / tiles_w, i = t % a.oH, b = t / a.oH;
    if (tid < NPIX) {
      const int ci = i + tid / PW, cj = tw * PT + tid % PW;
      if (ci < a.oH && cj < a.oW) {
        const int bp = __ldg(a.base_plane + (b * H + 2 * ci) * W + 2 * cj);
        e = make_int2(((b * a.oH + ci) * a.oW + cj) * oD, (bp + SD - 1) / SD);   // as in sc_tap_t
      }
    } else if (tid >= 64 && tid < 64 + 4 * PT) {
      const int f = tid - 64, q = f / 4, cls = f % 4;   // classes in the accumulators' order
      const int r = 2 * i + (cls < 2), c = 2 * (tw * PT + q) + (cls == 1 || cls == 2);
      if (r < H && c < W) {
        const int pix = (b * H + r) * W + c;
        e = make_int2(pix * D, __ldg(a.base_plane + pix));
      }
    }
    return e;
  };
  auto keep = [&](int buf, const int2& e) {
    if (tid < NPIX) coarse_s[buf][tid] = e;
    else if (tid >= 64 && tid < 64 + 4 * PT) fine_s[buf][tid - 64] = e;
  };
  struct Step {   // one staging and its MMAs: a pass over a tile; the same in every thread
    int tile, z0;
    unsigned now, left;   // fine pixels of this pass, still to do
  };
  auto floor_sd = [](int x) { return SD == 1 ? x : x >> 1; };
  auto window = [&](Step& s, const int2& e) {   // lane i: fine pixel i
    const int lo = floor_sd(e.y - 1), hi = floor_sd(e.y + D);   // coarse planes that its taps read
    s.z0 = __reduce_min_sync(0xffffffffu, (s.left >> lane) & 1u ? lo : 0x7fffffff);
    s.now = __ballot_sync(0xffffffffu, ((s.left >> lane) & 1u) && (unsigned)hi - (unsigned)s.z0 < (unsigned)RP);
    if (s.now == 0) s.now = s.left;   // base planes at the ends of the integers: the passes end all the same
    s.left &= ~s.now;
  };
  auto fine_entry = [&](int buf) { return lane < 4 * PT ? fine_s[buf][lane] : make_int2(-1, 0); };
  auto open = [&](Step& s, int buf) -> unsigned {       // the fine pixels of a rough tile, which gets none here; otherwise zero
    const int2 e = fine_entry(buf);
    s.left = __ballot_sync(0xffffffffu, e.x >= 0 && (P == 1 || lane % 4 / 2 == half));
    const unsigned all = s.left;
    window(s, e);
    if (s.left == 0) return 0;
    Step t = s;
    for (int pass = 1; pass < 4 && t.left != 0; ++pass) window(t, e);
    if (t.left == 0) return 0;
    s.now = s.left = 0;
    return all;
  };
  constexpr int NI = (G::ROWS * KR + 255) / 256, RSTEP = 256 / KR;
  const int chunk = tid % KR, row0 = tid / KR;
  constexpr int VEC = (int)sizeof(T) / 2;               // 16-byte words of a chunk of eight channels
  uint4 val[NI][VEC];
  auto request = [&](const Step& s, int buf) {
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const int row = row0 + i * RSTEP;
#pragma unroll
      for (int k = 0; k < VEC; ++k) val[i][k] = padv;
      if ((i + 1) * RSTEP > G::ROWS && row >= G::ROWS) continue;
      const int2 e = coarse_s[buf][row / RP];
      const int plane = row % RP + s.z0 - e.y;
      if (e.x >= 0 && !oob(plane, oD)) {
#pragma unroll
        for (int k = 0; k < VEC; ++k) val[i][k] = __ldg(reinterpret_cast<const uint4*>(src + (size_t)(e.x + plane) * CR) + chunk * VEC + k);
      }
    }
  };

  Step cur, nxt;
  cur.tile = blockIdx.x;
  int2 ahead = entry(cur.tile);
  keep(0, ahead);
  __syncthreads();
  auto mark = [&](int tile) {                           // a rough tile of this CTA, by their order
    const int turn = min((tile - (int)blockIdx.x) / (int)gridDim.x, 63);
    if (tid == 0) rough_s[turn / 32] |= 1u << (turn % 32);
  };
  if (tid == 0) rough_s[0] = rough_s[1] = 0;
  if (open(cur, 0) != 0) mark(cur.tile);
  request(cur, 0);
  ahead = entry(cur.tile + (int)gridDim.x);
  // filter tiles: offset order; the loop of stage_filter_tiles with slots of its own
  unsigned top = 0;
  for (int e = tid; e < 27 * COUT * KC; e += 256) {
    const int kg = e % KC, n = (e / KC) % COUT, t = e / (KC * COUT);
    unsigned char* o = sB + (up_slot(t / 9, t / 3 % 3) * 3 + t % 3) * B_TAP_BYTES + (n / 8) * B_SBO + kg * B_LBO + (n % 8) * 16;
    const T* from = static_cast<const T*>(a.filters) + ((size_t)(26 - t) * NR + n) * CR + kg * 8;
    const bool is = kg * 8 < CR && n < NR;
    if constexpr (P == 1) {
      *reinterpret_cast<uint4*>(o) = is ? __ldg(reinterpret_cast<const uint4*>(from)) : make_uint4(0, 0, 0, 0);
    } else {
      float v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = is ? __ldg(from + i) : 0.f;
      top = max(top, top_bits(v));
      unsigned p[3][4];
      split3(v, p);
#pragma unroll
      for (int q = 0; q < 3; ++q) *reinterpret_cast<uint4*>(o + q * G::PIECE) = make_uint4(p[q][0], p[q][1], p[q][2], p[q][3]);
    }
  }
  unsigned w_top = 0;                                   // float32: the filter's largest magnitude
  bool plain = false;
  if constexpr (P > 1) {
    if (tid < 4) top_s[tid] = 0;
    __syncthreads();
    top = __reduce_max_sync(0xffffffffu, top);
    if (lane == 0) atomicMax(&top_s[3], top);
    __syncthreads();
    w_top = top_s[3];
  }
  for (int e = tid; e < 8 * NR; e += 256) {
    const int n = e % NR, par = e / NR % 2, cls = e / NR / 2, pr = cls < 2, pc = cls == 1 || cls == 2;
    float sum = 0.f;
    if (padded) {
      for (int t = 0; t < 27; ++t) {
        const int fr = t / 9, fc = t / 3 % 3, fz = t % 3;
        if ((fr != 1) == pr && (fc != 1) == pc && (SD == 1 || (fz != 1) == par)) continue;   // the tap exists
        for (int k = 0; k < CR; ++k) sum += ScIo<T>::ld(static_cast<const T*>(a.filters) + ((size_t)(26 - t) * NR + n) * CR + k);
      }
    }
    pad_s[cls][par][n] = padf * sum;
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base_s;
  const uint32_t mbar = smem_u32(&mbar_s);
  auto idesc = [](int n) { return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n * N3 >> 3) << 17) | ((128u >> 4) << 24); };
  const uint64_t da0 = umma_desc(smem_u32(sX), A_LBO, A_SBO);
  const uint64_t db0 = umma_desc(smem_u32(sB), B_LBO, B_SBO);
  uint32_t phase = 0;
  int buf = 0;
  auto next = [](int b) { return b == 2 ? 0 : b + 1; };

  auto put = [&](int row, const uint4 (&v)[VEC]) -> unsigned {   // this thread's chunk of a row; float32: its largest magnitude
    unsigned char* o = sX + chunk * A_LBO + row * 16;
    if constexpr (P == 1) {
      *reinterpret_cast<uint4*>(o) = v[0];
      return 0;
    } else {
      const uint4 lo = v[0], hi = v[VEC - 1];
      const float x[8] = {__uint_as_float(lo.x), __uint_as_float(lo.y), __uint_as_float(lo.z), __uint_as_float(lo.w),
                          __uint_as_float(hi.x), __uint_as_float(hi.y), __uint_as_float(hi.z), __uint_as_float(hi.w)};
      unsigned p[3][4];
      split3(x, p);
#pragma unroll
      for (int q = 0; q < 3; ++q) *reinterpret_cast<uint4*>(o + q * KC * A_LBO) = make_uint4(p[q][0], p[q][1], p[q][2], p[q][3]);
      return top_bits(x);
    }
  };
  // epilogue of the fine pixels `now`, whose windows begin at first(entry): the classes are dealt out to the two halves of the warps
  auto finish = [&](unsigned now, int buf, auto first) {
    if (now == 0) return;
    constexpr int NE = P == 1 ? NR : 8;                 // channels at a time
    const int m = tid & 127, q = m / RP, w = m % RP;
    if (P > 1 && plain) {
      if constexpr (P > 1) up_plain<CR, NR, SD, PW>(a, coarse_s[buf], fine_s[buf], now, padf, a.pad_zero || (!padded && w_top < 0x7f800000u));
    } else {
#pragma unroll 1
      for (int l = tid / 128 * (NCLS / 2); l < (tid / 128 + 1) * (NCLS / 2); ++l) {
        const int cls = P == 1 ? l : half * 2 + l;
        const int2 e = fine_s[buf][q * 4 + cls];
        const bool mine = (now >> (q * 4 + cls)) & 1u;
#pragma unroll 1
        for (int c0 = 0; c0 < NR; c0 += NE) {
          uint32_t t[P == 1 ? 1 : 2][3][NE];
          const uint32_t col = tmem + ((uint32_t)(m / 32 * 32) << 16) + l * N3 + c0;
#pragma unroll
          for (int g = 0; g < (P == 1 ? 1 : 2); ++g)
#pragma unroll
            for (int fz = 0; fz < 3; ++fz) tmem_ld<NE>(col + g * NCLS * N3 + fz * COUT, t[g][fz]);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          float s[2][NE];
#pragma unroll
          for (int k = 0; k < NE; ++k) {
            float f[3];
#pragma unroll
            for (int fz = 0; fz < 3; ++fz) {
              f[fz] = __uint_as_float(t[0][fz][k]);
              if constexpr (P > 1) f[fz] += __uint_as_float(t[1][fz][k]);
            }
            const float above = __shfl_down_sync(0xffffffffu, f[2], 1);
            if (SD == 1) {
              s[0][k] = __shfl_up_sync(0xffffffffu, f[0], 1) + f[1] + above;
              s[1][k] = 0.f;
            } else {
              s[0][k] = f[1];
              s[1][k] = f[0] + above;
            }
            if (padded) {
              s[0][k] += pad_s[cls][0][c0 + k];
              s[1][k] += pad_s[cls][1][c0 + k];
            }
          }
#pragma unroll
          for (int p = 0; p < SD; ++p) {
            const int d = (w + first(e)) * SD + p - e.y;
            if (!mine || oob(d, D)) continue;
            T* o = dst + (size_t)(e.x + d) * NR + c0;
            if constexpr (P == 1) {
#pragma unroll
              for (int k = 0; k < NE; k += 8) {
                uint32_t h[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                  const __nv_bfloat162 b2 = __floats2bfloat162_rn(s[p][k + 2 * i], s[p][k + 2 * i + 1]);
                  h[i] = *reinterpret_cast<const uint32_t*>(&b2);
                }
                *reinterpret_cast<uint4*>(o + k) = make_uint4(h[0], h[1], h[2], h[3]);
              }
            } else {
#pragma unroll
              for (int k = 0; k < NE; k += 4) *reinterpret_cast<float4*>(o + k) = make_float4(s[p][k], s[p][k + 1], s[p][k + 2], s[p][k + 3]);
            }
          }
        }
      }
    }
  };

  while (true) {
    const bool again = cur.left != 0;
    // the next step's tables; their buffer was last read two steps ago, before the barrier behind the last staging
    if (again) keep(next(buf), tid < NPIX ? coarse_s[buf][tid] : tid >= 64 && tid < 64 + 4 * PT ? fine_s[buf][tid - 64] : make_int2(0, 0));
    else keep(next(buf), ahead);
    top = 0;
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      if ((i + 1) * RSTEP > G::ROWS && row0 + i * RSTEP >= G::ROWS) continue;
      top = max(top, put(row0 + i * RSTEP, val[i]));
    }
    if constexpr (P > 1) {
      top = __reduce_max_sync(0xffffffffu, top);
      if (lane == 0) atomicMax(&top_s[buf], top);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if constexpr (P > 1) {
      plain = !pieces_fit<CR>(top_s[buf], w_top);
      if (tid == 0) top_s[next(next(buf))] = 0;         // read in the last step, written two steps on
    }
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int k16 = 0; k16 < CIN / 16; ++k16) {
        const uint64_t da = umma_desc_advance(da0, k16 * 2 * A_LBO), db = umma_desc_advance(db0, k16 * 2 * B_LBO);
        auto slot = [&](int s) { return umma_desc_advance(db, s * 3 * B_TAP_BYTES); };
        if constexpr (P > 1) {
          // pieces (p, q): x1*w1 | x1*w2, x2*w1, x1*w3, x2*w2, x3*w1
          constexpr int PQ[6][2] = {{0, 0}, {0, 1}, {1, 0}, {0, 2}, {1, 1}, {2, 0}};
#pragma unroll
          for (int c = 0; c < 6; ++c) {
            const uint64_t dx = umma_desc_advance(da, PQ[c][0] * KC * A_LBO);
            auto piece = [&](int s) { return umma_desc_advance(slot(s), PQ[c][1] * G::PIECE); };
            const uint32_t acc = tmem + (c == 0 ? 0 : NCLS * N3);
            const uint32_t add = k16 != 0 || c > 1 ? 1u : 0u;
            umma_bf16(acc, dx, piece(half == 0 ? 0 : 2), idesc(2), add);
            if (half == 0) {
              umma_bf16(acc, umma_desc_advance(dx, PW * RP * 16), piece(4), idesc(2), 1u);
              umma_bf16(acc + N3, umma_desc_advance(dx, RP * 16), piece(6), idesc(1), 1u);
              umma_bf16(acc + N3, umma_desc_advance(dx, (PW + 1) * RP * 16), piece(8), idesc(1), 1u);
            } else {
              umma_bf16(acc, umma_desc_advance(dx, RP * 16), piece(7), idesc(1), 1u);
            }
          }
          continue;
        }
        umma_bf16(tmem, da, slot(0), idesc(4), k16 != 0 ? 1u : 0u);                                        // offset (0,0): all classes
        umma_bf16(tmem, umma_desc_advance(da, PW * RP * 16), slot(4), idesc(2), 1u);                       // (1,0): (1,0), (1,1)
        umma_bf16(tmem + N3, umma_desc_advance(da, RP * 16), slot(6), idesc(2), 1u);                       // (0,1): (1,1), (0,1)
        umma_bf16(tmem + N3, umma_desc_advance(da, (PW + 1) * RP * 16), slot(8), idesc(1), 1u);            // (1,1): (1,1)
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
    }
    // ---- while they run: the next step's pixels and rows ---------------------------------------------------------
    nxt = cur;
    bool go = true;
    if (!again) {
      nxt.tile = cur.tile + (int)gridDim.x;
      go = nxt.tile < ntiles;
      if (go && open(nxt, next(buf)) != 0) mark(nxt.tile);
    } else {
      window(nxt, fine_entry(next(buf)));
    }
    if (go) {
      request(nxt, next(buf));
      if (!again) ahead = entry(nxt.tile + (int)gridDim.x);
    }
    bool done = true;
    if (tid < 32) done = mbar_wait(mbar, phase);
    phase ^= 1;
    if (!__syncthreads_and(done)) {
      if (tid == 0) note_timeout();
      if (tid == 0) rough_s[0] = rough_s[1] = 0;
      break;
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

    finish(cur.now, buf, [&](const int2&) { return cur.z0; });
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (!go) break;
    cur = nxt;
    buf = next(buf);
  }

  __syncthreads();
  if ((rough_s[0] | rough_s[1]) != 0) {
    const int columns = P == 1 ? 9 : half == 0 ? 6 : 3;
    bool ok = true;
    int turn = 0;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x, turn += turn < 63) {
      if (!((rough_s[turn / 32] >> (turn % 32)) & 1u)) continue;
      __syncthreads();                                  // the tables and the largest magnitude have been read
      keep(0, entry(tile));
      if (tid == 0) top_s[0] = 0;
      __syncthreads();
      Step s;
      const unsigned now = open(s, 0);
      if (now == 0) continue;
      for (int c0 = 0; ok && c0 < columns; c0 += G::SL) {
        const int n = min(G::SL, columns - c0);
        unsigned most = 0;
        for (int row = row0; row < n * 128; row += RSTEP) {
          const int slot = up_column(P == 1 ? -1 : half, c0 + row / 128), q = row % 128 / RP;
          const int2 f = fine_s[0][q * 4 + up_class(slot)], e = coarse_s[0][up_below(slot) * PW + q + up_right(slot)];
          const int plane = floor_sd(f.y - 1) + row % RP - e.y;
          const bool in = f.x >= 0 && e.x >= 0 && !oob(plane, oD);
          uint4 v[VEC];
#pragma unroll
          for (int k = 0; k < VEC; ++k) {
            v[k] = padv;
            if (in) v[k] = __ldg(reinterpret_cast<const uint4*>(src + (size_t)(e.x + plane) * CR) + chunk * VEC + k);
          }
          most = max(most, put(row, v));
        }
        if constexpr (P > 1) {
          most = __reduce_max_sync(0xffffffffu, most);
          if (lane == 0) atomicMax(&top_s[0], most);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        if (tid == 0) {
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          for (int i = 0; i < n; ++i) {                 // columns 0 .. 3 are the first of their classes
            const int slot = up_column(P == 1 ? -1 : half, c0 + i);
            const uint32_t acc = tmem + (up_class(slot) - (P == 1 ? 0 : 2 * half)) * N3;
#pragma unroll
            for (int k16 = 0; k16 < CIN / 16; ++k16) {
              const uint64_t dx = umma_desc_advance(da0, i * 128 * 16 + k16 * 2 * A_LBO);
              const uint64_t dw = umma_desc_advance(db0, slot * 3 * B_TAP_BYTES + k16 * 2 * B_LBO);
              const uint32_t add = slot >= 4 || k16 != 0 ? 1u : 0u;
              umma_bf16(acc, dx, dw, idesc(1), add);
              if constexpr (P > 1) {
#pragma unroll
                for (int p = 0; p < 3; ++p)
#pragma unroll
                  for (int r = p == 0 ? 1 : 0; r < 3 - p; ++r)
                    umma_bf16(acc + NCLS * N3, umma_desc_advance(dx, p * KC * A_LBO), umma_desc_advance(dw, r * G::PIECE), idesc(1), p == 0 && r == 1 ? add : 1u);
              }
            }
          }
          asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
        }
        bool done = true;
        if (tid < 32) done = mbar_wait(mbar, phase);
        phase ^= 1;
        ok = __syncthreads_and(done);
        if (!ok && tid == 0) note_timeout();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      }
      if (!ok) break;
      if constexpr (P > 1) plain = !pieces_fit<CR>(top_s[0], w_top);
      finish(now, 0, [&](const int2& e) { return floor_sd(e.y - 1); });
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (tid < 32) {
    uint32_t ncols = 256;
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols) : "memory");
  }
}

template <typename T, int CIN, int COUT, int RP, int SD>
int launch_up(const ScArgs& a, cudaStream_t st) {
  typedef UpGeo<T, CIN, COUT, RP> G;
  auto k = sc_up_kernel<T, CIN, COUT, RP, SD>;
  if (int e = grant_smem(k, G::SMEM)) return e;
  const int tw = (a.oW + G::PT - 1) / G::PT;
  const long long ntiles = (long long)a.B * a.oH * tw;
  constexpr long long slots = 148LL * G::CTAS * G::NCLS / 4;
  k<<<dim3((unsigned)(ntiles < slots ? ntiles : slots), 4 / G::NCLS), 256, G::SMEM, st>>>(a, (int)ntiles, tw);
  return (int)cudaGetLastError();
}
template <typename T, int CIN, int COUT>
int launch_depth(const ScArgs& a, cudaStream_t st) {
  if (a.sd == 2) return launch_up<T, CIN, COUT, 16, 2>(a, st);
  return a.D <= 10 ? launch_up<T, CIN, COUT, 16, 1>(a, st) : launch_up<T, CIN, COUT, 32, 1>(a, st);
}

}  // namespace

// 3x3x3, dilation 1 and 31-bit voxel counts are the caller's conditions.  Bands of few planes leave most of a window's 16 rows empty; there the
// gather is the faster kernel (us of it and of this one, replayed from a graph):
//   * bfloat16, 16 produced channels, fewer than four planes on large images: 180x230x3 16 <- 16 15.0, 15.9; five planes 18.6, 16.1; 146x180x3
//     14.0, 11.9.  At depth stride 1 fewer than nine planes on very small ones (a tile of eight pixels takes as long as its four
//     classes): 48x60x6 8.2, 9.2, 9 planes 9.4, 9.2; 96x130x6 13.2, 11.2; stride 2 8.2, 6.8.
//   * float32 with eight channels on either side, fewer than five planes (eight on both: six) on large images: 180x230x3 8 <- 8 26.5, 35.9, 8 <- 16
//     30.6, 36.3, 16 <- 8 32.2, 39.6, 16 <- 16 43.5, 41.0; five planes 34.3, 35.7, 39.7, 36.5, 41.2, 39.9; 146x180x3
//     23.9, 24.5, 26.6, 25.8, 28.1, 27.0.
bool sc_up_supported(int dtype, const ScArgs& a) {
  if (a.sr != 2 || a.sc != 2 || a.sd > 2 || a.Cin > 16 || a.D > 24) return false;
  const long long pixels = (long long)a.B * a.H * a.W;
  if (dtype == 0) return pixels < 34000 || a.Cin + a.Cout == 32 || a.D >= (a.Cin + a.Cout == 16 ? 6 : 5);
  if (a.Cin < 16) return true;
  return pixels >= 34000 ? a.D >= 4 || a.Cout > 16 : pixels >= 6000 || a.sd == 2 || a.D >= 9;
}
int sc_up_launch(const ScArgs& a, cudaStream_t st) {
#define CHOP_CASE(I, O) if (a.Cout == I && a.Cin == O) return launch_depth<__nv_bfloat16, I, O>(a, st);
  CHOP_CASE(8, 8) CHOP_CASE(16, 8) CHOP_CASE(32, 8) CHOP_CASE(8, 16) CHOP_CASE(16, 16) CHOP_CASE(32, 16)
#undef CHOP_CASE
  return -4;
}
// float32, where this is faster than sc_tile.cu and no less exact.  Transposed forward, us there and here (produced < gathered):
// strides (2,2,2), 256x320x9 16<16 152, 73; 8<16 96, 62; 16<8 94, 68; 8<8 74, 60; at 17 planes 269, 87; 168, 74; 161, 89; 125, 72;
// (2,2,1) 189x251x7 16<16 79, 46; 8<16 59, 64; 16<8 57, 64; 8<8 47, 58.  (At 17 planes and depth stride 1 but for 16<16 called one by one, the
// others replayed from a graph.)  2-norm of the error against float64: (2,2,2) 16 gathered channels
// 8.6e-8 there, 6.2e-8 here, 8 8.0e-8, 4.7e-8; 32 8.9e-8, 9.5e-8 (and at depth stride 1 slower), so those stay there.
bool sc_up_f32_supported(int dtype, const ScArgs& a) {
  return dtype == 0 && sc_up_supported(dtype, a) && a.fh == 3 && a.fw == 3 && a.fd == 3 && a.dr == 1 && a.dc == 1 && a.dd == 1 &&
         (a.Cin == 8 || a.Cin == 16) && (a.Cout == 16 || (a.Cout == 8 && a.sd == 2)) && (a.sd == 2 || a.Cin == 16) &&
         a.nvox_in < (1LL << 31) - 4096;
}
int sc_up_f32_launch(const ScArgs& a, cudaStream_t st) {
  if (a.Cout == 16 && a.Cin == 16) return launch_depth<float, 16, 16>(a, st);
  if (a.sd != 2) return -4;
  if (a.Cout == 8 && a.Cin == 8) return launch_up<float, 8, 8, 16, 2>(a, st);
  if (a.Cout == 16 && a.Cin == 8) return launch_up<float, 16, 8, 16, 2>(a, st);
  if (a.Cout == 8 && a.Cin == 16) return launch_up<float, 8, 16, 16, 2>(a, st);
  return -4;
}
int sc_up_timeouts() { return timeouts_here(); }
int sc_up_publish_mirror(int* dptr, cudaStream_t st) { return (int)publish_mirror_here(dptr, st); }
int sc_up_clear_timeouts() { return (int)clear_timeouts_here(); }

}  // namespace chop
