// Stride-1 manifold convolution on the tensor cores with every voxel staged ONCE per tile: 3x3x3, dilation 1, bands of up to 24
// planes; bfloat16 with 8, 16 or 32 channels, and float32 (in three bfloat16 pieces, below) where that pays; float32 accumulation.
//
// sc_umma_rows_kernel (sc_umma.cu) stages each neighbour pixel nine times, once per filter column, because a column's rows
// have to be shifted by base_plane[pixel] - base_plane[neighbour].  In ABSOLUTE depth there is no shift: here a tile is
// R x PT output pixels, and the (R+2) x (PT+2) pixels around them are staged once, each as a window of RP rows for the
// absolute planes z0 .. z0+RP-1, default_value where a plane lies outside a pixel's band.  Rows are linear in shared memory
// (SBO = 128), so the A operand of filter column (fr, fc) for the PT pixels of image row r is the stage's address plus
// ((r + fr)*(PT+2) + fc)*RP rows, the same for all 128 MMA rows (PT*RP <= 128).
//   * An M = 128 operand costs the tensor core 32 cycles of shared-memory reads whatever N is, so N is filled: the three
//     depth taps of a column are side by side in N - accumulator row z holds the sums for the taps that read plane z, and the
//     epilogue adds rows z-1, z and z+1 with two shuffles per channel - and so are the filter rows: the staged row hr is
//     filter row fr of output row hr - fr, and the output rows' accumulators lie side by side, last row first.
//   * A pixel's D planes and one on either side must lie in the window: base_plane may vary by RP-2-D over the tile.  A tile
//     that varies more takes a second pass with the window moved; one that would need a third is "rough" (a random base
//     plane, not a depth map) and stages its filter columns one by one, each pixel's rows shifted as in sc_umma_rows_kernel, as many
//     columns a step as shared memory holds beside the other CTAs (all nine of 8 or 16 bfloat16 channels, five otherwise).
//
// Base planes of 64 planes over the image (two sinusoid periods), D = 9: 1.00 passes a tile at 256x320 pixels, 1.4 at 100x125.
// Bound: the shared-memory data pipe (58 % load-store, of which half is the epilogue's tensor-memory reads and shuffles; 32 %
// MMA operands) and, with four CTAs an SM, a tile's chain of staging, MMAs and epilogue.  256x320x9, 3x3x3, bfloat16, us of
// sc_umma_rows_kernel and here, replayed from a graph: 16 -> 16 channels 54, 36, 8 -> 8 47, 27, 32 -> 32 208, 87, 32 -> 16 123, 62; at 17 planes
// 92, 65, 338, 152.
// Tiles of four rows with 256 threads: 45; of one row: 49; windows that do not divide 32 rows (25 for 17 planes): 108.
// Base planes that vary: smooth / smooth with up to eight planes of noise on it / random, us of sc_umma_rows_kernel | with the window's
// rows as the rough tile's buffer | here: 256x320x9 16 -> 16 57 / 56 / 53 | 37 / 96 / 94 | 36 / 65 / 59; 8 -> 8 51 / 50 / 50 | 34 / 73 / 71 |
// 33 / 52 / 49; 32 -> 32 210 / 210 / 198 | 98 / 255 / 250 | 84 / 182 / 176; 16 -> 32 76 / 74 / 70 | 64 / 126 / 123 | 59 / 91 / 84; objects in
// front of a background, sharp edges: 16 -> 16 57 | 49 | 44.  float32 189x251x7 16 -> 16, sc_tile.cu first, which leaves out taps that no voxel
// of a warp has: 138 / 135 / 61 | 81 / 157 / 182 | 75 / 144 / 143.
//
// float32: a value is the exact sum of three bfloat16 pieces, x = x1 + x2 + x3, and x*w the sum of the six products
// x1w1, x1w2, x2w1, x1w3, x2w2, x3w1 (what is left out is below 2^-24 of it).  Steps that the pieces cannot hold (pieces_fit) are
// computed by plain multiply-adds (band_plain).  189x251x7, 16 -> 16 channels: 135 us with a thread per four voxels (sc_tile.cu),
// 127 in runs of planes (sc_run.cu), 71 here; 16 -> 32 320, 238, 140.  Bound: 84 % of the shared-memory data pipe (operands 39,
// load-store 45) at eight warps an SM; when it took 88 us, 72 with a quarter of the MMAs, 90 without the loads, 85 without splitting.  Three
// groups of four warps around one filter 92 us, a thread per four channels instead of eight 99.
#include "sc_entry.h"
#include "sc_umma_common.cuh"
#include "smem_grant.h"

namespace chop {
namespace {

// RP: rows of a pixel's window.  R: image rows of a tile.
// bfloat16: one where two would leave room for two CTAs only (tensor memory: R*3*channels of 512 columns): 16 -> 32 channels
// 64 us with one, 74 with two; 32 -> 32, where shared memory allows two CTAs anyway, 131 and 100.  float32: one (three pieces).
template <typename T> struct BandType;
template <> struct BandType<__nv_bfloat16> {
  static constexpr int P = 1;
  static constexpr int rows(int cr, int nr) { return nr > 16 && cr <= 16 ? 1 : 2; }
};
template <> struct BandType<float> {
  static constexpr int P = 3;
  static constexpr int rows(int, int) { return 1; }
};
template <typename T, int CR, int NR, int RP> struct BandGeo {
  static constexpr int P = BandType<T>::P;            // bfloat16 pieces of a value
  static constexpr int PT = 128 / RP;                 // pixels of an image row that make one MMA block
  static constexpr int R = BandType<T>::rows(CR, NR); // MMA blocks of a tile
  static constexpr int PW = PT + 2, NPIX = (R + 2) * PW;
  static constexpr int ROWS = NPIX * RP;              // staged rows
  static constexpr int FILTER = P * 27 * pad16(NR) * pad16(CR) * 2;
  static constexpr int ROW = P * (pad16(CR) / 8) * 16;   // bytes of a staged row
  static constexpr int COLS = R * P * 3 * pad16(NR);  // accumulators
  static constexpr uint32_t TMEM = COLS <= 64 ? 64 : COLS <= 128 ? 128 : 256;
  // CTAs that an SM holds with the window alone; the filter columns per step of a rough tile fill what that leaves of shared memory
  static constexpr int PER_SM = 224 * 1024;
  static constexpr int BY_SMEM = PER_SM / (FILTER + (ROWS + 4) * ROW + 3072), BY_TMEM = 512 / TMEM;
  static constexpr int CTAS = BY_SMEM < 1 ? 1 : BY_SMEM < BY_TMEM ? BY_SMEM : BY_TMEM;
  static constexpr int FIT = (PER_SM / CTAS - FILTER - 3072 - 4 * ROW) / (128 * ROW);
  static constexpr int GROUPS = FIT >= 9 ? 1 : FIT >= 5 ? 2 : 3;   // steps per image row of a rough tile
  static constexpr int CG = (9 + GROUPS - 1) / GROUPS;
  static constexpr int SROWS = CG * 128 > ROWS ? CG * 128 : ROWS;
  static constexpr int NRB = SROWS + 4;               // K-chunk stride 64 bytes off a multiple of 128 (bank conflicts)
  static constexpr size_t SMEM = (size_t)FILTER + (size_t)NRB * ROW + 1024;
  static_assert(FIT >= 3, "rough tiles");
  static_assert(PT * RP == 128 && 32 % RP == 0 && ROWS % 8 == 0 && NPIX <= 128 && R * PT <= 32 && COLS <= 256 && (P == 1 || R == 1), "tile");
};

// The filter in three pieces: tile [filter column][filter row][piece][depth tap], each as in stage_filter_tiles; channels n0 ..
// n0 + NR - 1 of NF produced ones.  Returns the largest magnitude that this thread has seen.
template <int CR, int NR, int NF, bool DGRAD>
__device__ __forceinline__ unsigned stage_filter_pieces(const float* flt, int n0, unsigned char* sB, int tid, uint32_t lbo, uint32_t sbo, int tap_bytes) {
  constexpr int COUT = pad16(NR), KC = pad16(CR) / 8;
  unsigned top = 0;
#pragma unroll 1
  for (int e = tid; e < 27 * COUT * KC; e += 128) {
    const int kg = e % KC, n = (e / KC) % COUT, t = e / (KC * COUT);
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int k = kg * 8 + i;
      v[i] = kg * 8 >= CR || n >= NR ? 0.f
             : __ldg(DGRAD ? flt + ((size_t)(26 - t) * NF + n0 + n) * CR + k : flt + ((size_t)t * CR + k) * NF + n0 + n);
    }
    top = max(top, top_bits(v));
    unsigned p[3][4];
    split3(v, p);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const int slot = ((t / 3 % 3 * 3 + t / 9) * 3 + q) * 3 + t % 3;
      *reinterpret_cast<uint4*>(sB + slot * tap_bytes + (n / 8) * sbo + kg * lbo + (n % 8) * 16) = make_uint4(p[q][0], p[q][1], p[q][2], p[q][3]);
    }
  }
  return top;
}

// The same sums by plain multiply-adds, for a step whose values are not for the pieces: output pixels `todo` of image row r.  A thread
// holds four channels of a voxel.  Taps that are padding add nothing in gradients, and where a zero meets a finite filter; a zero times
// an infinite weight is not a number.  189x251x7, 16 -> 16 channels, every value near 2^-110: 138 us on the CUDA cores (sc_tile.cu), 1380 a
// channel per thread, 1104 here; ordinary values 81.  Not inlined and with no more than this around it: 88 with the test of the padding in the caller.
template <int CR, int NR, int NF, bool DGRAD>
__device__ __noinline__ void band_plain(const ScArgs& a, const int2* tab, int pw, int r, unsigned todo, int n0, float pad, unsigned w_top) {
  const bool skip = a.pad_zero || (pad == 0.f && w_top < 0x7f800000u);
  const float* src = static_cast<const float*>(DGRAD ? a.out_grad : a.images);
  const float* flt = static_cast<const float*>(a.filters) + (DGRAD ? (size_t)n0 * CR : n0);
  float* dst = static_cast<float*>(DGRAD ? a.images_grad : a.output) + n0;
  const bool aligned = (reinterpret_cast<size_t>(flt) & 15) == 0;
  const float4 pad4 = make_float4(pad, pad, pad, pad);
  const int D = a.D;
  constexpr int N4 = NR / 4;
  for (int e = threadIdx.x; e < (pw - 2) * D * N4; e += 128) {
    const int n = e % N4 * 4, d = e / N4 % D, q = e / N4 / D;
    if (!((todo >> q) & 1u)) continue;
    const int2 o = tab[(r + 1) * pw + q + 1];
    float s[4] = {0.f, 0.f, 0.f, 0.f};
    for (int t = 0; t < 27; ++t) {
      const int2 nb = tab[(r + t / 9) * pw + q + t / 3 % 3];
      const int plane = d + o.y - nb.y - 1 + t % 3;
      const bool in = nb.x >= 0 && !oob(plane, D);
      if (!in && skip) continue;
      const float4* x = reinterpret_cast<const float4*>(src + (size_t)(in ? nb.x + plane : 0) * CR);
      const float* w = flt + (DGRAD ? ((size_t)(26 - t) * NF + n) * CR : (size_t)t * CR * NF + n);
#pragma unroll 1
      for (int k = 0; k < CR; k += 4) plain_fma<!DGRAD>(s, in ? __ldg(x + k / 4) : pad4, w + (size_t)k * (DGRAD ? 1 : NF), DGRAD ? CR : NF, aligned);
    }
    *reinterpret_cast<float4*>(dst + ((size_t)o.x + d) * NF + n) = make_float4(s[0], s[1], s[2], s[3]);
  }
}

// NR: produced channels of a CTA, NF: of the convolution (float32: 32 are produced by two CTAs, blockIdx.y).
template <typename T, int CR, int NF, bool DGRAD, int RP, int NR>
__global__ void __launch_bounds__(128, (BandGeo<T, CR, NR, RP>::CTAS))
sc_band_kernel(const ScArgs a, const int ntiles, const int tiles_w, const int tiles_h) {
  extern __shared__ __align__(1024) unsigned char smem[];
  typedef BandGeo<T, CR, NR, RP> G;
  constexpr int PT = G::PT, R = G::R, PW = G::PW, NPIX = G::NPIX, NRB = G::NRB, CG = G::CG, P = G::P;
  __shared__ __align__(8) uint64_t mbar_s;
  __shared__ uint32_t tmem_base_s;
  __shared__ int2 tab_s[3][NPIX];                       // per pixel around the tile: first voxel (-1: outside the image), base plane
  __shared__ unsigned top_s[4];                         // float32: largest magnitude of a step, three steps in turn
  constexpr int CIN = pad16(CR), COUT = pad16(NR), KC = CIN / 8, KR = CR / 8, N3 = 3 * COUT;
  constexpr uint32_t B_LBO = 128, B_SBO = KC * 128;     // filter tiles: K-chunks adjacent, then 8-row groups, taps behind each other
  constexpr uint32_t A_LBO = NRB * 16, A_SBO = 128;     // stage: rows linear, K-chunks NRB rows apart
  constexpr int B_TAP_BYTES = COUT * CIN * 2;
  unsigned char* sB = smem;                             // 27 taps
  unsigned char* sX = smem + G::FILTER;      // [piece][K-chunk][row]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n0 = NF > NR ? (int)blockIdx.y * NR : 0;
  const T* src = static_cast<const T*>(DGRAD ? a.out_grad : a.images);
  T* dst = static_cast<T*>(DGRAD ? a.images_grad : a.output) + n0;

  if (KR < KC)   // the padding channels stay zero
    for (int e = tid; e < P * G::SROWS; e += 128)
      *reinterpret_cast<uint4*>(sX + (e / G::SROWS * KC + 1) * A_LBO + e % G::SROWS * 16) = make_uint4(0, 0, 0, 0);
  constexpr uint32_t TCOLS = G::TMEM;
  if (warp == 0) {
    uint32_t slot = smem_u32(&tmem_base_s), ncols = TCOLS;
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&mbar_s)), "r"(1) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }

  const int H = a.H, W = a.W, D = a.D;
  uint4 padv = make_uint4(0, 0, 0, 0);                  // 16 bytes of padding values
  if (!a.pad_zero) {
    unsigned d32;
    if constexpr (P == 1) {
      const unsigned d16 = __ldg(static_cast<const unsigned short*>(a.default_value));
      d32 = d16 | (d16 << 16);
    } else {
      d32 = __ldg(static_cast<const unsigned*>(a.default_value));
    }
    padv = make_uint4(d32, d32, d32, d32);
  }
  auto entry = [&](int tile) {   // this thread's entry of a tile's table
    int2 e = make_int2(-1, 0);
    if (tid < NPIX && tile < ntiles) {
      const int tw = tile % tiles_w, t = tile / tiles_w, th = t % tiles_h, b = t / tiles_h;
      const int r = th * R - 1 + tid / PW, c = tw * PT - 1 + tid % PW;
      if (!oob(r, H) && !oob(c, W)) {
        const int pix = (b * H + r) * W + c;
        e = make_int2(pix * D, __ldg(a.base_plane + pix));   // voxel indices fit 31 bits (checked on the host)
      }
    }
    return e;
  };

  // A step is one staging of the buffer and the MMAs over it: a pass of a tile, or a (row, group of filter columns) of a
  // rough one.  All of this is the same in every thread.
  struct Step {
    int tile;         // -1: none
    int z0;           // smooth: first plane of the window
    unsigned now;     // smooth: the output pixels that this pass produces
    unsigned left;    // smooth: those still to do; rough: all bits
    int sub;          // rough: row*GROUPS + group, otherwise -1
  };
  // lane i of every warp stands for output pixel (i / PT, i % PT) of the tile
  const int slack = RP - 2 - D;
  auto window = [&](Step& s, int bp) {   // the next pass over the pixels in s.left
    const int lo = __reduce_min_sync(0xffffffffu, (s.left >> lane) & 1u ? bp : 0x7fffffff);
    s.z0 = lo - 1;
    s.now = __ballot_sync(0xffffffffu, ((s.left >> lane) & 1u) && (unsigned)bp - (unsigned)lo <= (unsigned)slack);
    s.left &= ~s.now;
  };
  auto out_entry = [&](const int2* tab) { return lane < R * PT ? tab[(lane / PT + 1) * PW + lane % PT + 1] : make_int2(-1, 0); };
  auto open = [&](Step& s, const int2* tab) {
    const int2 e = out_entry(tab);
    s.left = __ballot_sync(0xffffffffu, e.x >= 0);
    s.sub = -1;
    const unsigned all = s.left;
    window(s, e.y);
    if (s.left != 0) {
      Step u = s;
      window(u, e.y);
      if (u.left != 0) {   // a third pass would be needed
        s.sub = 0;
        s.left = all;
      }
    }
  };
  auto more = [&](const Step& s) { return s.sub >= 0 ? s.sub + 1 < R * G::GROUPS : s.left != 0; };

  constexpr int NI = (G::ROWS * KR + 127) / 128;        // chunks of eight channels that a thread stages per step
  constexpr int RSTEP = 128 / KR;                       // rows between them
  constexpr int VEC = (int)sizeof(T) / 2;               // 16-byte words of a chunk
  const int chunk = tid % KR, row0 = tid / KR;
  uint4 val[NI][VEC];
  // A rough tile's step: rows of CG filter columns, UC of them at a time in `val`.  Column c is staged in rows c*128 .., RPC chunks
  // of it by a thread, all of the same window row.
  constexpr int RPC = 128 / RSTEP, UC = NI / RPC;
  static_assert(RSTEP % RP == 0 && UC >= 1, "rough tiles");
  auto request_columns = [&](const Step& s, const int2* tab, int c0) {
    const int2* at = tab + s.sub / G::GROUPS * PW + row0 / RP;
    const int first = s.sub % G::GROUPS * CG;
    int from[RPC];
#pragma unroll
    for (int j = 0; j < RPC; ++j) from[j] = row0 % RP - 1 + at[PW + 1 + j * (RSTEP / RP)].y;
#pragma unroll
    for (int u = 0; u < UC; ++u) {
      const int col = first + c0 + u;
      if (c0 + u >= CG || col >= 9) continue;
#pragma unroll
      for (int j = 0; j < RPC; ++j) {
        const int2 e = at[col / 3 * PW + col % 3 + j * (RSTEP / RP)];
        const int plane = from[j] - e.y;
        const bool in = e.x >= 0 && !oob(plane, D);
#pragma unroll
        for (int k = 0; k < VEC; ++k) {
          val[u * RPC + j][k] = padv;
          if (in) val[u * RPC + j][k] = __ldg(reinterpret_cast<const uint4*>(src + (size_t)(e.x + plane) * CR) + chunk * VEC + k);
        }
      }
    }
  };
  // The chunks of a row are fetched by neighbouring lanes, a pixel's planes by the lanes behind: consecutive addresses.
  auto request = [&](const Step& s, const int2* tab) {
    if (s.sub >= 0) {
      request_columns(s, tab, 0);
      return;
    }
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const int row = row0 + i * RSTEP;
      int2 e = make_int2(-1, 0);
      int plane = 0;
      if ((i + 1) * RSTEP <= G::ROWS || row < G::ROWS) {   // a last, partial round
        e = tab[row / RP];
        plane = row % RP + s.z0 - e.y;
      }
      const bool in = e.x >= 0 && !oob(plane, D);
#pragma unroll
      for (int k = 0; k < VEC; ++k) {
        val[i][k] = padv;
        if (in) val[i][k] = __ldg(reinterpret_cast<const uint4*>(src + (size_t)(e.x + plane) * CR) + chunk * VEC + k);
      }
    }
  };

  Step cur, nxt;
  cur.tile = blockIdx.x;
  int2 ahead = entry(cur.tile);
  if (tid < NPIX) tab_s[0][tid] = ahead;
  __syncthreads();
  open(cur, tab_s[0]);
  request(cur, tab_s[0]);
  ahead = entry(cur.tile + (int)gridDim.x);             // of the tile after the present one
  unsigned w_top = 0;                                   // float32: the filter's largest magnitude
  if constexpr (P == 1) {
    stage_filter_tiles<CR, NR, DGRAD, true>(static_cast<const unsigned short*>(a.filters), sB, tid, B_LBO, B_SBO, B_TAP_BYTES);
  } else {
    const unsigned top = __reduce_max_sync(0xffffffffu, stage_filter_pieces<CR, NR, NF, DGRAD>(static_cast<const float*>(a.filters), n0, sB, tid, B_LBO, B_SBO, B_TAP_BYTES));
    if (lane == 0) top_s[warp] = top;
    __syncthreads();
    w_top = max(max(top_s[0], top_s[1]), max(top_s[2], top_s[3]));
    __syncthreads();
    if (tid < 3) top_s[tid] = 0;
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

  unsigned top = 0;
  bool plain = false;                                   // float32: this step's values are not for the pieces
  auto store = [&](int i, int row) {
    unsigned char* o = sX + chunk * A_LBO + row * 16;
    if constexpr (P == 1) {
      *reinterpret_cast<uint4*>(o) = val[i][0];
    } else {
      const uint4 lo = val[i][0], hi = val[i][VEC - 1];
      const float v[8] = {__uint_as_float(lo.x), __uint_as_float(lo.y), __uint_as_float(lo.z), __uint_as_float(lo.w),
                          __uint_as_float(hi.x), __uint_as_float(hi.y), __uint_as_float(hi.z), __uint_as_float(hi.w)};
      top = max(top, top_bits(v));
      unsigned p[3][4];
      split3(v, p);
#pragma unroll
      for (int q = 0; q < 3; ++q) *reinterpret_cast<uint4*>(o + q * KC * A_LBO) = make_uint4(p[q][0], p[q][1], p[q][2], p[q][3]);
    }
  };
  // Piece p of the gathered values meets pieces 0 .. P-1-p of the weights, side by side in N: accumulators [piece sum][depth tap],
  // the products x1*w1 | x1*w2, x2*w1 | x1*w3, x2*w2, x3*w1.  Apart from one another the small ones cost the large ones no bits: a
  // chain of 9*CIN/16 additions in tensor memory each, against 27*CIN/4 in registers before.
  while (true) {
    const bool again = more(cur);
    // the table of the next step; its buffer was last read two steps ago, before the barrier behind the last staging
    if (tid < NPIX) tab_s[next(buf)][tid] = again ? tab_s[buf][tid] : ahead;
    top = 0;
    if (cur.sub < 0) {
#pragma unroll
      for (int i = 0; i < NI; ++i)
        if ((i + 1) * RSTEP <= G::ROWS || row0 + i * RSTEP < G::ROWS)
          store(i, row0 + i * RSTEP);
    } else {
#pragma unroll 1
      for (int c0 = 0; c0 < CG; c0 += UC) {
        if (c0 > 0) request_columns(cur, tab_s[buf], c0);
#pragma unroll
        for (int i = 0; i < UC * RPC; ++i)
          if (c0 + i / RPC < CG && cur.sub % G::GROUPS * CG + c0 + i / RPC < 9) store(i, row0 + c0 * 128 + i * RSTEP);
      }
    }
    if constexpr (P > 1) {
      top = __reduce_max_sync(0xffffffffu, top);
      if (lane == 0) atomicMax(&top_s[buf], top);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if constexpr (P > 1) {
      if (cur.sub < 0 || cur.sub % G::GROUPS == 0) plain = false;
      plain = plain || !pieces_fit<CR>(top_s[buf], w_top);
      if (tid == 0) top_s[next(next(buf))] = 0;         // read in the last step, written two steps on
    }
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (cur.sub < 0) {
#pragma unroll
        for (int hr = 0; hr < R + 2; ++hr) {            // staged row: filter row fr of output row hr - fr
          const int lo = hr < R ? 0 : hr - R + 1, hi = hr < 2 ? hr : 2;
#pragma unroll
          for (int fc = 0; fc < 3; ++fc) {
#pragma unroll
            for (int k16 = 0; k16 < CIN / 16; ++k16) {
              const uint64_t da = umma_desc_advance(da0, (hr * PW + fc) * RP * 16 + k16 * 2 * A_LBO);
              const uint64_t db = umma_desc_advance(db0, fc * 9 * P * B_TAP_BYTES + k16 * 2 * B_LBO);
              if constexpr (P > 1) {                    // R == 1: staged row hr is filter row hr
#pragma unroll
                for (int p = 0; p < P; ++p)
                  umma_bf16(tmem + p * N3, umma_desc_advance(da, p * KC * A_LBO), umma_desc_advance(db, hr * P * 3 * B_TAP_BYTES),
                            idesc(P - p), (hr | fc | k16 | p) != 0 ? 1u : 0u);
                continue;
              }
              const bool fresh = lo == 0 && fc == 0 && k16 == 0;   // the first sums of output row hr
              const int from = fresh ? 1 : lo;
              if (fresh) umma_bf16(tmem + (R - 1 - hr) * N3, da, db, idesc(1), 0u);
              if (from <= hi) umma_bf16(tmem + (R - 1 - hr + from) * N3, da, umma_desc_advance(db, from * 3 * B_TAP_BYTES), idesc(hi - from + 1), 1u);
            }
          }
        }
      } else {
        const int blk = cur.sub / G::GROUPS, first = (cur.sub % G::GROUPS) * CG;
        for (int i = 0; i < CG && first + i < 9; ++i) {
#pragma unroll
          for (int k16 = 0; k16 < CIN / 16; ++k16) {
            const uint64_t da = umma_desc_advance(da0, i * 128 * 16 + k16 * 2 * A_LBO);
            const int col = first + i;
            const uint64_t db = umma_desc_advance(db0, (col % 3 * 3 + col / 3) * P * 3 * B_TAP_BYTES + k16 * 2 * B_LBO);
#pragma unroll
            for (int p = 0; p < P; ++p)
              umma_bf16(tmem + (R - 1 - blk) * N3 + p * N3, umma_desc_advance(da, p * KC * A_LBO), db, idesc(P - p),
                        (first | i | k16 | p) != 0 ? 1u : 0u);
          }
        }
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
    }
    // ---- while they run: the next step's pixels and rows ---------------------------------------------------------
    nxt = cur;
    bool go = true;
    if (!again) {
      nxt.tile = cur.tile + (int)gridDim.x;
      go = nxt.tile < ntiles;
      if (go) open(nxt, tab_s[next(buf)]);
    } else if (cur.sub >= 0) {
      ++nxt.sub;
    } else {
      window(nxt, out_entry(tab_s[next(buf)]).y);
    }
    if (go) {
      request(nxt, tab_s[next(buf)]);
      if (!again) ahead = entry(nxt.tile + (int)gridDim.x);
    }

    // one warp polls the mbarrier (every poll is a shared-memory access); the others wait at the hardware barrier
    bool done = true;
    if (warp == 0) done = mbar_wait(mbar, phase);
    phase ^= 1;
    if (!__syncthreads_and(done)) {
      if (tid == 0) note_timeout();
      break;
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

    // ---- epilogue: accumulator row = (pixel q, window row w); taps fz of rows w-1, w, w+1 make output row w -----------
    constexpr int NE = P > 1 || NR < 16 ? 8 : 16;       // channels at a time
    const int q = tid / RP, w = tid % RP;
#pragma unroll 1
    for (int r = 0; r < R; ++r) {
      const int2 e = tab_s[buf][(r + 1) * PW + q + 1];
      bool mine;
      int d;
      unsigned todo = (cur.now >> (r * PT)) & ((1u << PT) - 1u);
      if (cur.sub < 0) {
        mine = (todo >> q) & 1u;
        d = w + cur.z0 - e.y;
      } else {
        todo = __ballot_sync(0xffffffffu, lane < PT && tab_s[buf][(r + 1) * PW + lane % PT + 1].x >= 0);
        if (cur.sub != r * G::GROUPS + G::GROUPS - 1) todo = 0;   // not the row's last group of filter columns
        mine = e.x >= 0;
        d = w - 1;
      }
      if (todo == 0) continue;
      if constexpr (P > 1) {
        if (plain) {
          band_plain<CR, NR, NF, DGRAD>(a, tab_s[buf], PW, r, todo, n0, __uint_as_float(padv.x), w_top);
          continue;
        }
      }
      mine = mine && !oob(d, D);
      T* o = dst + (size_t)(mine ? e.x + d : 0) * NF;
#pragma unroll 1
      for (int c = 0; c < NR; c += NE) {
        uint32_t t[P][3][NE];
        const uint32_t col = tmem + ((uint32_t)(warp * 32) << 16) + (R - 1 - r) * N3 + c;
#pragma unroll
        for (int p = 0; p < P; ++p)
#pragma unroll
          for (int fz = 0; fz < 3; ++fz) tmem_ld<NE>(col + p * N3 + fz * COUT, t[p][fz]);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        float s[NE];
#pragma unroll
        for (int k = 0; k < NE; ++k) {
          float f[3];
#pragma unroll
          for (int fz = 0; fz < 3; ++fz) {
            f[fz] = __uint_as_float(t[P - 1][fz][k]);   // the small products first
#pragma unroll
            for (int p = P - 2; p >= 0; --p) f[fz] += __uint_as_float(t[p][fz][k]);
          }
          const float below = __shfl_up_sync(0xffffffffu, f[0], 1);
          const float above = __shfl_down_sync(0xffffffffu, f[2], 1);
          s[k] = below + f[1] + above;
        }
        if (mine) {
          if constexpr (P == 1) {
#pragma unroll
            for (int k = 0; k < NE; k += 8) {
              uint32_t h[4];
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const __nv_bfloat162 b = __floats2bfloat162_rn(s[k + 2 * i], s[k + 2 * i + 1]);
                h[i] = *reinterpret_cast<const uint32_t*>(&b);
              }
              *reinterpret_cast<uint4*>(o + c + k) = make_uint4(h[0], h[1], h[2], h[3]);
            }
          } else {
#pragma unroll
            for (int k = 0; k < NE; k += 4) *reinterpret_cast<float4*>(o + c + k) = make_float4(s[k], s[k + 1], s[k + 2], s[k + 3]);
          }
        }
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (!go) break;
    cur = nxt;
    buf = next(buf);
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    uint32_t ncols = TCOLS;
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols) : "memory");
  }
}

// Windows of 16 rows for bands of up to 10 planes, of 32 rows for up to 24: base_plane may vary by four planes at least.
template <typename T, int CIN, int COUT, bool DGRAD, int RP>
int launch_rp(const ScArgs& a, cudaStream_t st) {
  constexpr int NR = BandType<T>::P > 1 && COUT > 16 ? 16 : COUT;
  typedef BandGeo<T, CIN, NR, RP> G;
  auto k = sc_band_kernel<T, CIN, COUT, DGRAD, RP, NR>;
  if (int e = grant_smem(k, G::SMEM)) return e;
  const int tw = (a.W + G::PT - 1) / G::PT, th = (a.H + G::R - 1) / G::R;
  const long long ntiles = (long long)a.B * tw * th;    // at most as many as pixels: 31 bits
  constexpr long long slots = 148LL * G::CTAS / (COUT / NR);
  k<<<dim3((unsigned)(ntiles < slots ? ntiles : slots), COUT / NR), 128, G::SMEM, st>>>(a, (int)ntiles, tw, th);
  return (int)cudaGetLastError();
}
template <typename T, int CIN, int COUT, bool DGRAD>
int launch_band(const ScArgs& a, cudaStream_t st) {
  if (a.D <= 10) return launch_rp<T, CIN, COUT, DGRAD, 16>(a, st);
  return launch_rp<T, CIN, COUT, DGRAD, 32>(a, st);
}
#define CHOP_CASE(T, I, O)                                                            \
  if (!dgrad && a.Cin == I && a.Cout == O) return launch_band<T, I, O, false>(a, st); \
  if (dgrad && a.Cout == I && a.Cin == O) return launch_band<T, I, O, true>(a, st);

}  // namespace

// Where this beats sc_umma_rows_kernel, whose cost follows D + 2 rows a pixel where this one's follows the window:
//   * 32 produced channels of 8 or 16 gathered ones (tiles of one row: three staged pixels per pixel) need a well filled
//     window.  256x320, 16 -> 32: D = 5 57 us there, 61 here; 9 80, 64; 13 (32-row window) 102, 115; 17 131, 119.
//   * 16-row windows on small images, where few tiles share the chip and their base planes are steep (two passes): 60x75x9
//     14 there, 16 here for 16 -> 16 and 27, 36 for 32 -> 32; 100x125x9 20, 23 and 47, 44; 120x150x9 25, 23 and 61, 49.
bool sc_band_better(const ScArgs& a, int cin, int cout) {
  if (a.D > 24) return false;
  const int rp = a.D <= 10 ? 16 : 32;
  if (BandType<__nv_bfloat16>::rows(cin, cout) == 1 && 16 * (a.D + 2) < 9 * rp) return false;
  return rp == 32 || (long long)a.B * a.H * a.W >= 16000;
}

// float32, where this beats sc_run_kernel and is no less exact.  189x251x7, us there and here: 16 -> 16 127, 88; 16 -> 32 238, 166;
// 16 -> 8 79, 84; 8 -> 8 49, 70; 8 -> 16 73, 74; 256x320x9 254, 140; 493, 268; 155, 134; 87, 112; 134, 117; 60x75x9, 16 -> 16 29, 30
// (when these were compared; 16 -> 16 and 16 -> 32 now 71, 139 and 135, 239).
// 2-norm of the error against float64 over that of the result: 16 gathered channels 1.31 to 1.38e-7 here, 1.80 to 1.92e-7 there.  32, whose
// chains are twice as long, 2.5 to 2.6e-7 here and 1.85 to 1.90e-7 there: less exact, so they stay there, although 256x320x9 32 -> 32
// would take 625 us instead of 1134, 32 -> 16 314 instead of 575.
bool sc_band_f32_better(const ScArgs& a, int cin, int cout) { return cin == 16 && cout >= 16 && a.D >= 5 && a.D <= 24; }

int sc_band_launch(const ScArgs& a, bool dgrad, cudaStream_t st) {
  typedef __nv_bfloat16 bf;
  CHOP_CASE(bf, 8, 8) CHOP_CASE(bf, 8, 16) CHOP_CASE(bf, 8, 32) CHOP_CASE(bf, 16, 8) CHOP_CASE(bf, 16, 16) CHOP_CASE(bf, 16, 32)
  CHOP_CASE(bf, 32, 8) CHOP_CASE(bf, 32, 16) CHOP_CASE(bf, 32, 32)
  return -4;
}
int sc_band_f32_launch(const ScArgs& a, bool dgrad, cudaStream_t st) {
  if (!dgrad && a.Cin == 16 && a.Cout == 16) return launch_band<float, 16, 16, false>(a, st);
  if (!dgrad && a.Cin == 16 && a.Cout == 32) return launch_band<float, 16, 32, false>(a, st);
  if (dgrad && a.Cout == 16 && a.Cin == 16) return launch_band<float, 16, 16, true>(a, st);
  if (dgrad && a.Cout == 16 && a.Cin == 32) return launch_band<float, 16, 32, true>(a, st);
  return -4;
}
#undef CHOP_CASE

int sc_band_timeouts() { return timeouts_here(); }
int sc_band_publish_mirror(int* dptr, cudaStream_t st) { return (int)publish_mirror_here(dptr, st); }
int sc_band_clear_timeouts() { return (int)clear_timeouts_here(); }

}  // namespace chop
