// Stride-1 manifold convolution on the tensor cores with every voxel staged ONCE per tile: 3x3x3, dilation 1, bfloat16
// storage, float32 accumulation, 8, 16 or 32 channels, bands of up to 24 planes.
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
//     plane, not a depth map) and stages its filter columns one by one, each pixel's rows shifted as in sc_umma_rows_kernel.
//
// Base planes of 64 planes over the image (two sinusoid periods), D = 9: 1.00 passes a tile at 256x320 pixels, 1.4 at 100x125.
// Bound: the shared-memory data pipe (56 % load-store, of which half is the epilogue's tensor-memory reads and shuffles; 35 %
// MMA operands) and, with four CTAs an SM, a tile's chain of staging, MMAs and epilogue.  256x320x9, 3x3x3, bfloat16, us:
// 16 -> 16 channels 59 -> 41, 8 -> 8 51 -> 33, 32 -> 32 213 -> 100, 32 -> 16 129 -> 74; at 17 planes 97 -> 72, 344 -> 182.
// Tiles of four rows with 256 threads: 45; of one row: 49; windows that do not divide 32 rows (25 for 17 planes): 108.
#include "sc_entry.h"
#include "sc_umma_common.cuh"
#include "smem_grant.h"

namespace chop {
namespace {

// RP: rows of a pixel's window.  R: image rows of a tile.
// One where two would leave room for two CTAs only (tensor memory: R*3*channels of 512 columns): 16 -> 32 channels 64 us
// with one, 74 with two; 32 -> 32, where shared memory allows two CTAs anyway, 131 and 100.
constexpr int band_tile_rows(int cr, int nr) { return nr > 16 && cr <= 16 ? 1 : 2; }
template <int CR, int NR, int RP> struct BandGeo {
  static constexpr int PT = 128 / RP;                 // pixels of an image row that make one MMA block
  static constexpr int R = band_tile_rows(CR, NR);        // MMA blocks of a tile
  static constexpr int NTHR = 128;                     // one thread per accumulator row
  static constexpr int PW = PT + 2, NPIX = (R + 2) * PW;
  static constexpr int ROWS = NPIX * RP;              // staged rows
  static constexpr int NRB = ROWS + 4;                // K-chunk stride 64 bytes off a multiple of 128 (bank conflicts)
  static constexpr int CG = ROWS / 128;               // filter columns per step of a rough tile
  static constexpr int GROUPS = (9 + CG - 1) / CG;
  static constexpr size_t SMEM = (size_t)27 * pad16(NR) * pad16(CR) * 2 + (size_t)(pad16(CR) / 8) * NRB * 16 + 1024;
  static constexpr uint32_t TMEM = R * 3 * pad16(NR) <= 64 ? 64 : R * 3 * pad16(NR) <= 128 ? 128 : 256;
  static constexpr int BY_SMEM = (int)((size_t)220 * 1024 / (SMEM + 2048)), BY_TMEM = 512 / TMEM;
  static constexpr int CTAS = BY_SMEM < BY_TMEM ? BY_SMEM : BY_TMEM;
  static_assert(PT * RP == 128 && 32 % RP == 0 && ROWS % 8 == 0 && NPIX <= NTHR && R * PT <= 32 && R * 3 * pad16(NR) <= 256, "tile");
};

template <int CR, int NR, bool DGRAD, int RP>
__global__ void __launch_bounds__(BandGeo<CR, NR, RP>::NTHR, BandGeo<CR, NR, RP>::CTAS)
sc_band_kernel(const ScArgs a, const int ntiles, const int tiles_w, const int tiles_h) {
  extern __shared__ __align__(1024) unsigned char smem[];
  typedef BandGeo<CR, NR, RP> G;
  constexpr int PT = G::PT, R = G::R, PW = G::PW, NPIX = G::NPIX, NRB = G::NRB, CG = G::CG, NTHR = G::NTHR;
  __shared__ __align__(8) uint64_t mbar_s;
  __shared__ uint32_t tmem_base_s;
  __shared__ int2 tab_s[3][NPIX];                       // per pixel around the tile: first voxel (-1: outside the image), base plane
  constexpr int CIN = pad16(CR), COUT = pad16(NR), KC = CIN / 8, KR = CR / 8, N3 = 3 * COUT;
  constexpr uint32_t B_LBO = 128, B_SBO = KC * 128;     // filter tiles: K-chunks adjacent, then 8-row groups, taps behind each other
  constexpr uint32_t A_LBO = NRB * 16, A_SBO = 128;     // stage: rows linear, K-chunks NRB rows apart
  constexpr int B_TAP_BYTES = COUT * CIN * 2;
  unsigned char* sB = smem;                             // 27 taps
  unsigned char* sX = smem + 27 * B_TAP_BYTES;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const __nv_bfloat16* src = static_cast<const __nv_bfloat16*>(DGRAD ? a.out_grad : a.images);
  __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(DGRAD ? a.images_grad : a.output);

  if (KR < KC)   // the padding channels stay zero
    for (int e = tid; e < G::ROWS; e += NTHR) *reinterpret_cast<uint4*>(sX + A_LBO + e * 16) = make_uint4(0, 0, 0, 0);
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
  uint4 padv = make_uint4(0, 0, 0, 0);
  if (!a.pad_zero) {
    const unsigned d16 = __ldg(static_cast<const unsigned short*>(a.default_value));
    const unsigned d32 = d16 | (d16 << 16);
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

  constexpr int NI = (G::ROWS * KR + NTHR - 1) / NTHR;  // 16-byte chunks a thread stages per step
  constexpr int RSTEP = NTHR / KR;                      // rows between them
  const int chunk = tid % KR, row0 = tid / KR;
  uint4 val[NI];
  // The chunks of a row are fetched by neighbouring lanes, a pixel's planes by the lanes behind: consecutive addresses.
  auto request = [&](const Step& s, const int2* tab) {
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const int row = row0 + i * RSTEP;
      int2 e = make_int2(-1, 0);
      int plane = 0;
      if ((i + 1) * RSTEP > G::ROWS && row >= G::ROWS) {   // a last, partial round
      } else if (s.sub < 0) {
        e = tab[row / RP];
        plane = row % RP + s.z0 - e.y;
      } else {
        const int blk = s.sub / G::GROUPS, col = (s.sub % G::GROUPS) * CG + row / 128, q = row % 128 / RP;
        if (col < 9) {
          const int2 o = tab[(blk + 1) * PW + q + 1];
          e = tab[(blk + col / 3) * PW + q + col % 3];
          plane = row % RP - 1 + o.y - e.y;
        }
      }
      val[i] = padv;
      if (e.x >= 0 && !oob(plane, D)) val[i] = __ldg(reinterpret_cast<const uint4*>(src + (size_t)(e.x + plane) * CR) + chunk);
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
  stage_filter_tiles<CR, NR, DGRAD, true, NTHR>(static_cast<const unsigned short*>(a.filters), sB, tid, B_LBO, B_SBO, B_TAP_BYTES);
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

  while (true) {
    const bool again = more(cur);
    // the table of the next step; its buffer was last read two steps ago, before the barrier behind the last staging
    if (tid < NPIX) tab_s[next(buf)][tid] = again ? tab_s[buf][tid] : ahead;
#pragma unroll
    for (int i = 0; i < NI; ++i)
      if ((i + 1) * RSTEP <= G::ROWS || row0 + i * RSTEP < G::ROWS)
        *reinterpret_cast<uint4*>(sX + chunk * A_LBO + (row0 + i * RSTEP) * 16) = val[i];
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
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
              const uint64_t db = umma_desc_advance(db0, fc * 9 * B_TAP_BYTES + k16 * 2 * B_LBO);
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
            const uint64_t db = umma_desc_advance(db0, (col % 3 * 3 + col / 3) * 3 * B_TAP_BYTES + k16 * 2 * B_LBO);
            umma_bf16(tmem + (R - 1 - blk) * N3, da, db, idesc(1), (first | i | k16) != 0 ? 1u : 0u);
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
    constexpr int NE = NR < 16 ? NR : 16;               // channels at a time
    const int q = tid / RP, w = tid % RP;
#pragma unroll 1
    for (int r = 0; r < R; ++r) {
      const int2 e = tab_s[buf][(r + 1) * PW + q + 1];
      bool mine;
      int d;
      if (cur.sub < 0) {
        mine = (cur.now >> (r * PT + q)) & 1u;
        d = w + cur.z0 - e.y;
        if (((cur.now >> (r * PT)) & ((1u << PT) - 1u)) == 0) continue;
      } else {
        if (cur.sub != r * G::GROUPS + G::GROUPS - 1) continue;   // the row's last group of filter columns
        mine = e.x >= 0;
        d = w - 1;
      }
      mine = mine && !oob(d, D);
      uint4* o = reinterpret_cast<uint4*>(dst + (size_t)(mine ? e.x + d : 0) * NR);
#pragma unroll 1
      for (int n0 = 0; n0 < NR; n0 += NE) {
        uint32_t t0[NE], t1[NE], t2[NE];
        const uint32_t col = tmem + ((uint32_t)(warp * 32) << 16) + (R - 1 - r) * N3 + n0;
        tmem_ld<NE>(col, t0);
        tmem_ld<NE>(col + COUT, t1);
        tmem_ld<NE>(col + 2 * COUT, t2);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        uint32_t h[NE / 2];
#pragma unroll
        for (int k = 0; k < NE; k += 2) {
          float s[2];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const float below = __uint_as_float(__shfl_up_sync(0xffffffffu, t0[k + i], 1));
            const float above = __uint_as_float(__shfl_down_sync(0xffffffffu, t2[k + i], 1));
            s[i] = below + __uint_as_float(t1[k + i]) + above;
          }
          const __nv_bfloat162 p = __floats2bfloat162_rn(s[0], s[1]);
          h[k / 2] = *reinterpret_cast<const uint32_t*>(&p);
        }
        if (mine) {
#pragma unroll
          for (int k = 0; k < NE / 8; ++k) o[n0 / 8 + k] = make_uint4(h[4 * k], h[4 * k + 1], h[4 * k + 2], h[4 * k + 3]);
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
template <int CIN, int COUT, bool DGRAD, int RP>
int launch_rp(const ScArgs& a, cudaStream_t st) {
  typedef BandGeo<CIN, COUT, RP> G;
  auto k = sc_band_kernel<CIN, COUT, DGRAD, RP>;
  if (int e = grant_smem(k, G::SMEM)) return e;
  const int tw = (a.W + G::PT - 1) / G::PT, th = (a.H + G::R - 1) / G::R;
  const long long ntiles = (long long)a.B * tw * th;    // at most as many as pixels: 31 bits
  constexpr long long slots = 148LL * G::CTAS;
  k<<<(unsigned)(ntiles < slots ? ntiles : slots), G::NTHR, G::SMEM, st>>>(a, (int)ntiles, tw, th);
  return (int)cudaGetLastError();
}
template <int CIN, int COUT, bool DGRAD>
int launch_band(const ScArgs& a, cudaStream_t st) {
  if (a.D <= 10) return launch_rp<CIN, COUT, DGRAD, 16>(a, st);
  return launch_rp<CIN, COUT, DGRAD, 32>(a, st);
}

}  // namespace

// Where this beats sc_umma_rows_kernel, whose cost follows D + 2 rows a pixel where this one's follows the window:
//   * 32 produced channels of 8 or 16 gathered ones (tiles of one row: three staged pixels per pixel) need a well filled
//     window.  256x320, 16 -> 32: D = 5 57 us there, 61 here; 9 80, 64; 13 (32-row window) 102, 115; 17 131, 119.
//   * 16-row windows on small images, where few tiles share the chip and their base planes are steep (two passes): 60x75x9
//     14 there, 16 here for 16 -> 16 and 27, 36 for 32 -> 32; 100x125x9 20, 23 and 47, 44; 120x150x9 25, 23 and 61, 49.
bool sc_band_better(const ScArgs& a, int cin, int cout) {
  if (a.D > 24) return false;
  const int rp = a.D <= 10 ? 16 : 32;
  if (band_tile_rows(cin, cout) == 1 && 16 * (a.D + 2) < 9 * rp) return false;
  return rp == 32 || (long long)a.B * a.H * a.W >= 16000;
}

int sc_band_launch(const ScArgs& a, bool dgrad, cudaStream_t st) {
#define CHOP_CASE(I, O)                                                            \
  if (!dgrad && a.Cin == I && a.Cout == O) return launch_band<I, O, false>(a, st); \
  if (dgrad && a.Cout == I && a.Cin == O) return launch_band<I, O, true>(a, st);
  CHOP_CASE(8, 8) CHOP_CASE(8, 16) CHOP_CASE(8, 32) CHOP_CASE(16, 8) CHOP_CASE(16, 16) CHOP_CASE(16, 32) CHOP_CASE(32, 8)
  CHOP_CASE(32, 16) CHOP_CASE(32, 32)
#undef CHOP_CASE
  return -4;
}

int sc_band_timeouts() { return timeouts_here(); }
int sc_band_publish_mirror(int* dptr) { return (int)publish_mirror_here(dptr); }
int sc_band_clear_timeouts() { return (int)clear_timeouts_here(); }

}  // namespace chop
