// What the tensor-core convolution kernels of sc_umma.cu, sc_band.cu and sc_up.cu share: descriptors, tcgen05 wrappers, the bounded
// wait and its bookkeeping, the filter tiles, the three pieces of a float32.  Everything has internal linkage: each of the three
// files has its own counter of abandoned waits, which sc_umma.cu adds up.
#pragma once
#include <cuda_bf16.h>

#include "sc_common.cuh"

namespace chop {
namespace {

__device__ int g_umma_timeouts = 0;
// Host-visible mirror of the counter: a mapped, pinned int that sc_umma_watch() publishes to the device on request.
// A kernel that gives up a wait also bumps it, so a host can notice without synchronising with the device.
__device__ int* g_umma_host_mirror = nullptr;
__device__ __forceinline__ void note_timeout() {
  atomicAdd(&g_umma_timeouts, 1);
  int* h = g_umma_host_mirror;
  if (h) {
    atomicAdd_system(h, 1);
    __threadfence_system();
  }
}
// Host side of one file's counter: its value (-1: error), the mirror's device address, a reset.
inline int timeouts_here() {
  int v = -1;
  return cudaMemcpyFromSymbol(&v, g_umma_timeouts, sizeof(int)) == cudaSuccess ? v : -1;
}
inline cudaError_t publish_mirror_here(int* dptr, cudaStream_t st) {   // the stream is waited for: a capture elsewhere goes on
  const cudaError_t e = cudaMemcpyToSymbolAsync(g_umma_host_mirror, &dptr, sizeof(dptr), 0, cudaMemcpyHostToDevice, st);
  return e != cudaSuccess ? e : cudaStreamSynchronize(st);
}
inline cudaError_t clear_timeouts_here() {
  const int zero = 0;
  return cudaMemcpyToSymbol(g_umma_timeouts, &zero, sizeof(int));
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor, K-major, no swizzle: start address, leading byte offset (distance
// between core matrices adjacent in K), stride byte offset (distance between 8-row groups), version 1.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
  d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;
  return d;
}

// The descriptor of the same layout `bytes` further on (the start-address field counts 16-byte units and a CTA's
// shared memory cannot carry out of it).  Issuing an MMA then costs one addition per operand instead of
// rebuilding the descriptor; a single thread issues them all, so this is the critical path of a tile.
__device__ __forceinline__ uint64_t umma_desc_advance(uint64_t desc, uint32_t bytes) { return desc + (uint64_t)(bytes >> 4); }

__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
      "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity) {
  uint32_t ok = 0;
  for (int it = 0; it < (1 << 24) && !ok; ++it) {
    asm volatile(
        "{\n.reg .pred P1;\nmbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\nselp.u32 %0, 1, 0, P1;\n}\n"
        : "=r"(ok)
        : "r"(mbar), "r"(parity)
        : "memory");
  }
  return ok != 0;
}

template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t* r);
template <>
__device__ __forceinline__ void tmem_ld<16>(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                 "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(taddr)
               : "memory");
}
template <>
__device__ __forceinline__ void tmem_ld<8>(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
template <>
__device__ __forceinline__ void tmem_ld<32>(uint32_t taddr, uint32_t* r) {
  tmem_ld<16>(taddr, r);
  tmem_ld<16>(taddr + 16, r + 16);
}

// Filter [27][Cin_f][Cout_f] -> canonical K-major B tiles in shared memory, B[n][k] of tap t at sB + t*tap_bytes
// (forward: n = output channel, k = input channel; DGRAD: the flipped tap with the channels swapped, whose rows are
// contiguous in the filter tensor).  One 16-byte chunk (eight k of one n) per thread and step, its loads independent of
// each other: every CTA repeats this, so it must not be a chain of dependent scalar loads.
// CR, NR: the channels the tensors have.  Eight are padded to 16 (the K of an MMA, the least N at M = 128) with zeros.
// The tensor pipe is idle most of the time anyway: 180x230x9, 3x3x3, bf16 forward / image gradient / filter gradient took
// 91 / 110 / 127 us for 8 -> 16 channels on the CUDA cores and take 30 / 31 / 21 here, 32 -> 8 191 / 159 / 236 and 68 / 35 / 120.
__host__ __device__ constexpr int pad16(int c) { return c < 16 ? 16 : c; }
// COLS: the tiles in the order [filter column][filter row][depth tap], not the filter's [row][column][depth].
template <int CR, int NR, bool DGRAD, bool COLS = false>
__device__ __forceinline__ void stage_filter_tiles(const unsigned short* flt, unsigned char* sB, int tid, uint32_t lbo,
                                                   uint32_t sbo, int tap_bytes) {
  constexpr int COUT = pad16(NR), KC = pad16(CR) / 8;
#pragma unroll 2
  for (int e = tid; e < 27 * COUT * KC; e += 128) {
    const int kg = e % KC, n = (e / KC) % COUT, t = e / (KC * COUT);
    uint4 w = make_uint4(0, 0, 0, 0);
    if (kg * 8 >= CR || n >= NR) {
    } else if (DGRAD) {
      w = __ldg(reinterpret_cast<const uint4*>(flt + ((size_t)(26 - t) * NR + n) * CR + kg * 8));  // f[flip t][ci = n][oc = k]
    } else {
      unsigned h[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) h[i] = __ldg(flt + ((size_t)t * CR + kg * 8 + i) * NR + n);        // f[t][ci = k][oc = n]
      w = make_uint4(h[0] | (h[1] << 16), h[2] | (h[3] << 16), h[4] | (h[5] << 16), h[6] | (h[7] << 16));
    }
    const int slot = COLS ? (t / 3 % 3 * 3 + t / 9) * 3 + t % 3 : t;
    *reinterpret_cast<uint4*>(sB + slot * tap_bytes + (n / 8) * sbo + kg * lbo + (n % 8) * 16) = w;
  }
}

// Eight float32 values as three bfloat16 pieces each, every piece the nearest to what is left: x = x1 + x2 + x3, exactly from
// |x| = 2^-109 on (the remainders have 15 and 6 significant bits; below, x3 is rounded to a multiple of 2^-133).  Cut off instead of rounded, all pieces of a value have its sign and the products
// that are left out add up: 2-norm error of the transposed forward, strides (2,2,2), 16 channels, 1.02e-7.
__device__ __forceinline__ void split3(const float (&v)[8], unsigned (&p)[3][4]) {
#pragma unroll
  for (int i = 0; i < 8; i += 2) {
    float a = v[i], b = v[i + 1];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
      p[q][i / 2] = *reinterpret_cast<const unsigned*>(&h);
      if (q < 2) {
        a = __fsub_rn(a, __uint_as_float(p[q][i / 2] << 16));
        b = __fsub_rn(b, __uint_as_float(p[q][i / 2] & 0xffff0000u));
      }
    }
  }
}
// Largest magnitude, as bits.
__device__ __forceinline__ unsigned top_bits(const float (&v)[8]) {
  unsigned m = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) m = max(m, __float_as_uint(v[i]) & 0x7fffffffu);
  return m;
}
// Whether sums of 27*CR products x*w can be made of pieces; x: largest magnitude of a step's values (top_bits), w: of the filter.
//   * Finite, and not rounded to an infinity: that times a zero piece is not a number.
//   * No sum of so many products, rounded up to the next power of two, can pass the largest float: x1*w1 and the small products are
//     added up apart, so an overflow would be an infinity too early, or two of them with different signs.
//   * Neither x nor w nor their product below 2^-100, so that the third pieces (2^-17 of the value) and what they are multiplied to are
//     normal numbers.  Smaller values beside these lose bits below 2^-133, the end of bfloat16's subnormal numbers.
template <int CR>
__device__ __forceinline__ bool pieces_fit(unsigned x, unsigned w) {
  constexpr int LOG = CR == 8 ? 8 : CR == 16 ? 9 : 10;  // 27*CR <= 2^LOG
  constexpr unsigned INF = 0x7f7f0000u;
  if (x >= INF || w >= INF) return false;
  if (x == 0 || w == 0) return true;
  const int ex = (int)(x >> 23) - 127, ew = (int)(w >> 23) - 127;   // the values are below 2^(e + 1)
  return ex >= -100 && ew >= -100 && ex + ew >= -100 && ex + ew + 2 + LOG <= 127;
}

// For sums that the pieces cannot hold: s[j] += x . (the weights of produced channel j), four gathered and four produced channels.
// The filter may lie at any address.  w: FWD weight [0][0] of rows of NF produced channels, otherwise of rows of CR gathered ones.
__device__ __forceinline__ float4 ld4_any(const float* p, bool aligned) {
  return aligned ? __ldg(reinterpret_cast<const float4*>(p)) : make_float4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3));
}
template <bool FWD>
__device__ __forceinline__ void plain_fma(float (&s)[4], const float4& x, const float* w, int pitch, bool aligned) {
  const float4 a = ld4_any(w, aligned), b = ld4_any(w + pitch, aligned), c = ld4_any(w + 2 * pitch, aligned), d = ld4_any(w + 3 * pitch, aligned);
  if (FWD) {
    s[0] = fmaf(x.w, d.x, fmaf(x.z, c.x, fmaf(x.y, b.x, fmaf(x.x, a.x, s[0]))));
    s[1] = fmaf(x.w, d.y, fmaf(x.z, c.y, fmaf(x.y, b.y, fmaf(x.x, a.y, s[1]))));
    s[2] = fmaf(x.w, d.z, fmaf(x.z, c.z, fmaf(x.y, b.z, fmaf(x.x, a.z, s[2]))));
    s[3] = fmaf(x.w, d.w, fmaf(x.z, c.w, fmaf(x.y, b.w, fmaf(x.x, a.w, s[3]))));
  } else {
    s[0] = fmaf(x.w, a.w, fmaf(x.z, a.z, fmaf(x.y, a.y, fmaf(x.x, a.x, s[0]))));
    s[1] = fmaf(x.w, b.w, fmaf(x.z, b.z, fmaf(x.y, b.y, fmaf(x.x, b.x, s[1]))));
    s[2] = fmaf(x.w, c.w, fmaf(x.z, c.z, fmaf(x.y, c.y, fmaf(x.x, c.x, s[2]))));
    s[3] = fmaf(x.w, d.w, fmaf(x.z, d.z, fmaf(x.y, d.y, fmaf(x.x, d.x, s[3]))));
  }
}

}  // namespace
}  // namespace chop
