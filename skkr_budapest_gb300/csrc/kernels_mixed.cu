// Split-precision kernels: FP64-accurate complex products on the 5th-generation
// tensor cores (tcgen05.mma, BF16 operands, FP32 accumulation in TMEM) and a
// refined inverse.
//
// Products (Ozaki-style splitting).  Every row i of A gets a power-of-two
// scale sigma_i >= max_j |A_ij| (re and im together), every column j of B a
// scale tau_j.  The scaled entries in [-1, 1] are cut into S exact slices of
// 8 significant bits by repeated rounding:
//     x/sigma = sum_p s_p 2^(-7-8(p-1)),   s_p integers, |s_p| <= 128,
// which BF16 stores exactly.  Slice p of A is stored as s_p 2^(-8(p-1)) and
// slice q of B as s_q 2^(-8(q-3)); then every slice product A_p B_q carries
// its true relative weight, and all products of one "level" p+q land in the
// same accumulator with a common factor 2^-30 sigma_i tau_j.  Each level has
// its own TMEM accumulator: the tensor core aligns addends to the largest
// exponent and truncates, so sums of one level stay exact (integer multiples
// of the level's unit, at most (c+1) K 2^14 units, within FP32's 24 bits for
// K <= 256 and c <= 3) whereas mixing levels would drop the low bits of the
// smaller one.  Products with p+q > S+1 are dropped: S slices keep S(S+1)/2
// products in S levels (S x 64 TMEM columns) and give about 2^-8S relative to
// sigma_i tau_j.
//
// Complex to real: [Cr Ci] = [Ar Ai] [[Br Bi], [-Bi Br]], i.e. a real GEMM of
// M = n, N = 2n, K' = 2K.  The real depth K' runs over groups of 16 complex
// indices, each group [Re 16 | Im 16] (kpos below), so that one 32-wide
// k-block holds both parts of 16 complex indices; B' columns 2j and 2j+1
// are Re and Im of output column j.
//
// Staging layouts (bf16, K-major for both UMMA operands, tiled by k-block so
// that one TMA box is one contiguous block):
//   A'[item][s][kb][M'][32]   M' = 128 * mtiles, kb < kblocks = ceil(K/16)
//   B'[item][s][kb][N'][32]   N' = 64 * ntiles (zero padded)
// A tiles reach shared memory by TMA (3-D tensor maps, 64-byte swizzle).  B
// tiles either the same way from B' or, fused, straight from the FP64 B: TMA
// brings its values into a ring of shared memory and converting warps form
// the slices beside the tensor core.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>
#include <string>
#include <cstring>
#include <vector>

#include "../../include/skkr_gpu.h"
#include "kernels.h"
#include "slicing.cuh"

namespace {

constexpr int NT = 64;            // N tile (TMEM columns per accumulator)
constexpr int MT = 128;           // M tile (UMMA M)
constexpr int KB = 32;            // K per k-block (one 64-byte swizzle row of bf16)
constexpr int OZ_SMEM_MAX = 232448;  // shared memory one CTA may use (opt-in)
constexpr int OZ_A_SLICE = MT * KB * 2, OZ_B_SLICE = NT * KB * 2;  // bytes of one slice's A / B tile of a k-block
// accumulator sets: up to four slices (4 x 64 columns) leave room for a second
// set, so that one tile's MMAs run while the previous tile's sums are read
__host__ __device__ constexpr int oz_bufs(int S) { return S <= 4 ? 2 : 1; }
// Shared memory of S slices: a ring of A k-blocks (TMA), one of B k-blocks
// (TMA, or formed here: fused) and, fused, one of FP64 k-blocks of B, the raw
// values the conversion reads (32 columns of 16 values, as two TMA boxes of
// eight values = 128 bytes per column, 128-byte swizzle).
constexpr int OZ_RAW_BYTES = (NT / 2) * 16 * 16;
constexpr int OZ_SMEM_RINGS = OZ_SMEM_MAX - 1024 - 4096;  // alignment, OzShared
__host__ __device__ constexpr int oz_min(int a, int b) { return a < b ? a : b; }
__host__ __device__ constexpr int oz_a_stages(int S, bool fused) {
  return !fused ? oz_min(6, OZ_SMEM_RINGS / (S * (OZ_A_SLICE + OZ_B_SLICE))) : S <= 3 ? 4 : S <= 6 ? 3 : 2;
}
__host__ __device__ constexpr int oz_b_stages(int S, bool fused) {
  return !fused ? oz_a_stages(S, false) : S <= 3 ? 4 : S == 4 ? 3 : 2;
}
__host__ __device__ constexpr int oz_ring_bytes(int S, bool fused) {
  return S * (oz_a_stages(S, fused) * OZ_A_SLICE + oz_b_stages(S, fused) * OZ_B_SLICE);
}
__host__ __device__ constexpr int oz_raw_stages(int S) {
  return oz_min(8, (OZ_SMEM_RINGS - oz_ring_bytes(S, true)) / OZ_RAW_BYTES);
}
constexpr long long WAIT_LIMIT = 1LL << 22;
// The TMA lane of A (warp 0), the MMA lane (warp 1), the column scales (warp
// 2), the TMA lane of B's raw values (warp 3), the epilogue (warps 4-11) and
// the conversion of B: one group of four warps (16 warps in all, 128 registers
// a thread), or two groups taking alternate k-blocks where the epilogue does
// with 96 registers (up to four slices: few MMAs per k-block, so that the
// conversion sets the pace).
constexpr int OZ_EPI0 = 4, OZ_EPI_WARPS = 8, OZ_CONV0 = 12;
__host__ __device__ constexpr int oz_conv_groups(int S) { return S <= 4 ? 2 : 1; }
__host__ __device__ constexpr int oz_threads(int S) { return 32 * (OZ_CONV0 + 4 * oz_conv_groups(S)); }
constexpr int OZ_SCALE_RING = 4;  // tiles the column scales may run ahead of the conversion
constexpr int OZ_EXP_RING = 16;   // tiles whose column scales are kept

// ------------------------------------------------------------------ PTX helpers
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// bounded wait: false when the limit is reached
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity) {
  for (long long i = 0; i < WAIT_LIMIT; i++)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}
__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *tm, int c0, int c1, int c2,
                                            uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::
          "r"(smem_u32(dst)),
      "l"((uint64_t)tm), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar))
      : "memory");
}
// a load that the compiler keeps in program order (a batch of them is then in
// flight together)
__device__ __forceinline__ uint32_t load_u32(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ void tma_load_4d(void *dst, const CUtensorMap *tm, int c0, int c1, int c2, int c3,
                                            uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::
          "r"(smem_u32(dst)),
      "l"((uint64_t)tm), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(bar))
      : "memory");
}
// the 128-byte line of p towards L2
__device__ __forceinline__ void prefetch_l2(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
// bytes (a multiple of 16, 16-byte aligned) of global memory towards L2
__device__ __forceinline__ void bulk_prefetch_l2(const void *p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tmem_alloc(uint32_t *dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma_bf16(uint32_t dtmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(dtmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// 8 / 4 consecutive accumulator columns of this warp's 32 TMEM lanes, without
// the wait (tmem_ld_wait after a batch of loads)
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t *r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t *r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// UMMA shared-memory descriptor: K-major, 64-byte swizzle (rows of 32 bf16),
// 8-row groups 512 bytes apart (tile base 512-byte aligned).
__device__ __forceinline__ uint64_t sdesc_sw64(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
  d |= (uint64_t)1 << 16;           // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(512 >> 4) << 32;  // stride byte offset: 8 rows x 64 bytes
  d |= (uint64_t)1 << 46;           // descriptor version
  d |= (uint64_t)4 << 61;           // 64-byte swizzle
  return d;
}
// instruction descriptor: BF16 x BF16 -> FP32, K-major A and B, M x N
__host__ __device__ constexpr uint32_t idesc_bf16(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// ------------------------------------------------------------------ slicing
// (abs_bits, scale_exp, slice_digits, digit_bits, slice4: slicing.cuh)

// element (row r, K' index kk) of one slice region in the k-block tiled layout
__device__ __forceinline__ long long tiled(int r, int kk, int rows) {
  return ((long long)(kk >> 5) * rows + r) * 32 + (kk & 31);
}
// K' index of the real (im = 0) or imaginary (im = 1) part of complex index k
__host__ __device__ __forceinline__ int kpos(int k, int im) { return ((k >> 4) << 5) + (im << 4) + (k & 15); }

// the S words at dst + p sstride, sign bits flipped by `flip` (0 or 0x80008000)
template <int S>
__device__ __forceinline__ void store_words(const uint32_t (&w)[S][2], uint32_t flip, __nv_bfloat16 *dst,
                                            long long sstride) {
#pragma unroll
  for (int p = 0; p < S; p++)
    *reinterpret_cast<uint2 *>(dst + p * sstride) = make_uint2(w[p][0] ^ flip, w[p][1] ^ flip);
}
// one element, slices p = 0..S-1 (the shapes of no four-element group)
template <int S, int DB>
__device__ __forceinline__ void store1(const int (&dg)[S], int wshift, uint16_t flip, __nv_bfloat16 *dst,
                                       long long sstride) {
#pragma unroll
  for (int p = 0; p < S; p++) {
    const float sc = pow2f(wshift - DB * p);
    const uint16_t h = (uint16_t)(digit_bits(dg[p], sc, -12582912.0f * sc) >> 16) ^ flip;
    *reinterpret_cast<uint16_t *>(dst + p * sstride) = h;
  }
}

// A' = [Re A, Im A] (n x 2K, in the K' order) from the n x K complex A; rows scaled by their
// max over these K columns.  32 rows per block: the row maxima, then 32 x 32
// tiles transposed through shared memory, each thread taking four
// consecutive columns of one row (8-byte stores of every slice) when K is a
// multiple of four, one element otherwise.
// H (n <= 64, see k_ozaki): row 64 + r of A' is [Im A, Re A] and row r
// [Re A, -Im A].
template <int S, int DB, int H>
__global__ void __launch_bounds__(256) k_split_a(MatRef A, int n, int K, int nc, const int *__restrict__ act,
                                                 __nv_bfloat16 *__restrict__ out, int Mp, int Kp,
                                                 int *__restrict__ sigma) {
  const int item = blockIdx.y, kk0 = item / nc, cc = item % nc;
  if (act && !act[item]) return;
  const zd *a = mat_ptr(A, kk0, cc);
  const int r0 = blockIdx.x * 32, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __shared__ unsigned long long red[8][32];
  __shared__ int sc[32];
  __shared__ zd T[32][33];
  unsigned long long m = 0;
  const int row = r0 + lane;
  if (row < n)
    for (int k = w; k < K; k += 8) {
      zd v = a[row + (long long)k * A.ld];
      const unsigned long long bx = abs_bits(v.x), by = abs_bits(v.y);
      m = bx > m ? bx : m;
      m = by > m ? by : m;
    }
  red[w][lane] = m;
  __syncthreads();
  if (w == 0) {
    unsigned long long mm = 0;
    for (int q = 0; q < 8; q++) mm = red[q][lane] > mm ? red[q][lane] : mm;
    const int es = scale_exp(mm);
    sc[lane] = es;
    if (r0 + lane < (H ? MT / 2 : Mp)) sigma[(long long)item * Mp + r0 + lane] = es;
    if (H && r0 + lane < MT / 2) sigma[(long long)item * Mp + MT / 2 + r0 + lane] = es;
  }
  __syncthreads();
  const long long sstride = (long long)Mp * Kp;
  __nv_bfloat16 *base = out + (long long)item * S * sstride;
  const bool vec = (K & 3) == 0;
  for (int c0 = 0; c0 < K; c0 += 32) {
    for (int q = w; q < 32; q += 8) {
      int col = c0 + q;
      T[lane][q] = (row < n && col < K) ? a[row + (long long)col * A.ld] : make_double2(0.0, 0.0);
    }
    __syncthreads();
    if (vec) {
      // thread t: row r0 + t / 8, columns c0 + 4 (t % 8) .. +3
      const int q = threadIdx.x >> 3, c4 = (threadIdx.x & 7) * 4, r = r0 + q, col = c0 + c4;
      if (r < n && col < K) {
        double re[4], im[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
          re[e] = T[q][c4 + e].x;
          im[e] = T[q][c4 + e].y;
        }
        uint32_t wr[S][2], wi[S][2];
        slice4<S, DB>(re, im, sc[q], 0, wr, wi);
        store_words<S>(wr, 0u, base + tiled(r, kpos(col, 0), Mp), sstride);
        store_words<S>(wi, H ? 0x80008000u : 0u, base + tiled(r, kpos(col, 1), Mp), sstride);
        if (H) {
          store_words<S>(wi, 0u, base + tiled(MT / 2 + r, kpos(col, 0), Mp), sstride);
          store_words<S>(wr, 0u, base + tiled(MT / 2 + r, kpos(col, 1), Mp), sstride);
        }
      }
    } else {
      for (int q = w; q < 32; q += 8) {
        const int r = r0 + q, col = c0 + lane;
        if (r < n && col < K) {
          const int es = sc[q];
          const zd v = T[q][lane];
          int dr[S], di[S];
          slice_digits<S, DB>(v.x, es, dr);
          slice_digits<S, DB>(v.y, es, di);
          store1<S, DB>(dr, 0, 0, base + tiled(r, kpos(col, 0), Mp), sstride);
          store1<S, DB>(di, 0, H ? 0x8000 : 0, base + tiled(r, kpos(col, 1), Mp), sstride);
          if (H) {
            store1<S, DB>(di, 0, 0, base + tiled(MT / 2 + r, kpos(col, 0), Mp), sstride);
            store1<S, DB>(dr, 0, 0, base + tiled(MT / 2 + r, kpos(col, 1), Mp), sstride);
          }
        }
      }
    }
    __syncthreads();
  }
}

// B'^T from the K x n complex B: one warp per column j; rows 2j and 2j+1 of
// B'^T are [Re B(:,j), -Im B(:,j)] and [Im B(:,j), Re B(:,j)] (columns scaled
// by their max over these K rows), so that the real and imaginary parts of an
// output element land in adjacent accumulator columns of one thread.  Each
// lane takes four consecutive rows k (8-byte stores) when K is a multiple of
// four, one row otherwise; each digit is formed once and stored twice, -Im
// with its sign bit flipped.
// H (n <= 64): row j of B'^T is [Re B(:,j), Im B(:,j)].
template <int S, int DB, int H>
__global__ void __launch_bounds__(256, 3) k_split_b(MatRef B, int n, int K, int nc, const int *__restrict__ act,
                                                 __nv_bfloat16 *__restrict__ out, int Np, int Kp,
                                                 int *__restrict__ tau) {
  const int item = blockIdx.y, kk0 = item / nc, cc = item % nc;
  if (act && !act[item]) return;
  const int lane = threadIdx.x & 31, j = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (j >= n) return;
  const zd *b = mat_ptr(B, kk0, cc) + (long long)j * B.ld;
  unsigned long long m = 0;
  for (int k = lane; k < K; k += 32) {
    zd v = b[k];
    const unsigned long long bx = abs_bits(v.x), by = abs_bits(v.y);
    m = bx > m ? bx : m;
    m = by > m ? by : m;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long t = __shfl_xor_sync(0xffffffffu, m, o);
    m = t > m ? t : m;
  }
  const int es = scale_exp(m);
  if (lane == 0) tau[(long long)item * n + j] = es;
  const long long sstride = (long long)Np * Kp;
  __nv_bfloat16 *base = out + (long long)item * S * sstride;
  if ((K & 3) == 0) {
    for (int k = 4 * lane; k < K; k += 128) {
      double re[4], im[4];
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const zd v = b[k + e];
        re[e] = v.x;
        im[e] = v.y;
      }
      uint32_t wr[S][2], wi[S][2];
      slice4<S, DB>(re, im, es, 16, wr, wi);
      if (H) {
        store_words<S>(wr, 0u, base + tiled(j, kpos(k, 0), Np), sstride);
        store_words<S>(wi, 0u, base + tiled(j, kpos(k, 1), Np), sstride);
        continue;
      }
      store_words<S>(wr, 0u, base + tiled(2 * j, kpos(k, 0), Np), sstride);
      store_words<S>(wi, 0x80008000u, base + tiled(2 * j, kpos(k, 1), Np), sstride);
      store_words<S>(wi, 0u, base + tiled(2 * j + 1, kpos(k, 0), Np), sstride);
      store_words<S>(wr, 0u, base + tiled(2 * j + 1, kpos(k, 1), Np), sstride);
    }
  } else {
    for (int k = lane; k < K; k += 32) {
      const zd v = b[k];
      int dr[S], di[S];
      slice_digits<S, DB>(v.x, es, dr);
      slice_digits<S, DB>(v.y, es, di);
      if (H) {
        store1<S, DB>(dr, 16, 0, base + tiled(j, kpos(k, 0), Np), sstride);
        store1<S, DB>(di, 16, 0, base + tiled(j, kpos(k, 1), Np), sstride);
        continue;
      }
      store1<S, DB>(dr, 16, 0, base + tiled(2 * j, kpos(k, 0), Np), sstride);
      store1<S, DB>(di, 16, 0x8000, base + tiled(2 * j, kpos(k, 1), Np), sstride);
      store1<S, DB>(di, 16, 0, base + tiled(2 * j + 1, kpos(k, 0), Np), sstride);
      store1<S, DB>(dr, 16, 0, base + tiled(2 * j + 1, kpos(k, 1), Np), sstride);
    }
  }
}

// ------------------------------------------------------------------ the GEMM
struct OzArgs {
  int n, mtiles, ntiles, kblocks, nc, mode;
  int tiles;            // items x mtiles x ntiles
  const int *sigma;     // [item][M']  row scale exponents of A
  const int *tau;       // [item][n]   column scale exponents of B (staged B)
  MatRef B;             // the FP64 K x n operand B (fused B)
  int K;
  MatRef C, D, E;
  const int *act;
  int *err;
};

// The exact integer sum of one level, from its FP32 accumulator (integer
// times 2^(16 - DB l))
template <int DB>
__device__ __forceinline__ int level_int(uint32_t v, int l) {
  return __float2int_rn(__uint_as_float(v) * pow2f(DB * l - 16));
}
// The weighted sum of the S levels of one output in units of level
// min(S - 1, 5) (weight 2^(-5 DB) of level 0 at most: 62 bits hold it, as
// |N_0| <= 2^22); seven slices round level 6 into that unit.  Eight, which
// stand for FP64, keep what the levels 6 and 7 add: the lowest bit tells the
// unit, 1 for level 6 while the sum stays below 2^55 units of level 5 (it then
// fits there), 0 for level 5 above, where a double's last place is eight of
// them.  In level 5's unit throughout, an output far below sigma_i tau_j lost
// digits that its slices hold: 2^-55 sigma_i tau_j, now 2^-60; 110 products of
// n = 128 take 67.2 us as before with staged B, 75 for 70 with fused B.  32 x
// 32 + 64 bit multiply-adds with constant powers of two.
template <int S, int DB, int W>
__device__ __forceinline__ long long levels_sum(const uint32_t (&v)[S][W], int t) {
  constexpr int B1 = 1 << DB, B2 = 1 << (2 * DB);
  const long long hi = (long long)level_int<DB>(v[0][t], 0) * B2 +
                       ((long long)level_int<DB>(v[1][t], 1) * B1 + level_int<DB>(v[2][t], 2));
  if constexpr (S == 3) return hi;
  if constexpr (S == 4) return hi * B1 + level_int<DB>(v[3][t], 3);
  if constexpr (S == 5)
    return hi * B2 + ((long long)level_int<DB>(v[3][t], 3) * B1 + level_int<DB>(v[4][t], 4));
  if constexpr (S >= 6) {
    long long lo = (long long)level_int<DB>(v[3][t], 3) * B2 +
                   ((long long)level_int<DB>(v[4][t], 4) * B1 + level_int<DB>(v[5][t], 5));
    if constexpr (S == 7) lo += (level_int<DB>(v[6][t], 6) + B1 / 2) >> DB;
    const long long sum = (hi << (3 * DB)) + lo;
    if constexpr (S < 8) return sum;
    // level 6 with level 7 rounded into it; the sum's upper word decides the unit.  (Both
    // values, then the choice: chosen terms cost twice the spilled registers.)
    const int low = level_int<DB>(v[6][t], 6) + ((level_int<DB>(v[7][t], 7) + B1 / 2) >> DB);
    const bool small = (unsigned)((int)(sum >> 32) + (1 << 23) - 1) < (1u << 24) - 2u;
    const long long fine = (sum << DB) + ((low + 1) | 1);
    const long long coarse = (sum + ((low + B1) >> DB)) & ~1ll;
    return small ? fine : coarse;
  }
}
// round-to-nearest-even double of a * 2^e from integer operations only (the
// FP64 pipe of this GPU is ~1/40 of the integer rate): normalise with a
// leading-zero count, keep 53 bits, round on the dropped 11, add e to the
// exponent (the leading one and a carry of the rounding add into the exponent
// field).  Equal to __ll2double_rn(a) * 2^e for normal results; a result
// below the normal range is 0, one above it infinite.
__device__ __forceinline__ double fix_to_double(long long a, int e) {
  const unsigned long long sign = (unsigned long long)a & 0x8000000000000000ull;
  unsigned long long m = a < 0 ? 0ull - (unsigned long long)a : (unsigned long long)a;
  const int lz = __clzll((long long)m);
  m <<= (lz & 63);                             // leading one at bit 63
  unsigned long long mant = m >> 11;           // 53 significant bits
  mant += (((unsigned)m & 0x7FFu) + ((unsigned)mant & 1u)) > 0x400u ? 1ull : 0ull;
  const int bx = 63 - lz + e + 1022;           // biased exponent less the leading one
  unsigned long long r = ((unsigned long long)(unsigned)bx << 52) + mant;
  r = bx >= 2046 ? 0x7FF0000000000000ull : r;
  r = (a == 0 || bx < 0) ? 0ull : r;
  return __longlong_as_double((long long)(sign | r));
}
// levels_sum's value, e the exponent of level min(S - 1, 5)'s unit
template <int S, int DB>
__device__ __forceinline__ double level_value(long long a, int e) {
  if constexpr (S < 8) return fix_to_double(a, e);
  return fix_to_double(a & ~1ll, e - ((a & 1) ? DB : 0));
}

// byte offset of bf16 (row r, column t < 32) in a K-major tile of 64-byte rows
// with the 64-byte swizzle, as TMA lays it out and the UMMA descriptor reads
// it: the 16-byte chunk index XORed with address bits 7-8 (bits 1-2 of r)
__device__ __forceinline__ uint32_t sw64_off(int r, int t) {
  return (uint32_t)(r * 64 + ((((t >> 3) ^ (r >> 1)) & 3) << 4) + ((t & 7) << 1));
}

// One CTA's walk over its tiles (t = blockIdx.x, + gridDim.x, ...; the N tiles
// of an item side by side, so that they read its A slices from L2 together),
// tiles of masked items left out; the mask of the tile after next is loaded
// ahead.  Every role walks the same list.
struct TileWalk {
  const OzArgs &g;
  int t, i, next_on;  // tile, its number in this CTA's list, mask of the next candidate
  __device__ __forceinline__ explicit TileWalk(const OzArgs &g_) : g(g_), t((int)blockIdx.x - (int)gridDim.x), i(-1) {
    next_on = on(t + (int)gridDim.x);
    step();
  }
  __device__ __forceinline__ int on(int u) const {
    return (g.act && u < g.tiles) ? g.act[u / (g.mtiles * g.ntiles)] : 1;
  }
  __device__ __forceinline__ void step() {
    int keep;
    do {
      t += (int)gridDim.x;
      keep = next_on;
      next_on = on(t + (int)gridDim.x);
    } while (t < g.tiles && !keep);
    i++;
  }
  __device__ __forceinline__ bool valid() const { return t < g.tiles; }
  __device__ __forceinline__ int item() const { return t / (g.mtiles * g.ntiles); }
  __device__ __forceinline__ int mt() const { return t % (g.mtiles * g.ntiles) / g.ntiles; }
  __device__ __forceinline__ int nt() const { return t % g.ntiles; }
};

struct OzShared {
  __align__(8) uint64_t a_full[6], a_empty[6], b_full[6], b_empty[6], raw_full[8], raw_empty[8];
  uint64_t acc_full[2], acc_empty[2], sc_full[OZ_SCALE_RING], sc_empty[OZ_SCALE_RING], done;
  uint32_t tmem_base;
  volatile int failed;
  volatile int a_issued, raw_issued;      // k-blocks asked for (counts over all tiles)
  short col_exp[OZ_EXP_RING][NT];         // column scale exponents of each tile's complex columns
};

// the warp waits for a phase of a barrier; false (for the whole warp) once
// anything failed
__device__ __forceinline__ bool oz_warp_wait(OzShared &sh, uint64_t *bar, uint32_t parity, bool skip = false) {
  if (skip || __all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  int ok = 1;
  if ((threadIdx.x & 31) == 0) ok = !sh.failed && mbar_wait(bar, parity);
  ok = __shfl_sync(0xffffffffu, ok, 0);
  if (!ok) sh.failed = 1;
  return ok != 0;
}

// n rows of an operand's tile's columns towards L2, one column per lane
__device__ __forceinline__ void oz_prefetch(const zd *p, int ld, int rows, int cols) {
  for (int c = threadIdx.x & 31; c < cols; c += 32)
    bulk_prefetch_l2(p + (long long)c * ld, (uint32_t)rows * (uint32_t)sizeof(zd));
}

// raw blocks (32 columns each) of a k-block of fused B
template <int H>
__device__ __forceinline__ int oz_raw_passes(const OzArgs &g) {
  return H && g.n > 32 ? 2 : 1;
}

// Scale exponents of the columns c0 .. c0 + 7 of B (nj columns from b) over the
// whole depth: column c0 + lane % 8's in every lane, 0 past the last.
__device__ __forceinline__ int oz_exps8(const OzArgs &g, const zd *b, int c0, int nj) {
  const int lane = threadIdx.x & 31;
  unsigned m[8];
#pragma unroll
  for (int c = 0; c < 8; c++) m[c] = 0;
#pragma unroll 1
  for (int kc = 0; kc < g.K; kc += 128) {
    // indices past the end repeat the last one: every load is valid and
    // all of them are in flight together
    unsigned v[8][8];
#pragma unroll
    for (int c = 0; c < 8; c++)
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const uint32_t *q = reinterpret_cast<const uint32_t *>(b + min(kc + lane + 32 * e, g.K - 1) +
                                                               (long long)min(c0 + c, nj - 1) * g.B.ld);
        v[c][2 * e] = load_u32(q + 1);
        v[c][2 * e + 1] = load_u32(q + 3);
      }
#pragma unroll
    for (int c = 0; c < 8; c++)
#pragma unroll
      for (int e = 0; e < 8; e++) m[c] = max(m[c], v[c][e] & 0x7FFFFFFFu);
  }
  int mine = 0;
#pragma unroll
  for (int c = 0; c < 8; c++) {
    const unsigned t = __reduce_max_sync(0xffffffffu, m[c]);
    if ((lane & 7) == c && c0 + c < nj) mine = scale_exp((unsigned long long)t << 32);
  }
  return mine;
}

// The scale role (warp 2, fused B only): the exponents of each tile's 32
// columns of B over the whole depth K, into the ring the conversion and the
// epilogue read, with the columns of B two tiles ahead started towards L2.
// Only the exponent field of a value matters (scale_exp), so the maxima run on
// the upper words, and only those are loaded (64 loads of a lane in flight:
// the role's pace is its load latency).  The first tile's are the conversion
// warps' own work, which have nothing else yet: four warps at once (30
// products of n = 128, one tile an SM, eight slices: 49 -> 44 us).  A ring slot of exponents is free
// again when the role returns to it: it runs at most four tiles ahead of the
// conversion, the conversion at most four k-blocks, hence five tiles, ahead of
// the MMAs, and those wait for the epilogue of the tile oz_bufs before.
template <int H>
__device__ __forceinline__ void oz_scales(const OzArgs &g, OzShared &sh) {
  constexpr int NC = H ? NT : NT / 2;  // complex columns of a tile
  const int lane = threadIdx.x & 31;
  auto prefetch_b = [&](const TileWalk &w) {
    const int item = w.item(), j0 = w.nt() * NC;
    if (w.valid())
      oz_prefetch(mat_ptr(g.B, item / g.nc, item % g.nc) + (long long)j0 * g.B.ld, g.B.ld, g.K,
                  g.n - j0 < NC ? g.n - j0 : NC);
  };
  TileWalk wp(g);
  prefetch_b(wp);
  wp.step();
  prefetch_b(wp);
  if (wp.valid()) wp.step();
  prefetch_b(wp);
  TileWalk w(g);
  if (w.valid()) w.step();
  for (; w.valid(); w.step()) {
    const int item = w.item(), j0 = w.nt() * NC, nj = g.n - j0 < NC ? g.n - j0 : NC;
    if (wp.valid()) wp.step();
    prefetch_b(wp);
    if (!oz_warp_wait(sh, &sh.sc_empty[w.i % OZ_SCALE_RING], ((w.i / OZ_SCALE_RING) - 1) & 1, w.i < OZ_SCALE_RING))
      break;
    const zd *b = mat_ptr(g.B, item / g.nc, item % g.nc) + (long long)j0 * g.B.ld;
    int mine = 0, mine1 = 0;  // columns lane and 32 + lane
#pragma unroll 1
    for (int c0 = 0; c0 < nj; c0 += 8) {
      const int e = oz_exps8(g, b, c0, nj);
      if ((lane & ~7) == (c0 & 31)) (H && c0 >= 32 ? mine1 : mine) = e;
    }
    sh.col_exp[w.i % OZ_EXP_RING][lane] = (short)mine;
    if (H) sh.col_exp[w.i % OZ_EXP_RING][lane + 32] = (short)mine1;
    __syncwarp();
    if (lane < 4) mbar_arrive(&sh.sc_full[w.i % OZ_SCALE_RING]);  // (as the four conversion warps for the first tile)
  }
}

// The conversion role (fused B): the S B tiles of every k-block, eight columns
// per warp.  A thread takes one column and the four complex indices
// 16 kb + 4 (lane % 4) .. +3, forms their digits once and stores them four
// times (rows 2j and 2j+1, the Re and Im halves of the k-block, -Im with
// flipped sign bits).  Each thread orders its stores before the tensor core's
// reads (proxy fence); lane 0, after the warp's barrier, arrives on the
// stage's full barrier.  (Values outside the matrix arrive as zeros.)
// H: 64 columns of one row each, in passes of 32 columns that each take a raw
// block; two stores a value.
template <int S, int DB, int NB, int NRAW, int H>
__device__ __forceinline__ void oz_convert(const OzArgs &g, OzShared &sh, unsigned char *sb0, const unsigned char *raw) {
  const int cw = (threadIdx.x >> 5) - OZ_CONV0, lane = threadIdx.x & 31;
  const int nkb = g.kblocks, jl = 8 * (cw & 3) + (lane >> 2), kq = 4 * (lane & 3);
  const int r = H ? jl : 2 * jl, npass = oz_raw_passes<H>(g);
  const uint32_t o0 = sw64_off(r, kq), o1 = sw64_off(r, kq + 16), o2 = sw64_off(r + 1, kq),
                 o3 = sw64_off(r + 1, kq + 16);
  // this thread's 16-byte values in a raw block: box kq / 8, row jl, chunks kq % 8 .. +3 XORed with jl % 8
  const unsigned char *src = raw + (kq >> 3) * (OZ_RAW_BYTES / 2) + jl * 128;
  for (TileWalk w(g); w.valid(); w.step()) {
    if (w.i == 0 && cw < 4) {  // the first tile's scales: eight columns a warp (and a pass)
      const int j0 = w.nt() * (H ? NT : NT / 2), nj = min(g.n - j0, H ? NT : NT / 2);
      const zd *b = mat_ptr(g.B, w.item() / g.nc, w.item() % g.nc) + (long long)j0 * g.B.ld;
#pragma unroll 1
      for (int c0 = 8 * cw; c0 < 32 * npass; c0 += 32) {
        const int e = oz_exps8(g, b, c0, nj);
        if (lane < 8) sh.col_exp[0][c0 + lane] = (short)e;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh.sc_full[0]);
    }
    if (!oz_warp_wait(sh, &sh.sc_full[w.i % OZ_SCALE_RING], (w.i / OZ_SCALE_RING) & 1)) return;
    for (int kb = cw >> 2; kb < nkb; kb += oz_conv_groups(S)) {
      const int kc = w.i * nkb + kb, st = kc % NB;
#pragma unroll 1
      for (int pass = 0; pass < npass; pass++) {
        const int rc = kc * npass + pass, rr = rc % NRAW, es = sh.col_exp[w.i % OZ_EXP_RING][jl + 32 * pass];
        if (!oz_warp_wait(sh, &sh.raw_full[rr], (rc / NRAW) & 1)) return;
        double re[4], im[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const zd v = *reinterpret_cast<const zd *>(src + rr * OZ_RAW_BYTES + ((((kq & 7) + e) ^ (jl & 7)) << 4));
          re[e] = v.x;
          im[e] = v.y;
        }
        uint32_t wr[S][2], wi[S][2];
        if constexpr (DB == 8) slice4b<S>(re, im, es, wr, wi);
        else slice4<S, DB>(re, im, es, 16, wr, wi);
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh.raw_empty[rr]);
        // the stores come after the tensor core's reads of the stage
        if (pass == 0 && !oz_warp_wait(sh, &sh.b_empty[st], ((kc / NB) - 1) & 1, kc < NB)) return;
        unsigned char *sb = sb0 + st * (S * OZ_B_SLICE) + pass * (32 * KB * 2);
#pragma unroll
        for (int p = 0; p < S; p++) {
          unsigned char *tp = sb + p * OZ_B_SLICE;
          *reinterpret_cast<uint2 *>(tp + o0) = make_uint2(wr[p][0], wr[p][1]);
          if constexpr (H) {
            *reinterpret_cast<uint2 *>(tp + o1) = make_uint2(wi[p][0], wi[p][1]);
          } else {
            *reinterpret_cast<uint2 *>(tp + o1) = make_uint2(wi[p][0] ^ 0x80008000u, wi[p][1] ^ 0x80008000u);
            *reinterpret_cast<uint2 *>(tp + o2) = make_uint2(wi[p][0], wi[p][1]);
            *reinterpret_cast<uint2 *>(tp + o3) = make_uint2(wr[p][0], wr[p][1]);
          }
        }
      }
      // every lane's stores visible to the tensor core, then one arrival per warp
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh.b_full[st]);
    }
    if (lane == 0) mbar_arrive(&sh.sc_empty[w.i % OZ_SCALE_RING]);
  }
}

// The epilogue role (warps 4-11): warp w reads TMEM lanes 32 (w % 4) .. +31
// (rows of the M tile) and one half of the tile's 64 columns, as one 64-bit
// integer per output.  With one accumulator set the level sums of the whole
// tile are combined first and the accumulators handed back to the MMAs; the
// rounding to FP64 and the update of C, D, E run beside the next tile's MMAs.
template <int S, int DB, int FB>
__device__ __forceinline__ void oz_epilogue(const OzArgs &g, OzShared &sh, uint32_t tbase) {
  constexpr int NBUF = oz_bufs(S), CH = S <= 6 ? 8 : 4;  // columns per TMEM load (registers)
  constexpr bool EARLY = NBUF == 1;  // hand the accumulators back before the rounding
  constexpr int NA = EARLY ? 32 : CH, NO = EARLY ? 8 : 4;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int quarter = warp & 3, half = (warp - OZ_EPI0) >> 2;
  const int mode = g.mode;
  const bool rd = mode == 1 || mode == 5 || mode == 2 || mode == 3, rd_c = mode == 1 || mode == 5;
  const double nan = __longlong_as_double(0x7FF8000000000000ll);
  for (TileWalk w(g); w.valid(); w.step()) {
    const int item = w.item(), kk = item / g.nc, cc = item % g.nc, buf = w.i % NBUF;
    const int row = w.mt() * MT + quarter * 32 + lane, j0 = w.nt() * (NT / 2) + half * 16;
    // level 0 carries 2^(sigma_i + tau_j - 2 (DB - 1)); levels_sum is in units of level min(S - 1, 5)
    const int sig = row < g.n ? g.sigma[(long long)item * (g.mtiles * MT) + row] : 0;
    const int erow = sig - 2 * (DB - 1) - DB * (S - 1 < 5 ? S - 1 : 5);
    const int nq = row < g.n ? g.n - j0 : 0;  // columns of this thread's row inside the matrix
    zd *pc = mat_ptr(g.C, kk, cc) + row + (long long)j0 * g.C.ld;
    zd *pd = mat_ptr(g.D, kk, cc) + row + (long long)j0 * g.D.ld;
    zd *pe = mat_ptr(g.E, kk, cc) + row + (long long)j0 * g.E.ld;
    // modes that read the old C (1, 5) or D (2, 3) load it ahead
    const zd *src = rd_c ? pc : pd;
    const long long sld = rd_c ? g.C.ld : g.D.ld;
    // the column scales: of the scale role (fused B), or of the split
    auto ce = [&](int q) {
      return FB ? (int)sh.col_exp[w.i % OZ_EXP_RING][half * 16 + q] : g.tau[(long long)item * g.n + j0 + q];
    };
    zd old[NO];
    auto load_old = [&](const zd *src, long long sld, int q0) {  // columns q0 .. q0 + NO - 1
#pragma unroll
      for (int q = 0; q < NO; q++)
        if (q0 + q < nq) old[q] = src[(q0 + q) * sld];
    };
    // one output (column q of this thread's row) into C (mode 2: into D), `o` its old C or D
    auto emit = [&](zd val, int q, zd o) {
      zd *out = (mode == 2 ? pd : pc) + q * (long long)(mode == 2 ? g.D.ld : g.C.ld);
      if (mode == 0) *out = val;
      else if (mode == 4) *out = make_double2(row == j0 + q ? 1.0 - val.x : -val.x, -val.y);
      else if (mode == 5) *out = zadd(o, val);
      else *out = zsub(o, val);
    };
    // the level sums in FP64; a row of A or a column of B that holds an infinity or a NaN has no digits
    auto value = [&](long long ar, long long ai, int q) {
      const int tj = ce(q);
      zd val = make_double2(level_value<S, DB>(ar, erow + tj), level_value<S, DB>(ai, erow + tj));
      if (sig == SCALE_NONFINITE || tj == SCALE_NONFINITE) val = make_double2(nan, nan);
      return val;
    };
    if (!EARLY && rd) load_old(src, sld, 0);
    if (rd) {
      // the next tile's old values towards L2: 16 columns x 512 bytes of this
      // warp, one 128-byte line per lane and step
      TileWalk wn = w;
      wn.step();
      if (wn.valid()) {
        const int in = wn.item(), rn = wn.mt() * MT + quarter * 32 + 8 * (lane & 3), jn = wn.nt() * (NT / 2) + half * 16;
        const MatRef &M = rd_c ? g.C : g.D;
        const zd *p = mat_ptr(M, in / g.nc, in % g.nc) + rn;
        const zd *pe2 = mat_ptr(g.E, in / g.nc, in % g.nc) + rn;
#pragma unroll
        for (int q = 0; q < 16; q += 8) {
          const int j = jn + q + (lane >> 2);
          if (rn < g.n && j < g.n) {
            prefetch_l2(p + (long long)j * M.ld);
            if (mode == 2) prefetch_l2(pe2 + (long long)j * g.E.ld);
          }
        }
      }
    }
    if (!oz_warp_wait(sh, &sh.acc_full[buf], (w.i / NBUF) & 1)) break;
    tc_fence_after();
    const uint32_t ta = tbase + ((uint32_t)(quarter * 32) << 16) + buf * 256 + half * 32;
    long long acc[NA];
#pragma unroll
    for (int c0 = 0; c0 < 32; c0 += CH) {
      uint32_t v[S][CH];
#pragma unroll
      for (int l = 0; l < S; l++) {
        if constexpr (CH == 8) tmem_ld8(ta + l * NT + c0, v[l]);
        else tmem_ld4(ta + l * NT + c0, v[l]);
      }
      tmem_ld_wait();
#pragma unroll
      for (int t = 0; t < CH; t++) acc[(EARLY ? c0 : 0) + t] = levels_sum<S, DB, CH>(v, t);
      if constexpr (!EARLY) {
        const int q0 = c0 / 2;
#pragma unroll
        for (int q = 0; q < CH / 2; q++)
          if (q0 + q < nq) {
            const zd val = value(acc[2 * q], acc[2 * q + 1], q0 + q);
            emit(val, q0 + q, old[q]);
            if (mode == 2) pe[(q0 + q) * (long long)g.E.ld] = zsub(pe[(q0 + q) * (long long)g.E.ld], val);
          }
        if (rd && q0 + NO < 16) load_old(src, sld, q0 + NO);
        __syncwarp();
      }
    }
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(&sh.acc_empty[buf]);
    if constexpr (EARLY) {
#pragma unroll
      for (int q0 = 0; q0 < 16; q0 += NO) {
        if (rd) load_old(src, sld, q0);
#pragma unroll
        for (int q = 0; q < NO; q++)
          if (q0 + q < nq) {
            const zd val = value(acc[(2 * (q0 + q)) % NA], acc[(2 * (q0 + q) + 1) % NA], q0 + q);
            emit(val, q0 + q, old[q]);
            acc[(2 * (q0 + q)) % NA] = __double_as_longlong(val.x);  // for E
            acc[(2 * (q0 + q) + 1) % NA] = __double_as_longlong(val.y);
          }
      }
      if (mode == 2) {
#pragma unroll
        for (int q0 = 0; q0 < 16; q0 += NO) {
          load_old(pe, g.E.ld, q0);
#pragma unroll
          for (int q = 0; q < NO; q++)
            if (q0 + q < nq)
              pe[(q0 + q) * (long long)g.E.ld] =
                  zsub(old[q], make_double2(__longlong_as_double(acc[(2 * (q0 + q)) % NA]),
                                            __longlong_as_double(acc[(2 * (q0 + q) + 1) % NA])));
        }
      }
    }
  }
}

// The epilogue role for stacked operands (H): rows 0-63 of the tile hold the
// real, rows 64-127 the imaginary parts, a TMEM column is one complex column;
// a thread updates one part of 32 outputs.  (The two parts of a row come from
// different warps: their 8-byte accesses meet in the cache.)
template <int S, int DB, int FB>
__device__ __forceinline__ void oz_epilogue_h(const OzArgs &g, OzShared &sh, uint32_t tbase) {
  constexpr int NBUF = oz_bufs(S), CH = S <= 6 ? 8 : 4;  // columns per TMEM load
  constexpr bool EARLY = NBUF == 1;                      // hand the accumulators back before the rounding
  constexpr int NA = EARLY ? 32 : CH, NO = 8;  // sums held, old values in a batch
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int quarter = warp & 3, half = (warp - OZ_EPI0) >> 2;
  const int mode = g.mode, part = quarter >> 1, row = (quarter & 1) * 32 + lane, j0 = half * 32;
  const int nq = row < g.n ? g.n - j0 : 0;  // columns of this thread's row inside the matrix
  const bool rd = mode == 1 || mode == 5 || mode == 2 || mode == 3, rd_c = mode == 1 || mode == 5;
  const double nan = __longlong_as_double(0x7FF8000000000000ll);
  for (TileWalk w(g); w.valid(); w.step()) {
    const int item = w.item(), kk = item / g.nc, cc = item % g.nc, buf = w.i % NBUF;
    const int sig = row < g.n ? g.sigma[(long long)item * MT + part * (MT / 2) + row] : 0;
    const int erow = sig - 2 * (DB - 1) - DB * (S - 1 < 5 ? S - 1 : 5);
    auto at = [&](const MatRef &M) {
      return reinterpret_cast<double *>(mat_ptr(M, kk, cc) + row + (long long)j0 * M.ld) + part;
    };
    double *pc = at(g.C), *pd = at(g.D), *pe = at(g.E);
    const double *src = rd_c ? pc : pd;
    const long long sld = 2ll * (rd_c ? g.C.ld : g.D.ld), eld = 2ll * g.E.ld, old_ld = 2ll * (mode == 2 ? g.D.ld : g.C.ld);
    double *out = mode == 2 ? pd : pc;
    auto ce = [&](int q) {
      return FB ? (int)sh.col_exp[w.i % OZ_EXP_RING][j0 + q] : g.tau[(long long)item * g.n + j0 + q];
    };
    if (rd) {
      // the next tile's old values towards L2: 32 columns x 512 bytes, shared with the warp of the other part
      TileWalk wn = w;
      wn.step();
      if (wn.valid()) {
        const int in = wn.item(), rn = (quarter & 1) * 32 + 8 * (lane & 3);
        const MatRef &M = rd_c ? g.C : g.D;
        const zd *p = mat_ptr(M, in / g.nc, in % g.nc) + rn;
        const zd *pe2 = mat_ptr(g.E, in / g.nc, in % g.nc) + rn;
#pragma unroll
        for (int q = 0; q < 16; q += 8) {
          const int j = j0 + 16 * part + q + (lane >> 2);
          if (rn < g.n && j < g.n) {
            prefetch_l2(p + (long long)j * M.ld);
            if (mode == 2) prefetch_l2(pe2 + (long long)j * g.E.ld);
          }
        }
      }
    }
    long long acc[NA];
    double old[NO];
    auto load_old = [&](const double *p, long long ld, int q0) {  // columns q0 .. q0 + NO - 1
#pragma unroll
      for (int q = 0; q < NO; q++)
        if (q0 + q < nq) old[q] = p[(q0 + q) * ld];
    };
    auto emit = [&](int q0) {  // columns q0 .. q0 + NO - 1 into C (mode 2: into D)
#pragma unroll
      for (int q = 0; q < NO; q++)
        if (q0 + q < nq) {
          const int tj = ce(q0 + q);
          double val = level_value<S, DB>(acc[(q0 + q) % NA], erow + tj);
          if (sig == SCALE_NONFINITE || tj == SCALE_NONFINITE) val = nan;
          const double unit = part == 0 && row == j0 + q0 + q ? 1.0 : 0.0;
          out[(q0 + q) * old_ld] = mode == 0 ? val : mode == 4 ? unit - val : mode == 5 ? old[q] + val : old[q] - val;
          acc[(q0 + q) % NA] = __double_as_longlong(val);  // for E
        }
    };
    auto emit_e = [&](int q0) {
#pragma unroll
      for (int q = 0; q < NO; q++)
        if (q0 + q < nq) pe[(q0 + q) * eld] = old[q] - __longlong_as_double(acc[(q0 + q) % NA]);
    };
    if (!EARLY && rd) load_old(src, sld, 0);
    if (!oz_warp_wait(sh, &sh.acc_full[buf], (w.i / NBUF) & 1)) break;
    tc_fence_after();
    const uint32_t ta = tbase + ((uint32_t)(quarter * 32) << 16) + buf * 256 + half * 32;
#pragma unroll
    for (int c0 = 0; c0 < 32; c0 += CH) {
      uint32_t v[S][CH];
#pragma unroll
      for (int l = 0; l < S; l++) {
        if constexpr (CH == 8) tmem_ld8(ta + l * NT + c0, v[l]);
        else tmem_ld4(ta + l * NT + c0, v[l]);
      }
      tmem_ld_wait();
#pragma unroll
      for (int t = 0; t < CH; t++) acc[(c0 + t) % NA] = levels_sum<S, DB, CH>(v, t);
      if constexpr (!EARLY) {
        emit(c0);
        if (mode == 2) {
          load_old(pe, eld, c0);
          emit_e(c0);
        }
        if (rd && c0 + CH < 32) load_old(src, sld, c0 + CH);
        __syncwarp();
      }
    }
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(&sh.acc_empty[buf]);
    if constexpr (EARLY) {
#pragma unroll
      for (int q0 = 0; q0 < 32; q0 += NO) {
        if (rd) load_old(src, sld, q0);
        emit(q0);
      }
      if (mode == 2) {
#pragma unroll
        for (int q0 = 0; q0 < 32; q0 += NO) {
          load_old(pe, eld, q0);
          emit_e(q0);
        }
      }
    }
  }
}

// Sliced product, persistent: one CTA per SM walks its output tiles (128 rows
// x 32 complex columns) with the roles below running side by side, so that
// the loads, the conversion of B and the rounding of one tile hide behind
// another tile's MMAs.  (Before, one CTA of 128 x 48 per tile did these in
// turn: of the 16.7 us a six-slice tile of it took, 4.4 were launch, TMEM
// allocation and pipeline fill, 5 the epilogue, 5.2 the MMAs.)
// What bounds it, 590 products of n = 128 from cold operands, before -> now:
// staged B, six slices 293 -> 187 us (MMAs 12.5 of a tile's 21 thousand
// cycles, the hand-over of the accumulators 4, operand loads 4; DRAM floor
// 125 us); staged three slices 184 -> 112 us (epilogue: 64-bit integer
// arithmetic at half the FP32 rate); fused B, seven slices 391 -> 258 us,
// three slices 280 -> 164 us (conversion, likewise integer arithmetic);
// R = I - AX and X += XR of the Newton step 422 + 316 -> 258 + 187 us.
// The 64-bit sums that the epilogue holds from five slices on spill 80 to 170
// bytes a thread at 128 registers (H = 0).  More epilogue or conversion warps
// do not pay where they cost registers: 20 warps with 96 spill more (six
// slices 187 -> 244 us); neither does redistributing registers with setmaxnreg (291 us).
// Every level p + q has its own accumulator (64 TMEM columns each), so that
// every level sum stays an exact integer while its bound allows (levels 0..3
// always), and the slices of B lie side by side in a stage: A_p against up
// to four of them is ONE instruction of N = 64..256 whose columns land in the
// consecutive accumulators p + q.  A slice of A is then read once per 256
// columns instead of once per pair.
// FB = 0: B tiles by TMA from the staged B'; FB = 1: B fused, its tiles
// formed by the conversion role from the FP64 B, which tmB then maps (g.B is
// the same operand).
// H = 1 (up to 64 rows): the tile is the whole product, with the real and the
// imaginary parts of A stacked, [Re A, -Im A; Im A, Re A] (64 + 64 rows)
// times [Re B; Im B] (one row of B'^T, one accumulator column per complex
// column).  The other form would fill half the rows of every tile and form
// every digit of B four times instead of twice; the integers summed are the
// same, so are the results bit for bit.  1640 products of n = 54: staged B, six
// slices 276 -> 156 us; fused B, seven slices 418 -> 209, three 311 -> 183.
template <int S, int DB, int FB, int H>
__global__ void __launch_bounds__(oz_threads(S), 1) k_ozaki(const __grid_constant__ CUtensorMap tmA,
                                                         const __grid_constant__ CUtensorMap tmB,
                                                         const __grid_constant__ OzArgs g) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  constexpr int NA = oz_a_stages(S, FB > 0), NB = oz_b_stages(S, FB > 0), NBUF = oz_bufs(S);
  constexpr int NRAW = FB > 0 ? oz_raw_stages(S) : 1;
  static_assert(NA >= 2 && NB >= 2 && (FB == 0 || NRAW >= 2), "the rings must fit the shared memory");
  unsigned char *sA = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char *sB = sA + NA * S * OZ_A_SLICE, *raw = sB + NB * S * OZ_B_SLICE;  // (all 1024-byte aligned)
  __shared__ OzShared sh;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (warp == 0) {
    tmem_alloc(&sh.tmem_base, 512);
    tmem_relinquish();
  }
  if (threadIdx.x == 32) {
    sh.failed = 0;
    sh.a_issued = 0;
    sh.raw_issued = 0;
    for (int i = 0; i < 6; i++) {
      mbar_init(&sh.a_full[i], 1);
      mbar_init(&sh.a_empty[i], 1);
      mbar_init(&sh.b_full[i], FB ? 4 : 1);  // fused B: the four warps of a group
      mbar_init(&sh.b_empty[i], 1);
    }
    for (int i = 0; i < 8; i++) {
      mbar_init(&sh.raw_full[i], 1);
      mbar_init(&sh.raw_empty[i], 4);
    }
    for (int i = 0; i < OZ_SCALE_RING; i++) {
      mbar_init(&sh.sc_full[i], 4);
      mbar_init(&sh.sc_empty[i], 4 * oz_conv_groups(S));
    }
    for (int i = 0; i < NBUF; i++) {
      mbar_init(&sh.acc_full[i], 1);
      mbar_init(&sh.acc_empty[i], OZ_EPI_WARPS);
    }
    mbar_init(&sh.done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = sh.tmem_base;
  const int nkb = g.kblocks;

  if (warp == 0) {
    // TMA producer (with staged B both operands, in rings of equal length)
    if (lane == 0) {
      int kc = 0;
      for (TileWalk w(g); w.valid() && !sh.failed; w.step()) {
        const int item = w.item(), mt = w.mt(), nt = w.nt();
        for (int kb = 0; kb < nkb; kb++, kc++) {
          const int st = kc % NA;
          if (sh.failed || (kc >= NA && !mbar_wait(&sh.a_empty[st], ((kc / NA) - 1) & 1))) {
            sh.failed = 1;
            break;
          }
          mbar_expect_tx(&sh.a_full[st], S * OZ_A_SLICE);
          if (FB == 0) mbar_expect_tx(&sh.b_full[st], S * OZ_B_SLICE);
#pragma unroll
          for (int sl = 0; sl < S; sl++) {
            const int z = (item * S + sl) * nkb + kb;
            tma_load_3d(sA + (st * S + sl) * OZ_A_SLICE, &tmA, 0, mt * MT, z, &sh.a_full[st]);
            if (FB == 0) tma_load_3d(sB + (st * S + sl) * OZ_B_SLICE, &tmB, 0, nt * NT, z, &sh.b_full[st]);
          }
          sh.a_issued = kc + 1;
        }
      }
    }
  } else if (warp == 1) {
    // MMA issuer
    if (lane == 0) {
      int kc = 0;
      for (TileWalk w(g); w.valid() && !sh.failed; w.step()) {
        const int buf = w.i % NBUF;
        if (w.i >= NBUF && !mbar_wait(&sh.acc_empty[buf], ((w.i / NBUF) - 1) & 1)) {
          sh.failed = 1;
          break;
        }
        const uint32_t td = tbase + buf * 256;
        for (int kb = 0; kb < nkb; kb++, kc++) {
          const int sa = kc % NA, sb = kc % NB;
          if (sh.failed || !mbar_wait(&sh.a_full[sa], (kc / NA) & 1) || !mbar_wait(&sh.b_full[sb], (kc / NB) & 1)) {
            sh.failed = 1;
            break;
          }
          tc_fence_after();
          const uint32_t a0 = smem_u32(sA) + sa * (S * OZ_A_SLICE), b0 = smem_u32(sB) + sb * (S * OZ_B_SLICE);
#pragma unroll
          for (int k = 0; k < KB / 16; k++)
#pragma unroll
            for (int p = 0; p < S; p++)
#pragma unroll
              for (int q = 0; q < S - p; q += 4) {  // p + q <= S - 1; up to four slices of B at once
                const int nb = S - p - q < 4 ? S - p - q : 4;
                umma_bf16(td + (p + q) * NT, sdesc_sw64(a0 + p * OZ_A_SLICE + 32 * k),
                          sdesc_sw64(b0 + q * OZ_B_SLICE + 32 * k), idesc_bf16(MT, NT * nb),
                          (kb == 0 && k == 0 && p == 0) ? 0u : 1u);
              }
          umma_commit(&sh.a_empty[sa]);  // the stages are free once these MMAs have read them
          umma_commit(&sh.b_empty[sb]);
        }
        umma_commit(&sh.acc_full[buf]);  // accumulators complete
      }
      umma_commit(&sh.done);
    }
  } else if (warp == 2) {
    if constexpr (FB > 0) oz_scales<H>(g, sh);
  } else if (warp == 3) {
    // fused B: the FP64 k-blocks of B into their ring
    if (FB > 0 && lane == 0) {
      const int npass = oz_raw_passes<H>(g);
      int rc = 0;
      for (TileWalk w(g); w.valid() && !sh.failed; w.step()) {
        const int kk = w.item() / g.nc, cc = w.item() % g.nc, j0 = w.nt() * (NT / 2);
        const int mc = map_at(g.B, cc);
        for (int kp = 0; kp < nkb * npass; kp++, rc++) {
          const int r = rc % NRAW, kb = kp / npass, jp = j0 + (kp % npass) * 32;
          if (sh.failed || (rc >= NRAW && !mbar_wait(&sh.raw_empty[r], ((rc / NRAW) - 1) & 1))) {
            sh.failed = 1;
            break;
          }
          mbar_expect_tx(&sh.raw_full[r], OZ_RAW_BYTES);
          unsigned char *dst = raw + r * OZ_RAW_BYTES;
          tma_load_4d(dst, &tmB, 32 * kb, jp, mc, kk, &sh.raw_full[r]);
          tma_load_4d(dst + OZ_RAW_BYTES / 2, &tmB, 32 * kb + 16, jp, mc, kk, &sh.raw_full[r]);
          sh.raw_issued = rc + 1;
        }
      }
    }
  } else if (warp < OZ_CONV0) {
    if constexpr (H) oz_epilogue_h<S, DB, FB>(g, sh, tbase);
    else oz_epilogue<S, DB, FB>(g, sh, tbase);
  } else if constexpr (FB > 0) {
    oz_convert<S, DB, NB, NRAW, H>(g, sh, sB, raw);
  }
  __syncthreads();
  // every MMA issued is complete (bounded wait) before the accumulators go
  if (!mbar_wait(&sh.done, 0)) sh.failed = 1;
  __syncthreads();
  if (sh.failed && threadIdx.x == 0) {
    atomicOr(g.err, 1);
    // copies asked for but perhaps not consumed: let them land (bounded) before exit
    for (int kc = sh.a_issued > NA ? sh.a_issued - NA : 0; kc < sh.a_issued; kc++) {
      mbar_wait(&sh.a_full[kc % NA], (kc / NA) & 1);
      if (FB == 0) mbar_wait(&sh.b_full[kc % NB], (kc / NB) & 1);
    }
    for (int rc = sh.raw_issued > NRAW ? sh.raw_issued - NRAW : 0; rc < sh.raw_issued; rc++)
      mbar_wait(&sh.raw_full[rc % NRAW], (rc / NRAW) & 1);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tbase, 512);
}

// ------------------------------------------------------------------ FP32 GJ
// Gauss-Jordan with column pivoting (main/gjinv.f: in row i the pivot is the
// largest |a(i, j)| over the columns not yet used, first index on ties) in
// complex FP32, in panels of eight rows.  The pivot columns are not swapped
// into place: step i eliminates with the pivot (i, kp) where it lies and
// records sigma(i) = kp, which is Gauss-Jordan on A P (P the column
// permutation); the array then holds (A P)^-1 with its columns stored at the
// positions of A P's, so A^-1(sigma(r), c) is found at (r, sigma(c)) and the
// store permutes both indices.  The result (written as FP64) only seeds the
// Newton refinement.
//
// The last N / 32 warps factor the panel: a lane holds one column of the eight
// rows in registers, and eight Gauss-Jordan steps run on those rows alone.
// With the panel P (eight rows of the inverse tableau) and its pivot columns
// K, every other row takes one update of depth eight,
//   a(r, :) <- (a(r, :) with the columns K zeroed) - sum_q a(r, K_q) P(q, :),
// and the panel's own rows become P.  The other
// W warps do that on the matrix in shared memory (column-major): a warp takes
// four columns at a time, a lane the rows lane + 32 a, with the lane's
// multipliers in registers and P broadcast.  Each warp forms its columns of
// the next panel's rows first and hands them over, so that the next panel is
// factored while the update runs.
//
// Why panels: a rank-1 update per pivot needs a block barrier, the pivot
// search and the multipliers' selects every step, 1750 clocks of which 128
// were multiply-adds (n = 64); in panels a step takes one barrier of N / 32
// warps and a chain of about 300 clocks, beside the update.  Why shared
// memory: the columns K and the rows of a panel lie at run-time indices, which
// registers answer with selects over the whole tile (45 us for 42 items of
// n = 64).  Before and after: 57 and 30 us (42 items of n = 64), 99 and 57
// (420), 277 and 149 (1640 of n = 54).  At n = 128 the whole matrix takes
// 104 us (42 items, one wave) and 305 us (420), where the 2 x 2 block form on
// 64-row inverses took 214 and 468 (and would take 160 and 384 on this one).
// The FP32 multiply-adds alone are 32 us a wave at n = 128; loading and
// storing with conversions (two a clock per SM) 16, the panel chain and the
// barriers the rest.

__device__ __forceinline__ unsigned long long pk2(float x, float y) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 upk2(unsigned long long r) {
  float2 v;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(r));
  return v;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b,
                                                   unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
constexpr int GJ_NB = 8;                                         // rows of a panel
constexpr int GJ_BAR_PANEL = 1, GJ_BAR_RAW = 2, GJ_BAR_MUL = 3, GJ_BAR_STEP = 4;  // named barriers

template <int ID>
__device__ __forceinline__ void bar_sync_n(int threads) {
  asm volatile("bar.sync %0, %1;" ::"n"(ID), "r"(threads) : "memory");
}
template <int ID>
__device__ __forceinline__ void bar_arrive_n(int threads) {
  asm volatile("bar.arrive %0, %1;" ::"n"(ID), "r"(threads) : "memory");
}

// N: rows and columns, padded to 32.  The leading dimension N + 8 puts the
// eight rows of a panel in four neighbouring columns on different banks.
template <int N>
struct GjShared {
  unsigned long long m[N][N + 8];  // [column][row], (re, im) pairs
  alignas(16) unsigned long long p[2][N][GJ_NB + 2];  // the panel, handed over and back: [column][row] (80 bytes a column: no
                                          // bank conflicts between eight columns)
  ulonglong2 pcol[2][N / 32][GJ_NB / 2 + 1];  // proposed pivot columns of a step, 1/pivot
  unsigned pkey[2][N / 32];        // and their keys
  alignas(16) int slot[2][N];      // q of a panel's pivot column, else -1
  int kcol[2][GJ_NB];              // pivot columns of a panel
  int sig[N], sinv[N];
};

// Eight Gauss-Jordan steps on the panel of rows i0 .. i0 + 7, column j in this
// thread.  Each warp proposes the best pivot of its 32 columns together with
// its column and reciprocal, so that a step takes one barrier of the panel
// warps.  used: this column has been a pivot (or is >= n).  Rows >= n are unit
// rows and pivot on themselves.
template <int N>
__device__ __forceinline__ void gj_panel(GjShared<N> &sh, int buf, int i0, int n, int j, bool &used) {
  constexpr int PW = N / 32;
  const int pw = j >> 5, lane = j & 31;
  unsigned long long v[GJ_NB];
#pragma unroll
  for (int q = 0; q < GJ_NB; q++) v[q] = sh.p[buf][j][q];
  int mine = -1;
#pragma unroll
  for (int q = 0; q < GJ_NB; q++) {
    const int i = i0 + q;
    // largest |a(i, j)|^2 over the unused columns: its bits order as integers;
    // the last seven carry the column (first index on ties, that is within
    // 2^-16), so that one reduction gives both.  NaN comes last.
    const float2 w = upk2(v[q]);
    const float mm = w.x * w.x + w.y * w.y;
    const unsigned inv = 127u - (unsigned)j;
    unsigned key = mm >= 0.f ? ((__float_as_uint(mm) | 0x80000000u) & ~127u) | inv : 128u | inv;
    key = used ? 0u : key;
    key = i < n ? key : j == i ? 0xFFFFFF80u | inv : 0u;
    const float rden = __frcp_rn(mm);
    unsigned kmax = __reduce_max_sync(0xFFFFFFFFu, key);
    ulonglong2(&pc)[PW][GJ_NB / 2 + 1] = sh.pcol[q & 1];
    if (key == kmax && key != 0u) {
#pragma unroll
      for (int r = 0; r < GJ_NB; r += 2) pc[pw][r / 2] = make_ulonglong2(v[r], v[r + 1]);
      pc[pw][GJ_NB / 2].x = pk2(w.x * rden, -w.y * rden);
    }
    int win = 0;
    if (PW > 1) {
      if (lane == 0) sh.pkey[q & 1][pw] = kmax;
      bar_sync_n<GJ_BAR_STEP>(PW * 32);
      kmax = sh.pkey[q & 1][0];
#pragma unroll
      for (int o = 1; o < PW; o++) {
        const unsigned k = sh.pkey[q & 1][o];
        win = k > kmax ? o : win;
        kmax = k > kmax ? k : kmax;
      }
    } else {
      __syncwarp();
    }
    const int kp = 127 - (int)(kmax & 127u);
    const float2 d = upk2(pc[win][GJ_NB / 2].x);
    float2 c[GJ_NB];
#pragma unroll
    for (int r = 0; r < GJ_NB; r += 2) {
      const ulonglong2 t = pc[win][r / 2];
      c[r] = upk2(t.x);
      c[r + 1] = upk2(t.y);
    }
    const bool hit = j == kp;
    if (hit) {
      used = true;
      mine = q;
      sh.sig[i] = kp;
      sh.sinv[kp] = i;
      sh.kcol[buf][q] = kp;
    }
    // the pivot row times 1/pivot, then the other rows minus a(r, kp) times
    // it; the pivot column starts from the unit column
    const float2 x = hit ? make_float2(1.f, 0.f) : w;
    const float2 o = make_float2(x.x * d.x - x.y * d.y, x.x * d.y + x.y * d.x);
    v[q] = pk2(o.x, o.y);
    const unsigned long long ps = pk2(o.y, -o.x);
#pragma unroll
    for (int rr = 1; rr < GJ_NB; rr++) {
      const int r = (q + rr) % GJ_NB;  // the next pivot row first
      v[r] = fma2(pk2(c[r].y, c[r].y), ps, fma2(pk2(-c[r].x, -c[r].x), v[q], hit ? 0ull : v[r]));
    }
  }
#pragma unroll
  for (int q = 0; q < GJ_NB; q += 2) *reinterpret_cast<ulonglong2 *>(&sh.p[buf][j][q]) = make_ulonglong2(v[q], v[q + 1]);
  sh.slot[buf][j] = mine;
}

// u -= c p
__device__ __forceinline__ void gj_fms(float2 &u, float2 c, float2 p) {
  u.x = fmaf(-c.x, p.x, u.x);
  u.y = fmaf(-c.x, p.y, u.y);
  u.x = fmaf(c.y, p.y, u.x);
  u.y = fmaf(-c.y, p.x, u.y);
}

static_assert(offsetof(GjShared<32>, slot) % 16 == 0 && offsetof(GjShared<64>, slot) % 16 == 0 &&
                  offsetof(GjShared<96>, slot) % 16 == 0 && offsetof(GjShared<128>, slot) % 16 == 0 &&
                  offsetof(GjShared<96>, p) % 16 == 0 && offsetof(GjShared<96>, pcol) % 16 == 0,
              "16-byte shared loads");

// RA rows a lane (N = 32 RA), W update warps, MINB blocks per SM
template <int RA, int W, int MINB>
__global__ void __launch_bounds__((W + RA) * 32, MINB) k_cgj32(const __grid_constant__ MatRef A,
                                                            const __grid_constant__ MatRef X, int n, int nc,
                                                            const int *__restrict__ act) {
  constexpr int N = 32 * RA, T = W * 32, TALL = T + N;
  const int item = blockIdx.x, kk = item / nc, cc = item % nc;
  if (act && !act[item]) return;
  extern __shared__ __align__(16) char gj_smem[];
  GjShared<N> &sh = *reinterpret_cast<GjShared<N> *>(gj_smem);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, np = (n + GJ_NB - 1) / GJ_NB, ncols = np * GJ_NB;
  if (w >= W) {  // the panel warps
    const int j = threadIdx.x - T;
    bool used = j >= n;
    for (int p = 0; p < np; p++) {
      bar_sync_n<GJ_BAR_RAW>(TALL);  // the rows of panel p are in p[p & 1]
      gj_panel<N>(sh, p & 1, p * GJ_NB, n, j, used);
      bar_arrive_n<GJ_BAR_PANEL>(TALL);
    }
    return;
  }
  {
    const zd *a = mat_ptr(A, kk, cc);
    constexpr int LB = RA >= 3 ? 2 : 4;  // columns in flight
    for (int j0 = w; j0 < N; j0 += LB * W) {
      zd z[LB][RA];
#pragma unroll
      for (int e = 0; e < LB; e++)
#pragma unroll
        for (int ia = 0; ia < RA; ia++) {
          const int r = lane + 32 * ia, j = j0 + e * W;
          z[e][ia] = r < n && j < n ? a[r + (long long)j * A.ld] : make_double2(r == j ? 1.0 : 0.0, 0.0);
        }
#pragma unroll
      for (int e = 0; e < LB; e++) {
        const int j = j0 + e * W;
        if (j >= N) break;
#pragma unroll
        for (int ia = 0; ia < RA; ia++) {
          const unsigned long long v = pk2((float)z[e][ia].x, (float)z[e][ia].y);
          sh.m[j][lane + 32 * ia] = v;
          if (ia == 0 && lane < GJ_NB) {
            sh.p[0][j][lane] = v;
            sh.p[1][j][lane] = 0ull;  // (columns past ncols stay so)
          }
        }
      }
    }
  }
  bar_arrive_n<GJ_BAR_RAW>(TALL);
  for (int p = 0; p < np; p++) {
    const int i0 = p * GJ_NB, buf = p & 1;
    bar_sync_n<GJ_BAR_PANEL>(TALL);  // panel p factored, every earlier update finished
    int kc[GJ_NB];
#pragma unroll
    for (int q = 0; q < GJ_NB; q++) kc[q] = sh.kcol[buf][q];
    if (p + 1 < np) {  // the next panel's rows: eight rows, four columns a warp
      const int rn = lane & 7, r1 = i0 + GJ_NB + rn;
      float2 cn[GJ_NB];
#pragma unroll
      for (int q = 0; q < GJ_NB; q++) cn[q] = upk2(sh.m[kc[q]][r1]);
      for (int j = 4 * w + (lane >> 3); j < ncols; j += 4 * W) {
        float2 u = upk2(sh.slot[buf][j] < 0 ? sh.m[j][r1] : 0ull);
#pragma unroll
        for (int q = 0; q < GJ_NB; q += 2) {
          const ulonglong2 t = *reinterpret_cast<const ulonglong2 *>(&sh.p[buf][j][q]);
          gj_fms(u, cn[q], upk2(t.x));
          gj_fms(u, cn[q + 1], upk2(t.y));
        }
        sh.p[buf ^ 1][j][rn] = pk2(u.x, u.y);
      }
      bar_arrive_n<GJ_BAR_RAW>(TALL);
    }
    float2 c[GJ_NB][RA];  // (of the panel's own rows too: they are overwritten below)
#pragma unroll
    for (int q = 0; q < GJ_NB; q++)
#pragma unroll
      for (int ia = 0; ia < RA; ia++) c[q][ia] = upk2(sh.m[kc[q]][lane + 32 * ia]);
    bar_sync_n<GJ_BAR_MUL>(T);  // multipliers and next rows read: the matrix may change
    for (int j0 = 4 * w; j0 < ncols; j0 += 4 * W) {
      const int4 sl = *reinterpret_cast<const int4 *>(&sh.slot[buf][j0]);
      const int sle[4] = {sl.x, sl.y, sl.z, sl.w};
      if ((sl.x & sl.y & sl.z & sl.w) >= 0) {  // a column of K among them
#pragma unroll
        for (int e = 0; e < 4; e++)
          if (sle[e] >= 0)
#pragma unroll
            for (int ia = 0; ia < RA; ia++) sh.m[j0 + e][lane + 32 * ia] = 0ull;
      }
      float2 u[4][RA];
#pragma unroll
      for (int e = 0; e < 4; e++)
#pragma unroll
        for (int ia = 0; ia < RA; ia++) u[e][ia] = upk2(sh.m[j0 + e][lane + 32 * ia]);
#pragma unroll
      for (int q = 0; q < GJ_NB; q += 2)
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const ulonglong2 t = *reinterpret_cast<const ulonglong2 *>(&sh.p[buf][j0 + e][q]);
#pragma unroll
          for (int ia = 0; ia < RA; ia++) gj_fms(u[e][ia], c[q][ia], upk2(t.x));
#pragma unroll
          for (int ia = 0; ia < RA; ia++) gj_fms(u[e][ia], c[q + 1][ia], upk2(t.y));
        }
#pragma unroll
      for (int e = 0; e < 4; e++)
#pragma unroll
        for (int ia = 0; ia < RA; ia++) sh.m[j0 + e][lane + 32 * ia] = pk2(u[e][ia].x, u[e][ia].y);
      __syncwarp();
      sh.m[j0 + (lane >> 3)][i0 + (lane & 7)] = sh.p[buf][j0 + (lane >> 3)][lane & 7];  // the panel's rows
    }
  }
  bar_sync_n<GJ_BAR_MUL>(T);
  // place (r, j) holds A^-1(sigma(r), sigma^-1(j))
  zd *x = mat_ptr(X, kk, cc);
#pragma unroll 4
  for (int j = w; j < n; j += W) {
    const unsigned long long *col = sh.m[sh.sig[j]];
#pragma unroll
    for (int ia = 0; ia < RA; ia++) {
      const int r = lane + 32 * ia;
      if (r < n) {
        const float2 v = upk2(col[sh.sinv[r]]);
        x[r + (long long)j * X.ld] = make_double2((double)v.x, (double)v.y);
      }
    }
  }
}

// ------------------------------------------------------------------ host side

// resolved once per process (thread-safe static initialisation: contexts may
// run from several host threads)
static PFN_cuTensorMapEncodeTiled_v12000 encoder() {
  static const PFN_cuTensorMapEncodeTiled_v12000 fn = []() -> PFN_cuTensorMapEncodeTiled_v12000 {
    cudaDriverEntryPointQueryResult q;
    void *p = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) !=
            cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return nullptr;
    return (PFN_cuTensorMapEncodeTiled_v12000)p;
  }();
  return fn;
}
int get_encoder() { return encoder() ? 0 : -1; }

// tiled staging: dims {32, rows, regions * kblocks}; one box = one contiguous block
int make_map(CUtensorMap *m, void *base, int rows, long long depth, int boxrows) {
  cuuint64_t dims[3] = {(cuuint64_t)KB, (cuuint64_t)rows, (cuuint64_t)depth};
  cuuint64_t strides[2] = {(cuuint64_t)KB * 2, (cuuint64_t)KB * 2 * rows};
  cuuint32_t box[3] = {(cuuint32_t)KB, (cuuint32_t)boxrows, 1};
  cuuint32_t es[3] = {1, 1, 1};
  CUresult r = encoder()(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, base, dims, strides, box, es,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -1;
}

// the FP64 operand B (K rows, n columns, nk x nc items): dims {2 K doubles,
// columns, class blocks, k points}; one box = eight complex values of 32
// columns.  False where a stride cannot be mapped (the caller stages B then).
bool make_raw_map(CUtensorMap *m, const MatRef &B, int n, int K, int nk, int nc) {
  int cmax = 0;
  for (int c = 0; c < nc; c++) {
    if (B.map[c] < 0) return false;
    cmax = std::max(cmax, B.map[c]);
  }
  const long long sc = cmax > 0 ? B.sc : (long long)n * B.ld, sk = nk > 1 ? B.sk : sc * (cmax + 1);
  const long long top = 1LL << 35;
  if (B.ld < K || sc <= 0 || sk <= 0 || sc >= top || sk >= top) return false;
  cuuint64_t dims[4] = {(cuuint64_t)2 * K, (cuuint64_t)n, (cuuint64_t)cmax + 1, (cuuint64_t)nk};
  cuuint64_t strides[3] = {(cuuint64_t)B.ld * sizeof(zd), (cuuint64_t)sc * sizeof(zd), (cuuint64_t)sk * sizeof(zd)};
  cuuint32_t box[4] = {16, NT / 2, 1, 1}, es[4] = {1, 1, 1, 1};
  return encoder()(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, B.base, dims, strides, box, es,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// above half of an SM's shared memory for every S, so that no second CTA
// (whose 512-column TMEM allocation would wait) becomes resident
size_t oz_smem_bytes(int S, bool fused) {
  return (size_t)oz_ring_bytes(S, fused) + (fused ? (size_t)oz_raw_stages(S) * OZ_RAW_BYTES : 0) + 1024;
}

}  // namespace

// ---------------------------------------------------------------------------
// Split operands live in staging slots (MIXED_SLOTS per side) so that an
// operand used by several products is split once.  A slot records the layout
// its zero padding was made for and the slices / digit base of its contents.
struct Stage {
  void *p = nullptr;       // [item][S][kblocks][rows][32] bf16 slices
  size_t cap = 0;
  int *scale = nullptr;    // row (A) / column (B) scale exponents
  size_t scap = 0;
  int n = -1, K = -1;      // padding layout of p
  int S = 0, DB = 0;       // the operand held: slices, digit base, dims, items
  int cn = -1, cK = -1;
  long long items = 0;
  bool fused = false;      // B only: not split; each product forms its tiles from src
  MatRef src;
};

constexpr int OZ_FORMS = 6 * 2 * 3;  // k_ozaki's instances: slices, staged or fused B, digit base or stacked

struct MixedWork {
  Stage A[MIXED_SLOTS], B[MIXED_SLOTS];
  zd *acopy = nullptr, *rbuf = nullptr, *big = nullptr;
  size_t ac_cap = 0, rb_cap = 0, big_cap = 0;
  double *rnorm = nullptr;
  size_t rn_cap = 0;
  int *err = nullptr;
  unsigned long long *dmax = nullptr;  // running max of accepted Newton residual norms (double bits)
  unsigned long long *nfb = nullptr;   // inverses redone in FP64 (residual above the limit)
  int *flag = nullptr;                 // per-item FP64 fallback mask
  size_t flag_cap = 0;
  int *mark = nullptr;                 // per-item mask of the further Newton steps
  size_t mark_cap = 0;
  int *cnt = nullptr;                  // count of marked items (device scalar)
  unsigned long long *nref = nullptr;  // [0] inverses that took further Newton steps, [1] kernels run by the
                                       // IF bodies of captured further steps (device counts)
  cudaStream_t side = nullptr;         // captures the bodies of conditional graph nodes
  // of the device this context lives on: its SMs, and which forms of k_ozaki
  // have had their shared memory limit raised (a kernel's attributes belong to
  // the device that is current when they are set, and end with its context)
  int sms = 0;
  bool smem_set[OZ_FORMS] = {};
  bool fuse_b = true;      // B operands formed inside the product (mixed_set_fused)
};

void mixed_set_fused(MixedWork *w, bool on) { w->fuse_b = on; }

// the callers' streams are non-blocking: free the old buffer only once the
// device is idle (cudaFree does not wait for those streams)
static int grow(void **p, size_t *cap, size_t bytes, bool zero) {
  if (bytes <= *cap) return 0;
  std::lock_guard<std::recursive_mutex> lk(skkr_device_mutex());
  if (*p) {
    cudaDeviceSynchronize();
    cudaFree(*p);
  }
  *p = nullptr;
  *cap = 0;
  if (cudaMalloc(p, bytes) != cudaSuccess) return SKKR_ERR_NOMEM;
  // cudaMemset runs on the legacy default stream, which the non-blocking
  // streams do not wait for: finish it before the buffer is used
  if (zero && (cudaMemset(*p, 0, bytes) != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess))
    return SKKR_ERR_NOMEM;
  *cap = bytes;
  return 0;
}

MixedWork *mixed_create() {
  std::lock_guard<std::recursive_mutex> lk(skkr_device_mutex());
  MixedWork *w = new MixedWork();
  int dev = 0;
  if (cudaMalloc(&w->err, sizeof(int)) != cudaSuccess ||
      cudaMalloc(&w->dmax, sizeof(unsigned long long)) != cudaSuccess ||
      cudaMalloc(&w->nfb, sizeof(unsigned long long)) != cudaSuccess ||
      cudaMalloc(&w->cnt, sizeof(int)) != cudaSuccess ||
      cudaMalloc(&w->nref, 2 * sizeof(unsigned long long)) != cudaSuccess ||
      cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&w->sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || w->sms < 1 ||
      cudaStreamCreateWithFlags(&w->side, cudaStreamNonBlocking) != cudaSuccess) {
    void *ps[] = {w->err, w->dmax, w->nfb, w->cnt, w->nref};
    for (void *p : ps)
      if (p) cudaFree(p);
    delete w;
    return nullptr;
  }
  cudaMemset(w->err, 0, sizeof(int));
  cudaMemset(w->dmax, 0, sizeof(unsigned long long));
  cudaMemset(w->nfb, 0, sizeof(unsigned long long));
  cudaMemset(w->nref, 0, 2 * sizeof(unsigned long long));
  cudaDeviceSynchronize();  // default-stream memsets, before the non-blocking streams use the flags
  return w;
}

int mixed_resid_reset(MixedWork *w, cudaStream_t st) {
  return (cudaMemsetAsync(w->err, 0, sizeof(int), st) == cudaSuccess &&
          cudaMemsetAsync(w->dmax, 0, sizeof(unsigned long long), st) == cudaSuccess &&
          cudaMemsetAsync(w->nfb, 0, sizeof(unsigned long long), st) == cudaSuccess &&
          cudaMemsetAsync(w->nref, 0, 2 * sizeof(unsigned long long), st) == cudaSuccess)
             ? 0
             : SKKR_ERR_CUDA;
}

int mixed_resid_read(MixedWork *w, double *out, long long *fallbacks, long long *refined, cudaStream_t st) {
  unsigned long long h[3] = {0, 0, 0};
  if (cudaMemcpyAsync(&h[0], w->dmax, sizeof(h[0]), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaMemcpyAsync(&h[1], w->nfb, sizeof(h[1]), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaMemcpyAsync(&h[2], w->nref, sizeof(h[2]), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return SKKR_ERR_CUDA;
  double v;
  memcpy(&v, &h[0], sizeof(v));
  *out = v;
  if (fallbacks) *fallbacks = (long long)h[1];
  if (refined) *refined = (long long)h[2];
  return 0;
}

int *mixed_error_ptr(MixedWork *w) { return w->err; }

long long mixed_graph_kernels(MixedWork *w, cudaStream_t st) {
  unsigned long long h = 0;
  if (cudaMemcpyAsync(&h, w->nref + 1, sizeof(h), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return 0;
  return (long long)h;
}

void mixed_destroy(MixedWork *w) {
  if (!w) return;
  std::lock_guard<std::recursive_mutex> lk(skkr_device_mutex());
  cudaDeviceSynchronize();
  for (int i = 0; i < MIXED_SLOTS; i++) {
    void *q[] = {w->A[i].p, w->A[i].scale, w->B[i].p, w->B[i].scale};
    for (void *p : q)
      if (p) cudaFree(p);
  }
  void *ps[] = {w->acopy, w->rbuf, w->big, w->rnorm, w->err, w->dmax, w->nfb, w->flag, w->mark, w->cnt, w->nref};
  for (void *p : ps)
    if (p) cudaFree(p);
  if (w->side) cudaStreamDestroy(w->side);
  delete w;
}

int mixed_error_flag(MixedWork *w) {
  int h = 0;
  if (cudaMemcpy(&h, w->err, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
  return h;
}

// up to 64 rows the real and imaginary parts of A are stacked in one tile
// (k_ozaki's H; depths of the eight-bit digits)
static bool oz_stacked(int n, int K) { return n <= MT / 2 && K <= 128; }

// dims of the staged real problem for complex n x K times K x n
static void oz_dims(int n, int K, int *Mp, int *Np, int *Kp, int *mtiles, int *ntiles, int *kblocks) {
  *mtiles = (n + MT - 1) / MT;
  *Mp = *mtiles * MT;
  *ntiles = oz_stacked(n, K) ? 1 : (2 * n + NT - 1) / NT;
  *Np = *ntiles * NT;
  *kblocks = (2 * K + KB - 1) / KB;
  *Kp = *kblocks * KB;
}

// digit base for depth K: 8 bits while 2K <= 256, 7 bits above so that the
// FP32 level sums stay exact integers
static int oz_digits(int K) { return K <= 128 ? 8 : 7; }

// side 1 with fuse_b: the slot only records B (the product reads it when it
// runs: B must not change in between, which every caller keeps); `real`
// (an operand several products read) splits it all the same
template <int S, int DB, int H>
static int split_s(MixedWork *w, int side, int slot, const MatRef &M, int n, int K, int nk, int nc,
                   const int *act, cudaStream_t st, bool real = false) {
  int Mp, Np, Kp, mtiles, ntiles, kblocks;
  oz_dims(n, K, &Mp, &Np, &Kp, &mtiles, &ntiles, &kblocks);
  const long long items = (long long)nk * nc;
  Stage &sg = side == 0 ? w->A[slot] : w->B[slot];
  sg.S = S;
  sg.DB = DB;
  sg.cn = n;
  sg.cK = K;
  sg.items = items;
  sg.fused = side == 1 && !real && w->fuse_b;
  if (sg.fused) {
    sg.src = M;
    return 0;
  }
  const int rows = side == 0 ? Mp : Np;
  int rc;
  // a buffer cannot be reallocated inside a captured graph: the eager run
  // before any capture sizes every slot (mixed_zinv reserves its further steps')
  if ((size_t)items * S * rows * Kp * 2 > sg.cap && stream_capturing(st)) return SKKR_ERR_CUDA;
  if ((rc = grow(&sg.p, &sg.cap, (size_t)items * S * rows * Kp * 2, true))) return rc;
  if ((rc = grow((void **)&sg.scale, &sg.scap, (size_t)items * (side == 0 ? Mp : n) * sizeof(int), false)))
    return rc;
  if (sg.n != n || sg.K != K) {
    // padding (rows beyond the operand, K' places of complex indices >= K)
    // must be zero; a new layout clears what an earlier one wrote there
    if (cudaMemsetAsync(sg.p, 0, sg.cap, st) != cudaSuccess) return SKKR_ERR_CUDA;
    sg.n = n;
    sg.K = K;
  }
  const long long active_s = act ? skkr_active_items(items) : items;
  // split traffic: FP64 operand read + S bf16 slices of the real embedding written
  const double split_bytes = (double)active_s * n * K * (16.0 + S * 2.0 * 2.0);
  if (side == 0) {
    dim3 ga((n + 31) / 32, items);
    kstat_begin(KS_OTHER, split_bytes, st);
    k_split_a<S, DB, H><<<ga, 256, 0, st>>>(M, n, K, nc, act, (__nv_bfloat16 *)sg.p, Mp, Kp, sg.scale);
  } else {
    dim3 gb((n + 7) / 8, items);
    kstat_begin(KS_OTHER, 2.0 * split_bytes, st);
    k_split_b<S, DB, H><<<gb, 256, 0, st>>>(M, n, K, nc, act, (__nv_bfloat16 *)sg.p, Np, Kp, sg.scale);
  }
  kstat_end(st);
  SKKR_LAUNCHED();
  return 0;
}

template <int S, int DB, int FB, int H>
static int oz_launch(MixedWork *w, const CUtensorMap &ma, const CUtensorMap &mb, const OzArgs &g, cudaStream_t st) {
  const size_t smem = oz_smem_bytes(S, FB > 0);
  bool &set = w->smem_set[((S - 3) * 2 + (FB > 0)) * 3 + (H ? 2 : DB - 7)];
  if (!set &&
      cudaFuncSetAttribute(k_ozaki<S, DB, FB, H>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
          cudaSuccess)
    return SKKR_ERR_CUDA;
  set = true;
  k_ozaki<S, DB, FB, H><<<std::min(g.tiles, w->sms), oz_threads(S), smem, st>>>(ma, mb, g);
  return 0;
}

template <int S, int DB, int H>
static int gemm_s(MixedWork *w, int mode, int sa, int sb, const MatRef &C, const MatRef &D, const MatRef &E,
                  int n, int K, int nk, int nc, const int *act, cudaStream_t st) {
  if (get_encoder()) return SKKR_ERR_CUDA;
  int Mp, Np, Kp, mtiles, ntiles, kblocks;
  oz_dims(n, K, &Mp, &Np, &Kp, &mtiles, &ntiles, &kblocks);
  const long long items = (long long)nk * nc;
  const Stage &A = w->A[sa];
  Stage &B = w->B[sb];
  if (A.fused || A.S != S || B.S != S || A.DB != DB || B.DB != DB || A.cn != n || B.cn != n || A.cK != K ||
      B.cK != K || A.items != items || B.items != items)
    return SKKR_ERR_ARG;  // the slots do not hold splits of this product's operands
  CUtensorMap ma, mb;
  // a fused B that the product writes over (C, D or E) is split first, so
  // that no CTA reads an element another one has already replaced; so is one
  // whose strides no tensor map takes
  auto over = [&](const MatRef &out) { return mref_overlap(B.src, out, nk, nc, n, K, n); };
  if (B.fused && (over(C) || over(D) || over(E) || !make_raw_map(&mb, B.src, n, K, nk, nc))) {
    const int rc = split_s<S, DB, H>(w, 1, sb, B.src, n, K, nk, nc, act, st, true);
    if (rc) return rc;
  }
  if (make_map(&ma, A.p, Mp, items * S * kblocks, MT)) return SKKR_ERR_CUDA;
  if (!B.fused && make_map(&mb, B.p, Np, items * S * kblocks, NT)) return SKKR_ERR_CUDA;
  OzArgs g;
  g.n = n;
  g.mtiles = mtiles;
  g.ntiles = ntiles;
  g.kblocks = kblocks;
  g.nc = nc;
  g.mode = mode;
  g.sigma = A.scale;
  g.tau = B.scale;
  g.B = B.src;
  g.K = K;
  g.C = C;
  g.D = D;
  g.E = E;
  g.act = act;
  g.err = w->err;
  const long long active = act ? skkr_active_items(items) : items;
  // algorithmic BF16 tensor work: S(S+1)/2 real products of n x 2K x 2n per item
  // FP64-equivalent: one complex n x K by K x n product per item
  kstat_begin2(KS_OZAKI, (double)(S * (S + 1) / 2) * 8.0 * n * (double)n * K * (double)active,
               8.0 * n * (double)n * K * (double)active, st);
  g.tiles = (int)(items * mtiles * ntiles);
  const int rc = B.fused ? oz_launch<S, DB, 1, H>(w, ma, mb, g, st) : oz_launch<S, DB, 0, H>(w, ma, mb, g, st);
  kstat_end(st);
  if (rc) return rc;
  SKKR_LAUNCHED();
  return 0;
}

// f<S, DB, H>(...) for S = 3..8, the digit base of the depth and the form of the size
#define OZ_CASE(S, f, ...)                                                      \
  case S:                                                                       \
    return stacked ? f<S, 8, 1>(__VA_ARGS__) : d8 ? f<S, 8, 0>(__VA_ARGS__) : f<S, 7, 0>(__VA_ARGS__);
#define OZ_DISPATCH(S, n, K, f, ...)                                            \
  do {                                                                          \
    const bool d8 = oz_digits(K) == 8, stacked = oz_stacked(n, K);              \
    switch (S) {                                                                \
      OZ_CASE(3, f, __VA_ARGS__)                                                \
      OZ_CASE(4, f, __VA_ARGS__)                                                \
      OZ_CASE(5, f, __VA_ARGS__)                                                \
      OZ_CASE(6, f, __VA_ARGS__)                                                \
      OZ_CASE(7, f, __VA_ARGS__)                                                \
      OZ_CASE(8, f, __VA_ARGS__)                                                \
      default: return SKKR_ERR_ARG;                                             \
    }                                                                           \
  } while (0)

int mixed_split(MixedWork *w, int side, int slot, int S, const MatRef &M, int n, int K, int nk, int nc,
                const int *act, cudaStream_t st, bool reused) {
  if (n < 1 || n > 256 || K < 1 || K > 256 || nk * (long long)nc > 65535 || slot < 0 ||
      slot >= MIXED_SLOTS || (side != 0 && side != 1))
    return SKKR_ERR_ARG;
  OZ_DISPATCH(S, n, K, split_s, w, side, slot, M, n, K, nk, nc, act, st, reused);
}

int mixed_gemm_staged(MixedWork *w, int mode, int S, int sa, int sb, const MatRef &C, const MatRef &D,
                      const MatRef &E, int n, int K, int nk, int nc, const int *act, cudaStream_t st) {
  if (sa < 0 || sa >= MIXED_SLOTS || sb < 0 || sb >= MIXED_SLOTS) return SKKR_ERR_ARG;
  OZ_DISPATCH(S, n, K, gemm_s, w, mode, sa, sb, C, D, E, n, K, nk, nc, act, st);
}

int mixed_zgemm_k(MixedWork *w, int mode, int S, const MatRef &A, const MatRef &B, const MatRef &C,
                  const MatRef &D, const MatRef &E, int n, int K, int nk, int nc, const int *act,
                  cudaStream_t st) {
  int rc = mixed_split(w, 0, 0, S, A, n, K, nk, nc, act, st);
  if (!rc) rc = mixed_split(w, 1, 0, S, B, n, K, nk, nc, act, st);
  if (!rc) rc = mixed_gemm_staged(w, mode, S, 0, 0, C, D, E, n, K, nk, nc, act, st);
  return rc;
}

int mixed_zgemm(MixedWork *w, int mode, int S, const MatRef &A, const MatRef &B, const MatRef &C,
                const MatRef &D, const MatRef &E, int n, int nk, int nc, const int *act, cudaStream_t st) {
  return mixed_zgemm_k(w, mode, S, A, B, C, D, E, n, n, nk, nc, act, st);
}

// Newton residual check per item: an item whose last residual norm
// |I - A X|_F is above `limit` (or not finite) is marked for an FP64
// Gauss-Jordan redo; the others fold their norm into the running maximum
// (non-negative doubles order like their bit patterns: integer atomicMax)
__global__ void k_newton_check(const double *__restrict__ rn, const int *__restrict__ act, int items,
                               double limit, int *__restrict__ flag, unsigned long long *dmax,
                               unsigned long long *nfb) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= items) return;
  const int a = act ? act[i] : 1;
  const double r = rn[i];
  const int f = a && !(r <= limit);
  flag[i] = f;
  if (f) atomicAdd(nfb, 1ull);
  else if (a) atomicMax(dmax, (unsigned long long)__double_as_longlong(r));
}

// Items whose residual is above `limit` but below `basin` (Newton's
// quadratic regime) are marked for a further step.  One block: the count of
// marked items goes to *count (eager runs read it on the host), is added to
// *nref on the first further step, and, inside a captured graph, decides the
// IF node of the step (cudaGraphSetConditional).
__global__ void __launch_bounds__(1024) k_newton_select(const double *__restrict__ rn, const int *__restrict__ act,
                                                        int items, double limit, double basin, int *__restrict__ mark,
                                                        int *count, unsigned long long *nref, int first,
                                                        cudaGraphConditionalHandle cond, int use_cond,
                                                        int body_kernels) {
  __shared__ int part[32];
  int v = 0;
  for (int i = threadIdx.x; i < items; i += blockDim.x) {
    const int a = act ? act[i] : 1;
    const double r = rn[i];
    const int m = a && r > limit && r < basin;
    mark[i] = m;
    v += m;
  }
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    int t = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += part[w];
    *count = t;
    if (first && t) nref[0] += (unsigned long long)t;
    if (use_cond) {
      cudaGraphSetConditional(cond, t > 0 ? 1u : 0u);
      if (t > 0) nref[1] += (unsigned long long)body_kernels;
    }
  }
}

// Inside a stream capture: an IF node whose condition a kernel captured
// before it sets, with its body captured on `side`.  cond_handle creates the
// handle on the graph being captured (the setter needs it as an argument);
// cond_if_begin appends the node after the stream's current dependencies and
// starts the capture of its body; cond_if_end closes that capture.
int cond_handle(cudaStream_t st, cudaGraphConditionalHandle *h) {
  cudaStreamCaptureStatus cs;
  cudaGraph_t g;
  if (cudaStreamGetCaptureInfo(st, &cs, nullptr, &g, nullptr, nullptr, nullptr) != cudaSuccess ||
      cs != cudaStreamCaptureStatusActive)
    return SKKR_ERR_CUDA;
  return cudaGraphConditionalHandleCreate(h, g, 0, 0) == cudaSuccess ? 0 : SKKR_ERR_CUDA;
}

int cond_begin(cudaStream_t st, cudaStream_t side, cudaGraphConditionalHandle h, int type) {
  cudaStreamCaptureStatus cs;
  cudaGraph_t g;
  const cudaGraphNode_t *deps = nullptr;
  const cudaGraphEdgeData *ed = nullptr;
  size_t nd = 0;
  if (cudaStreamGetCaptureInfo(st, &cs, nullptr, &g, &deps, &ed, &nd) != cudaSuccess ||
      cs != cudaStreamCaptureStatusActive)
    return SKKR_ERR_CUDA;
  cudaGraphNodeParams p = {};
  p.type = cudaGraphNodeTypeConditional;
  p.conditional.handle = h;
  p.conditional.type = (cudaGraphConditionalNodeType)type;
  p.conditional.size = 1;
  cudaGraphNode_t node;
  if (cudaGraphAddNode(&node, g, deps, ed, nd, &p) != cudaSuccess) return SKKR_ERR_CUDA;
  if (cudaStreamUpdateCaptureDependencies(st, &node, nullptr, 1, cudaStreamSetCaptureDependencies) != cudaSuccess)
    return SKKR_ERR_CUDA;
  return cudaStreamBeginCaptureToGraph(side, p.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                       cudaStreamCaptureModeRelaxed) == cudaSuccess
             ? 0
             : SKKR_ERR_CUDA;
}

int cond_end(cudaStream_t side) {
  cudaGraph_t body = nullptr;
  return cudaStreamEndCapture(side, &body) == cudaSuccess ? 0 : SKKR_ERR_CUDA;
}

bool stream_capturing(cudaStream_t st) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  return cudaStreamIsCapturing(st, &cs) == cudaSuccess && cs == cudaStreamCaptureStatusActive;
}

// ---------------------------------------------------------------------------
// Autotuned thread layout of the FP32 Gauss-Jordan.  A size class fixes the
// rows per lane (32 RA >= n); its layouts differ in the number of update
// warps and in the blocks per SM.  Every
// layout gives the same inverse bit for bit (each element takes the same
// sequence of updates, the pivot search is deterministic), so the first
// batch of each (size class, batch size) key times the layouts once on the
// real operands and later calls use the fastest.  A capture in progress
// before a key is tuned takes the first layout.
using GjLaunch = void (*)(const MatRef &, const MatRef &, int, int, const int *, unsigned, cudaStream_t);

template <int RA, int W, int MINB>
static void gj_launch(const MatRef &A, const MatRef &X, int n, int nc, const int *act, unsigned items,
                      cudaStream_t st) {
  constexpr size_t smem = sizeof(GjShared<32 * RA>);
  if (smem > 48 * 1024)
    cudaFuncSetAttribute(k_cgj32<RA, W, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  k_cgj32<RA, W, MINB><<<items, (W + RA) * 32, smem, st>>>(A, X, n, nc, act);
}

struct GjClass {
  int nmax;
  int nv;
  GjLaunch f[2];
  const char *name[2];
};

static const GjClass GJ_CLASSES[4] = {
    {32, 2, {gj_launch<1, 4, 6>, gj_launch<1, 2, 8>}, {"4+1 warps", "2+1 warps"}},
    {64, 2, {gj_launch<2, 4, 4>, gj_launch<2, 8, 3>}, {"4+2 warps", "8+2 warps"}},
    {96, 2, {gj_launch<3, 6, 2>, gj_launch<3, 12, 1>}, {"6+3 warps", "12+3 warps"}},
    {128, 2, {gj_launch<4, 12, 1>, gj_launch<4, 8, 1>}, {"12+4 warps", "8+4 warps"}},
};

namespace {
std::mutex g_tune_mu;
std::map<std::pair<int, int>, int> g_tuned;  // (class, batch bucket) -> layout
int g_tune_force = 0;                         // > 0: always layout g_tune_force - 1 (tests)
}  // namespace

static GjLaunch gj_choose(int n, long long items, const MatRef &A, const MatRef &X, int nc, const int *act,
                          cudaStream_t st) {
  const int cls = (n - 1) / 32;
  const GjClass &C = GJ_CLASSES[cls];
  std::lock_guard<std::mutex> lk(g_tune_mu);
  if (g_tune_force > 0) return C.f[std::min(g_tune_force - 1, C.nv - 1)];
  // batches below one wave, below four waves, and larger
  const int bucket = items < 152 ? 0 : items < 608 ? 1 : 2;
  auto it = g_tuned.find({cls, bucket});
  if (it != g_tuned.end()) return C.f[it->second];
  if (C.nv == 1) {
    g_tuned[{cls, bucket}] = 0;
    return C.f[0];
  }
  if (stream_capturing(st)) return C.f[0];
  cudaEvent_t e0, e1;
  if (cudaEventCreate(&e0) != cudaSuccess) return C.f[0];
  if (cudaEventCreate(&e1) != cudaSuccess) {
    cudaEventDestroy(e0);
    return C.f[0];
  }
  // each layout: one warm run, then the best of three timed runs; a later
  // layout replaces the current choice only when it is 5 % faster (the
  // layouts are listed in order of preference)
  int best = 0;
  float tbest = 1e30f;
  for (int v = 0; v < C.nv; v++) {
    C.f[v](A, X, n, nc, act, (unsigned)items, st);  // warm (module load, caches)
    float tv = 1e30f;
    for (int rep = 0; rep < 3; rep++) {
      cudaEventRecord(e0, st);
      C.f[v](A, X, n, nc, act, (unsigned)items, st);
      cudaEventRecord(e1, st);
      float ms = 1e30f;
      if (cudaEventSynchronize(e1) == cudaSuccess && cudaEventElapsedTime(&ms, e0, e1) == cudaSuccess)
        tv = std::min(tv, ms);
    }
    if (tv < 0.95f * tbest) {
      tbest = tv;
      best = v;
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  g_tuned[{cls, bucket}] = best;
  return C.f[best];
}

int gj_tune_force(int v) {
  std::lock_guard<std::mutex> lk(g_tune_mu);
  g_tune_force = v;
  if (v == 0) g_tuned.clear();
  return 0;
}

std::string gj_tune_report() {
  std::lock_guard<std::mutex> lk(g_tune_mu);
  std::string r;
  static const char *bn[3] = {"<1 wave", "<4 waves", ">=4 waves"};
  for (auto &kv : g_tuned) {
    const GjClass &C = GJ_CLASSES[kv.first.first];
    r += "n<=" + std::to_string(C.nmax) + " " + bn[kv.first.second] + ": " + C.name[kv.second] + "; ";
  }
  return r;
}

// X = A^-1: FP32 Gauss-Jordan, then `newton` steps X += X (I - A X) with the
// residual product at S = sres slices and the correction at S = scorr.  An
// item is accepted when the residual before the last correction is at most
// `limit`.  X may be A itself (`inplace`); otherwise the two must not overlap.
int mixed_zinv(MixedWork *w, const MatRef &A, const MatRef &X, int n, int nk, int nc, const int *act,
               int newton, int sres, int scorr, double limit, bool inplace, cudaStream_t st) {
  if (n < 1 || n > 128 || newton < 1) return SKKR_ERR_ARG;
  const long long items = (long long)nk * nc, MB = (long long)n * n;
  int rc;
  if (inplace && (rc = grow((void **)&w->acopy, &w->ac_cap, (size_t)items * MB * sizeof(zd), false))) return rc;
  if ((rc = grow((void **)&w->rbuf, &w->rb_cap, (size_t)items * MB * sizeof(zd), false))) return rc;
  if ((rc = grow((void **)&w->rnorm, &w->rn_cap, (size_t)items * sizeof(double), false))) return rc;
  if ((rc = grow((void **)&w->flag, &w->flag_cap, (size_t)items * sizeof(int), false))) return rc;
  if ((rc = grow((void **)&w->mark, &w->mark_cap, (size_t)items * sizeof(int), false))) return rc;
  // the further Newton steps split X (and, unless B is fused, R) into slot 5
  // at sres slices (the standard correction uses fewer): reserve that size while
  // not capturing, so that a captured step never has to grow the slot
  if (!stream_capturing(st)) {
    int Mp, Np, Kp, mt, ntl, kbl;
    oz_dims(n, n, &Mp, &Np, &Kp, &mt, &ntl, &kbl);
    if ((rc = grow(&w->A[5].p, &w->A[5].cap, (size_t)items * sres * Mp * Kp * 2, true))) return rc;
    if (!w->fuse_b && (rc = grow(&w->B[5].p, &w->B[5].cap, (size_t)items * sres * Np * Kp * 2, true))) return rc;
  }
  // A itself serves the Gauss-Jordan start, the residuals and the FP64 redo
  // unless X overwrites it (in place): then a copy does
  const MatRef Ac = inplace ? mref(w->acopy, (long long)nc * MB, MB, n) : A;
  MatRef R = mref(w->rbuf, (long long)nc * MB, MB, n);
  if (inplace) launch_zaxpby(Ac, A, nullptr, 0, nullptr, 0, n, nk, nc, act, st);
  kstat_begin(KS_GJ, 8.0 * n * (double)n * n * (double)(act ? skkr_active_items(items) : items), st);
  gj_choose(n, items, Ac, X, nc, act, st)(Ac, X, n, nc, act, (unsigned)items, st);
  SKKR_LAUNCHED();
  kstat_end(st);
  // A is split once (A slot 0) for the residuals of every Newton step
  if ((rc = mixed_split(w, 0, 0, sres, Ac, n, n, nk, nc, act, st))) return rc;
  for (int it = 0; it < newton; it++) {
    // R = I - A X
    if ((rc = mixed_split(w, 1, 0, sres, X, n, n, nk, nc, act, st))) return rc;
    if ((rc = mixed_gemm_staged(w, 4, sres, 0, 0, R, R, R, n, n, nk, nc, act, st))) return rc;
    if (it == newton - 1) launch_fnorm(R, n, nk, nc, act, w->rnorm, st);
    // X = X + X R (slot 5: slot 0 keeps A)
    if ((rc = mixed_split(w, 0, 5, scorr, X, n, n, nk, nc, act, st))) return rc;
    if ((rc = mixed_split(w, 1, 5, scorr, R, n, n, nk, nc, act, st))) return rc;
    if ((rc = mixed_gemm_staged(w, 5, scorr, 5, 5, X, X, X, n, n, nk, nc, act, st))) return rc;
  }
  // Items above the limit but inside Newton's basin (|R| < 1/2) take up to
  // NEWTON_EXTRA further steps with the correction at sres slices as well:
  // the 3-slice correction leaves about cond(A) 2^-24 |R| in the next
  // residual, which stalls ill-conditioned items.  Each step runs only if an
  // item is marked: inside a captured graph an IF node decides on the
  // device; run eagerly, the host reads the count.
  const bool cap = stream_capturing(st);
  const long long hint = skkr_active_items(-1);
  for (int e = 0; e < NEWTON_EXTRA; e++) {
    cudaGraphConditionalHandle h = 0;
    if (cap && (rc = cond_handle(st, &h))) return rc;
    // the IF body below launches 2 sliced products, 1 norm and the splits:
    // 3, or 1 with the B operands fused
    const int nbody = w->fuse_b ? 4 : 6;
    k_newton_select<<<1, 1024, 0, st>>>(w->rnorm, act, (int)items, limit, 0.5, w->mark, w->cnt, w->nref, e == 0,
                                        h, cap ? 1 : 0, nbody);
    SKKR_LAUNCHED();
    const long long l_body = g_skkr_launches;
    cudaStream_t sx = st;
    if (cap) {
      if ((rc = cond_begin(st, w->side, h, cudaGraphCondTypeIf))) return rc;
      sx = w->side;
    } else {
      int marked = 0;
      if (cudaMemcpyAsync(&marked, w->cnt, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
          cudaStreamSynchronize(st) != cudaSuccess)
        return SKKR_ERR_CUDA;
      if (marked == 0) break;
      skkr_set_active_items(marked);
    }
    const int *mk = w->mark;
    auto step = [&]() -> int {
      int r;
      if ((r = mixed_split(w, 1, 0, sres, X, n, n, nk, nc, mk, sx))) return r;
      if ((r = mixed_gemm_staged(w, 4, sres, 0, 0, R, R, R, n, n, nk, nc, mk, sx))) return r;
      launch_fnorm(R, n, nk, nc, mk, w->rnorm, sx);
      if ((r = mixed_split(w, 0, 5, sres, X, n, n, nk, nc, mk, sx))) return r;
      if ((r = mixed_split(w, 1, 5, sres, R, n, n, nk, nc, mk, sx))) return r;
      return mixed_gemm_staged(w, 5, sres, 5, 5, X, X, X, n, n, nk, nc, mk, sx);
    };
    rc = step();
    if (cap) {  // close the body's capture whatever happened inside it
      const int rc2 = cond_end(w->side);
      if (!rc) rc = rc2;
      // the body's kernels are counted when they run (nref[1]), not here
      g_skkr_launches = l_body;
      g_skkr_if_captured += nbody;
    }
    if (rc) return rc;
    skkr_set_active_items(hint);
  }
  // An ill-conditioned A (cond ~ 1e7 and above) leaves the FP32 start outside
  // Newton's basin: such items are inverted again in FP64 (copy A, column-
  // pivoting Gauss-Jordan), masked so that the others are untouched.  The
  // residual before the last correction bounds the final error by its square.
  k_newton_check<<<(unsigned)((items + 255) / 256), 256, 0, st>>>(w->rnorm, act, (int)items, limit, w->flag,
                                                                   w->dmax, w->nfb);
  SKKR_LAUNCHED();
  launch_zaxpby(X, Ac, nullptr, 0, nullptr, 0, n, nk, nc, w->flag, st);
  launch_zgj(X, n, nk, nc, w->flag, st);
  return 0;
}

// ---------------------------------------------------------------------------
// FP64 products and inverses on the tensor cores.  Eight slices of eight bits
// hold a 64-bit fixed-point value per element, in units of 2^-63 of its row's
// (A) or column's (B) scale sigma_i, tau_j (the power of two above its
// largest), and the slice pairs past level 7 are left out.  An output errs by
//   2^-53 |C_ij| + 2^-60 sigma_i tau_j
// at a depth of 128 (the second term as a root mean square over digits;
// 2^-53 sigma_i tau_j if every digit left out were the largest and of one
// sign), where FP64's own 2K roundings are relative to sum_k |a_ik| |b_kj|.
// That sum is of the order of sigma_i tau_j for operands of even scale, and
// the error is below FP64's; it is far below it where a row's large elements
// meet a column's small ones, and there the error is above FP64's: callers
// keep strongly graded blocks on the FP64 pipe (choose_engine in capi.cu).
// (The sums of levels 4 to 7 leave FP32's exact integers only where nearly all
// digits are the largest and of one sign, by a unit of that level.)  The
// depth is cut into `halves` above 128, where the level sums would leave
// FP32's integers, and for BdG blocks (electron-first layout): each half then
// has its own row and column scales, so that the O(Delta) electron-hole blocks
// keep their own relative precision beside the diagonal ones.  590 products of
// n = 128: 8.01 ms on the FP64 pipe (99.5 % of its rate), 0.28 ms staged, 0.30 fused.
int wide_zgemm(MixedWork *w, int mode, const MatRef &A, const MatRef &B, const MatRef &C, const MatRef &D,
               const MatRef &E, int n, bool halves, int nk, int nc, const int *act, cudaStream_t st) {
  if (n <= 128 && !halves) return mixed_zgemm(w, mode, WIDE_SLICES, A, B, C, D, E, n, nk, nc, act, st);
  // A B = A[:, :h] B[:h, :] + A[:, h:] B[h:, :]; every mode but 0, 3 and 4 is additive per half
  const int h = n / 2, m2 = mode == 0 ? 5 : (mode == 3 || mode == 4) ? 1 : mode;
  const MatRef A2 = mref_offset(A, (long long)h * A.ld), B2 = mref_offset(B, h);
  const int rc = mixed_zgemm_k(w, mode, WIDE_SLICES, A, B, C, D, E, n, h, nk, nc, act, st);
  if (rc) return rc;
  return mixed_zgemm_k(w, m2, WIDE_SLICES, A2, B2, C, D, E, n, n - h, nk, nc, act, st);
}

// X = A^-1 to FP64 accuracy.  Up to 128 rows: mixed_zinv with eight-slice
// residuals, four-slice corrections and the acceptance limit at 1e-9, whose
// square is below FP64's rounding.  Above, and in `halves` (n even): the 2 x 2
// block form (X11 = A11^-1, U = X11 A12, T = A21 X11, S = A22 - A21 U, Y = S^-1) with
// such inverses and products, then one Newton step on the whole matrix, which also checks it.  What is not accepted is inverted by the
// FP64 Gauss-Jordan, as are odd sizes above 128.  30 inverses of n = 256:
// 18.9 ms by k_zgj (one block, hence one SM, per matrix).
int wide_zinv(MixedWork *w, const MatRef &A, const MatRef &X, int n, bool halves, int nk, int nc, const int *act,
              bool inplace, cudaStream_t st) {
  if (n <= 128 && !halves) return mixed_zinv(w, A, X, n, nk, nc, act, 2, WIDE_SLICES, 4, WIDE_LIMIT, inplace, st);
  if (n > 256) return SKKR_ERR_ARG;
  if (n & 1) {
    if (!inplace) launch_zaxpby(X, A, nullptr, 0, nullptr, 0, n, nk, nc, act, st);
    launch_zgj(X, n, nk, nc, act, st);
    return 0;
  }
  const int h = n / 2;
  const long long items = (long long)nk * nc, HB = (long long)h * h, NN = (long long)n * n;
  // per item: X11, U, T, S, Y (h x h each), R and, in place, A (n x n each); then one zero block
  const long long per = 5 * HB + (inplace ? 2 : 1) * NN;
  int rc;
  const size_t need = ((size_t)items * per + HB) * sizeof(zd);
  if (need > w->big_cap && stream_capturing(st)) return SKKR_ERR_CUDA;
  if ((rc = grow((void **)&w->big, &w->big_cap, need, false))) return rc;
  if ((rc = grow((void **)&w->rnorm, &w->rn_cap, (size_t)items * sizeof(double), false))) return rc;
  if ((rc = grow((void **)&w->flag, &w->flag_cap, (size_t)items * sizeof(int), false))) return rc;
  auto blk = [&](long long off, int ld) { return mref(w->big + HB + off, nc * per, per, ld); };
  const MatRef Z = mref(w->big, 0, 0, h), X11 = blk(0, h), U = blk(HB, h), T = blk(2 * HB, h), S = blk(3 * HB, h),
               Y = blk(4 * HB, h), R = blk(5 * HB, n), Ac = inplace ? blk(5 * HB + NN, n) : A;
  if (cudaMemsetAsync(w->big, 0, HB * sizeof(zd), st) != cudaSuccess) return SKKR_ERR_CUDA;
  if (inplace) launch_zaxpby(Ac, A, nullptr, 0, nullptr, 0, n, nk, nc, act, st);
  auto sub = [&](const MatRef &M, int r, int c) { return mref_offset(M, r + (long long)c * M.ld); };
  const MatRef A12 = sub(Ac, 0, h), A21 = sub(Ac, h, 0), A22 = sub(Ac, h, h);
  const MatRef Xa = X, X12 = sub(X, 0, h), X21 = sub(X, h, 0), X22 = sub(X, h, h);
  auto prod = [&](int mode, const MatRef &a, const MatRef &b, const MatRef &c, const MatRef &d) {
    return wide_zgemm(w, mode, a, b, c, d, c, h, false, nk, nc, act, st);
  };
  if ((rc = wide_zinv(w, Ac, X11, h, false, nk, nc, act, false, st))) return rc;
  if ((rc = prod(0, X11, A12, U, U))) return rc;    // U = X11 A12
  if ((rc = prod(0, A21, X11, T, T))) return rc;    // T = A21 X11
  if ((rc = prod(3, A21, U, S, A22))) return rc;    // S = A22 - A21 U
  if ((rc = wide_zinv(w, S, Y, h, false, nk, nc, act, false, st))) return rc;
  launch_zaxpby(X22, Y, nullptr, 0, nullptr, 0, h, nk, nc, act, st);
  if ((rc = prod(3, U, Y, X12, Z))) return rc;      // X12 = -U Y
  if ((rc = prod(3, Y, T, X21, Z))) return rc;      // X21 = -Y T
  if ((rc = prod(3, X12, T, Xa, X11))) return rc;   // X11 - X12 T
  // one Newton step: R = I - A X, X += X R
  if ((rc = wide_zgemm(w, 4, Ac, X, R, R, R, n, true, nk, nc, act, st))) return rc;
  launch_fnorm(R, n, nk, nc, act, w->rnorm, st);
  const MatRef Xr = sub(X, 0, h), R2 = mref_offset(R, h);
  if ((rc = mixed_split(w, 0, 1, 4, X, n, h, nk, nc, act, st))) return rc;
  if ((rc = mixed_split(w, 0, 2, 4, Xr, n, h, nk, nc, act, st))) return rc;
  if ((rc = mixed_split(w, 1, 1, 4, R, n, h, nk, nc, act, st))) return rc;
  if ((rc = mixed_split(w, 1, 2, 4, R2, n, h, nk, nc, act, st))) return rc;
  if ((rc = mixed_gemm_staged(w, 5, 4, 1, 1, X, X, X, n, h, nk, nc, act, st))) return rc;
  if ((rc = mixed_gemm_staged(w, 5, 4, 2, 2, X, X, X, n, h, nk, nc, act, st))) return rc;
  k_newton_check<<<(unsigned)((items + 255) / 256), 256, 0, st>>>(w->rnorm, act, (int)items, WIDE_LIMIT, w->flag,
                                                                   w->dmax, w->nfb);
  SKKR_LAUNCHED();
  launch_zaxpby(X, Ac, nullptr, 0, nullptr, 0, n, nk, nc, w->flag, st);
  launch_zgj(X, n, nk, nc, w->flag, st);
  return 0;
}
