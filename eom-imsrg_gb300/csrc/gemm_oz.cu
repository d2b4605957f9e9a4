// FP64 matrix products on the BF16 tensor cores, by exact integer digits.
//
// GB300's FP64 pipe does 1.2 TFLOP/s, its BF16 tensor cores about 1900: an FP64 product made of many exact BF16
// products is still much the faster one.  The scheme is that of Ozaki, Ogita, Oishi and Rump (Numer. Algorithms 59,
// 2012): every row of an operand gets a power of two 2^e above its largest element, every element becomes the integer
// a 2^(62-e) (rounded to nearest), written in eight balanced base-256 digits d_0 .. d_7 (|d| <= 128, exact in BF16's
// eight significant bits):  a = 2^e sum_s d_s 2^(-6-8s).  The products of digits i and j all carry the weight
// 2^(ea+eb-12-8(i+j)), so the 36 slice products with i + j = d <= 7 go into one of eight FP32 accumulators per d.
// A digit product is at most 2^14 and an accumulator takes at most 8 of them for each of 128 values of K before it is
// read out: 8 * 128 * 2^14 = 2^24, so every sum is an integer that FP32 holds exactly.  The accumulators are then
// added up in 64-bit integers (four of them in each, H and L), and only the finished sum T = H 2^32 + L is rounded,
// once, to FP64.  What is lost: 2^-63 of the row's power of two for each element, and the digit products with
// i + j >= 8, together below K 2^-59 of the two powers of two (K^(1/2) 2^-62 for digits that behave as random ones),
// against a rounding of 2^-53 of the running sum at every step of a chain of FP64 FMAs.
//
// The powers of two say little about an element where the large elements of a row meet the small ones of a column, and an
// FMA chain would be far better there.  So a ninth slice holds every element's magnitude, |a| 2^-ea in BF16, and its product
// gives each output element's sum of |a||b| 2^-(ea+eb), term by term, before the digits.  Digits are kept from
// 2^-6 on: then K 2^-59 is within K 2^-53 of the sum of |a||b|, the error bound of the FMAs, for every element (what is usual,
// K^(1/2) 2^-62, is there at most K^(1/2) 2^-56 of the sum, where a chain of roundings usually comes to 2^-55 of it, and far below
// that where the sum is of the size of the powers of two, as most are).  Elements below that are noted and left to
// k_gemm_fp64_rest: fewer than one in 10^5 of random operators' products, one in 300 to 3000 of those with a flow's Omega, whose
// elements fall off faster ([Omega, [Omega, H]] at eMax 10 9.6 ms, 8.4 with no such care; with 2^-6 K^(1/4), so that the usual
// errors match too, 11.6; with 2^-6 K^(1/2) 14).  The ninth product costs 2 of 74 MMAs and a reading more of the accumulators for
// each term.
//
// Rows that hold an Inf or a NaN have no such form: the split raises a flag, this kernel then leaves the outputs alone
// and k_gemm_fp64_rest, launched behind it with the same flag, computes the whole list.
//
// Measured at eMax 10 (GB300): the ladder's list (33 G multiply-adds, K up to 1291) 63.2 -> 3.0 ms, the cross-coupled
// list (9.1 G, K up to 74) 17.7 -> 1.7 ms against k_gemm_fp64; error of W1 and W2 against extended precision at eMax 8
// 6.6e-17 (norm), 6.2e-16 before.  An MMA takes about 51 clocks, near the 48 that reading its 6 KB of operands from
// shared memory takes; a list of small K is bound by the readers' integer instructions (about 60 an output element).
//
// k_oz_split writes the digits straight in the form that tcgen05.mma reads from shared memory (K-major rows of 64
// bytes, 64-byte swizzle), so a stage of the GEMM's pipeline is filled by a few untiled bulk copies.
// k_oz_gemm is persistent and warp-specialised: warp 0 copies, warp 1 issues the MMAs, sixteen warps read the
// accumulators out of TMEM.  All of TMEM (512 columns) holds the eight 128 x 64 accumulators of one tile; each has
// its own full / empty barrier, so the readers empty one while the MMAs go on in the others.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <map>
#include <queue>
#include <tuple>

#include "engine.h"
#include "gemm_oz.h"
#include "kernels.h"
#include "umma.cuh"

namespace imsrg {

namespace {

constexpr int S = kOzSlices;
constexpr int kSliceBytes = kOzTileM * kOzBlockK * 2;  // 8 KiB: 128 rows of 64 bytes
constexpr int kBlockBytes = S * kSliceBytes;           // 64 KiB
constexpr int kStageA = kBlockBytes, kStageB = kBlockBytes / 2;
constexpr int kStageBytes = kStageA + kStageB;
constexpr int kStages = 2;
constexpr int kMagBlocks = S;    // K blocks of magnitudes in a stage
constexpr int kChunkBlocks = 4;  // K blocks between two readings of the accumulators: K = 128
constexpr int kEpiWarps = 16;
constexpr int kThreads = 32 * (2 + kEpiWarps);
constexpr size_t kSmem = (size_t)kStages * kStageBytes + 1024 + 256 + 2 * 32 * kEpiWarps;

// The accumulators in the order in which they are issued and read.  The last one holds the sums of magnitudes before a term's
// first digits: its own digits come last, so that the readers of the tile before delay those alone.
__host__ __device__ constexpr int oz_order(int x) { return x < S - 1 ? S - 2 - x : S - 1; }

// the exponent e with |a| < 2^e of the largest high word of a row's magnitudes (subnormals count as 2^-1022)
__device__ __forceinline__ int oz_exp(unsigned maxhi) { return max((int)(maxhi >> 20), 1) - 1022; }

// a 2^(62-e) to the nearest integer, as the biased digits: byte 7 - s is d_s + 128.  mag: |a| 2^-e rounded down to BF16, at
// least 2^-62 unless a is zero (a product of two is then above the smallest normal number).
__device__ __forceinline__ unsigned long long oz_digits(double a, int e, unsigned& mag) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(a);
  const int ea = (int)(b >> 52) & 0x7FF;
  const unsigned long long m = (b & 0xFFFFFFFFFFFFFull) | (ea ? 1ull << 52 : 0ull);
  const int sh = max(ea, 1) - 1075 + 62 - e;  // <= 9
  unsigned long long i;
  if (sh >= 0) i = m << sh;
  else if (sh > -55) i = (m + (1ull << (-sh - 1))) >> -sh;
  else i = 0;
  const int z = __clzll((long long)(i | 1ull));
  mag = m ? (unsigned)(128 - z) << 7 | ((unsigned)((i << z) >> 56) & 0x7Fu) : 0u;
  if (b >> 63) i = 0ull - i;
  return (i + 0x0080808080808080ull) ^ 0x8000000000000000ull;
}
// the BF16 values of digit s of two elements, packed (low half: the first)
__device__ __forceinline__ unsigned oz_pair(unsigned long long x, unsigned long long y, int s) {
  const unsigned bx = (unsigned)(x >> (56 - 8 * s)) & 0xFFu, by = (unsigned)(y >> (56 - 8 * s)) & 0xFFu;
  const float fx = __uint_as_float(0x4B000000u | bx) - 8388736.0f, fy = __uint_as_float(0x4B000000u | by) - 8388736.0f;
  return __byte_perm(__float_as_uint(fx), __float_as_uint(fy), 0x7632);
}

}  // namespace

// One CTA per 32 rows of an operand: the row exponents, then the digits and magnitudes.  Bound by memory: 8 bytes read (twice,
// the second time from L2) and 18 written an element.
__global__ void __launch_bounds__(256) k_oz_split(const OzOperand* __restrict__ ops, const OzChunk* __restrict__ chunks,
                                                  GemmOperands in, char* __restrict__ buf, char* __restrict__ mag,
                                                  int* __restrict__ exps, int* flag) {
  __shared__ unsigned mx[32];
  const OzChunk ch = chunks[blockIdx.x];
  const OzOperand o = ops[ch.op];
  const double* A = in.in[o.id] + o.off;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nr = min(32, o.rows - ch.r0);
  if (threadIdx.x < 32) mx[threadIdx.x] = 0u;
  __syncthreads();
  if (o.ks == 1) {  // K contiguous: a warp per row
    for (int r = warp; r < nr; r += 8) {
      const double* row = A + (int64_t)(ch.r0 + r) * o.rs;
      unsigned m = 0u;
      for (int k = lane; k < o.K; k += 32) m = max(m, (unsigned)__double2hiint(row[k]) & 0x7FFFFFFFu);
      m = __reduce_max_sync(0xffffffffu, m);
      if (lane == 0) mx[r] = m;
    }
  } else if (lane < nr) {  // rows contiguous: lanes along the rows
    const double* col = A + ch.r0 + lane;
    unsigned m = 0u;
    for (int k = warp; k < o.K; k += 8) m = max(m, (unsigned)__double2hiint(col[(int64_t)k * o.ks]) & 0x7FFFFFFFu);
    atomicMax(&mx[lane], m);
  }
  __syncthreads();
  if (threadIdx.x < nr) {
    exps[o.exp0 + ch.r0 + threadIdx.x] = oz_exp(mx[threadIdx.x]);
    if (mx[threadIdx.x] >= 0x7FF00000u) *flag = 1;  // Inf or NaN
  }
  const int rb = ch.r0 >> 7, rin = ch.r0 & 127;
  char* blk = buf + (o.blk0 + (int64_t)rb * o.nkb) * kBlockBytes;
  char* mblk = mag + (o.blk0 + (int64_t)rb * o.nkb) * kSliceBytes;
  if (o.ks == 1) {  // two rows of 32 K a warp pass, two K a thread
    const int half = lane >> 4, k2 = (lane & 15) * 2;
    for (int x = warp; x < o.nkb * 16; x += 8) {
      const int kb = x >> 4, r = (x & 15) * 2 + half, k = kb * 32 + k2;
      if (r >= nr) continue;
      const double* row = A + (int64_t)(ch.r0 + r) * o.rs;
      const int e = oz_exp(mx[r]);
      unsigned m0, m1;
      const unsigned long long d0 = oz_digits(k < o.K ? row[k] : 0.0, e, m0), d1 = oz_digits(k + 1 < o.K ? row[k + 1] : 0.0, e, m1);
      const int rr = rin + r, at = rr * 64 + (((k2 >> 3) ^ ((rr >> 1) & 3)) << 4) + (k2 & 7) * 2;
      char* dst = blk + (int64_t)kb * kBlockBytes + at;
#pragma unroll
      for (int s = 0; s < S; ++s) *reinterpret_cast<unsigned*>(dst + s * kSliceBytes) = oz_pair(d0, d1, s);
      *reinterpret_cast<unsigned*>(mblk + (int64_t)kb * kSliceBytes + at) = m0 | m1 << 16;
    }
  } else if (lane < nr) {  // lanes along the rows, eight K (16 bytes of a slice's row) a thread
    const double* col = A + ch.r0 + lane;
    const int e = oz_exp(mx[lane]), rr = rin + lane;
    for (int x = warp; x < o.nkb * 4; x += 8) {
      const int kb = x >> 2, c = x & 3, k0 = kb * 32 + c * 8;
      unsigned long long d[8];
      unsigned m[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) d[u] = oz_digits(k0 + u < o.K ? col[(int64_t)(k0 + u) * o.ks] : 0.0, e, m[u]);
      const int at = rr * 64 + ((c ^ ((rr >> 1) & 3)) << 4);
      char* dst = blk + (int64_t)kb * kBlockBytes + at;
#pragma unroll
      for (int s = 0; s < S; ++s)
        *reinterpret_cast<uint4*>(dst + s * kSliceBytes) = make_uint4(oz_pair(d[0], d[1], s), oz_pair(d[2], d[3], s),
                                                                      oz_pair(d[4], d[5], s), oz_pair(d[6], d[7], s));
      *reinterpret_cast<uint4*>(mblk + (int64_t)kb * kSliceBytes + at) =
          make_uint4(m[0] | m[1] << 16, m[2] | m[3] << 16, m[4] | m[5] << 16, m[6] | m[7] << 16);
    }
  }
}

namespace {

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
// shared-memory matrix descriptor: K-major operand rows of 64 bytes, 64-byte swizzle, 8-row groups 512 bytes apart
constexpr uint32_t kDescHi = (uint32_t)(512 >> 4) | 1u << 14 | 4u << 29;  // bits 32-63: SBO, version, swizzle
__device__ __forceinline__ uint32_t oz_desc_lo(uint32_t saddr) { return ((saddr & 0x3FFFFu) >> 4) | 1u << 16; }
__device__ __forceinline__ void oz_umma(uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n .reg .b64 da, db;\n setp.ne.b32 p, %4, 0;\n"
      " mov.b64 da, {%1, %5};\n mov.b64 db, {%2, %5};\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n}\n" ::"r"(tmem_d),
      "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(kDescHi)
      : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// +-(H 2^32 + L) 2^e rounded to nearest (ties away from zero), |H| < 2^55, in integer instructions (three FP64
// instructions here would take longer than all of these)
__device__ __forceinline__ double oz_value(long long H, long long L, bool neg, int e) {
  const long long h0 = H + (L >> 32), sg = h0 >> 63;
  const unsigned s32 = (unsigned)sg, l = ((unsigned)L ^ s32) - s32;
  unsigned long long h = (unsigned long long)(h0 ^ sg) + (unsigned long long)(l == 0u ? s32 & 1u : 0u);
  unsigned low = l;
  int ex = 95 + e + 1023;  // exponent field of the leading bit of h 2^32 + l, still without its leading zeros
  if (h == 0ull) {
    h = (unsigned long long)l << 32;
    low = 0u;
    ex -= 64;
  }
  const int z = __clzll((long long)h);
  unsigned long long m = (h << (z & 63)) | (((unsigned long long)low << 31) >> ((63 - z) & 63));
  m = (m >> 11) + ((m >> 10) & 1ull);
  ex -= z;  // a carry out of the mantissa moves the exponent up by itself
  const int exc = min(max(ex, 1), 2045);
  const unsigned sign = ((s32 & 1u) ^ (neg ? 1u : 0u)) << 31;
  double v = __hiloint2double((int)(((unsigned)(m >> 32) + ((unsigned)(exc - 1) << 20)) | sign), (int)(unsigned)m);
  if (h == 0ull) v = 0.0;
  else if (ex != exc)  // a subnormal result or an overflow
    v *= __hiloint2double((min(max(ex - exc, -1022), 1023) + 1023) << 20, 0);
  return v;
}
// acc + v 2^s
template <int SH>
__device__ __forceinline__ void oz_mad(long long& acc, int v) {
  asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(acc) : "r"(v), "n"(1 << SH));
}

}  // namespace

__global__ void __launch_bounds__(kThreads, 1)
    k_oz_gemm(const OzProb* __restrict__ probs, const OzTile* __restrict__ tiles, const int* __restrict__ start, GemmOperands out,
              const char* __restrict__ buf, const char* __restrict__ mag, const int* __restrict__ exps, int* flag,
              OzRedo* __restrict__ redo, int max_redo, int* err, unsigned long long wait_ns, int unarmed_it) {
  if (*flag) return;  // a row with an Inf or a NaN: k_gemm_fp64_rest computes the list
  extern __shared__ uint8_t oz_smem[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(oz_smem) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + (size_t)kStages * kStageBytes);
  uint64_t* empty = full + kStages;
  uint64_t* dfull = empty + kStages;
  uint64_t* dempty = dfull + S;
  uint64_t* drain = dempty + S;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* consumed = reinterpret_cast<volatile int*>(tmem_slot + 2);
  unsigned short* coarse = reinterpret_cast<unsigned short*>(tmem_slot + 4);  // a word for each reader's 16 elements
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int d = 0; d < S; ++d) {
      mbar_init(&dfull[d], 1);
      mbar_init(&dempty[d], kEpiWarps);
    }
    mbar_init(drain, 1);
    *abort_flag = 0;
    *consumed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int t0 = start[blockIdx.x], t1 = start[blockIdx.x + 1];  // this CTA's tiles

  int it = 0;  // stages filled (copies) or taken (MMAs)
  if (warp == 0) {
    if (elect_one()) {  // ---- copies
      bool ok = true;
      for (int t = t0; t < t1 && ok; ++t) {
        const OzTile tile = tiles[t];
        const OzProb& P = probs[tile.prob];
        for (int term = 0; term < P.nterm && ok; ++term) {
          const int nkb = P.t[term].nkb;
          const int64_t ablk = P.t[term].a_blk + (int64_t)(tile.m0 >> 7) * nkb, bblk = P.t[term].b_blk + (int64_t)(tile.n0 >> 7) * nkb;
          const int half = ((tile.n0 >> 6) & 1) * (kSliceBytes / 2);
          for (int kb0 = 0; kb0 < nkb; kb0 += kMagBlocks, ++it) {  // the magnitudes of up to eight K blocks in one stage
            const int s = it % kStages, n = min(kMagBlocks, nkb - kb0);
            if (!mbar_wait(&empty[s], ((it / kStages) & 1) ^ 1, abort_flag, err, 1, wait_ns)) { ok = false; break; }
            // test switch (imsrg_test_unarmed_stage): CTA 0 issues no copy for this stage and nothing arrives on its barrier
            if (it == unarmed_it && blockIdx.x == 0) continue;
            mbar_expect_tx(&full[s], (uint32_t)(n * (kSliceBytes + kSliceBytes / 2)));
            const uint32_t st = smem_u32(smem + (size_t)s * kStageBytes);
            bulk_load(st, mag + (ablk + kb0) * kSliceBytes, (uint32_t)(n * kSliceBytes), &full[s]);
            for (int j = 0; j < n; ++j)
              bulk_load(st + kStageA + j * (kSliceBytes / 2), mag + (bblk + kb0 + j) * kSliceBytes + half, kSliceBytes / 2, &full[s]);
          }
          if (!ok) break;
          const char* a = buf + ablk * kBlockBytes;
          // a tile of 64 columns takes the upper or the lower half of every slice of its operand block
          const char* b = buf + bblk * kBlockBytes + half;
          for (int kb = 0; kb < nkb; ++kb, ++it) {
            const int s = it % kStages;
            if (!mbar_wait(&empty[s], ((it / kStages) & 1) ^ 1, abort_flag, err, 1, wait_ns)) { ok = false; break; }
            mbar_expect_tx(&full[s], (uint32_t)kStageBytes);
            const uint32_t st = smem_u32(smem + (size_t)s * kStageBytes);
            bulk_load(st, a + (int64_t)kb * kBlockBytes, kStageA, &full[s]);
#pragma unroll
            for (int sl = 0; sl < S; ++sl)
              bulk_load(st + kStageA + sl * (kSliceBytes / 2), b + (int64_t)kb * kBlockBytes + sl * kSliceBytes,
                        kSliceBytes / 2, &full[s]);
          }
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {  // ---- MMAs
      int cc = 0, cm = 0;  // cc: chunks so far; cm: sums of magnitudes so far
      bool ok = true;
      for (int t = t0; t < t1 && ok; ++t) {
        const OzTile tile = tiles[t];
        const OzProb& P = probs[tile.prob];
        const int nterm = P.nterm;
        // FP32 accumulators, BF16 operands, both K-major, N = w, M = 128
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(tile.w >> 3) << 17) | (8u << 24);
        for (int term = 0; term < nterm && ok; ++term) {
          const int nkb = P.t[term].nkb;
          {  // the sums of magnitudes
            if (!mbar_wait(&dempty[S - 1], ((cc + cm) & 1) ^ 1, abort_flag, err, 2, wait_ns)) { ok = false; break; }
            tc_fence_after();
            for (int kb0 = 0; kb0 < nkb; kb0 += kMagBlocks, ++it) {
              const int s = it % kStages, n = min(kMagBlocks, nkb - kb0);
              if (!mbar_wait(&full[s], (it / kStages) & 1, abort_flag, err, 3, wait_ns)) { ok = false; break; }
              tc_fence_after();
              const uint32_t st = smem_u32(smem) + (uint32_t)(s * kStageBytes);
              const uint32_t da = oz_desc_lo(st), db = oz_desc_lo(st + kStageA);
              for (int j = 0; j < n; ++j)
#pragma unroll
                for (int ks = 0; ks < 2; ++ks)
                  oz_umma(tmem_base + (S - 1) * kOzTileN, da + ((j * kSliceBytes + ks * 32) >> 4),
                          db + ((j * (kSliceBytes / 2) + ks * 32) >> 4), idesc, (kb0 == 0 && j == 0 && ks == 0) ? 0u : 1u);
              umma_commit(&empty[s]);
              *consumed = it + 1;
            }
            if (!ok) break;
            umma_commit(&dfull[S - 1]);
            ++cm;
          }
          for (int kb = 0; kb < nkb && ok; ++kb, ++it) {
            const int s = it % kStages;
            const bool first = (kb & (kChunkBlocks - 1)) == 0, last = (kb & (kChunkBlocks - 1)) == kChunkBlocks - 1 || kb == nkb - 1;
            if (!mbar_wait(&full[s], (it / kStages) & 1, abort_flag, err, 3, wait_ns)) { ok = false; break; }
            tc_fence_after();
            const uint32_t st = smem_u32(smem) + (uint32_t)(s * kStageBytes);
            const uint32_t da = oz_desc_lo(st), db = oz_desc_lo(st + kStageA);
#pragma unroll
            for (int x = 0; x < S; ++x) {
              const int d = oz_order(x);
              if (first) {
                if (!mbar_wait(&dempty[d], ((d == S - 1 ? cc + cm : cc) & 1) ^ 1, abort_flag, err, 2, wait_ns)) { ok = false; break; }
                tc_fence_after();
              }
#pragma unroll
              for (int i = 0; i <= d; ++i)
#pragma unroll
                for (int ks = 0; ks < 2; ++ks)
                  oz_umma(tmem_base + d * kOzTileN, da + ((i * kSliceBytes + ks * 32) >> 4),
                          db + (((d - i) * (kSliceBytes / 2) + ks * 32) >> 4), idesc,
                          (first && i == 0 && ks == 0) ? 0u : 1u);
              if (last) umma_commit(&dfull[d]);
            }
            if (!ok) break;
            umma_commit(&empty[s]);
            *consumed = it + 1;
            if (last) ++cc;
          }
        }
      }
    }
  } else {
    // ---- readers: warp (quad, grp) has rows 32 quad .. + 31 and columns 16 grp .. + 15 of the tile
    const int quad = warp & 3, grp = (warp - 2) >> 2;
    const uint32_t tm = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(grp * 16);
    int cc = 0, cm = 0;
    bool ok = true;
    for (int t = t0; t < t1 && ok; ++t) {
      const OzTile tile = tiles[t];
      const OzProb& P = probs[tile.prob];
      const int m = tile.m0 + quad * 32 + lane, n = tile.n0 + grp * 16;
      const bool mine = grp * 16 < tile.w;
      const int nterm = P.nterm;
      for (int term = 0; term < nterm && ok; ++term) {
        const OzTerm& T = P.t[term];
        const int nchunk = (T.nkb + kChunkBlocks - 1) / kChunkBlocks;
        const int ea = __ldg(exps + T.a_exp + min(m, P.M - 1)) - 68, eb = __ldg(exps + T.b_exp + min(n + (lane & 15), P.N - 1));
        // elements whose sum of magnitudes is too small for the digits: noted for k_gemm_fp64_rest
        {
          ok = __all_sync(0xffffffffu, mbar_wait(&dfull[S - 1], (cc + cm) & 1, abort_flag, err, 4, wait_ns));
          if (!ok) break;
          tc_fence_after();
          unsigned c16 = 0u;
          if (mine) {
            uint32_t r[16];
            tmem_ld16(tm + (uint32_t)((S - 1) * kOzTileN), r);
            const unsigned least = __float_as_uint(kOzLeast) - 1u;
#pragma unroll
            for (int j = 0; j < 16; ++j) c16 |= r[j] - 1u < least ? 1u << j : 0u;  // 0 < sum < least, by the bits
            if (c16) c16 = m < P.M ? c16 & ((1u << min(max(P.N - n, 0), 16)) - 1u) : 0u;
            if (__any_sync(0xffffffffu, c16 != 0u)) {
              const bool many = __reduce_add_sync(0xffffffffu, __popc(c16)) > kOzSingles;  // these from the end backwards
              int x = 0;
              if (lane == 0) x = many ? max_redo - 1 - atomicAdd(flag + 2, 1) : atomicAdd(flag + 1, 1);
              x = __shfl_sync(0xffffffffu, x, 0);
              if (lane == 0) *reinterpret_cast<int4*>(&redo[x]) = make_int4(P.src, T.src, tile.m0 + quad * 32, n);
              redo[x].mask[lane] = (unsigned short)c16;
            }
            if (P.accum) coarse[threadIdx.x - 64] = (unsigned short)c16;
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&dempty[S - 1]);
          ++cm;
        }
        long long H[16], L[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) H[j] = L[j] = 0;
        for (int c = 0; c < nchunk && ok; ++c, ++cc) {
#pragma unroll
          for (int x = 0; x < S; ++x) {
            const int d = oz_order(x);
            // the warp goes on or gives up as one (the TMEM loads below are the whole warp's)
            ok = __all_sync(0xffffffffu, mbar_wait(&dfull[d], (d == S - 1 ? cc + cm : cc) & 1, abort_flag, err, 4, wait_ns));
            if (!ok) break;
            tc_fence_after();
            if (mine) {
#pragma unroll
              for (int h = 0; h < 16; h += 8) {
                uint32_t r[8];
                tmem_ld8(tm + (uint32_t)(d * kOzTileN + h), r);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                  // d <= 2: at most 2^22 in magnitude (the leading digit is at most 64), so that adding 3 2^22 leaves the
                  // integer in the low bits; the conversion instruction has a sixteenth of that rate
                  const int v = d <= 2 ? __float_as_int(__uint_as_float(r[j]) + 12582912.0f) - 0x4B400000
                                       : __float2int_rn(__uint_as_float(r[j]));
                  if (d == 0) oz_mad<24>(H[h + j], v);
                  else if (d == 1) oz_mad<16>(H[h + j], v);
                  else if (d == 2) oz_mad<8>(H[h + j], v);
                  else if (d == 3) H[h + j] += v;
                  else if (d == 4) oz_mad<24>(L[h + j], v);
                  else if (d == 5) oz_mad<16>(L[h + j], v);
                  else if (d == 6) oz_mad<8>(L[h + j], v);
                  else L[h + j] += v;
                }
              }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&dempty[d]);
          }
        }
        if (!ok) break;
        if (!mine) continue;
        const OzProb* Q = &P;  // its fields are read again here: kept from the start they cost registers, which are short
        asm volatile("" : "+l"(Q));
        const int M = Q->M, ldc = Q->ldc, nn = Q->N - n, sel = Q->t[term].alpha & 3, alpha_neg = Q->t[term].alpha & kAlphaNeg;
        const bool accum = Q->accum != 0;
        double* C = out.out[Q->c_id] + Q->c_off + m + (int64_t)n * ldc;
        const bool neg = ((sel == kAlphaHL && out.hL < 0) || (sel == kAlphaHR && out.hR < 0)) != (alpha_neg != 0);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          double v = oz_value(H[j], L[j], neg, ea + __shfl_sync(0xffffffffu, eb, j));
          if (m < M && j < nn) {
            double* c = C + (int64_t)j * ldc;
            if (accum) {  // a reduction: other kernels may add to the same elements
              if (!((coarse[threadIdx.x - 64] >> j) & 1)) atomicAdd(c, v);
            } else {
              if (term > 0) v += *c;
              *c = v;
            }
          }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  __syncwarp();
  if (*abort_flag && warp < 2 && elect_one()) {  // a wait ran out: what is in flight into or out of this CTA's memory ends first
    if (warp == 0) {
      for (int j = *consumed; j < it; ++j)
        if (j != unarmed_it || blockIdx.x) mbar_drain(&full[j % kStages], (j / kStages) & 1);
    } else {
      umma_commit(drain);
      mbar_drain(drain, 0);
    }
  }
  __syncwarp();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
}

// ---------------------------------------------------------------- host side
void build_oz_plan(const std::vector<GemmProb>& probs, int ncta, OzPlan& P) {
  P.ops.clear(); P.chunks.clear(); P.probs.clear(); P.tiles.clear();
  P.max_redo = 0;
  P.blocks = 0;
  P.nexp = 0;
  std::map<std::tuple<int, int64_t, int, int, int, int>, int> seen;  // operands used by several products are split once
  auto operand = [&](int id, int64_t off, int rows, int K, int rs, int ks) {
    const auto key = std::make_tuple(id, off, rows, K, rs, ks);
    const auto it = seen.find(key);
    if (it != seen.end()) return it->second;
    OzOperand o{};
    o.id = id; o.off = off; o.rows = rows; o.K = K; o.rs = rs; o.ks = ks;
    o.nkb = (K + kOzBlockK - 1) / kOzBlockK;
    o.exp0 = P.nexp;
    o.blk0 = P.blocks;
    P.nexp += rows;
    P.blocks += (int64_t)((rows + kOzTileM - 1) / kOzTileM) * o.nkb;
    const int x = (int)P.ops.size();
    for (int r0 = 0; r0 < rows; r0 += 32) P.chunks.push_back(OzChunk{x, r0});
    P.ops.push_back(o);
    seen[key] = x;
    return x;
  };
  for (const GemmProb& g : probs) {
    if (g.M <= 0 || g.N <= 0) continue;
    OzProb p{};
    p.src = (int)(&g - probs.data());
    p.c_off = g.c_off; p.M = g.M; p.N = g.N; p.ldc = g.ldc; p.c_id = g.c_id; p.accum = g.accum;
    for (int i = 0; i < g.nterm; ++i) {
      const GemmTerm& t = g.t[i];
      if (t.K <= 0) continue;
      const int a = operand(t.a_id, t.a_off, g.M, t.K, t.ta ? t.lda : 1, t.ta ? 1 : t.lda);
      const int b = operand(t.b_id, t.b_off, g.N, t.K, t.tb ? 1 : t.ldb, t.tb ? t.ldb : 1);
      OzTerm& o = p.t[p.nterm++];
      o.a_blk = P.ops[a].blk0; o.b_blk = P.ops[b].blk0;
      o.a_exp = P.ops[a].exp0; o.b_exp = P.ops[b].exp0;
      o.nkb = P.ops[a].nkb;
      o.alpha = t.alpha;
      o.src = i;
    }
    if (!p.nterm) continue;
    const int x = (int)P.probs.size();
    P.probs.push_back(p);
    for (int m0 = 0; m0 < g.M; m0 += kOzTileM)
      for (int n0 = 0; n0 < g.N; n0 += kOzTileN)
        P.tiles.push_back(OzTile{x, m0, n0, std::min(kOzTileN, (g.N - n0 + 15) / 16 * 16)});
    for (int k = 0; k < p.nterm; ++k) P.max_redo += (int64_t)((g.M + 31) / 32) * ((g.N + 15) / 16);
  }
  // every tile to the CTA with the least work so far, the longest tiles first.  The work of a tile in clocks: a K block
  // takes 72 MMAs that read 4 KB of A and w / 32 KB of B from shared memory, a reading of the accumulators about 4000.
  auto work = [&](const OzTile& t) {
    double c = 2000.0;
    for (int i = 0; i < P.probs[t.prob].nterm; ++i) {
      const int nkb = P.probs[t.prob].t[i].nkb;
      c += std::max(72.0 * (32 + t.w / 4) * nkb, 4000.0 * ((nkb + kChunkBlocks - 1) / kChunkBlocks)) + 3000.0;
    }
    return c;
  };
  std::vector<std::pair<double, int>> order;
  for (int i = 0; i < (int)P.tiles.size(); ++i) order.push_back({-work(P.tiles[i]), i});
  std::stable_sort(order.begin(), order.end(), [](const auto& a, const auto& b) { return a.first < b.first; });
  P.ncta = std::min<int>((int)P.tiles.size(), ncta);
  std::priority_queue<std::pair<double, int>, std::vector<std::pair<double, int>>, std::greater<>> load;
  std::vector<std::vector<OzTile>> mine(P.ncta);
  for (int c = 0; c < P.ncta; ++c) load.push({0.0, c});
  for (const auto& o : order) {
    auto l = load.top();
    load.pop();
    mine[l.second].push_back(P.tiles[o.second]);
    load.push({l.first - o.first, l.second});
  }
  P.tiles.clear();
  P.start.assign(1, 0);
  for (const auto& m : mine) {
    P.tiles.insert(P.tiles.end(), m.begin(), m.end());
    P.start.push_back((int)P.tiles.size());
  }
}

}  // namespace imsrg

using namespace imsrg;

// Tables and operand blocks of a plan.  The blocks' padding rows hold whatever was there: a row of A or of B reaches the elements
// of that row or column alone, and those past the problem's edge are not stored.  (Padding in K is written by the split.)  Where
// the device has no room for them the list stays on k_gemm_fp64.
imsrg_status Ctx::oz_prepare(OzPlan& P, const std::vector<GemmProb>& probs, OzPool* pool) {
  if (P.state) return IMSRG_OK;
  P.state = -1;
  cudaDeviceGetAttribute(&oz_sms, cudaDevAttrMultiProcessorCount, device);
  double macs = 0.0;
  for (const GemmProb& g : probs)
    for (int i = 0; i < g.nterm; ++i)
      macs += (double)((g.M + 15) / 16 * 16) * ((g.N + 15) / 16 * 16) * g.t[i].K;
  if (macs < kOzMinMacs) {
    const std::vector<GemmTile> t = build_tiles(probs, 16, 16);
    if (t.empty()) return IMSRG_OK;
    if (cudaMalloc(&P.tables, sizeof(GemmTile) * t.size()) != cudaSuccess) {
      cudaGetLastError();
      P.tables = nullptr;
      return IMSRG_OK;
    }
    CK_TC(put(P.tables, t.data(), sizeof(GemmTile) * t.size(), "cudaMemcpy(FP64 product tiles)"));
    P.d_small = static_cast<const GemmTile*>(P.tables);
    P.nsmall = (int)t.size();
    P.state = 2;
    return IMSRG_OK;
  }
  build_oz_plan(probs, oz_sms, P);
  if (P.tiles.empty()) return IMSRG_OK;
  auto al = [](size_t b) { return (b + 255) & ~size_t(255); };
  const size_t bo = al(sizeof(OzOperand) * P.ops.size()), bc = al(sizeof(OzChunk) * P.chunks.size()),
               bp = al(sizeof(OzProb) * P.probs.size()), bt = al(sizeof(OzTile) * P.tiles.size()),
               bs = al(sizeof(int) * P.start.size()), be = al(sizeof(int) * ((size_t)P.nexp + 3)),
               br = al(sizeof(OzRedo) * (size_t)P.max_redo);
  const size_t bb = (size_t)P.blocks * (kBlockBytes + kSliceBytes);
  char *t = nullptr, *buf = nullptr;
  const bool have = pool && pool->bytes >= bb;
  if ((!have && (!room_for(bb) || cudaMalloc(&buf, bb) != cudaSuccess)) ||
      cudaMalloc(&t, bo + bc + bp + bt + bs + be + br) != cudaSuccess) {
    cudaGetLastError();
    if (buf) cudaFree(buf);
    return IMSRG_OK;
  }
  if (!pool) {
    P.own = buf;
  } else if (!have) {  // in place of a smaller one
    CK_TC(cuda(cudaStreamSynchronize(stream), "cudaStreamSynchronize(FP64 product operands)"));
    if (pool->buf) cudaFree(pool->buf);
    pool->buf = buf;
    pool->bytes = bb;
  }
  P.pool = pool;
  P.tables = t;
  std::vector<char> h(bo + bc + bp + bt + bs);
  std::memcpy(h.data(), P.ops.data(), sizeof(OzOperand) * P.ops.size());
  std::memcpy(h.data() + bo, P.chunks.data(), sizeof(OzChunk) * P.chunks.size());
  std::memcpy(h.data() + bo + bc, P.probs.data(), sizeof(OzProb) * P.probs.size());
  std::memcpy(h.data() + bo + bc + bp, P.tiles.data(), sizeof(OzTile) * P.tiles.size());
  std::memcpy(h.data() + bo + bc + bp + bt, P.start.data(), sizeof(int) * P.start.size());
  CK_TC(put(t, h.data(), h.size(), "cudaMemcpy(FP64 product plan)"));
  P.d_ops = reinterpret_cast<const OzOperand*>(t);
  P.d_chunks = reinterpret_cast<const OzChunk*>(t + bo);
  P.d_probs = reinterpret_cast<const OzProb*>(t + bo + bc);
  P.d_tiles = reinterpret_cast<const OzTile*>(t + bo + bc + bp);
  P.d_start = reinterpret_cast<const int*>(t + bo + bc + bp + bt);
  P.exps = reinterpret_cast<int*>(t + bo + bc + bp + bt + bs);
  P.flag = P.exps + P.nexp;
  P.redo = reinterpret_cast<OzRedo*>(t + bo + bc + bp + bt + bs + be);
  CK_TC(cuda(cudaFuncSetAttribute(k_oz_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem),
             "smem attr (FP64 products)"));
  P.state = 1;
  return IMSRG_OK;
}

void Ctx::oz_release(OzPlan& P) {
  if (P.own) cudaFree(P.own);
  if (P.tables) cudaFree(P.tables);
  P = OzPlan();
}

// The grouped FP64 products of a list (d_probs, d_tiles: the same list for k_gemm_fp64).
imsrg_status Ctx::gemm_fp64(OzPlan& P, const std::vector<GemmProb>& probs, const GemmProb* d_probs,
                            const GemmTile* d_tiles, int ntiles, const GemmOperands& ops, OzPool* pool) {
  if (!ntiles) return IMSRG_OK;
  CK_TC(oz_prepare(P, probs, pool));
  if (P.state == 2) {
    k_gemm_fp64_small<<<P.nsmall, 256, 0, stream>>>(d_probs, P.d_small, ops);
    return launched("k_gemm_fp64_small");
  }
  if (P.state > 0) {
    CK_TC(cuda(cudaMemsetAsync(P.flag, 0, 3 * sizeof(int), stream), "memset(FP64 product flags)"));
    char *buf = P.buf(), *mag = buf + (size_t)P.blocks * kBlockBytes;
    k_oz_split<<<(int)P.chunks.size(), 256, 0, stream>>>(P.d_ops, P.d_chunks, ops, buf, mag, P.exps, P.flag);
    CK_TC(launched("k_oz_split"));
    const int unarmed = tc_unarmed_next ? 0 : -1;  // one-shot test switch
    tc_unarmed_next = 0;
    k_oz_gemm<<<P.ncta, kThreads, kSmem, stream>>>(P.d_probs, P.d_tiles, P.d_start, ops, buf, mag, P.exps, P.flag, P.redo,
                                                   (int)P.max_redo, const_cast<int*>(wait_err), tc_wait_ns, unarmed);
    CK_TC(launched("k_oz_gemm"));
    k_gemm_fp64_rest<<<4 * oz_sms, 256, 0, stream>>>(d_probs, d_tiles, ntiles, ops, P.flag, P.redo, (int)P.max_redo);
    return launched("k_gemm_fp64_rest");
  }
  k_gemm_fp64<<<ntiles, 256, 0, stream>>>(d_probs, d_tiles, ops);
  return launched("k_gemm_fp64");
}
