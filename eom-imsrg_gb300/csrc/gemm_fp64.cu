// Grouped FP64 GEMM over a static problem/tile list on the FP64 pipe: the lists that have no digit plan
// (gemm_oz.cu), those with a non-finite operand, and the elements that the digits are too coarse for.
//
// One CTA per 64x64 output tile, 256 threads each accumulating a 4x4 sub-tile with
// DFMA; K is staged through shared memory in chunks of 16 with loads coalesced along
// whichever dimension is contiguous for the operand's transpose flag.  On GB300 the
// FP64 pipe, not HBM, bounds this kernel, so the tile only has to keep DFMA busy.
#include "gemm.h"
#include "gemm_oz.h"
#include "kernels.h"

namespace imsrg {

namespace {
constexpr int BM = 64, BN = 64, BK = 16;
constexpr int kRestParts = 16;  // warps that share the single elements of a piece
constexpr int kRestK = 32;      // K of a stage of a fuller piece

__device__ __forceinline__ double alpha_of(int code, int hL, int hR) {
  const int sel = code & 3;
  double a = (sel == kAlphaHL) ? (double)hL : (sel == kAlphaHR ? (double)hR : 1.0);
  return (code & kAlphaNeg) ? -a : a;
}

// one 64 x 64 output tile on 256 threads
__device__ __forceinline__ void gemm_tile(const GemmProb& P, const GemmTile& tile, const GemmOperands& ops, double (&As)[BK][BM + 1],
                                          double (&Bs)[BK][BN + 1]) {
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  double acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.0;

  for (int t = 0; t < P.nterm; ++t) {
    const GemmTerm& T = P.t[t];
    const double* A = ops.in[T.a_id] + T.a_off;
    const double* B = ops.in[T.b_id] + T.b_off;
    const double alpha = alpha_of(T.alpha, ops.hL, ops.hR);
    for (int k0 = 0; k0 < T.K; k0 += BK) {
      // A tile: op(A)(m, k), m in [m0, m0+64), k in [k0, k0+16)
      if (T.ta == 0) {
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          const int m = tid & 63, k = (tid >> 6) + 4 * s;
          const int gm = tile.m0 + m, gk = k0 + k;
          As[k][m] = (gm < P.M && gk < T.K) ? alpha * A[gm + (int64_t)gk * T.lda] : 0.0;
        }
      } else {
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          const int k = tid & 15, m = (tid >> 4) + 16 * s;
          const int gm = tile.m0 + m, gk = k0 + k;
          As[k][m] = (gm < P.M && gk < T.K) ? alpha * A[gk + (int64_t)gm * T.lda] : 0.0;
        }
      }
      // B tile: op(B)(k, n)
      if (T.tb == 0) {
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          const int k = tid & 15, n = (tid >> 4) + 16 * s;
          const int gn = tile.n0 + n, gk = k0 + k;
          Bs[k][n] = (gn < P.N && gk < T.K) ? B[gk + (int64_t)gn * T.ldb] : 0.0;
        }
      } else {
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          const int n = tid & 63, k = (tid >> 6) + 4 * s;
          const int gn = tile.n0 + n, gk = k0 + k;
          Bs[k][n] = (gn < P.N && gk < T.K) ? B[gn + (int64_t)gk * T.ldb] : 0.0;
        }
      }
      __syncthreads();
#pragma unroll
      for (int kk = 0; kk < BK; ++kk) {
        double a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = As[kk][tx + 16 * i];
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = Bs[kk][ty + 16 * j];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
      }
      __syncthreads();
    }
  }
  double* C = ops.out[P.c_id] + P.c_off;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gm = tile.m0 + tx + 16 * i, gn = tile.n0 + ty + 16 * j;
      if (gm < P.M && gn < P.N) {
        double* c = C + gm + (int64_t)gn * P.ldc;
        if (P.accum) atomicAdd(c, acc[i][j]);  // other kernels may add to the same elements
        else *c = acc[i][j];
      }
    }
}

}  // namespace

__global__ void __launch_bounds__(256) k_gemm_fp64(const GemmProb* __restrict__ probs,
                                                   const GemmTile* __restrict__ tiles, GemmOperands ops) {
  __shared__ double As[BK][BM + 1];
  __shared__ double Bs[BK][BN + 1];
  const GemmTile tile = tiles[blockIdx.x];
  gemm_tile(probs[tile.prob], tile, ops, As, Bs);
}

// noted elements in the rows before this lane's
__device__ __forceinline__ int elements_before(unsigned mask, int lane) {
  const int own = __popc(mask);
  int n = own;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, n, o);
    if (lane >= o) n += y;
  }
  return n - own;
}

// What the digit products of a list (gemm_oz.cu) leave: the whole list where an operand is not finite, otherwise the noted
// elements, and those alone.  A piece's few elements are shared by kRestParts warps, an element at a time with K across the
// lanes: a chain of uncoalesced reads is what one takes, and many warps wait side by side.  A fuller piece takes a CTA: its
// rows and columns come through shared memory, read along their contiguous index, and a thread has one or two of the elements,
// so that the FP64 pipe does no more than their products.  ([Omega, [Omega, H]] of an eMax 10 flow: whole columns of the
// pieces 10.7 ms, an element a lane straight from memory 11.9, so 9.6.)
__global__ void __launch_bounds__(256) k_gemm_fp64_rest(const GemmProb* __restrict__ probs, const GemmTile* __restrict__ tiles,
                                                        int ntiles, GemmOperands ops, const int* __restrict__ flags,
                                                        const OzRedo* __restrict__ redo, int max_redo) {
  __shared__ double sh[2][BK][BM + 1];
  if (flags[0]) {
    for (int x = blockIdx.x; x < ntiles; x += gridDim.x) {
      const GemmTile tile = tiles[x];
      gemm_tile(probs[tile.prob], tile, ops, sh[0], sh[1]);
    }
    return;
  }
  const int few = flags[1], many = flags[2], tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  auto put = [&](const GemmProb& P, int m, int c, double v) {
    double* at = ops.out[P.c_id] + P.c_off + m + (int64_t)c * P.ldc;
    if (P.accum) atomicAdd(at, v);
    else *at = v;
  };
  for (int64_t x = blockIdx.x * 8 + warp; x < (int64_t)few * kRestParts; x += gridDim.x * 8) {
    const OzRedo& r = redo[x / kRestParts];
    const unsigned mask = r.mask[lane];
    const int count = __reduce_add_sync(0xffffffffu, __popc(mask));
    const GemmProb& P = probs[r.prob];
    const int t0 = P.accum ? r.term : 0, t1 = P.accum ? r.term + 1 : P.nterm;
    const int before = elements_before(mask, lane);
    for (int e = (int)(x % kRestParts); e < count; e += kRestParts) {
      const int row = 31 - __clz(__ballot_sync(0xffffffffu, before <= e));
      unsigned bits = __shfl_sync(0xffffffffu, mask, row);
      for (int k = e - __shfl_sync(0xffffffffu, before, row); k > 0; --k) bits &= bits - 1u;
      const int m = r.m + row, c = r.n + __ffs((int)bits) - 1;
      double s = 0.0;
      for (int t = t0; t < t1; ++t) {
        const GemmTerm& T = P.t[t];
        const double* A = ops.in[T.a_id] + T.a_off + (T.ta ? (int64_t)m * T.lda : m);
        const double* B = ops.in[T.b_id] + T.b_off + (T.tb ? c : (int64_t)c * T.ldb);
        const int64_t sa = T.ta ? 1 : T.lda, sb = T.tb ? T.ldb : 1;
        double v = 0.0;
#pragma unroll 4
        for (int k = lane; k < T.K; k += 32) v = fma(A[k * sa], B[k * sb], v);
        s = fma(alpha_of(T.alpha, ops.hL, ops.hR), v, s);
      }
#pragma unroll
      for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) put(P, m, c, s);
    }
  }
  double(*As)[33] = reinterpret_cast<double(*)[33]>(&sh[0][0][0]);                // [K][row]
  double(*Bs)[17] = reinterpret_cast<double(*)[17]>(&sh[0][0][0] + kRestK * 33);  // [K][column]
  static_assert(kRestK * (33 + 17) <= 2 * BK * (BM + 1), "a stage fits the buffers of a tile");
  for (int x = blockIdx.x; x < many; x += gridDim.x) {
    const OzRedo& r = redo[max_redo - 1 - x];
    const unsigned mask = r.mask[lane];
    const int before = elements_before(mask, lane);
    const int count = __shfl_sync(0xffffffffu, before + __popc(mask), 31);
    int row[2], col[2];  // this thread's elements: tid and tid + 256 of the piece's
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int e = min(tid + 256 * j, count - 1);
      row[j] = 0;  // the last row with no more than e elements before it
#pragma unroll
      for (int o = 16; o; o >>= 1)
        if (__shfl_sync(0xffffffffu, before, row[j] + o) <= e) row[j] += o;
      unsigned bits = __shfl_sync(0xffffffffu, mask, row[j]);
      for (int k = e - __shfl_sync(0xffffffffu, before, row[j]); k > 0; --k) bits &= bits - 1u;
      col[j] = __ffs((int)bits) - 1;
    }
    const GemmProb& P = probs[r.prob];
    const int t0 = P.accum ? r.term : 0, t1 = P.accum ? r.term + 1 : P.nterm;
    double acc[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
    for (int t = t0; t < t1; ++t) {
      const GemmTerm& T = P.t[t];
      const double* A = ops.in[T.a_id] + T.a_off;
      const double* B = ops.in[T.b_id] + T.b_off;
      const double alpha = alpha_of(T.alpha, ops.hL, ops.hR);
      const int K = T.K, lda = T.lda, ldb = T.ldb, ta = T.ta, tb = T.tb;
      double a[4], b[2];
      auto load = [&](int k0) {  // lanes along the contiguous index of each operand
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int y = warp + 8 * i, gm = r.m + (ta ? y : lane), gk = k0 + (ta ? lane : y);
          a[i] = (gm < P.M && gk < K) ? alpha * A[ta ? gk + (int64_t)gm * lda : gm + (int64_t)gk * lda] : 0.0;
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int c = tb ? lane & 15 : warp + 8 * i, k = tb ? 2 * (warp + 8 * i) + (lane >> 4) : lane, gn = r.n + c, gk = k0 + k;
          b[i] = (gn < P.N && gk < K) ? B[tb ? gn + (int64_t)gk * ldb : gk + (int64_t)gn * ldb] : 0.0;
        }
      };
      load(0);
      for (int k0 = 0; k0 < K; k0 += kRestK) {
#pragma unroll
        for (int i = 0; i < 4; ++i) (ta ? As[lane][warp + 8 * i] : As[warp + 8 * i][lane]) = a[i];
#pragma unroll
        for (int i = 0; i < 2; ++i) (tb ? Bs[2 * (warp + 8 * i) + (lane >> 4)][lane & 15] : Bs[lane][warp + 8 * i]) = b[i];
        __syncthreads();
        if (k0 + kRestK < K) load(k0 + kRestK);
        if (tid - lane < count) {
          const int kn = min(kRestK, K - k0);
#pragma unroll 4
          for (int k = 0; k < kn; k += 2) {  // an odd K ends on zeros
            acc[0][0] = fma(As[k][row[0]], Bs[k][col[0]], acc[0][0]);
            acc[0][1] = fma(As[k + 1][row[0]], Bs[k + 1][col[0]], acc[0][1]);
          }
          if (tid - lane + 256 < count) {
#pragma unroll 4
            for (int k = 0; k < kn; k += 2) {
              acc[1][0] = fma(As[k][row[1]], Bs[k][col[1]], acc[1][0]);
              acc[1][1] = fma(As[k + 1][row[1]], Bs[k + 1][col[1]], acc[1][1]);
            }
          }
        }
        __syncthreads();
      }
    }
#pragma unroll
    for (int j = 0; j < 2; ++j)
      if (tid + 256 * j < count) put(P, r.m + row[j], r.n + col[j], acc[j][0] + acc[j][1]);
  }
}

// The same list in 16 x 16 output tiles, one thread an element: for small channels, where a 64 x 64 tile is mostly padding
// (the FP64 pipe does two FMAs a clock and SM, so a padded tile costs what a full one does) and leaves SMs idle.  The next
// 16 x 16 blocks of A and B are loaded while the present ones are multiplied.
__global__ void __launch_bounds__(256) k_gemm_fp64_small(const GemmProb* __restrict__ probs,
                                                         const GemmTile* __restrict__ tiles, GemmOperands ops) {
  __shared__ double As[2][16][17];
  __shared__ double Bs[2][16][17];
  const GemmTile tile = tiles[blockIdx.x];
  const GemmProb& P = probs[tile.prob];
  const int x = threadIdx.x & 15, y = threadIdx.x >> 4;
  const int gm = tile.m0 + x, gn = tile.n0 + y, M = P.M, N = P.N;
  double acc = 0.0;
  int buf = 0;
  for (int t = 0; t < P.nterm; ++t) {
    const GemmTerm& T = P.t[t];
    const double* A = ops.in[T.a_id] + T.a_off;
    const double* B = ops.in[T.b_id] + T.b_off;
    const double alpha = alpha_of(T.alpha, ops.hL, ops.hR);
    const int K = T.K, lda = T.lda, ldb = T.ldb;
    // lanes along the contiguous index of each operand
    auto load = [&](int k0, double& a, double& b) {
      const int am = tile.m0 + (T.ta ? y : x), ak = k0 + (T.ta ? x : y);
      a = (am < M && ak < K) ? A[T.ta ? ak + (int64_t)am * lda : am + (int64_t)ak * lda] : 0.0;
      const int bn = tile.n0 + (T.tb ? x : y), bk = k0 + (T.tb ? y : x);
      b = (bn < N && bk < K) ? B[T.tb ? bn + (int64_t)bk * ldb : bk + (int64_t)bn * ldb] : 0.0;
    };
    double a, b;
    load(0, a, b);
    for (int k0 = 0; k0 < K; k0 += 16, buf ^= 1) {
      if (T.ta) As[buf][x][y] = a; else As[buf][y][x] = a;  // [k][m]
      if (T.tb) Bs[buf][y][x] = b; else Bs[buf][x][y] = b;  // [k][n]
      __syncthreads();
      if (k0 + 16 < K) load(k0 + 16, a, b);
      const int kn = min(16, K - k0);
      double s = 0.0;
      for (int k = 0; k < kn; ++k) s = fma(As[buf][k][x], Bs[buf][k][y], s);
      acc = fma(alpha, s, acc);
    }
  }
  if (gm < M && gn < N) {
    double* c = ops.out[P.c_id] + P.c_off + gm + (int64_t)gn * P.ldc;
    if (P.accum) atomicAdd(c, acc);
    else *c = acc;
  }
}

}  // namespace imsrg
