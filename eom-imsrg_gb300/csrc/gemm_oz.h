// FP64 grouped GEMMs on the BF16 tensor cores by exact integer digits (gemm_oz.cu): plans.
#pragma once
#include <cstddef>
#include <cstdint>
#include <vector>

#include "gemm.h"

namespace imsrg {

constexpr int kOzSlices = 8;     // base-256 digits of an operand element
constexpr int kOzBlockK = 32;    // K of an operand block (64 bytes of BF16 a row)
constexpr int kOzTileM = 128;    // rows of an operand block and of an output tile
// Multiply-adds of a list, in 16 x 16 tiles, from which the digits pay: the FP64 pipe does 600 per ns, the digit kernels take
// about 30 us before they have done any (ladder / cross-coupled list at eMax 4, 5 and 8 M: 56 / 30 us by digits, 32 / 20 on
// the FP64 pipe; at eMax 5, 33 and 40 M: 74 / 43 and 86 / 74).
constexpr double kOzMinMacs = 2e7;
constexpr int kOzTileN = 64;     // widest output tile

// One operand: op(A) as rows of M (or op(B) as rows of N) over K, cut into blocks of 128 rows x 32 K, each block
// holding its eight digit slices one after the other; a ninth slice of magnitudes is kept apart, so that those of one row
// block lie one K block after the other.  Element (r, k) is at off + r * rs + k * ks of array id.
struct OzOperand {
  int64_t off;
  int id, rows, K, nkb;
  int rs, ks;       // strides of a row and of K (one of the two is 1)
  int exp0;         // first of its row exponents
  int64_t blk0;     // first block: (row block rb, K block kb) is blk0 + rb * nkb + kb
};
// rows r0 .. r0 + 31 of an operand, one CTA of the split
struct OzChunk {
  int op, r0;
};
struct OzTerm {
  int64_t a_blk, b_blk;
  int a_exp, b_exp, nkb, alpha;
  int src;  // the same term of GemmProb
};
struct OzProb {
  int64_t c_off;
  int M, N, ldc, c_id, nterm, accum;
  int src;  // the same problem of the GemmProb list
  OzTerm t[kMaxTerms];
};
// Elements of a 32 x 16 piece of an output that one term's digits are too coarse for (gemm_oz.cu): rows m + lane, columns
// n + bit.  With accum that term alone is still to be added, otherwise the whole element is still to be assigned.
struct OzRedo {
  int prob, term, m, n;  // of the GemmProb list
  unsigned short mask[32];
};
constexpr int kOzSingles = 16;  // most elements of an entry that are redone one by one
// smallest sum of |a||b| 2^-(ea+eb) that the digits are used for: they lose at most K 8.03 2^-62 (seven digit products of 2^14 at
// 2^-76, what follows them, and 2^-63 for each operand), FMAs K 2^-53 of the sum
constexpr float kOzLeast = 1.01f / 64;
// rows m0 .. m0 + 127 and columns n0 .. n0 + w - 1 of a problem (w a multiple of 16, n0 of 64)
struct OzTile {
  int prob, m0, n0, w;
};

// Operand blocks of plans that run one after the other on one stream, as large as the largest of them needs.
struct OzPool {
  char* buf = nullptr;
  size_t bytes = 0;
};

// The digit plan of a problem list; `state` 0: not prepared, 1: ready, 2: a small list, for k_gemm_fp64_small (its tiles in
// `tables`), -1: the list stays on k_gemm_fp64.
struct OzPlan {
  int state = 0;
  std::vector<OzOperand> ops;
  std::vector<OzChunk> chunks;
  std::vector<OzProb> probs;
  std::vector<OzTile> tiles;  // CTA by CTA
  std::vector<int> start;     // first tile of every CTA
  int ncta = 0;
  int64_t blocks = 0;
  int nexp = 0;
  void* tables = nullptr;
  char* own = nullptr;   // operand blocks, then their magnitude slices; in a pool where there is one
  OzPool* pool = nullptr;
  char* buf() const { return pool ? pool->buf : own; }
  int* exps = nullptr;   // row exponents, then the flags
  int* flag = nullptr;   // [0] an operand is not finite; entries of redo with [1] few and [2] many elements (from its end)
  OzRedo* redo = nullptr;
  int64_t max_redo = 0;
  const GemmTile* d_small = nullptr;
  int nsmall = 0;
  const OzOperand* d_ops = nullptr;
  const OzChunk* d_chunks = nullptr;
  const OzProb* d_probs = nullptr;
  const OzTile* d_tiles = nullptr;
  const int* d_start = nullptr;
};

// ncta: the CTAs of the persistent kernel
void build_oz_plan(const std::vector<GemmProb>& probs, int ncta, OzPlan& P);

}  // namespace imsrg
