// eddy_internal.h -- layouts shared by the host side (eddy_api.cu) and the
// sm_103a kernels (eddy_kernels.cu) of libeddy_gpu.
//
// Vocabulary follows the reference: a gene set of g genes, n samples split
// into class 1 (label 0, nA samples) and class 2 (label 1, nB samples); a
// "unit" is one gene set under one labelling (one permutation); each unit
// has S = nA + nB + 2 leave-one-out networks (kernel1.cu:85-88, 412-416);
// pair p enumerates (row, col), row > col, row-major lower triangle
// (main.cu:615-632).
#pragma once
#include <stdint.h>

namespace eddy {

constexpr int kFastMaxN = 32767;    // samples of a table at most that FP32 decides
constexpr int kMaxSetGenes = 512;   // genes of a set at most
constexpr int kDofSlots = 3;        // dof 1, 2, 4 (dof 0 never gives an edge)
constexpr int kMaxBdeuParents = 3;  // kernel5.cu:119-130 caps at 1 + 3
constexpr int kDivisors = 15;       // distinct q and q*r of the BDeu terms
constexpr uint32_t kUnitOk = 0;
constexpr uint32_t kUnitKeepFull = 1u;       // no room for a kept unit's outputs
constexpr uint32_t kUnitHashCollision = 2u;  // equal hash, unequal networks
constexpr uint32_t kUnitBadShape = 4u;

// Decision thresholds for one (alpha selector, dof) in chi-square units.
// True scale (the reference's FP64 chi-square): edge is certain on
// (chiB, kLo), certainly absent below chiA and above kHi; [chiA, chiB] and
// [kLo, kHi] need the exact FP64 re-evaluation.  f* are the same bounds
// moved inward by the FP32 chi-square error so they apply to FP32 values.
struct Thr {
  float chiA, chiB, kLo, kHi;   // true scale, rounded outward
  float fA, fB, fKlo, fKhi;     // FP32-value scale
};

struct SetDev {
  int g, n, W, c;         // genes, samples, 64-bit words per sample row, pairs
  int nA, nB, S;          // class sizes (fixed under permutation), networks
  int mp;                 // -mp
  int GW;                 // 32-bit words per network row bitset (ceil(g/32))
  int bonf;               // Bonferroni on
  int exact_all;          // pathological alphas: every table goes exact
  int core;               // every value of the set is -1/0/1: the tensor-core
                          // path counts 4 cells per table and derives the
                          // other 5 from the genes' class counts
  double alpha_edge, alpha_edge_prior;
  Thr thr[2][kDofSlots];  // [0] = no prior (alpha_edge), [1] = prior pairs
  const uint64_t *planes; // [g][3][W]  bit s of plane (i, a) = (x_i(s) == a-1)
  const uint64_t *planesT; // [W][g][3] the same planes word-major (follows planes)
  const uint64_t *valid;  // [W] all-sample mask
  const uint32_t *codes;  // [g][n16] states 0-3 (st_of), two bits each, 16
                          // samples a word
  int n16;                // code_words(n)
  const uint16_t *ctot;   // [c][9]  permutation-invariant full-sample table
  const uint8_t *prior;   // [c]     prior bit of pair p
  const int64_t *lg;      // [kDivisors][n+1] fixed-point lgamma(m+4/d)-lgamma(4/d)
  int lg_stride;          // n+1
  int lg_shift;           // fixed-point scale 2^lg_shift
  uint64_t salt;          // network hash salt
};

// One set of a preparation: where its arrays go, its first gene among the
// genes of all the sets and its first block of 128 pairs among theirs.
struct PrepSet {
  uint64_t *planes;  // and the word-major copy behind them
  uint32_t *codes;
  uint16_t *ctot;
  int g, c, gene0, pblk0;
};

// Decision masks of a batch, per set: [nb][c] u32 (class 1 in bits 0-9,
// class 2 in bits 16-25), followed by a bitmap per unit of the 32-pair
// chunks that hold a nonzero mask ([nb][chunk_words(c)] u32).  Between
// batches the whole buffer is zero: the decision kernels only set bits
// (and a chunk's bit with every nonzero mask in it), and the unit kernel
// clears each mask word and chunk bit it reads.
#ifdef __CUDACC__
#define EDDY_HD __host__ __device__
#else
#define EDDY_HD
#endif
// 32-bit words of a gene's packed states (two bits a sample).
EDDY_HD constexpr int code_words(int n) { return (n + 15) >> 4; }
EDDY_HD constexpr int chunk_words(int c) { return ((c + 31) / 32 + 31) / 32; }
// u32 words of one set's decision masks and chunk bitmaps for nb units
EDDY_HD constexpr size_t dmask_words(int nb, int c) {
  return (size_t)nb * (c > 0 ? c : 1) + (size_t)nb * chunk_words(c > 0 ? c : 1);
}
EDDY_HD constexpr size_t dmask_bytes(int B, int c) { return sizeof(uint32_t) * dmask_words(B, c); }

// One gene set of a batch.  A batch holds the units (labellings) of one or
// more sets of the same sample count: set k's units are [u0, u0 + nb) of
// the batch, in order.  Its decision masks and per-unit scratch are its
// slices of the batch's buffers; in the contingency GEMM its units are the
// A-operand rows [128 mb0, 128 (mb0 + mblocks)) (the rest of the last
// block is padding) and its pair groups the column groups [grp0, grp0 +
// groups) of the batch's operand Y, full-sample tables and group table, and
// its tiles are [tile0, tile0 + ntn * mblocks) of the launch.
struct BatchSet {
  SetDev sd;
  int u0, nb;          // units
  int mb0, mblocks;    // A-operand row blocks of 128 units
  int tile0, ntn;      // contingency tiles (ntn column tiles per row block)
  int grp0;            // first column group of the set in the batch's Y
  int gc0;             // first gene of the set in the batch's gene counts
  int marg_b0;         // first block of its class-count work (4-cell layout)
  int pad_;
  long long dm0;       // u32 words: its decision masks, then its chunk bitmap
  long long mg0;       // u32 words (4-cell layout): class counts [g][128
                       // mblocks], then the class-1 sizes [128 mblocks]
};
#ifdef __CUDACC__
__device__ __forceinline__ uint32_t *unit_dmask(uint32_t *dmask, const BatchSet &bs, int u) {
  return dmask + bs.dm0 + (size_t)(u - bs.u0) * bs.sd.c;
}
__device__ __forceinline__ uint32_t *unit_chunks(uint32_t *dmask, const BatchSet &bs, int u) {
  return dmask + bs.dm0 + (size_t)bs.nb * bs.sd.c + (size_t)(u - bs.u0) * chunk_words(bs.sd.c);
}
// marks the chunk of pair p in a unit's chunk bitmap
__device__ __forceinline__ void mark_chunk(uint32_t *ucb, int p) {
  atomicOr(ucb + (p >> 10), 1u << ((p >> 5) & 31));
}
#endif

// Detailed outputs of a kept unit, packed by the kernel into one buffer for
// all of a batch's (KeepMeta: where, and the counts its layout follows from):
// the likelihoods and node-summed scores of its U unique networks (class 1's,
// then class 2's), their ids, edge ranges (epn, U + 1), per-node edge
// positions (U x g) and edges (E), and the uncapped parent lists of the two
// full networks: per-node positions within each class (2 g) and edges (E2,
// the first E2a of class 1).
struct KeepMeta {
  unsigned long long off;  // 8-byte words
  int U, E, E2, E2a;
  int u, pad_;             // its unit in the batch, + 1 (0: none, the unit did
                           // not finish)
};
struct KeepLayout {
  size_t lval, dist, ids, epn, nodes, edges, lnodes, ledges, words;  // bytes; 8-byte words
};
EDDY_HD inline KeepLayout keep_layout(int g, int U, int E, int E2) {
  KeepLayout k;
  k.lval = 0;
  k.dist = k.lval + 16 * (size_t)U;
  k.ids = k.dist + 16 * (size_t)U;
  k.epn = k.ids + 4 * (size_t)U;
  k.nodes = k.epn + 4 * ((size_t)U + 1);
  k.edges = k.nodes + 4 * (size_t)U * g;
  k.lnodes = k.edges + 4 * (size_t)E;
  k.ledges = k.lnodes + 8 * (size_t)g;
  k.words = (k.ledges + 4 * (size_t)E2 + 7) / 8;
  return k;
}

// Per-batch pointers for the unit kernel.
// Byte offsets of a unit's arrays in its block's scratch and in its shared
// memory (eddy_kernels.cu), for the largest set of a batch.
struct UnitLayout {
  uint32_t phi[2], ent, ment, mdh, msc, vcan, sel, hs, dist, sig, urep, wl, vrep, ubits, htab;
  uint32_t bkey, bsc, bpos, vcnt, krow, vinf, uv, vw, xs, dc, moves, cp, ikey, isc;
  uint32_t total;
};
struct UnitSlices {
  uint32_t mA, mB, pcA, pcB, rows, cnt3, fcnt, fend, fps, fh, phs, phe, moff, nst, big, need, nobs;
  uint32_t used, chg, dmap, itk, acc, tq, fsc, ent;
  uint32_t total;
};

struct BatchDev {
  int B;                       // units in the batch
  int nsets;                   // sets in the batch
  int memo_max;                // most entries of a row whose lists are formed
                               // per subset of them (EDDY_MEMO_MAX lowers it)
  const BatchSet *sets;        // [nsets]
  const int32_t *uslot;        // [B] set of each unit (index into sets)
  const uint64_t *masks;       // [B][W] class-1 sample mask per unit
  uint32_t *dmask;             // decision masks and chunk bitmaps (per set: dm0)
  uint8_t *scratch;            // unit scratch: a slot of lay.total bytes per block of the
                               // unit kernel, then one per kept unit
  UnitLayout lay;
  UnitSlices sm;
  int words_kept;              // variants whose sample words the scratch keeps
  int blocks, threads;         // of the unit kernel
  unsigned *taken;             // units taken past the first of every block, 0 before
                               // (not read when every unit has a block)
  double *js;                  // [B]
  int32_t *U;                  // [B]
  uint32_t *status;            // [B]
  int32_t *keep_slot;          // [B] -1 or slot of detailed output
  KeepMeta *kmeta;             // [1 + slots]: entry 0's off counts the words taken,
                               // entry 1 + slot is a kept unit's
  uint64_t *kbuf;              // the kept units' packed outputs (KeepLayout)
  unsigned long long kcap;     // its 8-byte words
  unsigned long long *cycles;  // [2] SM cycles of the unit kernel's blocks, and of their
                               // normalisation and JS, added up (null: not wanted)
};

}  // namespace eddy
