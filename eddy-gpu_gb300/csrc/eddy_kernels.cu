// eddy_kernels.cu -- sm_103a kernels of the EDDY hot path.
//
//   k_planes / k_ctot   set preparation: per-gene state bit-planes over the
//                       samples and the permutation-invariant full-sample
//                       3x3 table of every pair.
//   k_counter_masks     counter-based labelling (Philox-4x32-10) -> class-1
//                       sample masks, a warp per unit.
//   k_pairs             contingency counts of class 1 for every (unit, pair)
//                       (class 2 = full table - class 1), and the 10-bit
//                       leave-one-out decision mask per class: the reference's
//                       run2/run2Scalable (kernel1.cu:389-477) over all S
//                       networks collapsed to <= 10 distinct tables per class.
//   k_units             a block per unit at a time: full networks, flip lists, the
//                       capped parent lists that left-out samples change
//                       (kernel2.cu:114-142, kernel3.cu:134-165), network
//                       hashing and first-occurrence dedup with exact
//                       verification (kernel4.cu:72-84, main.cu:1060-1121),
//                       BDeu over the unique networks in fixed point
//                       (kernel5.cu:237-257), normalisation and JS
//                       (main.cu:1293-1428).
//   k_pack              the networks of the units kept for output files.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <climits>

#include "eddy_device.cuh"
#include "eddy_kernels.h"

namespace eddy {

// ----------------------------------------------------------- set prep
// The sets of a batch are prepared together, two launches however many
// there are (a launch per set and array was 85% launch overhead: 2341 sets
// of 5-300 genes x 1000 samples took 36 ms in them, now 1.4 ms).

// last k of [0, n) whose first (nondecreasing, first(0) = 0) is not past i
template <class First>
__device__ __forceinline__ int owner_of(int n, int i, First first) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (first(mid) <= i) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// the low 16 bits of x, one to every second bit
__device__ __forceinline__ uint32_t spread16(uint32_t x) {
  x &= 0xFFFFu;
  x = (x | (x << 8)) & 0x00FF00FFu;
  x = (x | (x << 4)) & 0x0F0F0F0Fu;
  x = (x | (x << 2)) & 0x33333333u;
  return (x | (x << 1)) & 0x55555555u;
}

// One warp per gene of a set: its state bit-planes (gene-major and
// word-major) and packed states, 64 samples at a time by ballots over
// coalesced byte loads, four words' loads in flight.  rows: the row of vals
// of each gene (null: the gene's position).  Warp 0 also writes the all-sample
// mask `valid`.
__global__ void __launch_bounds__(128) k_planes(const PrepSet *__restrict__ sets, int ns, int genes,
                                                const int8_t *__restrict__ vals,
                                                const int32_t *__restrict__ rows, int n, int W,
                                                uint64_t *valid) {
  const int wi = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (wi >= genes) return;
  const PrepSet &ps = sets[owner_of(ns, wi, [&](int k) { return sets[k].gene0; })];
  const int i = wi - ps.gene0, g = ps.g, n16 = code_words(n);
  const int8_t *row = vals + (size_t)(rows ? rows[wi] : wi) * n;
  uint64_t *planesT = ps.planes + (size_t)g * 3 * W;
  if (wi == 0)
    for (int w = lane; w < W; w += 32) valid[w] = n - 64 * w >= 64 ? ~0ull : (1ull << (n - 64 * w)) - 1ull;
  constexpr int kWords = 4;
  for (int w0 = 0; w0 < W; w0 += kWords) {
    int8_t x[2 * kWords];
#pragma unroll
    for (int q = 0; q < 2 * kWords; q++) {
      const int s = 64 * w0 + 32 * q + lane;
      x[q] = s < n ? row[s] : (int8_t)2;
    }
#pragma unroll
    for (int q = 0; q < kWords; q++) {
      const int w = w0 + q;
      if (w >= W) break;
      uint32_t b0[2], b1[2];  // bits of the states (0-3)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int st = st_of(x[2 * q + h]);
        b0[h] = __ballot_sync(0xffffffffu, st & 1);
        b1[h] = __ballot_sync(0xffffffffu, st & 2);
      }
      const uint64_t lo = b0[0] | ((uint64_t)b0[1] << 32), hi = b1[0] | ((uint64_t)b1[1] << 32);
      // lanes 0-2: the planes; 4-6: their word-major copy; 8-11: the codes
      const int a = lane & 3;
      const uint64_t pl = a == 0 ? ~lo & ~hi : a == 1 ? lo & ~hi : hi & ~lo;
      if (lane < 3) ps.planes[((size_t)i * 3 + a) * W + w] = pl;
      else if (lane >= 4 && lane < 7) planesT[(size_t)w * g * 3 + (size_t)i * 3 + a] = pl;
      else if (lane >= 8 && lane < 12 && 4 * w + a < n16)
        ps.codes[(size_t)i * n16 + 4 * w + a] =
            spread16((uint32_t)(lo >> (16 * a))) | (spread16((uint32_t)(hi >> (16 * a))) << 1);
    }
  }
}

// The permutation-invariant full-sample 3x3 table of every pair, blocks of
// 128 pairs of a set.
__global__ void __launch_bounds__(128) k_ctot(const PrepSet *__restrict__ sets, int ns, int W) {
  const PrepSet &ps =
      sets[owner_of(ns, (int)blockIdx.x, [&](int k) { return sets[k].pblk0; })];
  const int p = ((int)blockIdx.x - ps.pblk0) * 128 + threadIdx.x;
  if (p >= ps.c) return;
  int row, col;
  pair_rc(p, row, col);
  const uint64_t *T = ps.planes + (size_t)ps.g * 3 * W;  // word-major: consecutive columns
  int cnt[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  for (int w = 0; w < W; w++, T += 3 * ps.g) {
    const uint64_t r0 = T[3 * row], r1 = T[3 * row + 1], r2 = T[3 * row + 2];
    const uint64_t c0 = T[3 * col], c1 = T[3 * col + 1], c2 = T[3 * col + 2];
    cnt[0] += __popcll(r0 & c0); cnt[1] += __popcll(r0 & c1); cnt[2] += __popcll(r0 & c2);
    cnt[3] += __popcll(r1 & c0); cnt[4] += __popcll(r1 & c1); cnt[5] += __popcll(r1 & c2);
    cnt[6] += __popcll(r2 & c0); cnt[7] += __popcll(r2 & c1); cnt[8] += __popcll(r2 & c2);
  }
  for (int k = 0; k < 9; k++) ps.ctot[(size_t)p * 9 + k] = (uint16_t)cnt[k];
}

// ---------------------------------------------------- counter labelling
__device__ __forceinline__ void philox10(uint32_t c[4], uint32_t k0, uint32_t k1) {
  for (int r = 0; r < 10; r++) {
    uint32_t hi0 = __umulhi(0xD2511F53u, c[0]), lo0 = 0xD2511F53u * c[0];
    uint32_t hi1 = __umulhi(0xCD9E8D57u, c[2]), lo1 = 0xCD9E8D57u * c[2];
    uint32_t n0 = hi1 ^ c[1] ^ k0, n2 = hi0 ^ c[3] ^ k1;
    c[0] = n0; c[1] = lo1; c[2] = n2; c[3] = lo0;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
}

// A warp per unit.  key(s) = word s mod 4 of Philox(ctr = (s / 4, perm, set,
// 0), key = seed); the nA samples with the smallest (key, s) are class 1.
// Selection: a histogram of the keys' top 8 bits finds the bin that holds the
// nA-th smallest key; the samples of that bin (about n / 256 of them) are
// ranked by (key, s) against each other, which gives the last one in, (T,
// sT); sample s is in when (key, s) <= (T, sT).  The same set as sorting the
// pairs and taking the first nA.  (A block of 128 threads per unit, 2048
// bins, waited at its barriers: 4.5 ms for 339000 units of 1000 samples, now
// 0.9 ms.)
constexpr int kCmWarps = 4, kCmBins = 256, kCmShift = 24;
constexpr int kCmMaxSamples = 4096;  // (more: the labellings come from the host)
__host__ __device__ constexpr int cm_words(int n) { return ((n + 3) & ~3) + kCmBins; }  // a warp's shared memory
__global__ void __launch_bounds__(32 * kCmWarps) k_counter_masks(int n, int nA, int W, uint64_t seed,
                                                                 const int32_t *unit_set,
                                                                 const int32_t *unit_perm,
                                                                 const uint64_t *mask0,
                                                                 uint64_t *masks, int B) {
  extern __shared__ __align__(16) uint32_t cm_smem[];
  const int lane = threadIdx.x & 31, u = blockIdx.x * kCmWarps + (threadIdx.x >> 5);
  if (u >= B) return;
  // the unit's keys, then the histogram, then (in its place) the bin's samples
  uint32_t *key = cm_smem + (threadIdx.x >> 5) * cm_words(n), *hist = key + ((n + 3) & ~3);
  uint16_t *cand = reinterpret_cast<uint16_t *>(hist);
  const int perm = unit_perm[u];
  uint64_t *out = masks + (size_t)u * W;
  if (perm == 0) {
    for (int w = lane; w < W; w += 32) out[w] = mask0[w];
    return;
  }
#pragma unroll
  for (int i = 0; i < kCmBins / 32; i++) hist[32 * i + lane] = 0u;
  __syncwarp();
  const uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32), set = (uint32_t)unit_set[u];
  // one Philox call gives the keys of four samples
  for (int s4 = lane; 4 * s4 < n; s4 += 32) {
    uint32_t c[4] = {(uint32_t)s4, (uint32_t)perm, set, 0u};
    philox10(c, k0, k1);
    *reinterpret_cast<uint4 *>(key + 4 * s4) = make_uint4(c[0], c[1], c[2], c[3]);
#pragma unroll
    for (int j = 0; j < 4; j++)
      if (4 * s4 + j < n) atomicAdd(&hist[c[j] >> kCmShift], 1u);
  }
  __syncwarp();
  // the bin of the nA-th smallest key, and the samples it has to give: a lane
  // sums eight bins, then a scan of the sums
  constexpr int kPer = kCmBins / 32;
  int h[kPer], loc = 0;
#pragma unroll
  for (int j = 0; j < kPer; j++) loc += h[j] = (int)hist[lane * kPer + j];
  int before = loc;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, before, o);
    if (lane >= o) before += y;
  }
  before -= loc;
  __syncwarp();
  const int owner = 31 - __clz(__ballot_sync(0xffffffffu, before < nA && nA <= before + loc));
  int bin = 0, need = 0;
#pragma unroll
  for (int j = 0; j < kPer; j++) {
    if (before < nA && nA <= before + h[j]) {
      bin = lane * kPer + j;
      need = nA - before;
    }
    before += h[j];
  }
  bin = __shfl_sync(0xffffffffu, bin, owner);
  need = __shfl_sync(0xffffffffu, need, owner);
  // the bin's samples in order, as many as the histogram's place holds
  constexpr int kCand = 2 * kCmBins;
  int cnt = 0;
  for (int s0 = 0; s0 < n; s0 += 32) {
    const bool in = s0 + lane < n && (int)(key[s0 + lane] >> kCmShift) == bin;
    const unsigned bal = __ballot_sync(0xffffffffu, in);
    const int at = cnt + __popc(bal & ((1u << lane) - 1u));
    if (in && at < kCand) cand[at] = (uint16_t)(s0 + lane);
    cnt += __popc(bal);
  }
  __syncwarp();
  // rank of each of them by (key, s): the one of rank need - 1 is the last in
  const bool listed = cnt <= kCand;
  uint32_t T = 0u;
  int sT = -1;
  for (int c = lane; c < (listed ? cnt : n); c += 32) {
    const int s = listed ? cand[c] : c;
    const uint32_t k = key[s];
    int rank = 0;
    if (!listed && (int)(k >> kCmShift) != bin) continue;
    for (int d = 0; d < (listed ? cnt : n); d++) {
      const int t = listed ? cand[d] : d;
      const uint32_t kt = key[t];
      rank += ((int)(kt >> kCmShift) == bin && (kt < k || (kt == k && t < s))) ? 1 : 0;
    }
    if (rank == need - 1) {
      T = k;
      sT = s;
    }
  }
  const int last = 31 - __clz(__ballot_sync(0xffffffffu, sT >= 0));
  T = __shfl_sync(0xffffffffu, T, last);
  sT = __shfl_sync(0xffffffffu, sT, last);
  uint32_t *out32 = reinterpret_cast<uint32_t *>(out);
  uint32_t mine = 0u;
  for (int w = 0; w < 2 * W; w++) {
    const int s = 32 * w + lane;
    const uint32_t k = s < n ? key[s] : 0u;
    const uint32_t bal = __ballot_sync(0xffffffffu, s < n && (k < T || (k == T && s <= sT)));
    if (lane == (w & 31)) mine = bal;
    if ((w & 31) == 31 || w == 2 * W - 1)
      if (lane <= (w & 31)) out32[(w & ~31) + lane] = mine;
  }
}

// ------------------------------------------------------------ k_pairs
// Contingency counts by popcounts and the ten decisions of both classes,
// for batches of few units per set (and as the second path of any batch):
// no operand is built, and a unit costs only its own pairs where the
// contraction computes 128 rows whatever the batch holds.
//
// A block takes a 32 x 32 tile of one unit's pairs (rows above columns), a
// lane one column gene, a warp four row genes, so a lane's three plane words
// of 64 samples serve four pairs; the masked row planes are staged in shared
// memory kPairWords words at a time.  Where the tiles are too few for the GPU
// a block takes half or a quarter of one (launch_pairs).  A set without missing values counts
// cells (-1,-1), (-1,0), (0,-1), (0,0) and derives the other five from the
// genes' class-1 counts.  Bound by POPC (32 a word and lane in that case, 72
// otherwise).
constexpr int kPairTile = 32, kPairWords = 16, kPairWarps = 8;

// The tables of a tile that the packed forms leave: their decisions are shared
// out over the block, the FP32 ones a lane per table, the exact FP64 ones a
// lane per decision.  (With each lane deciding its own tables a warp waited for
// ten exact decisions one after the other of the few lanes that had any: every
// decision in FP64, 8 genes x 40 samples, 700 units 3.19 ms a call, now 0.50; 60
// x 400 at alpha 1e-9, where 5% of the tables needs them, 100 units 1.53, now
// 0.19.)
constexpr int kTileThreads = 32 * kPairWarps, kTileStep = 2 * kTileThreads;
struct TileGeneral {
  // counts (nine of 16 bits), then prior | class << 1 in the fifth word's high
  // half, and the pair
  uint32_t table[2 * kTileStep][6];
  // of kTileThreads of them at a time: decisions known so far, the bits that
  // share the full table's, and what is left, item * 10 + slot (0: the full
  // table)
  uint32_t bits[kTileThreads];
  uint16_t shared0[kTileThreads], exact[10 * kTileThreads];
};
__device__ __forceinline__ void tile_table(const uint32_t *w, int *t) {
#pragma unroll
  for (int k = 0; k < 9; k++) t[k] = (int)((w[k >> 1] >> (16 * (k & 1))) & 0xFFFFu);
}
// The masks of the n tables listed in G into the unit's (*left: 0 before and
// after).  Returns the exact evaluations of this thread, and in the high half
// the tables a filter settled.
__device__ __noinline__ uint64_t tile_general(TileGeneral &G, int n, int *left, const SetDev &sd,
                                              uint32_t *udm, uint32_t *ucb) {
  unsigned nexact = 0, nfilt = 0;
  const int tid = threadIdx.x;
#pragma unroll 1
  for (int k0 = 0; k0 < n; k0 += kTileThreads) {
    const uint32_t *w = G.table[k0 + tid];
    if (k0 + tid < n) {
      int t[9];
      tile_table(w, t);
      const int prior = (w[4] >> 16) & 1;
      TabInfo ti;
      table_info(t, ti);
      uint32_t bits = 0u, shared0 = 1u;
      if (quick_zero(ti, prior, sd)) {
        nfilt++;
      } else {
        const int bit0 = fast_decision(ti, prior, sd);
        if (loo_safe(ti, prior, sd)) {
          shared0 = 0x3FFu;
          nfilt++;
        } else {
#pragma unroll
          for (int cell = 0; cell < 9; cell++) {
            if (t[cell] == 0) {
              shared0 |= 2u << cell;
              continue;
            }
            t[cell]--;
            TabInfo tj;
            table_info(t, tj);
            t[cell]++;
            const int bit = fast_decision(tj, prior, sd);
            if (bit == 2) G.exact[atomicAdd(left, 1)] = (uint16_t)(10 * tid + 1 + cell);
            else bits |= (uint32_t)bit << (1 + cell);
          }
        }
        if (bit0 == 2) G.exact[atomicAdd(left, 1)] = (uint16_t)(10 * tid);
        else if (bit0) bits |= shared0;
      }
      G.bits[tid] = bits;
      G.shared0[tid] = (uint16_t)shared0;
    }
    __syncthreads();
    const int ne = *left;
    for (int e = tid; e < ne; e += kTileThreads) {
      const int k = G.exact[e] / 10, slot = G.exact[e] - 10 * k;
      const uint32_t *x = G.table[k0 + k];
      int t[9];
      tile_table(x, t);
#pragma unroll
      for (int c = 0; c < 9; c++) t[c] -= slot == 1 + c ? 1 : 0;
      nexact++;
      if (exact_decision(t[0], t[1], t[2], t[3], t[4], t[5], t[6], t[7], t[8], (x[4] >> 16) & 1, sd))
        atomicOr(&G.bits[k], slot ? 1u << slot : (uint32_t)G.shared0[k]);
    }
    __syncthreads();
    if (tid == 0) *left = 0;
    if (k0 + tid < n && G.bits[tid]) {
      atomicOr(&udm[w[5]], G.bits[tid] << ((w[4] >> 17) & 1 ? 16 : 0));
      mark_chunk(ucb, (int)w[5]);
    }
    __syncthreads();
  }
  return (uint64_t)nexact | ((uint64_t)nfilt << 32);
}

template <bool kCore, int kPairRows>
__device__ __forceinline__ void pairs_tile(const BatchSet &bs, int u, int row0, int tc, int W,
                                           const uint64_t *__restrict__ mask, uint32_t *dmask,
                                           TileGeneral &G, int *listed, unsigned &nexact,
                                           unsigned &nfilt, unsigned &ntab) {
  constexpr int kSt = kCore ? 2 : 3, kCells = kSt * kSt, kRows = kPairWarps * kPairRows;
  // the masked row planes (+ 1: fewer bank conflicts), then in their place the
  // tables the packed forms leave
  using Rows = uint64_t[kRows][kSt][kPairWords + 1];
  static_assert(sizeof(Rows) <= sizeof(TileGeneral), "room");
  Rows &rowp = *reinterpret_cast<Rows *>(&G);
  int &items = listed[0], &left = listed[1];  // tables; their exact decisions
  __shared__ int n1;  // the unit's class-1 samples
  __shared__ uint64_t mw[kPairWords];
  __shared__ int marg[2][kPairTile][2];  // class-1 counts of states -1, 0: rows, columns
  const SetDev &sd = bs.sd;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = sd.g;
  const int col = tc * kPairTile + lane;
  const bool cl = col < g;
  int cnt[kPairRows][kCells];
  int cm[2] = {0, 0}, rm[2] = {0, 0}, nc = 0;
#pragma unroll
  for (int i = 0; i < kPairRows; i++)
#pragma unroll
    for (int k = 0; k < kCells; k++) cnt[i][k] = 0;
  for (int w0 = 0; w0 < W; w0 += kPairWords) {
    const int nw = min(kPairWords, W - w0);
    __syncthreads();
    if (threadIdx.x < nw) mw[threadIdx.x] = mask[w0 + threadIdx.x];
    // the masked row planes, word by word from the gene-major planes
    for (int i = threadIdx.x; i < kRows * kSt * nw; i += blockDim.x) {
      const int w = i % nw, ra = i / nw, r = ra / kSt, a = ra % kSt, row = row0 + r;
      rowp[r][a][w] = row < g ? sd.planes[((size_t)row * 3 + a) * W + w0 + w] & mask[w0 + w] : 0ull;
    }
    __syncthreads();
    for (int w = 0; w < nw; w++) {
      uint64_t c[kSt];
#pragma unroll
      for (int b = 0; b < kSt; b++)
        c[b] = cl ? sd.planesT[(size_t)(w0 + w) * 3 * g + 3 * col + b] : 0ull;
      if (kCore) {
        // the genes' counts: columns by warp 0, rows by warp 1 (and the
        // class size by warp 2)
        if (warp == 0) {
          const uint64_t m = mw[w];
          cm[0] += __popcll(c[0] & m);
          cm[1] += __popcll(c[1] & m);
        } else if (warp == 1) {
          rm[0] += __popcll(rowp[lane % kRows][0][w]);
          rm[1] += __popcll(rowp[lane % kRows][1][w]);
        } else if (warp == 2) {
          nc += __popcll(mw[w]);
        }
      }
#pragma unroll
      for (int i = 0; i < kPairRows; i++)
#pragma unroll
        for (int a = 0; a < kSt; a++) {
          const uint64_t x = rowp[warp * kPairRows + i][a][w];
#pragma unroll
          for (int b = 0; b < kSt; b++) cnt[i][a * kSt + b] += __popcll(x & c[b]);
        }
    }
  }
  if (kCore) {
    if (warp == 0) {
      marg[1][lane][0] = cm[0];
      marg[1][lane][1] = cm[1];
    } else if (warp == 1) {
      marg[0][lane][0] = rm[0];
      marg[0][lane][1] = rm[1];
    } else if (warp == 2 && lane == 0) {
      n1 = nc;
    }
  }
  if (threadIdx.x == 0) items = left = 0;
  __syncthreads();
  uint32_t *udm = unit_dmask(dmask, bs, u), *ucb = unit_chunks(dmask, bs, u);
#pragma unroll
  for (int i = 0; i < kPairRows; i++) {
    const int r = warp * kPairRows + i, row = row0 + r;
    const bool live = row < g && col < row;
    const int p = live ? row * (row - 1) / 2 + col : 0;
    int t[2][9], prior = 0;
    uint32_t m = 0u;
    unsigned unc = 0u;
    if (__any_sync(0xffffffffu, live)) {
      if (kCore) {
        t[0][0] = cnt[i][0], t[0][1] = cnt[i][1], t[0][3] = cnt[i][2], t[0][4] = cnt[i][3];
        t[0][2] = marg[0][r][0] - t[0][0] - t[0][1];
        t[0][5] = marg[0][r][1] - t[0][3] - t[0][4];
        t[0][6] = marg[1][lane][0] - t[0][0] - t[0][3];
        t[0][7] = marg[1][lane][1] - t[0][1] - t[0][4];
        t[0][8] = n1 - marg[0][r][0] - marg[0][r][1] - t[0][6] - t[0][7];
      } else {
#pragma unroll
        for (int k = 0; k < 9; k++) t[0][k] = cnt[i][k];
      }
      const uint16_t *ct = sd.ctot + (size_t)p * 9;
#pragma unroll
      for (int k = 0; k < 9; k++) t[1][k] = (int)ct[k] - t[0][k];
      prior = sd.prior[p] ? 1 : 0;
      const Thr &T = sd.thr[prior][2];
      f32x2 o[9];
#pragma unroll
      for (int k = 0; k < 9; k++) o[k] = f2_pack((float)t[0][k], (float)t[1][k]);
      const unsigned want = live ? ~quick_zero_f2(o, sd.exact_all ? -1.f : T.chiA) & 3u : 0u;
      if (live) {
        nfilt += 2 - __popc(want);
        ntab += 2;
      }
      if (__any_sync(0xffffffffu, want)) {
        f32x2 R[3], C[3];
#pragma unroll
        for (int a = 0; a < 3; a++) {
          R[a] = f2_add(f2_add(o[3 * a], o[3 * a + 1]), o[3 * a + 2]);
          C[a] = f2_add(f2_add(o[a], o[3 + a]), o[6 + a]);
        }
        unc = want & loo_f2(o, R, C, f2_add(f2_add(R[0], R[1]), R[2]), T, sd.exact_all != 0, m);
        m = (want & 1u ? m & 0x3FFu : 0u) | (want & 2u ? m & 0x3FF0000u : 0u);
#pragma unroll
        for (int cls = 0; cls < 2; cls++) {
          const uint32_t mm = (m >> (16 * cls)) & 0x3FFu;
          // (the ten tables agree: settled at once)
          nfilt += (((want & ~unc) >> cls) & 1u) && (mm == 0u || mm == 0x3FFu);
        }
      }
    }
    // (masks that are zero already are: the buffer starts at zero)
    if (m) udm[p] = m;
    const unsigned nz = __ballot_sync(0xffffffffu, m != 0u);
    if (nz) {
      // the row's 32 pairs lie in two chunks at most
      const int p0 = row * (row - 1) / 2 + tc * kPairTile, cut = 32 - (p0 & 31);
      const unsigned first = cut >= 32 ? ~0u : (1u << cut) - 1u;
      if (lane == 0 && (nz & first)) mark_chunk(ucb, p0);
      if (lane == 1 && (nz & ~first)) mark_chunk(ucb, p0 + cut);
    }
    // what is left goes into the list, which has room for two steps
    const unsigned b0 = __ballot_sync(0xffffffffu, unc & 1u);
    const unsigned b1 = __ballot_sync(0xffffffffu, (unc & 2u) != 0u), below = (1u << lane) - 1u;
    const int cnt = __popc(b0) + __popc(b1);
    int at = 0;
    if (cnt) {
      if (lane == 0) at = atomicAdd(&items, cnt);
      at = __shfl_sync(0xffffffffu, at, 0);
#pragma unroll
      for (int cls = 0; cls < 2; cls++)
        if ((unc >> cls) & 1u) {
          uint32_t *w = G.table[at + (cls ? __popc(b0) + __popc(b1 & below) : __popc(b0 & below))];
#pragma unroll
          for (int k = 0; k < 4; k++)
            w[k] = (uint32_t)t[cls][2 * k] | ((uint32_t)t[cls][2 * k + 1] << 16);
          w[4] = (uint32_t)t[cls][8] | ((uint32_t)(prior | (cls << 1)) << 16);
          w[5] = (uint32_t)p;
        }
    }
    // (a barrier: the masks stored above are there before bits are added)
    if (!__syncthreads_or(i == kPairRows - 1 ? cnt != 0 || items > 0 : at + cnt > kTileStep)) continue;
    const uint64_t c = tile_general(G, items, &left, sd, udm, ucb);
    nexact += (unsigned)c;
    nfilt += (unsigned)(c >> 32);
    if (i < kPairRows - 1) {
      if (threadIdx.x == 0) items = 0;
      __syncthreads();
    }
  }
}

template <int kPairRows>
__global__ void __launch_bounds__(32 * kPairWarps, 2) k_pairs(const BatchSet *__restrict__ sets,
                                                           const int32_t *__restrict__ uslot,
                                                           const uint64_t *masks, int W,
                                                           uint32_t *dmask,
                                                           unsigned long long *stats) {
  const int u = blockIdx.y;
  const BatchSet &bs = sets[uslot[u]];
  // tile of the lower triangle, row by row
  int tr = (int)((sqrtf(8.f * (float)blockIdx.x + 1.f) - 1.f) * 0.5f);
  while (tr * (tr + 1) / 2 > (int)blockIdx.x) tr--;
  while ((tr + 1) * (tr + 2) / 2 <= (int)blockIdx.x) tr++;
  const int tc = (int)blockIdx.x - tr * (tr + 1) / 2;
  const int row0 = tr * kPairTile + (int)blockIdx.z * kPairWarps * kPairRows;
  if (row0 >= bs.sd.g) return;
  __shared__ __align__(16) TileGeneral G;
  __shared__ int listed[2];
  unsigned nexact = 0, nfilt = 0, ntab = 0;
  const uint64_t *mask = masks + (size_t)u * W;
  if (bs.sd.core) pairs_tile<true, kPairRows>(bs, u, row0, tc, W, mask, dmask, G, listed, nexact, nfilt, ntab);
  else pairs_tile<false, kPairRows>(bs, u, row0, tc, W, mask, dmask, G, listed, nexact, nfilt, ntab);
  if (stats) {
    // warp-aggregated counters
    for (int o = 16; o > 0; o >>= 1) {
      nexact += __shfl_down_sync(0xffffffffu, nexact, o);
      nfilt += __shfl_down_sync(0xffffffffu, nfilt, o);
      ntab += __shfl_down_sync(0xffffffffu, ntab, o);
    }
    if ((threadIdx.x & 31) == 0) {
      unsigned long long *sk = stats + 4 * (size_t)uslot[u];  // the set's row
      if (nexact) atomicAdd(&sk[0], (unsigned long long)nexact);
      if (ntab) atomicAdd(&sk[1], (unsigned long long)ntab);
      if (nfilt) atomicAdd(&sk[2], (unsigned long long)nfilt);
    }
  }
}

// ------------------------------------------------------------ k_units
// Kept flip entries of the two full networks' rows, one uint2 each:
//   x = column (9 bits) | node << 9
//   y = cells: bit 4a + b set when the entry fires for a left-out sample of
//       states a (node) and b (column), no bit for a missing value (3)
__device__ __forceinline__ uint32_t cells16(uint32_t fb) {
  return (fb & 7u) | (((fb >> 3) & 7u) << 4) | (((fb >> 6) & 7u) << 8);
}
// A row with at most E <= BatchDev::memo_max kept entries (and no more subsets of them
// than its class has samples) is a memo row: its capped list under every
// non-empty subset of its entries (a variant) is formed once per unit.  The
// other rows' lists are formed per left-out sample.  E is lowered until the
// unit's variants fit unit_variants(g), which rows of up to five entries
// always do, and the room for their sample words (BatchDev::words_kept).
__host__ __device__ constexpr int unit_variants(int g) { return 62 * g + 64; }
// slots of the table of the lists formed per sample (in the unit's scratch)
__host__ __device__ constexpr int big_slots(int g) {
  int s = 256;
  while (s < 16 * g && s < 8192) s <<= 1;
  return s;
}
// network table: slots held in shared memory (larger ones in the scratch)
constexpr int kSmSlots = 4096;
// genes of a set of c pairs (c = g (g - 1) / 2, so 1 + 8 c = (2 g - 1)^2)
static int genes_of_pairs(int c) {
  int r = (int)sqrt((double)(1 + 8 * (long long)c));
  while ((long long)r * r > 1 + 8 * (long long)c) r--;
  while ((long long)(r + 1) * (r + 1) <= 1 + 8 * (long long)c) r++;
  return (r + 1) / 2;
}

static UnitLayout unit_layout(int c, int S, int words_kept) {
  UnitLayout L;
  size_t o = 0;
  auto take = [&](size_t bytes) {
    const size_t at = o;
    o = (o + bytes + 255) & ~(size_t)255;
    return (uint32_t)at;
  };
  const size_t cc = c > 0 ? c : 1;
  const int g = genes_of_pairs(c);
  const size_t nv = unit_variants(g), nb = big_slots(g);
  L.dist = take(sizeof(int64_t) * 2 * (size_t)S);
  L.hs = take(sizeof(uint64_t) * (size_t)S);    // per network: hash, ~0 = its class's full one
  L.sig = take(sizeof(int32_t) * (size_t)S);    // class-1 samples then class-2 samples
  L.urep = take(sizeof(int32_t) * (size_t)S);   // unique networks in order
  L.wl = take(sizeof(int32_t) * (size_t)S);     // networks merged by hash, to verify
  L.vrep = take(sizeof(int32_t) * (size_t)S);   // and what they were merged with
  L.ubits = take(sizeof(uint32_t) * (size_t)((S + 31) / 32));
  int ht = 1;
  while (ht < 2 * (S + 2)) ht <<= 1;
  L.htab = take(ht > kSmSlots ? sizeof(int32_t) * (size_t)ht : 0);
  L.ment = take(sizeof(uint64_t) * nv);         // variants: key (or ~0: the full list)
  L.mdh = take(sizeof(uint64_t) * nv);          // hash less the full list's
  L.msc = take(2 * sizeof(int64_t) * nv);       // scores less the full list's, both classes
  L.vcan = take(sizeof(uint16_t) * nv);         // a variant with the same key, scored for it
  L.sel = take(sizeof(uint16_t) * nv);          // the variants to score
  L.vcnt = take(sizeof(uint16_t) * nv);         // their list lengths
  // a kept unit's rows, entry ranges (k_pack reads them)
  L.krow = take(sizeof(uint32_t) * (2 * (size_t)g * ((g + 31) / 32) + 4 * (size_t)g));
  L.vinf = take(sizeof(uint32_t) * nv);         // variants: entries and subset (variant_info)
  L.uv = take(sizeof(uint2) * nv);              // the used ones: number, info
  L.vw = take(sizeof(uint32_t) * (size_t)words_kept * class_words(S - 2));  // their words
  L.xs = take(2 * sizeof(int64_t) * (size_t)S); // per network: scores less the full one's
  L.dc = take(sizeof(int32_t) * (size_t)S);     // and its lists' edges (kept units)
  L.moves = take(sizeof(uint32_t) * 32 * ((size_t)(S - 2 + 63) / 64));  // pack_classes' masks
  L.cp = take(sizeof(uint2) * (size_t)g * ((S - 2) / 32 + 4));  // both classes' ClassPlanes
  L.bkey = take(sizeof(uint64_t) * nb);
  L.bsc = take(2 * sizeof(int64_t) * nb);
  L.bpos = take(sizeof(int32_t) * nb);
  L.ikey = take(sizeof(uint64_t) * (2 * g + nv + nb));    // the keys to score
  L.isc = take(2 * sizeof(int64_t) * (2 * g + nv + nb));  // and their scores
  for (int k = 0; k < 2; k++) L.phi[k] = take(sizeof(uint32_t) * cc);
  L.ent = take(2 * sizeof(uint2) * cc);
  L.total = (uint32_t)o;
  return L;
}

// Variants whose sample words take at most `bytes` of a unit's scratch.
static int words_kept(int c, int S, size_t bytes) {
  return (int)std::min<size_t>(unit_variants(genes_of_pairs(c)), bytes / (4 * class_words(S - 2)));
}

size_t unit_scratch_bytes(int c, int S, size_t words) {
  return unit_layout(c, S, words_kept(c, S, words)).total;
}

// Block-wide exclusive scan (blockDim multiple of 32, <= 1024).
template <class T>
__device__ __forceinline__ T block_scan(T v, T &total, T *sbuf) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  T x = v;
  for (int o = 1; o < 32; o <<= 1) {
    T y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sbuf[warp] = x;
  __syncthreads();
  if (warp == 0) {
    T t = (lane < nw) ? sbuf[lane] : (T)0;
    for (int o = 1; o < 32; o <<= 1) {
      T y = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += y;
    }
    sbuf[lane] = t;
  }
  __syncthreads();
  const T excl = x - v + (warp ? sbuf[warp - 1] : (T)0);
  total = sbuf[nw - 1];
  __syncthreads();
  return excl;
}

struct UnitPtrs {
  uint64_t *mA, *mB;      // [W]
  int *pcA, *pcB;         // [W]
  uint32_t *rows;         // [2][g][GW]
  uint16_t *cnt3;         // [2][g][3] state counts per class
  uint16_t *fcnt;         // [2][g] capped count of full networks
  int16_t *fend;          // [2][g] column of the mp-th parent (0x7FFF: fewer)
  uint16_t *fps;          // [2][g][3] first three parents
  unsigned long long *fh; // [2][g] node hash of full networks
  int *phs, *phe;         // [2][g] flip-entry range per row
  int *moff;              // [2][g] variants of the rows before
  int *nst;               // [2][g] scratch of the compaction
  uint16_t *big;          // [2][g] rows formed per sample, per class
  uint8_t *need;          // [g] 1 = full lists differ, 2 = scores needed
  uint8_t *nobs;          // [2][g] observed states per class
  uint32_t *used;         // [unit_variants / 32] variants some network uses
  unsigned long long *itk;   // [kItems] node-score items: t | np << 14 | parents
  long long *acc;            // [kItems][2] their scores per class
  int *tq;                   // [2 kItems + 1] task prefix per (item, class)
  uint32_t *chg;             // [class_words of both classes] networks with a changed list
  int8_t *dmap;              // [96] divisor map (copy of the constant one)
  long long *fsc;            // [2 full][2 data][g] base node scores
  uint2 *ent;                // [kEntCache] the kept flip entries
};

struct UnitSmem {
  // fixed part; variable arrays follow in dynamic shared memory
  SetDev sd;    // the unit's set (copied from the batch's set table)
  UnitPtrs P;   // the variable arrays (for the functions not inlined)
  unsigned long long HF[2];  // hashes of the two full networks
  long long base[2][2];      // [data class][full network of class]
  int flen[2];  // edges of the full networks' capped lists (kept units)
  int ndab;     // nodes whose full lists differ between the classes
  int split[2]; // class 2's first memo entry, first variant
  int nbig[2];  // rows formed per sample, per class
  int firstB0;  // first class-2 network equal to the class-2 full network
  int nchg;     // networks that differ from their class's full network
  int nver;     // networks merged by hash
  int nsel;     // variants to score
  int any;
  int next[2];  // the block's next unit (by turns)
  long long cycles[2];  // BatchDev::cycles of this block
  unsigned status;
  unsigned long long koff;  // a kept unit's region of the packed outputs
  int scan[32];
  unsigned long long scan64[32];
  long long red[6][32];
  double redd[3][32];
};

// BDeu work items (node scores) processed per round
constexpr int kItems = 512;
// the BDeu item arrays (keys, scores, task prefix) in one region that also
// holds the operands of the networks' sums (unit_walk) and then the network
// table
constexpr size_t kWorkBytes = sizeof(unsigned long long) * kItems + 2 * sizeof(long long) * kItems +
                              sizeof(int) * (2 * kItems + 4);
static_assert(kSmSlots * sizeof(int) <= kWorkBytes && kWorkBytes % 16 == 0, "work region");
// kept flip entries a unit holds in shared memory (more go to its scratch)
constexpr int kEntCache = 1280;

static UnitSlices unit_slices(int g, int W) {
  UnitSlices P;
  const int GW = (g + 31) / 32;
  size_t o = sizeof(UnitSmem);
  auto take = [&](size_t bytes) {
    o = (o + 15) & ~(size_t)15;
    const size_t at = o;
    o += bytes;
    return (uint32_t)at;
  };
  P.mA = take(2 * sizeof(uint64_t) * W);
  P.mB = P.mA + sizeof(uint64_t) * W;
  P.pcA = take(2 * sizeof(int) * W);
  P.pcB = P.pcA + sizeof(int) * W;
  P.rows = take(2 * sizeof(uint32_t) * (size_t)g * GW);
  P.cnt3 = take(2 * 3 * sizeof(uint16_t) * g);
  P.fcnt = take(2 * sizeof(uint16_t) * g);
  P.fend = take(2 * sizeof(uint16_t) * g);
  P.fps = take(2 * 3 * sizeof(uint16_t) * g);
  P.fh = take(2 * sizeof(unsigned long long) * g);
  P.phs = take(4 * sizeof(int) * g);
  P.moff = take(2 * sizeof(int) * g);
  P.nst = take(2 * sizeof(int) * g);
  P.big = take(2 * sizeof(uint16_t) * g);
  P.need = take(g);
  P.nobs = take(2 * g);
  P.used = take(sizeof(uint32_t) * ((unit_variants(g) + 31) / 32));
  P.chg = take(sizeof(uint32_t) * (2 * W + 2));
  P.dmap = take(96);
  // (the base scores follow the work region directly)
  P.itk = take(kWorkBytes + 4 * sizeof(long long) * g);
  P.acc = P.itk + sizeof(unsigned long long) * kItems;
  P.tq = P.acc + 2 * sizeof(long long) * kItems;
  P.fsc = P.itk + kWorkBytes;
  P.ent = take(sizeof(uint2) * kEntCache);
  P.total = (uint32_t)((o + 15) & ~(size_t)15);
  return P;
}
// (phe follows phs, both by the unit's own genes: they are copied as one)
__device__ __forceinline__ UnitPtrs unit_ptrs(char *base, const UnitSlices &o, int g) {
  UnitPtrs P;
  P.mA = (uint64_t *)(base + o.mA);
  P.mB = (uint64_t *)(base + o.mB);
  P.pcA = (int *)(base + o.pcA);
  P.pcB = (int *)(base + o.pcB);
  P.rows = (uint32_t *)(base + o.rows);
  P.cnt3 = (uint16_t *)(base + o.cnt3);
  P.fcnt = (uint16_t *)(base + o.fcnt);
  P.fend = (int16_t *)(base + o.fend);
  P.fps = (uint16_t *)(base + o.fps);
  P.fh = (unsigned long long *)(base + o.fh);
  P.phs = (int *)(base + o.phs);
  P.phe = P.phs + 2 * g;
  P.moff = (int *)(base + o.moff);
  P.nst = (int *)(base + o.nst);
  P.big = (uint16_t *)(base + o.big);
  P.need = (uint8_t *)(base + o.need);
  P.nobs = (uint8_t *)(base + o.nobs);
  P.used = (uint32_t *)(base + o.used);
  P.chg = (uint32_t *)(base + o.chg);
  P.dmap = (int8_t *)(base + o.dmap);
  P.itk = (unsigned long long *)(base + o.itk);
  P.acc = (long long *)(base + o.acc);
  P.tq = (int *)(base + o.tq);
  P.fsc = (long long *)(base + o.fsc);
  P.ent = (uint2 *)(base + o.ent);
  return P;
}

// Network s of a unit: class k (0 = class 1, 1 = class 2) and left-out
// sample sigma (-1 for the two full networks), kernel1.cu:85-88, 412-416.
// sig: class-1 samples then class-2 samples in index order.
__device__ __forceinline__ void net_of(int s, const SetDev &sd, const int *sig, int &k, int &sigma) {
  if (s == 0) { k = 0; sigma = -1; return; }
  if (s == sd.S - 1) { k = 1; sigma = -1; return; }
  // class-1 sample s-1 sits at s-1; class-2 sample s-nA-1 at nA+(s-nA-1) = s-1
  k = (s <= sd.nA) ? 0 : 1;
  sigma = sig[s - 1];
}

__device__ __forceinline__ void gen_for(ListGen &G, const SetDev &sd, const UnitPtrs &P,
                                        const uint2 *ent, int k, int t, int sigma) {
  const int i = k * sd.g + t;
  G.init(P.rows + (size_t)i * sd.GW, sd.GW, ent, P.phs[i], P.phe[i], sd.codes, sd.n16, t, sigma);
}

// Exact comparison of the capped lists of node t in two networks.
__device__ __noinline__ bool lists_equal(const SetDev &sd, const UnitPtrs &P, const uint2 *ent, int t,
                                         int k1, int sigma1, int k2, int sigma2) {
  ListGen a, b;
  gen_for(a, sd, P, ent, k1, t, sigma1);
  gen_for(b, sd, P, ent, k2, t, sigma2);
  for (int i = 0; i < sd.mp; i++) {
    int x = a.next(), y = b.next();
    if (x != y) return false;
    if (x < 0) return true;
  }
  return true;
}

// A capped list's key: node, count of the first three parents, the parents.
__device__ __forceinline__ unsigned long long list_key(int t, int cnt, const int *ps) {
  return (unsigned long long)t | ((unsigned long long)(cnt < 3 ? cnt : 3) << 14) |
         ((unsigned long long)(ps[0] & 0xFFFF) << 16) |
         ((unsigned long long)(ps[1] & 0xFFFF) << 32) | ((unsigned long long)(ps[2] & 0xFFFF) << 48);
}

// The list of row i = (k, t) for left-out sample sigma, when it differs
// from the full network's: its key, hash and length (false: the full list).  The
// lists differ exactly when the first column that a triggered entry
// toggles is not past the full list's end (an edge taken out there was in
// the list; one put in there belongs to it).
__device__ __noinline__ bool sample_list(const SetDev &sd, const UnitPtrs &P, const uint2 *ent, int k,
                                         int t, int sigma, unsigned long long &key,
                                         unsigned long long &hash, int &len) {
  const int i = k * sd.g + t;
  const uint32_t *cw = sd.codes + (sigma >> 4);
  const int sh = 2 * (sigma & 15);
  const int a4 = 4 * ((cw[(size_t)t * sd.n16] >> sh) & 3);
  int first = 0x7FFFFFFF;
  for (int e = P.phs[i]; e < P.phe[i]; e++) {
    const uint2 en = ent[e];
    const int col = en.x & 511;
    const int b = (cw[(size_t)col * sd.n16] >> sh) & 3;
    if ((en.y >> (a4 + b)) & 1u) {
      first = col;
      break;
    }
  }
  if (first > P.fend[i]) return false;
  ListGen G;
  gen_for(G, sd, P, ent, k, t, sigma);
  uint64_t h = node_hash_init(sd.salt, t);
  int cnt = 0, ps[3] = {0xFFFF, 0xFFFF, 0xFFFF};
  while (cnt < sd.mp) {
    const int j = G.next();
    if (j < 0) break;
    if (cnt < 3) ps[cnt] = j;
    h = node_hash_step(h, j);
    cnt++;
  }
  key = list_key(t, cnt, ps);
  hash = h;
  len = cnt;
  return true;
}

// The unit kernel's shared memory.  (Functions that are not inlined reach it by
// offset: through a pointer the loads would be generic ones.)
extern __shared__ __align__(16) char unit_smem[];

// divisor rows of a score's terms in one class (false: no observed
// configuration or child state, the score is 0)
__device__ __forceinline__ bool bdeu_rows(const SetDev &sd, const UnitPtrs &P, int cls, int t, int np,
                                          int p0, int p1, int p2, const int64_t *&LGq,
                                          const int64_t *&LGqr) {
  const uint8_t *no = P.nobs + cls * sd.g;
  const int q = no[p0] * (np > 1 ? no[p1] : 1) * (np > 2 ? no[p2] : 1), r = no[t];
  if (q == 0 || r == 0) return false;
  LGq = sd.lg + (size_t)P.dmap[q] * sd.lg_stride;
  LGqr = sd.lg + (size_t)P.dmap[q * r] * sd.lg_stride;
  return true;
}

// Node scores of `n` keys (t | np << 14 | p0 << 16 | p1 << 32 | p2 << 48; ~0:
// nothing to score, 0), kItems per round, as a flat task list over the block:
// task (key, class, parent configuration j); out: class-1 score, class-2
// score.  Fixed-point terms are summed with atomics: exact, in any order.
// Nodes without parents are scored from the state counts.
__device__ __noinline__ void bdeu_items(const UnitSlices &o, const ClassPlanes cpA,
                                        const ClassPlanes cpB, int n, const unsigned long long *keys,
                                        longlong2 *out) {
  UnitSmem &SM = *reinterpret_cast<UnitSmem *>(unit_smem);
  const SetDev &sd = SM.sd;
  const UnitPtrs P = unit_ptrs(unit_smem, o, sd.g);
  const int tid = threadIdx.x, nt = blockDim.x, g = sd.g;
#pragma unroll 1
  for (int b0 = 0; b0 < n; b0 += kItems) {
    const int m = n - b0 < kItems ? n - b0 : kItems;
    for (int i = tid; i < m; i += nt) {
      const unsigned long long key = keys[b0 + i];
      P.itk[i] = key;
      const int np = (key == ~0ull) ? 0 : (int)((key >> 14) & 3);
      for (int cls = 0; cls < 2; cls++) {
        P.tq[2 * i + cls] = np ? bdeu_tasks(np) : 0;
        P.acc[2 * i + cls] = (key != ~0ull && np == 0)
                                 ? bdeu_score0(sd, (int)(key & 0x3FFF), P.cnt3 + 3 * g * cls)
                                 : 0;
      }
    }
    __syncthreads();
    int running = 0;
    for (int c0 = 0; c0 < 2 * m; c0 += nt) {
      const int e = c0 + tid;
      const int v = e < 2 * m ? P.tq[e] : 0;
      int total;
      const int off = block_scan(v, total, SM.scan);
      if (e < 2 * m) P.tq[e] = running + off;
      running += total;
    }
    __syncthreads();
    // tasks in (item, class) order: a warp's consecutive lanes mostly share
    // one score, so their terms are summed in the warp (segmented) and each
    // score takes one atomic per warp
    const int lane = tid & 31;
    for (int base = tid - lane; base < running; base += nt) {
      const int task = base + lane;
      int seg = -1;
      long long term = 0;
      if (task < running) {
        int lo = 0, hi = 2 * m - 1;
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (P.tq[mid] <= task) lo = mid;
          else hi = mid - 1;
        }
        const int i = lo >> 1, cls = lo & 1, j = task - P.tq[lo];
        const unsigned long long key = P.itk[i];
        const int t = (int)(key & 0x3FFF), np = (int)((key >> 14) & 3);
        const int p0 = (int)((key >> 16) & 0xFFFF), p1 = (int)((key >> 32) & 0xFFFF),
                  p2 = (int)((key >> 48) & 0xFFFF);
        const int64_t *LGq, *LGqr;
        if (bdeu_rows(sd, P, cls, t, np, p0, p1, p2, LGq, LGqr))
          term = bdeu_config_term(cls ? cpB : cpA, t, np, p0, p1, p2, j, LGq, LGqr);
        seg = lo;
      }
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const long long y = __shfl_up_sync(0xffffffffu, term, d);
        const int sy = __shfl_up_sync(0xffffffffu, seg, d);
        if (lane >= d && sy == seg) term += y;
      }
      const int sn = __shfl_down_sync(0xffffffffu, seg, 1);
      if (seg >= 0 && (lane == 31 || sn != seg))
        atomicAdd((unsigned long long *)&P.acc[seg], (unsigned long long)term);
    }
    __syncthreads();
    for (int i = tid; i < m; i += nt) out[b0 + i] = make_longlong2(P.acc[2 * i], P.acc[2 * i + 1]);
    __syncthreads();
  }
}

// Both classes' scores of one key by one thread.
__device__ __noinline__ void key_scores(const SetDev &sd, const UnitPtrs &P, const ClassPlanes *cp,
                                        unsigned long long key, long long *s) {
  const int t = (int)(key & 0x3FFF), np = (int)((key >> 14) & 3);
  const int p0 = (int)((key >> 16) & 0xFFFF), p1 = (int)((key >> 32) & 0xFFFF),
            p2 = (int)((key >> 48) & 0xFFFF);
  for (int cls = 0; cls < 2; cls++) {
    if (np == 0) {
      s[cls] = bdeu_score0(sd, t, P.cnt3 + 3 * sd.g * cls);
      continue;
    }
    const int64_t *LGq, *LGqr;
    s[cls] = 0;
    if (bdeu_rows(sd, P, cls, t, np, p0, p1, p2, LGq, LGqr))
      for (int j = 0; j < bdeu_tasks(np); j++)
        s[cls] += bdeu_config_term(cp[cls], t, np, p0, p1, p2, j, LGq, LGqr);
  }
}

// The states of a unit's samples packed by class (ClassPlanes), a lane per
// gene, a warp per 32 genes and class: the class's bits of each sample word
// are moved together (Hacker's Delight's compress, its five move masks
// formed once per word and class) and appended to the gene's current output
// word; the lanes share the masks, so they fill and store words together.
//
// A warp's words are one chain of latencies.  With many of them (kLong) the
// warps that the genes leave over share the words, eight each at least, and a
// word's masks are loaded a word ahead as its planes are (cycles of a block:
// 10 genes x 16000 samples 235k -> 55k, 250 x 4000 133k -> 88k).  With few it
// costs more than it gives (5025 units of 51 x 66 2.82 -> 2.87 ms).
constexpr int kLongWords = 16;
template <bool kLong>
__device__ __noinline__ void pack_classes(const SetDev &sd, const UnitPtrs &P, uint32_t *moves,
                                          uint2 *out) {
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  const int g = sd.g, W32 = 2 * sd.W;
  for (int i = tid; i < 2 * W32; i += nt) {
    const int cls = i >= W32 ? 1 : 0;
    uint32_t m = reinterpret_cast<const uint32_t *>(cls ? P.mB : P.mA)[i - cls * W32];
    uint32_t *mv = moves + 8 * i;
    mv[5] = m;
    uint32_t mk = ~m << 1;
#pragma unroll
    for (int b = 0; b < 5; b++) {
      uint32_t mp = mk ^ (mk << 1);
      mp ^= mp << 2;
      mp ^= mp << 4;
      mp ^= mp << 8;
      mp ^= mp << 16;
      const uint32_t v = mp & m;
      mv[b] = v;
      m = (m ^ v) | (v >> (1 << b));
      mk &= ~mp;
    }
  }
  __syncthreads();
  const int gb = (g + 31) >> 5, segs = kLong ? max(1, min(nw / (2 * gb), sd.W / 8)) : 1;
  for (int task = warp; task < 2 * gb * segs; task += nw) {
    const int seg = kLong ? task / (2 * gb) : 0, ct = task - seg * 2 * gb, cls = ct >= gb ? 1 : 0;
    const int i = 32 * (ct - cls * gb) + lane;
    const bool live = i < g;
    // the sample words [ws, we): the class's output words [o0, o1) that start
    // there, the last of which is filled from the words behind
    int ws = 0, o0 = 0, o1 = class_words(cls ? sd.nB : sd.nA), fill = 0, at = 0;
    if (kLong) {
      const int *pc = cls ? P.pcB : P.pcA;
      const int we = sd.W * (seg + 1) / segs;
      ws = sd.W * seg / segs;
      o0 = (pc[ws] + 31) >> 5;
      if (we < sd.W) o1 = (pc[we] + 31) >> 5;
      if (o0 >= o1) continue;
      fill = pc[ws] & 31;
      at = pc[ws] >> 5;
    }
    const uint64_t *pl = sd.planesT + 3 * ((size_t)ws * g + (live ? i : g - 1));
    uint2 *dst = out + (cls ? (size_t)class_words(sd.nA) * g : 0) + (size_t)at * g + i;
    auto store = [&](uint32_t x, uint32_t y) {
      if (live && (!kLong || at >= o0)) *dst = make_uint2(x, y);
      dst += g;
      if (kLong) at++;
    };
    const uint2 *end = dst + (size_t)(o1 - at) * g;
    const uint4 *mv4 = reinterpret_cast<const uint4 *>(moves + 8 * (size_t)cls * W32);
    uint32_t a0 = 0u, a1 = 0u;
    uint64_t n0 = pl[0], n1 = pl[1], n2 = pl[2];  // the next word's planes
    uint4 mn[4];
#pragma unroll
    for (int x = 0; kLong && x < 4; x++) mn[x] = mv4[4 * ws + x];
#pragma unroll 1
    for (int w = ws; w < sd.W && (!kLong || at < o1); w++) {
      const uint64_t q0 = n0, q1 = n1, q2 = n2;
      uint4 mq[4];
#pragma unroll
      for (int x = 0; kLong && x < 4; x++) mq[x] = mn[x];
      if (w + 1 < sd.W) {
        pl += 3 * (size_t)g;
        n0 = pl[0];
        n1 = pl[1];
        n2 = pl[2];
#pragma unroll
        for (int x = 0; kLong && x < 4; x++) mn[x] = mv4[4 * (w + 1) + x];
      }
      const uint64_t mis = ~(q0 | q1 | q2), b0 = q1 | mis, b1 = q2 | mis;
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const uint4 u = kLong ? mq[2 * h] : mv4[4 * w + 2 * h], v = kLong ? mq[2 * h + 1] : mv4[4 * w + 2 * h + 1];
        const uint32_t mv[5] = {u.x, u.y, u.z, u.w, v.x};
        uint32_t x0 = (uint32_t)(b0 >> (32 * h)) & v.y, x1 = (uint32_t)(b1 >> (32 * h)) & v.y;
#pragma unroll
        for (int b = 0; b < 5; b++) {
          const uint32_t t0 = x0 & mv[b], t1 = x1 & mv[b];
          x0 = (x0 ^ t0) | (t0 >> (1 << b));
          x1 = (x1 ^ t1) | (t1 >> (1 << b));
        }
        a0 |= x0 << fill;
        a1 |= x1 << fill;
        const int c = __popc(v.y);
        if (fill + c >= 32) {
          if (!kLong || at < o1) store(a0, a1);
          a0 = fill ? x0 >> (32 - fill) : 0u;
          a1 = fill ? x1 >> (32 - fill) : 0u;
          fill -= 32;
        }
        fill += c;
      }
    }
    // past the class's last sample: no value
    if (fill && (!kLong || at < o1)) store(a0 | (~0u << fill), a1 | (~0u << fill));
    while (kLong ? at < o1 : dst != end) store(~0u, ~0u);
  }
  __syncthreads();
}

// Where a variant comes from: its row's first kept entry, their number and
// the subset of them that fires; bit 31: it has a list of its own (not the
// full network's).
__device__ __forceinline__ uint32_t variant_info(int e0, int e, int sub, bool live) {
  return (uint32_t)e0 | ((uint32_t)e << 14) | ((uint32_t)sub << 18) | (live ? 1u << 31 : 0u);
}
__device__ __forceinline__ uint32_t info_live(uint32_t x) { return (uint32_t)((int32_t)x >> 31); }
__device__ __forceinline__ int info_first(uint32_t x) { return (int)(x & 0x3FFFu); }
__device__ __forceinline__ int info_count(uint32_t x) { return (int)((x >> 14) & 15u); }
__device__ __forceinline__ int info_end(uint32_t x) { return info_first(x) + info_count(x); }

// The 32 samples of a class that fire an entry (t, j, cells): the OR over the
// cells (a, b) of state a of node t and state b of column j.
__device__ __forceinline__ uint32_t trigger_word(const uint2 *cw, uint2 en) {
  const uint2 a = cw[(en.x >> 9) & 511u], b = cw[en.x & 511u];
  const uint32_t j0 = ~(b.x | b.y), j1 = b.x & ~b.y, j2 = b.y & ~b.x;
  auto cells = [&](uint32_t f) {
    return ((f & 1u) ? j0 : 0u) | ((f & 2u) ? j1 : 0u) | ((f & 4u) ? j2 : 0u);
  };
  return (~(a.x | a.y) & cells(en.y)) | ((a.x & ~a.y) & cells(en.y >> 4)) |
         ((a.y & ~a.x) & cells(en.y >> 8));
}

constexpr int kFewVariants = 16;
constexpr int kUnitRegs = 80;

// Which of the unit's nvar variants (class 2's from vsplit on) some left-out
// sample changes its row to (P.used), which samples have a changed list
// (P.chg), and the variants' words (vw[v][stride]).
// 8, 16 or 32 words of the classes at a time, a lane per variant and word; the
// entries' trigger words are formed first, as many as `bytes` of the work
// region hold, word by word (a warp's 32 entries share their nodes' planes;
// an odd pitch keeps the lanes' words in different banks).  Both classes go by
// together and four variants of a lane at a time: bound by the chain from a
// variant's number to its words.  (The subsets' products from registers, a
// lane per row and word, unrolled: more instructions than the instruction
// cache holds beside the rest, 268k cycles of a block at 200 genes x 1000
// samples against 131k.)
template <int kThreads>
__device__ __noinline__ void mark_variants(const UnitSlices &o, const ClassPlanes cpA,
                                           const ClassPlanes cpB, int nA, int nB,
                                           const uint2 *ent, const uint32_t *vinf, int vsplit,
                                           int nvar, uint32_t *vw, int stride, int bytes) {
  uint32_t *T = (uint32_t *)(unit_smem + o.itk), *used = (uint32_t *)(unit_smem + o.used);
  uint32_t *chg = (uint32_t *)(unit_smem + o.chg);
  const int tid = threadIdx.x, lane = tid & 31, g = cpA.g;
  const int w1 = (nA + 31) >> 5, w2 = (nB + 31) >> 5, words = max(w1, w2);
  const int lw = words <= 8 ? 3 : words <= 16 ? 4 : 5, nw = 1 << lw;
  const int pitch = ((bytes >> (lw + 2)) - 1) | 1, w = tid & (nw - 1);
  constexpr int kAt = 4;  // loads in flight
  for (int w0 = 0; w0 < words; w0 += nw) {
    uint32_t c1 = 0u, c2 = 0u;
    for (int q = 0, qe; q < nvar; q = qe) {
      const int e0 = info_first(vinf[q]);
      qe = nvar;
      if (info_end(vinf[nvar - 1]) - e0 > pitch) {
        // the longest run of variants whose rows' entries fit
        int lo = q + 1;
        while (lo < qe) {
          const int mid = (lo + qe + 1) >> 1;
          if (info_end(vinf[mid - 1]) - e0 <= pitch) lo = mid;
          else qe = mid - 1;
        }
      }
      const int ne = info_end(vinf[qe - 1]) - e0;
      // class 1's entries end where class 2's variants begin
      const int esplit = vsplit <= q ? 0 : vsplit >= qe ? ne : info_first(vinf[vsplit]) - e0;
      __syncthreads();
      {
        const int n = ne * min(nw, words - w0);
        const int dx = kThreads / ne, de = kThreads - dx * ne;
        int x = tid / ne, e = tid - x * ne;
        for (int i = tid; i < n; i += kAt * kThreads) {
          uint32_t y[kAt];
          int at[kAt];
#pragma unroll
          for (int r = 0; r < kAt; r++) {
            const bool k1 = e < esplit, in = i + r * kThreads < n && w0 + x < (k1 ? w1 : w2);
            at[r] = x * pitch + e;
            y[r] = in ? trigger_word((k1 ? cpA.p : cpB.p) + (size_t)(w0 + x) * g, ent[e0 + e]) : 0u;
            e += de;
            x += dx;
            if (e >= ne) e -= ne, x++;
          }
#pragma unroll
          for (int r = 0; r < kAt; r++)
            if (i + r * kThreads < n) T[at[r]] = y[r];
        }
      }
      __syncthreads();
      const uint32_t *t0 = T + w * pitch - e0;
      for (int b = q + (tid >> lw); b - (tid >> lw) < qe; b += kAt * (kThreads >> lw)) {
        uint32_t info[kAt];
#pragma unroll
        for (int r = 0; r < kAt; r++) {
          const int v = b + r * (kThreads >> lw);
          info[r] = v < qe && w0 + w < words ? vinf[v] : 0u;
        }
        // (all loads before the stores, which might alias them)
        uint32_t y[kAt];
#pragma unroll
        for (int r = 0; r < kAt; r++) {
          const uint32_t *t = t0 + info_first(info[r]);
          const uint32_t sub = info[r] >> 18;
          const int cnt = info_count(info[r]);
          y[r] = info_live(info[r]);
#pragma unroll
          for (int j = 0; j < 4; j++)
            if (j < cnt) y[r] &= t[j] ^ (((sub >> j) & 1u) - 1u);
          for (int j = 4; j < cnt; j++) y[r] &= t[j] ^ (((sub >> j) & 1u) - 1u);
        }
#pragma unroll
        for (int r = 0; r < kAt; r++) {
          const int v = b + r * (kThreads >> lw);
          const uint32_t x = y[r];
          if (info[r]) vw[(size_t)v * stride + w0 + w] = x;
          if (v < vsplit) c1 |= x;
          else c2 |= x;
          const uint32_t any = __ballot_sync(0xffffffffu, x != 0u) >> (lane & ~(nw - 1));
          if (w == 0 && (any & (~0u >> (32 - nw)))) atomicOr(&used[v >> 5], 1u << (v & 31));
        }
      }
    }
    for (int o = nw; o < 32; o <<= 1) {
      c1 |= __shfl_xor_sync(0xffffffffu, c1, o);
      c2 |= __shfl_xor_sync(0xffffffffu, c2, o);
    }
    if (lane < nw && c1) atomicOr(&chg[w0 + w], c1);
    if (lane < nw && c2) atomicOr(&chg[cpA.words + w0 + w], c2);
  }
}

__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                         uint32_t a3, uint2 b) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b.x), "r"(b.y));
}

// What the left-out samples of a class of nk change: for every sample the sum
// over the used variants uv[0 .. nu) that it fires of the variant's hash
// difference and of its two score differences (and, J = 4, of its list's
// length difference), put(i, sums) for sample i of the class.
//
// The sums are a contraction of the samples' bits with the variants' values,
// so they go through the matrix units: the values' eight bytes are the
// columns of bf16 operand B (0 .. 255, exact), the bits, as 0 or 2, are
// operand A (a sample fires at most one variant of a row, so a column sums to
// at most 2 x 512 x 255: exact in FP32), and the bytes' sums are put together
// modulo 2^64.  A warp takes 32 samples, eight words of the class at a time;
// the variants go by in blocks of 160, the next one's words and values loaded
// while this one's are multiplied.  mma.sync tiles, M = samples, N = 24, K =
// variants: a block's operands are read once, so the descriptors, fences and
// TMEM round trips of tcgen05.mma would cost more than the 60 instructions a
// warp issues for it.  The bits pass into registers by shift and mask: a pair
// of variants' words is held as its low and its high halves, so that bit r of
// both variants lands in the exponents' top bits of one register.
template <int kThreads, int J, class Word, class Value, class Put>
__device__ __noinline__ void unit_walk(uint32_t region, int nk, int nu, Word word, Value value,
                                       Put put) {
  constexpr int kUnitWarps = 8;                            // words of a step (warps past them help to stage)
  constexpr int kK = 160;                                  // variants of a block
  constexpr int kB = (kK / 2 * J + kThreads - 1) / kThreads;  // pairs of values
  static_assert(kK * (4 * kUnitWarps + 16 * J) <= (int)kWorkBytes, "work region");
  uint2 *A = (uint2 *)(unit_smem + region);                          // [kK / 16][8 words][4][2]
  uint32_t *B = (uint32_t *)(A + kK / 2 * kUnitWarps);     // [kK / 16][J][8][4][2]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, words = (nk + 31) >> 5;
  const int r8 = lane >> 2, t4 = lane & 3, aw = tid & (kUnitWarps - 1), ap = tid / kUnitWarps;
  const uint32_t sh0 = 14 - r8, sh1 = (6 - r8) & 31;
  auto bits = [](uint32_t x, uint32_t sh) { return __funnelshift_l(x, x, sh) & 0x40004000u; };
  constexpr int kPairs = kThreads / kUnitWarps;          // pairs of operand A at a time
  constexpr int kAp = (kK / 2 + kPairs - 1) / kPairs;
  for (int w0 = 0; w0 < words; w0 += kUnitWarps) {
    float acc[2][J][4];
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
      for (int j = 0; j < J; j++)
#pragma unroll
        for (int q = 0; q < 4; q++) acc[m][j][q] = 0.f;
    uint32_t xa[kAp][2];
    unsigned long long xb[kB][2];
    auto load = [&](int q) {
#pragma unroll
      for (int r = 0; r < kAp; r++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int p = ap + r * kPairs, i = q + 2 * p + h;
          xa[r][h] = 2 * p < kK && i < nu && w0 + aw < words ? word(i, w0 + aw) : 0u;
        }
#pragma unroll
      for (int r = 0; r < kB; r++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int x = tid + r * kThreads, j = x / (kK / 2), i = q + 2 * (x - j * (kK / 2)) + h;
          xb[r][h] = j < J && i < nu ? value(i, j) : 0ull;
        }
    };
    // (one copy of each part's code: the next block's loads, this block's
    // products, then the operands)
#pragma unroll 1
    for (int q = 0; q < nu + kK; q += kK) {
      if (q < nu) load(q);
      if (q > 0 && warp < kUnitWarps && w0 + warp < words) {
        const int steps = (min(kK, nu - (q - kK)) + 15) >> 4;
        const uint4 *a4 = reinterpret_cast<const uint4 *>(A) + warp * 4 + t4;
        const uint2 *b2 = reinterpret_cast<const uint2 *>(B) + lane;
#pragma unroll 2
        for (int ks = 0; ks < steps; ks++, a4 += 4 * kUnitWarps, b2 += 32 * J) {
          const uint4 a = *a4;
          const uint32_t l0 = bits(a.x, sh0), l1 = bits(a.x, sh1), l2 = bits(a.z, sh0), l3 = bits(a.z, sh1);
          const uint32_t h0 = bits(a.y, sh0), h1 = bits(a.y, sh1), h2 = bits(a.w, sh0), h3 = bits(a.w, sh1);
#pragma unroll
          for (int j = 0; j < J; j++) {
            const uint2 b = b2[32 * j];
            mma_bf16(acc[0][j], l0, l1, l2, l3, b);
            mma_bf16(acc[1][j], h0, h1, h2, h3, b);
          }
        }
      }
      if (q >= nu) break;
      __syncthreads();
#pragma unroll
      for (int r = 0; r < kAp; r++) {
        const int p = ap + r * kPairs;
        if (2 * p < kK)
          A[(((p >> 3) * kUnitWarps + aw) * 4 + (p & 3)) * 2 + ((p >> 2) & 1)] = make_uint2(
              __byte_perm(xa[r][0], xa[r][1], 0x5410), __byte_perm(xa[r][0], xa[r][1], 0x7632));
      }
#pragma unroll
      for (int r = 0; r < kB; r++) {
        const int x = tid + r * kThreads, j = x / (kK / 2), p = x - j * (kK / 2);
        if (j >= J) continue;
        uint32_t *b = B + ((p >> 3) * J + j) * 64 + 2 * (p & 3) + ((p >> 2) & 1);
#pragma unroll
        for (int l = 0; l < 8; l++) {
          // a byte as a float: 2^23 + x, less 2^23
          float f[2];
#pragma unroll
          for (int h = 0; h < 2; h++)
            f[h] = __uint_as_float(__byte_perm((uint32_t)(xb[r][h] >> (l < 4 ? 0 : 32)), 0x4B000000u,
                                               0x7540u + (l & 3))) - 8388608.f;
          b[8 * l] = __byte_perm(__float_as_uint(f[0]), __float_as_uint(f[1]), 0x7632);
        }
      }
      __syncthreads();
    }
    if (warp >= kUnitWarps || w0 + warp >= words) continue;
    // a lane's two bytes' sums of samples r8 + 8 x, the four lanes' together
    // the value's; lane t4 keeps sample r8 + 8 t4
    unsigned long long sum[J];
#pragma unroll
    for (int j = 0; j < J; j++) {
      sum[j] = 0ull;
#pragma unroll
      for (int x = 0; x < 4; x++) {
        const unsigned lo = (unsigned)(acc[x >> 1][j][2 * (x & 1)] * 0.5f);
        const unsigned hi = (unsigned)(acc[x >> 1][j][2 * (x & 1) + 1] * 0.5f);
        unsigned long long y = ((unsigned long long)lo + ((unsigned long long)hi << 8)) << (16 * t4);
        y += __shfl_xor_sync(0xffffffffu, y, 1);
        y += __shfl_xor_sync(0xffffffffu, y, 2);
        if (x == t4) sum[j] = y;
      }
    }
    const int i = 32 * (w0 + warp) + r8 + 8 * t4;
    if (i < nk) put(i, sum);
  }
}

// Normalisation (main.cu:1302-1404) and JS (main.cu:1406-1428) of a unit
// from its unique networks' node-summed fixed-point scores dist[U], dist[S
// + U]: per class min, max and mean of the scores (exact integers),
// likelihoods exp((d - mean) 10 / (max - min)) normalised to sum 1, then the
// two KL terms of kool() (routines.cu:42-60), zeros skipped, in FP64.  The
// exponentials replace the scores in dist.  The even lanes take class 1, the
// odd ones class 2 (one copy of the code for both, and its latency: FP64's is
// most of a small unit's JS).  Sums are formed in a fixed order, the same in
// both classes: a thread's networks in turn, then a tree over the warp, then
// the warps in turn.  The first 256 threads take part, whatever the block
// has, so that a unit's JS is the same bits in every batch (a set's block
// size depends on the sets beside it).  pl, ql: the kept normalised
// likelihoods, or null.
//
// Inside k_units rather than after it: FP64 is slow on this part (about two
// operations a cycle and SM, ~128 cycles to a dependent one), and here its
// waits pass under the other blocks' integer work.  As a kernel of its own,
// a warp per unit or more units a warp, it took 6.0 ms for 10000 units of
// 1000 networks, 18.4 ms for 75000 of 400 and 68 us for one unit of 300.
static __device__ __noinline__ double unit_js(long long *dist, int S, int U, UnitSmem &SM, double *pl,
                                              double *ql) {
  constexpr int kJsThreads = 256, us = kJsThreads / 2;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // the warps that hold networks, and the lanes of a warp that do (the sums
  // over the others' zeros are left out: each costs a dependent FP64 add)
  const int nw = min(kJsThreads >> 5, (2 * U + 31) >> 5), lanes = min(2 * U, 32);
  const int cls = tid & 1, u0 = tid < kJsThreads ? tid >> 1 : U;
  long long *d = dist + (cls ? S : 0);
  long long mn = LLONG_MAX, mx = LLONG_MIN;
  unsigned long long sum = 0;  // modulo 2^64
  for (int uu = u0; uu < U; uu += us) {
    const long long a = d[uu];
    mn = min(mn, a);
    mx = max(mx, a);
    sum += (unsigned long long)a;
  }
#pragma unroll
  for (int o = 16; o > 1; o >>= 1) {
    mn = min(mn, (long long)__shfl_xor_sync(0xffffffffu, mn, o));
    mx = max(mx, (long long)__shfl_xor_sync(0xffffffffu, mx, o));
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
  }
  if (lane < 2) {
    SM.red[3 * lane][warp] = mn;
    SM.red[3 * lane + 1][warp] = mx;
    SM.red[3 * lane + 2][warp] = (long long)sum;
  }
  __syncthreads();
  mn = LLONG_MAX;
  mx = LLONG_MIN;
  sum = 0;
#pragma unroll 1
  for (int w = 0; w < nw; w++) {
    mn = min(mn, SM.red[3 * cls][w]);
    mx = max(mx, SM.red[3 * cls + 1][w]);
    sum += (unsigned long long)SM.red[3 * cls + 2][w];
  }
  // one score for all networks in a class: no JS
  const bool flat = __any_sync(0xffffffffu, mn == mx) != 0;
  if (flat && !pl) return __longlong_as_double(0x7ff8000000000000ll);
  // the sums of the scores less the smallest: exact
  sum -= (unsigned long long)U * (unsigned long long)mn;
  const double mean = (double)(long long)sum / (double)U, scale = 10.0 / (double)(mx - mn);
  auto exponent = [&](int uu) { return ((double)(d[uu] - mn) - mean) * scale; };
  // equal exponents in both classes throughout (two networks ranked alike,
  // above all): equal likelihoods, every term of the JS is log(1)
  double x = 0.0;
  if (U <= us) {
    if (u0 < U) x = exponent(u0);
    const bool differ = x != __shfl_xor_sync(0xffffffffu, x, 1);
    if (!pl && !__syncthreads_or(differ)) return 0.0;
  }
  double z = 0.0;
#pragma unroll 1
  for (int uu = u0; uu < U; uu += us) {
    const double e = exp(U <= us ? x : exponent(uu));
    d[uu] = __double_as_longlong(e);
    z += e;
  }
#pragma unroll
  for (int o = 16; o > 1; o >>= 1)
    if (o < lanes) z += __shfl_xor_sync(0xffffffffu, z, o);
  if (lane < 2) SM.redd[lane][warp] = z;
  __syncthreads();
  z = SM.redd[cls][0];
#pragma unroll 1
  for (int w = 1; w < nw; w++) z += SM.redd[cls][w];
  // a network's likelihoods P and Q in the two lanes, and its two terms
  double t = 0.0;
#pragma unroll 1
  for (int b = 0; b < U; b += us) {
    const int uu = b + u0;
    const double p = uu < U ? __longlong_as_double(d[uu]) / z : 0.0;
    const double m = (p + __shfl_xor_sync(0xffffffffu, p, 1)) / 2;
    double y = 0.0;
    if (p != 0 && m != 0) y = 0.5 * (p * log(p / m));
    t += y + __shfl_xor_sync(0xffffffffu, y, 1);
    if (pl && uu < U) (cls ? ql : pl)[uu] = p;
  }
#pragma unroll
  for (int o = 16; o > 1; o >>= 1)
    if (o < lanes) t += __shfl_xor_sync(0xffffffffu, t, o);
  if (lane == 0) SM.redd[2][warp] = t;
  __syncthreads();
  t = SM.redd[2][0];
#pragma unroll 1
  for (int w = 1; w < nw; w++) t += SM.redd[2][w];
  if (flat) return __longlong_as_double(0x7ff8000000000000ll);
  return t / log(2.0);
}

// One block per unit.  A left-out sample changes only rows whose flip
// entries it triggers, and both a network's hash and its score are sums over
// rows, so nothing is kept per network but those sums: which samples change a
// row to which list (variant) is found 32 samples at a time, and the sums are
// a product of the samples' bits with the variants' values (unit_walk).
// 10000 units of 200 genes x 1000 samples near the threshold: 44.0 ms with a
// warp per network that lists its changed nodes, 14.3 with a lane per left-out
// sample that walks the rows and sums a list of its changes, 12.2 now; 301
// units of 387 x 600 35.0, 2.8, 2.4 ms (all but the first with the
// normalisation and JS, then 6.0 ms more).  Bound by issue and the waits
// between dependent steps (0.68 million warp instructions a unit at the first
// shape, 45% of the issue slots), a third of the time in the node scores'
// population counts, whose rate (16 a cycle and SM) they reach.
template <int kThreads>
__device__ __forceinline__ void run_unit(const BatchDev &bd, int u, char *smraw) {
  UnitSmem &SM = *reinterpret_cast<UnitSmem *>(smraw);
  // (not a constant: the loops would be unrolled past the instruction cache)
  const int nt = blockDim.x, nw = nt >> 5;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // the unit's set: its descriptor into shared memory, its slices of the
  // batch's masks
  const BatchSet &bs = bd.sets[bd.uslot[u]];
  const int ul = u - bs.u0, bs_nb = bs.nb;
  const long long bs_dm0 = bs.dm0;
  const int keep = bd.keep_slot ? bd.keep_slot[u] : -1;
  uint8_t *scr = bd.scratch + (size_t)(keep < 0 ? (int)blockIdx.x : bd.blocks + keep) * bd.lay.total;
  {
    const int *src = reinterpret_cast<const int *>(&bs.sd);
    int *dst = reinterpret_cast<int *>(&SM.sd);
    for (int i = tid; i < (int)(sizeof(SetDev) / sizeof(int)); i += nt) dst[i] = src[i];
  }
  if (tid == 0) SM.any = 0;
  __syncthreads();
  const SetDev &sd = SM.sd;
  const int g = sd.g, W = sd.W, GW = sd.GW, S = sd.S, c = sd.c, nA = sd.nA, nB = sd.nB;
  uint32_t *ucb = bd.dmask + bs_dm0 + (size_t)bs_nb * c + (size_t)ul * chunk_words(c);
  uint32_t *dm = bd.dmask + bs_dm0 + (size_t)ul * c;
  // a unit without a nonzero mask has empty networks only: one unique
  // network, no JS
  for (int i = tid; i < chunk_words(c); i += nt)
    if (ucb[i]) SM.any = 1;
  __syncthreads();
  if (!SM.any && keep < 0) {
    if (tid == 0) {
      bd.js[u] = __longlong_as_double(0x7ff8000000000000ll);
      bd.U[u] = 1;
      bd.status[u] = 0u;
    }
    return;
  }
  const UnitPtrs P = unit_ptrs(smraw, bd.sm, g);
  const UnitLayout &L = bd.lay;
  if (tid == 0) SM.P = P;
  uint32_t *phi[2] = {(uint32_t *)(scr + L.phi[0]), (uint32_t *)(scr + L.phi[1])};
  long long *dist = (long long *)(scr + L.dist);
  int *sig = (int *)(scr + L.sig);

  // ---- P0: init
  if (tid == 0) {
    SM.HF[0] = SM.HF[1] = 0;
    SM.flen[0] = SM.flen[1] = 0;
    SM.ndab = 0;
    SM.status = 0;
    SM.nbig[0] = SM.nbig[1] = 0;
    SM.firstB0 = S - 1;
    SM.nchg = SM.nver = SM.nsel = 0;
    SM.split[0] = SM.split[1] = 0;
    for (int a = 0; a < 2; a++)
      for (int b = 0; b < 2; b++) SM.base[a][b] = 0;
  }
  for (int w = tid; w < W; w += nt) {
    uint64_t m = bd.masks[(size_t)u * W + w];
    P.mA[w] = m;
    P.mB[w] = sd.valid[w] & ~m;
  }
  for (int i = tid; i < 2 * g * GW; i += nt) P.rows[i] = 0;
  // entry ranges of rows: start = INT_MAX, end = 0 until an entry lands
  for (int i = tid; i < 4 * g; i += nt) P.phs[i] = (i < 2 * g) ? 0x7fffffff : 0;
  for (int i = tid; i < 2 * W + 2; i += nt) P.chg[i] = 0u;
  for (int i = tid; i < 82; i += nt) P.dmap[i] = c_dmap[i];
  __syncthreads();

  // ---- P1: full-network rows and flip lists, from the 32-pair chunks that
  // hold a nonzero mask (the decision kernel's bitmap; the other chunks are
  // all zero).  Each nonzero mask word read is set back to zero.  Warp w
  // owns the rows whose pairs start in [w c/nw, (w+1) c/nw) and walks its
  // flagged chunks in pair order, four loads at a time.  Edge bits go into
  // the row bitsets; the flip entries (column, cells << 16) land, in pair
  // order, in the warp's own segment of the list (which starts at its first
  // pair); a row's entry range is the min / max position of its entries
  // (rows without entries keep start > end).
  {
    const long long p_lo = (long long)warp * c / nw, p_hi = (long long)(warp + 1) * c / nw;
    int r0, c0;
    pair_rc((int)(p_lo < c ? p_lo : 0), r0, c0);
    if (c0 != 0) r0++;  // rows are owned by the warp holding their first pair
    int r1 = g;
    if (p_hi < c) {
      int c1;
      pair_rc((int)p_hi, r1, c1);
      if (c1 != 0) r1++;
    }
    if (p_lo >= c) r0 = g;
    if (r0 < 1) r0 = 1;  // row 0 has no pairs
    const int pa = r0 * (r0 - 1) / 2, pb = r0 < r1 ? r1 * (r1 - 1) / 2 : pa;
    int wpos0 = pa, wpos1 = pa;
    const uint32_t below = (1u << lane) - 1u;
    const uint32_t *cbits = ucb;
    const int k0 = pa >> 5, k1 = (pb + 31) >> 5;  // chunks [k0, k1)
    auto chunk = [&](int k, uint32_t m) {
      const int p = 32 * k + lane;
      const bool in = p >= pa && p < pb;
      int t = 0, j = 0;
      if (in) pair_rc(p, t, j);
      if (in && (m & 1u)) atomicOr(&P.rows[((size_t)0 * g + t) * GW + (j >> 5)], 1u << (j & 31));
      if (in && ((m >> 16) & 1u))
        atomicOr(&P.rows[((size_t)1 * g + t) * GW + (j >> 5)], 1u << (j & 31));
#pragma unroll
      for (int cls = 0; cls < 2; cls++) {
        const uint32_t mm = (m >> (16 * cls)) & 0x3FFu;
        const uint32_t fb = (mm >> 1) ^ ((mm & 1u) ? 0x1FFu : 0u);
        const bool flag = in && fb != 0u;
        const uint32_t bal = __ballot_sync(0xffffffffu, flag);
        const int wpos = cls ? wpos1 : wpos0;
        const int pos = wpos + __popc(bal & below);
        if (flag) {
          phi[cls][pos] = (uint32_t)j | (cells16(fb) << 16);
          atomicMin(&P.phs[cls * g + t], pos);
          atomicMax(&P.phe[cls * g + t], pos + 1);
        }
        if (cls) wpos1 += __popc(bal); else wpos0 += __popc(bal);
      }
    };
    for (int kw = k0 >> 5; pa < pb && kw <= (k1 - 1) >> 5; kw++) {
      uint32_t bits = cbits[kw];
      if (kw == (k0 >> 5)) bits &= ~0u << (k0 & 31);
      if (kw == ((k1 - 1) >> 5) && (k1 & 31)) bits &= ~0u >> (32 - (k1 & 31));
      while (bits) {
        int ks[4];
        uint32_t mv[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
          ks[q] = -1;
          if (bits) {
            ks[q] = 32 * kw + __ffs(bits) - 1;
            bits &= bits - 1;
          }
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const int p = 32 * ks[q] + lane;
          mv[q] = (ks[q] >= 0 && p >= pa && p < pb) ? dm[p] : 0u;
        }
#pragma unroll
        for (int q = 0; q < 4; q++)
          if (ks[q] >= 0) {
            chunk(ks[q], mv[q]);
            if (mv[q]) dm[32 * ks[q] + lane] = 0u;  // read once: left zero
          }
      }
    }
  }
  __syncthreads();
  // every warp has read the unit's chunk bitmap: zero it for the next batch
  for (int i = tid; i < chunk_words(c); i += nt) ucb[i] = 0u;

  // ---- P1b: only flip entries that can change a capped list are kept.
  // Node t's capped list is its first mp parents.  If R of the row's
  // entries are edges of the full network (the flips that can remove an
  // edge), every network of the class has at least mp edges in the columns
  // up to the (mp + R)-th edge of the full row, so its capped list lies
  // there: entries at later columns change no list and no network, and are
  // dropped (networks that differ only in them are the same network).  A
  // row's entries are contiguous and in column order.
  int kept = 0;
  for (int i = tid; i < 2 * g; i += nt) {
    const int e0 = P.phs[i], e1 = P.phe[i];
    if (e0 >= e1) continue;
    const int k = i / g, t = i - k * g;
    const uint32_t *row = P.rows + (size_t)i * GW;
    int R = 0;
    for (int e = e0; e < e1; e++) {
      const int j = phi[k][e] & 0xFFFF;
      R += (row[j >> 5] >> (j & 31)) & 1u;
    }
    int need = sd.mp + R, reach = t;  // t: every column of the row
    for (int w = 0; w < GW; w++) {
      uint32_t x = row[w];
      const int pc = __popc(x);
      if (pc >= need) {
        for (int q = 1; q < need; q++) x &= x - 1;
        reach = 32 * w + __ffs(x) - 1;
        break;
      }
      need -= pc;
    }
    int e = e0;
    while (e < e1 && (int)(phi[k][e] & 0xFFFF) <= reach) e++;
    if (e == e0) {
      P.phs[i] = 0x7fffffff;
      P.phe[i] = 0;
    } else {
      P.phe[i] = e;
    }
    kept += e - e0;
  }
  const bool entries = __syncthreads_or(kept) != 0;

  // ---- P1c: the kept entries compacted: memo rows' in (class, node)
  // order, then the other rows', in shared memory when they fit.  moff is
  // the variants of the rows before (a variant's row is the last one whose
  // moff is not past it).
  const uint2 *ent = P.ent;
  int nmemo = 0, nvar = 0, E = bd.memo_max;
  auto memo_row = [&](int i, int e) {
    return e >= 1 && e <= E && (1 << e) <= (i < g ? nA : nB) + 8;
  };
  if (entries) {
    // packed: memo entries (14 bits), other entries (20), variants (30)
    constexpr int kO = 14, kV = 34;
    unsigned long long running;
    while (true) {
      running = 0ull;
      for (int i0 = 0; i0 < 2 * g; i0 += nt) {
        const int i = i0 + tid;
        const int e = (i < 2 * g && P.phs[i] < P.phe[i]) ? P.phe[i] - P.phs[i] : 0;
        const bool mr = memo_row(i, e);
        const unsigned long long v =
            mr ? (unsigned long long)e | ((unsigned long long)((1 << e) - 1) << kV)
               : (unsigned long long)e << kO;
        unsigned long long total;
        const unsigned long long off = running + block_scan(v, total, SM.scan64);
        if (i < 2 * g) {
          const int me = (int)(off & ((1u << kO) - 1));
          P.moff[i] = (int)(off >> kV);
          P.nst[i] = mr ? me : (int)((off >> kO) & 0xFFFFF);
          if (i == g) {
            SM.split[0] = me;
            SM.split[1] = P.moff[i];
          }
        }
        running += total;
      }
      nvar = (int)(running >> kV);
      if (nvar <= min(unit_variants(g), bd.words_kept) || E <= 0) break;
      E--;
      __syncthreads();
    }
    nmemo = (int)(running & ((1u << kO) - 1));
    const int nbig = (int)((running >> kO) & 0xFFFFF);
    uint2 *dst = nmemo + nbig <= kEntCache ? P.ent : (uint2 *)(scr + L.ent);
    ent = dst;
    __syncthreads();
    for (int i = tid; i < 2 * g; i += nt) {
      const int e0 = P.phs[i], e1 = P.phe[i];
      if (e0 >= e1) {
        P.phs[i] = P.phe[i] = 0;
        continue;
      }
      const int k = i / g, t = i - k * g, e = e1 - e0;
      const bool mr = memo_row(i, e);
      const int at = P.nst[i] + (mr ? 0 : nmemo);
      for (int q = 0; q < e; q++) {
        const uint32_t x = phi[k][e0 + q];
        dst[at + q] = make_uint2((x & 0xFFFFu) | ((uint32_t)t << 9), x >> 16);
      }
      P.phs[i] = at;
      P.phe[i] = at + e;
      if (!mr) P.big[k * g + atomicAdd(&SM.nbig[k], 1)] = (uint16_t)t;
    }
  } else {
    for (int i = tid; i < 2 * g; i += nt) P.phs[i] = P.phe[i] = 0;
  }
  for (int i = tid; i < (nvar + 31) / 32; i += nt) P.used[i] = 0u;
  __syncthreads();

  // ---- P2: capped lists of the two full networks; their hashes summed per
  // warp, then one atomic per warp and class
  unsigned long long hsum[2] = {0ull, 0ull};
  int csum[2] = {0, 0};
  for (int i = tid; i < 2 * g; i += nt) {
    const int k = i >= g ? 1 : 0, t = i - k * g;
    const uint32_t *row = P.rows + (size_t)i * GW;
    uint64_t h = node_hash_init(sd.salt, t);
    int cnt = 0, last = -1;
    int ps[3] = {0xFFFF, 0xFFFF, 0xFFFF};
    for (int w = 0; w < GW && cnt < sd.mp; w++)
      for (uint32_t x = row[w]; x && cnt < sd.mp; x &= x - 1) {
        last = 32 * w + __ffs(x) - 1;
        if (cnt < 3) ps[cnt] = last;
        h = node_hash_step(h, last);
        cnt++;
      }
    P.fcnt[i] = (uint16_t)cnt;
    P.fend[i] = (int16_t)(cnt < sd.mp ? 0x7FFF : last);
    for (int q = 0; q < 3; q++) P.fps[i * 3 + q] = (uint16_t)ps[q];
    P.fh[i] = h;
    hsum[k] += h;
    csum[k] += cnt;
  }
  if (keep >= 0)
    for (int k = 0; k < 2; k++) {
      const int x = __reduce_add_sync(0xffffffffu, csum[k]);
      if (lane == 0) atomicAdd(&SM.flen[k], x);
    }
  for (int o = 16; o > 0; o >>= 1) {
    hsum[0] += __shfl_xor_sync(0xffffffffu, hsum[0], o);
    hsum[1] += __shfl_xor_sync(0xffffffffu, hsum[1], o);
  }
  if (lane == 0) {
    atomicAdd(&SM.HF[0], hsum[0]);
    atomicAdd(&SM.HF[1], hsum[1]);
  }
  __syncthreads();
  // nodes whose capped lists differ between the full networks
  {
    int nd = 0;
    for (int t = tid; t < g; t += nt) {
      const uint32_t *ra = P.rows + (size_t)t * GW, *rb = P.rows + (size_t)(g + t) * GW;
      bool same = P.fcnt[t] == P.fcnt[g + t];
      int left = P.fcnt[t];
      for (int w = 0; same && w < GW && left > 0; w++) {
        // the words agree up to the column of the last one in the list
        const uint32_t x = ra[w] ^ rb[w];
        uint32_t m = ra[w];
        const int pc = __popc(m);
        if (pc >= left) {
          for (int q = 1; q < left; q++) m &= m - 1;
          same = (x & ((m & -m) | ((m & -m) - 1u))) == 0u;
          left = 0;
        } else {
          same = x == 0u;
          left -= pc;
        }
      }
      P.need[t] = same ? 0 : 1;
      nd += same ? 0 : 1;
    }
    if (nd) atomicAdd(&SM.ndab, nd);
  }

  // ---- the variants of the memo rows: key (node, first three parents)
  // and hash of each list that differs from the full one
  unsigned long long *ment = (unsigned long long *)(scr + L.ment);
  uint16_t *vcnt = (uint16_t *)(scr + L.vcnt);
  unsigned long long *mdh = (unsigned long long *)(scr + L.mdh);
  uint32_t *vinf = (uint32_t *)(scr + L.vinf);
  for (int v = tid; v < nvar; v += nt) {
    int lo = 0, hi = 2 * g - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (P.moff[mid] <= v) lo = mid;
      else hi = mid - 1;
    }
    const int i = lo, k = i >= g ? 1 : 0, t = i - k * g;
    const int sub = v - P.moff[i] + 1;
    const int e0 = P.phs[i], e1 = P.phe[i];
    unsigned long long key = ~0ull, dh = 0ull;
    int len = 0;
    if ((int)(ent[e0 + __ffs(sub) - 1].x & 511u) <= P.fend[i]) {
      const uint32_t *row = P.rows + (size_t)i * GW;
      uint64_t h = node_hash_init(sd.salt, t);
      int cnt = 0, ps[3] = {0xFFFF, 0xFFFF, 0xFFFF};
      int e = e0, col = ent[e0].x & 511;
      for (int w = 0; w < GW && cnt < sd.mp; w++) {
        uint32_t x = row[w];
        while (e < e1 && (col >> 5) == w) {
          if ((sub >> (e - e0)) & 1) x ^= 1u << (col & 31);
          if (++e < e1) col = ent[e].x & 511;
        }
        for (; x && cnt < sd.mp; x &= x - 1) {
          const int j = 32 * w + __ffs(x) - 1;
          if (cnt < 3) ps[cnt] = j;
          h = node_hash_step(h, j);
          cnt++;
        }
      }
      key = list_key(t, cnt, ps);
      len = cnt;
      dh = h - P.fh[i];
      // two lists of a node with one hash: another salt
      if (dh == 0ull) atomicOr(&SM.status, kUnitHashCollision);
    }
    ment[v] = key;
    mdh[v] = dh;
    vinf[v] = variant_info(e0, e1 - e0, sub, dh != 0ull);
    if (keep >= 0) vcnt[v] = (uint16_t)len;
  }
  // sample lists of both classes in index order (network -> left-out
  // sample)
  if (warp == 0) {
    for (int cls = 0; cls < 2; cls++) {
      const uint64_t *m = cls ? P.mB : P.mA;
      int *pc = cls ? P.pcB : P.pcA;
      int run = 0;
      for (int w0 = 0; w0 < W; w0 += 32) {
        int w = w0 + lane;
        int v = (w < W) ? __popcll(m[w]) : 0;
        int x = v;
        for (int o = 1; o < 32; o <<= 1) {
          int y = __shfl_up_sync(0xffffffffu, x, o);
          if (lane >= o) x += y;
        }
        if (w < W) pc[w] = run + x - v;
        run += __shfl_sync(0xffffffffu, x, 31);
      }
    }
  }
  const int nbigs = SM.nbig[0] + SM.nbig[1];
  const int KB = big_slots(g);
  unsigned long long *bkey = (unsigned long long *)(scr + L.bkey);
  if (nbigs)
    for (int i = tid; i < KB; i += nt) bkey[i] = ~0ull;
  __syncthreads();
  const bool networks = entries || keep >= 0;
  if (networks) {
    for (int i = tid; i < 64 * W; i += nt) {
      const int w = i >> 6, bit = i & 63;
      const uint64_t below64 = (bit ? (~0ull >> (64 - bit)) : 0ull);
      const uint64_t a = P.mA[w], b = P.mB[w];
      if ((a >> bit) & 1ull) sig[P.pcA[w] + __popcll(a & below64)] = i;
      else if ((b >> bit) & 1ull) sig[nA + P.pcB[w] + __popcll(b & below64)] = i;
    }
    __syncthreads();
  }

  // a changed node's key (node, first three parents) unless it equals the
  // full network's: the items scored in the BDeu phase
  auto differs = [&](int k, unsigned long long e) -> bool {
    const int t = (int)(e & 0x3FFF), np = (int)((e >> 14) & 3);
    const int i = k * g + t, fnp = P.fcnt[i] < 3 ? P.fcnt[i] : 3;
    if (np != fnp) return true;
    for (int q = 0; q < np; q++)
      if ((int)((e >> (16 + 16 * q)) & 0xFFFF) != (int)P.fps[i * 3 + q]) return true;
    return false;
  };
  // slot of a key in the table of lists formed per sample (-1: no room)
  constexpr int kProbes = 32;
  auto big_slot = [&](unsigned long long key, bool insert) -> int {
    unsigned slot = (unsigned)(mix64(key) & (KB - 1));
    for (int pr = 0; pr < kProbes; pr++, slot = (slot + 1u) & (KB - 1)) {
      // a slot only ever goes from empty to its final key
      unsigned long long cur = insert ? *(volatile unsigned long long *)&bkey[slot] : bkey[slot];
      if (insert && cur == ~0ull) cur = atomicCAS(&bkey[slot], ~0ull, key);
      if (cur == key || (insert && cur == ~0ull)) return (int)slot;
      if (cur == ~0ull) return -1;
    }
    return -1;
  };
  // ---- P3: which variants the left-out samples change their rows to, and
  // which samples have a changed list (both from the trigger words of the
  // entries, 32 samples of a class at a time)
  const int n = sd.n, vsplit = SM.split[1];
  unsigned long long *hs = (unsigned long long *)(scr + L.hs);
  auto as_key = [](unsigned long long h) { return h == ~0ull ? ~1ull : h; };
  uint2 *cpw = (uint2 *)(scr + L.cp);
  const int cw1 = class_words(nA);
  const ClassPlanes cp[2] = {{cpw, g, cw1}, {cpw + (size_t)cw1 * g, g, class_words(nB)}};
  if (networks || SM.ndab) {
    uint32_t *moves = (uint32_t *)(scr + L.moves);
    if (W >= kLongWords) pack_classes<true>(sd, SM.P, moves, cpw);
    else pack_classes<false>(sd, SM.P, moves, cpw);
  }
  uint2 *uv = (uint2 *)(scr + L.uv);
  uint32_t *vw = (uint32_t *)(scr + L.vw);
  const int vws = max(cw1, class_words(nB));
  int nul = 0, ulsplit = 0;
  if (entries) {
    // (the base scores' room behind the work region is free until then)
    if (nvar)
      mark_variants<kThreads>(bd.sm, cp[0], cp[1], nA, nB, ent, vinf, vsplit, nvar, vw, vws,
                    (int)(kWorkBytes + 4 * sizeof(long long) * (size_t)g));
    // the rows formed per sample: their hash differences, and their keys
    // into the table
    for (int s0 = 32 * warp; nbigs && s0 < n; s0 += nt) {
      const int s = 1 + s0 + lane;
      if (s > n) continue;
      const int k = s <= nA ? 0 : 1, sg = sig[s - 1], i = s - 1 - (k ? nA : 0);
      unsigned long long dh = 0ull;
      bool chg = false;
      for (int r = 0; r < SM.nbig[k]; r++) {
        const int t = P.big[k * g + r];
        unsigned long long key, h;
        int len;
        if (!sample_list(sd, SM.P, ent, k, t, sg, key, h, len)) continue;
        const unsigned long long d = h - P.fh[k * g + t];
        if (d == 0ull) atomicOr(&SM.status, kUnitHashCollision);
        dh += d;
        chg = true;
        if (differs(k, key)) big_slot(key, true);
      }
      hs[s] = dh;
      if (chg) atomicOr(&P.chg[(k ? cw1 : 0) + (i >> 5)], 1u << (i & 31));
    }
    __syncthreads();
    // changed networks, the first unchanged one of class 2
    for (int i = tid; i < cw1 + class_words(nB); i += nt) {
      const uint32_t x = P.chg[i];
      if (x) atomicAdd(&SM.nchg, __popc(x));
      const int at = 32 * (i - cw1), left = nB - at;
      if (at < 0 || left <= 0) continue;
      const uint32_t same = ~x & (left >= 32 ? ~0u : (1u << left) - 1u);
      if (same) atomicMin(&SM.firstB0, 1 + nA + at + __ffs(same) - 1);
    }
    // the used variants in order
    for (int w0 = 0; w0 < (nvar + 31) >> 5; w0 += nt) {
      const int w = w0 + tid;
      const uint32_t word = w < (nvar + 31) >> 5 ? P.used[w] : 0u;
      int total;
      int at = nul + block_scan(__popc(word), total, SM.scan);
      for (uint32_t x = word; x; x &= x - 1) {
        const int v = 32 * w + __ffs(x) - 1;
        uv[at++] = make_uint2((unsigned)v, vinf[v]);
      }
      nul += total;
    }
    __syncthreads();
    int hi = nul;  // class 1's
    while (ulsplit < hi) {
      const int mid = (ulsplit + hi) >> 1;
      if ((int)uv[mid].x < vsplit) ulsplit = mid + 1;
      else hi = mid;
    }
  } else {
    if (tid == 0) SM.firstB0 = nA + 1;  // the first class-2 network
    __syncthreads();
  }
  const int firstB0 = SM.firstB0;

  auto report = [&](int U) {
    if (tid != 0) return;
    bd.js[u] = __longlong_as_double(0x7ff8000000000000ll);
    bd.U[u] = SM.status ? -1 : U;
    bd.status[u] = SM.status;
  };
  // one network has no JS (the range of its scores is empty), whatever its
  // score is
  if ((SM.nchg == 0 && !SM.ndab && keep < 0) || SM.status) {
    report(1);
    return;
  }

  // ---- P4: BDeu.  The JS takes only differences of the networks' scores,
  // so the nodes that every network scores alike are left out (unless the
  // scores themselves are kept): needed are the nodes whose full lists
  // differ between the classes and those of rows with entries.
  for (int i = tid; i < g * 3; i += nt) {
    // state counts per class from the word-major planes: a warp's loads of
    // a word are 32 consecutive planes
    const uint64_t *pl = sd.planesT + i;
    int a = 0, b = 0;
    for (int w = 0; w < W; w++) {
      const uint64_t x = pl[(size_t)w * 3 * g];
      a += __popcll(x & P.mA[w]);
      b += __popcll(x & P.mB[w]);
    }
    P.cnt3[i] = (uint16_t)a;
    P.cnt3[3 * g + i] = (uint16_t)b;
  }
  __syncthreads();
  for (int i = tid; i < 2 * g; i += nt) {
    const uint16_t *c3 = P.cnt3 + 3 * i;
    P.nobs[i] = (uint8_t)((c3[0] > 0) + (c3[1] > 0) + (c3[2] > 0));
  }
  for (int t = tid; t < g; t += nt)
    if (keep >= 0 || P.need[t] || P.phs[t] < P.phe[t] || P.phs[g + t] < P.phe[g + t]) P.need[t] |= 2;
  __syncthreads();
  // the keys to score, all in one list: the needed nodes' lists in the two
  // full networks (a class-2 node whose first parents equal the class-1
  // one's has its scores), then the used variants' distinct keys, then the
  // keys of the lists formed per sample.  A table in the work region (free
  // until the scores) gives each key its first variant: 38 bits of key (genes
  // below 512) and 16 of the variant a slot.  A variant that finds no room is
  // scored on its own.  (Scored in two rounds, the full networks' first, a
  // small unit's waits came twice: one labelling of 20 genes x 200 samples
  // 55 us in the unit kernel for 52.)
  auto same_as_class1 = [&](int t) -> bool {
    const int a = P.fcnt[t] < 3 ? P.fcnt[t] : 3, b = P.fcnt[g + t] < 3 ? P.fcnt[g + t] : 3;
    if (a != b) return false;
    for (int q = 0; q < a; q++)
      if (P.fps[t * 3 + q] != P.fps[(g + t) * 3 + q]) return false;
    return true;
  };
  longlong2 *msc = (longlong2 *)(scr + L.msc);
  longlong2 *bsc = (longlong2 *)(scr + L.bsc);
  uint16_t *vcan = (uint16_t *)(scr + L.vcan), *sel = (uint16_t *)(scr + L.sel);
  unsigned long long *ikey = (unsigned long long *)(scr + L.ikey);
  longlong2 *isc = (longlong2 *)(scr + L.isc);
  int *bpos = (int *)(scr + L.bpos);
  int nsel = 0, nbk = 0;
  for (int i = tid; i < 2 * g; i += nt) {
    const int k = i >= g ? 1 : 0, t = i - k * g;
    const int ps[3] = {P.fps[i * 3], P.fps[i * 3 + 1], P.fps[i * 3 + 2]};
    ikey[i] = (P.need[t] & 2) && !(k == 1 && same_as_class1(t)) ? list_key(t, P.fcnt[i], ps) : ~0ull;
  }
  if (SM.nchg) {
    constexpr int kKeySlots = 2048;
    static_assert(kKeySlots * sizeof(unsigned long long) <= kWorkBytes, "key table");
    unsigned long long *kt = P.itk;
    int slots = 64;
    while (slots < 2 * nul && slots < kKeySlots) slots <<= 1;
    for (int i = tid; i < slots; i += nt) kt[i] = ~0ull;
    __syncthreads();
    for (int q = tid; q < nul; q += nt) {
      const int v = (int)uv[q].x;
      const unsigned long long key = ment[v];
      if (!differs(v >= vsplit ? 1 : 0, key)) {
        msc[v] = make_longlong2(0, 0);
        vcan[v] = (uint16_t)v;
        continue;
      }
      const unsigned long long k38 = (key & 511u) | (((key >> 14) & 3u) << 9) |
                                     (((key >> 16) & 511u) << 11) | (((key >> 32) & 511u) << 20) |
                                     (((key >> 48) & 511u) << 29);
      int can = v;
      unsigned slot = (unsigned)(mix64(k38) & (slots - 1));
      for (int pr = 0; pr < 32; pr++, slot = (slot + 1u) & (slots - 1)) {
        unsigned long long cur = *(volatile unsigned long long *)&kt[slot];
        if (cur == ~0ull) cur = atomicCAS(&kt[slot], ~0ull, (k38 << 16) | (unsigned)v);
        if (cur == ~0ull) break;
        if (cur >> 16 == k38) {
          can = (int)(cur & 0xFFFFu);
          break;
        }
      }
      vcan[v] = (uint16_t)can;
      if (can == v) {
        const int at = atomicAdd(&SM.nsel, 1);
        sel[at] = (uint16_t)v;
        ikey[2 * g + at] = key;
      }
    }
    __syncthreads();
    nsel = SM.nsel;
    for (int i0 = 0; nbigs && i0 < KB; i0 += nt) {
      const bool has = i0 + tid < KB && bkey[i0 + tid] != ~0ull;
      int total;
      const int off = block_scan(has ? 1 : 0, total, SM.scan);
      if (has) {
        bpos[nbk + off] = i0 + tid;
        ikey[2 * g + nsel + nbk + off] = bkey[i0 + tid];
      }
      nbk += total;
    }
  }
  __syncthreads();
  bdeu_items(bd.sm, cp[0], cp[1], 2 * g + nsel + nbk, ikey, isc);
  for (int i = tid; i < 2 * g; i += nt) {
    const int k = i >= g ? 1 : 0, t = i - k * g;
    const longlong2 x = isc[k == 1 && same_as_class1(t) ? t : i];
    P.fsc[(k * 2 + 0) * g + t] = x.x;
    P.fsc[(k * 2 + 1) * g + t] = x.y;
  }
  __syncthreads();
  if (warp < 4) {
    // warp 2 k + cls: the sum of full network k's scores over class cls
    long long s = 0;
    for (int t = lane; t < g; t += 32) s += P.fsc[warp * g + t];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) SM.base[warp & 1][warp >> 1] = s;
  }
  if (SM.nchg) {
    for (int i = tid; i < nsel + nbk; i += nt) {
      const longlong2 x = isc[2 * g + i];
      if (i < nsel) {
        const int v = sel[i], k = v >= vsplit ? 1 : 0, t = (int)(ikey[2 * g + i] & 0x3FFF);
        msc[v] = make_longlong2(x.x - P.fsc[(k * 2 + 0) * g + t], x.y - P.fsc[(k * 2 + 1) * g + t]);
      } else {
        bsc[bpos[i - nsel]] = x;
      }
    }
    __syncthreads();
    for (int q = tid; q < nul; q += nt) {
      const int v = (int)uv[q].x, c = vcan[v];
      if (c == v) continue;
      // the same list of the same node, in either class
      const int t = (int)(ment[v] & 0x3FFF), k = v >= vsplit ? 1 : 0, kc = c >= vsplit ? 1 : 0;
      longlong2 x = msc[c];
      x.x += P.fsc[(kc * 2 + 0) * g + t] - P.fsc[(k * 2 + 0) * g + t];
      x.y += P.fsc[(kc * 2 + 1) * g + t] - P.fsc[(k * 2 + 1) * g + t];
      msc[v] = x;
    }
  }
  __syncthreads();
  // ---- P5: the networks' hashes and scores, less their class's full one's
  longlong2 *xs = (longlong2 *)(scr + L.xs);
  int *dc = (int *)(scr + L.dc);
  if (SM.nchg)
    for (int k = 0; k < 2; k++) {
      const int nk = k ? nB : nA, s1 = 1 + (k ? nA : 0);
      const uint2 *u = uv + (k ? ulsplit : 0);
      const int nu = k ? nul - ulsplit : ulsplit;
      const uint32_t *chg = P.chg + (k ? cw1 : 0);
      const uint16_t *fc = P.fcnt + k * g;
      const unsigned long long HF = SM.HF[k];
      const bool big = nbigs > 0;
      auto put = [=](int i, const unsigned long long *x) {
        const int s = s1 + i;
        const bool c = ((chg[i >> 5] >> (i & 31)) & 1u) != 0u;
        const unsigned long long h = HF + x[0] + (big ? hs[s] : 0ull);
        hs[s] = !c ? ~0ull : h == ~0ull ? ~1ull : h;
        xs[s] = make_longlong2((long long)x[1], (long long)x[2]);
        if (keep >= 0) dc[s] = (int)x[3];
      };
      auto word = [=](int i, int w) -> uint32_t {
        return vw[(size_t)u[i].x * vws + w];
      };
      auto value = [=](int i, int j) -> unsigned long long {
        const int v = (int)u[i].x;
        if (j == 0) return mdh[v];
        if (j < 3) return (unsigned long long)reinterpret_cast<const long long *>(msc + v)[j - 1];
        return (unsigned long long)((long long)vcnt[v] - fc[(int)(ment[v] & 0x3FFF)]);
      };
      if (nu <= kFewVariants) {
        // few: a lane per sample adds up its own
        for (int i = tid; i < nk; i += nt) {
          unsigned long long x[4] = {0ull, 0ull, 0ull, 0ull};
          for (int q = 0; q < nu; q++)
            if ((word(q, i >> 5) >> (i & 31)) & 1u)
              for (int j = 0; j < (keep < 0 ? 3 : 4); j++) x[j] += value(q, j);
          put(i, x);
        }
      } else if (keep < 0) {
        unit_walk<kThreads, 3>(bd.sm.itk, nk, nu, word, value, put);
      } else {
        unit_walk<kThreads, 4>(bd.sm.itk, nk, nu, word, value, put);
      }
    }
  __syncthreads();

  // ---- P6: first-occurrence dedup.  Networks without changed nodes are
  // their class's full network: class-1 ones duplicate network 0, class-2
  // ones the first of them (firstB0).  So the unique networks are the
  // candidates -- network 0, firstB0 and the changed networks -- that are
  // the first occurrence of their hash: a table of network ids, compared by
  // hash, keeps the smallest id of each.
  int *urep = (int *)(scr + L.urep);
  int *wl = (int *)(scr + L.wl), *vrep = (int *)(scr + L.vrep);
  int U;
  if (SM.nchg == 0) {
    U = SM.ndab ? 2 : 1;
    if (tid == 0) {
      urep[0] = 0;
      if (U == 2) urep[1] = firstB0;
    }
    __syncthreads();
  } else {
    int slots = 64;
    while (slots < 2 * (SM.nchg + 2)) slots <<= 1;
    int *tab = slots <= kSmSlots ? (int *)P.itk : (int *)(scr + L.htab);
    const unsigned tmask = (unsigned)slots - 1u;
    uint32_t *ubits = (uint32_t *)(scr + L.ubits);
    const int nbw = (S + 31) >> 5;
    for (int i = tid; i < slots; i += nt) tab[i] = -1;
    for (int i = tid; i < nbw; i += nt) ubits[i] = 0u;
    if (tid == 0) {
      hs[0] = as_key(SM.HF[0]);
      hs[firstB0] = as_key(SM.HF[1]);
      if (firstB0 != S - 1) hs[S - 1] = ~0ull;
    }
    __syncthreads();
    for (int s = tid; s < S; s += nt) {
      const unsigned long long key = hs[s];
      if (key == ~0ull) continue;
      for (unsigned slot = (unsigned)(mix64(key) & tmask);; slot = (slot + 1u) & tmask) {
        int cur = *(volatile int *)&tab[slot];
        if (cur < 0) {
          cur = atomicCAS(&tab[slot], -1, s);
          if (cur < 0) break;
        }
        if (hs[cur] == key) {
          atomicMin(&tab[slot], s);
          break;
        }
      }
    }
    __syncthreads();
    for (int s = tid; s < S; s += nt) {
      const unsigned long long key = hs[s];
      if (key == ~0ull) continue;
      unsigned slot = (unsigned)(mix64(key) & tmask);
      int r = tab[slot];
      while (hs[r] != key) r = tab[slot = (slot + 1u) & tmask];
      if (r == s) {
        atomicOr(&ubits[s >> 5], 1u << (s & 31));
      } else {
        // merged by hash: checked list by list below
        const int q = atomicAdd(&SM.nver, 1);
        wl[q] = s;
        vrep[q] = r;
      }
    }
    __syncthreads();
    // unique networks in network order: the set bits before each one
    int running = 0;
    for (int w0 = 0; w0 < nbw; w0 += nt) {
      const int w = w0 + tid;
      const uint32_t word = w < nbw ? ubits[w] : 0u;
      int total;
      const int off = block_scan(__popc(word), total, SM.scan);
      int at = running + off;
      for (uint32_t x = word; x; x &= x - 1) urep[at++] = 32 * w + __ffs(x) - 1;
      running += total;
    }
    U = running;
    __syncthreads();
    // exact check of every hash merge, a lane per merged network: in one
    // class the rows' triggered entries agree, or else their lists do; in
    // two, the lists of all nodes
    const int nver = SM.nver;
    for (int wi = tid; wi < nver; wi += nt) {
      const int s = wl[wi], r = vrep[wi];
      int ks, ss, kr, sr;
      net_of(s, sd, sig, ks, ss);
      net_of(r, sd, sig, kr, sr);
      // a network without changes is compared as its class's full network
      if (s == firstB0) ss = -1;
      if (r == firstB0) sr = -1;
      bool ok = true;
      if (ks == kr && ss >= 0 && sr >= 0) {
        const uint32_t *ca = sd.codes + (ss >> 4), *cb = sd.codes + (sr >> 4);
        const int ha = 2 * (ss & 15), hb = 2 * (sr & 15), n16 = sd.n16;
        auto agree = [&](uint2 en) {
          const uint32_t t = (en.x >> 9) & 511u, j = en.x & 511u;
          const uint32_t a = 4u * ((ca[t * n16] >> ha) & 3u) + ((ca[j * n16] >> ha) & 3u);
          const uint32_t b = 4u * ((cb[t * n16] >> hb) & 3u) + ((cb[j * n16] >> hb) & 3u);
          return (((en.y >> a) ^ (en.y >> b)) & 1u) == 0u;
        };
        auto row = [&](int t) { return lists_equal(sd, SM.P, ent, t, ks, ss, kr, sr); };
        // the class's memo entries in a flat walk (a row that disagrees is
        // compared once: the walk goes on behind it), then the other rows
        const int e1 = ks ? nmemo : SM.split[0];
        for (int e = ks ? SM.split[0] : 0; ok && e < e1; e++) {
          const uint2 en = ent[e];
          if (agree(en)) continue;
          const int t = (en.x >> 9) & 511;
          ok = row(t);
          e = P.phe[ks * g + t] - 1;
        }
        for (int q = 0; ok && q < SM.nbig[ks]; q++) ok = row(P.big[ks * g + q]);
      } else if (ks != kr && ss < 0 && sr < 0) {
        ok = SM.ndab == 0;  // the two full networks
      } else {
        // (a row without entries has its class's full list, the same in both
        // classes but for the nodes marked)
        for (int t = 0; ok && t < g; t++) {
          if (P.phs[ks * g + t] >= P.phe[ks * g + t] && P.phs[kr * g + t] >= P.phe[kr * g + t] &&
              (ks == kr || !(P.need[t] & 1)))
            continue;
          ok = lists_equal(sd, SM.P, ent, t, ks, ss, kr, sr);
        }
      }
      if (!ok) atomicOr(&SM.status, kUnitHashCollision);
    }
    __syncthreads();
  }
  report(U);
  if ((U == 1 && keep < 0) || SM.status) return;

  // unique networks: base of their class plus the differences, and those of
  // the rows formed per sample
  for (int uu = tid; uu < U; uu += nt) {
    const int s = urep[uu], k = s <= nA ? 0 : 1;
    long long d1 = SM.base[0][k], d2 = SM.base[1][k];
    int edges = SM.flen[k];
    if (s != 0 && s != firstB0) {
      const longlong2 x = xs[s];
      d1 += x.x;
      d2 += x.y;
      if (keep >= 0) edges += dc[s];
      for (int r = 0; r < SM.nbig[k]; r++) {
        const int t = P.big[k * g + r];
        unsigned long long key, h;
        int len;
        if (!sample_list(sd, SM.P, ent, k, t, sig[s - 1], key, h, len)) continue;
        edges += len - P.fcnt[k * g + t];
        if (!differs(k, key)) continue;
        const int slot = big_slot(key, false);
        long long sc[2];
        if (slot >= 0) {
          sc[0] = bsc[slot].x;
          sc[1] = bsc[slot].y;
        } else {
          key_scores(sd, SM.P, cp, key, sc);  // the table had no room
        }
        d1 += sc[0] - P.fsc[(k * 2 + 0) * g + t];
        d2 += sc[1] - P.fsc[(k * 2 + 1) * g + t];
      }
    }
    dist[uu] = d1;
    dist[S + uu] = d2;
    if (keep >= 0) wl[uu] = edges;
  }

  __syncthreads();
  // ---- P7: detailed outputs of kept units, packed: a region of the
  // batch's buffer, its edge ranges and the full networks' edge lists;
  // k_pack writes the unique networks' lists
  double *pl = nullptr, *ql = nullptr;
  if (keep >= 0) {
    // edge ranges (in place), and the uncapped rows' counts
    int E = 0, E2 = 0;
    for (int u0 = 0; u0 < U; u0 += nt) {
      int total;
      const int off = block_scan(u0 + tid < U ? wl[u0 + tid] : 0, total, SM.scan);
      if (u0 + tid < U) wl[u0 + tid] = E + off;
      E += total;
    }
    auto row_edges = [&](int i) {
      int x = 0;
      for (int w = 0; w < GW; w++) x += __popc(P.rows[(size_t)i * GW + w]);
      return x;
    };
    for (int i0 = 0; i0 < 2 * g; i0 += nt) {
      const int i = i0 + tid;
      int total;
      const int off = block_scan(i < 2 * g ? row_edges(i) : 0, total, SM.scan);
      if (i < 2 * g) P.nst[i] = E2 + off;
      E2 += total;
    }
    __syncthreads();
    const int E2a = P.nst[g];
    const KeepLayout KL = keep_layout(g, U, E, E2);
    if (tid == 0) {
      SM.koff = atomicAdd(&bd.kmeta[0].off, (unsigned long long)KL.words);
      KeepMeta m;
      m.off = SM.koff;
      m.U = U;
      m.E = E;
      m.E2 = E2;
      m.E2a = E2a;
      m.u = SM.koff + KL.words <= bd.kcap ? u + 1 : 0;
      m.pad_ = 0;
      bd.kmeta[1 + keep] = m;
    }
    __syncthreads();
    if (SM.koff + KL.words > bd.kcap) {
      // (the host makes room for the words counted and runs the unit again)
      if (tid == 0) {
        bd.U[u] = -1;
        bd.status[u] = kUnitKeepFull;
      }
      return;
    }
    uint8_t *kb = reinterpret_cast<uint8_t *>(bd.kbuf + SM.koff);
    int *ids = (int *)(kb + KL.ids), *epn = (int *)(kb + KL.epn);
    int *lnodes = (int *)(kb + KL.lnodes), *ledges = (int *)(kb + KL.ledges);
    double *kd = (double *)(kb + KL.dist);
    const double fx = ldexp(1.0, -sd.lg_shift);
    for (int uu = tid; uu < U; uu += nt) {
      ids[uu] = urep[uu];
      epn[uu] = wl[uu];
      kd[uu] = (double)dist[uu] * fx;
      kd[U + uu] = (double)dist[S + uu] * fx;
    }
    if (tid == 0) epn[U] = E;
    for (int i = tid; i < 2 * g; i += nt) {
      const int at = P.nst[i];
      lnodes[i] = at - (i >= g ? E2a : 0);
      int q = at;
      for (int w = 0; w < GW; w++)
        for (uint32_t x = P.rows[(size_t)i * GW + w]; x; x &= x - 1) ledges[q++] = 32 * w + __ffs(x) - 1;
    }
    // what k_pack reads: the rows, the entry ranges and the entries
    uint32_t *kr = (uint32_t *)(scr + L.krow);
    for (int i = tid; i < 2 * g * GW; i += nt) kr[i] = P.rows[i];
    for (int i = tid; i < 4 * g; i += nt) kr[2 * g * GW + i] = (uint32_t)P.phs[i];
    if (ent == P.ent) {
      int n = nmemo;
      for (int k = 0; k < 2; k++)
        for (int r = 0; r < SM.nbig[k]; r++) n = max(n, P.phe[k * g + P.big[k * g + r]]);
      uint2 *dst = (uint2 *)(scr + L.ent);
      for (int i = tid; i < n; i += nt) dst[i] = P.ent[i];
    }
    pl = (double *)(kb + KL.lval);
    ql = pl + U;
    __syncthreads();
  }

  // ---- P8: normalisation and JS
  if (tid == 0) SM.cycles[1] -= clock64();
  const double js = unit_js(dist, S, U, SM, pl, ql);
  if (tid == 0) {
    SM.cycles[1] += clock64();
    bd.js[u] = js;
  }
}

// A block per place on the GPU, each unit taken when a block is free, so that
// a batch holds the scratch of those blocks only (1.5 GB for 33 GB at 10000
// units of 200 genes x 1000 samples; as fast as a block and a scratch per unit,
// 14.9 ms for 15.0).  The layouts, computed on the host, come with the
// parameters: with each block's own (every thread's, before) 14.9 ms against
// 12.0, 19.7 against 16.6 ms for 2000 small sets.
template <int kThreads>
__global__ void __maxnreg__(kUnitRegs) k_units(const __grid_constant__ BatchDev bd) {
  UnitSmem &SM = *reinterpret_cast<UnitSmem *>(unit_smem);
  int turn = 0;
  if (threadIdx.x == 0) {
    SM.cycles[0] = -clock64();
    SM.cycles[1] = 0;
  }
  for (int u = blockIdx.x; u < bd.B; turn ^= 1) {
    int next = bd.B;
    if (threadIdx.x == 0 && (int)gridDim.x < bd.B) next = (int)(gridDim.x + atomicAdd(bd.taken, 1u));
    run_unit<kThreads>(bd, u, unit_smem);
    if (threadIdx.x == 0) SM.next[turn] = next;
    __syncthreads();
    u = SM.next[turn];
  }
  if (threadIdx.x == 0 && bd.cycles) {
    atomicAdd(bd.cycles, (unsigned long long)(SM.cycles[0] + clock64()));
    atomicAdd(bd.cycles + 1, (unsigned long long)SM.cycles[1]);
  }
}

// The unique networks' capped parent lists of the kept units (their edge
// positions and edges in the packed outputs), a warp per network: in the
// unit's own block they took 2.3 ms for 1000 networks of 200 genes.
__global__ void __launch_bounds__(256) k_pack(const __grid_constant__ BatchDev bd) {
  const KeepMeta km = bd.kmeta[1 + blockIdx.x];
  if (km.u == 0) return;
  const int u = km.u - 1, lane = threadIdx.x & 31, wpg = (blockDim.x >> 5) * gridDim.y;
  const BatchSet &bs = bd.sets[bd.uslot[u]];
  const SetDev &sd = bs.sd;
  const int g = sd.g, GW = sd.GW;
  uint8_t *scr = bd.scratch + (size_t)(bd.blocks + (int)blockIdx.x) * bd.lay.total;
  const UnitLayout &L = bd.lay;
  const KeepLayout KL = keep_layout(g, km.U, km.E, km.E2);
  uint8_t *kb = reinterpret_cast<uint8_t *>(bd.kbuf + km.off);
  const int *ids = (const int *)(kb + KL.ids), *epn = (const int *)(kb + KL.epn);
  int *nodes = (int *)(kb + KL.nodes), *edges = (int *)(kb + KL.edges);
  const int *sig = (const int *)(scr + L.sig);
  const uint2 *ent = (const uint2 *)(scr + L.ent);
  UnitPtrs P{};
  P.rows = (uint32_t *)(scr + L.krow);
  P.phs = (int *)(P.rows + 2 * g * GW);
  P.phe = P.phs + 2 * g;
  // fn(j) for the parents of node t, in order, in the network of left-out
  // sample sigma of class k
  auto parents = [&](int k, int t, int sigma, auto &&fn) {
    const int i = k * g + t;
    int cnt = 0;
    if (sigma < 0 || P.phs[i] >= P.phe[i]) {
      const uint32_t *row = P.rows + (size_t)i * GW;
      for (int w = 0; w < GW && cnt < sd.mp; w++)
        for (uint32_t x = row[w]; x && cnt < sd.mp; x &= x - 1, cnt++) fn(32 * w + __ffs(x) - 1);
    } else {
      ListGen G;
      gen_for(G, sd, P, ent, k, t, sigma);
      for (int j; cnt < sd.mp && (j = G.next()) >= 0; cnt++) fn(j);
    }
    return cnt;
  };
  for (int uu = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5); uu < km.U; uu += wpg) {
    int k, sigma, run = 0;
    net_of(ids[uu], sd, sig, k, sigma);
    int *dst = edges + epn[uu];
    for (int t0 = 0; t0 < g; t0 += 32) {
      const int t = t0 + lane;
      const int cnt = t < g ? parents(k, t, sigma, [](int) {}) : 0;
      int incl = cnt;
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      if (t < g) {
        const int at = run + incl - cnt;
        nodes[(size_t)uu * g + t] = at;
        int q = at;
        parents(k, t, sigma, [&](int j) { dst[q++] = j; });
      }
      run += __shfl_sync(0xffffffffu, incl, 31);
    }
  }
}

// ------------------------------------------------------------ launchers
// A kernel's limit of dynamic shared memory belongs to the process: every
// launcher sets the largest value any of its launches can need, and the same
// one each time, so a launch of one thread fits whatever another thread
// launches meanwhile.  (It is a limit only: a launch takes what it asks for.)
cudaError_t launch_prep(const PrepSet *sets, int ns, int genes, int pair_blocks, const int8_t *vals,
                        const int32_t *rows, int n, int W, uint64_t *valid, cudaStream_t st) {
  if (genes <= 0) return cudaSuccess;
  k_planes<<<(genes + 3) / 4, 128, 0, st>>>(sets, ns, genes, vals, rows, n, W, valid);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  if (pair_blocks > 0) k_ctot<<<pair_blocks, 128, 0, st>>>(sets, ns, W);
  return cudaGetLastError();
}

cudaError_t launch_counter_masks(int n, int nA, int W, uint64_t seed, const int32_t *unit_set,
                                 const int32_t *unit_perm, const uint64_t *mask0, uint64_t *masks,
                                 int B, cudaStream_t st) {
  const size_t smem = sizeof(uint32_t) * kCmWarps * (size_t)cm_words(n);
  if (n > kCmMaxSamples) return cudaErrorInvalidValue;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(k_counter_masks, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)sizeof(uint32_t) * kCmWarps * cm_words(kCmMaxSamples));
    if (e != cudaSuccess) return e;
  }
  k_counter_masks<<<(B + kCmWarps - 1) / kCmWarps, 32 * kCmWarps, smem, st>>>(n, nA, W, seed, unit_set,
                                                                              unit_perm, mask0, masks, B);
  return cudaGetLastError();
}

cudaError_t launch_pairs(const BatchSet *sets, const int32_t *uslot, const uint64_t *masks,
                         uint32_t *dmask, int B, int W, int gmax, int sms, bool exact_all,
                         unsigned long long *stats, cudaStream_t st) {
  if (gmax < 2) return cudaSuccess;
  const int t = (gmax + kPairTile - 1) / kPairTile;
  const dim3 grid(t * (t + 1) / 2, B);
  const long long tiles = (long long)grid.x * B;
  // grid.y holds at most 65535 units (a batch has at most 32768)
  // A block's time is a chain over the sample words, then over its warps'
  // rows (their general and exact decisions above all), so while the quarters
  // or halves of all tiles fit on the GPU together they are quicker: one tile
  // of 100 samples, most tables on the general path, 0.060 / 0.035 / 0.021 ms
  // (whole, halves, quarters), of 10000 samples 0.096 / 0.071 / 0.054, of
  // 65000 with exact decisions 1.71 / 0.96 / 0.59; 112 tiles of 10000 samples
  // 0.097 / 0.079 / 0.093, 448 0.199 / 0.212 / 0.236.  (The figures of general
  // and exact decisions are from before the block shared them.)  Where every
  // decision is exact, a tile is FP64 work for one SM and quarters spread it
  // better however many there are: 10 units of 120 genes x 150 samples 3.26
  // -> 2.03 ms a call, 700 of 60 x 400 32.6 -> 30.8, of 200 x 1000 404 -> 402.
  const auto launch = [&](auto *kernel, int parts) {
    kernel<<<dim3(grid.x, grid.y, parts), 32 * kPairWarps, 0, st>>>(sets, uslot, masks, W, dmask, stats);
  };
  if (4 * tiles <= 2 * sms || exact_all) launch(k_pairs<1>, 4);
  else if (2 * tiles <= 2 * sms) launch(k_pairs<2>, 2);
  else launch(k_pairs<4>, 1);
  return cudaGetLastError();
}

constexpr int kSmBytes = 227 << 10;  // a block's most
void plan_units(BatchDev &bd, int gmax, double pairs, int n, int sms, size_t words) {
  const int c = gmax * (gmax - 1) / 2;
  bd.words_kept = words_kept(c, n + 2, words);
  bd.lay = unit_layout(c, n + 2, bd.words_kept);
  bd.sm = unit_slices(gmax, (n + 63) / 64);
  // a block per place on the GPU (an SM: 227 KB of shared memory, 1 KB a
  // block of it the system's, and 64 K registers)
  // Where shared memory leaves room for fewer than three blocks of 256
  // threads (sets above about 240 genes), blocks of 384 give an SM more
  // warps: 24 for 16 where two blocks fit (up to about 380 genes), 12 for 8
  // where one does.  n = 600, 3000 units of 245 / 300 / 378 genes (two
  // blocks) 5.85 -> 5.07, 9.17 -> 7.73, 14.7 -> 11.9 ms, of 387 / 512 (one)
  // 22.6 -> 17.6, 38.8 -> 29.8; 301 units of 387 genes 2.43 -> 1.87.  With
  // three blocks the registers are full already, and blocks of 384 come two
  // an SM: 230 genes 4.67 -> 4.76, 200 x 1000 12.2 -> 13.4.  A batch of mostly
  // smaller sets keeps 256, which suits its units (150 co-expressed sets of
  // 8-250 genes 24.8 ms, with 384 25.5).
  const int fit = kSmBytes / (int)(bd.sm.total + 1024), warps = 65536 / (kUnitRegs * 32);
  bd.threads = fit < 3 && 2.0 * pairs >= (double)bd.B * c ? 384 : 256;
  bd.blocks = std::min(bd.B, std::max(1, std::min(fit, 32 * warps / bd.threads)) * sms);
}

template <int kThreads>
static cudaError_t launch_units_of(const BatchDev &bd, cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute(k_units<kThreads>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       kSmBytes);
  if (e != cudaSuccess) return e;
  k_units<kThreads><<<bd.blocks, kThreads, bd.sm.total, st>>>(bd);
  return cudaGetLastError();
}
cudaError_t launch_units(const BatchDev &bd, cudaStream_t st) {
  return bd.threads == 384 ? launch_units_of<384>(bd, st) : launch_units_of<256>(bd, st);
}

cudaError_t launch_pack(const BatchDev &bd, int kept, int S, cudaStream_t st) {
  if (kept <= 0) return cudaSuccess;
  k_pack<<<dim3(kept, std::min(64, (S + 7) / 8)), 256, 0, st>>>(bd);
  return cudaGetLastError();
}

cudaError_t set_divisor_map(const int8_t *map82) {
  return cudaMemcpyToSymbol(c_dmap, map82, 82);
}

}  // namespace eddy
