// eddy_kernels.h -- host-callable launchers of the sm_103a kernels.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "eddy_internal.h"

namespace eddy {
// A unit's scratch, with `words` bytes at most of its variants' sample words
// (4 MB hold all of them up to 387 genes x 900 samples).
constexpr size_t kVariantWords = (size_t)4 << 20;
size_t unit_scratch_bytes(int c, int S, size_t words = kVariantWords);
constexpr int kMemoMax = 8;  // BatchDev::memo_max unless lowered
// State planes, packed states and full-sample tables of the sets of a table
// on the device (genes and pair_blocks: of all of them).
cudaError_t launch_prep(const PrepSet *sets, int ns, int genes, int pair_blocks, const int8_t *vals,
                        const int32_t *rows, int n, int W, uint64_t *valid, cudaStream_t st);
constexpr int prep_pair_blocks(int c) { return (c + 127) / 128; }
cudaError_t launch_counter_masks(int n, int nA, int W, uint64_t seed, const int32_t *unit_set,
                                 const int32_t *unit_perm, const uint64_t *mask0, uint64_t *masks,
                                 int B, cudaStream_t st);
// Popcount contingency and decision kernel for a batch (sets: its device
// set table, uslot: each unit's set; gmax: the largest set; sms: the GPU's SMs;
// exact_all: every set decides in FP64 throughout).
cudaError_t launch_pairs(const BatchSet *sets, const int32_t *uslot, const uint64_t *masks,
                         uint32_t *dmask, int B, int W, int gmax, int sms, bool exact_all,
                         unsigned long long *stats, cudaStream_t st);
// Network, BDeu and JS kernel of a batch; before, its layouts and blocks
// (bd.B units of `pairs` pairs together, the largest set of gmax genes, n
// samples).
void plan_units(BatchDev &bd, int gmax, double pairs, int n, int sms, size_t words = kVariantWords);
cudaError_t launch_units(const BatchDev &bd, cudaStream_t st);
// Lists of the kept units' unique networks, after launch_units (S: networks).
cudaError_t launch_pack(const BatchDev &bd, int kept, int S, cudaStream_t st);
cudaError_t set_divisor_map(const int8_t *map82);
}  // namespace eddy
