// The stable radix passes of k_sort.cu, for the entries built on them.
#pragma once

#include "vkc_internal.h"

namespace vkc {

// Exclusive scan of m u32 counts into out, with scan_counts_sum_words(m) words of scratch in sums.
int64_t scan_counts_sum_words(int64_t m);
void scan_counts(vkc_ctx *ctx, const unsigned *c, int64_t m, unsigned *sums, unsigned *out);

// Scratch tables of a pass: radix_table_words(n) words each.
struct RadixTables {
    unsigned *counts, *offs, *sums;
};
void radix_table_words(int64_t n, int64_t *count_words, int64_t *sum_words);

// Images and payloads of n rows: the first pass reads img_first and pay_first, the others the buffer
// the pass before wrote (the first one writes buffer 0).
template <class IMG, class PAY> struct RadixPairs {
    const IMG *img_first;
    const PAY *pay_first;
    IMG *img[2];
    PAY *pay[2];
};
// One stable pass per entry of `shifts` (8-bit digits, least first). *which: the buffer that holds the
// result. Enqueue only: no host synchronisation and no allocation. (32-bit images with 64-bit
// payloads.)
template <class IMG, class PAY>
vkc_status radix_pairs(vkc_ctx *ctx, const RadixPairs<IMG, PAY> &p, int64_t n, const int *shifts, int passes,
                       const RadixTables &t, int *which);

// The key digits of a batched argsort, least first: bit offsets of bytes (run: one after the other).
struct BatchDigits {
    int n, run;
    int shift[8];
};

// Batched argsort, each array for itself: tiles of `tile` rows of one array each (2048 or 3072), a pass per key digit, from
// the keys to the outputs' positions. img[] and pos[] are two buffers of n rows each (images of 32 bits
// for up to four digits, else 64); the tables hold 256 counts a tile. Enqueue only.
struct SortSeg {
    const unsigned long long *keys;
    long long *out;
    int64_t base, n;  // its rows of the concatenation
    int64_t tile0;    // its first tile
};
struct BatchSegs {
    const SortSeg *segs;   // in the concatenation's order
    const int *tile_seg;   // each tile's array
    int tiles, tile;
    BatchDigits digits;
};
vkc_status radix_segs(vkc_ctx *ctx, const BatchSegs &b, void *const img[2], unsigned *const pos[2], int64_t n,
                      const RadixTables &t);

// Batched argsort over n rows of all the arrays, concatenated: row i has the image (array number <<
// index_shift) + key digits in images[] (64 bits when `wide`, else 32); the passes over `shifts` sort
// the rows by it, and the last one writes every row's position in its array to that array's output.
// img[] and pos[] are two buffers each (images may be img[1]: the second pass is the first to write
// it). Enqueue only.
struct BatchOut {
    const int64_t *bases;           // first row of each array
    const unsigned long long *outs; // each array's output (an address)
    int index_shift;
};
vkc_status radix_batch(vkc_ctx *ctx, bool wide, const void *images, void *const img[2], unsigned *const pos[2],
                       const BatchOut &batch, int64_t n, const int *shifts, int passes, const RadixTables &t);

// The same for digits that do not fit one image: radix_batch_keys orders the rows by their 64-bit key
// images (images may be img[1]; the result is in buffer (passes - 1) & 1), radix_batch_numbers then by
// the array numbers of the ordered rows (one or two digits), through img_tmp and pay_tmp, and writes
// the outputs. Enqueue only.
vkc_status radix_batch_keys(vkc_ctx *ctx, const void *images, void *const img[2], unsigned *const pos[2], int64_t n,
                            const int *shifts, int passes, const RadixTables &t);
vkc_status radix_batch_numbers(vkc_ctx *ctx, const unsigned *numbers, const unsigned *pay, unsigned *img_tmp,
                               unsigned *pay_tmp, const BatchOut &batch, int64_t n, int passes, const RadixTables &t);

}  // namespace vkc
