// sort.cuh — stable LSD radix sort of (32-bit cell key, 32-bit particle id) pairs.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace rrsph {

constexpr int kSortThreads = 256;
constexpr int kSortItems = 4;
constexpr int kSortTile = kSortThreads * kSortItems;  // keys per tile
constexpr int kRadix = 256;                           // 8-bit digits

inline uint32_t sort_tiles(uint32_t n) { return (n + kSortTile - 1) / kSortTile; }
// Scratch words the sort needs for n keys: per-tile digit counts + digit totals.
inline size_t sort_scratch_words(uint32_t n) { return (size_t)kRadix * sort_tiles(n) + kRadix; }

// Sorts n pairs by the low `bits` bits of the keys, stably (equal keys keep
// their input order): reads keys_in/vals_in (not modified), leaves the result
// in keys_out/vals_out, and uses keys_tmp/vals_tmp (n words each) and counts
// (sort_scratch_words(n) words) as working memory. Launches 3 kernels per
// 8-bit digit on `stream`; adds them to *launches.
void radix_sort_pairs_into(const uint32_t* keys_in, const uint32_t* vals_in, uint32_t* keys_out, uint32_t* vals_out,
                           uint32_t* keys_tmp, uint32_t* vals_tmp, uint32_t* counts, uint32_t n, int bits,
                           cudaStream_t stream, unsigned long long* launches);

// The grid's sort as a counting sort over the cells, for tables of up to
// kCountCells cells and 64 per particle: every particle takes a place in its cell by an
// atomic count, one pass over the cells turns the counts into the cell table
// (empty cells start at kEmpty) and the particles are
// scattered to their cells; the reorder that follows orders each cell's ids.
// Three launches for any key length against three per 8 bits, and the table with
// them: 409k flume (2M cells) 55 -> 23 us, 6k dam break (8k cells) 28 -> 15 us.
// Above the limits the pass over the cells would cost more than the radix sort.
constexpr uint32_t kCountCells = 1u << 24;
constexpr uint32_t kCountTile = 1024;  // cells per block of the pass over the cells
inline bool cell_sort_fits(uint64_t max_cells, uint64_t n) { return max_cells <= kCountCells && max_cells <= 64 * n + 65536; }
inline uint32_t cell_tiles(uint32_t max_cells) { return (max_cells + kCountTile - 1) / kCountTile; }
// Working words: a count per cell (in whole tiles) and per tile, zero before and after.
inline size_t cell_sort_words(uint32_t max_cells) { return (size_t)cell_tiles(max_cells) * (kCountTile + 1); }
// keys: cell per particle id. place: n words of working memory. scattered[n] gets
// the ids grouped by cell, in any order inside a cell. cell_start and cell_end
// hold whole tiles. Launches 3 kernels on `stream`; adds them to *launches.
void cell_sort(const uint32_t* keys, uint32_t* place, uint32_t* scattered, uint32_t* cell_start, uint32_t* cell_end,
               uint32_t* counts, uint32_t n, uint32_t max_cells, cudaStream_t stream, unsigned long long* launches);

}  // namespace rrsph
