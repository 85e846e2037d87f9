// Row tiles (tile_kernels.cu): the execution layout shared by single matrices and batches.
#pragma once

#include <stdint.h>

#include <functional>
#include <vector>

#include <cuda_runtime.h>

namespace spmv {

// A converted matrix the layout is built from: CSR rows (V = 1, P = row_ptr) or column-major
// slices of V rows (P = slice pointer).
struct TileSource {
	const int32_t * P;
	int V;
	const int32_t * cols;
	const double * vals;
	const float * vals_f;        // FP32 variant: the rounded values (long rows read them)
	const int32_t * ymap;        // row map of sorted slices, or null
	int64_t m;                   // rows
	int64_t entries;             // stored entries
	bool split;                  // csr_naive arithmetic: product and sum rounded separately
	// Padded slices: the CSR row_ptr (null: rows have no padding), and the column that pads a
	// row, PAD_OWN for the row's own last one.
	const int32_t * rp;
	int32_t pad_col;
	int64_t x_off, y_off;        // batches: offsets into the concatenated x and y
};

constexpr int32_t PAD_OWN = -1, PAD_SPLIT = -2;

// A row summed by a whole warp from the format's own arrays.
struct LongUnit {
	const int32_t * cols;        // first entry; the others follow `stride` apart
	const void * vals;
	int32_t n;
	int32_t stride;
	int32_t x_off;
	int32_t split;               // csr_naive arithmetic (batches)
	int32_t row;                 // y index
	int32_t padded, pad_col;     // the row ends in padding; its column (PAD_OWN: that of the last entry)
};

// What the staged kernel that would run instead takes, beside a launch: its stored entries, each
// `base` + (mean row length) / `per_length` ps, at most `most`, times `uneven` where the widest
// slice is over twice the mean; or its longest row, from `chain_from` entries on, at `chain` ns an entry
// (both, where that is over eight times the mean).
struct StagedTime {
	double base, per_length, most, uneven, chain;
	int chain_from;
};

struct TilePlan {
	bool built = false;
	int faster = 0;              // not built: the kernel that takes less time (4, 10)
	int32_t pad_col = PAD_OWN;
	bool f32 = false, mixed = false, wide = false, staged = false;
	bool split = false;          // csr_naive arithmetic (MIXED batches: by slice)
	int lanes = 0;               // csr_vec: its lanes; 0: rows summed in order
	int32_t * sptr = nullptr;
	int32_t * tcols = nullptr;
	void * vals = nullptr;
	int32_t * slot_row = nullptr;
	int32_t * slot_cnt = nullptr;
	int32_t * pad = nullptr;     // MIXED batches: a slice's pad column, PAD_OWN or PAD_SPLIT
	int4 * ranges = nullptr;
	LongUnit * longs = nullptr;
	int64_t nranges = 0, nlong = 0, grid = 0;
};

// Where a layout's arrays live: those of a handle or a batch.
struct TileMemory {
	std::function<int(void **, size_t)> take;
	std::function<void(void *)> drop;        // before the owner's end
};

// Builds the layout; p.built stays false, and nothing of it stays allocated, where it does not pay
// (padding above a third of the entries, rows too few and long for its warps), does not fit 32-bit
// indices or finds no memory (a second copy of the entries, which the staged kernels do without).
// lanes: 4 or 8 for csr_vec's row sums, else 0.  staged: the alternative, null: none.
int build_tiles(TilePlan & p, const std::vector<TileSource> & src, int lanes, bool f32, bool mixed,
		const StagedTime * staged, int num_sms, cudaStream_t s, const TileMemory & memory);
int launch_tiles(const TilePlan & p, const void * x, void * y, cudaStream_t s);

}  // namespace spmv
