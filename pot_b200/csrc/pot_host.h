// Host-side launch wrappers shared by the kernel translation units, and the
// per-kernel event timer used when POT_OPT_TIMING is set.
#pragma once

#include <cstddef>
#include <cstdint>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "pot_internal.cuh"

namespace pot {

// Records a start/stop event pair around each kernel when enabled; the
// pairs are resolved into per-name totals at the next sync point.
class Timer {
public:
	bool enabled = false;
	cudaStream_t stream = nullptr;
	uint64_t launches = 0;  // kernels enqueued through ScopedKernel scopes (always counted)

	void begin(const char* name);
	void end();
	void resolve();   // stream must be idle
	void reset();
	int report(int max, const char** names, double* ms, uint64_t* launches) const;
	~Timer();

private:
	struct Pending { int kind; cudaEvent_t a, b; };
	std::vector<const char*> names_;
	std::vector<double> ms_;
	std::vector<uint64_t> count_;
	std::vector<Pending> pending_;
	std::vector<cudaEvent_t> pool_;
	int open_kind_ = -1;
	cudaEvent_t open_a_ = nullptr;
	cudaEvent_t take();
	int kind_of(const char* name);
};

struct ScopedKernel {
	Timer& t;
	ScopedKernel(Timer& tm, const char* name, int kernels = 1) : t(tm)
	{
		t.launches += (uint64_t)kernels;
		t.begin(name);
	}
	~ScopedKernel() { t.end(); }
};

// ---- sort.cu ------------------------------------------------------------
constexpr int RS_BINS = 256;
constexpr int OS_MAX_PASSES = 8;  // radix passes at most (64-bit keys, 8 bits each)
constexpr int OS_THREADS = 256;
// Keys per thread of a radix pass (a tile has OS_THREADS times as many).
// Small runs take small tiles: the pass is then one tile's latency, which
// ranking eight keys a thread sets (eight passes of 8,193 keys 97 -> 86 us,
// of 32,001 102 -> 86; at 128,001 102 and 106, at 1,000,001 245 and 215).  A
// packed batch's passes, whose launch fills the device, take eight.
constexpr uint32_t OS_SMALL_N = 100000u;
constexpr uint32_t OS_ITEMS_MAX = 8;
__host__ __device__ inline uint32_t os_items(uint32_t n) { return n < OS_SMALL_N ? 4u : OS_ITEMS_MAX; }
constexpr int TILE_THREADS = 256;  // of the cell numbering and the due list
constexpr int CELL_TILE = 2048;   // key pairs per tile of the cell numbering
constexpr int DUE_TILE = 4096;    // slots per tile of the due list (whole blocks of the reorder)
constexpr int REORDER_THREADS = 256;

// Words of a step that start at zero: the radix sort's digit counts, the keys
// kernel's block counter, the count of node records given out, a tile ticket
// counter per radix pass, the due
// slots of each DUE_TILE and the passes' look-back status words, 256 a tile.
// The words of the passes in use come last, so that one memset clears a
// step's.  The cell counts of each CELL_TILE need no clearing.
struct StepWords {
	uint32_t* hist;      // [OS_MAX_PASSES * 256]
	unsigned int* pass_ctr;  // [OS_MAX_PASSES]
	unsigned int* keys_ctr;
	unsigned int* rec_ctr;
	uint32_t* cell;      // [cell_tiles(n)]
	uint32_t* due;       // [due_tiles(n)]
	uint32_t* status;    // [passes * radix_rows(n) * 256]
	__host__ __device__ static uint32_t radix_tiles(uint32_t n, uint32_t items)
	{
		return (n + OS_THREADS * items - 1) / (OS_THREADS * items);
	}
	// status rows a pass: the tiles of a single run's, which are the more
	__host__ __device__ static uint32_t radix_rows(uint32_t n) { return radix_tiles(n, os_items(n)); }
	__host__ __device__ static uint32_t cell_tiles(uint32_t n) { return (n + CELL_TILE - 1) / CELL_TILE; }
	__host__ __device__ static uint32_t due_tiles(uint32_t n) { return (n + DUE_TILE - 1) / DUE_TILE; }
	// words before the status rows, which start on a 256-byte boundary
	__host__ __device__ static uint32_t head(uint32_t n)
	{
		return (uint32_t)(OS_MAX_PASSES * RS_BINS + 16 + cell_tiles(n) + due_tiles(n) + 63) & ~63u;
	}
	__host__ __device__ StepWords(uint32_t* w, uint32_t n)
	{
		hist = w;
		pass_ctr = w + OS_MAX_PASSES * RS_BINS;
		keys_ctr = pass_ctr + OS_MAX_PASSES;
		rec_ctr = keys_ctr + 1;
		cell = w + OS_MAX_PASSES * RS_BINS + 16;
		due = cell + cell_tiles(n);
		status = w + head(n);
	}
	__host__ __device__ static size_t words(uint32_t n, int passes)
	{
		return head(n) + (size_t)passes * radix_rows(n) * RS_BINS;
	}
};

// 8-bit passes of the sort from low_bit
int radix_passes(int low_bit);
// Clear the step's words; the keys kernel then counts the digits into hist.
void step_words_clear(uint32_t* words, uint32_t n, int low_bit, cudaStream_t s);
// After step_words_clear and the keys kernel's digit counts: LSD radix sort
// of (keys, vals) on bits [low_bit, 64) in 8-bit passes; result in
// keys[0]/vals[0] when the number of passes is even, keys[1]/vals[1]
// otherwise (returns the index).
int radix_sort_pairs(uint64_t* keys[2], uint32_t* vals[2], uint32_t n, uint32_t* words, int low_bit, cudaStream_t s,
                     Timer& tm, int* err);

}  // namespace pot
