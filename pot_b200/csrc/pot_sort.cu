// The 64-bit LSD radix sort of (Morton key, slot) pairs that orders particles
// each step.  A pass (k_os_pass) waits inside the kernel: each tile spins in
// its decoupled look-back on the status words of tiles that took an earlier
// ticket (and are therefore resident), with LOOKBACK_SPIN_CAP as the limit
// after which it records POT_E_ITER and finishes.
#include <algorithm>

#include "pot_tree.cuh"

namespace pot {

// ---------------------------------------------------------------------------
// block-level helpers
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v)
{
	const int lane = threadIdx.x & 31;
#pragma unroll
	for (int o = 1; o < 32; o <<= 1) {
		uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
		if (lane >= o) v += t;
	}
	return v;
}

// Exclusive block scan of one value per thread (whole warps, at most 32);
// returns the exclusive prefix, writes the block total to *total.
__device__ uint32_t block_excl_scan(uint32_t v, uint32_t* total)
{
	__shared__ uint32_t warp_tot[32];
	__shared__ uint32_t s_total;
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
	const int nw = (int)(blockDim.x >> 5);
	uint32_t inc = warp_incl_scan(v);
	if (lane == 31) warp_tot[w] = inc;
	__syncthreads();
	if (w == 0) {
		uint32_t t = (lane < nw) ? warp_tot[lane] : 0u;
		uint32_t ti = warp_incl_scan(t);
		if (lane < nw) warp_tot[lane] = ti - t;
		if (lane == 31) s_total = ti;
	}
	__syncthreads();
	const uint32_t excl = inc - v + warp_tot[w];
	*total = s_total;
	__syncthreads();  // warp_tot / s_total are reused by the next call
	return excl;
}

// ---------------------------------------------------------------------------
// radix sort: one kernel per 8-bit pass with decoupled look-back
// ---------------------------------------------------------------------------
// Tiles of OS_TILE keys.  The grid is the blocks the device holds at once;
// each block takes the next tile index from a counter (so tiles start in
// index order) until none is left, ranks its keys stably per digit, publishes
// its per-digit counts, and obtains the exclusive prefix of each digit over
// all earlier tiles by looking back at their published words (aggregate or
// inclusive prefix).  Every wait has an iteration cap; reaching it records
// POT_E_ITER and the pass completes with wrong order but without hanging.
// The keys are then staged in shared memory in digit order and written out
// contiguously per digit.
constexpr uint32_t LB_AGG = 1u << 30;
constexpr uint32_t LB_PRE = 2u << 30;
constexpr uint32_t LB_COUNT = (1u << 30) - 1u;
constexpr long LOOKBACK_SPIN_CAP = 1L << 24;
constexpr int OS_LOOKBACK = 8;      // earlier tiles read per round of the look-back

template <int OS_ITEMS, class G>
__device__ __forceinline__ void os_pass_body(G grd, const uint64_t* __restrict__ kin,
                                             const uint32_t* __restrict__ vin, size_t n, int shift,
                                             const uint32_t* __restrict__ goff, uint32_t* __restrict__ status,
                                             unsigned int* __restrict__ tile_ctr, uint64_t* __restrict__ kout,
                                             uint32_t* __restrict__ vout, int* __restrict__ err)
{
	constexpr int NW = OS_THREADS / 32, OS_TILE = OS_THREADS * OS_ITEMS;
	__shared__ uint32_t s_tile;
	__shared__ uint32_t s_wcnt[NW][RS_BINS];  // per-warp running count, then per-warp exclusive prefix
	__shared__ uint32_t s_loc[RS_BINS];       // digit start inside the staged tile
	__shared__ uint32_t s_glob[RS_BINS];      // digit start in the output
	__shared__ uint64_t s_key[OS_TILE];
	__shared__ uint32_t s_val[OS_TILE];
	const int t = threadIdx.x, w = t >> 5, lane = t & 31;
	const uint32_t lt_mask = (1u << lane) - 1u;
	for (;;) {  // tiles in ticket order until none is left
		if (t == 0) s_tile = atomicAdd(tile_ctr, 1u);
#pragma unroll
		for (int k = 0; k < NW; k++) s_wcnt[k][t] = 0;
		__syncthreads();
		const uint32_t tile = s_tile;
		const size_t base = (size_t)tile * OS_TILE;
		if (base >= n) return;
		// warp w holds OS_ITEMS rounds of 32 consecutive keys of the tile, so a key's index in the tile is (warp, round, lane) in order
		uint64_t key[OS_ITEMS];
		uint32_t val[OS_ITEMS];
		uint32_t rank[OS_ITEMS];
		int dig[OS_ITEMS];
#pragma unroll
		for (int r = 0; r < OS_ITEMS; r++) {
			const size_t i = base + (size_t)(w * 32 * OS_ITEMS + r * 32 + lane);
			dig[r] = RS_BINS;
			key[r] = 0;
			val[r] = 0;
			if (i < n) {
				key[r] = kin[i];
				val[r] = vin[i];
				dig[r] = (int)((key[r] >> shift) & 0xFF);
			}
		}
		// stable ranks inside the warp: a running count per digit in the warp's
		// own row, updated once per round by the lowest lane of each digit
#pragma unroll
		for (int r = 0; r < OS_ITEMS; r++) {
			const int d = dig[r];
			const uint32_t peers = __match_any_sync(0xffffffffu, d);
			const uint32_t before = d < RS_BINS ? s_wcnt[w][d] : 0u;
			rank[r] = before + __popc(peers & lt_mask);
			__syncwarp();
			if (d < RS_BINS && (peers & lt_mask) == 0u) s_wcnt[w][d] = before + __popc(peers);
			__syncwarp();
		}
		__syncthreads();
		// digit t: each warp's exclusive prefix over the warps before it, and
		// the tile's count
		uint32_t cnt = 0;
#pragma unroll
		for (int k = 0; k < NW; k++) {
			const uint32_t c = s_wcnt[k][t];
			s_wcnt[k][t] = cnt;
			cnt += c;
		}
		// publish this tile's count of digit t, then look back for its prefix,
		// OS_LOOKBACK earlier tiles per round of reads
		volatile uint32_t* st = status;
		st[(size_t)tile * RS_BINS + t] = (tile == 0 ? LB_PRE : LB_AGG) | cnt;
		uint32_t excl = 0;
		if (tile > 0) {
			long spins = 0;
			int64_t j = (int64_t)tile - 1;  // next tile to read
			bool found = false;
			while (!found) {
				uint32_t v[OS_LOOKBACK];
#pragma unroll
				for (int q = 0; q < OS_LOOKBACK; q++) v[q] = j - q >= 0 ? st[(size_t)(j - q) * RS_BINS + t] : 0u;
				int used = 0;
				bool stalled = false;
#pragma unroll
				for (int q = 0; q < OS_LOOKBACK; q++) {
					if (found || stalled) continue;
					const uint32_t flag = v[q] & ~LB_COUNT;
					if (flag == 0) {  // not yet published (tile 0 always is, so j - q >= 0 here)
						stalled = true;
						continue;
					}
					excl += v[q] & LB_COUNT;
					used++;
					if (flag == LB_PRE) found = true;
				}
				if (found) break;
				j -= used;
				if (used == 0 && ++spins > LOOKBACK_SPIN_CAP) {
					atomicCAS(err, 0, POT_E_ITER);
					break;
				}
			}
			st[(size_t)tile * RS_BINS + t] = LB_PRE | (excl + cnt);
		}
		s_glob[t] = goff[t] + excl;
		// digit starts inside the tile
		{
			uint32_t tot;
			const uint32_t e = block_excl_scan(cnt, &tot);
			s_loc[t] = e;
		}
		__syncthreads();
#pragma unroll
		for (int r = 0; r < OS_ITEMS; r++) {
			if (dig[r] < RS_BINS) {
				const uint32_t p = s_loc[dig[r]] + s_wcnt[w][dig[r]] + rank[r];
				s_key[p] = key[r];
				s_val[p] = val[r];
			}
		}
		__syncthreads();
		const uint32_t nt = (uint32_t)((n - base) < (size_t)OS_TILE ? (n - base) : (size_t)OS_TILE);
		for (uint32_t i = t; i < nt; i += OS_THREADS) {
			const uint64_t k = s_key[i];
			const int d = (int)((k >> shift) & 0xFF);
			const uint32_t o = s_glob[d] + (i - s_loc[d]);
			kout[o] = k;
			vout[o] = s_val[i];
		}
		__syncthreads();  // the next tile reuses the shared arrays
	}
}

template <int ITEMS>
__global__ void __launch_bounds__(OS_THREADS) k_os_pass(const uint64_t* __restrict__ kin,
                                                        const uint32_t* __restrict__ vin, size_t n, int shift,
                                                        const uint32_t* __restrict__ goff,
                                                        uint32_t* __restrict__ status,
                                                        unsigned int* __restrict__ tile_ctr,
                                                        uint64_t* __restrict__ kout, uint32_t* __restrict__ vout,
                                                        int* __restrict__ err)
{
	os_pass_body<ITEMS>(GridSelf {}, kin, vin, n, shift, goff, status, tile_ctr, kout, vout, err);
}

static inline int os_passes(int low_bit) { return (63 - low_bit + 7) / 8; }

// Blocks of k_os_pass resident on the device at once: the pass's grid, each
// block taking tiles until none is left (no second wave of blocks).
template <int ITEMS>
static uint32_t os_resident()
{
	static uint32_t n = 0;
	if (!n) {
		int dev = 0, sms = 0, per = 0;
		cudaGetDevice(&dev);
		cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
		cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_os_pass<ITEMS>, OS_THREADS, 0);
		n = (uint32_t)std::max(1, sms) * (uint32_t)std::max(1, per);
	}
	return n;
}

int radix_passes(int low_bit) { return os_passes(low_bit); }

void step_words_clear(uint32_t* words, uint32_t n, int low_bit, cudaStream_t s)
{
	cudaMemsetAsync(words, 0, sizeof(uint32_t) * StepWords::words(n, os_passes(low_bit)), s);
}

template <int ITEMS>
static int sort_passes(uint64_t* keys[2], uint32_t* vals[2], uint32_t n, uint32_t* words, int low_bit, cudaStream_t s,
                       Timer& tm, int* err)
{
	const StepWords W(words, n);
	const uint32_t tiles = StepWords::radix_tiles(n, ITEMS);
	const int npass = os_passes(low_bit);
	int src = 0;
	for (int p = 0; p < npass; p++) {
		ScopedKernel k(tm, "sort_pass");
		const uint32_t grid = std::min<uint32_t>(tiles, os_resident<ITEMS>());
		k_os_pass<ITEMS><<<grid, OS_THREADS, 0, s>>>(keys[src], vals[src], n, low_bit + 8 * p, W.hist + p * RS_BINS,
		                                             W.status + (size_t)p * tiles * RS_BINS, W.pass_ctr + p,
		                                             keys[src ^ 1], vals[src ^ 1], err);
		src ^= 1;
	}
	return src;
}

int radix_sort_pairs(uint64_t* keys[2], uint32_t* vals[2], uint32_t n, uint32_t* words, int low_bit, cudaStream_t s,
                     Timer& tm, int* err)
{
	if (n == 0) return 0;
	return os_items(n) == 4 ? sort_passes<4>(keys, vals, n, words, low_bit, s, tm, err)
	                        : sort_passes<(int)OS_ITEMS_MAX>(keys, vals, n, words, low_bit, s, tm, err);
}

}  // namespace pot

// ---------------------------------------------------------------------------
// packed batch: the sort of every member in one launch per pass
// ---------------------------------------------------------------------------
namespace pot {

// What the single run clears with a memset before its keys.
__global__ void __launch_bounds__(OS_THREADS) kp_sort_clear(PackDev B)
{
	const SegBlock sb = seg_block(B.pre[PS_TILES], B.M);
	const MemberView& v = B.mv[sb.m];
	const size_t n = StepWords::words(v.P.n, (int)B.npass);
	for (size_t i = (size_t)sb.id * OS_THREADS + threadIdx.x; i < n; i += (size_t)sb.n * OS_THREADS) v.words[i] = 0u;
}

// Pass p: every member's tiles; a tile's index within its member comes from
// the member's own ticket counter, so the look-back waits only on tiles of
// the same member that took earlier tickets (and are therefore resident).
__global__ void __launch_bounds__(OS_THREADS) kp_os_pass(PackDev B, int p)
{
	const SegBlock sb = seg_block(B.pre[PS_TILES], B.M);
	const MemberView& v = B.mv[sb.m];
	const StepWords W(v.words, v.P.n);
	const int src = p & 1;
	os_pass_body<(int)OS_ITEMS_MAX>(GridSeg { sb.id, sb.n }, v.keys[src], v.vals[src], (size_t)v.P.n,
	                                (int)v.P.key_bits + 8 * p, W.hist + p * RS_BINS,
	                                W.status + (size_t)p * StepWords::radix_rows(v.P.n) * RS_BINS, W.pass_ctr + p,
	                                v.keys[src ^ 1], v.vals[src ^ 1], &v.rec->status);
}

void pack_sort_begin(const PackDev& B, cudaStream_t s)
{
	kp_sort_clear<<<B.blocks[PS_TILES], OS_THREADS, 0, s>>>(B);
}

void pack_sort(const PackDev& B, cudaStream_t s)
{
	for (uint32_t p = 0; p < B.npass; p++) kp_os_pass<<<B.blocks[PS_TILES], OS_THREADS, 0, s>>>(B, (int)p);
}

}  // namespace pot
