// Morton keys, per-step reorder, octree build and upward moments.
//
// Topology.  The reference inserts particles one by one into a pointer
// octree whose root is [0, 2 r mpp]^3 and whose cells split at the midpoint
// (x1 + x2) / 2 of their faces until every leaf holds one particle
// (pot.c:1457-1643).  The final tree does not depend on insertion order: a
// cell is internal exactly when two or more particles lie in it.  So it is
// rebuilt here from sorted keys:
//   * key = 21 levels x 3 bits of the comparisons `x < mid` the reference's
//     descent makes (pot.c:1522-1553), computed with the same midpoint
//     arithmetic, so cell membership is bit-identical;
//   * with keys sorted, the cell of level l containing particle i holds
//     more than L particles iff keys i and i + L share its 3l-bit prefix;
//     pair i = (i, i + L) "owns" the cells whose first particle is i, i.e.
//     the levels (lvl[i-1], lvl[i]], which numbers cells in pre-order;
//   * a cell's last particle and its 8 children are found by searches over
//     its key range that make several independent reads per round
//     (cell_end, child_starts).
// Leaf size L = 1 reproduces the reference's tree; L > 1 gives bucket leaves.
//
// Moments.  Net charge q, absolute charge aq and the |q|-weighted centre of
// a cell are the reference's running update over its children in the
// member order gxlylz, gxlygz, lxlylz, lxlygz, lxgylz, lxgygz, gxgylz, gxgygz
// (pot.c:1290-1402), evaluated bottom-up with arrival counters and unfused
// double operations, which makes them bit-identical too.
#include "pot_tree.cuh"

namespace pot {

// 63-bit key: level 1 in bits 62..60, digit = gx << 2 | gy << 1 | gz.
__device__ __forceinline__ uint64_t morton_key(double x, double y, double z, double w)
{
	double lx = 0.0, hx = w, ly = 0.0, hy = w, lz = 0.0, hz = w;
	uint64_t key = 0;
#pragma unroll 3
	for (int l = 0; l < MAX_LEVELS; l++) {
		const double mx = dmul(dadd(lx, hx), 0.5);
		const double my = dmul(dadd(ly, hy), 0.5);
		const double mz = dmul(dadd(lz, hz), 0.5);
		const uint32_t bx = (x < mx) ? 0u : 1u;
		const uint32_t by = (y < my) ? 0u : 1u;
		const uint32_t bz = (z < mz) ? 0u : 1u;
		if (bx) lx = mx; else hx = mx;
		if (by) ly = my; else hy = my;
		if (bz) lz = mz; else hz = mz;
		key = (key << 3) | (uint64_t)((bx << 2) | (by << 1) | bz);
	}
	return key;
}

// spread the low 21 bits of v to every third bit
__device__ __forceinline__ uint64_t spread3(uint64_t v)
{
	v &= 0x1FFFFFull;
	v = (v | (v << 32)) & 0x1F00000000FFFFull;
	v = (v | (v << 16)) & 0x1F0000FF0000FFull;
	v = (v | (v << 8)) & 0x100F00F00F00F00Full;
	v = (v | (v << 4)) & 0x10C30C30C30C30C3ull;
	v = (v | (v << 2)) & 0x1249249249249249ull;
	return v;
}

// Fast form: the same key layout from the scaled coordinate, cell j of level
// 21 being [j, j + 1) * w / 2^21; it differs from the midpoint descent only
// for points within rounding of a cell face, which the fast form tolerates.
__device__ __forceinline__ uint64_t scaled_key(double x, double y, double z, double scale)
{
	const double m = 2097151.0;
	const uint64_t ix = (uint64_t)fmin(fmax(x * scale, 0.0), m);
	const uint64_t iy = (uint64_t)fmin(fmax(y * scale, 0.0), m);
	const uint64_t iz = (uint64_t)fmin(fmax(z * scale, 0.0), m);
	return (spread3(ix) << 2) | (spread3(iy) << 1) | spread3(iz);
}

// Keys of every particle (grid-stride) and the digit counts of each of the
// radix sort's npass 8-bit passes from low_bit, counted in shared memory and
// added once per block to hist[p * 256 + d]: the sort then needs no read of
// the keys of its own for them.
template <class G>
__device__ __forceinline__ void keys_body(G grd, const double4* __restrict__ pos, uint64_t* __restrict__ keys,
                                          uint32_t* __restrict__ vals, const Params& P, RunRec* rec, int begin_step,
                                          uint32_t* hist, unsigned int* ctr, int low_bit, int npass)
{
	__shared__ uint32_t h[OS_MAX_PASSES][RS_BINS];
	__shared__ bool s_last;
	for (int i = threadIdx.x; i < npass * RS_BINS; i += blockDim.x) (&h[0][0])[i] = 0;
	__syncthreads();
	if (grd.id() == 0 && threadIdx.x == 0) {
		rec->n_overflow = 0;
		for (int k = 0; k < 2; k++) rec->n_groups[k] = rec->n_groups_all[k] = 0;
	}
	if (begin_step && grd.id() == 0 && threadIdx.x == 0) {
		const unsigned long long t = rec->t_steps + 1;
		rec->t_steps = t;
		rec->n_due = 0;
		rec->n_rein = 0;
		rec->n_nodes = 0;
		rec->work_ctr = 0;
		rec->work_ctr2 = 0;
		rec->stack_max = 0;
		rec->grain_due = (t % P.tss[SP_DUST]) == 0 ? 1u : 0u;
		rec->chi_failed = 0;
		rec->wall_warn = rec->warn & WARN_WALL;
		rec->dq = 0;
		rec->de = 0;
		rec->nabs_ion = 0;
		rec->nabs_e = 0;
		for (int k = 0; k < 3; k++) { rec->sumv_ion[k] = 0; rec->sumv_e[k] = 0; }
		rec->interactions = 0;
		rec->far_cells = 0;
		rec->n_pushed = 0;
		rec->n_collected = 0;
		rec->n_wall = 0;
		rec->n_bounced = 0;
		rec->done_ctr = 0;
		rec->grain_slot = 0xFFFFFFFFu;
	}
	for (uint32_t s = grd.id() * blockDim.x + threadIdx.x; s < P.n; s += grd.n() * blockDim.x) {
		const double4 p = pos[s];
		if (isnan(p.x) || isnan(p.y) || isnan(p.z)) {
			set_status(rec, POT_E_NONFINITE);
		} else if (p.x < 0.0 || p.x > P.root_w || p.y < 0.0 || p.y > P.root_w || p.z < 0.0 || p.z > P.root_w) {
			set_status(rec, POT_E_DOMAIN);  // build_tree returns NULL, pot.c:1491-1500
		}
		// A spheroidal grain is not a tree source (pot-spheroid.c:1516-1518): the
		// largest key sorts it to the last slot, outside [0, n_tree).  No
		// particle of the spherical domain lies in that corner cell.
		const uint64_t k = (P.shape && (int)p.w == SP_DUST) ? 0x7FFFFFFFFFFFFFFFull
		                   : P.form == POT_FORM_FAST       ? scaled_key(p.x, p.y, p.z, 2097152.0 / P.root_w)
		                                                   : morton_key(p.x, p.y, p.z, P.root_w);
		keys[s] = k;
		vals[s] = s;
		for (int q = 0; q < npass; q++) atomicAdd(&h[q][(k >> (low_bit + 8 * q)) & 0xFF], 1u);
	}
	__syncthreads();
	for (int i = threadIdx.x; i < npass * RS_BINS; i += blockDim.x) {
		const uint32_t c = (&h[0][0])[i];
		if (c) atomicAdd(&hist[i], c);
	}
	// the last block turns each pass's counts into the digits' starts in the
	// sorted order (one warp a pass, eight digits a lane)
	__threadfence();
	__syncthreads();
	if (threadIdx.x == 0) s_last = atomicAdd(ctr, 1u) + 1u == grd.n();
	__syncthreads();
	const int p = (int)(threadIdx.x >> 5), lane = (int)(threadIdx.x & 31u);
	if (!s_last || p >= npass) return;
	__threadfence();
	uint4* row = reinterpret_cast<uint4*>(hist + p * RS_BINS) + 2 * lane;
	uint4 a = __ldcg(row), b = __ldcg(row + 1);
	const uint32_t sum = a.x + a.y + a.z + a.w + b.x + b.y + b.z + b.w;
	uint32_t run = sum;
#pragma unroll
	for (int o = 1; o < 32; o <<= 1) {
		const uint32_t v = __shfl_up_sync(0xffffffffu, run, o);
		if (lane >= o) run += v;
	}
	run -= sum;
	uint32_t c;
	c = a.x; a.x = run; run += c;
	c = a.y; a.y = run; run += c;
	c = a.z; a.z = run; run += c;
	c = a.w; a.w = run; run += c;
	c = b.x; b.x = run; run += c;
	c = b.y; b.y = run; run += c;
	c = b.z; b.z = run; run += c;
	b.w = run;
	row[0] = a;
	row[1] = b;
}

__global__ void __launch_bounds__(256) k_keys(const double4* __restrict__ pos, uint64_t* __restrict__ keys,
                                              uint32_t* __restrict__ vals, Params P, RunRec* rec, int begin_step,
                                              uint32_t* words, int low_bit, int npass)
{
	const StepWords W(words, P.n);
	keys_body(GridSelf {}, pos, keys, vals, P, rec, begin_step, W.hist, W.keys_ctr, low_bit, npass);
}

// Gather the state into the new Morton order, write the tree sources and
// mark the particles due this step (electrons every step, ions every
// tss[ION] steps, the grain every tss[DUST] steps, pot.c:2430-2434).
// One slot of the reorder; returns whether the particle is due.
__device__ __forceinline__ bool reorder_one(uint32_t s, const uint32_t* __restrict__ perm,
                                            const double4* __restrict__ pos_in,
                                            const double4* __restrict__ vel_in, const uint32_t* __restrict__ pid_in,
                                            double4* __restrict__ pos_out, double4* __restrict__ vel_out,
                                            uint32_t* __restrict__ pid_out, double4* __restrict__ src64,
                                            float4* __restrict__ src32, const Params& P, RunRec* rec)
{
	const uint32_t j = perm[s];
	const double4 p = pos_in[j];
	const double4 v = vel_in[j];
	const uint32_t id = pid_in[j];
	const int sp = (int)p.w;
	const double q = sp == SP_DUST ? (double)rec->grain_q : (sp == SP_ION ? 1.0 : -1.0);
	pos_out[s] = p;
	vel_out[s] = v;
	pid_out[s] = id;
	src64[s] = make_double4(p.x, p.y, p.z, q);
	if (src32) {
		src32[s] = make_float4((float)((p.x - P.rad) * P.inv_rad), (float)((p.y - P.rad) * P.inv_rad),
		                       (float)((p.z - P.rad) * P.inv_rad), (float)q);
	}
	if (sp == SP_DUST) rec->grain_slot = s;
	return (rec->t_steps % P.tss[sp]) == 0;
}

template <class G>
__device__ __forceinline__ void reorder_body(G grd, const uint32_t* __restrict__ perm,
                                             const double4* __restrict__ pos_in,
                                             const double4* __restrict__ vel_in, const uint32_t* __restrict__ pid_in,
                                             double4* __restrict__ pos_out, double4* __restrict__ vel_out,
                                             uint32_t* __restrict__ pid_out, double4* __restrict__ src64,
                                             float4* __restrict__ src32, uint8_t* __restrict__ due,
                                             uint32_t* __restrict__ due_tiles, const Params& P, RunRec* rec)
{
	const uint32_t s = grd.id() * REORDER_THREADS + threadIdx.x;
	// the due slots of each DUE_TILE (a block lies inside one)
	bool is_due = false;
	if (s < P.n) {
		is_due = reorder_one(s, perm, pos_in, vel_in, pid_in, pos_out, vel_out, pid_out, src64, src32, P, rec);
		due[s] = is_due ? 1 : 0;
	}
	__shared__ uint32_t wcnt[REORDER_THREADS / 32];
	const uint32_t c = __popc(__ballot_sync(0xffffffffu, is_due));
	if ((threadIdx.x & 31) == 0) wcnt[threadIdx.x >> 5] = c;
	__syncthreads();
	if (threadIdx.x == 0) {
		uint32_t t = 0;
		for (uint32_t w = 0; w < REORDER_THREADS / 32; w++) t += wcnt[w];
		if (t) atomicAdd(&due_tiles[(grd.id() * REORDER_THREADS) / DUE_TILE], t);
	}
}

__global__ void __launch_bounds__(REORDER_THREADS)
k_reorder(const uint32_t* __restrict__ perm, const double4* __restrict__ pos_in, const double4* __restrict__ vel_in,
          const uint32_t* __restrict__ pid_in, double4* __restrict__ pos_out,
          double4* __restrict__ vel_out, uint32_t* __restrict__ pid_out, double4* __restrict__ src64,
          float4* __restrict__ src32, uint8_t* __restrict__ due, uint32_t* words, Params P, RunRec* rec)
{
	reorder_body(GridSelf {}, perm, pos_in, vel_in, pid_in, pos_out, vel_out, pid_out, src64, src32, due,
	             StepWords(words, P.n).due, P, rec);
}

// Exclusive prefix of tile `tile` over the tiles' counts, by the whole block:
// each block adds up the counts of the tiles before its own (at most some
// thousands of words from L2), so a scan needs no launch between the kernel
// that counts and the one that places.
__device__ __forceinline__ uint32_t tiles_before(const uint32_t* __restrict__ counts, uint32_t tile)
{
	__shared__ uint32_t part[TILE_THREADS / 32];
	uint32_t s = 0;
	for (uint32_t i = threadIdx.x; i < tile; i += TILE_THREADS) s += counts[i];
	s = __reduce_add_sync(0xffffffffu, s);
	if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
	__syncthreads();
	uint32_t t = 0;
#pragma unroll
	for (int k = 0; k < TILE_THREADS / 32; k++) t += part[k];
	__syncthreads();
	return t;
}

// Exclusive block scan of one value per thread (TILE_THREADS threads);
// *total = block sum.
__device__ __forceinline__ uint32_t tile_scan(uint32_t v, uint32_t* total)
{
	__shared__ uint32_t wsum[TILE_THREADS / 32];
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
	uint32_t incl = v;
#pragma unroll
	for (int o = 1; o < 32; o <<= 1) {
		const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
		if (lane >= o) incl += u;
	}
	if (lane == 31) wsum[w] = incl;
	__syncthreads();
	uint32_t before = 0, tot = 0;
#pragma unroll
	for (int k = 0; k < TILE_THREADS / 32; k++) {
		const uint32_t c = wsum[k];
		if (k < w) before += c;
		tot += c;
	}
	__syncthreads();
	*total = tot;
	return before + incl - v;
}

// The due list: due_list[k] is the k-th due slot, due_prefix[s] the number of
// due slots before s; one DUE_TILE a block, 16 slots a thread.
template <class G>
__device__ __forceinline__ void due_list_body(G grd, const uint8_t* __restrict__ due,
                                              const uint32_t* __restrict__ counts, uint32_t* __restrict__ due_list,
                                              uint32_t* __restrict__ due_prefix, const Params& P, RunRec* rec)
{
	constexpr int ITEMS = DUE_TILE / TILE_THREADS;  // 16: one 16-byte load of flags
	const uint32_t tile = grd.id(), n = P.n, s0 = tile * DUE_TILE + threadIdx.x * ITEMS;
	const uint32_t base = tiles_before(counts, tile);
	uint32_t bits = 0;
	if (s0 + ITEMS <= n) {
		const uint4 f = *reinterpret_cast<const uint4*>(due + s0);
		const uint32_t q[4] = { f.x, f.y, f.z, f.w };
#pragma unroll
		for (int k = 0; k < ITEMS; k++) bits |= ((q[k >> 2] >> (8 * (k & 3))) & 1u) << k;
	} else {
		for (int k = 0; k < ITEMS; k++)
			if (s0 + (uint32_t)k < n && due[s0 + k]) bits |= 1u << k;
	}
	uint32_t total;
	uint32_t run = base + tile_scan(__popc(bits), &total);
	if (threadIdx.x == 0 && (uint64_t)(tile + 1) * DUE_TILE >= n) {
		rec->n_due = base + total;
		due_prefix[n] = base + total;
	}
#pragma unroll
	for (int k = 0; k < ITEMS; k += 4) {
		uint4 o;
		uint32_t* const op = &o.x;
#pragma unroll
		for (int u = 0; u < 4; u++) {
			const uint32_t s = s0 + (uint32_t)(k + u);
			op[u] = run;
			if ((bits >> (k + u)) & 1u) due_list[run++] = s;
		}
		if (s0 + (uint32_t)(k + 4) <= n) {
			*reinterpret_cast<uint4*>(due_prefix + s0 + k) = o;
		} else {
			for (int u = 0; u < 4; u++)
				if (s0 + (uint32_t)(k + u) < n) due_prefix[s0 + k + u] = op[u];
		}
	}
}

__global__ void __launch_bounds__(TILE_THREADS)
k_due_list(const uint8_t* __restrict__ due, const uint32_t* __restrict__ words_due, uint32_t* __restrict__ due_list,
           uint32_t* __restrict__ due_prefix, Params P, RunRec* rec)
{
	due_list_body(GridSelf {}, due, words_due, due_list, due_prefix, P, rec);
}

__device__ __forceinline__ int lcp_levels(uint64_t a, uint64_t b)
{
	const uint64_t x = a ^ b;
	if (x == 0) return MAX_LEVELS;
	return (__clzll((long long)x) - 1) / 3;
}

// Common levels of the keys of slots i and i + L, capped at max_level - 1 (a
// cell of the deepest level cannot split).
__device__ __forceinline__ int pair_levels(uint64_t a, uint64_t b, int max_level, RunRec* rec)
{
	const int l = lcp_levels(a, b);
	if (l == MAX_LEVELS && max_level == MAX_LEVELS && rec) atomicOr(&rec->warn, 1u);
	return l < max_level - 1 ? l : max_level - 1;
}

// Cell numbering in two launches over tiles of CELL_TILE key pairs.  Pair i
// owns the cells of levels (lvl8[i-1], lvl8[i]], lvl8[i] its common levels:
// the first launch counts the cells each tile owns, the second adds up the
// counts before its tile, numbers its cells (base[i]: pair i's first) and
// writes their first slot and level.
struct PairLevels {
	int lv[CELL_TILE / TILE_THREADS + 1];  // lv[0]: the pair before this thread's first
	uint32_t sum;
	uint32_t same;  // bit k: slots i0 + k and i0 + k + 1 have one key
	__device__ __forceinline__ PairLevels(const uint64_t* __restrict__ keys, uint32_t i0, uint32_t n_pairs, uint32_t L,
	                                      int max_level, RunRec* rec)
	{
		lv[0] = i0 > 0 && i0 - 1 < n_pairs ? pair_levels(keys[i0 - 1], keys[i0 - 1 + L], max_level, nullptr) : -1;
		sum = same = 0;
		uint64_t next = i0 < n_pairs ? keys[i0] : 0;
#pragma unroll
		for (int k = 0; k < CELL_TILE / TILE_THREADS; k++) {
			const uint32_t i = i0 + (uint32_t)k;
			const uint64_t key = next;
			lv[k + 1] = -1;
			if (i < n_pairs) {
				next = keys[i + 1];
				if (next == key) same |= 1u << k;
				lv[k + 1] = pair_levels(key, L == 1 ? next : keys[i + L], max_level, rec);
			}
			if (lv[k + 1] > lv[k]) sum += (uint32_t)(lv[k + 1] - lv[k]);
		}
	}
};

// Two particles at one position, slots i and i + 1 with one key: the
// reference's insertion would split forever (pot.c:1466-1470) or fail at a
// reallocation (pot.c:1578-1586).
__device__ __forceinline__ void check_coincident(uint32_t i, const uint32_t* __restrict__ perm,
                                                 const double4* __restrict__ pos_in, RunRec* rec)
{
	const double4 p = pos_in[perm[i]], o = pos_in[perm[i + 1]];
	if (p.x == o.x && p.y == o.y && p.z == o.z) set_status(rec, POT_E_COINCIDENT);
}

// The positions of neighbours with one key are compared here, ahead of all that
// can find the tree too large, so that the status names the cause.
template <class G>
__device__ __forceinline__ void cell_count_body(G grd, const uint64_t* __restrict__ keys,
                                                const uint32_t* __restrict__ perm, const double4* __restrict__ pos_in,
                                                uint32_t n_pairs, uint32_t L, int max_level,
                                                uint32_t* __restrict__ counts, RunRec* rec)
{
	const uint32_t i0 = grd.id() * CELL_TILE + threadIdx.x * (CELL_TILE / TILE_THREADS);
	const PairLevels p(keys, i0, n_pairs, L, max_level, rec);
	for (uint32_t same = p.same; same; same &= same - 1u) check_coincident(i0 + (uint32_t)__ffs(same) - 1u, perm, pos_in, rec);
	// the last L - 1 neighbours, beyond the pairs (i, i + L)
	if (grd.id() == 0 && threadIdx.x + 1 < L) {
		const uint32_t i = n_pairs + threadIdx.x;
		if (keys[i] == keys[i + 1]) check_coincident(i, perm, pos_in, rec);
	}
	uint32_t total;
	tile_scan(p.sum, &total);
	if (threadIdx.x == 0) counts[grd.id()] = total;
}

template <class G>
__device__ __forceinline__ void cell_number_body(G grd, const uint64_t* __restrict__ keys, uint32_t n_pairs, uint32_t L,
                                                 int max_level, const uint32_t* __restrict__ counts, const TreeDev& T,
                                                 RunRec* rec)
{
	const uint32_t tile = grd.id(), i0 = tile * CELL_TILE + threadIdx.x * (CELL_TILE / TILE_THREADS);
	const PairLevels p(keys, i0, n_pairs, L, max_level, nullptr);
	const uint32_t base = tiles_before(counts, tile);
	uint32_t total;
	uint32_t run = base + tile_scan(p.sum, &total);
	if (threadIdx.x == 0 && (uint64_t)(tile + 1) * CELL_TILE >= n_pairs) rec->n_nodes = base + total;
#pragma unroll
	for (int k = 0; k < CELL_TILE / TILE_THREADS; k++) {
		const uint32_t i = i0 + (uint32_t)k;
		if (i >= n_pairs) break;
		T.lvl8[i] = (int8_t)p.lv[k + 1];
		T.base[i] = run;
		for (int l = p.lv[k] + 1; l <= p.lv[k + 1]; l++, run++) {
			if (run >= T.cap) {
				set_status(rec, POT_E_CAPACITY);
				break;
			}
			T.first[run] = i;
			T.level[run] = (uint8_t)l;
		}
	}
}

__global__ void __launch_bounds__(TILE_THREADS) k_cell_count(const uint64_t* __restrict__ keys,
                                                             const uint32_t* __restrict__ perm,
                                                             const double4* __restrict__ pos_in, uint32_t n_pairs,
                                                             uint32_t L, int max_level, uint32_t* __restrict__ counts,
                                                             RunRec* rec)
{
	cell_count_body(GridSelf {}, keys, perm, pos_in, n_pairs, L, max_level, counts, rec);
}

__global__ void __launch_bounds__(TILE_THREADS) k_cell_number(const uint64_t* __restrict__ keys, uint32_t n_pairs,
                                                              uint32_t L, int max_level,
                                                              const uint32_t* __restrict__ counts, TreeDev T,
                                                              RunRec* rec)
{
	cell_number_body(GridSelf {}, keys, n_pairs, L, max_level, counts, T, rec);
}

// The searches below run over a cell's sorted key range, where the tested
// property holds on a prefix of the range.  They make several independent
// reads per round, so that the chain of dependent loads -- which sets the
// time of the cells near the root -- is short.

// First index in [a, b) at which `pred` fails, b if it holds throughout:
// seven probes per round keep one eighth of the range; the last eight or
// fewer are read at once.
template <class Pred>
__device__ __forceinline__ uint32_t first_fail8(const uint64_t* __restrict__ keys, uint32_t a, uint32_t b, Pred pred)
{
	while (b - a > 8u) {
		const uint64_t span = b - a;
		uint32_t p[7];
		bool ok[7];
#pragma unroll
		for (int i = 0; i < 7; i++) p[i] = a + (uint32_t)((span * (uint64_t)(i + 1)) >> 3);  // a < p[0] < ... < p[6] < b
#pragma unroll
		for (int i = 0; i < 7; i++) ok[i] = pred(keys[p[i]]);
		uint32_t na = a, nb = b;
#pragma unroll
		for (int i = 0; i < 7; i++)
			if (ok[i]) na = p[i] + 1;  // the last probe that holds
#pragma unroll
		for (int i = 6; i >= 0; i--)
			if (!ok[i]) nb = p[i];  // the first probe that fails
		a = na;
		b = nb;
	}
	uint32_t c = 0;
#pragma unroll
	for (int i = 0; i < 8; i++) c += (a + (uint32_t)i < b && pred(keys[a + i])) ? 1u : 0u;
	return a + c;
}

// One past the last slot of the cell that starts at slot f with key prefix
// pfx (key >> shift): f + 2^e is probed for seven exponents per round until
// one leaves the cell, then the bracket is searched.
__device__ __forceinline__ uint32_t cell_end(const uint64_t* __restrict__ keys, uint32_t f, uint32_t n, int shift,
                                             uint64_t pfx)
{
	const auto same = [=](uint64_t k) { return (k >> shift) == pfx; };
	uint32_t a = f + 1, b = n;
	for (int e0 = 0; e0 < 32; e0 += 7) {
		uint64_t q[7];
		bool ok[7];
#pragma unroll
		for (int i = 0; i < 7; i++) {
			q[i] = (uint64_t)f + (1ull << (e0 + i));
			ok[i] = q[i] < n && same(keys[q[i]]);
		}
		bool left = false;
#pragma unroll
		for (int i = 0; i < 7; i++)
			if (ok[i]) a = (uint32_t)q[i] + 1;
#pragma unroll
		for (int i = 6; i >= 0; i--) {
			if (!ok[i]) {
				b = q[i] < n ? (uint32_t)q[i] : n;
				left = true;
			}
		}
		if (left) break;
	}
	return first_fail8(keys, a, b, same);
}

// s[c] for c = 1..7: the first slot of [f, e) whose child digit at `shift`
// is >= c; seven bisections side by side.
__device__ __forceinline__ void child_starts(const uint64_t* __restrict__ keys, uint32_t f, uint32_t e, int shift,
                                             uint32_t s[9])
{
	uint32_t lo[7], hi[7];
#pragma unroll
	for (int c = 0; c < 7; c++) {
		lo[c] = f;
		hi[c] = e;
	}
	for (uint32_t span = e - f; span > 0u; span >>= 1) {
#pragma unroll
		for (int c = 0; c < 7; c++) {
			if (lo[c] < hi[c]) {
				const uint32_t m = lo[c] + ((hi[c] - lo[c]) >> 1);
				if (((keys[m] >> shift) & 7u) < (uint32_t)(c + 1)) lo[c] = m + 1; else hi[c] = m;
			}
		}
	}
#pragma unroll
	for (int c = 0; c < 7; c++) s[c + 1] = lo[c];
}

// n consecutive items for each lane, from one counter, by a whole warp.
__device__ __forceinline__ uint32_t warp_take(unsigned int* ctr, uint32_t n)
{
	const int lane = threadIdx.x & 31;
	uint32_t incl = n;
#pragma unroll
	for (int o = 1; o < 32; o <<= 1) {
		const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
		if (lane >= o) incl += u;
	}
	uint32_t base = 0;
	if (lane == 31) base = atomicAdd(ctr, incl);
	return __shfl_sync(0xffffffffu, base, 31) + incl - n;
}

// Extents and children of the cells and, fast form, the places of their
// children's records, for the children there are.  Against eight places a cell a
// run takes 874 bytes a particle instead of 1,738 with leaf size 1, 423 instead
// of 475 with 16, and the walk reads fewer lines (678 -> 664 us at 1,000,001
// particles; this kernel 29 -> 30).  Places come from a counter, a warp's cells
// together: which warp comes first moves records, not what is computed.
template <class G>
__device__ __forceinline__ void finish_nodes_body(G grd, const uint64_t* __restrict__ keys, uint32_t n, uint32_t L,
                                                  const int8_t* __restrict__ lvl8, const uint32_t* __restrict__ base,
                                                  const TreeDev& T, unsigned int* rec_ctr, const Params& P, RunRec* rec)
{
	const bool fast = P.form == POT_FORM_FAST;
	const uint32_t M = rec->n_nodes;
	if (M > T.cap) {
		if (grd.id() == 0 && threadIdx.x == 0) set_status(rec, POT_E_CAPACITY);
		return;
	}
	const uint32_t whole = (M + 31u) & ~31u;  // whole warps
	for (uint32_t k = grd.id() * blockDim.x + threadIdx.x; k < whole; k += grd.n() * blockDim.x) {
		int l = 0;
		uint64_t pfx = 0;
		uint32_t s[9], nch = 0;
		if (k < M) {
			const uint32_t f = T.first[k];
			l = T.level[k];
			const int shift = 63 - 3 * l;
			pfx = keys[f] >> shift;
			// last particle of the cell
			const uint32_t last = cell_end(keys, f, n, shift, pfx) - 1;
			T.last[k] = last;
			// children by digit at the next level
			s[0] = f;
			s[8] = last + 1;
			child_starts(keys, f, last + 1, shift - 3, s);
#pragma unroll
			for (int c = 0; c < 8; c++) nch += s[c + 1] != s[c] ? 1u : 0u;
		}
		uint32_t place = fast ? 1u + warp_take(rec_ctr, nch) : 0u;
		if (k >= M) continue;
		T.ctr[k] = place;  // plain form: no arrivals yet
		int nint = 0;
#pragma unroll
		for (int c = 0; c < 8; c++) {
			const uint32_t cnt = s[c + 1] - s[c];
			int32_t code;
			if (cnt == 0) {
				code = CH_EMPTY;
			} else if (cnt <= L || l + 1 >= (int)P.max_level) {
				if (L == 1 && cnt == 1) {
					code = leaf_code(s[c]);
				} else if (L == 1) {
					const uint32_t j = atomicAdd(&rec->n_overflow, 1u);
					atomicOr(&rec->warn, 1u);
					if (j < OVF_CAP) {
						T.ovf[j] = make_uint2(s[c], cnt);
						code = leaf_code(n + j);
					} else {
						set_status(rec, POT_E_CAPACITY);
						code = CH_EMPTY;
					}
				} else {
					const uint32_t e = 8u * k + (uint32_t)c;
					code = leaf_code(e);
					T.lrange[e] = make_uint2(s[c], cnt);
				}
			} else {
				const uint32_t sc = s[c];
				const int lo = sc == 0 ? 0 : lvl8[sc - 1] + 1;
				const uint32_t kc = base[sc] + (uint32_t)(l + 1 - lo);
				if (sc + L >= n || kc >= M || kc <= k) {
					// cannot happen for a consistent key order; never write out of range
					set_status(rec, POT_E_CAPACITY);
					code = CH_EMPTY;
				} else {
					code = (int32_t)kc;
					T.parent[kc] = (int32_t)(fast ? place : k);
					nint++;
				}
			}
			T.child[8u * k + (uint32_t)c] = code;
			place += cnt != 0 ? 1u : 0u;
		}
		T.nint[k] = (uint8_t)nint;
		if (k == 0) T.parent[0] = -1;
		// x-extent of the cell by the reference's halving (pot.c:1262)
		double lo = 0.0, hi = P.root_w;
		for (int lev = 1; lev <= l; lev++) {
			const uint32_t bit = (uint32_t)(pfx >> (3 * (l - lev) + 2)) & 1u;
			const double mid = dmul(dadd(lo, hi), 0.5);
			if (bit) lo = mid; else hi = mid;
		}
		const double w = dsub(hi, lo);
		T.w2[k] = dmul(w, w);
	}
}

__global__ void k_finish_nodes(const uint64_t* __restrict__ keys, uint32_t n, uint32_t L,
                               const int8_t* __restrict__ lvl8, const uint32_t* __restrict__ base, TreeDev T,
                               unsigned int* rec_ctr, Params P, RunRec* rec)
{
	finish_nodes_body(GridSelf {}, keys, n, L, lvl8, base, T, rec_ctr, P, rec);
}

// running |q|-weighted update of pot.c:1290-1310
__device__ __forceinline__ void add_moment(int& q, uint32_t& aq, double& cx, double& cy, double& cz, int cq,
                                           uint32_t caq, double ccx, double ccy, double ccz)
{
	const double a0 = (double)aq, a1 = (double)caq, den = (double)(aq + caq);
	cx = ddiv(dadd(dmul(a0, cx), dmul(a1, ccx)), den);
	cy = ddiv(dadd(dmul(a0, cy), dmul(a1, ccy)), den);
	cz = ddiv(dadd(dmul(a0, cz), dmul(a1, ccz)), den);
	q += cq;
	aq += caq;
}

// DIPOLES (pot.c:1290-1310): the node's dipole moves to the new centre of
// |q|, then the child's, moved there too, is added; q and |q| last
__device__ __forceinline__ void add_moment_dip(int& q, uint32_t& aq, double& cx, double& cy, double& cz, double& px,
                                               double& py, double& pz, int cq, uint32_t caq, double ccx, double ccy,
                                               double ccz, double cpx, double cpy, double cpz)
{
	const double ox = cx, oy = cy, oz = cz;
	const double a0 = (double)aq, a1 = (double)caq, den = (double)(aq + caq);
	cx = ddiv(dadd(dmul(a0, cx), dmul(a1, ccx)), den);
	cy = ddiv(dadd(dmul(a0, cy), dmul(a1, ccy)), den);
	cz = ddiv(dadd(dmul(a0, cz), dmul(a1, ccz)), den);
	const double qd = (double)q, cqd = (double)cq;
	px = dsub(px, dmul(dsub(cx, ox), qd));
	py = dsub(py, dmul(dsub(cy, oy), qd));
	pz = dsub(pz, dmul(dsub(cz, oz), qd));
	px = dadd(px, dsub(cpx, dmul(dsub(cx, ccx), cqd)));
	py = dadd(py, dsub(cpy, dmul(dsub(cy, ccy), cqd)));
	pz = dadd(pz, dsub(cpz, dmul(dsub(cz, ccz), cqd)));
	q += cq;
	aq += caq;
}

// The moments of cell k's children in member order, children with buckets or
// dipoles among them.
struct CellMoments {
	int q;
	uint32_t aq;
	double c[3], p[3];
};
__device__ __noinline__ CellMoments cell_moments_general(const TreeDev& T, const double4* __restrict__ src64,
                                                         const Params& P, uint32_t k)
{
	const bool dip = T.dip != nullptr;
	int q = 0;
	uint32_t aq = 0;
	double cx = 0.0, cy = 0.0, cz = 0.0;
	double px = 0.0, py = 0.0, pz = 0.0;
	for (int s = 0; s < 8; s++) {
		const int d = slot_digit(s);
		const int32_t code = T.child[8u * k + (uint32_t)d];
		if (code == CH_EMPTY) continue;
		int cq;
		uint32_t caq;
		double ccx, ccy, ccz;
		double cpx = 0.0, cpy = 0.0, cpz = 0.0;
		if (code >= 0) {
			cq = __ldcg(&T.q[code]);
			caq = __ldcg(&T.aq[code]);
			const double2* cp2 = reinterpret_cast<const double2*>(&T.cq[code]);
			const double2 c01 = __ldcg(cp2), c23 = __ldcg(cp2 + 1);
			const double4 c = make_double4(c01.x, c01.y, c23.x, c23.y);
			ccx = c.x; ccy = c.y; ccz = c.z;
			if (dip) {
				const double2* dp2 = reinterpret_cast<const double2*>(&T.dip[code]);
				const double2 d01 = __ldcg(dp2), d23 = __ldcg(dp2 + 1);
				cpx = d01.x; cpy = d01.y; cpz = d23.x;
			}
		} else if (leaf_payload(code) < P.n_tree) {
			const double4 sp = src64[leaf_payload(code)];
			cq = (int)sp.w;
			caq = (uint32_t)abs(cq);
			ccx = sp.x; ccy = sp.y; ccz = sp.z;
		} else {
			// overflow bucket: its own running moments over its particles
			const uint32_t e = leaf_payload(code);
			const uint2 r = T.ovf[e - P.n_tree];
			cq = 0;
			caq = 0;
			ccx = ccy = ccz = 0.0;
			for (uint32_t j = r.x; j < r.x + r.y; j++) {
				const double4 sp = src64[j];
				const int pq = (int)sp.w;
				const uint32_t paq = (uint32_t)abs(pq);
				if (!paq) continue;
				if (dip) {
					add_moment_dip(cq, caq, ccx, ccy, ccz, cpx, cpy, cpz, pq, paq, sp.x, sp.y, sp.z, 0.0, 0.0,
					               0.0);
				} else {
					add_moment(cq, caq, ccx, ccy, ccz, pq, paq, sp.x, sp.y, sp.z);
				}
			}
		}
		if (caq) {
			if (dip) {
				add_moment_dip(q, aq, cx, cy, cz, px, py, pz, cq, caq, ccx, ccy, ccz, cpx, cpy, cpz);
			} else {
				add_moment(q, aq, cx, cy, cz, cq, caq, ccx, ccy, ccz);
			}
		}
	}
	return CellMoments { q, aq, { cx, cy, cz }, { px, py, pz } };
}

// Plain form (leaf size 1): the reference's running update bottom-up, a thread
// a cell, the last child's thread going on to the parent.  The chain of cells
// from the deepest pair to the root sets the time, so a cell's child codes are
// loaded at once and its children's moments two ahead of their update: 64 -> 51
// us at 8,193 particles, 81 -> 65 at 150,001, 268 -> 222 at 1,000,001.
__global__ void __launch_bounds__(256, 3) k_moments(TreeDev T, const double4* __restrict__ src64, Params P, RunRec* rec)
{
	const uint32_t M = rec->n_nodes;
	if (M > T.cap) return;
	const bool dip = T.dip != nullptr;
	for (uint32_t k0 = blockIdx.x * blockDim.x + threadIdx.x; k0 < M; k0 += gridDim.x * blockDim.x) {
		if (T.nint[k0] != 0) continue;
		uint32_t k = k0;
		for (;;) {
			const int4* row = reinterpret_cast<const int4*>(&T.child[8u * k]);
			const int4 r0 = row[0], r1 = row[1];
			// member order (slot_digit)
			const int32_t code[8] = { r1.x, r1.y, r0.x, r0.y, r0.z, r0.w, r1.z, r1.w };
			const int32_t p = T.parent[k];
			// parents precede children in pre-order; a cell that none claimed (keys
			// out of order after a sort that gave up) holds any value
			const bool orphan = k != 0 && (p < 0 || (uint32_t)p >= k);
			const uint32_t nint = k != 0 && !orphan ? T.nint[p] : 0u;
			bool plain = !dip;
#pragma unroll
			for (int s = 0; s < 8; s++) plain = plain && (code[s] >= CH_EMPTY || leaf_payload(code[s]) < P.n_tree);
			int q = 0;
			uint32_t aq = 0;
			double cx = 0.0, cy = 0.0, cz = 0.0, px = 0.0, py = 0.0, pz = 0.0;
			if (plain) {
				// the next two children's moments are on the way during a child's
				// update (its divisions)
				double4 ch[3];
				uint32_t ca[3];
				const auto fetch = [&](int32_t cd, double4& m, uint32_t& w) {
					w = 0;
					if (cd >= 0) {
						const double2* cp = reinterpret_cast<const double2*>(&T.cq[cd]);
						const double2 a = __ldcg(cp), b = __ldcg(cp + 1);
						m = make_double4(a.x, a.y, b.x, b.y);  // its charge is in .w, exactly
						w = __ldcg(&T.aq[cd]);
					} else if (cd != CH_EMPTY) {
						m = src64[leaf_payload(cd)];
						w = (uint32_t)abs((int)m.w);
					}
				};
				fetch(code[0], ch[0], ca[0]);
				fetch(code[1], ch[1], ca[1]);
#pragma unroll
				for (int s = 0; s < 8; s++) {
					if (s < 6) fetch(code[s + 2], ch[(s + 2) % 3], ca[(s + 2) % 3]);
					asm volatile("" ::: "memory");
					const double4 m = ch[s % 3];
					const uint32_t w = ca[s % 3];
					if (w) add_moment(q, aq, cx, cy, cz, (int)m.w, w, m.x, m.y, m.z);
				}
			} else {
				const CellMoments m = cell_moments_general(T, src64, P, k);
				q = m.q;
				aq = m.aq;
				cx = m.c[0]; cy = m.c[1]; cz = m.c[2];
				px = m.p[0]; py = m.p[1]; pz = m.p[2];
			}
			T.q[k] = q;
			T.aq[k] = aq;
			T.cq[k] = make_double4(cx, cy, cz, (double)q);
			if (dip) T.dip[k] = make_double4(px, py, pz, 0.0);
			if (k == 0) break;
			if (orphan) {
				set_status(rec, POT_E_CAPACITY);
				break;
			}
			__threadfence();
			const uint32_t arrived = atomicAdd(&T.ctr[p], 1u) + 1u;
			if (arrived != nint) break;
			__threadfence();
			k = (uint32_t)p;
		}
	}
}

// ---------------------------------------------------------------------------
// Fast form moments from prefix sums.  With particles in Morton order every
// cell and bucket leaf is a contiguous slot range [a, b), so its net charge,
// absolute charge and |q|-weighted position sums are differences of
// exclusive prefix sums P[b] - P[a] of (q, |q|, |q|(x - c), |q|(y - c),
// |q|(z - c)), c the domain centre.  FP64 sums: with |x - c| <= R the
// cancellation error of a difference is ~1e-16 of the largest prefix, far
// below the FP32 resolution the fast walk uses.
// ---------------------------------------------------------------------------
struct Mom5 {
	double q, a, x, y, z;
};

__device__ __forceinline__ Mom5 mom_add(const Mom5& u, const Mom5& v)
{
	return Mom5 { u.q + v.q, u.a + v.a, u.x + v.x, u.y + v.y, u.z + v.z };
}

// K = 0: (q, |q|, |q| x, |q| y, |q| z); K = 1 (DIPOLES): (q x, q y, q z, 0, 0);
// positions relative to the domain centre c
template <int K>
__device__ __forceinline__ Mom5 mom_of(const double4& p, double c)
{
	if (K == 1) return Mom5 { p.w * (p.x - c), p.w * (p.y - c), p.w * (p.z - c), 0.0, 0.0 };
	const double a = fabs(p.w);
	return Mom5 { p.w, a, a * (p.x - c), a * (p.y - c), a * (p.z - c) };
}

__device__ __forceinline__ Mom5 mom_shfl_up(const Mom5& m, int o)
{
	return Mom5 { __shfl_up_sync(0xffffffffu, m.q, o), __shfl_up_sync(0xffffffffu, m.a, o),
	              __shfl_up_sync(0xffffffffu, m.x, o), __shfl_up_sync(0xffffffffu, m.y, o),
	              __shfl_up_sync(0xffffffffu, m.z, o) };
}

constexpr int MOM_THREADS = 256;
constexpr int MOM_ITEMS = 16;
constexpr int MOM_TILE = MOM_THREADS * MOM_ITEMS;

// exclusive block scan of one Mom5 per thread; *tot = block total
__device__ Mom5 mom_block_excl(Mom5 v, Mom5* tot)
{
	__shared__ Mom5 wsum[MOM_THREADS / 32];
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
	Mom5 inc = v;
#pragma unroll
	for (int o = 1; o < 32; o <<= 1) {
		const Mom5 t = mom_shfl_up(inc, o);
		if (lane >= o) inc = mom_add(inc, t);
	}
	if (lane == 31) wsum[w] = inc;
	__syncthreads();
	if (threadIdx.x == 0) {
		Mom5 run = Mom5 { 0, 0, 0, 0, 0 };
		for (int k = 0; k < MOM_THREADS / 32; k++) {
			const Mom5 t = wsum[k];
			wsum[k] = run;
			run = mom_add(run, t);
		}
		*tot = run;
	}
	__syncthreads();
	const Mom5 excl = mom_add(wsum[w], Mom5 { inc.q - v.q, inc.a - v.a, inc.x - v.x, inc.y - v.y, inc.z - v.z });
	__syncthreads();
	return excl;
}

// Each warp owns a contiguous chunk of MOM_ITEMS * 32 particles of the tile
// and walks it 32 at a time (coalesced loads).
__device__ __forceinline__ Mom5 mom_warp_incl(Mom5 v)
{
	const int lane = threadIdx.x & 31;
#pragma unroll
	for (int o = 1; o < 32; o <<= 1) {
		const Mom5 t = mom_shfl_up(v, o);
		if (lane >= o) v = mom_add(v, t);
	}
	return v;
}

__device__ __forceinline__ Mom5 mom_shfl(const Mom5& m, int src)
{
	return Mom5 { __shfl_sync(0xffffffffu, m.q, src), __shfl_sync(0xffffffffu, m.a, src),
	              __shfl_sync(0xffffffffu, m.x, src), __shfl_sync(0xffffffffu, m.y, src),
	              __shfl_sync(0xffffffffu, m.z, src) };
}

template <int K, class G>
__device__ __forceinline__ void mom_reduce_body(G grd, const double4* __restrict__ src64, uint32_t n, double c,
                                                Mom5* __restrict__ bsum)
{
	__shared__ Mom5 tot;
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
	const size_t base = (size_t)grd.id() * MOM_TILE + (size_t)w * (MOM_ITEMS * 32);
	Mom5 s = Mom5 { 0, 0, 0, 0, 0 };
	for (int k = 0; k < MOM_ITEMS; k++) {
		const size_t i = base + (size_t)k * 32 + lane;
		if (i < n) s = mom_add(s, mom_of<K>(src64[i], c));
	}
	mom_block_excl(s, &tot);
	if (threadIdx.x == 0) bsum[grd.id()] = tot;
}

template <int K>
__global__ void __launch_bounds__(MOM_THREADS) k_mom_reduce(const double4* __restrict__ src64, uint32_t n, double c,
                                                            Mom5* __restrict__ bsum)
{
	mom_reduce_body<K>(GridSelf {}, src64, n, c, bsum);
}

// Sum of the block totals before block `id`, added in a fixed order: block
// scans of MOM_THREADS totals and a running carry.  Every block works its
// own out, so no launch is needed between the totals and their use.
__device__ Mom5 mom_before(const Mom5* __restrict__ bsum, uint32_t id)
{
	__shared__ Mom5 tot, mine;
	Mom5 carry = Mom5 { 0, 0, 0, 0, 0 };
	for (uint32_t base = 0;; base += MOM_THREADS) {
		const uint32_t i = base + threadIdx.x;
		const Mom5 v = i <= id ? bsum[i] : Mom5 { 0, 0, 0, 0, 0 };  // its own enters the scan it is left out of
		const Mom5 e = mom_block_excl(v, &tot);
		if (i == id) mine = mom_add(carry, e);
		if (id < base + MOM_THREADS) break;
		carry = mom_add(carry, tot);
		__syncthreads();
	}
	__syncthreads();
	return mine;
}

template <int K, class G>
__device__ __forceinline__ void mom_down_body(G grd, const double4* __restrict__ src64, uint32_t n, double c,
                                              const Mom5* __restrict__ bsum, Mom5* __restrict__ pre)
{
	__shared__ Mom5 tot;
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
	const size_t base = (size_t)grd.id() * MOM_TILE + (size_t)w * (MOM_ITEMS * 32);
	// this warp's chunk total, then its offset among the block's warps
	Mom5 s = Mom5 { 0, 0, 0, 0, 0 };
	for (int k = 0; k < MOM_ITEMS; k++) {
		const size_t i = base + (size_t)k * 32 + lane;
		if (i < n) s = mom_add(s, mom_of<K>(src64[i], c));
	}
	// reduce the per-lane partial sums to the warp total on lane 0
	Mom5 wt = s;
#pragma unroll
	for (int o = 16; o; o >>= 1) {
		wt = mom_add(wt, Mom5 { __shfl_xor_sync(0xffffffffu, wt.q, o), __shfl_xor_sync(0xffffffffu, wt.a, o),
		                        __shfl_xor_sync(0xffffffffu, wt.x, o), __shfl_xor_sync(0xffffffffu, wt.y, o),
		                        __shfl_xor_sync(0xffffffffu, wt.z, o) });
	}
	const Mom5 mine = lane == 0 ? wt : Mom5 { 0, 0, 0, 0, 0 };
	const Mom5 before = mom_before(bsum, grd.id());
	Mom5 carry = mom_add(before, mom_block_excl(mine, &tot));  // valid on lane 0
	carry = mom_shfl(carry, 0);
	for (int k = 0; k < MOM_ITEMS; k++) {
		const size_t i = base + (size_t)k * 32 + lane;
		const Mom5 v = i < n ? mom_of<K>(src64[i], c) : Mom5 { 0, 0, 0, 0, 0 };
		const Mom5 inc = mom_warp_incl(v);
		if (i < n) {
			pre[i] = mom_add(carry, Mom5 { inc.q - v.q, inc.a - v.a, inc.x - v.x, inc.y - v.y, inc.z - v.z });
			if (i + 1 == n) pre[n] = mom_add(carry, inc);
		}
		carry = mom_add(carry, mom_shfl(inc, 31));
	}
}

template <int K>
__global__ void __launch_bounds__(MOM_THREADS) k_mom_down(const double4* __restrict__ src64, uint32_t n, double c,
                                                          const Mom5* __restrict__ bsum, Mom5* __restrict__ pre)
{
	mom_down_body<K>(GridSelf {}, src64, n, c, bsum, pre);
}

__device__ __forceinline__ Mom5 mom_range(const Mom5* __restrict__ pre, uint32_t a, uint32_t b)
{
	const Mom5 u = pre[b], v = pre[a];
	return Mom5 { u.q - v.q, u.a - v.a, u.x - v.x, u.y - v.y, u.z - v.z };
}

// DIPOLES: the dipole about the centre of |q| from the prefix sums of q x
// (pd) and the cell's charge and centre (relative to the domain centre),
// p = sum q (x - c) = sum q x - Q c
__device__ __forceinline__ double3 dipole_of(const Mom5& pd, double q, double cx, double cy, double cz)
{
	return make_double3(pd.q - q * cx, pd.a - q * cy, pd.x - q * cz);
}

__device__ __forceinline__ void put_rec(NodeRec* rec, float x, float y, float z, float q, float r2, uint32_t base,
                                        uint32_t info)
{
	uint4* o = reinterpret_cast<uint4*>(rec);
	o[0] = make_uint4(__float_as_uint(x), __float_as_uint(y), __float_as_uint(z), __float_as_uint(q));
	o[1] = make_uint4(__float_as_uint(r2), base, info, 0u);
}

// Eight lanes a cell: each writes its child's record if that is a leaf, the
// first the cell's own moments and record.
template <class G>
__device__ __forceinline__ void moments_prefix_body(G grd, const TreeDev& T, const Mom5* __restrict__ pre,
                                                    const Mom5* __restrict__ pre_d, const Params& P, RunRec* rec)
{
	const uint32_t M = rec->n_nodes;
	if (M > T.cap) return;
	const uint32_t L = P.leaf_size, d = threadIdx.x & 7u, spare = T.spare;
	const uint32_t n = (8u * M + 31u) & ~31u;  // whole warps
	for (uint32_t i = grd.id() * blockDim.x + threadIdx.x; i < n; i += grd.n() * blockDim.x) {
		const uint32_t k = i >> 3;
		const int32_t code = k < M ? T.child[i] : CH_EMPTY;
		const uint32_t mask = (__ballot_sync(0xffffffffu, code != CH_EMPTY) >> (threadIdx.x & 24u)) & 0xFFu;
		// Of a cell that no parent claimed (keys out of order after a sort that
		// gave up) the place holds any value: none leads past the records.
		const uint32_t base = k < M ? T.ctr[k] : 0u;
		if (code < CH_EMPTY) {
			const uint32_t e = leaf_payload(code);
			const uint32_t o = min(base + __popc(mask & ((1u << d) - 1u)), spare);
			if (L > 1) {
				const float w_child = 0.5f * (float)(sqrt(T.w2[k]) * P.inv_rad);
				const uint2 r = T.lrange[e];
				const Mom5 lm = mom_range(pre, r.x, r.x + r.y);
				const double li = lm.a > 0.0 ? 1.0 / lm.a : 0.0;
				put_rec(&T.nrec[o], (float)(lm.x * li * P.inv_rad), (float)(lm.y * li * P.inv_rad),
				        (float)(lm.z * li * P.inv_rad), (float)llrint(lm.q), w_child * w_child / P.oap2_f, r.x,
				        NR_LEAF | r.y);
				if (pre_d) {
					const double3 dl = dipole_of(mom_range(pre_d, r.x, r.x + r.y), (double)llrint(lm.q), lm.x * li,
					                             lm.y * li, lm.z * li);
					T.drec[o] = make_float4((float)(dl.x * P.inv_rad), (float)(dl.y * P.inv_rad),
					                        (float)(dl.z * P.inv_rad), 0.f);
				}
			} else {
				const uint2 r = e < P.n_tree ? make_uint2(e, 1u) : T.ovf[e - P.n_tree];
				put_rec(&T.nrec[o], 0.f, 0.f, 0.f, 0.f, 0.f, r.x, NR_LEAF | NR_UNTESTED | r.y);
			}
		}
		if (d != 0 || k >= M) continue;
		const uint32_t a = T.first[k], b = T.last[k] + 1;
		const Mom5 m = mom_range(pre, a, b);
		const double inv = m.a > 0.0 ? 1.0 / m.a : 0.0;
		const double cx = m.x * inv, cy = m.y * inv, cz = m.z * inv;  // relative to the centre
		const int q = (int)llrint(m.q);
		T.q[k] = q;
		T.aq[k] = (uint32_t)llrint(m.a);
		T.cq[k] = make_double4(cx + P.rad, cy + P.rad, cz + P.rad, (double)q);
		const uint32_t o = k == 0 ? 0u : min((uint32_t)T.parent[k], spare);
		put_rec(&T.nrec[o], (float)(cx * P.inv_rad), (float)(cy * P.inv_rad), (float)(cz * P.inv_rad), (float)q,
		        (float)(T.w2[k] * P.inv_rad * P.inv_rad / P.oap2), base, __popc(mask));
		if (pre_d) {
			const double3 dc = dipole_of(mom_range(pre_d, a, b), (double)q, cx, cy, cz);
			T.dip[k] = make_double4(dc.x, dc.y, dc.z, 0.0);
			T.drec[o] = make_float4((float)(dc.x * P.inv_rad), (float)(dc.y * P.inv_rad), (float)(dc.z * P.inv_rad), 0.f);
		}
	}
}

__global__ void k_moments_prefix(TreeDev T, const Mom5* __restrict__ pre, const Mom5* __restrict__ pre_d, Params P,
                                 RunRec* rec)
{
	moments_prefix_body(GridSelf {}, T, pre, pre_d, P, rec);
}

// Blocks of the cells' moments kernel: eight lanes a cell, of which there are
// about n / 2 with leaf size 1 and n / (2 L) or fewer with larger leaves.
uint32_t mom_cell_blocks(size_t n, uint32_t leaf) { return (uint32_t)((std::max(n / 4, 4 * n / leaf) + 256) / 256); }

size_t mom_prefix_entries(size_t n) { return n + 1; }
size_t mom_block_entries(size_t n) { return (n + MOM_TILE - 1) / MOM_TILE + 1; }

// ---------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------
static inline uint32_t blocks_for(size_t n, int threads) { return (uint32_t)((n + threads - 1) / threads); }

// The keys kernel's grid: a block per 256 particles up to eight blocks per
// SM, then grid-stride (each block adds its digit counts once).
uint32_t keys_blocks(size_t n) { return std::min<uint32_t>(blocks_for(n, 256), 148u * 8u); }

void launch_keys(const double4* pos, uint64_t* keys, uint32_t* vals, const Params& P, RunRec* rec,
                 int begin_step, uint32_t* words, cudaStream_t s, Timer& tm)
{
	ScopedKernel k(tm, "keys");
	k_keys<<<keys_blocks(P.n), 256, 0, s>>>(pos, keys, vals, P, rec, begin_step, words, (int)P.key_bits,
	                                        radix_passes((int)P.key_bits));
}

void launch_reorder(const uint32_t* perm, const double4* pos_in, const double4* vel_in, const uint32_t* pid_in,
                    double4* pos_out, double4* vel_out, uint32_t* pid_out, double4* src64, float4* src32,
                    uint8_t* due, uint32_t* words, const Params& P, RunRec* rec, cudaStream_t s, Timer& tm)
{
	ScopedKernel k(tm, "reorder");
	k_reorder<<<blocks_for(P.n, REORDER_THREADS), REORDER_THREADS, 0, s>>>(perm, pos_in, vel_in, pid_in, pos_out, vel_out,
	                                                                       pid_out, src64, src32, due, words, P, rec);
}

void launch_due_list(const uint8_t* due, uint32_t* words, uint32_t* due_list, uint32_t* due_prefix, const Params& P,
                     RunRec* rec, cudaStream_t s, Timer& tm)
{
	ScopedKernel k(tm, "due_list");
	k_due_list<<<StepWords::due_tiles(P.n), TILE_THREADS, 0, s>>>(due, StepWords(words, P.n).due, due_list, due_prefix,
	                                                             P, rec);
}

// Topology from the sorted keys: cell numbering, extents and children.
void launch_cells(const uint64_t* keys, const uint32_t* perm, const double4* pos_in, TreeDev& T, const Params& P,
                  RunRec* rec, uint32_t* words, cudaStream_t s, Timer& tm)
{
	const uint32_t n = P.n_tree, L = P.leaf_size;
	const uint32_t n_pairs = n - L;  // n_tree > L is checked at creation
	{
		ScopedKernel k(tm, "tree_cells", 2);
		uint32_t* counts = StepWords(words, P.n).cell;
		const uint32_t nb = StepWords::cell_tiles(n_pairs);
		k_cell_count<<<nb, TILE_THREADS, 0, s>>>(keys, perm, pos_in, n_pairs, L, (int)P.max_level, counts, rec);
		k_cell_number<<<nb, TILE_THREADS, 0, s>>>(keys, n_pairs, L, (int)P.max_level, counts, T, rec);
	}
	ScopedKernel k(tm, "tree_finish");
	k_finish_nodes<<<blocks_for(n, 256), 256, 0, s>>>(keys, n, L, T.lvl8, T.base, T, StepWords(words, P.n).rec_ctr, P,
	                                                  rec);
}

// Fast form: prefix sums of the moments over the reordered particles.
void launch_mom_sums(TreeDev& T, const double4* src64, const Params& P, cudaStream_t s, Timer& tm)
{
	if (P.form != POT_FORM_FAST) return;
	const uint32_t n = P.n_tree, nb = (uint32_t)((n + MOM_TILE - 1) / MOM_TILE);
	ScopedKernel k(tm, "moment_sums", T.mom_pre_d ? 4 : 2);
	Mom5* bs = reinterpret_cast<Mom5*>(T.mom_blk);
	k_mom_reduce<0><<<nb, MOM_THREADS, 0, s>>>(src64, n, P.rad, bs);
	k_mom_down<0><<<nb, MOM_THREADS, 0, s>>>(src64, n, P.rad, bs, reinterpret_cast<Mom5*>(T.mom_pre));
	if (T.mom_pre_d) {  // DIPOLES: prefix sums of q x as well
		Mom5* bs_d = reinterpret_cast<Mom5*>(T.mom_blk_d);
		k_mom_reduce<1><<<nb, MOM_THREADS, 0, s>>>(src64, n, P.rad, bs_d);
		k_mom_down<1><<<nb, MOM_THREADS, 0, s>>>(src64, n, P.rad, bs_d, reinterpret_cast<Mom5*>(T.mom_pre_d));
	}
}

// The cells' moments, from the prefix sums (fast form) or bottom-up.
void launch_moments(TreeDev& T, const double4* src64, const Params& P, RunRec* rec, cudaStream_t s, Timer& tm)
{
	const uint32_t n = P.n_tree;
	ScopedKernel k(tm, "tree_moments");
	if (P.form == POT_FORM_FAST) {
		k_moments_prefix<<<mom_cell_blocks(n, P.leaf_size), 256, 0, s>>>(
			T, reinterpret_cast<const Mom5*>(T.mom_pre), reinterpret_cast<const Mom5*>(T.mom_pre_d), P, rec);
	} else {
		k_moments<<<blocks_for(n, 256), 256, 0, s>>>(T, src64, P, rec);
	}
}

}  // namespace pot

// ---------------------------------------------------------------------------
// packed batch: the same kernels, one launch over every member
// ---------------------------------------------------------------------------
namespace pot {

__global__ void __launch_bounds__(256) kp_keys(PackDev B, int k)
{
	const SegBlock sb = seg_block(B.pre[PS_KEYS], B.M);
	const MemberView& v = B.mv[sb.m];
	const StepWords W(v.words, v.P.n);
	keys_body(GridSeg { sb.id, sb.n }, v.pos[pack_in(v, k)], v.keys[0], v.vals[0], v.P, v.rec, 1, W.hist, W.keys_ctr,
	          (int)v.P.key_bits, (int)B.npass);
}

__global__ void __launch_bounds__(REORDER_THREADS) kp_reorder(PackDev B, int k)
{
	const SegBlock sb = seg_block(B.pre[PS_N256], B.M);
	const MemberView& v = B.mv[sb.m];
	const uint32_t a = pack_in(v, k), b = pack_out(v, k);
	reorder_body(GridSeg { sb.id, sb.n }, v.vals[v.kb], v.pos[a], v.vel[a], v.pid[a], v.pos[b], v.vel[b],
	             v.pid[b], v.src64, v.src32, v.due, StepWords(v.words, v.P.n).due, v.P, v.rec);
}

__global__ void __launch_bounds__(TILE_THREADS) kp_due_list(PackDev B)
{
	const SegBlock sb = seg_block(B.pre[PS_DUE], B.M);
	const MemberView& v = B.mv[sb.m];
	due_list_body(GridSeg { sb.id, sb.n }, v.due, StepWords(v.words, v.P.n).due, v.due_list, v.due_prefix, v.P, v.rec);
}

__global__ void __launch_bounds__(TILE_THREADS) kp_cell_count(PackDev B, int k)
{
	const SegBlock sb = seg_block(B.pre[PS_CELLS], B.M);
	const MemberView& v = B.mv[sb.m];
	cell_count_body(GridSeg { sb.id, sb.n }, v.keys[v.kb], v.vals[v.kb], v.pos[pack_in(v, k)],
	                v.P.n_tree - v.P.leaf_size, v.P.leaf_size,
	                (int)v.P.max_level, StepWords(v.words, v.P.n).cell, v.rec);
}

__global__ void __launch_bounds__(TILE_THREADS) kp_cell_number(PackDev B)
{
	const SegBlock sb = seg_block(B.pre[PS_CELLS], B.M);
	const MemberView& v = B.mv[sb.m];
	cell_number_body(GridSeg { sb.id, sb.n }, v.keys[v.kb], v.P.n_tree - v.P.leaf_size, v.P.leaf_size,
	                 (int)v.P.max_level, StepWords(v.words, v.P.n).cell, v.T, v.rec);
}

__global__ void kp_finish_nodes(PackDev B)
{
	const SegBlock sb = seg_block(B.pre[PS_FINISH], B.M);
	const MemberView& v = B.mv[sb.m];
	finish_nodes_body(GridSeg { sb.id, sb.n }, v.keys[v.kb], v.P.n_tree, v.P.leaf_size, v.T.lvl8, v.T.base, v.T,
	                  StepWords(v.words, v.P.n).rec_ctr, v.P, v.rec);
}

__global__ void __launch_bounds__(MOM_THREADS) kp_mom_reduce(PackDev B)
{
	const SegBlock sb = seg_block(B.pre[PS_MOM], B.M);
	const MemberView& v = B.mv[sb.m];
	mom_reduce_body<0>(GridSeg { sb.id, sb.n }, v.src64, v.P.n_tree, v.P.rad, reinterpret_cast<Mom5*>(v.T.mom_blk));
}

__global__ void __launch_bounds__(MOM_THREADS) kp_mom_down(PackDev B)
{
	const SegBlock sb = seg_block(B.pre[PS_MOM], B.M);
	const MemberView& v = B.mv[sb.m];
	mom_down_body<0>(GridSeg { sb.id, sb.n }, v.src64, v.P.n_tree, v.P.rad, reinterpret_cast<Mom5*>(v.T.mom_blk),
	                 reinterpret_cast<Mom5*>(v.T.mom_pre));
}

__global__ void kp_moments_prefix(PackDev B)
{
	const SegBlock sb = seg_block(B.pre[PS_MOMPRE], B.M);
	const MemberView& v = B.mv[sb.m];
	moments_prefix_body(GridSeg { sb.id, sb.n }, v.T, reinterpret_cast<const Mom5*>(v.T.mom_pre), nullptr, v.P,
	                    v.rec);
}

static_assert(MOM_TILE == (int)PACK_MOM_TILE, "moment tile");

void pack_keys(const PackDev& B, int k, cudaStream_t s)
{
	kp_keys<<<B.blocks[PS_KEYS], 256, 0, s>>>(B, k);
}

void pack_reorder(const PackDev& B, int k, cudaStream_t s)
{
	kp_reorder<<<B.blocks[PS_N256], REORDER_THREADS, 0, s>>>(B, k);
}

void pack_due_list(const PackDev& B, cudaStream_t s)
{
	kp_due_list<<<B.blocks[PS_DUE], TILE_THREADS, 0, s>>>(B);
}

void pack_cells(const PackDev& B, int k, cudaStream_t s)
{
	kp_cell_count<<<B.blocks[PS_CELLS], TILE_THREADS, 0, s>>>(B, k);
	kp_cell_number<<<B.blocks[PS_CELLS], TILE_THREADS, 0, s>>>(B);
	kp_finish_nodes<<<B.blocks[PS_FINISH], 256, 0, s>>>(B);
}

void pack_mom_sums(const PackDev& B, cudaStream_t s)
{
	kp_mom_reduce<<<B.blocks[PS_MOM], MOM_THREADS, 0, s>>>(B);
	kp_mom_down<<<B.blocks[PS_MOM], MOM_THREADS, 0, s>>>(B);
}

void pack_moments(const PackDev& B, cudaStream_t s)
{
	kp_moments_prefix<<<B.blocks[PS_MOMPRE], 256, 0, s>>>(B);
}

}  // namespace pot
