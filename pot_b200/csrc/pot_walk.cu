// Barnes-Hut walks fused with the Boris push, grain absorption and the
// boundary test; potential energies, point queries, edge potential (chi_b).
//
// Plain form (POT_FORM_PLAIN): FP64, leaf size 1.  Every target makes its own
// accept/open decisions with the reference's unfused opening test
// (pot.c:1719-1772), so its terms are exactly the reference's; the terms
// (pot.c:1737-1749, 1789-1798) are evaluated and summed in FP64 with fused
// multiply-adds, where the reference accumulates in x87 long double.
//
// Fast form (POT_FORM_FAST): see pot_walk_fast.cu.
#include "pot_push.cuh"

namespace pot {

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31u; }

// One 32-byte load of data that the kernel does not write.
__device__ __forceinline__ double4 ld_nc(const double4* p)
{
	double4 r;
	asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(r.x), "=d"(r.y), "=d"(r.z), "=d"(r.w) : "l"(p));
	return r;
}

// A target's sum: the field, or the potential in x.
struct PlainAcc {
	double x, y, z;
};

// 1 / sqrt(x) to FP64 rounding, for normal positive x and without branches:
// the hardware's approximation y0 keeps 20 fraction bits, so y0^2 is exact
// and e = 1 - x y0^2 has one rounding of its own; then x^(-p/2) is
// y0^p (1 - e)^(-p/2), the binomial series in e (|e| < 2^-17) to third order.
struct Rsqrt {
	double y0, y02, e;
	__device__ __forceinline__ explicit Rsqrt(double x)
	{
		asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(x));
		y02 = y0 * y0;
		e = fma(-x, y02, 1.0);
	}
	// s x^(-1/2), s / x and s x^(-3/2)
	__device__ __forceinline__ double p1(double s) const
	{
		const double w = s * y0;
		return fma(w, e * fma(e, fma(e, 0.3125, 0.375), 0.5), w);
	}
	__device__ __forceinline__ double p2(double s) const
	{
		const double w = s * y02;
		return fma(w, e * fma(e, 1.0 + e, 1.0), w);
	}
	__device__ __forceinline__ double p3(double s) const
	{
		const double w = s * (y02 * y0);
		return fma(w, e * fma(e, fma(e, 2.1875, 1.875), 1.5), w);
	}
};

// One term of the sum at offset (dx, dy, dz), squared distance d2 (of a
// particle, softened; of a cell, not): kq is QE q / (4 pi eps0).  A term
// whose bit is not set (on) adds zero; dip implies on.
template <bool PHI, bool DIP>
__device__ __forceinline__ void plain_term(PlainAcc& E, bool on, bool dip, const double4& pd, double kq, double dx,
                                           double dy, double dz, double d2)
{
	const Rsqrt r(d2);
	if (PHI) {
		double v = r.p1(kq);  // pot.c:1960-1973
		if (DIP && dip) v += r.p3(fma(dx, pd.x, fma(dy, pd.y, dz * pd.z)));
		E.x += on ? v : 0.0;
	} else {
		double es = r.p3(kq);  // pot.c:1737-1749, 1789-1798
		if (DIP && dip) {  // DIPOLES, pot.c:1739-1745: (q + 3 (p.r) / r^2) r / r^3 - p / r^3
			es = r.p3(kq + 3.0 * r.p2(fma(dx, pd.x, fma(dy, pd.y, dz * pd.z))));
			const double n3 = r.p3(-1.0);
			E.x = fma(n3, pd.x, E.x);
			E.y = fma(n3, pd.y, E.y);
			E.z = fma(n3, pd.z, E.z);
		}
		es = on ? es : 0.0;
		E.x = fma(es, dx, E.x);
		E.y = fma(es, dy, E.y);
		E.z = fma(es, dz, E.z);
	}
}

// The walk: a warp walks the tree once for G targets, keeping every target's
// own decisions.  A stack entry is a node and the mask of the targets that
// have opened all of its ancestors.  Each lane takes one node a round and
// makes the reference's unfused test (pot.c:1719-1803) for each of the G
// targets: a cell some of them accept goes to a list with their mask, and
// its children are pushed with the mask of those that open it; a particle
// goes to the list with its mask less the target that is that particle.
// Whole 32-entry lists are then evaluated with the lanes split into G targets
// by 32 / G entries, each lane skipping the entries its target's bit is not
// set in.  So every target's terms are the reference's; only the order of
// its FP64 sum differs.
//
// What bounds it: with many targets instruction issue and the FP64 pipe (at
// 1,000,001 particles 68 % of issue slots, 50 % of the FP64 pipe, 73 % of the
// shared-memory wavefronts, 26 of 32 lanes active); with few, the latency of
// each warp's chain of rounds (8,193 particles: 12 warps an SM, 23 % of issue
// slots over the launch).  A walk of one thread per target, the form before, ran
// 17 of 32 lanes on average through three divergent paths and waited on its
// stack in local memory.  Sharing a node's load, stack
// entry and list entry between G neighbours, and evaluating branch-free
// lists, took a step's walk from 958 to 54 us on the 8,193-particle plasma,
// from 2,570 to 291 us at 60,001 particles (theta 0.4) and from 9.18 to
// 2.57 ms at 1,000,001.  The sums' error against a long double walk fell
// with it (RMS 7.0e-16 to 3.9e-16 on the 8,193-particle plasma).
//
// Stack: a round that pops t nodes leaves at most 7 t more than it found, so
// t is cut (down to 1, a depth-first descent, which needs at most 7 entries
// for each of the 21 levels) when the stack nears its capacity: no tree can
// overflow it.
constexpr int PW_WARPS = 4;  // warps per block
constexpr int PW_CAP = 640;
constexpr int PW_RESERVE = 7 * (MAX_LEVELS + 1);
// The list: its first 32 entries are evaluated before anything is appended to
// 32 or more, so an append (of a round's nodes or of 32 of a bucket's
// particles, at most one entry a lane) starts from 31 or fewer and ends with 63
// or fewer.
constexpr int PW_LIST = 64;
constexpr uint32_t PW_PART = 1u << 31;  // list word: a particle (softened); the low bits the targets' mask
template <int G, bool DIP> struct PwSmem {
	int2 stack[PW_CAP];       // node code, targets' mask
	double4 src[PW_LIST];     // the list: position and charge
	double4 dip[DIP ? PW_LIST : 1];
	uint32_t word[PW_LIST];
	double2 txy[G];           // the targets
	double tz[G];
	uint32_t self[G];
};

// The list's first 32 entries (unused ones have no bit set) against the lane's
// target, G entries a lane.
template <int G, bool PHI, bool DIP>
__device__ __forceinline__ void plain_eval(PlainAcc& E, uint32_t t, uint32_t sub, double x, double y, double z,
                                           const PwSmem<G, DIP>& sm, const Params& P, uint32_t& n_inter, int& rc)
{
#pragma unroll(G < 4 ? G : 4)
	for (int k = 0; k < G; k++) {
		const int i = k * (32 / G) + (int)sub;
		const uint32_t w = sm.word[i];
		const double4 c = sm.src[i];
		const bool on = ((w >> t) & 1u) != 0u, part = (w & PW_PART) != 0u;
		const double dx = x - c.x, dy = y - c.y, dz = z - c.z;
		double d2 = fma(dx, dx, fma(dy, dy, dz * dz));
		if (!PHI && on && part && d2 == 0.0) rc = POT_E_COINCIDENT;
		if (part) d2 += P.soft2;
		// only a cell's entry has a dipole; what lies in sm.dip of any other is
		// whatever was there before
		plain_term<PHI, DIP>(E, on, on && !part, sm.dip[DIP ? i : 0], c.w, dx, dy, dz, d2);
		n_inter += on ? 1u : 0u;
	}
}

// Evaluate the list's first 32 of n >= 32 entries; those beyond move to the
// front.
template <int G, bool PHI, bool DIP>
__device__ __forceinline__ void plain_flush(PlainAcc& E, int& n, uint32_t t, uint32_t sub, double x, double y, double z,
                                            PwSmem<G, DIP>& sm, const Params& P, uint32_t& n_inter, int& rc)
{
	const uint32_t lane = lane_id();
	plain_eval<G, PHI, DIP>(E, t, sub, x, y, z, sm, P, n_inter, rc);
	n -= 32;
	__syncwarp();
	if ((int)lane < n) {
		sm.src[lane] = sm.src[32 + lane];
		sm.word[lane] = sm.word[32 + lane];
		if (DIP) sm.dip[DIP ? lane : 0] = sm.dip[DIP ? 32 + lane : 0];
	}
	__syncwarp();
}

// Sums of the warp's nt <= G targets: lane l holds target l % G's point and
// slot (0xFFFFFFFF for none) and its share of the lists; the lanes l < G
// return the targets' sums.  n_inter counts the lane's terms; rc is set for a
// target at a particle's position, whose sum is zero.
template <int G, bool PHI, bool DIP>
__device__ PlainAcc plain_walk(uint32_t nt, double x, double y, double z, uint32_t me, const TreeDev& T,
                               const double4* __restrict__ src64, const Params& P, PwSmem<G, DIP>& sm,
                               uint32_t& n_inter, int& rc)
{
	const uint32_t lane = lane_id(), t = lane % G, sub = lane / G;
	const uint32_t lt = (1u << lane) - 1u;
	PlainAcc E { 0.0, 0.0, 0.0 };
	if (lane < G) {
		sm.txy[lane] = make_double2(x, y);
		sm.tz[lane] = z;
		sm.self[lane] = me;
	}
	sm.src[lane] = make_double4(0.0, 0.0, 0.0, 0.0);  // unused entries are evaluated too
	const double ke = QE / P.k4;
	int len = 0, n = 0;
	// the round's node: the root on lane 0
	int32_t code = lane == 0 ? 0 : CH_EMPTY;
	uint32_t mask = (1u << nt) - 1u;
	double4 c = make_double4(0.0, 0.0, 0.0, 0.0);
	double w2 = 0.0;
	if (code == 0) {
		c = ld_nc(&T.cq[0]);
		w2 = __ldg(&T.w2[0]);
	}
	__syncwarp();
	while (__any_sync(0xffffffffu, code != CH_EMPTY)) {
		const bool cell = code >= 0;
		const uint32_t e = leaf_payload(code);
		const bool over = code < CH_EMPTY && e >= P.n_tree;  // overflow bucket (see OVF_CAP)
		uint32_t acc = 0, opn = 0;
		if (cell) {
#pragma unroll
			for (int k = 0; k < G; k++) {
				const double2 q = sm.txy[k];
				const double d2 = dsq3(dsub(q.x, c.x), dsub(q.y, c.y), dsub(sm.tz[k], c.z));
				if (w2 < dmul(P.oap2, d2)) acc |= 1u << k;
			}
			opn = mask & ~acc;
			acc &= mask;
			if (DIP ? T.aq[code] == 0 : c.w == 0.0) acc = 0;
		} else if (code != CH_EMPTY && !over) {
			acc = mask;
#pragma unroll
			for (int k = 0; k < G; k++)
				if (sm.self[k] == e) acc &= ~(1u << k);
		}
		// the children of the opened nodes, appended with a warp scan
		int4 c0 = make_int4(CH_EMPTY, CH_EMPTY, CH_EMPTY, CH_EMPTY), c1 = c0;
		int nch = 0;
		if (opn) {
			const int4* cp = reinterpret_cast<const int4*>(&T.child[8u * (uint32_t)code]);
			c0 = __ldg(cp);
			c1 = __ldg(cp + 1);
			nch = (c0.x != CH_EMPTY) + (c0.y != CH_EMPTY) + (c0.z != CH_EMPTY) + (c0.w != CH_EMPTY) +
			      (c1.x != CH_EMPTY) + (c1.y != CH_EMPTY) + (c1.z != CH_EMPTY) + (c1.w != CH_EMPTY);
		}
		// the list
		const uint32_t am = __ballot_sync(0xffffffffu, acc != 0u);
		if (acc) {
			const int i = n + __popc(am & lt);
			sm.src[i] = make_double4(c.x, c.y, c.z, ke * c.w);
			sm.word[i] = acc | (cell ? 0u : PW_PART);
			if (DIP && cell) {
				const double4 d = T.dip[code];
				sm.dip[i] = make_double4(ke * d.x, ke * d.y, ke * d.z, 0.0);
			}
		}
		n += __popc(am);
		int incl = nch;
#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			const int v = __shfl_up_sync(0xffffffffu, incl, o);
			if ((int)lane >= o) incl += v;
		}
		int w = len + incl - nch;
		len += __shfl_sync(0xffffffffu, incl, 31);
		if (opn) {
			const int32_t cc[8] = { c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w };
#pragma unroll
			for (int d = 0; d < 8; d++)
				if (cc[d] != CH_EMPTY) sm.stack[w++] = make_int2(cc[d], (int)opn);
		}
		__syncwarp();
		uint32_t om = __ballot_sync(0xffffffffu, over);
		while (om) {  // every particle of an overflow bucket, 32 at a time
			const int b = __ffs(om) - 1;
			om &= om - 1u;
			const uint2 r = T.ovf[__shfl_sync(0xffffffffu, e, b) - P.n_tree];
			const uint32_t bm = __shfl_sync(0xffffffffu, mask, b);
			for (uint32_t j0 = r.x; j0 < r.x + r.y; j0 += 32) {
				// the nodes before it, or the 32 particles before these, may have left
				// up to 63 entries
				if (n >= 32) plain_flush<G, PHI, DIP>(E, n, t, sub, x, y, z, sm, P, n_inter, rc);
				const uint32_t j = j0 + lane;
				if (j < r.x + r.y) {
					uint32_t m = bm;
					for (int k = 0; k < G; k++)
						if (sm.self[k] == j) m &= ~(1u << k);
					const double4 p = src64[j];
					sm.src[n + (int)lane] = make_double4(p.x, p.y, p.z, ke * p.w);
					sm.word[n + (int)lane] = m | PW_PART;
				}
				n += (int)min(32u, r.x + r.y - j0);
				__syncwarp();
			}
		}
		// the next round's nodes, whose loads are in flight while the list is
		// evaluated
		int take = min(len, 32);
		if (len + 7 * take > PW_CAP - PW_RESERVE) take = max(1, min(take, (PW_CAP - PW_RESERVE - len) / 7));
		int2 next = make_int2(CH_EMPTY, 0);
		if ((int)lane < take) next = sm.stack[len - 1 - (int)lane];
		len -= take;
		double4 cn = c;
		if (next.x >= 0) {
			cn = ld_nc(&T.cq[next.x]);
			w2 = __ldg(&T.w2[next.x]);
		} else if (next.x != CH_EMPTY && leaf_payload(next.x) < P.n_tree) {
			cn = ld_nc(&src64[leaf_payload(next.x)]);
		}
		if (n >= 32) plain_flush<G, PHI, DIP>(E, n, t, sub, x, y, z, sm, P, n_inter, rc);
		__syncwarp();
		code = next.x;
		mask = (uint32_t)next.y;
		c = cn;
	}
	if (n > 0) {
		if ((int)lane >= n) sm.word[lane] = 0u;
		__syncwarp();
		plain_eval<G, PHI, DIP>(E, t, sub, x, y, z, sm, P, n_inter, rc);
		__syncwarp();
	}
#pragma unroll
	for (int o = G; o < 32; o <<= 1) {
		E.x += __shfl_xor_sync(0xffffffffu, E.x, o);
		if (!PHI) {
			E.y += __shfl_xor_sync(0xffffffffu, E.y, o);
			E.z += __shfl_xor_sync(0xffffffffu, E.z, o);
		}
	}
	if (!PHI) {  // a target at a particle's position has no field, whichever lane met it
		constexpr uint32_t LANES = G == 2 ? 0x55555555u : (G == 4 ? 0x11111111u : 0x01010101u);  // of target 0
		static_assert(G == 2 || G == 4 || G == 8, "targets per warp");
		if (__ballot_sync(0xffffffffu, rc != POT_OK) & (LANES << t)) {
			rc = POT_E_COINCIDENT;
			E = PlainAcc { 0.0, 0.0, 0.0 };
		}
	}
	return E;
}

// Deterministic block sum of three doubles (fixed shuffle and warp order).
__device__ void block_sum3(double v[3], double* __restrict__ out)
{
	__shared__ double part[32][3];
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
	for (int k = 0; k < 3; k++)
		for (int o = 16; o; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
	if (lane == 0)
		for (int k = 0; k < 3; k++) part[w][k] = v[k];
	__syncthreads();
	if (threadIdx.x == 0) {
		double t[3] = { 0.0, 0.0, 0.0 };
		for (int j = 0; j < (int)(blockDim.x >> 5); j++)
			for (int k = 0; k < 3; k++) t[k] += part[j][k];
		for (int k = 0; k < 3; k++) out[k] = t[k];
	}
}

// compute_epe of move_particles (pot.c:2771-2804), plain form: every
// particle's potential at its step-start position; per-block partial sums
// of q e phi per species (slots assigned to warps statically).
template <int G, bool DIP>
__global__ void __launch_bounds__(PW_WARPS * 32) k_epe_plain(const double4* __restrict__ pos, TreeDev T,
                                                             const double4* __restrict__ src64,
                                                             double* __restrict__ partial, Params P, RunRec* rec)
{
	__shared__ PwSmem<G, DIP> smem[PW_WARPS];
	PwSmem<G, DIP>& sm = smem[threadIdx.x >> 5];
	double acc[3] = { 0.0, 0.0, 0.0 };
	if (warp_status(rec) == POT_OK) {
		const uint32_t gs = rec->grain_slot;
		const uint32_t warps = gridDim.x * PW_WARPS;
		for (uint32_t b = blockIdx.x * PW_WARPS + (threadIdx.x >> 5); b * G < P.n; b += warps) {
			const uint32_t s = b * G + lane_id() % G, nt = min((uint32_t)G, P.n - b * G);
			const bool has = s < P.n;
			double4 p = make_double4(0.0, 0.0, 0.0, 0.0);
			if (has) p = src64[s];
			int rc = POT_OK;
			uint32_t ni = 0;
			const PlainAcc r = plain_walk<G, true, DIP>(nt, p.x, p.y, p.z, s, T, src64, P, sm, ni, rc);
			if (!has || lane_id() >= G) continue;
			double phi = r.x;
			if (s == gs) {
				rec->phi_grain = phi;
				continue;
			}
			if (P.shape) {  // pot-spheroid.c:2107-2109: the grain's own potential first
				phi = spheroid_phi(P, (double)rec->grain_q, dsub(p.x, rec->grain_pos[0]), dsub(p.y, rec->grain_pos[1]),
				                   dsub(p.z, rec->grain_pos[2])) + phi;
			}
			const int sp = (int)pos[s].w;
			acc[sp] += (QE * p.w) * phi;
		}
	}
	block_sum3(acc, &partial[3 * blockIdx.x]);
}

// Fixed-order sum of per-block (or per-group) partials into rec->epe.
__global__ void __launch_bounds__(1024) k_epe_final(const double* __restrict__ partial, const unsigned int* count,
                                                    uint32_t fixed, RunRec* rec)
{
	const uint32_t n = count ? count[0] + count[1] : fixed;
	double v[3] = { 0.0, 0.0, 0.0 };
	for (uint32_t i = threadIdx.x; i < n; i += blockDim.x)
		for (int k = 0; k < 3; k++) v[k] += partial[3 * i + k];
	__shared__ double out[3];
	block_sum3(v, out);
	__syncthreads();
	if (threadIdx.x == 0) {
		rec->epe[SP_ION] = out[SP_ION];
		rec->epe[SP_E] = out[SP_E];
	}
}

__device__ __forceinline__ void warp_add_u64(unsigned long long* dst, unsigned long long v)
{
#pragma unroll
	for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
	if (lane_id() == 0 && v) atomicAdd(dst, v);
}

// The walk fused with the push.  STG 0: Boris (half drift, field, kick,
// rotate, kick, half drift), then absorption and the boundary.  The
// non-Boris integrators take two launches: STG 1 evaluates the field at the
// old position and writes the intermediate state, its acceleration and its
// source entry (sb); STG 2 evaluates the field at the intermediate state over
// those sources (leaf particles moved, cells as built) and finishes the step
// (pot.c:2533-2639), then absorption and the boundary against the
// start-of-step position in src64.
// Each warp takes G targets (neighbours in Morton order) from the run's work
// counter, finds their fields (plain_walk) and pushes them.
template <int STG, int G, bool DIP>
__global__ void __launch_bounds__(PW_WARPS * 32) k_push_plain(double4* __restrict__ pos, double4* __restrict__ vel,
                                                              TreeDev T, const double4* __restrict__ src64,
                                                              const uint32_t* __restrict__ due_list,
                                                              uint32_t* __restrict__ rein_list, Params P, RunRec* rec,
                                                              StageBufs sb)
{
	__shared__ PwSmem<G, DIP> smem[PW_WARPS];
	PwSmem<G, DIP>& sm = smem[threadIdx.x >> 5];
	if (warp_status(rec) != POT_OK) return;
	const uint32_t n_due = rec->n_due;
	const unsigned long long t = rec->t_steps;
	const bool grain_due = rec->grain_due != 0;
	const bool absorb_on = !(P.flags & FLAG_NO_GRAIN) && t >= P.t_settle;
	double gx = rec->grain_pos[0], gy = rec->grain_pos[1], gz = rec->grain_pos[2];
	if (STG == 2 && grain_due && rec->grain_slot < P.n) {
		const double4 g = pos[rec->grain_slot];  // the grain's intermediate position
		gx = g.x; gy = g.y; gz = g.z;
	}
	const double qg = (double)rec->grain_q;
	const double4* __restrict__ src = STG == 2 ? sb.src64b : src64;
	unsigned long long n_inter = 0, n_push = 0;
	for (;;) {
		uint32_t base = 0;
		if (lane_id() == 0) base = atomicAdd(&rec->work_ctr, (uint32_t)G);
		base = __shfl_sync(0xffffffffu, base, 0);
		if (base >= n_due) break;
		const uint32_t i = base + lane_id() % G, nt = min((uint32_t)G, n_due - base);
		const bool has = i < n_due;
		uint32_t s = 0xFFFFFFFFu;
		double3 h = make_double3(0.0, 0.0, 0.0);
		if (has) {
			s = due_list[i];
			const double4 p = pos[s];
			h = make_double3(p.x, p.y, p.z);
			if (STG == 0) {
				const double4 v = vel[s];
				const double half = 0.5 * (P.dt * (double)P.tss[(int)p.w]);
				h = make_double3(fma(half, v.x, p.x), fma(half, v.y, p.y), fma(half, v.z, p.z));
			}
		}
		uint32_t ni = 0;
		int rc = POT_OK;
		const PlainAcc r = plain_walk<G, false, DIP>(nt, h.x, h.y, h.z, s, T, src, P, sm, ni, rc);
		if (rc != POT_OK) set_status(rec, rc);
		n_inter += ni;
		if (!has || lane_id() >= G) continue;
		const double4 p = pos[s];
		double4 v = vel[s];
		const int sp = (int)p.w;
		const double dt = P.dt * (double)P.tss[sp];
		double E[3] = { r.x, r.y, r.z };
		if (P.shape && sp != SP_DUST && rc == POT_OK) {
			// a spheroidal grain's own field first (pot-spheroid.c:1815-1819)
			spheroid_field(P, qg, dsub(h.x, gx), dsub(h.y, gy), dsub(h.z, gz), E);
			E[0] += r.x;
			E[1] += r.y;
			E[2] += r.z;
		}
		const double charge = sp == SP_DUST ? qg : (sp == SP_ION ? 1.0 : -1.0);
		const double qom = (QE * charge) / mass_of(sp, P);
		if (STG == 1) {
			const double3 a1 = accel_lorentz(E, v, qom, P);
			double4 pm = p;
			half_first(pm, v, a1, dt, P);
			pos[s] = pm;
			vel[s] = v;
			sb.acc[s] = make_double4(a1.x, a1.y, a1.z, 0.0);
			sb.src64b[s] = make_double4(pm.x, pm.y, pm.z, src64[s].w);
			continue;
		}
		n_push++;
		double3 xn;
		if (STG == 0) {
			boris(v, h, E, qom, dt, P, xn);
		} else {
			const double4 a = sb.acc[s];
			half_second(xn, v, p, make_double3(a.x, a.y, a.z), accel_lorentz(E, v, qom, P), dt, P);
		}
		uint32_t reason = 0;
		if (!grain_due) reason = after_push(sp, STG == 0 ? p : src64[s], xn, v, P, rec, absorb_on, gx, gy, gz);
		pos[s] = make_double4(xn.x, xn.y, xn.z, p.w);
		vel[s] = v;
		if (reason) rein_list[atomicAdd(&rec->n_rein, 1u)] = s | (reason << 30);
	}
	warp_add_u64(&rec->interactions, n_inter);
	warp_add_u64(&rec->n_pushed, n_push);
}

// ---------------------------------------------------------------------------
// potential: warp-cooperative phi_at (pot.c:1818-1901)
// ---------------------------------------------------------------------------
constexpr int PHI_STACK = 2048;

// One warp evaluates the potential at (x, y, z); `stack` is this warp's
// shared-memory stack.  Nodes are processed 32 at a time; children of opened
// cells are pushed with a warp prefix sum.  Returns NaN on stack overflow.
__device__ double warp_phi(double x, double y, double z, const TreeDev& T, const double4* __restrict__ src64,
                           const Params& P, int32_t* stack)
{
	const uint32_t lane = lane_id();
	int len = 1;
	if (lane == 0) stack[0] = 0;
	__syncwarp();
	double acc = 0.0;
	bool overflow = false;
	while (len > 0) {
		const int take = len < 32 ? len : 32;
		const int32_t code = (int)lane < take ? stack[len - 1 - (int)lane] : CH_EMPTY;
		__syncwarp();
		len -= take;
		int32_t ch[8];
		int nch = 0;
		if (code >= 0) {
			const double4 c = T.cq[code];
			const double dx = dsub(x, c.x), dy = dsub(y, c.y), dz = dsub(z, c.z);
			const double dist2 = dsq3(dx, dy, dz);
			if (T.w2[code] < dmul(P.oap2, dist2)) {
				if (T.dip) {
					if (T.aq[code] != 0) {  // DIPOLES, pot.c:1860-1868
						const double dist = sqrt(dist2);
						const double4 pd = T.dip[code];
						const double rp = dadd(dadd(dmul(dx, pd.x), dmul(dy, pd.y)), dmul(dz, pd.z));
						acc += dmul(ddiv(QE, P.k4), dadd(ddiv(c.w, dist), ddiv(rp, dmul(dist, dist2))));
					}
				} else if (c.w != 0.0) {
					acc += ddiv(dmul(QE, c.w), dmul(P.k4, sqrt(dist2)));
				}
			} else {
				const int32_t* cp = &T.child[8u * (uint32_t)code];
#pragma unroll
				for (int s = 0; s < 8; s++) {
					const int32_t cc = cp[slot_digit(s)];
					if (cc != CH_EMPTY) ch[nch++] = cc;
				}
			}
		} else if (code != CH_EMPTY) {
			const uint32_t e = leaf_payload(code);
			uint32_t j0 = e, j1 = e + 1;
			if (P.leaf_size > 1 || e >= P.n_tree) {
				const uint2 r = P.leaf_size > 1 ? T.lrange[e] : T.ovf[e - P.n_tree];
				j0 = r.x;
				j1 = r.x + r.y;
			}
			for (uint32_t j = j0; j < j1; j++) {
				const double4 p = src64[j];
				const double d2 = dsq3(dsub(x, p.x), dsub(y, p.y), dsub(z, p.z));
				acc += ddiv(dmul(QE, p.w), dmul(P.k4, sqrt(dadd(d2, P.soft2))));
			}
		}
		int incl = nch;
#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			const int tv = __shfl_up_sync(0xffffffffu, incl, o);
			if ((int)lane >= o) incl += tv;
		}
		const int total = __shfl_sync(0xffffffffu, incl, 31);
		if (len + total > PHI_STACK) {
			overflow = true;
			break;
		}
		const int off = len + incl - nch;
		for (int j = 0; j < nch; j++) stack[off + j] = ch[j];
		__syncwarp();
		len += total;
	}
#pragma unroll
	for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
	return overflow ? __longlong_as_double(0x7ff8000000000000ll) : acc;
}

// The spheroid's term of phi_at (pot-spheroid.c:1924-1953), which the
// reference evaluates at the point's own coordinates rather than relative
// to the grain; reproduced as written.  Zero for a spherical grain, whose
// charge is a tree source.
__device__ __forceinline__ double spheroid_phi_at(const Params& P, const RunRec* rec, double x, double y, double z)
{
	if (!P.shape) return 0.0;
	double u, v, w;
	sph_to_frame(P, x, y, z, u, v, w);
	return spheroid_phi_frame(P, (double)rec->grain_q, u, v, w);
}

// measure_chi_b (pot.c:2251-2279) as a run of P = chi_ranks MPI ranks does
// it (pot.c:2409-2418): rank k samples phi at azimuth 2 pi k / P in the x-y
// plane through the grain, the samples are summed and divided by P; every 20
// steps.  Four warps share the samples; the sum is taken in rank order.
template <class G>
__device__ __forceinline__ void chi_b_body(G grd, const TreeDev& T, const double4* __restrict__ src64,
                                           const Params& P, RunRec* rec, int force)
{
	__shared__ int32_t stack[4][PHI_STACK];
	__shared__ double sample[64];
	__shared__ int bad;
	if (!(P.flags & FLAG_SCEPTIC)) return;
	if (!force && (rec->t_steps % 20) != 0) return;
	if (block_status(rec) != POT_OK) return;
	const uint32_t w = threadIdx.x >> 5;
	if (threadIdx.x == 0) bad = 0;
	__syncthreads();
	const double zen = PI_REF / 2.0;
	const double r = P.rad;
	for (uint32_t k = w; k < P.chi_ranks; k += 4) {
		const double azi = 2.0 * PI_REF * k / P.chi_ranks;
		const double x = rec->grain_pos[0] + (r * cos(azi) * sin(zen));
		const double y = rec->grain_pos[1] + (r * sin(azi) * sin(zen));
		const double z = rec->grain_pos[2] + (r * cos(zen));
		const double phi = spheroid_phi_at(P, rec, x, y, z) + warp_phi(x, y, z, T, src64, P, stack[w]);
		if (lane_id() == 0) {
			sample[k] = phi / (KB * P.Ti / (1 * QE));
			if (isnan(phi)) bad = 1;
		}
	}
	__syncthreads();
	if (threadIdx.x == 0) {
		if (bad) {
			rec->chi_failed = 1;  // the step ends with POT_E_WALK (finish_step_body)
		} else {
			double sum = 0.0;
			for (uint32_t k = 0; k < P.chi_ranks; k++) sum += sample[k];
			rec->chi_b = sum / P.chi_ranks;
		}
	}
}

__global__ void __launch_bounds__(128) k_chi_b(TreeDev T, const double4* __restrict__ src64, Params P, RunRec* rec,
                                               int force)
{
	chi_b_body(GridSelf {}, T, src64, P, rec, force);
}

__global__ void k_phi_query(TreeDev T, const double4* __restrict__ src64, const double* __restrict__ xyz,
                            uint32_t nq, double* __restrict__ phi, Params P, RunRec* rec)
{
	__shared__ int32_t stack[4][PHI_STACK];
	const uint32_t w = threadIdx.x >> 5;
	for (uint32_t q = blockIdx.x * 4 + w; q < nq; q += gridDim.x * 4) {
		const double v = spheroid_phi_at(P, rec, xyz[3 * q], xyz[3 * q + 1], xyz[3 * q + 2]) +
		                 warp_phi(xyz[3 * q], xyz[3 * q + 1], xyz[3 * q + 2], T, src64, P, stack[w]);
		if (lane_id() == 0) {
			phi[q] = v;
			if (isnan(v)) set_status(rec, POT_E_WALK);
		}
	}
}

template <int G, bool DIP>
__global__ void __launch_bounds__(PW_WARPS * 32) k_field_query_plain(TreeDev T, const double4* __restrict__ src64,
                                                                     const double* __restrict__ xyz,
                                                                     const uint32_t* __restrict__ self_slot,
                                                                     uint32_t nq, double* __restrict__ E, Params P,
                                                                     RunRec* rec)
{
	__shared__ PwSmem<G, DIP> smem[PW_WARPS];
	PwSmem<G, DIP>& sm = smem[threadIdx.x >> 5];
	const uint32_t base = (blockIdx.x * PW_WARPS + (threadIdx.x >> 5)) * G;
	if (base >= nq) return;
	const uint32_t q = base + lane_id() % G, nt = min((uint32_t)G, nq - base);
	const bool has = q < nq;
	double3 h = make_double3(0.0, 0.0, 0.0);
	uint32_t self = 0xFFFFFFFFu;
	if (has) {
		h = make_double3(xyz[3 * (size_t)q], xyz[3 * (size_t)q + 1], xyz[3 * (size_t)q + 2]);
		self = self_slot[q];
	}
	uint32_t ni = 0;
	int rc = POT_OK;
	const PlainAcc r = plain_walk<G, false, DIP>(nt, h.x, h.y, h.z, self, T, src64, P, sm, ni, rc);
	if (rc != POT_OK) set_status(rec, rc);
	if (!has || lane_id() >= G) return;
	double e[3] = { 0.0, 0.0, 0.0 };
	if (P.shape && self != rec->grain_slot && rc == POT_OK) {
		spheroid_field(P, (double)rec->grain_q, dsub(h.x, rec->grain_pos[0]), dsub(h.y, rec->grain_pos[1]),
		               dsub(h.z, rec->grain_pos[2]), e);
	}
	E[3 * (size_t)q] = e[0] + r.x;
	E[3 * (size_t)q + 1] = e[1] + r.y;
	E[3 * (size_t)q + 2] = e[2] + r.z;
}

// ---------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------
void launch_push_fast(double4* pos, double4* vel, const TreeDev& T, const float4* src32, const double4* src64,
                      const uint32_t* due_list, const uint2* groups, uint32_t* rein_list, const Params& P,
                      RunRec* rec, const StageBufs& sb, cudaStream_t s, Timer& tm);
void launch_epe_fast(const double4* pos, const TreeDev& T, const float4* src32, const double4* src64,
                     uint2* groups_all, double* partial, const Params& P, RunRec* rec, cudaStream_t s, Timer& tm);
void launch_field_query_fast(const TreeDev& T, const float4* src32, const double* xyz, const uint32_t* self_slot,
                             uint32_t nq, double* E, const Params& P, RunRec* rec, cudaStream_t s, Timer& tm);

static int sm_count()
{
	static int n = 0;
	if (!n) {
		int dev = 0;
		cudaGetDevice(&dev);
		cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
		if (n <= 0) n = 148;
	}
	return n;
}

// Targets per warp of the plain walk for n targets.  More targets share each
// node's load, test round and stack entry, fewer make more warps: with 4,096
// targets (8,193 particles) the walk takes 55, 63, 88 and 138 us with 2, 4, 8
// and 16 targets a warp, with 15,000 132, 115, 129 and 209, with 30,000 399,
// 294, 288 and 380, with 500,000 4,990, 3,248, 2,647 and 2,570.  With dipoles
// (the reference's off-by-default variant) one size is compiled, the one for
// many targets: 2, 4 and 8 targets take 71, 88 and 126 us with 4,096, 203, 171
// and 180 with 15,000, 401, 303 and 296 with 30,000, 8,320, 5,450 and 4,363 with
// 500,000.
static int plain_group(uint32_t n) { return n < 8192u ? 2 : (n < 32768u ? 4 : 8); }

template <int STG, int G, bool DIP>
static void push_plain(double4* pos, double4* vel, const TreeDev& T, const double4* src64, const uint32_t* due_list,
                       uint32_t* rein_list, const Params& P, RunRec* rec, const StageBufs& sb, cudaStream_t s)
{
	static const int per = [] {  // set once, also by threads that step their first runs together
		int n = 0;
		cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_push_plain<STG, G, DIP>, PW_WARPS * 32, 0);
		return n > 0 ? n : 1;
	}();
	k_push_plain<STG, G, DIP><<<sm_count() * per, PW_WARPS * 32, 0, s>>>(pos, vel, T, src64, due_list, rein_list, P,
	                                                                    rec, sb);
}

template <int STG>
static void push_plain_stage(double4* pos, double4* vel, const TreeDev& T, const double4* src64,
                             const uint32_t* due_list, uint32_t* rein_list, const Params& P, RunRec* rec,
                             const StageBufs& sb, cudaStream_t s)
{
	const int G = plain_group(P.n / 2);  // at least the electrons are due
	if (T.dip) push_plain<STG, 8, true>(pos, vel, T, src64, due_list, rein_list, P, rec, sb, s);
	else if (G == 4) push_plain<STG, 4, false>(pos, vel, T, src64, due_list, rein_list, P, rec, sb, s);
	else if (G == 2) push_plain<STG, 2, false>(pos, vel, T, src64, due_list, rein_list, P, rec, sb, s);
	else push_plain<STG, 8, false>(pos, vel, T, src64, due_list, rein_list, P, rec, sb, s);
}

void launch_chi_b(const TreeDev& T, const double4* src64, const Params& P, RunRec* rec, int force,
                  cudaStream_t s, Timer& tm)
{
	if (!(P.flags & FLAG_SCEPTIC)) return;
	ScopedKernel k(tm, "chi_b");
	k_chi_b<<<1, 128, 0, s>>>(T, src64, P, rec, force);
}

void launch_push(double4* pos, double4* vel, const TreeDev& T, const double4* src64, const float4* src32,
                 const uint32_t* due_list, const uint2* groups, uint32_t* rein_list, const Params& P, RunRec* rec,
                 const StageBufs& sb, cudaStream_t s, Timer& tm)
{
	if (P.form == POT_FORM_FAST) {
		launch_push_fast(pos, vel, T, src32, src64, due_list, groups, rein_list, P, rec, sb, s, tm);
		return;
	}
	ScopedKernel k(tm, sb.stage == 0 ? "walk_push_plain" : (sb.stage == 1 ? "walk_half1_plain" : "walk_half2_plain"));
	if (sb.stage == 0) push_plain_stage<0>(pos, vel, T, src64, due_list, rein_list, P, rec, sb, s);
	else if (sb.stage == 1) push_plain_stage<1>(pos, vel, T, src64, due_list, rein_list, P, rec, sb, s);
	else push_plain_stage<2>(pos, vel, T, src64, due_list, rein_list, P, rec, sb, s);
}

void launch_epe(const double4* pos, const TreeDev& T, const double4* src64, const float4* src32, uint2* groups_all,
                double* partial, const Params& P, RunRec* rec, cudaStream_t s, Timer& tm)
{
	if (P.form == POT_FORM_FAST) {
		launch_epe_fast(pos, T, src32, src64, groups_all, partial, P, rec, s, tm);
		ScopedKernel k(tm, "epe_final");
		k_epe_final<<<1, 1024, 0, s>>>(partial, rec->n_groups_all, 0, rec);
		return;
	}
	ScopedKernel k(tm, "epe_plain", 2);
	const int G = plain_group(P.n), th = PW_WARPS * 32;
	if (T.dip) k_epe_plain<8, true><<<EPE_BLOCKS, th, 0, s>>>(pos, T, src64, partial, P, rec);
	else if (G == 2) k_epe_plain<2, false><<<EPE_BLOCKS, th, 0, s>>>(pos, T, src64, partial, P, rec);
	else if (G == 4) k_epe_plain<4, false><<<EPE_BLOCKS, th, 0, s>>>(pos, T, src64, partial, P, rec);
	else k_epe_plain<8, false><<<EPE_BLOCKS, th, 0, s>>>(pos, T, src64, partial, P, rec);
	k_epe_final<<<1, 1024, 0, s>>>(partial, nullptr, EPE_BLOCKS, rec);
}

void launch_field_query(const TreeDev& T, const double4* src64, const float4* src32, const double* xyz,
                        const uint32_t* self_slot, uint32_t nq, double* E, const Params& P, RunRec* rec,
                        cudaStream_t s, Timer& tm)
{
	if (P.form == POT_FORM_FAST) {
		launch_field_query_fast(T, src32, xyz, self_slot, nq, E, P, rec, s, tm);
		return;
	}
	ScopedKernel k(tm, "field_query");
	const int G = T.dip ? 8 : plain_group(nq);
	const uint32_t per = PW_WARPS * (uint32_t)G, nb = (nq + per - 1) / per;
	const int th = PW_WARPS * 32;
	if (T.dip) k_field_query_plain<8, true><<<nb, th, 0, s>>>(T, src64, xyz, self_slot, nq, E, P, rec);
	else if (G == 2) k_field_query_plain<2, false><<<nb, th, 0, s>>>(T, src64, xyz, self_slot, nq, E, P, rec);
	else if (G == 4) k_field_query_plain<4, false><<<nb, th, 0, s>>>(T, src64, xyz, self_slot, nq, E, P, rec);
	else k_field_query_plain<8, false><<<nb, th, 0, s>>>(T, src64, xyz, self_slot, nq, E, P, rec);
}

void launch_phi_query(const TreeDev& T, const double4* src64, const double* xyz, uint32_t nq, double* phi,
                      const Params& P, RunRec* rec, cudaStream_t s, Timer& tm)
{
	ScopedKernel k(tm, "phi_query");
	const uint32_t nb = (nq + 3) / 4;
	k_phi_query<<<nb < 4096 ? nb : 4096, 128, 0, s>>>(T, src64, xyz, nq, phi, P, rec);
}

}  // namespace pot

// ---------------------------------------------------------------------------
// packed batch: chi_b of every member
// ---------------------------------------------------------------------------
namespace pot {

__global__ void __launch_bounds__(128) kp_chi_b(PackDev B)
{
	const SegBlock sb = seg_block(B.pre[PS_ONE], B.M);
	const MemberView& v = B.mv[sb.m];
	chi_b_body(GridSeg { sb.id, sb.n }, v.T, v.src64, v.P, v.rec, 0);
}

void pack_chi_b(const PackDev& B, cudaStream_t s)
{
	kp_chi_b<<<B.blocks[PS_ONE], 128, 0, s>>>(B);
}

}  // namespace pot
