// Tree storage and launchers shared by the tree and walk translation units.
#pragma once

#include "pot_host.h"

namespace pot {

// A tree node as the FP32 walk reads it, in units of the domain radius from
// the domain centre.  A cell: centre of charge and charge, critical radius
// squared (accepted when d^2 > r2), the index of its first child's record and
// how many children it has.  A leaf: the same moments, its first slot and, with
// NR_LEAF, its particle count; a leaf of a leaf-size-1 tree has no moments
// (NR_UNTESTED: always opened).
constexpr uint32_t NR_LEAF = 1u << 31, NR_UNTESTED = 1u << 30, NR_COUNT = NR_UNTESTED - 1u;
struct __align__(32) NodeRec {
	float x, y, z, q;
	float r2;
	uint32_t base;
	uint32_t info;
	uint32_t pad;
};

// Internal nodes in pre-order, structure of arrays; `cap` entries each
// (the leaf table of bucket leaves has 8 * cap entries).
struct TreeDev {
	uint32_t cap;
	int8_t* lvl8;      // [n] common levels of pair (i, i + L), capped at 20
	uint32_t* base;    // [n] index of pair i's first cell (prefix of the cells owned)
	uint32_t* first;   // first particle (Morton slot)
	uint32_t* last;    // last particle
	uint8_t* level;    // depth (root 0)
	int32_t* child;    // [8 * cap] child codes by octal digit
	int32_t* parent;   // the parent cell, -1 for the root; fast form: the cell's own record
	uint8_t* nint;     // internal children
	uint32_t* ctr;     // arrivals in the upward pass; fast form: the first child's record
	int32_t* q;        // net charge (Tree.q)
	uint32_t* aq;      // absolute charge (Tree.aq)
	double4* cq;       // centre of |q| and q
	double* w2;        // (x2 - x1)^2
	double4* dip;      // DIPOLES: dipole moment about cq (FP64, both forms); null otherwise
	// FP32 walk (fast form only; null otherwise): one 32-byte record per node, so
	// that a walk reads everything it needs of a node with one load.  The root's
	// is record 0; a cell's children have consecutive records in digit order
	// (k_finish_nodes gives them out), at most `cap` of cells and n of leaves.
	NodeRec* nrec;     // [spare + 1]
	uint32_t spare;    // a record no node has
	uint2* lrange;     // [8 * cap] bucket-leaf (first slot, count)
	uint2* ovf;        // [OVF_CAP] leaf-size-1 overflow buckets (first slot, count)
	// fast form: exclusive prefix sums of (q, |q|, |q| x, |q| y, |q| z), 5 doubles each
	double* mom_pre;   // [n + 1]
	double* mom_blk;   // [blocks + 1]
	// fast form with DIPOLES: prefix sums of (q x, q y, q z) in the same layout,
	// and the nodes' dipoles in FP32 units of q R
	double* mom_pre_d;
	double* mom_blk_d;
	float4* drec;      // [spare + 1], indexed as nrec
};

// One member run of a packed batch as the batched kernels see it: the
// run's parameters, tree, record and device arrays (those of its context).
// Buffer parity: at step k of a graph launch a member's state is in
// pos[cur ^ (k & 1)]; kb is the key buffer holding the sorted keys (the
// number of radix passes is the same for every member of a batch).
struct MemberView {
	Params P;
	TreeDev T;
	RunRec* rec;
	StepHist* hist;
	double4* pos[2];
	double4* vel[2];
	uint32_t* pid[2];
	double4* src64;
	float4* src32;
	uint64_t* keys[2];
	uint32_t* vals[2];
	uint32_t* words;       // the step's cleared words (StepWords)
	uint8_t* due;
	uint32_t* due_list;
	uint32_t* due_prefix;
	uint2* groups;
	uint32_t* rein_list;
	uint32_t cur;
	uint32_t kb;
};

// A packed batch's step: each kernel of the step is one launch over every
// member (pot_batch.cu builds this).  pre[stage] is the exclusive prefix of
// the members' block counts for that stage's kernels (device, M + 1
// entries), blocks[stage] its total.  Stages:
//   PS_KEYS    keys_blocks(n): keys and the sort's digit counts
//   PS_N256    blocks_for(n, 256): reorder
//   PS_DUE     due_tiles(n): due list
//   PS_TILES   the sort's tiles: clearing the step's words, each pass
//   PS_CELLS   cell_tiles(n_tree - L): cell numbering
//   PS_FINISH  blocks_for(n_tree, 256)
//   PS_MOM     moment tiles over n_tree: prefix sums
//   PS_MOMPRE  mom_cell_blocks(n_tree, leaf size): cell moments from the sums
//   PS_GROUPS  target groups
//   PS_ONE     one block per member: chi_b
//   PS_SMALL   4-148 blocks per member (one per 8,192 particles): the step's
//              end (one warp per reinjected particle)
enum PackStage : int {
	PS_KEYS, PS_N256, PS_DUE, PS_TILES, PS_CELLS, PS_FINISH, PS_MOM, PS_MOMPRE, PS_GROUPS, PS_ONE, PS_SMALL, PS_COUNT
};
struct PackDev {
	const MemberView* mv;           // [M], device
	uint32_t M;
	uint32_t npass;                 // radix passes, the same for every member
	const uint32_t* pre[PS_COUNT];
	uint32_t blocks[PS_COUNT];
	uint32_t* gpre;                 // [2 M + 1] prefix of the members' target groups this step (device)
	unsigned int* ctr;              // the batch walk's work counter (device)
};
// The member's state at step k of a graph launch is in buffer cur ^ (k & 1)
// until the reorder, which writes the other buffer.
__device__ __forceinline__ uint32_t pack_in(const MemberView& v, int k) { return v.cur ^ (uint32_t)(k & 1); }
__device__ __forceinline__ uint32_t pack_out(const MemberView& v, int k) { return v.cur ^ (uint32_t)(k & 1) ^ 1u; }

// the packed step's launches, in stream order (tree.cu, sort.cu, walk.cu,
// walk_fast.cu, inject.cu)
void pack_sort_begin(const PackDev& B, cudaStream_t s);
void pack_keys(const PackDev& B, int k, cudaStream_t s);
void pack_sort(const PackDev& B, cudaStream_t s);
void pack_reorder(const PackDev& B, int k, cudaStream_t s);
void pack_due_list(const PackDev& B, cudaStream_t s);
void pack_cells(const PackDev& B, int k, cudaStream_t s);
void pack_mom_sums(const PackDev& B, cudaStream_t s);
void pack_moments(const PackDev& B, cudaStream_t s);
void pack_groups(const PackDev& B, cudaStream_t s);
void pack_chi_b(const PackDev& B, cudaStream_t s);
void pack_push(const PackDev& B, int k, uint32_t tpl, cudaStream_t s);
void pack_finish_step(const PackDev& B, int k, cudaStream_t s);
constexpr uint32_t PACK_MOM_TILE = 256 * 16;  // moment prefix-sum tile (tree.cu MOM_TILE)

uint32_t mom_cell_blocks(size_t n, uint32_t leaf);
size_t mom_prefix_entries(size_t n);
size_t mom_block_entries(size_t n);
void launch_keys(const double4* pos, uint64_t* keys, uint32_t* vals, const Params& P, RunRec* rec,
                 int begin_step, uint32_t* words, cudaStream_t s, Timer& tm);
uint32_t keys_blocks(size_t n);
void launch_reorder(const uint32_t* perm, const double4* pos_in, const double4* vel_in, const uint32_t* pid_in,
                    double4* pos_out, double4* vel_out, uint32_t* pid_out, double4* src64, float4* src32,
                    uint8_t* due, uint32_t* words, const Params& P, RunRec* rec, cudaStream_t s, Timer& tm);
void launch_due_list(const uint8_t* due, uint32_t* words, uint32_t* due_list, uint32_t* due_prefix, const Params& P,
                     RunRec* rec, cudaStream_t s, Timer& tm);
void launch_cells(const uint64_t* keys, const uint32_t* perm, const double4* pos_in, TreeDev& T, const Params& P,
                  RunRec* rec, uint32_t* words, cudaStream_t s, Timer& tm);
void launch_mom_sums(TreeDev& T, const double4* src64, const Params& P, cudaStream_t s, Timer& tm);
void launch_moments(TreeDev& T, const double4* src64, const Params& P, RunRec* rec, cudaStream_t s, Timer& tm);

// ---- branches of a step --------------------------------------------------
// A captured step runs on three streams: while the main one reorders the
// state and sums its moments, the second builds the tree's topology from the
// sorted keys (and later measures chi_b beside the walk) and the third lists
// the due particles and makes the target groups.  Without side streams the
// same launches follow each other on the main one.
struct StepStreams {
	cudaStream_t main = nullptr, side[2] = { nullptr, nullptr };
	cudaEvent_t ev[6] = {};
	bool forked = false;
	cudaStream_t tree() const { return forked ? side[0] : main; }
	cudaStream_t list() const { return forked ? side[1] : main; }
	// what `to` enqueues next waits for what `from` holds now
	void order(int e, cudaStream_t from, cudaStream_t to) const
	{
		if (from == to) return;
		cudaEventRecord(ev[e], from);
		cudaStreamWaitEvent(to, ev[e], 0);
	}
	bool create()  // side streams and events, once
	{
		if (side[0]) return true;
		for (auto& e : ev)
			if (!e && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) return false;
		if (!side[1] && cudaStreamCreateWithFlags(&side[1], cudaStreamNonBlocking) != cudaSuccess) return false;
		return cudaStreamCreateWithFlags(&side[0], cudaStreamNonBlocking) == cudaSuccess;
	}
	void destroy()
	{
		for (auto& e : ev)
			if (e) cudaEventDestroy(e);
		for (auto& s : side)
			if (s) cudaStreamDestroy(s);
		*this = StepStreams();
	}
};

// walk.cu
size_t macro_scratch_doubles();
void launch_macro(const double4* pos, const double4* vel, const Params& P, double* scratch, RunRec* rec,
                  cudaStream_t s, Timer& tm);
void launch_chi_b(const TreeDev& T, const double4* src64, const Params& P, RunRec* rec, int force,
                  cudaStream_t s, Timer& tm);
// Buffers of the non-Boris integrators' two-launch step: stage 0 is the
// one-launch Boris step; stage 1 writes each due particle's first-half
// acceleration (acc) and its intermediate source entry (src64b, and src32b in
// the fast form); stage 2 reads them.
struct StageBufs {
	int stage;
	double4* acc;
	double4* src64b;
	float4* src32b;
};
void launch_push(double4* pos, double4* vel, const TreeDev& T, const double4* src64, const float4* src32,
                 const uint32_t* due_list, const uint2* groups, uint32_t* rein_list, const Params& P, RunRec* rec,
                 const StageBufs& sb, cudaStream_t s, Timer& tm);
// Target groups of at most P.group_max due particles, each inside one tree
// cell.  With gcell (a byte per tree cell) and gblk (group_blocks() + 1
// words) the groups are laid out in tree pre-order, so that the walk's
// concurrent warps work on neighbouring groups; with gcell == nullptr they
// are built by one launch, in the order their cells finish.
uint32_t group_blocks();
void launch_groups(const TreeDev& T, const uint32_t* dpre, uint2* groups, uint8_t* gcell, uint32_t* gblk,
                   const Params& P, RunRec* rec, cudaStream_t s, Timer& tm);
void launch_epe(const double4* pos, const TreeDev& T, const double4* src64, const float4* src32, uint2* groups_all,
                double* partial, const Params& P, RunRec* rec, cudaStream_t s, Timer& tm);
void launch_field_query(const TreeDev& T, const double4* src64, const float4* src32, const double* xyz,
                        const uint32_t* self_slot, uint32_t nq, double* E, const Params& P, RunRec* rec,
                        cudaStream_t s, Timer& tm);
void launch_phi_query(const TreeDev& T, const double4* src64, const double* xyz, uint32_t nq, double* phi,
                      const Params& P, RunRec* rec, cudaStream_t s, Timer& tm);

// inject.cu
// The state a step started from: slot s of its order was perm[s] of pos and vel.
struct StepStart {
	const uint32_t* perm;
	const double4* pos;
	const double4* vel;
};
void launch_finish_step(double4* pos, double4* vel, const uint32_t* pid, const uint32_t* due_list, uint32_t* rein_list,
                        const double4* src64, StepHist* hist, const StepStart& from, const Params& P, RunRec* rec,
                        int epe, cudaStream_t s, Timer& tm);
void launch_init(double4* pos, double4* vel, uint32_t* pid, const Params& P, RunRec* rec, cudaStream_t s,
                 Timer& tm);

}  // namespace pot
