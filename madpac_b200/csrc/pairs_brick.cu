// Single-box pair kernels: one CTA per brick of 2x2x2 linked cells (the per-brick work is in
// brick.cuh, which also documents the staging, filter and compute passes).
//
//   k_pairs_brick  filter + exact evaluation every call (the drop-in traversal)
//   k_build_lists  Verlet-skin mode, build step: each molecule's candidates within rc + skin
//   k_pairs_list   Verlet-skin mode, every step: exact evaluation of the lists at the current
//                  positions
// In the Verlet-skin mode the build is launched every step and returns at once unless a device flag
// (set by the Leapfrog pre-kick when a molecule moved more than skin/2 since the build) is set.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>
#include <utility>

#include "brick.cuh"
#include "md_internal.h"

namespace mdgpu {
namespace {

// Resident CTAs per SM of the traversal (registers and the usual shared memory are sized for it). 250,047
// molecules at rc = 2.5, us per traversal: three, with 80 registers, 125; two, with 128, 146; four, with 64, 137.
// At rc = 3.0, where the regions leave room for two in each case: 187, 179 and 226.
constexpr int kTraverseMinBlocks = 3;

template <bool kSingle, bool kLjIsRc>
__global__ void __launch_bounds__(brick::kThreads, kTraverseMinBlocks)
    k_pairs_brick(const __grid_constant__ brick::Const p, const __grid_constant__ brick::Box bx,
                  const double* __restrict__ rx, const double* __restrict__ ry,
                  const double* __restrict__ rz, const int32_t* __restrict__ cid,
                  const int32_t* __restrict__ cstart, const PairParams* __restrict__ pp,
                  double* __restrict__ fx, double* __restrict__ fy, double* __restrict__ fz,
                  double* __restrict__ partials, int* __restrict__ status,
                  brick::Lists lists, unsigned* ticket, double* scalars) {
	extern __shared__ __align__(16) unsigned char smem[];
	__shared__ int s_item;
	brick::load_params(smem, brick::layout(p.s_cap, true, brick::kHitWords), pp, p.ns);
	// every brick, one CTA each, or (lists.counts) those that k_pairs_sparse left: a resident grid takes
	// them from a queue
	const bool queue = lists.counts != nullptr;
	const int nwork = queue ? (int) *(volatile unsigned*) lists.counts : 0;
	int b = (int) blockIdx.x;
	do {
		if (queue) {
			__syncthreads();
			if (threadIdx.x == 0) s_item = (int) atomicAdd(lists.counts + 1, 1u);
			__syncthreads();
			if (s_item >= nwork) break;
			b = lists.blist[s_item];
		}
		brick::pairs<kSingle, kLjIsRc, brick::kHitWords>(p, bx, b, b, smem, rx, ry, rz, cid, cstart, fx, fy, fz,
		                                                 partials, status);
	} while (queue);
	// U6 sum, virial sum and pair count over every brick, by the last CTA (ticket null: by a later launch)
	if (ticket) last_block_sum(ticket, partials, gridDim.x, 3, scalars);
}

// The sparse bricks of a traversal (vapour: a few molecules), one warp each; the others go to counts[0],
// blist. A CTA of the dense kernel spends 9000 cycles on such a brick, most of them waiting for its
// staging's loads; here as many bricks as warps fit wait at once. Measured, us per traversal: the 786,432-
// molecule slab 532 -> 394 (its sparse bricks 26), a vapour of 100,000 at density 0.02 987 -> 45.
template <bool kSingle, bool kLjIsRc>
__global__ void __launch_bounds__(brick::kThreads, 4)
    k_pairs_sparse(brick::Const p, brick::Box bx, int nbricks, const double* __restrict__ rx,
                   const double* __restrict__ ry, const double* __restrict__ rz, const int32_t* __restrict__ cid,
                   const int32_t* __restrict__ cstart, const PairParams* __restrict__ pp, double* __restrict__ fx,
                   double* __restrict__ fy, double* __restrict__ fz, double* __restrict__ partials,
                   int* __restrict__ status, brick::Lists lists) {
	__shared__ brick::SparseTraverse s_warp[brick::kWarps];
	const int b = (int) blockIdx.x * brick::kWarps + (int) (threadIdx.x >> 5);
	if (b >= nbricks) return;
	if (!brick::pairs_sparse<kSingle, kLjIsRc>(p, bx, b, s_warp[threadIdx.x >> 5], pp, rx, ry, rz, cid, cstart, fx, fy,
	                                           fz, partials, status) &&
	    (threadIdx.x & 31) == 0)
		lists.blist[atomicAdd(lists.counts, 1u)] = b;
}

// Verlet-skin build step (runs only when *gate is this step's id): the lists, no forces.
constexpr int kBuildMinBlocks = 3;
__global__ void __launch_bounds__(brick::kThreads, kBuildMinBlocks)
    k_build_lists(brick::Box bx, int nbricks, int s_cap, const double* __restrict__ rx,
                  const double* __restrict__ ry, const double* __restrict__ rz, const int32_t* __restrict__ cstart,
                  const int* __restrict__ gate, int step, brick::Lists lists) {
	if (*gate != step) return;
	if (lists.pst && blockIdx.x == 0 && threadIdx.x == 0) lists.pst->built = step;   // pruned lists: prune now
	extern __shared__ __align__(16) unsigned char smem[];
	// a resident grid walks the bricks: a step without a build costs one launch of that grid only
	for (int b = blockIdx.x; b < nbricks; b += gridDim.x) {
		brick::build_lists(bx, b, s_cap, smem, rx, ry, rz, cstart, lists, b);
		__syncthreads();
	}
}

// Resident CTAs per SM of the list kernels (registers and shared memory are sized for it). The FP64 form
// stages only images and component ids (25 bytes per molecule, 40 with the FP32 form's split positions), so
// three CTAs hold its regions too: 400,009 molecules, us per step, one species 190 at the start, 132 with two
// CTAs, 113 with three; two species 204, 142, 143; 1,048,576 with pruned lists 295 with two, 254 with three.
constexpr int kListMinBlocks = 3;

// The list evaluation of a step. With pruned lists (lists.pst set) it comes in two variants, launched
// one after the other in every step: kPrune runs in the steps that prune (the lists were built in
// this step, or the summed largest drifts since the last prune reached half_prune), reads the build
// lists and writes the inner lists (po) besides the forces; the plain variant runs in the other
// steps and reads the inner lists. Both decide from values that no CTA of their launch changes (not
// from the rebuild flag, which the fused kick of this step may set for the next one).
template <bool kFP64, bool kSingle, bool kLjIsRc, bool kPrune = false>
__global__ void __launch_bounds__(brick::kThreads, kListMinBlocks)
    k_pairs_list(brick::Const p, brick::Box bx, const double* __restrict__ rx, const double* __restrict__ ry,
                 const double* __restrict__ rz, const int32_t* __restrict__ cid,
                 const int32_t* __restrict__ cstart, const PairParams* __restrict__ pp,
                 double* __restrict__ fx, double* __restrict__ fy, double* __restrict__ fz,
                 double* __restrict__ partials, int* __restrict__ status,
                 brick::Lists lists, unsigned* tickets, double* scalars, brick::Kick kick, double* record,
                 brick::PruneOut po, double half_prune) {
	if (lists.pst) {
		const PruneState* st = lists.pst;
		if (kPrune) {
			const double moved = st->acc + sqrt((double) __uint_as_float(st->dmax[lists.step & 1]));
			if (st->built != lists.step && moved < half_prune) return;
			if (blockIdx.x == 0 && threadIdx.x == 0) {
				lists.pst->pruned = lists.step;
				lists.pst->count++;
			}
		} else if (st->pruned == lists.step) {
			return;   // the prune variant evaluated this step
		}
	}
	extern __shared__ __align__(16) unsigned char smem[];
	__shared__ int s_item;
	brick::load_params(smem, brick::layout(p.s_cap, kFP64), pp, p.ns);
	if (threadIdx.x == 0) brick::drift_slot() = 0u;   // read after the barriers below
	if (lists.kind == nullptr) {
		// every brick, one CTA each
		__syncthreads();
		brick::list_pairs<kFP64, kSingle, kLjIsRc, true, kPrune>(p, bx, blockIdx.x, blockIdx.x, smem, rx, ry, rz, cid,
		                                                         cstart, fx, fy, fz, partials, status, lists, kick, po);
	} else {
		// the dense bricks of the last build (the sparse ones go to k_pairs_list_sparse): a resident
		// grid takes them from a queue
		const int nwork = (int) *(volatile unsigned*) (lists.counts + 1);
		for (;;) {
			__syncthreads();
			if (threadIdx.x == 0) s_item = (int) atomicAdd(lists.counts + 2, 1u);
			__syncthreads();
			const int item = s_item;
			if (item >= nwork) break;
			const int b = lists.blist[item];
			brick::list_pairs<kFP64, kSingle, kLjIsRc, true, kPrune>(p, bx, b, b, smem, rx, ry, rz, cid, cstart, fx, fy,
			                                                         fz, partials, status, lists, kick, po);
		}
	}
	__syncthreads();
	brick::drift_flush(kick.dmax);
	// U6 sum, virial sum, pair count (and sum m v^2 of the closing kick) of the step over every
	// brick's partials, summed by the last CTA to finish, which also writes the step record
	// {Upot, virial, sum m v^2, pairs} and resets both work queues
	if (last_block_sum(tickets, partials, lists.nbricks, kick.mode ? 4 : 3, scalars) && threadIdx.x == 0) {
		lists.counts[2] = 0u;
		lists.counts[3] = 0u;
		if (lists.pst) {
			// the drift into this step's positions joins the sum, which a prune at this step restarts
			PruneState* st = lists.pst;
			const int par = lists.step & 1;
			st->acc = kPrune ? 0.0 : st->acc + sqrt((double) __uint_as_float(st->dmax[par]));
			st->dmax[par] = 0u;
		}
		if (record) {
			record[0] = scalars[0] * 0.5 / 6.;
			record[1] = scalars[1] * 0.5;
			record[2] = scalars[3];
			record[3] = scalars[2] * 0.5;
		}
	}
}

// Sparse bricks (few molecules, e.g. a vapour), one warp each: every warp of a resident grid takes
// the sparse bricks of the last build from a queue.
template <bool kFP64, bool kSingle, bool kLjIsRc>
__global__ void __launch_bounds__(brick::kThreads, 2)
    k_pairs_list_sparse(brick::Const p, brick::Box bx, const double* __restrict__ rx,
                        const double* __restrict__ ry, const double* __restrict__ rz,
                        const int32_t* __restrict__ cid, const int32_t* __restrict__ cstart,
                        const PairParams* __restrict__ pp, double* __restrict__ fx, double* __restrict__ fy,
                        double* __restrict__ fz, double* __restrict__ partials, int* __restrict__ status,
                        brick::Lists lists, brick::Kick kick) {
	extern __shared__ __align__(16) unsigned char smem[];
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	unsigned char* ws = smem + warp * brick::sparse_warp_bytes(kFP64);
	const brick::SmemLayout L = brick::layout(brick::kSparseCap, kFP64);
	double* pd = reinterpret_cast<double*>(ws + L.params);
	float* pf = reinterpret_cast<float*>(pd + 3 * brick::KK);
	for (int k = lane; k < p.ns * p.ns; k += 32) {
		pd[k] = pp->eps24[k];
		pd[brick::KK + k] = pp->sig2[k];
		pd[2 * brick::KK + k] = pp->shift6[k];
		pf[k] = (float) pp->eps24[k];
		pf[brick::KK + k] = (float) pp->sig2[k];
		pf[2 * brick::KK + k] = (float) pp->shift6[k];
	}
	if (!kFP64 && lane == 0)
		reinterpret_cast<float4*>(ws + L.hi)[brick::kSparseCap] =
		    make_float4(1e15f, 1e15f, 1e15f, __uint_as_float((256u << 18) | (256u << 9) | 256u));
	if (threadIdx.x == 0) brick::drift_slot() = 0u;
	__syncthreads();
	const int nwork = (int) *(volatile unsigned*) lists.counts;
	for (;;) {
		__syncwarp();
		int item = 0;
		if (lane == 0) item = (int) atomicAdd(lists.counts + 3, 1u);
		item = __shfl_sync(brick::kFull, item, 0);
		if (item >= nwork) break;
		const int b = lists.blist[lists.nbricks + item];
		brick::list_pairs_warp<kFP64, kSingle, kLjIsRc>(p, bx, b, ws, rx, ry, rz, cid, cstart, fx, fy, fz, partials,
		                                                status, lists, kick);
	}
	__syncthreads();
	brick::drift_flush(kick.dmax);
}

// Resident grid of a kernel: the CTAs that fit on the device at once (at most `cap`). The
// occupancy query is a host call of several microseconds; its answer per (kernel, shared memory)
// is kept, since small boxes stepped one launch at a time would otherwise pay it every step.
template <typename K>
int resident_grid(const Context* c, K kern, size_t smem, int cap) {
	static std::mutex mu;
	static std::map<std::pair<const void*, size_t>, int> known;
	const auto key = std::make_pair(reinterpret_cast<const void*>(kern), smem);
	int per_sm = 0;
	{
		std::lock_guard<std::mutex> lock(mu);
		auto it = known.find(key);
		if (it != known.end()) per_sm = it->second;
	}
	if (per_sm == 0) {
		if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, brick::kThreads, smem) != cudaSuccess ||
		    per_sm < 1)
			per_sm = 1;
		std::lock_guard<std::mutex> lock(mu);
		known[key] = per_sm;
	}
	return std::max(1, std::min(cap, per_sm * c->num_sms));
}

struct Plan {
	brick::Const p;
	brick::Box bx;
	size_t bytes;
	int nbricks;
};

// Shared memory per CTA with `ctas` of them per SM: the SM's 228 KB, less 1 KB reserved per CTA and a margin.
size_t share(const Context* c, int ctas) {
	return std::min((size_t) (224 / ctas - 2) * 1024, (size_t) device_max_optin(c->device));
}

// Whether a capacity of s_cap staged molecules, that of `ctas` CTAs per SM, holds a region of 64 cells with
// room for its fluctuations. The kernels take the most CTAs per SM for which it does: of a region above the
// capacity the traversal stages the parts one by one (30,000 molecules loaded at a density of 0.1 and then set
// to a droplet: 117 us per step), and the list kernels gather the candidates from global memory, ten times as
// slow. The skin cells of a small box can be much larger than the radius asks for (3 or 4 along an edge, two or
// three times the molecules), so the lists' last step is the whole SM for one CTA. A grid of one CTA per SM or
// less loses nothing by it and asks for the most room (with 3 cells along an edge a region holds some of them
// twice); a larger one asks for little (a liquid's regions differ by a percent or two, and the density around a
// molecule of a lattice is 6 % high already: with 1.15 for the step to three CTAs the FP64 form with pruned
// lists took two for 1,048,576 molecules, whose regions of 2,048 three hold: 0.445 ms per step against 0.374).
// 20 steps of FP64 runs with skin 0.3, at a density of 0.7 and a cutoff of 2.5, in ms, with one fixed capacity
// and with this rule: 1,500 molecules 11.2 and 1.4, 3,300 10.0 and 1.3, 5,000 23.7 and 1.7 (FP32 25.3 and
// 1.5), 8,000 4.8 and 1.3.
bool region_fits(const Context* c, const Grid& g, int kind, int ctas, int s_cap) {
	const double rho = c->rho_typ > 0.0 ? c->rho_typ : (double) c->n / (g.L[0] * g.L[1] * g.L[2]);
	const double region = 64.0 * rho * g.cell_length[0] * g.cell_length[1] * g.cell_length[2];
	const int64_t nbricks = (int64_t) ((g.nc[0] + 1) / 2) * ((g.nc[1] + 1) / 2) * ((g.nc[2] + 1) / 2);
	const double room = nbricks <= c->num_sms || (kind == 0 && ctas > 2) ? 1.3 : 1.05;
	return room * region + 64.0 <= s_cap;
}

// kind 0: plain traversal, 2: list evaluation of the skin mode.
Plan plan(Context* c, const Grid& g, double filter_radius, int kind) {
	const bool fp64 = kind == 0 || c->precision == MDGPU_FP64;   // the traversal evaluates both modes in FP64
	Plan P;
	brick::init_box(P.bx, g, filter_radius, 0, kind == 0 ? 0.0 : 0.5 * c->skin);
	const int words = kind == 2 ? 0 : brick::kHitWords;
	// The prune variant's ring takes its part of each share.
	const size_t ring = kind == 2 && pruning(c) ? brick::kPruneRingBytes : 0;
	int s_cap = 0;
	// the traversal stops at two CTAs, the batched ensemble's capacity: both then evaluate the same bricks in
	// parts, and a box steps bit for bit as it does alone. Parts reach regions of 5,900 molecules that way, as many
	// as one CTA per SM would stage whole.
	for (int ctas = kind == 2 ? kListMinBlocks : kTraverseMinBlocks; ctas >= (kind == 2 ? 1 : 2); ctas--) {
		s_cap = brick::capacity_for(share(c, ctas) - ring, fp64, words);
		if (region_fits(c, g, kind, ctas, s_cap)) break;
	}
	P.p = brick::make_const(c->sp.n, s_cap, c->rc, c->rc_lj);
	P.bytes = brick::layout(s_cap, fp64, words).total;
	P.nbricks = P.bx.nb[0] * P.bx.nb[1] * P.bx.nb[2];
	return P;
}

// Whether the traversal's last CTA sums the bricks' partials. It costs every CTA a fence and an atomic
// before it ends, which is cheaper than another launch up to about one resident round of CTAs (16,384
// molecules: 1 against 3 us), but not where many short CTAs follow one another (24,400 bricks of a slab:
// 47 against 8 us).
bool fold_in_traversal(const Context* c, const Plan& P) { return P.nbricks <= kTraverseMinBlocks * c->num_sms; }

template <typename K, typename... Extra>
cudaError_t go(Context* c, const Plan& P, K kern, const brick::Lists& lists, Extra... extra) {
	cudaError_t r = allow_dynamic_smem((const void*) kern, c->device, P.bytes);
	// the list kernel runs as a resident grid over a queue of the dense bricks when the sparse ones are
	// evaluated apart (lists.kind set, or lists.counts in the traversal); otherwise one CTA per brick
	const bool queue = lists.kind || (lists.counts && !lists.nbr);
	const int grid = queue ? resident_grid(c, kern, P.bytes, P.nbricks) : P.nbricks;
	if (r == cudaSuccess)
		kern<<<grid, brick::kThreads, P.bytes, c->stream>>>(P.p, P.bx, c->p.rx, c->p.ry, c->p.rz, c->p.cid,
		                                                         c->cell_start, c->d_pp, c->p.fx, c->p.fy, c->p.fz,
		                                                         c->partials, c->status, lists, extra...);
	return r;
}

// kind 0: plain traversal, 2: list evaluation of the skin mode (kPr: its prune variant)
template <int kKind, bool kPr = false>
cudaError_t dispatch(Context* c, const Plan& P, const brick::Lists& lists,
                     const brick::Kick& kick = brick::Kick{}, double* record = nullptr,
                     const brick::PruneOut& po = brick::PruneOut{}, double half_prune = 0.0) {
	const bool fp64 = c->precision == MDGPU_FP64;
	const bool single = c->sp.n == 1, ljrc = c->rc_lj == c->rc;
	if (kKind == 2) {
		unsigned* t = c->tickets;
		double* out = c->scalars;
		if (fp64 && ljrc)
			return single ? go(c, P, k_pairs_list<true, true, true, kPr>, lists, t, out, kick, record, po, half_prune)
			              : go(c, P, k_pairs_list<true, false, true, kPr>, lists, t, out, kick, record, po,
			                   half_prune);
		if (fp64)
			return single ? go(c, P, k_pairs_list<true, true, false, kPr>, lists, t, out, kick, record, po, half_prune)
			              : go(c, P, k_pairs_list<true, false, false, kPr>, lists, t, out, kick, record, po,
			                   half_prune);
		if (ljrc)
			return single ? go(c, P, k_pairs_list<false, true, true, kPr>, lists, t, out, kick, record, po, half_prune)
			              : go(c, P, k_pairs_list<false, false, true, kPr>, lists, t, out, kick, record, po,
			                   half_prune);
		return single ? go(c, P, k_pairs_list<false, true, false, kPr>, lists, t, out, kick, record, po, half_prune)
		              : go(c, P, k_pairs_list<false, false, false, kPr>, lists, t, out, kick, record, po,
		                   half_prune);
	}
	unsigned* t = fold_in_traversal(c, P) ? c->tickets + 2 : nullptr;
	if (ljrc) return single ? go(c, P, k_pairs_brick<true, true>, lists, t, c->scalars)
	                        : go(c, P, k_pairs_brick<false, true>, lists, t, c->scalars);
	return single ? go(c, P, k_pairs_brick<true, false>, lists, t, c->scalars)
	              : go(c, P, k_pairs_brick<false, false>, lists, t, c->scalars);
}

brick::Lists lists_of(Context* c) {
	brick::Lists l{};
	l.nbr = c->nbr;
	l.count = c->nbr_count;
	l.rx_ref = c->r_ref;
	l.ry_ref = c->r_ref + c->n;
	l.rz_ref = c->r_ref + 2 * c->n;
	l.n = c->n;
	l.cap = c->list_cap;
	l.builds = c->builds;
	l.kind = c->brick_kind;
	l.counts = c->brick_counts;
	l.blist = c->brick_list;
	l.nbricks = (int) skin_partials_needed(c);
	return l;
}

}  // namespace

// Whether a traversal looks for sparse bricks first: where there are several rounds of bricks and many
// are expected to be sparse -- a dilute fluid, or one that leaves much of the box nearly empty (the density
// around a typical molecule is well above the mean). A homogeneous liquid has none, and skips the launch.
bool sparse_traversal(const Context* c, const Plan& P) {
	if (!c->trav_list || P.nbricks > c->trav_cap || P.nbricks < sparse_min_bricks(c)) return false;
	const Grid& g = c->g;
	const double rho = (double) c->n / (g.L[0] * g.L[1] * g.L[2]);
	const double cell = g.cell_length[0] * g.cell_length[1] * g.cell_length[2];
	return 64.0 * rho * cell <= 0.75 * brick::kSparseCap || c->rho_typ > 1.5 * rho;
}

cudaError_t launch_pairs_brick(Context* c) {
	const Plan P = plan(c, c->g, c->rc, 0);
	prof_begin(c, 1);
	brick::Lists l{};
	cudaError_t e = cudaSuccess;
	const bool sparse = sparse_traversal(c, P);
	if (sparse) {
		l.counts = c->trav_counts;
		l.blist = c->trav_list;
		e = cudaMemsetAsync(l.counts, 0, sizeof(unsigned) * 2, c->stream);
		const bool single = c->sp.n == 1, ljrc = c->rc_lj == c->rc;
		auto ks = single ? (ljrc ? k_pairs_sparse<true, true> : k_pairs_sparse<true, false>)
		                 : (ljrc ? k_pairs_sparse<false, true> : k_pairs_sparse<false, false>);
		if (e == cudaSuccess)
			ks<<<(P.nbricks + brick::kWarps - 1) / brick::kWarps, brick::kThreads, 0, c->stream>>>(
			    P.p, P.bx, P.nbricks, c->p.rx, c->p.ry, c->p.rz, c->p.cid, c->cell_start, c->d_pp, c->p.fx, c->p.fy,
			    c->p.fz, c->partials, c->status, l);
	}
	if (e == cudaSuccess) e = dispatch<0>(c, P, l);
	if (e == cudaSuccess) e = cudaGetLastError();
	prof_end(c, 1, sparse ? 2 : 1);
	if (e != cudaSuccess || fold_in_traversal(c, P)) return e;
	return launch_reduce(c, P.nbricks, c->scalars, 3);
}

cudaError_t launch_pairs_skin(Context* c, int kick_mode, double dt, double* record) {
	brick::Lists l = lists_of(c);
	brick::Kick kick{};
	kick.mode = kick_mode;
	if (kick_mode) {
		kick.id = c->step_id + 1;   // the step whose rebuild a long drift asks for
		kick.dt = dt;
		kick.half2 = 0.25 * c->skin * c->skin;
		for (int k = 0; k < c->sp.n; k++) {
			kick.post[k] = (0.5 * dt) / c->sp.mass[k];
			kick.pre[k] = (.5 * dt) / c->sp.mass[k];
			kick.mass[k] = c->sp.mass[k];
		}
		kick.vx = c->p.vx;
		kick.vy = c->p.vy;
		kick.vz = c->p.vz;
		kick.ox = c->q.rx;
		kick.oy = c->q.ry;
		kick.oz = c->q.rz;
		kick.flag = c->rebuild;
		if (pruning(c) && kick_mode == 1) kick.dmax = &c->prune_st->dmax[(c->step_id + 1) & 1];
	}
	const Plan P = plan(c, c->gs, c->rc, 2);
	l.sentinel = P.p.s_cap;   // the evaluation kernel's sentinel slot terminates every list
	int launches = 2;
	// pruned lists: the prune variant of the evaluation reads the build lists (and writes the inner
	// ones) in the steps that prune, the plain variant reads the inner lists in the others; the
	// sparse bricks always evaluate their build lists; the build records its step in the prune state
	brick::Lists inner = l;
	brick::PruneOut po{};
	double half_prune = 0.0;
	const bool prune = pruning(c);
	if (prune) {
		l.pst = c->prune_st;
		l.step = c->step_id;
		inner = l;
		inner.nbr = c->nbr_in;
		inner.count = c->nbr_in_count;
		po.nbr = c->nbr_in;
		po.count = c->nbr_in_count;
		// the FP32 form's split positions: the lo parts (at most 256 steps each way per coordinate, plus
		// half a step of quantisation) move the distance by at most sqrt(3) * 513 steps; the float
		// arithmetic by a few 1e-7 of it
		const double lo = 520.0 * std::max(P.bx.lo_step[0], std::max(P.bx.lo_step[1], P.bx.lo_step[2]));
		const double rp = c->rc + c->prune + 1.7320508075688772 * lo;
		const double rp2 = rp * rp * (1.0 + 2e-6);
		po.rp2f = (float) rp2;
		if ((double) po.rp2f < rp2) po.rp2f = std::nextafter(po.rp2f, 2.0f * po.rp2f);
		// prune when the drifts reach half the inner skin, less a margin that keeps every pair left
		// out farther than rc (1 + 1e-5) from the other molecule until then
		half_prune = 0.5 * c->prune - 1e-5 * (c->rc + c->prune);
		launches++;
	}
	prof_begin(c, 1);
	// build (gated): half-precision staging only
	brick::Box bb{};
	brick::init_box(bb, c->gs, c->rc + c->skin, 0, 0.5 * c->skin);
	int s_cap = 0, ctas = kBuildMinBlocks;
	for (;; ctas--) {
		s_cap = 256;
		while (brick::build_bytes(s_cap + 64) <= share(c, ctas)) s_cap += 64;
		if (ctas == 1 || region_fits(c, c->gs, 2, ctas, s_cap)) break;
	}
	const size_t bbytes = brick::build_bytes(s_cap);
	const int nbricks = bb.nb[0] * bb.nb[1] * bb.nb[2];
	cudaError_t e = allow_dynamic_smem((const void*) k_build_lists, c->device, bbytes);
	const int grid = std::min(nbricks, ctas * c->num_sms);
	if (e == cudaSuccess)
		k_build_lists<<<grid, brick::kThreads, bbytes, c->stream>>>(bb, nbricks, s_cap, c->p.rx, c->p.ry, c->p.rz,
		                                                           c->cell_start, c->rebuild, c->step_id, l);
	// evaluation, every step: sparse bricks one warp each, then the others (whose last CTA sums the
	// partials of all bricks). When the last build of an earlier run found no sparse brick the
	// dense kernel takes every brick (kind not consulted) and the sparse kernel is not launched.
	const bool sparse = !c->h_sparse || *(volatile int*) c->h_sparse != 0;
	brick::Lists ld = l, ldi = inner;
	if (!sparse) ld.kind = ldi.kind = nullptr;
	if (e == cudaSuccess && sparse) {
		const bool fp64 = c->precision == MDGPU_FP64;
		const bool single = c->sp.n == 1, ljrc = c->rc_lj == c->rc;
		auto ks = fp64 ? (single ? (ljrc ? k_pairs_list_sparse<true, true, true> : k_pairs_list_sparse<true, true, false>)
		                         : (ljrc ? k_pairs_list_sparse<true, false, true>
		                                 : k_pairs_list_sparse<true, false, false>))
		               : (single ? (ljrc ? k_pairs_list_sparse<false, true, true> : k_pairs_list_sparse<false, true, false>)
		                         : (ljrc ? k_pairs_list_sparse<false, false, true>
		                                 : k_pairs_list_sparse<false, false, false>));
		const size_t sbytes = brick::kWarps * brick::sparse_warp_bytes(fp64);
		const brick::Const ps = brick::make_const(c->sp.n, brick::kSparseCap, c->rc, c->rc_lj);
		e = allow_dynamic_smem((const void*) ks, c->device, sbytes);
		const int sgrid = resident_grid(c, ks, sbytes, (P.nbricks + brick::kWarps - 1) / brick::kWarps);
		if (e == cudaSuccess)
			ks<<<sgrid, brick::kThreads, sbytes, c->stream>>>(ps, P.bx, c->p.rx, c->p.ry, c->p.rz, c->p.cid,
			                                                   c->cell_start, c->d_pp, c->p.fx, c->p.fy, c->p.fz,
			                                                   c->partials, c->status, l, kick);
	}
	if (e == cudaSuccess && prune) {
		Plan Pp = P;
		Pp.bytes += brick::kPruneRingBytes;
		e = dispatch<2, true>(c, Pp, ld, kick, record, po, half_prune);
	}
	if (e == cudaSuccess) e = dispatch<2>(c, P, prune ? ldi : ld, kick, record);
	if (e == cudaSuccess) e = cudaGetLastError();
	prof_end(c, 1, sparse ? launches + 1 : launches);
	return e;
}

int64_t skin_partials_needed(const Context* c) {
	return (int64_t) ((c->gs.nc[0] + 1) / 2) * ((c->gs.nc[1] + 1) / 2) * ((c->gs.nc[2] + 1) / 2);
}

}  // namespace mdgpu
