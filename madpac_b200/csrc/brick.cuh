// Pair traversal of one brick of 2x2x2 linked cells staged in shared memory (device function used
// by the single-box pair kernels and by the persistent multi-box step kernel).
//
// One CTA (8 warps) owns a brick of 2x2x2 cells and computes the full force on its molecules from every
// molecule of the 27 cells around theirs (periodic images at +-L, r_j + L / r_j - L as
// DomainDecompDummy::exchangeMolecules places halo images, parallel/DomainDecompDummy.cpp:64-70, 93-99;
// paths relative to madpac/mardyn/). Two ways lead there:
//
//  pairs       the drop-in traversal, every call: staging of the 4x4x4 cells around the brick, a packed
//              half-precision filter over the rows of 3 cells around each molecule's cell (rc plus a
//              margin covering the rounding) and the exact evaluation of its hits in FP64.
//  list_pairs  the Verlet-skin steps: the lists that build_lists made with the same filter are evaluated
//              at the current positions, in FP64 or (mixed form) in FP32 with FP64 accumulation.
//
// Staging copies the region's molecules to shared memory cell by cell (x fastest), so the 3 cells of each
// neighbour row of a cell form one contiguous slot range. The FP64 evaluations read the double image
// position x + shift. The FP32 lists read a local frame X = x + shift - c_brick + C, C = 1.5 * 2^k with
// all X of the region in [2^k, 2^(k+1)]: differences of their float "hi" parts are exact (Sterbenz), and
// the "lo" part X - hi is kept as 9-bit fixed point (steps of 1/512 ulp of the binade) in the 4th word
// of the same float4, with the component id: (hi_i - hi_j) + (lo_i - lo_j) is X_i - X_j to about 2e-9
// absolute, one 16-byte shared load per candidate.
// The exact cutoff test is dd < rc^2, strict as BlockTraverse.cpp:155, decided in FP64 as the reference
// decides it; the force law is PotForceLJ's (molecules/potforce.h:41-53). A brick whose region holds more
// molecules than the shared-memory capacity is evaluated in parts by the traversal (pairs_in_parts); the list
// kernels, whose capacity follows the density, gather its candidates straight from global memory.
//
// Each unordered pair is evaluated from both sides; energy and virial are halved on readout.
// Orders of staging, enumeration and accumulation are fixed: results are deterministic and do not
// depend on which CTA evaluates a brick. (Between launches of different capacity, one of which evaluates a
// brick whole and the other in parts, the order of a molecule's pairs and the last bits differ.)
#pragma once

#include <cuda_runtime.h>

#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>

#include "md_internal.h"
#include "pair_common.cuh"
#include "reduce.cuh"

namespace mdgpu {
namespace brick {

constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;
constexpr unsigned kFull = 0xffffffffu;
constexpr int KK = kMaxSpecies * kMaxSpecies;

// Constants shared by every brick of a launch.
struct Const {
	int ns;
	int s_cap;            // staged molecule capacity of the shared-memory layout
	float rc2f, band;     // float rc^2 and the band around it resolved in double
	float rclj2f;
	double rc2, rclj2;
};

// One periodic box as the brick code sees it: its cell grid, its bricks per dimension, the offset of
// its cells in the cell-start array, and the frame constants of the packed filter.
struct Box {
	Grid g;
	int nb[3];
	int32_t coff;
	float frame_c[3];     // C per dimension
	float rc2_h;          // rc^2 + margin covering half-precision rounding (packed filter)
	float lo_step[3];     // fixed-point step of the lo parts: 2^(k-32) for the binade [2^k, 2^(k+1))
	float lo_inv[3];      // 1 / lo_step
};

struct SmemLayout {
	size_t hi, img, comp, h16, cstart, lists, ccount, gstart, cell_k, cell_shift, params, total;
};

// Two consecutive staged molecules in half precision, relative to the brick centre: the packed
// filter tests two candidates per instruction.
struct __align__(16) HalfPair {
	__half2 x, y, z, pad;
};

__host__ __device__ inline size_t align16(size_t x) { return (x + 15) & ~size_t(15); }

// Shared memory of the list kernels (they read their lists from global memory): in the FP32 form the hi/lo
// positions with the far-away sentinel slot past the capacity, in the FP64 form the double images and the
// component ids. With words > 0 that of the traversal (pairs, fp64), which adds the packed half-precision
// copy for its filter and `words` hit words per lane.
__host__ __device__ inline SmemLayout layout(int s_cap, bool fp64, int words = 0) {
	SmemLayout L;
	size_t o = 0;
	const bool traverse = words > 0;
	L.hi = o;
	if (!fp64) o = align16(o + sizeof(float4) * (s_cap + 1));
	L.img = o;
	if (fp64) o = align16(o + sizeof(double) * 3 * s_cap);
	L.comp = o;
	if (fp64) o = align16(o + s_cap);
	L.h16 = o;
	if (traverse) o = align16(o + sizeof(HalfPair) * (s_cap / 2 + 20));  // 16-slot blocks may read past the end
	L.cstart = o;
	o = align16(o + sizeof(int) * 65);
	L.lists = o;
	if (traverse) o = align16(o + sizeof(unsigned) * kThreads * (words + 1));   // one past the last is read
	L.ccount = o;
	o = align16(o + sizeof(int) * 64);
	L.gstart = o;
	o = align16(o + sizeof(int) * 64);
	L.cell_k = o;
	if (!traverse) o = align16(o + sizeof(double) * 3 * 64);
	L.cell_shift = o;
	if (!traverse) o = align16(o + sizeof(double) * 3 * 64);
	L.params = o;
	o = align16(o + sizeof(double) * 3 * KK + sizeof(float) * 3 * KK);
	L.total = o;
	return L;
}

// Largest staged capacity (a multiple of 64) whose layout fits in `budget` bytes.
inline int capacity_for(size_t budget, bool fp64, int words = 0) {
	int s_cap = 256;
	while (layout(s_cap + 64, fp64, words).total <= budget) s_cap += 64;
	return s_cap > 65535 ? 65535 : s_cap;
}

// Frame constants of one box (host side).
// drift: how far a molecule may be outside its cell when staged (half the skin in the Verlet-skin
// mode, 0 otherwise).
inline void init_box(Box& b, const Grid& g, double rc, int32_t coff, double drift = 0.0) {
	b.g = g;
	b.coff = coff;
	for (int d = 0; d < 3; d++) {
		b.nb[d] = (g.nc[d] + 1) / 2;
		const double cl = g.cell_length[d];
		// smallest 2^k with the staged region X in [C - 2cl - drift, C + 2cl + drift] inside
		// [2^k, 2^(k+1)]
		double pk = 1.0;
		while (pk < 4.0 * cl + 2.0 * drift) pk *= 2.0;
		b.frame_c[d] = (float) (1.5 * pk);
		b.lo_step[d] = (float) std::ldexp(pk, -32);
		b.lo_inv[d] = (float) std::ldexp(1.0 / pk, 32);
	}
	// half-precision filter: coordinates within +-2 cells of the brick centre; each rounding is at
	// most half an ulp of the largest coordinate, plus the rounding of the packed r^2 itself
	const double cmax = 2.0 * std::max(g.cell_length[0], std::max(g.cell_length[1], g.cell_length[2])) + drift;
	const double uc = std::ldexp(1.0, std::ilogb(cmax) - 10);   // half ulp at cmax (10-bit mantissa)
	const double du = 2.0 * uc * 1.7320508;                     // |error of the difference vector|
	const double r2max = (rc + du) * (rc + du);
	const double ur2 = std::ldexp(1.0, std::ilogb(r2max) - 10);
	b.rc2_h = (float) (r2max + 4.0 * ur2 + 1e-3);
}

inline Const make_const(int ns, int s_cap, double rc, double rc_lj) {
	Const p{};
	p.ns = ns;
	p.s_cap = s_cap;
	p.rc2 = rc * rc;
	p.rclj2 = rc_lj * rc_lj;
	p.rc2f = (float) p.rc2;
	p.rclj2f = (float) p.rclj2;
	p.band = (float) (4e-6 * p.rc2);
	return p;
}

// Reciprocal by the hardware approximation (rcp.approx.ftz.f32, about 1 ulp).
__device__ __forceinline__ float rcp_approx(float x) {
	float r;
	asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
	return r;
}

// Copies the Comp2Param table to shared memory (double and float); the caller synchronises.
__device__ __forceinline__ void load_params(unsigned char* smem, const SmemLayout& L, const PairParams* pp, int ns) {
	double* s_pd = reinterpret_cast<double*>(smem + L.params);
	float* s_pf = reinterpret_cast<float*>(s_pd + 3 * KK);
	for (int k = threadIdx.x; k < ns * ns; k += kThreads) {
		s_pd[k] = pp->eps24[k];
		s_pd[KK + k] = pp->sig2[k];
		s_pd[2 * KK + k] = pp->shift6[k];
		s_pf[k] = (float) pp->eps24[k];
		s_pf[KK + k] = (float) pp->sig2[k];
		s_pf[2 * KK + k] = (float) pp->shift6[k];
	}
}

// Views of the shared-memory layout.
struct Smem {
	float4* hi;
	double* img;
	unsigned char* comp;  // component ids (FP64)
	HalfPair* h16;
	__half* h;
	int* cs;              // staged slot of each staged cell (65)
	unsigned* words;      // hit words of the traversal (a column per thread)
	int* cnt;
	int* gst;
	double* ck;           // frame offset and image shift of each staged cell (list kernels)
	double* csh;
	double* pd;           // eps24, sig2, shift6 (double)
	float* pf;            // the same as float
};

__device__ __forceinline__ Smem views(unsigned char* smem, const SmemLayout& L) {
	Smem S;
	S.hi = reinterpret_cast<float4*>(smem + L.hi);
	S.img = reinterpret_cast<double*>(smem + L.img);
	S.comp = smem + L.comp;
	S.h16 = reinterpret_cast<HalfPair*>(smem + L.h16);
	S.h = reinterpret_cast<__half*>(S.h16);
	S.cs = reinterpret_cast<int*>(smem + L.cstart);
	S.words = reinterpret_cast<unsigned*>(smem + L.lists);
	S.cnt = reinterpret_cast<int*>(smem + L.ccount);
	S.gst = reinterpret_cast<int*>(smem + L.gstart);
	S.ck = reinterpret_cast<double*>(smem + L.cell_k);
	S.csh = reinterpret_cast<double*>(smem + L.cell_shift);
	S.pd = reinterpret_cast<double*>(smem + L.params);
	S.pf = reinterpret_cast<float*>(S.pd + 3 * KK);
	return S;
}

// Warp w's brick cell: local (1 + (w&1), 1 + ((w>>1)&1), 1 + (w>>2)) in the 4x4x4 staged region;
// false when it lies beyond the grid (odd cell counts: the last brick of a dimension is partial).
__device__ __forceinline__ bool own_cell(const Box& bx, int brick, int w, int& icell) {
	const int bxi = brick % bx.nb[0];
	const int byi = (brick / bx.nb[0]) % bx.nb[1];
	const int bzi = brick / (bx.nb[0] * bx.nb[1]);
	const int il[3] = {1 + (w & 1), 1 + ((w >> 1) & 1), 1 + (w >> 2)};
	icell = il[0] + 4 * il[1] + 16 * il[2];
	return 2 * bxi + il[0] - 1 < bx.g.nc[0] && 2 * byi + il[1] - 1 < bx.g.nc[1] && 2 * bzi + il[2] - 1 < bx.g.nc[2];
}

// The packed 4th word of a staged molecule: lo parts as 9-bit fields (value + 256, bits 0-8, 9-17,
// 18-26) in steps of Box::lo_step, component id in bits 27-29.
__device__ __forceinline__ unsigned pack_lo(float lx, float ly, float lz, int cid, const Box& bx) {
	const float l[3] = {lx, ly, lz};
	unsigned w = (unsigned) cid << 27;
	for (int d = 0; d < 3; d++) {
		int q = __float2int_rn(l[d] * bx.lo_inv[d]);   // power-of-two step: exact product
		q = max(-255, min(255, q));
		w |= (unsigned) (q + 256) << (9 * d);
	}
	return w;
}

__device__ __forceinline__ int unpack_cid(unsigned w) { return (int) ((w >> 27) & 7u); }

// Component of a staged slot (FP64). The mask is a bounds guard only: no lane looks at a slot that nothing was
// staged to (idle lanes and the padding of lists look at a molecule of their own brick).
__device__ __forceinline__ int component(const Smem& S, int slot) { return S.comp[slot] & (kMaxSpecies - 1); }
static_assert((kMaxSpecies & (kMaxSpecies - 1)) == 0, "a power of two");

// What a staging stores: the list kernels' hi/lo frame positions (FP32) or double images and component ids
// (FP64), or the traversal's half-precision copy, double images and component ids.
enum Staging { kStageList32, kStageList64, kStageTraverse };

// Stages a molecule at double position (x, y, z), component q, at slot slot_s, with its cell's frame
// offset (kx, ky, kz) and image shift (shx, shy, shz). For the traversal the offset is that of the
// brick's centre, without the frame constant.
template <Staging kMode>
__device__ __forceinline__ void stage_at(const Box& bx, const Smem& S, int slot_s, double x, double y, double z, int q,
                                         double kx, double ky, double kz, double shx, double shy, double shz) {
	if (kMode != kStageList64) {
		const double Xd = __dadd_rn(x, kx), Yd = __dadd_rn(y, ky), Zd = __dadd_rn(z, kz);
		const float X = __double2float_rn(Xd), Y = __double2float_rn(Yd), Z = __double2float_rn(Zd);
		if (kMode == kStageTraverse) {
			// half-precision copy relative to the brick centre (slot pairs share one HalfPair)
			__half* hp = S.h + 8 * (slot_s >> 1) + (slot_s & 1);
			hp[0] = __float2half_rn(X);
			hp[2] = __float2half_rn(Y);
			hp[4] = __float2half_rn(Z);
		} else {
			const unsigned w = pack_lo(__double2float_rn(Xd - (double) X), __double2float_rn(Yd - (double) Y),
			                           __double2float_rn(Zd - (double) Z), q, bx);
			S.hi[slot_s] = make_float4(X, Y, Z, __uint_as_float(w));
		}
	}
	if (kMode != kStageList32) {
		S.comp[slot_s] = (unsigned char) q;
		S.img[3 * slot_s] = __dadd_rn(x, shx);
		S.img[3 * slot_s + 1] = __dadd_rn(y, shy);
		S.img[3 * slot_s + 2] = __dadd_rn(z, shz);
	}
}

// Staged coordinate l (0..3) of dimension d of a brick at coordinate b: the grid coordinate (periodic
// wrap), the image shift of its molecules and their frame offset, X = x + k, k = shift - c_brick + C.
__device__ __forceinline__ int staged_coord(const Box& bx, int d, int b, int l, double& sh, double& k) {
	int gc = 2 * b - 1 + l;
	sh = 0.0;
	if (gc < 0) {
		gc += bx.g.nc[d];
		sh = -bx.g.L[d];
	} else if (gc >= bx.g.nc[d]) {
		gc -= bx.g.nc[d];
		sh = bx.g.L[d];
	}
	k = (sh - (2 * b + 1) * bx.g.cell_length[d]) + (double) bx.frame_c[d];
	return gc;
}

// Part of a brick: node 1 is the brick, nodes 2 n and 2 n + 1 are the halves of node n, which split z, then y,
// then x. The own cells of a part are w (in binary zyx) with w >> (3 - level) == node - 2^level; it needs the
// cells next to those, 48, 36 or 27 of the 64. True for coordinate l of the staged cells in dimension d.
__device__ __forceinline__ int part_level(int node) { return 31 - __clz(node); }
__device__ __forceinline__ bool in_part(int node, int d, int l) {
	const int level = part_level(node);
	if (level < 3 - d) return true;
	return (unsigned) (l - ((node >> (level - 3 + d)) & 1)) <= 2u;
}

// Prefix sums (9) of the counts of a part's own cells (the other own cells, and cells beyond the grid, count as
// empty) and their staged cells (8), by one warp; the counts of staged cells 2 l and 2 l + 1 are in lane l's
// na and nb.
__device__ __forceinline__ void own_prefix(const Box& bx, int brick, int node, int na, int nb, int* s_own,
                                           int* s_ocell) {
	const int lane = threadIdx.x & 31;
	int ic = 0;
	const bool ok = lane < kWarps && own_cell(bx, brick, lane, ic) && ((8 + lane) >> (3 - part_level(node))) == node;
	const int a = __shfl_sync(kFull, na, ic >> 1), b = __shfl_sync(kFull, nb, ic >> 1);
	const int c = ok ? ((ic & 1) ? b : a) : 0;
	int own = c;
	for (int o = 1; o < kWarps; o <<= 1) {
		const int y = __shfl_up_sync(kFull, own, o);
		if (lane >= o) own += y;
	}
	if (lane < kWarps) {
		s_own[lane] = own - c;
		s_ocell[lane] = ic;
		if (lane == kWarps - 1) s_own[kWarps] = own;
	}
}

// Staging of the list kernels: the 4x4x4 cells around brick `brick`, cell by cell (their cells hold
// about 28 molecules, a warp's width). Returns false when the region exceeds the staged capacity
// (nothing staged then; the cell ranges S.gst/S.cnt are set either way). s_own and s_ocell: own_prefix.
// Ends with a CTA barrier.
template <bool kFP64, bool kWide>
__device__ __forceinline__ bool stage_cells(const Const& p, const Box& bx, int brick, const Smem& S, const double* rx,
                                            const double* ry, const double* rz, const int32_t* cid,
                                            const int32_t* cstart, int* s_own, int* s_ocell) {
	constexpr Staging kMode = kFP64 ? kStageList64 : kStageList32;
	const Grid& g = bx.g;
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int bc[3] = {brick % bx.nb[0], (brick / bx.nb[0]) % bx.nb[1], brick / (bx.nb[0] * bx.nb[1])};
	// staged cells k = lx + 4 ly + 16 lz, local l in 0..3, global 2b - 1 + l with periodic wrap
	if (tid < 64) {
		const int l[3] = {tid & 3, (tid >> 2) & 3, tid >> 4};
		int gc[3];
		for (int d = 0; d < 3; d++) gc[d] = staged_coord(bx, d, bc[d], l[d], S.csh[3 * tid + d], S.ck[3 * tid + d]);
		const int gcell = bx.coff + (gc[2] * g.nc[1] + gc[1]) * g.nc[0] + gc[0];
		const int st = cstart[gcell];
		S.gst[tid] = st;
		S.cnt[tid] = max(0, cstart[gcell + 1] - st);
	}
	__syncthreads();
	// exclusive scan of the 64 staged-cell counts (warp 0, two per lane)
	if (warp < 2) {
		const int a = S.cnt[2 * lane], b = S.cnt[2 * lane + 1];
		if (warp == 0) {
			int inc = a + b;
			for (int o = 1; o < 32; o <<= 1) {
				const int y = __shfl_up_sync(kFull, inc, o);
				if (lane >= o) inc += y;
			}
			const int excl = inc - (a + b);
			S.cs[2 * lane] = excl;
			S.cs[2 * lane + 1] = excl + a;
			if (lane == 31) S.cs[64] = inc;
		} else {
			own_prefix(bx, brick, 1, a, b, s_own, s_ocell);
		}
	}
	__syncthreads();
	const bool staged = S.cs[64] <= p.s_cap;
	// cell-major, each staged cell's molecules in their (id) order. A warp stages cells warp,
	// warp + 8, ...; kWide: four cells per round, every load of the round issued before the first
	// store (the stores to shared memory would otherwise hold back the next cell's loads). The
	// persistent ensemble kernel, at its register limit, stages one cell at a time.
	if (staged && !kWide) {
		for (int c = warp; c < 64; c += kWarps) {
			const int st = S.gst[c], cnt = S.cnt[c], base = S.cs[c];
			const double kx = S.ck[3 * c], ky = S.ck[3 * c + 1], kz = S.ck[3 * c + 2];
			const double shx = S.csh[3 * c], shy = S.csh[3 * c + 1], shz = S.csh[3 * c + 2];
			for (int e = lane; e < cnt; e += 32) {
				const int gi = st + e;
				stage_at<kMode>(bx, S, base + e, rx[gi], ry[gi], rz[gi], cid[gi], kx, ky, kz, shx, shy, shz);
			}
		}
	}
	if (staged && kWide) {
		auto one = [&](int c, int e, double x, double y, double z, int q) {
			stage_at<kMode>(bx, S, S.cs[c] + e, x, y, z, q, S.ck[3 * c], S.ck[3 * c + 1], S.ck[3 * c + 2], S.csh[3 * c],
			                S.csh[3 * c + 1], S.csh[3 * c + 2]);
		};
		for (int c0 = warp; c0 < 64; c0 += 4 * kWarps) {
			double x[4], y[4], z[4];
			int q[4];
#pragma unroll
			for (int u = 0; u < 4; u++) {
				const int c = c0 + u * kWarps;
				const int gi = S.gst[c] + lane;
				const bool a = lane < S.cnt[c];
				x[u] = a ? rx[gi] : 0.0;
				y[u] = a ? ry[gi] : 0.0;
				z[u] = a ? rz[gi] : 0.0;
				q[u] = a ? cid[gi] : 0;
			}
#pragma unroll
			for (int u = 0; u < 4; u++) {
				const int c = c0 + u * kWarps;
				const int cnt = S.cnt[c];
				if (lane < cnt) one(c, lane, x[u], y[u], z[u], q[u]);
				for (int e = lane + 32; e < cnt; e += 32) {
					const int gi = S.gst[c] + e;
					one(c, e, rx[gi], ry[gi], rz[gi], cid[gi]);
				}
			}
		}
	}
	__syncthreads();
	return staged;
}

// Staging of the traversal, whose cells hold few molecules (12 of a warp's 32 lanes at rc = 2.5 in a
// liquid): the 16 rows of four cells, which are contiguous slots, two rows per warp. Return value and
// arguments as stage_cells. Its CTA barrier at the end is its only one: every warp loads all cell starts
// and scans the counts itself (two cells per lane) instead of waiting for one warp's scan. Of a part (node > 1)
// only the cells that it needs are staged; the others count as empty.
__device__ __forceinline__ bool stage_rows(const Const& p, const Box& bx, int brick, int node, const Smem& S,
                                           const double* rx, const double* ry, const double* rz, const int32_t* cid,
                                           const int32_t* cstart, int* s_own, int* s_ocell) {
	const Grid& g = bx.g;
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const int bc[3] = {brick % bx.nb[0], (brick / bx.nb[0]) % bx.nb[1], brick / (bx.nb[0] * bx.nb[1])};
	// staged cells k = lx + 4 ly + 16 lz; this lane's: 2 lane and 2 lane + 1
	double t0, t1;
	const int gy = staged_coord(bx, 1, bc[1], (lane >> 1) & 3, t0, t1);
	const int gz = staged_coord(bx, 2, bc[2], lane >> 3, t0, t1);
	const int row0 = bx.coff + (gz * g.nc[1] + gy) * g.nc[0];
	const int ca = row0 + staged_coord(bx, 0, bc[0], 2 * (lane & 1), t0, t1);
	const int cb = row0 + staged_coord(bx, 0, bc[0], 2 * (lane & 1) + 1, t0, t1);
	const int sa = cstart[ca], ea = cstart[ca + 1], sb = cstart[cb], eb = cstart[cb + 1];
	int na = max(0, ea - sa), nb = max(0, eb - sb);
	if (node > 1) {
		const bool yz = in_part(node, 1, (lane >> 1) & 3) && in_part(node, 2, lane >> 3);
		if (!yz || !in_part(node, 0, 2 * (lane & 1))) na = 0;
		if (!yz || !in_part(node, 0, 2 * (lane & 1) + 1)) nb = 0;
	}
	int inc = na + nb;
	for (int o = 1; o < 32; o <<= 1) {
		const int y = __shfl_up_sync(kFull, inc, o);
		if (lane >= o) inc += y;
	}
	const int slot_a = inc - (na + nb);
	const int total = __shfl_sync(kFull, inc, 31);
	const bool staged = total <= p.s_cap;
	if (warp == 0) {
		S.cs[2 * lane] = slot_a;
		S.cs[2 * lane + 1] = slot_a + na;
		if (lane == 31) S.cs[64] = total;
		S.gst[2 * lane] = sa;
		S.gst[2 * lane + 1] = sb;
		S.cnt[2 * lane] = na;
		S.cnt[2 * lane + 1] = nb;
	} else if (warp == 1) {
		own_prefix(bx, brick, node, na, nb, s_own, s_ocell);
	}
	// lane 4 d + l holds the shift and the frame offset (of the brick's centre) of staged coordinate l of
	// dimension d
	double sh_l = 0.0, k_l = 0.0;
	if (lane < 12) {
		staged_coord(bx, lane >> 2, bc[lane >> 2], lane & 3, sh_l, k_l);
		k_l -= (double) bx.frame_c[lane >> 2];
	}
	if (staged) {
		for (int rr = 0; rr < 2; rr++) {
			// row `row`: its four cells' prefix counts, and the offset from a molecule's place in the row
			// to its index in the sorted arrays, per cell
			const int row = 2 * warp + rr;
			const int slot0 = __shfl_sync(kFull, slot_a, 2 * row);
			const int p1 = __shfl_sync(kFull, na, 2 * row);
			const int p2 = p1 + __shfl_sync(kFull, nb, 2 * row);
			const int p3 = p2 + __shfl_sync(kFull, na, 2 * row + 1);
			const int len = p3 + __shfl_sync(kFull, nb, 2 * row + 1);
			const int o0 = __shfl_sync(kFull, sa, 2 * row), o1 = __shfl_sync(kFull, sb, 2 * row) - p1;
			const int o2 = __shfl_sync(kFull, sa, 2 * row + 1) - p2, o3 = __shfl_sync(kFull, sb, 2 * row + 1) - p3;
			const double ky = __shfl_sync(kFull, k_l, 4 + (row & 3)), kz = __shfl_sync(kFull, k_l, 8 + (row >> 2));
			const double shy = __shfl_sync(kFull, sh_l, 4 + (row & 3)), shz = __shfl_sync(kFull, sh_l, 8 + (row >> 2));
			for (int e0 = 0; e0 < len; e0 += 64) {
				double x[2], y[2], z[2];
				int q[2], l[2];
#pragma unroll
				for (int u = 0; u < 2; u++) {
					const int e = e0 + 32 * u + lane;
					l[u] = (e >= p1 ? 1 : 0) + (e >= p2 ? 1 : 0) + (e >= p3 ? 1 : 0);
					const int gi = e + (e >= p2 ? (e >= p3 ? o3 : o2) : (e >= p1 ? o1 : o0));
					x[u] = y[u] = z[u] = 0.0;
					q[u] = 0;
					if (e < len) {
						x[u] = rx[gi];
						y[u] = ry[gi];
						z[u] = rz[gi];
						q[u] = cid[gi];
					}
				}
#pragma unroll
				for (int u = 0; u < 2; u++) {
					const double kx = __shfl_sync(kFull, k_l, l[u]), shx = __shfl_sync(kFull, sh_l, l[u]);
					const int e = e0 + 32 * u + lane;
					if (e < len)
						stage_at<kStageTraverse>(bx, S, slot0 + e, x[u], y[u], z[u], q[u], kx, ky, kz, shx, shy, shz);
				}
			}
		}
	}
	__syncthreads();
	return staged;
}

// Cutoff decision for a pair within a few ulp of rc (rare): recomputed from the FP64 positions in
// global memory with the FP64 path's operations (xi - (x_j + shift), sum of squares), so that the
// mixed mode evaluates exactly the pairs the FP64 mode evaluates. j is a staged slot; its cell is
// found by bisection of the staged-cell starts.
static __device__ __noinline__ bool exact_cut(const Smem& S, double rc2, int j, int gi, const double* rx, const double* ry,
                                       const double* rz) {
	int lo = 0, hi = 63;
	while (lo < hi) {
		const int mid = (lo + hi + 1) >> 1;
		if (S.cs[mid] <= j)
			lo = mid;
		else
			hi = mid - 1;
	}
	const int gj = S.gst[lo] + (j - S.cs[lo]);
	const double d0 = __dsub_rn(rx[gi], __dadd_rn(rx[gj], S.csh[3 * lo]));
	const double d1 = __dsub_rn(ry[gi], __dadd_rn(ry[gj], S.csh[3 * lo + 1]));
	const double d2 = __dsub_rn(rz[gi], __dadd_rn(rz[gj], S.csh[3 * lo + 2]));
	const double dd = __dadd_rn(__dadd_rn(__dmul_rn(d0, d0), __dmul_rn(d1, d1)), __dmul_rn(d2, d2));
	return dd < rc2;
}

// FP64 sums of one molecule's pairs: force, energy and virial before the pair parameters that the
// single-species form applies once per molecule (sums64_finish).
struct Sums64 {
	double x, y, z, u, w;
	int np, nlj;   // pairs within rc; pairs within rcLJ (where that is another radius)
};

// One candidate pair in FP64: d = r_i - r_j, branch-free (a pair outside the cutoffs, or v = false,
// adds zeros, provided that d and the pair parameters are finite: a caller without a partner passes a
// staged one). The squared distance and both cutoff tests keep the reference's operations and
// roundings (no contraction), so the pairs within rc are the reference's; the force law is
// PotForceLJ's (molecules/potforce.h:41-53), contracted: with s6 = (sig2/r^2)^3, m = s6^2 - s6 and
// e = s6^2 + m the sums are F += (e/r^2) d, U += m, W += e (the virial term d.f is e, as f = (e/r^2) d):
// 22 FP64 instructions against 38 and a division in the reference's order. A zero distance (its high
// word is zero) sets `same` and leaves non-finite sums. Returns the squared distance.
template <bool kSingle, bool kLjIsRc>
__device__ __forceinline__ double lj64(double d0, double d1, double d2, bool v, double rc2, double rclj2, double eps24,
                                     double sig2, double shift6, Sums64& s, bool& same) {
	const double dd = __dadd_rn(__dadd_rn(__dmul_rn(d0, d0), __dmul_rn(d1, d1)), __dmul_rn(d2, d2));
	const bool in = v && dd < rc2;
	const bool lj = kLjIsRc ? in : (in && dd < rclj2);
	s.np += in ? 1 : 0;
	if (!kLjIsRc) s.nlj += lj ? 1 : 0;
	same |= in && __double2hiint(dd) == 0;
	const double inv = lj ? rcp64(dd) : 0.0;
	const double s2 = sig2 * inv;
	const double s6 = s2 * s2 * s2;
	const double m = fma(s6, s6, -s6);
	double e = fma(s6, s6, m);
	if (kSingle) {
		s.u += m;
	} else {
		e *= eps24;
		s.u = fma(eps24, m, s.u) + (lj ? shift6 : 0.0);
	}
	const double fac = e * inv;
	s.x = fma(fac, d0, s.x);
	s.y = fma(fac, d1, s.y);
	s.z = fma(fac, d2, s.z);
	s.w += e;
	return dd;
}

// The pair parameters of a single-species molecule's sums.
template <bool kLjIsRc>
__device__ __forceinline__ void sums64_finish(Sums64& s, double eps24, double shift6) {
	s.x *= eps24;
	s.y *= eps24;
	s.z *= eps24;
	s.w *= eps24;
	s.u = fma(eps24, s.u, shift6 * (double) (kLjIsRc ? s.np : s.nlj));
}

// Neighbour lists of the Verlet-skin mode: entry k of molecule i (sorted slot) is a staged slot of
// i's brick region, stored at ((k/8)*n + i)*8 + k%8, so that one 16-byte load gives a lane 8 entries
// and a warp's loads are contiguous; count[i] entries, kListOverflow when more than cap were found.
struct Lists {
	unsigned short* nbr;
	unsigned short* count;
	double *rx_ref, *ry_ref, *rz_ref;   // positions at the build
	int64_t n;
	int cap;
	unsigned long long* builds;        // incremented once per build
	int sentinel;                      // staged slot of the list kernel's far-away sentinel
	unsigned char* kind;               // per brick: 1 = sparse (evaluated one warp per brick)
	// list kernels: sparse [0] and dense [1] bricks of the build (or null); traversal: bricks that are not
	// sparse [0] and the queue over them [1] (or null: no sparse bricks looked for)
	unsigned* counts;
	int32_t* blist;                    // dense bricks at [0, nbricks), sparse ones (lists only) from nbricks on
	int nbricks;
	PruneState* pst;                   // pruned lists: their state (the evaluation's last CTA updates it)
	int step;                          // id of the step being evaluated
};
// A brick is sparse when its whole staged region holds at most kSparseCap molecules and its own
// cells at most 32: one warp stages and evaluates it, without CTA-wide barriers.
constexpr int kSparseCap = 128;
constexpr unsigned short kListOverflow = 0xffff;

// Rows of the traversal's lanes: the 27 cells around a cell are 9 rows of 3 (row r: y offset r % 3 - 1,
// z offset r / 3 - 1), and the lanes of a molecule share its rows so that their hits are about equal
// (the middle row holds about 22 % of them, an edge row 12 %, a corner row 7 %). Entry lpm - 1 + sub:
// the rows of lane `sub` of lpm, one per 4 bits, 15 past the last.
static __constant__ unsigned long long kRowsOf[15] = {
    0xff876543210ull,                                                                // 1 lane
    0xf86204ull, 0xf7531ull,                                                         // 2 lanes
    0xfff04ull, 0xfff31ull, 0xfff75ull, 0xf862ull,                                   // 4 lanes
    0xff4ull, 0xff1ull, 0xff3ull, 0xff5ull, 0xff7ull, 0xf80ull, 0xf62ull, 0xffffull  // 8 lanes
};
__host__ __device__ constexpr int rows_per_lane(int lpm) { return lpm == 1 ? 9 : lpm == 2 ? 5 : lpm == 4 ? 3 : 2; }

// Hit words a lane collects before it evaluates them.
constexpr int kHitWords = 24;

// The molecules s_own, s_ocell of a staged region: forces to fx, fy, fz, sums to U, W, NP.
template <bool kSingle, bool kLjIsRc, int kWords>
__device__ __forceinline__ void pairs_staged(const Const& p, const Box& bx, const Smem& S, const int* s_own,
                                             const int* s_ocell, double* fx, double* fy, double* fz, int* status,
                                             double& U, double& W, double& NP, bool& same) {
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int ns = p.ns;
	const int n_own = s_own[kWarps];
	const int lpm = n_own > kThreads / 2 ? 1 : n_own > kThreads / 4 ? 2 : n_own > kThreads / 8 ? 4 : 8;
	const int lg = lpm == 1 ? 0 : lpm == 2 ? 1 : lpm == 4 ? 2 : 3;
	const int nrows = rows_per_lane(lpm);
	const int sub = lane & (lpm - 1);
	const unsigned long long rows = kRowsOf[lpm - 1 + sub];
	unsigned* const words = S.words + tid;
	const double eps24_d = S.pd[0], sig2_d = S.pd[KK], shift6_d = S.pd[2 * KK];
	for (int base0 = 0; base0 < n_own; base0 += kThreads >> lg) {
		const int t0 = base0 + ((warp * 32) >> lg);
		if (t0 >= n_own) break;   // this warp has no molecule (in this round or a later one)
		const int t = t0 + (lane >> lg);
		const bool act = t < n_own;
		int w = 0;
		if (act)
			while (w < kWarps - 1 && s_own[w + 1] <= t) w++;
		const int il0 = 1 + (w & 1), il1 = 1 + ((w >> 1) & 1), il2 = 1 + (w >> 2);
		const int oc = s_ocell[w];
		const int slot_i = S.cs[oc] + (act ? t - s_own[w] : 0);
		const int gi = S.gst[oc] + (act ? t - s_own[w] : 0);
		const double xi = S.img[3 * slot_i], yi = S.img[3 * slot_i + 1], zi = S.img[3 * slot_i + 2];
		const int ti = kSingle ? 0 : component(S, slot_i);
		Sums64 s64{0.0, 0.0, 0.0, 0.0, 0.0, 0, 0};
		int cnt = 0, hits = 0;   // words and hits collected

		// evaluates the collected words
		auto evaluate = [&]() {
			const int mx = __reduce_max_sync(kFull, hits);
			const unsigned* next = words;
			unsigned wd = 0u, nx = *next;   // this word's bits left; the next word
#pragma unroll 2
			for (int h = 0; h < mx; h++) {
				bool v = h < hits;
				if (v && (wd & 0xffffu) == 0u) {
					wd = nx;
					next += kThreads;   // (the word past the last one is never used)
				}
				nx = *next;
				const int bit = __ffs(wd) - 1;
				const int j = v ? (int) (wd >> 16) + ((bit & 7) << 1) + (bit >> 3) : slot_i;
				wd &= wd - 1u;
				v = v && j != slot_i;
				double e24 = 0.0, sg2 = sig2_d, sh6 = 0.0;
				if (!kSingle) {
					const int pk = ti * ns + component(S, j);
					e24 = S.pd[pk];
					sg2 = S.pd[KK + pk];
					sh6 = S.pd[2 * KK + pk];
				}
				lj64<kSingle, kLjIsRc>(__dsub_rn(xi, S.img[3 * j]), __dsub_rn(yi, S.img[3 * j + 1]),
				                       __dsub_rn(zi, S.img[3 * j + 2]), v, p.rc2, p.rclj2, e24, sg2, sh6, s64, same);
			}
			cnt = hits = 0;
		};

		// filter: packed half-precision test against rc^2 plus a margin covering its rounding
		const __half* hh = S.h + 8 * (slot_i >> 1) + (slot_i & 1);
		const __half2 xi2 = __half2half2(hh[0]), yi2 = __half2half2(hh[2]), zi2 = __half2half2(hh[4]);
		const __half2 rc2h = __float2half2_rn(bx.rc2_h);
		int q = 0, base = 0, left = 0;   // next row; this lane's next slot and what is left of its row
		unsigned first = 0u;             // the slot before an odd first slot belongs to another row
		for (bool more = true; more;) {
			// fill: blocks until a lane's words are full or the rows are done
			for (;;) {
				const int nblk = (__reduce_max_sync(kFull, left) + 15) >> 4;
				if (nblk <= 0) {
					if (q == nrows) {
						more = false;
						break;
					}
					const int r = (int) (rows >> (4 * q)) & 15;
					q++;
					left = 0;
					if (act && r < 9) {
						const int k0 = (il0 - 1) + 4 * (il1 + (r % 3) - 1) + 16 * (il2 + (r / 3) - 1);
						const int a = S.cs[k0];
						base = a & ~1;
						left = S.cs[k0 + 3] - base;
						first = (unsigned) (a & 1);
					}
					continue;
				}
				const int room = kWords - __reduce_max_sync(kFull, cnt);
				if (room == 0) break;
				const HalfPair* H = S.h16 + (base >> 1);
				for (int ib = min(nblk, room); ib > 0; ib--) {
					// bit k: slot base + 2k, bit 16 + k: slot base + 2k + 1
					unsigned m = 0u;
					if (left > 0) {
#pragma unroll
						for (int k = 0; k < 8; k++) {
							const HalfPair P = H[k];
							const __half2 dx = __hsub2(xi2, P.x), dy = __hsub2(yi2, P.y), dz = __hsub2(zi2, P.z);
							const __half2 d2 = __hfma2(dx, dx, __hfma2(dy, dy, __hmul2(dz, dz)));
							m |= __hlt2_mask(d2, rc2h) & ((1u << k) | (1u << (16 + k)));
						}
						// keep slots in [a, b)
						if (left < 16) m &= ((1u << ((left + 1) >> 1)) - 1u) | (((1u << (left >> 1)) - 1u) << 16);
						m &= ~first;
					}
					first = 0u;
					// even slots' bits in byte 0, odd slots' in byte 1, the block's first slot above
					words[cnt * kThreads] = __byte_perm(m, (unsigned) base, 0x5420);
					cnt += m != 0u ? 1 : 0;
					hits += __popc(m);
					base += 16;
					left -= 16;
					H += 8;
				}
			}
			evaluate();
		}
		if (kSingle) sums64_finish<kLjIsRc>(s64, eps24_d, shift6_d);
		U += s64.u;
		W += s64.w;
		NP += (double) s64.np;
		// the molecule's force: its lanes' sums in a fixed order
		for (int o = 1; o < lpm; o <<= 1) {
			s64.x += __shfl_xor_sync(kFull, s64.x, o);
			s64.y += __shfl_xor_sync(kFull, s64.y, o);
			s64.z += __shfl_xor_sync(kFull, s64.z, o);
		}
		if (act && sub == 0) {
			fx[gi] = s64.x;
			fy[gi] = s64.y;
			fz[gi] = s64.z;
			if (!(isfinite(s64.x) && isfinite(s64.y) && isfinite(s64.z))) atomicOr(status, kStatusNonFinite);
		}
	}
}

// A brick whose region exceeds the staged capacity: in the largest parts that fit, one after the other (kept out
// of the way of the ordinary bricks' code). Only a part of one own cell whose 27 cells do not fit gathers from
// global memory. 200,000 molecules at a density of 0.85, us per step: cutoff 3.7 (regions of 3,100; 2,500 fit)
// 1614 by gathering, 518 in parts; cutoff 4.4 3100 and 1311.
template <bool kSingle, bool kLjIsRc, int kWords>
__device__ __noinline__ void pairs_in_parts(const Const& p, const Box& bx, int brick, unsigned char* smem,
                                            const double* rx, const double* ry, const double* rz, const int32_t* cid,
                                            const int32_t* cstart, double* fx, double* fy, double* fz, int* s_own,
                                            int* s_ocell, int* status, double* sums) {
	const Smem S = views(smem, layout(p.s_cap, true, kWords));
	double U = 0.0, W = 0.0, NP = 0.0;
	bool same = false;
	int node = 2;
	do {
		const int level = part_level(node);
		int icell;
		if (own_cell(bx, brick, (node << (3 - level)) & 7, icell)) {   // (the first cell: the others lie beyond it)
			__syncthreads();   // before the next staging
			const bool staged = stage_rows(p, bx, brick, node, S, rx, ry, rz, cid, cstart, s_own, s_ocell);
			if (staged) {
				pairs_staged<kSingle, kLjIsRc, kWords>(p, bx, S, s_own, s_ocell, fx, fy, fz, status, U, W, NP, same);
			} else if (level < 3) {
				node *= 2;
				continue;
			} else {
				const int w = node & 7, gi0 = S.gst[s_ocell[w]];
				for (int t = threadIdx.x; t < s_own[kWarps]; t += kThreads) {
					const int gi = gi0 + t;
					PairSums s = gather_pairs<false>(gi, rx, ry, rz, cid, cstart, bx.g, S.pd, p.ns, p.rc2, p.rclj2, bx.coff);
					fx[gi] = s.F[0];
					fy[gi] = s.F[1];
					fz[gi] = s.F[2];
					U += s.U;
					W += s.W;
					NP += s.np;
					same |= s.same;
				}
			}
		}
		node++;
		while (!(node & 1)) node >>= 1;   // both halves done: the next of the level above
	} while (node > 1);
	if (same) atomicOr(status, kStatusSamePosition);
	sums[0] = U;
	sums[1] = W;
	sums[2] = NP;
}

// Forces on the molecules of brick `brick` (index within its box) of box `bx`; U, W and the pair
// count go to partials[slot]. The pair table must already be in shared memory (load_params).
// Ends with a CTA-wide barrier after which no thread reads the staged data.
//
// One evaluation, in FP64, serves both precision modes: what the FP32 form would save in the force law
// it spends on unpacking its split positions, here and in the staging (250,047 molecules at rc = 2.5:
// 121 us in FP64, 136 with an FP32 evaluation in the same structure).
//
// The brick's own molecules, of all its cells in one sequence, are spread over the CTA's lanes, lpm
// lanes per molecule: the largest of 1, 2, 4, 8 that the CTA's 256 lanes allow, so the warps that
// work are full whatever the cells hold (at rc = 2.5 a cell of a liquid holds 11-13 molecules: with
// one warp per cell, 60 % of every warp stood idle). A lane's filter walks its rows of three staged
// cells in blocks of 16 slots; lanes of other cells read other addresses in the same step. Hits stay
// a bit mask: one word per block (16 hit bits, the block's first slot above them), and the evaluation
// takes the bits of its words one by one, so the lanes of a warp wait for each other only at the end
// of a batch of words, not in every block.
//
// Bound by instruction issue (of 250,047 molecules at rc = 2.5: staging 25 %, filter 30 %, evaluation
// 45 %); three CTAs per SM. Measured, us per traversal, against one warp per cell with per-lane index
// lists and the reference's operation order: 250,047 molecules at rc = 2.5 121 (328), at rc = 3.0 190
// (381); 16,384 molecules of two species 26 (34).
template <bool kSingle, bool kLjIsRc, int kWords>
__device__ __forceinline__ void pairs(const Const& p, const Box& bx, int brick, int64_t slot, unsigned char* smem,
                                      const double* rx, const double* ry, const double* rz, const int32_t* cid,
                                      const int32_t* cstart, double* fx, double* fy, double* fz, double* partials,
                                      int* status) {
	const Smem S = views(smem, layout(p.s_cap, true, kWords));
	__shared__ int s_own[kWarps + 1], s_ocell[kWarps];
	double U = 0.0, W = 0.0, NP = 0.0;
	if (stage_rows(p, bx, brick, 1, S, rx, ry, rz, cid, cstart, s_own, s_ocell)) {
		bool same = false;
		pairs_staged<kSingle, kLjIsRc, kWords>(p, bx, S, s_own, s_ocell, fx, fy, fz, status, U, W, NP, same);
		if (same) atomicOr(status, kStatusSamePosition);
	} else {
		double sums[3];
		pairs_in_parts<kSingle, kLjIsRc, kWords>(p, bx, brick, smem, rx, ry, rz, cid, cstart, fx, fy, fz, s_own, s_ocell,
		                                         status, sums);
		U = sums[0];
		W = sums[1];
		NP = sums[2];
	}
	block_sum3_at(U, W, NP, partials, slot);
}

// Lanes per molecule for g molecules on one warp: the largest power of two with lpm * g <= 32.
__device__ __forceinline__ int lanes_per_molecule(int g) {
	int lpm = 1;
	while (lpm * 2 * g <= 32) lpm *= 2;
	return lpm;
}

// The traversal of a sparse brick by one warp, without CTA barriers. Its shared memory: the staged
// molecules' double images, component ids and staged cells, the cells' first slots and first molecules.
struct SparseTraverse {
	double img[3 * kSparseCap];
	int cs[65], gst[64];
	unsigned char comp[kSparseCap], cell[kSparseCap];
};

// Forces on the molecules of brick `brick` if it is sparse (see kSparseCap); false otherwise. Of the staged
// region each molecule tests all, lpm lanes per molecule: with a few molecules in all, a filter costs more
// than it saves. Candidates outside the 27 cells around the molecule's own are left out, as in pairs.
template <bool kSingle, bool kLjIsRc>
__device__ __forceinline__ bool pairs_sparse(const Const& p, const Box& bx, int brick, SparseTraverse& S,
                                             const PairParams* __restrict__ pp, const double* rx, const double* ry,
                                             const double* rz, const int32_t* cid, const int32_t* cstart, double* fx,
                                             double* fy, double* fz, double* partials, int* status) {
	const int lane = threadIdx.x & 31;
	const Grid& g = bx.g;
	const int bc[3] = {brick % bx.nb[0], (brick / bx.nb[0]) % bx.nb[1], brick / (bx.nb[0] * bx.nb[1])};
	// staged cells 2 lane and 2 lane + 1, as in stage_rows
	double t0, t1;
	const int gy = staged_coord(bx, 1, bc[1], (lane >> 1) & 3, t0, t1);
	const int gz = staged_coord(bx, 2, bc[2], lane >> 3, t0, t1);
	const int row0 = bx.coff + (gz * g.nc[1] + gy) * g.nc[0];
	const int ca = row0 + staged_coord(bx, 0, bc[0], 2 * (lane & 1), t0, t1);
	const int cb = row0 + staged_coord(bx, 0, bc[0], 2 * (lane & 1) + 1, t0, t1);
	const int sa = cstart[ca], ea = cstart[ca + 1], sb = cstart[cb], eb = cstart[cb + 1];
	const int na = max(0, ea - sa), nb = max(0, eb - sb);
	int inc = na + nb;
	for (int o = 1; o < 32; o <<= 1) {
		const int y = __shfl_up_sync(kFull, inc, o);
		if (lane >= o) inc += y;
	}
	const int slot_a = inc - (na + nb);
	const int total = __shfl_sync(kFull, inc, 31);
	// the own cells' counts in lanes 0..7, and their sum
	int ic = 0;
	const bool ok = lane < kWarps && own_cell(bx, brick, lane, ic);
	const int ia = __shfl_sync(kFull, na, ic >> 1), ib = __shfl_sync(kFull, nb, ic >> 1);
	const int c_own = ok ? ((ic & 1) ? ib : ia) : 0;
	const int n_own = __reduce_add_sync(kFull, c_own);
	if (total > kSparseCap || n_own > 32) return false;
	double U = 0.0, W = 0.0, NP = 0.0;
	if (n_own > 0) {
		S.cs[2 * lane] = slot_a;
		S.cs[2 * lane + 1] = slot_a + na;
		S.gst[2 * lane] = sa;
		S.gst[2 * lane + 1] = sb;
		if (lane == 31) S.cs[64] = total;
		__syncwarp();
		double sh_l = 0.0, k_l = 0.0;   // lane 4 d + l: the shift of staged coordinate l of dimension d
		if (lane < 12) staged_coord(bx, lane >> 2, bc[lane >> 2], lane & 3, sh_l, k_l);
		for (int t = lane; t < ((total + 31) & ~31); t += 32) {
			int c = 0;
			for (int step = 32; step; step >>= 1)
				if (S.cs[c + step] <= t) c += step;
			const double shx = __shfl_sync(kFull, sh_l, c & 3), shy = __shfl_sync(kFull, sh_l, 4 + ((c >> 2) & 3));
			const double shz = __shfl_sync(kFull, sh_l, 8 + (c >> 4));
			if (t < total) {
				const int gi = S.gst[c] + (t - S.cs[c]);
				S.img[3 * t] = __dadd_rn(rx[gi], shx);
				S.img[3 * t + 1] = __dadd_rn(ry[gi], shy);
				S.img[3 * t + 2] = __dadd_rn(rz[gi], shz);
				S.comp[t] = (unsigned char) cid[gi];
				S.cell[t] = (unsigned char) c;
			}
		}
		__syncwarp();
		int own = c_own;   // inclusive prefix of the own cells' counts in lanes 0..7
		for (int o = 1; o < kWarps; o <<= 1) {
			const int y = __shfl_up_sync(kFull, own, o);
			if (lane >= o) own += y;
		}
		const int lpm = lanes_per_molecule(n_own);
		const int sub = lane & (lpm - 1), t = lane / lpm;
		const bool act = t < n_own;
		int w = 0;
		for (int k = 0; k < kWarps - 1; k++) w += t >= __shfl_sync(kFull, own, k) ? 1 : 0;
		const int before = w > 0 ? w - 1 : 0;
		const int prev = __shfl_sync(kFull, own, before);
		const int oc = __shfl_sync(kFull, ic, w);
		const int e = act ? t - (w > 0 ? prev : 0) : 0;
		const int slot_i = min(S.cs[oc] + e, max(0, total - 1)), gi = S.gst[oc] + e;
		const double xi = S.img[3 * slot_i], yi = S.img[3 * slot_i + 1], zi = S.img[3 * slot_i + 2];
		const int ti = kSingle ? 0 : S.comp[slot_i];
		Sums64 s64{0.0, 0.0, 0.0, 0.0, 0.0, 0, 0};
		bool same = false;
		for (int j0 = 0; j0 < total; j0 += lpm) {
			const int j = min(j0 + sub, total - 1);
			const int cj = S.cell[j];
			const bool near = abs((cj & 3) - (oc & 3)) <= 1 && abs(((cj >> 2) & 3) - ((oc >> 2) & 3)) <= 1 &&
			                  abs((cj >> 4) - (oc >> 4)) <= 1;
			const bool v = act && j0 + sub < total && j != slot_i && near;
			const int pk = kSingle ? 0 : ti * p.ns + S.comp[j];
			lj64<kSingle, kLjIsRc>(__dsub_rn(xi, S.img[3 * j]), __dsub_rn(yi, S.img[3 * j + 1]),
			                       __dsub_rn(zi, S.img[3 * j + 2]), v, p.rc2, p.rclj2, pp->eps24[pk], pp->sig2[pk],
			                       pp->shift6[pk], s64, same);
		}
		if (kSingle) sums64_finish<kLjIsRc>(s64, pp->eps24[0], pp->shift6[0]);
		U = s64.u;
		W = s64.w;
		NP = (double) s64.np;
		for (int o = 1; o < lpm; o <<= 1) {
			s64.x += __shfl_xor_sync(kFull, s64.x, o);
			s64.y += __shfl_xor_sync(kFull, s64.y, o);
			s64.z += __shfl_xor_sync(kFull, s64.z, o);
		}
		if (act && sub == 0) {
			fx[gi] = s64.x;
			fy[gi] = s64.y;
			fz[gi] = s64.z;
			if (!(isfinite(s64.x) && isfinite(s64.y) && isfinite(s64.z))) atomicOr(status, kStatusNonFinite);
		}
		if (same) atomicOr(status, kStatusSamePosition);
		U = warp_sum(U);
		W = warp_sum(W);
		NP = warp_sum(NP);
		__syncwarp();   // the next brick of this warp stages into the same memory
	}
	if (lane == 0) {
		partials[4 * (int64_t) brick + 0] = U;
		partials[4 * (int64_t) brick + 1] = W;
		partials[4 * (int64_t) brick + 2] = NP;
		partials[4 * (int64_t) brick + 3] = 0.0;
	}
	return true;
}

// Entries of each lane's write-combining ring in build_lists: up to 7 unwritten entries plus the
// 32 that one block of candidates can add; a power of two for the index wrap.
constexpr int kBuildRing = 64;

// Shared-memory bytes of build_lists for a staged capacity s_cap.
__host__ __device__ inline size_t build_bytes(int s_cap) {
	return align16(sizeof(HalfPair) * (s_cap / 2 + 20)) + align16(sizeof(int) * 65) + 2 * align16(sizeof(int) * 64) +
	       align16(sizeof(double) * 3 * 64) + sizeof(unsigned short) * kBuildRing * kThreads;
}

// Bits [lo, hi) of a 16-bit field (0 <= lo, hi <= 16).
__device__ __forceinline__ unsigned range16(int lo, int hi) {
	const unsigned up = hi >= 16 ? 0xffffu : ((1u << hi) - 1u);
	return lo >= 16 ? 0u : up & ~((1u << lo) - 1u);
}

// Verlet-skin build for brick `brick`: stages the half-precision copy of the 4x4x4 cells around it
// (the same slots as stage() gives them) and writes to each own molecule's list every candidate
// that the packed filter finds within the list radius (bx.rc2_h holds rc + skin plus the rounding
// margin), with the positions of the build. No forces: list_pairs evaluates the lists.
__device__ __forceinline__ void build_lists(const Box& bx, int brick, int s_cap, unsigned char* smem,
                                            const double* rx, const double* ry, const double* rz,
                                            const int32_t* cstart, Lists lists, int64_t kind_slot) {
	HalfPair* s_h16 = reinterpret_cast<HalfPair*>(smem);
	__half* s_h = reinterpret_cast<__half*>(smem);
	size_t o = align16(sizeof(HalfPair) * (s_cap / 2 + 20));
	int* s_cs = reinterpret_cast<int*>(smem + o);
	o += align16(sizeof(int) * 65);
	int* s_cnt = reinterpret_cast<int*>(smem + o);
	o += align16(sizeof(int) * 64);
	int* s_gst = reinterpret_cast<int*>(smem + o);
	o += align16(sizeof(int) * 64);
	double* s_ck = reinterpret_cast<double*>(smem + o);
	o += align16(sizeof(double) * 3 * 64);
	const Grid& g = bx.g;
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	unsigned short* ring = reinterpret_cast<unsigned short*>(smem + o) + kBuildRing * tid;
	const int bc[3] = {brick % bx.nb[0], (brick / bx.nb[0]) % bx.nb[1], brick / (bx.nb[0] * bx.nb[1])};
	if (tid < 64) {
		const int l[3] = {tid & 3, (tid >> 2) & 3, tid >> 4};
		int gc[3];
		for (int d = 0; d < 3; d++) {
			int gcd = 2 * bc[d] - 1 + l[d];
			double sh = 0.0;
			if (gcd < 0) {
				gcd += g.nc[d];
				sh = -g.L[d];
			} else if (gcd >= g.nc[d]) {
				gcd -= g.nc[d];
				sh = g.L[d];
			}
			gc[d] = gcd;
			const double cbr = (2 * bc[d] + 1) * g.cell_length[d];
			s_ck[3 * tid + d] = (sh - cbr) + (double) bx.frame_c[d];
		}
		const int gcell = bx.coff + (gc[2] * g.nc[1] + gc[1]) * g.nc[0] + gc[0];
		const int st = cstart[gcell];
		s_gst[tid] = st;
		s_cnt[tid] = max(0, cstart[gcell + 1] - st);
	}
	__syncthreads();
	if (warp == 0) {
		const int a = s_cnt[2 * lane], b = s_cnt[2 * lane + 1];
		int inc = a + b;
		for (int of = 1; of < 32; of <<= 1) {
			const int y = __shfl_up_sync(kFull, inc, of);
			if (lane >= of) inc += y;
		}
		const int excl = inc - (a + b);
		s_cs[2 * lane] = excl;
		s_cs[2 * lane + 1] = excl + a;
		if (lane == 31) s_cs[64] = inc;
	}
	__syncthreads();
	const bool staged = s_cs[64] <= s_cap;
	if (staged) {
		for (int c = warp; c < 64; c += kWarps) {
			const int st = s_gst[c], cnt = s_cnt[c], base = s_cs[c];
			const double kx = s_ck[3 * c], ky = s_ck[3 * c + 1], kz = s_ck[3 * c + 2];
			for (int e = lane; e < cnt; e += 32) {
				const int gi = st + e;
				const float X = __double2float_rn(__dadd_rn(rx[gi], kx));
				const float Y = __double2float_rn(__dadd_rn(ry[gi], ky));
				const float Z = __double2float_rn(__dadd_rn(rz[gi], kz));
				const int slot_s = base + e;
				__half* hp = s_h + 8 * (slot_s >> 1) + (slot_s & 1);
				hp[0] = __float2half_rn(X - bx.frame_c[0]);
				hp[2] = __float2half_rn(Y - bx.frame_c[1]);
				hp[4] = __float2half_rn(Z - bx.frame_c[2]);
			}
		}
	}
	__syncthreads();
	int icell;
	if (own_cell(bx, brick, warp, icell)) {
		const int st = s_gst[icell], ncell = s_cnt[icell], i0 = s_cs[icell];
		const int il[3] = {1 + (warp & 1), 1 + ((warp >> 1) & 1), 1 + (warp >> 2)};
		if (!staged) {
			for (int e = lane; e < ncell; e += 32) {
				lists.count[st + e] = kListOverflow;
				lists.rx_ref[st + e] = rx[st + e];
				lists.ry_ref[st + e] = ry[st + e];
				lists.rz_ref[st + e] = rz[st + e];
			}
		} else {
			const __half2 rc2h = __float2half2_rn(bx.rc2_h);
			// each lane's entries go through its ring in shared memory and leave it in blocks of
			// 8 (one 16-byte store each); the rotation by lane spreads the ring writes over banks
			const int rot = 8 * (lane & 7);
			for (int b0 = 0; b0 < ncell; b0 += 32) {
				const bool act = b0 + lane < ncell;
				const int slot_i = i0 + (act ? b0 + lane : 0);
				const int gi = st + (slot_i - i0);
				const __half* hi = s_h + 8 * (slot_i >> 1) + (slot_i & 1);
				const __half2 xi2 = act ? __half2half2(hi[0]) : __float2half2_rn(60000.f);
				const __half2 yi2 = __half2half2(hi[2]);
				const __half2 zi2 = __half2half2(hi[4]);
				uint4* dst = reinterpret_cast<uint4*>(lists.nbr) + gi;
				int cnt = 0, done = 0;   // entries found; entries written (a multiple of 8)
				for (int r = 0; r < 9; r++) {
					const int ky = il[1] + (r % 3) - 1, kz = il[2] + (r / 3) - 1;
					const int k0 = (il[0] - 1) + 4 * ky + 16 * kz;
					const int a = s_cs[k0], b = s_cs[k0 + 3];
					for (int base = a & ~1; base < b; base += 32) {
						// bit k: slot base + 2k, bit 16 + k: slot base + 2k + 1
						unsigned mask = 0u;
#pragma unroll
						for (int k = 0; k < 16; k++) {
							const HalfPair H = s_h16[(base >> 1) + k];
							const __half2 dx = __hsub2(xi2, H.x), dy = __hsub2(yi2, H.y), dz = __hsub2(zi2, H.z);
							const __half2 d2 = __hfma2(dx, dx, __hfma2(dy, dy, __hmul2(dz, dz)));
							mask |= __hlt2_mask(d2, rc2h) & ((1u << k) | (1u << (16 + k)));
						}
						// keep slots in [a, b) and drop i itself
						const int lo = a - base, hi_b = b - base;
						mask &= range16(max(0, (lo + 1) >> 1), min(16, (hi_b + 1) >> 1)) |
						        (range16(max(0, lo >> 1), min(16, hi_b >> 1)) << 16);
						const int self = slot_i - base;
						if (self >= 0 && self < 32) mask &= ~(1u << ((self & 1) * 16 + (self >> 1)));
						if (!act) mask = 0u;
						while (mask) {
							const int bit = __ffs(mask) - 1;
							mask &= mask - 1u;
							ring[(cnt + rot) & (kBuildRing - 1)] = (unsigned short) (base + 2 * (bit & 15) + (bit >> 4));
							cnt++;
						}
						for (; done + 8 <= cnt; done += 8)
							if (done < lists.cap)
								dst[(int64_t) (done >> 3) * lists.n] =
								    *reinterpret_cast<const uint4*>(ring + ((done + rot) & (kBuildRing - 1)));
					}
				}
				if (act) {
					// the last block of 8, padded with the list kernel's sentinel slot
					if (cnt > done) {
						for (int k = cnt; k < done + 8; k++)
							ring[(k + rot) & (kBuildRing - 1)] = (unsigned short) lists.sentinel;
						if (done < lists.cap)
							dst[(int64_t) (done >> 3) * lists.n] =
							    *reinterpret_cast<const uint4*>(ring + ((done + rot) & (kBuildRing - 1)));
					}
					lists.count[gi] = cnt <= lists.cap ? (unsigned short) cnt : kListOverflow;
					lists.rx_ref[gi] = rx[gi];
					lists.ry_ref[gi] = ry[gi];
					lists.rz_ref[gi] = rz[gi];
				}
			}
		}
	}
	if (tid == 0) {
		int n_own = 0;
		for (int w = 0; w < kWarps; w++) {
			int ic;
			if (own_cell(bx, brick, w, ic)) n_own += s_cnt[ic];
		}
		const bool sparse = s_cs[64] <= kSparseCap && n_own <= 32;
		lists.kind[kind_slot] = sparse ? 1 : 0;
		if (lists.counts) {
			const unsigned at = atomicAdd(lists.counts + (sparse ? 0 : 1), 1u);
			lists.blist[(sparse ? lists.nbricks : 0) + (int) at] = (int32_t) kind_slot;
		}
		if (brick == 0) atomicAdd(lists.builds, 1ull);
	}
}

// What the list kernels do with a molecule's force once it is summed. Mode 0 stores it. Modes 1
// and 2 apply the closing kick of the step, v += (dt/2m) F, and add m v^2 to the step's sum
// (Molecule::upd_postF, molecules/Molecule.cpp:193-205); mode 2 (the last step of a run) stores F
// and v, mode 1 goes on with the opening kick and drift of the next step, v = 1*v + (dt/2m) F,
// r' = r + dt v (Molecule::upd_preF with vcorr = 1, Molecule.cpp:128-135), writes r' to the other
// position buffer (other bricks still stage r) and flags a rebuild with `id` when r' is farther than
// skin/2 from the position of the last build. Same operations and roundings as the Leapfrog kernels.
// The CTA's largest squared drift of a list kernel with pruned lists (float bits; set to 0 before the
// first finish, flushed by drift_flush).
__device__ __forceinline__ unsigned& drift_slot() {
	__shared__ unsigned s_drift;
	return s_drift;
}

struct Kick {
	int mode;
	int id;
	double dt;
	double half2;                 // (skin/2)^2
	double post[kMaxSpecies];     // (0.5 dt) / m of the closing kick
	double pre[kMaxSpecies];      // (0.5 dt) / m of the opening kick
	double mass[kMaxSpecies];
	double *vx, *vy, *vz;
	double *ox, *oy, *oz;         // positions after the drift (mode 1)
	int* flag;
	unsigned* dmax;               // mode 1 with pruned lists: the largest squared drift, as float bits
};

__device__ __forceinline__ double finish(const Kick& k, int64_t gi, double Fx, double Fy, double Fz, const double* rx,
                                         const double* ry, const double* rz, const int32_t* cid, const Lists& lists,
                                         double* fx, double* fy, double* fz, int* status) {
	if (!(Fx == Fx && Fy == Fy && Fz == Fz) || isinf(Fx) || isinf(Fy) || isinf(Fz)) atomicOr(status, kStatusNonFinite);
	if (k.mode != 1) {
		fx[gi] = Fx;
		fy[gi] = Fy;
		fz[gi] = Fz;
	}
	if (k.mode == 0) return 0.0;
	const int t = cid[gi];
	const double a = k.post[t];
	const double vx = __dadd_rn(k.vx[gi], __dmul_rn(a, Fx));
	const double vy = __dadd_rn(k.vy[gi], __dmul_rn(a, Fy));
	const double vz = __dadd_rn(k.vz[gi], __dmul_rn(a, Fz));
	const double v2 = __dadd_rn(__dadd_rn(__dmul_rn(vx, vx), __dmul_rn(vy, vy)), __dmul_rn(vz, vz));
	if (!(v2 == v2) || isinf(v2)) atomicOr(status, kStatusNonFinite);
	const double mv2 = __dmul_rn(k.mass[t], v2);
	if (k.mode == 2) {
		k.vx[gi] = vx;
		k.vy[gi] = vy;
		k.vz[gi] = vz;
		return mv2;
	}
	const double b = k.pre[t];
	const double wx = __dadd_rn(__dmul_rn(1.0, vx), __dmul_rn(b, Fx));
	const double wy = __dadd_rn(__dmul_rn(1.0, vy), __dmul_rn(b, Fy));
	const double wz = __dadd_rn(__dmul_rn(1.0, vz), __dmul_rn(b, Fz));
	const double x0 = rx[gi], y0 = ry[gi], z0 = rz[gi];
	const double x = __dadd_rn(x0, __dmul_rn(k.dt, wx));
	const double y = __dadd_rn(y0, __dmul_rn(k.dt, wy));
	const double z = __dadd_rn(z0, __dmul_rn(k.dt, wz));
	if (k.dmax) {
		// this drift's length squared, rounded up (the bits of a non-negative float order as it does)
		const double sx = x - x0, sy = y - y0, sz = z - z0;
		atomicMax(&drift_slot(), __float_as_uint(__double2float_ru(sx * sx + sy * sy + sz * sz)));
	}
	k.vx[gi] = wx;
	k.vy[gi] = wy;
	k.vz[gi] = wz;
	k.ox[gi] = x;
	k.oy[gi] = y;
	k.oz[gi] = z;
	const double dx = x - lists.rx_ref[gi], dy = y - lists.ry_ref[gi], dz = z - lists.rz_ref[gi];
	if (!(dx * dx + dy * dy + dz * dz <= k.half2)) *k.flag = k.id;
	return mv2;
}

// The CTA's largest squared drift into *dmax (thread 0, after a CTA barrier that follows every
// finish; the atomic is skipped when the value there is already as large).
__device__ __forceinline__ void drift_flush(unsigned* dmax) {
	if (dmax && threadIdx.x == 0 && drift_slot() > __ldcg(dmax)) atomicMax(dmax, drift_slot());
}

#ifndef MDGPU_LIST_ACC
#define MDGPU_LIST_ACC 1
#endif
// Independent FP32 partial sums per lane in list_chunk (entry u of a block of 8 goes to u % kListAcc).
constexpr int kListAcc = MDGPU_LIST_ACC;
static_assert(kListAcc == 1 || kListAcc == 2 || kListAcc == 4, "1, 2 or 4 partial sums");

// Word k of a block of 8 list entries (register selection; k need not be a constant).
__device__ __forceinline__ unsigned list_word(const uint4& v, int k) {
	return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w;
}

// The partial sums in a fixed order, in FP64.
__device__ __forceinline__ double acc_sum(const float* a) {
	if (kListAcc == 4) return ((double) a[0] + (double) a[1]) + ((double) a[2] + (double) a[3]);
	if (kListAcc == 2) return (double) a[0] + (double) a[1 % kListAcc];
	return (double) a[0];
}

// Where the evaluation of a prune step writes the inner lists: the entries of each molecule's build
// list whose squared staged distance is below rp2f, in list order, in the layout of Lists::nbr.
struct PruneOut {
	unsigned short* nbr;
	unsigned short* count;
	float rp2f;
};

// Entries of each thread's ring in shared memory in a prune step: up to 7 unwritten entries plus the
// 8 of one block; entry k of thread t at k * kThreads + t (a warp's stores of one entry each fall in
// 16 banks). The prune variant's shared memory is the layout's plus kPruneRingBytes.
constexpr int kPruneRing = 16;
constexpr size_t kPruneRingBytes = sizeof(unsigned short) * kPruneRing * kThreads;

// A warp evaluates the lists of the brick's own molecules t0 .. t1-1 (in the order of the own cells
// own[0..8] / ocell[0..7]), lpm lanes per molecule (a power of two, (t1 - t0) * lpm <= 32): lane
// sub = lane % lpm takes the blocks sub, sub + lpm, ... of its molecule's list, the lanes' forces
// are summed by a fixed butterfly and the molecule is finished by its first lane; U, W, the pair
// count and the same-position flag are accumulated into the caller's sums. kPrune (a prune step): the
// entries also pass the prune test into the molecule's inner list (po).
template <bool kFP64, bool kSingle, bool kLjIsRc, bool kClampJ = false, bool kPrune = false>
__device__ __forceinline__ void list_chunk(const Const& p, const Box& bx, const Smem& S, const int* s_own,
                                           const int* s_ocell, int t0, int t1, int lpm, const double* rx,
                                           const double* ry,
                                           const double* rz, const int32_t* cid, const int32_t* cstart, double* fx,
                                           double* fy, double* fz, int* status, const Lists& lists, const Kick& kick,
                                           double& U, double& W, double& NP, double& MV, bool& same,
                                           const PruneOut& po = PruneOut{}, unsigned short* ring = nullptr) {
	const int lane = threadIdx.x & 31;
	const int ns = p.ns;
	const float eps24_1 = S.pf[0], sig2_1 = S.pf[KK], shift6_1 = S.pf[2 * KK];
	const int sub = lane & (lpm - 1);
	const int t = t0 + lane / lpm;
	const bool act = t < t1;
	int w = 0;
	if (act)
		while (w < 7 && s_own[w + 1] <= t) w++;
	const int slot_i = act ? S.cs[s_ocell[w]] + (t - s_own[w]) : 0;
	float4 hi_i = make_float4(0.f, 0.f, 0.f, 0.f);
	double xi = 0, yi = 0, zi = 0;
	if (kFP64) {
		xi = S.img[3 * slot_i];
		yi = S.img[3 * slot_i + 1];
		zi = S.img[3 * slot_i + 2];
	}
	if (!kFP64) hi_i = S.hi[slot_i];
	const int ti = kSingle ? 0 : kFP64 ? component(S, slot_i) : unpack_cid(__float_as_uint(hi_i.w));
	const int gi = act ? S.gst[s_ocell[w]] + (t - s_own[w]) : S.gst[s_ocell[0]];
	int cnt = act ? (int) lists.count[gi] : 0;
	const bool ovf = cnt == kListOverflow;
	if (ovf && sub == 0) {
		// the list overflowed at the build: gather this molecule from global memory
		PairSums s = gather_pairs<!kFP64>(gi, rx, ry, rz, cid, cstart, bx.g, S.pd, ns, p.rc2, p.rclj2, bx.coff);
		MV += finish(kick, gi, s.F[0], s.F[1], s.F[2], rx, ry, rz, cid, lists, fx, fy, fz, status);
		U += s.U;
		W += s.W;
		NP += s.np;
		same |= s.same;
	}
	if (ovf) cnt = 0;
	const int mx = __reduce_max_sync(kFull, cnt);
	// blocks of 8 entries, one 16-byte load each, the next block loaded while this one is used;
	// this lane's blocks are sub, sub + lpm, ... (nk of them at most, the same bound in every lane)
	const uint4* my8 = reinterpret_cast<const uint4*>(lists.nbr) + gi;
	const int nb8 = (mx + 7) >> 3;
	const int nk = (nb8 + lpm - 1) / lpm;
	double Fx = 0.0, Fy = 0.0, Fz = 0.0;
	int anp = 0;
	// a prune step: kept entries go through this thread's ring and leave it in blocks of 8, the
	// lane's k-th block at inner block sub + k lpm (the blocks it would read at this split)
	int kept = 0, done = 0;
	uint4* const pdst = kPrune ? reinterpret_cast<uint4*>(po.nbr) + gi : nullptr;
	// branch-free: every entry is stored at the next free place, which only a kept entry takes
	// (at most 15 entries are unwritten, so the next free place is never one of them)
	auto keep = [&](unsigned e, bool k) {
		ring[(kept & (kPruneRing - 1)) * kThreads] = (unsigned short) e;
		kept += k ? 1 : 0;
	};
	auto flush = [&]() {
		unsigned v[4];
#pragma unroll
		for (int q = 0; q < 4; q++)
			v[q] = (unsigned) ring[((done + 2 * q) & (kPruneRing - 1)) * kThreads] |
			       ((unsigned) ring[((done + 2 * q + 1) & (kPruneRing - 1)) * kThreads] << 16);
		pdst[(int64_t) (sub + (done >> 3) * lpm) * lists.n] = make_uint4(v[0], v[1], v[2], v[3]);
		done += 8;
	};
	uint4 nxt = sub < nb8 ? my8[(int64_t) sub * lists.n] : make_uint4(0u, 0u, 0u, 0u);
	if (kFP64) {
		Sums64 s64{0.0, 0.0, 0.0, 0.0, 0.0, 0, 0};
		for (int k = 0; k < nk; k++) {
			const int b = sub + k * lpm;
			const uint4 cur = nxt;
			if (b + lpm < nb8) nxt = my8[(int64_t) (b + lpm) * lists.n];
			const unsigned e[4] = {cur.x, cur.y, cur.z, cur.w};
#pragma unroll
			for (int u = 0; u < 8; u++) {
				const int kk = 8 * b + u;
				const unsigned raw = (e[u >> 1] >> (16 * (u & 1))) & 0xffffu;
				// (a pruned list may hold sentinel slots before its end); what is no entry looks at the
				// molecule itself: nothing was staged to the sentinel's slot, whose bytes may be a NaN
				const bool v = kk < cnt && raw < (unsigned) p.s_cap;
				const int j = v ? (int) raw : slot_i;
				double e24 = 0.0, sg2 = S.pd[KK], sh6 = 0.0;
				if (!kSingle) {
					const int pk = ti * ns + component(S, j);
					e24 = S.pd[pk];
					sg2 = S.pd[KK + pk];
					sh6 = S.pd[2 * KK + pk];
				}
				const double dd =
				    lj64<kSingle, kLjIsRc>(__dsub_rn(xi, S.img[3 * j]), __dsub_rn(yi, S.img[3 * j + 1]),
				                           __dsub_rn(zi, S.img[3 * j + 2]), v, p.rc2, p.rclj2, e24, sg2, sh6, s64, same);
				if (kPrune) keep((unsigned) j, v && dd < (double) po.rp2f);
			}
			if (kPrune && kept - done >= 8) flush();
		}
		if (kSingle) sums64_finish<kLjIsRc>(s64, S.pd[0], S.pd[2 * KK]);
		Fx = s64.x;
		Fy = s64.y;
		Fz = s64.z;
		U += s64.u;
		W += s64.w;
		anp = s64.np;
	} else {
		// FP32, branch-free. Per coordinate e = fma(m_i - m_j, step, hi_i - hi_j) with m = 2^23 +
		// the 9-bit lo field (exact integer difference, one rounding). Single-species runs sum
		// fac/eps24, s6 (s6 - 1) and s6 (2 s6 - 1) and apply eps24 and shift6 per molecule.
		const unsigned wi = __float_as_uint(hi_i.w);
		const float mix = __uint_as_float(0x4B000000u | (wi & 511u));
		const float miy = __uint_as_float(0x4B000000u | ((wi >> 9) & 511u));
		const float miz = __uint_as_float(0x4B000000u | ((wi >> 18) & 511u));
		const int nblk = (cnt + 7) >> 3;
		const unsigned sent2 = (unsigned) p.s_cap | ((unsigned) p.s_cap << 16);
		float ax[kListAcc], ay[kListAcc], az[kListAcc], au[kListAcc], aw[kListAcc];
#pragma unroll
		for (int a = 0; a < kListAcc; a++) ax[a] = ay[a] = az[a] = au[a] = aw[a] = 0.f;
		int nlj = 0;   // pairs inside the LJ cutoff (shift6 terms)
		// one pair in FP32 with the given cutoff decision; sign +1 adds it, -1 removes it
		auto pair32 = [&](int j, bool in, float sign) {
			const float4 hj = S.hi[j];
			const unsigned wj = __float_as_uint(hj.w);
			const float e0 = fmaf(mix - __uint_as_float(0x4B000000u | (wj & 511u)), bx.lo_step[0], hi_i.x - hj.x);
			const float e1 = fmaf(miy - __uint_as_float(0x4B000000u | ((wj >> 9) & 511u)), bx.lo_step[1], hi_i.y - hj.y);
			const float e2 = fmaf(miz - __uint_as_float(0x4B000000u | ((wj >> 18) & 511u)), bx.lo_step[2], hi_i.z - hj.z);
			const float d2f = fmaf(e0, e0, fmaf(e1, e1, e2 * e2));
			const bool lj_in = kLjIsRc ? in : (in && d2f < p.rclj2f);
			anp += in ? (int) sign : 0;
			if (!kLjIsRc) nlj += lj_in ? (int) sign : 0;
			const float inv = lj_in ? rcp_approx(d2f) : 0.f;
			float eps24 = 1.f, sig2 = sig2_1, shift6 = 0.f;
			if (!kSingle) {
				const int pk = ti * ns + unpack_cid(wj);
				eps24 = S.pf[pk];
				sig2 = S.pf[KK + pk];
				shift6 = S.pf[2 * KK + pk];
			}
			const float s2 = sig2 * inv;
			const float s6 = s2 * s2 * s2;
			const float r = eps24 * (s6 * fmaf(2.f, s6, -1.f));
			const float fac = sign * r * inv;
			ax[0] = fmaf(fac, e0, ax[0]);
			ay[0] = fmaf(fac, e1, ay[0]);
			az[0] = fmaf(fac, e2, az[0]);
			au[0] += sign * (fmaf(eps24 * s6, s6 - 1.f, 0.f) + (lj_in ? shift6 : 0.f));
			aw[0] += sign * r;
		};
		for (int k = 0; k < nk; k++) {
			const int b = sub + k * lpm;
			uint4 cur = nxt;
			if (b + lpm < nb8) nxt = my8[(int64_t) (b + lpm) * lists.n];
			if (b >= nblk) cur = make_uint4(sent2, sent2, sent2, sent2);
			bool amb = false;
#pragma unroll
			for (int u = 0; u < 8; u++) {
				int j = (int) ((list_word(cur, u >> 1) >> (16 * (u & 1))) & 0xffffu);
				if (kClampJ) j = min(j, p.s_cap);   // a padding entry is the caller's sentinel slot
				const float4 hj = S.hi[j];
				const unsigned wj = __float_as_uint(hj.w);
				const float h0 = hi_i.x - hj.x, h1 = hi_i.y - hj.y, h2 = hi_i.z - hj.z;  // exact
				const float g0 = mix - __uint_as_float(0x4B000000u | (wj & 511u));
				const float g1 = miy - __uint_as_float(0x4B000000u | ((wj >> 9) & 511u));
				const float g2 = miz - __uint_as_float(0x4B000000u | ((wj >> 18) & 511u));
				const float e0 = fmaf(g0, bx.lo_step[0], h0);
				const float e1 = fmaf(g1, bx.lo_step[1], h1);
				const float e2 = fmaf(g2, bx.lo_step[2], h2);
				const float d2f = fmaf(e0, e0, fmaf(e1, e1, e2 * e2));
				const bool in = d2f < p.rc2f;
				if (kPrune) keep((unsigned) j, d2f < po.rp2f);   // padding is far: never kept
				// within a few ulp of rc: decided after the block as the FP64 computation does
				amb |= fabsf(d2f - p.rc2f) <= p.band;
				anp += in ? 1 : 0;
				const bool lj_in = kLjIsRc ? in : (in && d2f < p.rclj2f);
				if (!kLjIsRc) nlj += lj_in ? 1 : 0;
				const float inv = lj_in ? rcp_approx(d2f) : 0.f;
				const int a = u % kListAcc;
				if (kSingle) {
					const float s2 = sig2_1 * inv;
					const float s6 = s2 * s2 * s2;
					const float r = s6 * fmaf(2.f, s6, -1.f);
					const float facp = r * inv;
					ax[a] = fmaf(facp, e0, ax[a]);
					ay[a] = fmaf(facp, e1, ay[a]);
					az[a] = fmaf(facp, e2, az[a]);
					au[a] = fmaf(s6, s6 - 1.f, au[a]);
					aw[a] += r;
				} else {
					const int pk = ti * ns + unpack_cid(wj);
					const float eps24 = S.pf[pk], sig2 = S.pf[KK + pk], shift6 = S.pf[2 * KK + pk];
					const float s2 = sig2 * inv;
					const float s6 = s2 * s2 * s2;
					const float r = eps24 * (s6 * fmaf(2.f, s6, -1.f));
					const float fac = r * inv;
					ax[a] = fmaf(fac, e0, ax[a]);
					ay[a] = fmaf(fac, e1, ay[a]);
					az[a] = fmaf(fac, e2, az[a]);
					au[a] = fmaf(eps24 * s6, s6 - 1.f, au[a]) + (lj_in ? shift6 : 0.f);
					aw[a] += r;
				}
			}
			if (kPrune && kept - done >= 8) flush();
			if (__any_sync(kFull, amb)) {
				// rare: pairs within a few ulp of rc whose FP64 decision differs from the FP32 one
#pragma unroll 1
				for (int u = 0; u < 8; u++) {
					int j = (int) ((list_word(cur, u >> 1) >> (16 * (u & 1))) & 0xffffu);
					if (kClampJ) j = min(j, p.s_cap);
					const float4 hj = S.hi[j];
					const unsigned wj = __float_as_uint(hj.w);
					const float e0 = fmaf(mix - __uint_as_float(0x4B000000u | (wj & 511u)), bx.lo_step[0], hi_i.x - hj.x);
					const float e1 = fmaf(miy - __uint_as_float(0x4B000000u | ((wj >> 9) & 511u)), bx.lo_step[1], hi_i.y - hj.y);
					const float e2 = fmaf(miz - __uint_as_float(0x4B000000u | ((wj >> 18) & 511u)), bx.lo_step[2], hi_i.z - hj.z);
					const float d2f = fmaf(e0, e0, fmaf(e1, e1, e2 * e2));
					if (fabsf(d2f - p.rc2f) <= p.band) {
						const bool in_f = d2f < p.rc2f;
						const bool in_d = exact_cut(S, p.rc2, j, gi, rx, ry, rz);
						if (in_f != in_d) pair32(j, true, in_d ? 1.f : -1.f);
					}
				}
			}
			if ((k & 7) == 7 || k + 1 == nk) {
				// fold the FP32 partial sums of up to 64 entries into the FP64 accumulators
				const double sc = kSingle ? (double) eps24_1 : 1.0;
				Fx += sc * acc_sum(ax);
				Fy += sc * acc_sum(ay);
				Fz += sc * acc_sum(az);
				U += sc * acc_sum(au);
				W += sc * acc_sum(aw);
#pragma unroll
				for (int a = 0; a < kListAcc; a++) ax[a] = ay[a] = az[a] = au[a] = aw[a] = 0.f;
			}
		}
		if (kSingle) U += (double) shift6_1 * (double) (kLjIsRc ? anp : nlj);
		if (!(Fx == Fx && Fy == Fy && Fz == Fz) && act && !ovf) {
			// a zero distance gives 0 * inf: report it as the reference does (same position)
			for (int k = 0; k < cnt; k++) {
				const int j = lists.nbr[(((int64_t) (k >> 3) * lists.n + gi) << 3) + (k & 7)];
				const float4 hj = S.hi[min(j, p.s_cap)];
				const unsigned pos_bits = (1u << 27) - 1u;   // the lo fields, not the component id
				if (hj.x == hi_i.x && hj.y == hi_i.y && hj.z == hi_i.z &&
				    ((__float_as_uint(hj.w) ^ wi) & pos_bits) == 0u && j != slot_i)
					same = true;
			}
		}
	}
	NP += (double) anp;
	if (kPrune) {
		// each lane's last block padded with the sentinel slot; the list ends after the molecule's
		// last written block, and a lane's blocks below that end which it did not fill hold
		// sentinels only (the evaluation reads them as far away)
		if (kept > done) {
			for (int k = kept; k < done + 8; k++) ring[(k & (kPruneRing - 1)) * kThreads] = (unsigned short) lists.sentinel;
			flush();
		}
		int end = done > 0 ? sub + ((done >> 3) - 1) * lpm + 1 : 0;
		for (int o = 1; o < lpm; o <<= 1) end = max(end, __shfl_xor_sync(kFull, end, o));
		const unsigned s2 = (unsigned) lists.sentinel | ((unsigned) lists.sentinel << 16);
		for (int b = sub + (done >> 3) * lpm; b < end; b += lpm) pdst[(int64_t) b * lists.n] = make_uint4(s2, s2, s2, s2);
		if (act && sub == 0) po.count[gi] = ovf ? kListOverflow : (unsigned short) (8 * end);
	}
	// the molecule's force: its lanes' partial sums in a fixed order
	for (int o = 1; o < lpm; o <<= 1) {
		Fx += __shfl_xor_sync(kFull, Fx, o);
		Fy += __shfl_xor_sync(kFull, Fy, o);
		Fz += __shfl_xor_sync(kFull, Fz, o);
	}
	if (act && !ovf && sub == 0) MV += finish(kick, gi, Fx, Fy, Fz, rx, ry, rz, cid, lists, fx, fy, fz, status);
}

// Forces of brick `brick` from the neighbour lists that build_lists made on the same cell
// structure, at the current positions: staging as in pairs, then the molecules of the brick's
// own cells, 32 per warp regardless of their cell, each evaluate their list with the exact cutoff.
// Chunks of 64 entries are summed in FP32 and added to FP64 accumulators.
// Shared memory: layout(s_cap, kFP64) (no hit words, no half-precision copy).
// kPrune: a prune step (the build lists in, the inner lists out through po).
template <bool kFP64, bool kSingle, bool kLjIsRc, bool kWide = true, bool kPrune = false>
__device__ __forceinline__ void list_pairs(const Const& p, const Box& bx, int brick, int64_t slot,
                                           unsigned char* smem, const double* rx, const double* ry, const double* rz,
                                           const int32_t* cid, const int32_t* cstart, double* fx, double* fy,
                                           double* fz, double* partials, int* status, const Lists lists,
                                           const Kick& kick, const PruneOut& po = PruneOut{}) {
	const SmemLayout L = layout(p.s_cap, kFP64);
	const Smem S = views(smem, L);
	const int tid = threadIdx.x, warp = tid >> 5;
	const int ns = p.ns;
	__shared__ int s_own[kWarps + 1], s_ocell[kWarps];
	// sentinel slot: far from every molecule (entries past a list's end point to it)
	if (!kFP64 && tid == 0) S.hi[p.s_cap] = make_float4(1e15f, 1e15f, 1e15f, __uint_as_float((256u << 18) | (256u << 9) | 256u));
	const bool staged = stage_cells<kFP64, kWide>(p, bx, brick, S, rx, ry, rz, cid, cstart, s_own, s_ocell);
	const int n_own = s_own[kWarps];
	double U = 0.0, W = 0.0, NP = 0.0, MV = 0.0;
	bool same = false;
	if (!staged) {
		// over capacity: gather from global memory
		for (int t = tid; t < n_own; t += kThreads) {
			int w = 0;
			while (w < 7 && s_own[w + 1] <= t) w++;
			const int gi = S.gst[s_ocell[w]] + (t - s_own[w]);
			PairSums s = gather_pairs<!kFP64>(gi, rx, ry, rz, cid, cstart, bx.g, S.pd, ns, p.rc2, p.rclj2, bx.coff);
			MV += finish(kick, gi, s.F[0], s.F[1], s.F[2], rx, ry, rz, cid, lists, fx, fy, fz, status);
			U += s.U;
			W += s.W;
			NP += s.np;
			same |= s.same;
		}
	} else {
		// rounds of up to 256 molecules: the first as full warps of 32 (the fewest warp
		// instructions), a later one spread over every warp, g consecutive molecules with lpm lanes
		// each (lpm * g <= 32), so that no warp is left alone with a few long lists
		for (int base = 0; base < n_own; base += kThreads) {
			const int m = min(kThreads, n_own - base);
			const int g = base == 0 ? 32 : (m + kWarps - 1) / kWarps;
			const int lpm = lanes_per_molecule(g);
			const int w0 = base + warp * g, w1 = min(w0 + g, base + m);
			if (w0 < w1)
				list_chunk<kFP64, kSingle, kLjIsRc, false, kPrune>(p, bx, S, s_own, s_ocell, w0, w1, lpm, rx, ry, rz, cid,
				                                                   cstart, fx, fy, fz, status, lists, kick, U, W, NP,
				                                                   MV, same, po,
				                                                   reinterpret_cast<unsigned short*>(smem + L.total) + tid);
		}
	}
	if (same) atomicOr(status, kStatusSamePosition);
	block_sum3_at(U, W, NP, partials, slot, MV);
}

// A sparse brick (see kSparseCap) by one warp, in its own shared-memory area laid out as
// layout(kSparseCap, kFP64) plus 17 ints (own-cell prefix and cells): staging of the 4x4x4
// region flattened over its molecules (cell found by bisection of the staged-cell starts), then
// list_chunk; U, W, pair count to partials[brick]. Warp-level synchronisation only.
__host__ __device__ inline size_t sparse_warp_bytes(bool fp64) {
	return align16(layout(kSparseCap, fp64).total + sizeof(int) * 17);
}

template <bool kFP64, bool kSingle, bool kLjIsRc>
__device__ __forceinline__ void list_pairs_warp(const Const& p, const Box& bx, int brick, unsigned char* ws,
                                                const double* rx, const double* ry, const double* rz,
                                                const int32_t* cid, const int32_t* cstart, double* fx, double* fy,
                                                double* fz, double* partials, int* status, const Lists& lists,
                                                const Kick& kick) {
	const SmemLayout L = layout(kSparseCap, kFP64);
	const Smem S = views(ws, L);
	int* own = reinterpret_cast<int*>(ws + L.total);
	const int lane = threadIdx.x & 31;
	const Grid& g = bx.g;
	const int bc[3] = {brick % bx.nb[0], (brick / bx.nb[0]) % bx.nb[1], brick / (bx.nb[0] * bx.nb[1])};
	for (int c = lane; c < 64; c += 32) {
		const int l[3] = {c & 3, (c >> 2) & 3, c >> 4};
		int gc[3];
		for (int d = 0; d < 3; d++) gc[d] = staged_coord(bx, d, bc[d], l[d], S.csh[3 * c + d], S.ck[3 * c + d]);
		const int gcell = bx.coff + (gc[2] * g.nc[1] + gc[1]) * g.nc[0] + gc[0];
		const int st = cstart[gcell];
		S.gst[c] = st;
		S.cnt[c] = max(0, cstart[gcell + 1] - st);
	}
	__syncwarp();
	{
		const int a = S.cnt[2 * lane], b = S.cnt[2 * lane + 1];
		int inc = a + b;
		for (int o = 1; o < 32; o <<= 1) {
			const int y = __shfl_up_sync(kFull, inc, o);
			if (lane >= o) inc += y;
		}
		const int excl = inc - (a + b);
		S.cs[2 * lane] = excl;
		S.cs[2 * lane + 1] = excl + a;
		if (lane == 31) S.cs[64] = inc;
	}
	__syncwarp();
	const int total = S.cs[64];
	const bool staged = total <= kSparseCap;
	if (staged) {
		for (int t = lane; t < total; t += 32) {
			int lo = 0, hi = 63;
			while (lo < hi) {
				const int mid = (lo + hi + 1) >> 1;
				if (S.cs[mid] <= t)
					lo = mid;
				else
					hi = mid - 1;
			}
			const int gi = S.gst[lo] + (t - S.cs[lo]);
			stage_at<kFP64 ? kStageList64 : kStageList32>(bx, S, t, rx[gi], ry[gi], rz[gi], cid[gi], S.ck[3 * lo],
			                                              S.ck[3 * lo + 1], S.ck[3 * lo + 2], S.csh[3 * lo],
			                                              S.csh[3 * lo + 1], S.csh[3 * lo + 2]);
		}
	}
	if (lane == 0) {
		int acc = 0;
		for (int w = 0; w < 8; w++) {
			int ic;
			const bool ok = own_cell(bx, brick, w, ic);
			own[w] = acc;
			own[9 + w] = ic;
			acc += ok ? S.cnt[ic] : 0;
		}
		own[8] = acc;
	}
	__syncwarp();
	const int n_own = own[8];
	double U = 0.0, W = 0.0, NP = 0.0, MV = 0.0;
	bool same = false;
	if (staged) {
		for (int t0 = 0; t0 < n_own; t0 += 32) {
			const int g = min(32, n_own - t0);
			list_chunk<kFP64, kSingle, kLjIsRc, true>(p, bx, S, own, own + 9, t0, t0 + g, lanes_per_molecule(g), rx, ry,
			                                          rz, cid, cstart, fx, fy, fz, status, lists, kick, U, W, NP, MV,
			                                          same);
		}
	} else {
		for (int t = lane; t < n_own; t += 32) {
			int w = 0;
			while (w < 7 && own[w + 1] <= t) w++;
			const int gi = S.gst[own[9 + w]] + (t - own[w]);
			PairSums ps = gather_pairs<!kFP64>(gi, rx, ry, rz, cid, cstart, g, S.pd, p.ns, p.rc2, p.rclj2, bx.coff);
			MV += finish(kick, gi, ps.F[0], ps.F[1], ps.F[2], rx, ry, rz, cid, lists, fx, fy, fz, status);
			U += ps.U;
			W += ps.W;
			NP += ps.np;
			same |= ps.same;
		}
	}
	if (same) atomicOr(status, kStatusSamePosition);
	U = warp_sum(U);
	W = warp_sum(W);
	NP = warp_sum(NP);
	MV = warp_sum(MV);
	if (lane == 0) {
		partials[4 * (int64_t) brick + 0] = U;
		partials[4 * (int64_t) brick + 1] = W;
		partials[4 * (int64_t) brick + 2] = NP;
		partials[4 * (int64_t) brick + 3] = MV;
	}
}

}  // namespace brick
}  // namespace mdgpu
