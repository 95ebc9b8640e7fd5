// Cell-binned Verlet list build.
//
// Replaces simple_fill_cells / simple_update_neigh_list (src/CUDA/Lists/CUDA_simple_verlet.cuh:
// 14-95) and the host control of CUDASimpleVerletList::update (src/CUDA/Lists/
// CUDASimpleVerletList.cu:231-289).  Cells are filled by a counting sort (count, scan,
// scatter, then each particle placed by the rank of its caller's index within its cell), so there is no
// per-cell capacity to overflow and the neighbour order is deterministic run to run.  All of a build is
// one kernel, whose phases are separated by barriers of the blocks that run.  The geometry is the
// reference's fp32 geometry: cell coordinate ((x/L - floor(x/L)) * (1 - FLT_EPSILON)) * n and
// minimum-image squared distance against r_verlet^2, with IEEE division and the fused
// multiply-adds written out, so that oracle/dna2_oracle.c (oxo_verlet_f32) reproduces the
// pair set and the cell of every particle bit for bit.
#include "kernels.h"

#include <algorithm>
#include <atomic>
#include <cfloat>

namespace oxgb {

__device__ __forceinline__ int cell_coord(float x, float L, int n) {
	const float s = __fdiv_rn(x, L);
	return (int) (((s - floorf(s)) * (1.f - FLT_EPSILON)) * (float) n);
}

// Squared minimum-image separation in the reference's FP32 geometry (CUDABox.h:42-60: d - rint(d /
// L) L per axis, then the sum of squares as fused multiply-adds), with the image picked by a
// product with 1 / L rounded by the 1.5 * 2^23 addition instead of the IEEE quotient: the two
// images differ only where d / L sits within an ulp of a half-integer, i.e. |d| ~ L / 2, where both
// images leave a separation of ~L / 2 > the Verlet radius (L > 2 r_verlet).  So every pair that is
// listed, and its d^2, are exactly those of the quotient form (listed pairs have |d| < r_verlet,
// image 0 either way).
__device__ __forceinline__ float sqr_min_image_inv(float4 a, float4 b, float L, float inv) {
	float d[3] = {b.x - a.x, b.y - a.y, b.z - a.z};
#pragma unroll
	for(int k = 0; k < 3; k++) d[k] = __fmaf_rn(-__fsub_rn(__fmaf_rn(d[k], inv, 12582912.f), 12582912.f), L, d[k]);
	return __fmaf_rn(d[2], d[2], __fmaf_rn(d[1], d[1], __fmul_rn(d[0], d[0])));
}

// geometry of system s: box side, r_verlet^2, cells per side, first cell, bound of the
// Debye-Hueckel rows (squared, on backbone sites)
struct CellGeo {
	float box, rv2;
	int n, cell0;
	float dh2;
};

__device__ __forceinline__ int sys_of(const ListArgs &a, int i) { return a.sys ? a.sys[i] : 0; }

__device__ __forceinline__ CellGeo cell_geo(const ListArgs &a, int s) {
	if(!a.sys) return CellGeo{a.box, a.rverlet2, a.n_side, 0, a.dh_r2};
	return CellGeo{a.sys_box[s], a.sys_rv2[s], a.sys_nside[s], a.sys_cell0[s], a.sys_dh2 ? a.sys_dh2[s] : a.dh_r2};
}

// system s is rebuilt in this pass (always, unless per-system requests are given)
__device__ __forceinline__ bool rebuilt(const ListArgs &a, int s) { return !a.sys_stale || a.sys_stale[s] != 0; }


// ---------------------------------------------------------------- the blocks of a build
//
// One build is one launch: as a graph node of its own per phase it was a conditional (IF) node holding
// ten kernels, and that node alone cost 9 to 11 us per MD step whether the lists were stale or not (24
// nucleotides: 21.7 us per step with it, 12.7 without; 250,000: 117.5 and 106.6).  A kernel that reads
// the flag and returns costs about 1 us.
//
// Its phases are separated by barriers, so no block may wait for one that is not running: beside another
// program's kernel (a block here takes a whole SM's registers) some start when the others have finished.  A
// cooperative launch, which starts all blocks or none, had every build wait for whatever else the GPU ran:
// 40,000 nucleotides beside one-block kernels of 0.2 and 2 ms on another stream, 214 and 449 us per step
// (alone 53), a list of 16,000 1,948 us (alone 35); without it 53 to 54, and 37.  So the blocks that run share the
// work, which takes a build of the whole grid 1 to 2 us more.  The first phase is
// cut into as many items as the grid has blocks, each taken by whichever block asks for one; who asks before
// the last item is done is a member of the build, and the later phases and their barriers are the members'
// alone (their number changes no result).  A block that starts later finds the roll closed and leaves.  The
// last block of the grid to leave clears the barrier, the requests and the flag, which so stand for every
// block of the launch alike.
//
// A wait that should not end gives up after some seconds, flags the build and lets its block leave.  Such a
// block is missing at every later barrier, so no block gets beyond the phase after that one, and what a phase
// reads was written in full.  Its cell counts stay behind, on which no build may start: the roll stays closed to
// later ones until the host has cleared them (ListBuffers::reset).
//
// Measured, a rebuild / a step without one, before the one launch and now (us): 24 nucleotides 30 / 21.7 -> 11 / 14;
// 40,000 duplex nucleotides 75 / 47.7 -> 62 / 38; 250,000 strand nucleotides 230 / 117.5 -> 172 / 107;
// the plain list of 120,000 (no term lists) 97.3 -> 64.7.
constexpr int LIST_TPB = 1024;
// shared memory of a block that fills a whole system's cells (system_cells): padded counts, nucleotides
constexpr int LIST_LOCAL_SMEM = (LIST_LOCAL_CELLS + LIST_LOCAL_CELLS / 16 + 2 + LIST_LOCAL_N) * (int) sizeof(int);

// this block's number among the members, and how many they are (0: not a member); in shared memory, read where
// needed (the rows have no register to spare)
struct Member {
	int id, n;
};

// ListSync::roll: closed | a build gave up | arrivals << 32 | items taken << 16 | items done, in one word, so that
// ending an item and asking for the next is one atomic (as two words, one waits for the other); left: blocks that
// gave up << 16 | blocks
typedef unsigned long long Roll;
constexpr Roll ROLL_CLOSED = 1ull << 63, ROLL_FAILED = 1ull << 62, ROLL_ARRIVED = 1ull << 32, ROLL_TAKEN = 1ull << 16;
constexpr unsigned LEFT_FAILED = 0x10000u;

__device__ __forceinline__ unsigned roll_arrivals(Roll r) { return (unsigned) (r >> 32) & 0xffffu; }
__device__ __forceinline__ unsigned roll_taken(Roll r) { return (unsigned) (r >> 16) & 0xffffu; }
__device__ __forceinline__ unsigned roll_done(Roll r) { return (unsigned) r & 0xffffu; }

// (thread 0) polls *at until it is not `from`; false if the wait ran out
__device__ __forceinline__ bool poll(const ListArgs &a, const unsigned *at, unsigned from, unsigned &now) {
	now = from;
	for(int it = 0; now == from && it < a.wait_polls; it++) asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(now) : "l"(at) : "memory");
	return now != from;
}

// The first phase, item(k) for k = 0 .. gridDim.x - 1, and the roll; false if the wait ran out.  meanwhile(): work
// of every block, done while its arrival is on the way.
template <class Item, class Work>
__device__ __forceinline__ bool first_phase(const ListArgs &a, volatile Member &me, const Item &item, const Work &meanwhile) {
	const unsigned grid = gridDim.x;
	if(grid == 1) {
		meanwhile();
		item(0);
		if(threadIdx.x == 0) me.id = 0, me.n = 1;
		__syncthreads();
		return true;
	}
	ListSync *y = a.sync;
	__shared__ Roll roll;
	__shared__ int ok;
	Roll r = 0;
	if(threadIdx.x == 0) r = atomicAdd(&y->roll, ROLL_ARRIVED + ROLL_TAKEN);
	meanwhile();
	if(threadIdx.x == 0) {
		roll = r;
		me.id = (int) roll_arrivals(r);
		me.n = 0;
	}
	__syncthreads();
	if(roll & ROLL_CLOSED) return !(roll & ROLL_FAILED);
	unsigned closer = 0;  // (thread 0: the members, once this block has closed the roll)
	for(unsigned k = roll_taken(roll); k < grid; k = roll_taken(roll)) {
		item((int) k);
		__syncthreads();  // (everyone has read `roll`, too)
		if(threadIdx.x == 0) {
			asm volatile("atom.add.acq_rel.gpu.u64 %0, [%1], %2;" : "=l"(r) : "l"(&y->roll), "l"(ROLL_TAKEN + 1) : "memory");
			roll = r;
			if(roll_done(r) == grid - 1) {
				// (all have arrived, commonly; else nobody may any more)
				closer = roll_arrivals(r);
				if(closer < grid) closer = roll_arrivals(atomicOr(&y->roll, ROLL_CLOSED));
				asm volatile("st.release.gpu.u32 [%0], %1;" ::"l"(&y->members), "r"(closer) : "memory");
			}
		}
		__syncthreads();
	}
	if(threadIdx.x == 0) {
		ok = 1;
		if(closer == 0) ok = poll(a, &y->members, 0, closer);
		me.n = (int) closer;
	}
	__syncthreads();
	return ok != 0;
}

// the members' barrier; false if the wait ran out
__device__ __forceinline__ bool members_sync(const ListArgs &a, const volatile Member &me) {
	ListSync *y = a.sync;
	if(me.n == 1) {
		__syncthreads();
		return true;
	}
	__shared__ int ok;
	__syncthreads();
	if(threadIdx.x == 0) {
		unsigned gen, old;
		asm volatile("ld.relaxed.gpu.u32 %0, [%1];" : "=r"(gen) : "l"(&y->gen) : "memory");
		asm volatile("atom.add.acq_rel.gpu.u32 %0, [%1], 1;" : "=r"(old) : "l"(&y->count) : "memory");
		ok = 1;
		if(old == (unsigned) me.n - 1) {
			asm volatile("st.relaxed.gpu.u32 [%0], 0;" ::"l"(&y->count) : "memory");
			asm volatile("red.add.release.gpu.u32 [%0], 1;" ::"l"(&y->gen) : "memory");
		}
		else ok = poll(a, &y->gen, gen, gen);
	}
	__syncthreads();
	return ok != 0;
}

// ---------------------------------------------------------------- phases: cells

__device__ __forceinline__ int block_incl_scan(int v, int *warp_tot) {
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
	for(int off = 1; off < 32; off <<= 1) {
		const int u = __shfl_up_sync(0xffffffffu, v, off);
		if(lane >= off) v += u;
	}
	if(lane == 31) warp_tot[w] = v;
	__syncthreads();
	if(w == 0) {
		int t = lane < (int) (blockDim.x >> 5) ? warp_tot[lane] : 0;
#pragma unroll
		for(int off = 1; off < 32; off <<= 1) {
			const int u = __shfl_up_sync(0xffffffffu, t, off);
			if(lane >= off) t += u;
		}
		warp_tot[lane] = t;  // inclusive over warps
	}
	__syncthreads();
	return v + (w > 0 ? warp_tot[w - 1] : 0);
}


// this block's share of n items: a contiguous range
__device__ __forceinline__ void block_share(const volatile Member &me, int n, int &lo, int &hi) {
	lo = (int) ((long long) n * me.id / me.n);
	hi = (int) ((long long) n * (me.id + 1) / me.n);
}

// the cell of a nucleotide at r in a system of geometry g
__device__ __forceinline__ int cell_at(const ListArgs &a, const CellGeo &g, const float4 &r) {
	if(!(fabsf(r.x) < 1e7f && fabsf(r.y) < 1e7f && fabsf(r.z) < 1e7f)) {
		atomicOr(a.status, OXGB_ERR_NONFINITE);
		return g.cell0;
	}
	const int n = g.n;
	int cx = cell_coord(r.x, g.box, n), cy = cell_coord(r.y, g.box, n), cz = cell_coord(r.z, g.box, n);
	if(cx < 0 || cx >= n || cy < 0 || cy >= n || cz < 0 || cz >= n) {
		atomicOr(a.status, OXGB_ERR_CELL);
		cx = min(max(cx, 0), n - 1);
		cy = min(max(cy, 0), n - 1);
		cz = min(max(cz, 0), n - 1);
	}
	return g.cell0 + (cz * n + cy) * n + cx;
}

// the cell of every nucleotide of the systems to rebuild, and their numbers (cell_count is zero between
// builds): the item-th of gridDim.x parts
__device__ __forceinline__ void phase_count(const ListArgs &a, int item) {
	for(int i = item * LIST_TPB + threadIdx.x; i < a.N; i += gridDim.x * LIST_TPB) {
		const int s = sys_of(a, i);
		if(!rebuilt(a, s)) continue;
		const int c = cell_at(a, cell_geo(a, s), a.pos[i]);
		a.cell_of[i] = c;
		atomicAdd(a.cell_count + c, 1);
	}
}

// The number of nucleotides in cell c: counted in this build, or, in a system that is not rebuilt, its
// unchanged segment (every system keeps its total, so its segments keep their place)
__device__ __forceinline__ int cell_size(const ListArgs &a, int c) {
	if(a.cell_sys && !rebuilt(a, a.cell_sys[c])) return a.cell_start[c + 1] - a.cell_start[c];
	return __ldcg(a.cell_count + c);  // (counted by atomics: not through L1)
}

// sum of f(c) over this block's share of the cells, to scan_part[me.id]
template <class F>
__device__ __forceinline__ void phase_block_sum(const ListArgs &a, const volatile Member &me, int n_cells, const F &f) {
	__shared__ int wt[32];
	int lo, hi, v = 0;
	block_share(me, n_cells, lo, hi);
	for(int c = lo + threadIdx.x; c < hi; c += LIST_TPB) v += f(c);
	const int incl = block_incl_scan(v, wt);
	if(threadIdx.x == LIST_TPB - 1) a.scan_part[me.id] = incl;
}

// exclusive scan by one block of f(c) over the cells lo .. hi - 1, from `carry`: put(c, sum below c);
// returns the sum up to hi
template <class F, class P>
__device__ __forceinline__ int block_scan(int lo, int hi, int carry, const F &f, const P &put) {
	__shared__ int wt[32];
	for(int c0 = lo; c0 < hi; c0 += 4 * LIST_TPB) {
		const int base = c0 + (int) threadIdx.x * 4;
		int n[4], sum = 0;
#pragma unroll
		for(int k = 0; k < 4; k++) {
			n[k] = base + k < hi ? f(base + k) : 0;
			sum += n[k];
		}
		__syncthreads();  // the scratch of the scan before is free, and every f of this tile is read
		const int incl = block_incl_scan(sum, wt);
		int run = carry + incl - sum;
#pragma unroll
		for(int k = 0; k < 4; k++) {
			if(base + k < hi) put(base + k, run);
			run += n[k];
		}
		carry += wt[31];
	}
	return carry;
}

// exclusive scan of f(c), after phase_block_sum and a barrier: put(c, sum of f below c) for every cell
// of the block's share; the block of the last cell calls put(n_cells, total)
template <class F, class P>
__device__ __forceinline__ void phase_scan(const ListArgs &a, const volatile Member &me, int n_cells, const F &f, const P &put) {
	__shared__ int wt[32], before;
	int lo, hi, v = 0;
	block_share(me, n_cells, lo, hi);
	for(int b = threadIdx.x; b < me.id; b += LIST_TPB) v += a.scan_part[b];
	v = block_incl_scan(v, wt);
	if(threadIdx.x == LIST_TPB - 1) before = v;
	__syncthreads();
	const int total = block_scan(lo, hi, before, f, put);
	if(hi == n_cells && hi > lo && threadIdx.x == 0) put(n_cells, total);
}

// particles into their cells' segments, in arbitrary order (cell_tmp)
__device__ __forceinline__ void phase_scatter(const ListArgs &a, const volatile Member &me) {
	for(int i = me.id * LIST_TPB + threadIdx.x; i < a.N; i += me.n * LIST_TPB) {
		if(!rebuilt(a, sys_of(a, i))) continue;
		a.cell_tmp[atomicAdd(a.cell_cursor + a.cell_of[i], 1)] = i;
	}
}

// the caller's index of slot i (slot i itself while the engine was never sorted)
__device__ __forceinline__ int id_of(const ListArgs &a, int i) { return a.id ? a.id[i] : i; }

// what the rows read of nucleotide i at place p of the cell-sorted order, so that the candidates of
// neighbouring cells are read from consecutive addresses (w of the position: i)
__device__ __forceinline__ void sorted_copy(const ListArgs &a, int p, int i) {
	float4 r = a.pos[i];
	r.w = __int_as_float(i);
	a.spos[p] = r;
	if(a.sa1) {
		a.sa1[p] = a.fa1[i];
		a.sback[p] = a.fback[i];
	}
}

// the number of a cell's nucleotides (places b .. e - 1 of cell_tmp) with a caller's index below key
__device__ __forceinline__ int rank_in_cell(const ListArgs &a, int b, int e, int key) {
	int rank = 0;
	for(int k = b; k < e; k += 4) {
		int m[4];
#pragma unroll
		for(int u = 0; u < 4; u++) m[u] = k + u < e ? a.cell_tmp[k + u] : -1;
#pragma unroll
		for(int u = 0; u < 4; u++) rank += m[u] >= 0 && id_of(a, m[u]) < key;
	}
	return rank;
}

// each particle's rank by caller's index within its cell gives the deterministic order (cell_list)
__device__ __forceinline__ void phase_rank(const ListArgs &a, const volatile Member &me, bool copy) {
	for(int i = me.id * LIST_TPB + threadIdx.x; i < a.N; i += me.n * LIST_TPB) {
		if(!rebuilt(a, sys_of(a, i))) continue;
		const int c = a.cell_of[i], b = a.cell_start[c];
		const int p = b + rank_in_cell(a, b, a.cell_start[c + 1], id_of(a, i));
		a.cell_list[p] = i;
		if(copy) sorted_copy(a, p, i);
	}
}

// A system's cells by one block, with block barriers only (ListArgs::local_cells; no cell-order storage):
// counts, segments from the system's first nucleotide on, scatter and ranks.  For systems of a few thousand
// nucleotides this saves four grid barriers of about 2.5 us, and a batch's systems go side by side.  The
// counts, starts and scattered nucleotides stay in shared memory: through global memory each of the five
// dependent passes waited for L2 (rebuilds of two or so systems of a batch of 96, cells: 18 us; so: 11).
__device__ __forceinline__ void system_cells(const ListArgs &a, int s) {
	extern __shared__ int local_smem[];
	__shared__ int wt[32];
	int *cnt = local_smem, *tmp = cnt + LIST_LOCAL_CELLS + LIST_LOCAL_CELLS / 16 + 2;
	auto at = [](int c) { return c + (c >> 4); };  // (threads take runs of up to 16 cells: padded to miss bank conflicts)
	const int i0 = a.sys_off ? a.sys_off[s] : 0, i1 = a.sys_off ? a.sys_off[s + 1] : a.N;
	const CellGeo g = cell_geo(a, s);
	const int cells = g.n * g.n * g.n, t = threadIdx.x;
	constexpr int Q = LIST_LOCAL_N / LIST_TPB;  // nucleotides of a thread, whose loads overlap
	float4 r[Q];
	int c[Q], rank[Q];
#pragma unroll
	for(int q = 0; q < Q; q++) {
		const int i = i0 + t + q * LIST_TPB;
		if(i < i1) r[q] = a.pos[i];
	}
	for(int k = t; k < cells; k += LIST_TPB) cnt[at(k)] = 0;
	__syncthreads();
#pragma unroll
	for(int q = 0; q < Q; q++) {
		const int i = i0 + t + q * LIST_TPB;
		c[q] = rank[q] = 0;
		if(i < i1) {
			const int cell = cell_at(a, g, r[q]);
			a.cell_of[i] = cell;
			c[q] = cell - g.cell0;
			rank[q] = atomicAdd(cnt + at(c[q]), 1);
		}
	}
	__syncthreads();
	{
		const int w = (cells + LIST_TPB - 1) / LIST_TPB, lo = min(t * w, cells), hi = min(lo + w, cells);
		int sum = 0;
		for(int k = lo; k < hi; k++) sum += cnt[at(k)];
		int run = block_incl_scan(sum, wt) - sum;
		for(int k = lo; k < hi; k++) {
			const int n = cnt[at(k)];
			cnt[at(k)] = run;
			run += n;
		}
		if(t == 0) cnt[at(cells)] = i1 - i0;
	}
	__syncthreads();
	// (the next system's first cell starts where this one's last ends)
	for(int k = t; k <= cells; k += LIST_TPB) a.cell_start[g.cell0 + k] = i0 + cnt[at(k)];
#pragma unroll
	for(int q = 0; q < Q; q++) {
		const int i = i0 + t + q * LIST_TPB;
		if(i < i1) tmp[cnt[at(c[q])] + rank[q]] = i;
	}
	__syncthreads();
#pragma unroll
	for(int q = 0; q < Q; q++) {
		const int i = i0 + t + q * LIST_TPB;
		if(i >= i1) continue;
		const int b = cnt[at(c[q])], e = cnt[at(c[q] + 1)];
		int p = i0 + b;
		for(int k = b; k < e; k++) p += tmp[k] < i;
		a.cell_list[p] = i;
		sorted_copy(a, p, i);
	}
	__syncthreads();
}

// ---------------------------------------------------------------- phases: cell-order storage
// (CUDABaseBackend::_sort_particles, CUDABaseBackend.cu:263-281, with the cell order of this
// build in place of a Hilbert key: the order is the one the counting sort just produced)

// this build moves nucleotides: sorting on, and the build count a multiple of sort_every
__device__ __forceinline__ bool sort_now(const ListArgs &a) {
	return a.sort_every > 0 && a.id && (a.rebuilds ? *a.rebuilds : 0ull) % (unsigned long long) a.sort_every == 0ull;
}

// New slot k takes old slot perm[k] (rebuilt systems; the others stay): cell_list[k], or with the
// Hilbert order the nucleotide whose cell is at that position along the curve (hstart, the scan of the
// cells' sizes in that order), at its rank within the cell
__device__ __forceinline__ void phase_sort_perm(const ListArgs &a, const volatile Member &me) {
	for(int p = me.id * LIST_TPB + threadIdx.x; p < a.N; p += me.n * LIST_TPB) {
		int from = p, to = p;
		if(rebuilt(a, sys_of(a, p))) {
			from = a.cell_list[p];
			if(a.cell_hil) {
				const int c = a.cell_of[from];
				to = a.hstart[a.cell_hil[c]] + (p - a.cell_start[c]);
			}
		}
		a.perm[to] = from;
		a.inv[from] = to;
	}
}

// everything of old slot perm[k] into the staging buffer at k; bonds renumbered
__device__ __forceinline__ void phase_sort_gather(const ListArgs &a, const volatile Member &me) {
	const long long N = a.N;
	double4_32a *sd = reinterpret_cast<double4_32a *>(a.scratch);
	float4 *sf = reinterpret_cast<float4 *>(a.scratch + 4 * 32 * N);
	int2 *sb = reinterpret_cast<int2 *>(a.scratch + (4 * 32 + SORT_MIRRORS * 16) * N);
	int *si = reinterpret_cast<int *>(a.scratch + (4 * 32 + SORT_MIRRORS * 16 + 8) * N);
	for(int k = me.id * LIST_TPB + threadIdx.x; k < a.N; k += me.n * LIST_TPB) {
		const int from = a.perm[k];
#pragma unroll
		for(int t = 0; t < 4; t++) sd[t * N + k] = a.st[t][from];
#pragma unroll
		for(int t = 0; t < SORT_MIRRORS; t++)
			if(a.mir[t]) sf[t * N + k] = a.mir[t][from];
		const int2 b = a.bonds_rw[from];
		sb[k] = make_int2(b.x >= 0 ? a.inv[b.x] : -1, b.y >= 0 ? a.inv[b.y] : -1);
		si[k] = a.id[from];
		si[N + k] = a.cell_of[from];
		// segment entries name slots: renamed in place (each k touches its own entry)
		a.cell_list[k] = a.inv[a.cell_list[k]];
	}
}

// the staging buffer back into the arrays, and the inverse map
__device__ __forceinline__ void phase_sort_scatter(const ListArgs &a, const volatile Member &me) {
	const long long N = a.N;
	const double4_32a *sd = reinterpret_cast<const double4_32a *>(a.scratch);
	const float4 *sf = reinterpret_cast<const float4 *>(a.scratch + 4 * 32 * N);
	const int2 *sb = reinterpret_cast<const int2 *>(a.scratch + (4 * 32 + SORT_MIRRORS * 16) * N);
	const int *si = reinterpret_cast<const int *>(a.scratch + (4 * 32 + SORT_MIRRORS * 16 + 8) * N);
	for(int k = me.id * LIST_TPB + threadIdx.x; k < a.N; k += me.n * LIST_TPB) {
#pragma unroll
		for(int t = 0; t < 4; t++) a.st[t][k] = sd[t * N + k];
#pragma unroll
		for(int t = 0; t < SORT_MIRRORS; t++)
			if(a.mir[t]) a.mir[t][k] = sf[t * N + k];
		if(a.frame64) write_frame64(a.frame64, N, k, sd[3 * N + k], sb[k].x < 0 || sb[k].y < 0);
		a.bonds_rw[k] = sb[k];
		const int id = si[k];
		a.id[k] = id;
		a.slot[id] = k;
		a.cell_of[k] = si[N + k];
	}
}

__device__ __forceinline__ void phase_sorted_copies(const ListArgs &a, const volatile Member &me) {
	for(int p = me.id * LIST_TPB + threadIdx.x; p < a.N; p += me.n * LIST_TPB)
		if(rebuilt(a, sys_of(a, p))) sorted_copy(a, p, a.cell_list[p]);
}

// ---------------------------------------------------------------- the nucleotides to rebuild

// The nucleotides of the systems to rebuild, one system after the other, so that a build of a few systems
// of a batch is dealt over the whole grid (going through all nucleotides and skipping the others, two
// systems of a batch of 96 landed on 40 of 152 SMs and each group of lanes skipped a dozen nucleotides:
// 21 us for their rows; so: 12.6).  For batches of up to a block's threads; else all nucleotides, tested.
struct StaleSystems {
	int n, total;  // systems (0: all nucleotides), nucleotides
	int first[LIST_TPB], end[LIST_TPB];
	// the v-th nucleotide
	__device__ __forceinline__ int operator[](int v) const {
		if(n == 0) return v;
		int lo = 0, hi = n - 1;  // the first system whose end exceeds v
		while(lo < hi) {
			const int m = (lo + hi) / 2;
			if(end[m] > v) hi = m;
			else lo = m + 1;
		}
		return first[lo] + v - (lo > 0 ? end[lo - 1] : 0);
	}
};

// into shared memory; a barrier has to follow
__device__ __forceinline__ void list_stale_systems(const ListArgs &a, StaleSystems &y) {
	if(a.n_systems < 2 || !a.sys || !a.sys_stale || !a.sys_off || a.n_systems > LIST_TPB) {
		if(threadIdx.x == 0) y.n = 0, y.total = a.N;
		return;
	}
	__shared__ int wt[32];
	const int s = threadIdx.x;
	const bool on = s < a.n_systems && rebuilt(a, s);
	const int first = on ? a.sys_off[s] : 0, size = on ? a.sys_off[s + 1] - first : 0;
	const int k = block_incl_scan(on, wt);
	__syncthreads();
	const int end = block_incl_scan(size, wt);
	if(on) y.first[k - 1] = first, y.end[k - 1] = end;
	if(s == LIST_TPB - 1) y.n = k, y.total = end;
}

// ---------------------------------------------------------------- phases: rows

// A listed pair can have hydrogen bonding or cross stacking before the next rebuild only if its base
// sites (0.4 a1 from the centres), coaxial stacking only if its stacking sites (0.34 a1), are within
// their bounds.  Exactly symmetric in the two nucleotides, so the pair-term lists are symmetric.
__device__ __forceinline__ bool pair_sites_near(const ListArgs &a, float3 d, float4 a1i, float4 a1j) {
	const float bx = d.x + 0.4f * (a1j.x - a1i.x), by = d.y + 0.4f * (a1j.y - a1i.y), bz = d.z + 0.4f * (a1j.z - a1i.z);
	if(bx * bx + by * by + bz * bz < a.base_r2) return true;
	const float sx = d.x + 0.34f * (a1j.x - a1i.x), sy = d.y + 0.34f * (a1j.y - a1i.y), sz = d.z + 0.34f * (a1j.z - a1i.z);
	return sx * sx + sy * sy + sz * sz < a.stk_r2;
}

// the minimum-image separation vector of a listed pair (the reference's FP32 geometry, explicit
// fused multiply-adds), the image picked as in sqr_min_image_inv: the same integer as the IEEE
// quotient's rint for any pair closer than the Verlet radius, so the same vector
__device__ __forceinline__ float3 min_image_vec_inv(float4 a, float4 b, float L, float inv) {
	float d[3] = {b.x - a.x, b.y - a.y, b.z - a.z};
#pragma unroll
	for(int k = 0; k < 3; k++) d[k] = __fmaf_rn(-__fsub_rn(__fmaf_rn(d[k], inv, 12582912.f), 12582912.f), L, d[k]);
	return make_float3(d[0], d[1], d[2]);
}

// squared distance of the backbone sites of a listed pair (d: the centres' separation, bk: the
// backbone offsets)
__device__ __forceinline__ float back_sq(float3 d, float4 bki, float4 bkj) {
	const float x = d.x + bkj.x - bki.x, y = d.y + bkj.y - bki.y, z = d.z + bkj.z - bki.z;
	return x * x + y * y + z * z;
}

// A pair's excluded volume can act before the next rebuild only if one of its four site pairs
// (backbone-backbone, base-base, backbone-base both ways) is within that pair's cutoff plus twice
// the skin: the staleness test rebuilds before any site moves farther than the skin.  d is the
// centres' separation, a1 and bk the axes and backbone offsets (base site at 0.4 a1).
__device__ __forceinline__ bool ev_sites_near(const ListArgs &a, float3 d, float4 a1i, float4 bki, float4 a1j, float4 bkj) {
	const float ix = 0.4f * a1i.x, iy = 0.4f * a1i.y, iz = 0.4f * a1i.z;
	const float jx = 0.4f * a1j.x, jy = 0.4f * a1j.y, jz = 0.4f * a1j.z;
	auto sq = [](float x, float y, float z) { return x * x + y * y + z * z; };
	return sq(d.x + bkj.x - bki.x, d.y + bkj.y - bki.y, d.z + bkj.z - bki.z) < a.evs_r2[0] ||
			sq(d.x + jx - ix, d.y + jy - iy, d.z + jz - iz) < a.evs_r2[1] ||
			sq(d.x + jx - bki.x, d.y + jy - bki.y, d.z + jz - bki.z) < a.evs_r2[2] ||
			sq(d.x + bkj.x - ix, d.y + bkj.y - iy, d.z + bkj.z - iz) < a.evs_r2[2];
}

__device__ __forceinline__ void put(int *rows, bool col_major, long long N, int stride, int i, int k, int j) {
	if(col_major) rows[(long long) k * N + i] = j;
	else rows[(long long) i * stride + k] = j;
}


// K lanes per nucleotide (16 or 32).  The cells x - 1, x, x + 1 of a (z, y) row are consecutive cells, so
// their segments are one run of the cell-sorted order (two where the row wraps at the box face): nine
// rows, one per lane, in the serial scan order (dz, dy, dx from -1 to 1, each cell's segment by index).
// A scan over the nine lanes numbers the candidates; the group takes K of them at a time, each lane
// finding its candidate's row by a binary search of the scan, and reads them from consecutive addresses.
// The hits are compacted in order with a ballot and kept until K of them are there, which the lanes then
// put through the site tests of the Debye-Hueckel, excluded-volume and pair-term lists together (a third
// to a half of the candidates hits: tested where it is found, a hit would take its lane through them
// alone).  So every row comes out as a serial scan would write it.  (With 4 or 8 lanes, the groups of a
// warp reach those tests at different times and run them one after the other: 120 M warp instructions
// for 250,000 nucleotides.)
template <int K>
__device__ __forceinline__ void phase_rows(const ListArgs &a, const volatile Member &me, const StaleSystems &stale) {
	constexpr int G = LIST_TPB / K;
	__shared__ int2 kept[G][2 * K + 1];  // (place in the cell-sorted order, nucleotide); odd stride
	const int lane = threadIdx.x & 31, sub = lane % K, grp = (int) threadIdx.x / K;
	const unsigned gmask = (K == 32 ? 0xffffffffu : ((1u << (K & 31)) - 1u) << (lane - sub));
	const unsigned below = ((1u << lane) - 1u) & gmask;
	const bool terms = a.ev_nb != nullptr, dhl = a.dh_nb != nullptr;
	const long long N = a.N;
	// neighbouring nucleotides to the groups of a block (their rows' entries share sectors); where every
	// group gets one at most, to different blocks
	for(int v = stale.total <= me.n * G ? grp * me.n + me.id : me.id * G + grp; v < stale.total; v += me.n * G) {  // group-uniform
		const int i = stale[v];
		const int sy = sys_of(a, i);
		if(!rebuilt(a, sy)) continue;
		const CellGeo g = cell_geo(a, sy);
		const float4 r = a.pos[i];
		const int2 b = a.bonds[i];
		const int n = g.n;
		const int c = a.cell_of[i] - g.cell0;
		const int cx = c % n, cy = (c / n) % n, cz = c / (n * n);
		const float inv_box = __frcp_rn(g.box);
		float4 a1i = make_float4(0.f, 0.f, 0.f, 0.f), bki = a1i;
		if(terms || dhl) {
			a1i = a.fa1[i];
			bki = a.fback[i];
		}
		// the runs of a row: cells [x0, e0) and, where it wraps, [x1, e1)
		int x0, e0, x1 = 0, e1 = 0;
		if(cx > 0 && cx < n - 1) x0 = cx - 1, e0 = cx + 2;
		else if(cx == 0) x0 = n - 1, e0 = n, e1 = 2;  // cells n - 1 | 0, 1
		else x0 = n - 2, e0 = n, e1 = 1;              // cells n - 2, n - 1 | 0
		// this lane's row: its run at s0, and w0 where it wraps
		int s0 = 0, len = 0, w0 = 0, lenw = 0;
		if(sub < 9) {
			int z = cz + sub / 3 - 1, y = cy + sub % 3 - 1;
			z += z < 0 ? n : (z >= n ? -n : 0);
			y += y < 0 ? n : (y >= n ? -n : 0);
			const int *row = a.cell_start + g.cell0 + (z * n + y) * n;
			s0 = row[x0], len = row[e0] - s0;
			if(e1 > 0) w0 = row[x1], lenw = row[e1] - w0;
		}
		int incl = len + lenw;
#pragma unroll
		for(int off = 1; off < 16; off <<= 1) {
			const int u = __shfl_up_sync(gmask, incl, off, K);
			if(sub >= off) incl += u;
		}
		const int total = __shfl_sync(gmask, incl, 8, K);
		const int first = incl - len - lenw, wrap = first + len;
		int nk = 0, cnt = 0, nev = 0, npt = 0, ndh = 0;
		// the first m kept hits (m <= K), a lane each
		auto take = [&](int m) {
			__syncwarp(gmask);
			bool hev = false, hpt = false, hdh = false;
			int2 e = make_int2(0, 0);
			if(sub < m) {
				e = kept[grp][sub];
				if(cnt + sub < a.max_nb) put(a.nb, a.col_major != 0, N, a.max_nb, i, cnt + sub, e.y);
				if(terms || dhl) {
					const float4 rj = a.spos[e.x];
					const float3 d = min_image_vec_inv(r, rj, g.box, inv_box);
					const float4 bkj = a.sback[e.x];
					hdh = dhl && back_sq(d, bki, bkj) < g.dh2;
					if(terms && sqr_min_image_inv(r, rj, g.box, inv_box) < a.ev_r2) {
						const float4 a1j = a.sa1[e.x];
						hev = ev_sites_near(a, d, a1i, bki, a1j, bkj);
						hpt = pair_sites_near(a, d, a1i, a1j);
					}
				}
			}
			cnt += m;
			if(dhl) {
				const unsigned md = __ballot_sync(gmask, hdh) & gmask;
				const int k = ndh + __popc(md & below);
				if(hdh && k < a.max_nb) a.dh_nb[(long long) k * N + i] = e.y;
				ndh += __popc(md);
			}
			if(terms) {
				const unsigned me = __ballot_sync(gmask, hev) & gmask, mp = __ballot_sync(gmask, hpt) & gmask;
				const int ke = nev + __popc(me & below), kp = npt + __popc(mp & below);
				if(hev && ke < a.ev_cap) a.ev_nb[(long long) ke * N + i] = e.y;
				if(hpt && kp < a.pt_cap) a.pt_nb[(long long) kp * N + i] = e.y;
				nev += __popc(me);
				npt += __popc(mp);
			}
		};
		for(int t0 = 0; t0 < total; t0 += K) {
			const int t = t0 + sub;
			// the first row whose inclusive count exceeds t
			int l = 0;
#pragma unroll
			for(int step = 8; step > 0; step >>= 1) {
				const int v = __shfl_sync(gmask, incl, l + step - 1, K);
				if(v <= t) l += step;
			}
			int u = t + __shfl_sync(gmask, s0 - first, l, K);
			if(e1 > 0) {  // group-uniform
				const int at = __shfl_sync(gmask, wrap, l, K), to = __shfl_sync(gmask, w0 - wrap, l, K);
				if(t >= at) u = t + to;
			}
			bool hit = false;
			int j = -1;
			if(t < total) {
				const float4 rj = a.spos[u];
				j = __float_as_int(rj.w);
				hit = j != i && j != b.x && j != b.y && sqr_min_image_inv(r, rj, g.box, inv_box) < g.rv2;
			}
			const unsigned m = __ballot_sync(gmask, hit) & gmask;
			if(hit) kept[grp][nk + __popc(m & below)] = make_int2(u, j);
			nk += __popc(m);
			if(nk >= K) {  // group-uniform
				take(K);
				nk -= K;
				__syncwarp(gmask);
				int2 e = make_int2(0, 0);
				if(sub < nk) e = kept[grp][K + sub];
				__syncwarp(gmask);
				if(sub < nk) kept[grp][sub] = e;
			}
		}
		if(nk > 0) take(nk);
		__syncwarp(gmask);  // (the kept hits are read before the next nucleotide's are written)
		if(sub != 0) continue;
		if(cnt > a.max_nb) atomicOr(a.status, OXGB_ERR_NEIGH_OVERFLOW);
		if(a.term_max && cnt > a.term_max[3]) atomicMax(a.term_max + 3, cnt);
		a.nnb[i] = cnt;
		if(dhl) a.dh_n[i] = ndh;
		a.list_pos[i] = r;
		if(terms) {
			if(nev > a.ev_cap || npt > a.pt_cap) atomicOr(a.status, OXGB_ERR_NEIGH_OVERFLOW);
			if(a.term_max) {  // read first: the maxima rarely grow, so few atomics reach them
				if(nev > a.term_max[0]) atomicMax(a.term_max, nev);
				if(npt > a.term_max[1]) atomicMax(a.term_max + 1, npt);
			}
			a.ev_n[i] = nev;
			a.pt_n[i] = npt;
			a.list_a1[i] = a1i;
			a.list_back[i] = bki;
		}
	}
}

// The pair-term entries owned by a group of 32 nucleotides, together (ForceArgs::own): of every pair
// the nucleotide i with the lower caller's index keeps the entry, with the pair's position k in its
// list and m in the partner's (the lists are symmetric).  Four lanes per nucleotide over its entries; the
// search of the partner's list reads four entries at a time (a serial walk is a chain of dependent
// loads).  Their order within the group does not matter to the results.  A group that straddles systems
// is rebuilt if one of them is: the other lists are as they were.
__device__ __forceinline__ void phase_own(const ListArgs &a, const volatile Member &me) {
	constexpr int T = 4 * PAIR_GROUP, B = LIST_TPB / T;  // threads of a group, groups of a block
	__shared__ int count[B];
	const long long N = a.N;
	const int w = (int) threadIdx.x / T, t = (int) threadIdx.x % T, groups = (a.N + PAIR_GROUP - 1) / PAIR_GROUP;
	for(int g0 = me.id * B; g0 < groups; g0 += me.n * B) {
		const int g = g0 + w, i = g * PAIR_GROUP + t / 4;
		if(t == 0) count[w] = 0;
		__syncthreads();
		bool stale = false;
		if(a.n_systems > 1) {
			const int lo = g * PAIR_GROUP, hi = min(lo + PAIR_GROUP, a.N) - 1;
			if(lo < a.N)
				for(int s = sys_of(a, lo); s <= sys_of(a, hi); s++) stale |= rebuilt(a, s);
		}
		else stale = true;
		if(stale && i < a.N) {
			int2 *own = a.own + (long long) g * PAIR_GROUP * a.pt_cap;
			const int n = min(a.pt_n[i], a.pt_cap);
			const int key = id_of(a, i);
			for(int k = t & 3; k < n; k += 4) {
				const int j = a.pt_nb[(long long) k * N + i];
				if(id_of(a, j) < key) continue;
				int m = 255;
				const int nj = min(a.pt_n[j], a.pt_cap);
				for(int u = 0; u < nj && m == 255; u += 4) {
					int e[4];
#pragma unroll
					for(int v = 0; v < 4; v++) e[v] = u + v < nj ? a.pt_nb[(long long) (u + v) * N + j] : -1;
#pragma unroll
					for(int v = 0; v < 4; v++)
						if(e[v] == i) m = u + v;
				}
				if(m == 255) atomicOr(a.status, OXGB_ERR_NEIGH_OVERFLOW);  // an asymmetric (overflowed) list
				own[atomicAdd(&count[w], 1)] = make_int2(j, k | (m << 8) | (t / 4) << 16);
			}
		}
		__syncthreads();
		if(stale && t == 0 && g < groups) a.own_n[g] = count[w];
	}
}

// ---------------------------------------------------------------- the build

// the phases of a build; false if a wait ran out
template <int K>
__device__ __forceinline__ bool list_phases(const ListArgs &a, int n_cells) {
	__shared__ StaleSystems stale;
	__shared__ volatile Member me;
	const bool joined = first_phase(a, me, [&](int item) {
		if(!a.local_cells) return phase_count(a, item);
		for(int k = item; k < a.n_systems; k += gridDim.x)
			if(rebuilt(a, k)) system_cells(a, k);
	}, [&] { list_stale_systems(a, stale); });
	if(!joined) return false;
	if(me.n == 0) return true;
	if(!a.local_cells) {
		auto sync = [&] { return members_sync(a, me); };
		phase_block_sum(a, me, n_cells, [&](int c) { return cell_size(a, c); });
		if(!sync()) return false;
		phase_scan(a, me, n_cells, [&](int c) { return cell_size(a, c); }, [&](int c, int start) {
			a.cell_start[c] = start;
			if(c == n_cells) return;
			a.cell_cursor[c] = start;
			a.cell_count[c] = 0;  // for the next build (cells of systems that are not rebuilt hold zero)
		});
		if(!sync()) return false;
		phase_scatter(a, me);
		if(!sync()) return false;
		const bool sorting = sort_now(a);
		phase_rank(a, me, !sorting);
		if(!sync()) return false;
		if(sorting) {
			if(a.cell_hil) {
				for(int c = me.id * LIST_TPB + threadIdx.x; c < n_cells; c += me.n * LIST_TPB)
					a.hcount[a.cell_hil[c]] = a.cell_start[c + 1] - a.cell_start[c];
				if(!sync()) return false;
				phase_block_sum(a, me, n_cells, [&](int c) { return a.hcount[c]; });
				if(!sync()) return false;
				phase_scan(a, me, n_cells, [&](int c) { return a.hcount[c]; }, [&](int c, int start) { a.hstart[c] = start; });
				if(!sync()) return false;
			}
			phase_sort_perm(a, me);
			if(!sync()) return false;
			phase_sort_gather(a, me);
			if(!sync()) return false;
			phase_sort_scatter(a, me);
			if(!sync()) return false;
			phase_sorted_copies(a, me);
			if(!sync()) return false;
		}
	}
	phase_rows<K>(a, me, stale);
	if(a.own) {
		if(!members_sync(a, me)) return false;
		phase_own(a, me);
	}
	return true;
}

template <int K>
__global__ void __launch_bounds__(LIST_TPB, 1) k_list_build(ListArgs a, int n_cells) {
	pdl_trigger();  // (the next kernel's blocks wait for this one's end)
	pdl_wait();
	if(a.check_flag && *(volatile const int *) a.flag == 0) return;
	const bool whole = list_phases<K>(a, n_cells);
	// the last block to leave clears the barrier, and after a whole build counts it and clears the requests
	__shared__ int last;
	__syncthreads();
	if(threadIdx.x == 0) {
		if(!whole) atomicOr(a.status, OXGB_ERR_SYNC);
		__threadfence();
		last = 1;
		if(gridDim.x > 1) {
			const unsigned left = atomicAdd(&a.sync->left, whole ? 1u : LEFT_FAILED + 1);
			last = (left & (LEFT_FAILED - 1)) == gridDim.x - 1;
			if(last) {
				if(!whole || left >= LEFT_FAILED) last = 0;
				a.sync->roll = last ? 0 : ROLL_CLOSED | ROLL_FAILED;
				a.sync->members = a.sync->count = a.sync->left = 0;
			}
		}
	}
	__syncthreads();
	if(!last) return;
	if(a.sys_stale)
		for(int s = threadIdx.x; s < a.n_systems; s += LIST_TPB) a.sys_stale[s] = 0;
	if(threadIdx.x != 0) return;
	if(a.rebuilds) *a.rebuilds += 1;
	*a.flag = 0;
}

template <int K>
static cudaError_t launch_build(const ListArgs &a, int n_cells, cudaStream_t s) {
	// a block per SM (it takes the SM's registers), fewer where the nucleotides do not fill them
	static std::atomic<int> sms[64];  // per device (whoever comes first; the same value)
	int dev = 0;
	cudaError_t e = cudaGetDevice(&dev);
	if(e != cudaSuccess) return e;
	if(dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
	if(sms[dev].load() == 0) {
		int n = 0;
		if((e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
		if((e = cudaFuncSetAttribute(k_list_build<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, LIST_LOCAL_SMEM)) != cudaSuccess)
			return e;
		sms[dev].store(std::min(n, LIST_MAX_BLOCKS));
	}
	const long long threads = std::max((long long) a.N * K, (long long) n_cells / 8);
	const int blocks = (int) std::min<long long>(sms[dev].load(), (threads + LIST_TPB - 1) / LIST_TPB);
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = dim3(blocks > 0 ? blocks : 1);
	cfg.blockDim = dim3(LIST_TPB);
	cfg.dynamicSmemBytes = a.local_cells ? LIST_LOCAL_SMEM : 0;
	cfg.stream = s;
	cudaLaunchAttribute at[1];
	at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
	at[0].val.programmaticStreamSerializationAllowed = 1;
	cfg.attrs = at;
	cfg.numAttrs = a.pdl ? 1 : 0;
	return cudaLaunchKernelEx(&cfg, k_list_build<K>, a, n_cells);
}

cudaError_t launch_list_build(const ListArgs &a, cudaStream_t s) {
	const int n_cells = a.n_cells_total > 0 ? a.n_cells_total : a.n_side * a.n_side * a.n_side;
	return a.list_kind == OXGB_LIST_WARP ? launch_build<32>(a, n_cells, s) : launch_build<16>(a, n_cells, s);
}

}  // namespace oxgb
