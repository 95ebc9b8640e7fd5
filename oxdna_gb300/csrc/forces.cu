// oxDNA2 force and torque kernels.
//
// The engine's (mixed and FP64) evaluate bonds and pair terms once per pair, in blocks of their own
// (k_bonded_pairs), and Debye-Hueckel and the excluded volume from each end of a nucleotide's rows
// (k_nonbonded_*), with no atomics and a fixed summation order.  The reference layout (float4 positions
// with btype/index packed in w, float4 quaternions, int2 bonds and a neighbour matrix of any stride) has
// a kernel of its own, which accumulates into forces and torques initialised by the caller, exactly the
// contract of CUDABaseInteraction::compute_forces (k_forces_reference, at the end).  They replace the
// reference's thread-per-nucleotide dna_forces (src/CUDA/Interactions/CUDA_DNA.cuh:832-904).
#include "kernels.h"
#include "split.cuh"

#include <cuda_runtime.h>

namespace oxgb {

template <typename R>
struct KahanV {
	v3<R> s, c;
	OXGB_HD void add(v3<R> x) {
		kadd(s.x, c.x, x.x);
		kadd(s.y, c.y, x.y);
		kadd(s.z, c.z, x.z);
	}
	static OXGB_HD void kadd(R &sum, R &comp, R x) {
		const R y = x - comp;
		const R t = sum + y;
		comp = (t - sum) - y;
		sum = t;
	}
};

__device__ __forceinline__ int ref_type_of_btype(int bt) {
	return (bt > 0) ? (bt & 3) : 3 - ((3 - bt) & 3);
}

// the settings table of system sy (read through L1: a handful of values per thread, the same for all
// threads of a system)
template <typename R>
__device__ __forceinline__ const DNA2Table<R> &table_of(const ForceArgs &a, int sy) {
	return reinterpret_cast<const DNA2Table<R> *>(a.table)[sy];
}

// Debye-Hueckel of a pair in FP32 (dh_sites): the force on p over the vector from p's backbone site to
// q's, and the energy, at squared distance r2 < rc2; cut: the end charges' factor.  1 / r by a Newton step
// on the approximate reciprocal square root, both branches evaluated (a third of the pairs is inside
// the smoothing range, so a warp takes both anyway).
struct DebyeF {
	float rc, rc2, rhigh, mk, pre, b, half;
	__device__ __forceinline__ explicit DebyeF(const DNA2Table<float> &P)
		: rc(P.dh_rc), rc2(P.dh_rc * P.dh_rc), rhigh(P.dh_rhigh), mk(P.dh_minus_kappa), pre(P.dh_prefactor), b(P.dh_b),
		  half(P.dh_half_charged_ends ? 0.5f : 1.f) {}
	__device__ __forceinline__ float force(float r2, float cut, float &e) const {
		float v = rsqrtf(r2);
		v = v * fmaf(-0.5f * r2 * v, v, 1.5f);
		const float r = r2 * v;
		const float ex = pre * m_exp(mk * r), g = b * (r - rc);
		const bool in = r < rhigh;
		e = cut * (in ? ex * v : g * (r - rc));
		return -((in ? ex * (v - mk) * v : -2.f * g) * cut) * v;
	}
};

// ---------------------------------------------------------------- particle loaders

struct LoadMixed {
	// minimum image of q - p as hi + lo.  The image m = round(d / box) of a listed pair
	// (|q - p| < r_verlet, far below box / 2) has d / box at least 0.4 from a half-integer, so
	// the product with an approximate inverse rounds to the same integer as the quotient;
	// rounding by the 1.5 * 2^23 addition (|d / box| < 2^22) keeps it on the FMA pipe.
	// The FP32 difference of the hi parts is exact only for coordinates of one sign within a
	// factor of two of each other.  Otherwise -- coordinates on both sides of zero (a few per
	// cent of the nucleotides of a large box, in each dimension), or unwrapped coordinates a box
	// side or more apart -- it rounds at half an ulp of the result (2e-8 for a bonded
	// separation of 0.66, 3.8e-6 across the images of a box of 158), which the stiff excluded
	// volume (force slope up to 1.6e4) turns into force errors of 1e-4 and more.  The exact
	// remainder of the hi difference (two_sum) therefore always joins the low part.  The shift
	// by m box sides is then exact (the result is a small multiple of the ulp of d and of
	// box_hi); the box remainder goes to lo.  sep_soft leaves the remainder out, for
	// Debye-Hueckel and for screening: Debye-Hueckel's force slope is below 0.1, so the 3.8e-6
	// moves its force by less than 1e-6.
	template <bool EXACT = true>
	__device__ __forceinline__ Sep<float> sep(const float4 &ph, const float4 &pl, const float4 &qh, const float4 &ql,
			const DNA2Table<float> &P) const {
		const float qv[3] = {qh.x, qh.y, qh.z}, pv[3] = {ph.x, ph.y, ph.z};
		float d[3], l[3] = {ql.x - pl.x, ql.y - pl.y, ql.z - pl.z};
#pragma unroll
		for(int k = 0; k < 3; k++) {
			if(EXACT) {
				const F2 t = two_sum(qv[k], -pv[k]);
				d[k] = t.s;
				l[k] = __fadd_rn(l[k], t.e);
			}
			else {
				d[k] = qv[k] - pv[k];
			}
		}
#pragma unroll
		for(int k = 0; k < 3; k++) {
			const float m = __fsub_rn(__fmaf_rn(d[k], P.inv_box, 12582912.f), 12582912.f);
			d[k] = fmaf(-m, P.box_hi, d[k]);
			l[k] = fmaf(-m, P.box_lo, l[k]);
		}
		return Sep<float>{v3<float>{d[0], d[1], d[2]}, v3<float>{l[0], l[1], l[2]}};
	}
	__device__ __forceinline__ Sep<float> sep_soft(const float4 &ph, const float4 &pl, const float4 &qh, const float4 &ql,
			const DNA2Table<float> &P) const {
		return sep<false>(ph, pl, qh, ql, P);
	}
	// bonded neighbours: no periodic image; the hi difference's remainder as in sep
	__device__ __forceinline__ Sep<float> diff(const float4 &ph, const float4 &pl, const float4 &qh, const float4 &ql) const {
		const F2 x = two_sum(qh.x, -ph.x), y = two_sum(qh.y, -ph.y), z = two_sum(qh.z, -ph.z);
		return Sep<float>{v3<float>{x.s, y.s, z.s}, v3<float>{__fadd_rn(ql.x - pl.x, x.e), __fadd_rn(ql.y - pl.y, y.e),
				__fadd_rn(ql.z - pl.z, z.e)}};
	}
};

struct LoadRef {
	const float4 *pos, *quat;
	__device__ __forceinline__ NoRefine refine(int, int) const { return NoRefine{}; }
	__device__ __forceinline__ void load(int i, const DNA2Table<float> &P, const int2 b, Nuc<float> &n, float4 &hi,
			float4 &lo) const {
		hi = pos[i];
		lo = make_float4(0.f, 0.f, 0.f, 0.f);
		const float4 q = quat[i];
		quat_frame(q.x, q.y, q.z, q.w, n.a1, n.a2, n.a3);
		make_sites(n);
		n.btype = __float_as_int(hi.w) >> 22;
		n.type = ref_type_of_btype(n.btype);
		n.is_end = (b.x < 0 || b.y < 0);
	}
	__device__ __forceinline__ Sep<float> sep(const float4 &ph, const float4 &, const float4 &qh, const float4 &,
			const DNA2Table<float> &P) const {
		float d[3] = {qh.x - ph.x, qh.y - ph.y, qh.z - ph.z};
#pragma unroll
		for(int k = 0; k < 3; k++) d[k] = fmaf(-rintf(d[k] * P.inv_box), P.box_hi, d[k]);
		return Sep<float>{v3<float>{d[0], d[1], d[2]}, v3<float>{0.f, 0.f, 0.f}};
	}
	__device__ __forceinline__ Sep<float> diff(const float4 &ph, const float4 &, const float4 &qh, const float4 &) const {
		return Sep<float>{v3<float>{qh.x - ph.x, qh.y - ph.y, qh.z - ph.z}, v3<float>{0.f, 0.f, 0.f}};
	}
};

template <typename R>
struct Vec4Of;
template <>
struct Vec4Of<float> {
	using T = float4;
};
template <>
struct Vec4Of<double> {
	using T = double4_32a;
};

// FFS order parameters on the reference layout (hb_op_precalc, near_hb_op_precalc and
// dist_op_precalc, src/CUDA/Interactions/CUDA_DNA.cuh:910-1067): one thread per listed pair
// (op1[k], op2[k]), centre separation at its FP32 minimum image, base sites at POS_BASE a1.
//   MODE 0: the pair's hydrogen-bonding energy f1 f4(t1) f4(t2) f4(t3) f4(t4) f4(t7) f4(t8)
//           (no hb_multiplier, as the reference's kernel), 0 unless the bases are complementary
//           and their distance is inside the hydrogen-bonding window;
//   MODE 1: "nearly bonded": at least six of those seven factors on (f1 < 0, each f4 > 0);
//   MODE 2: the base-base distance.
template <int MODE>
__global__ void k_order_params(const float4 *poss, const float4 *quat, const int *op1, const int *op2, int n,
		const DNA2Table<float> *table, float *val, bool *flag) {
	const DNA2Table<float> &P = *table;
	const int k = blockIdx.x * blockDim.x + threadIdx.x;
	if(k >= n) return;
	const LoadRef ld{poss, quat};
	Nuc<float> p, q;
	float4 ph, pl, qh, ql;
	ld.load(op1[k], P, make_int2(0, 0), p, ph, pl);
	ld.load(op2[k], P, make_int2(0, 0), q, qh, ql);
	const v3<float> rb = site_vec(ld.sep(ph, pl, qh, ql, P), q.base, p.base);
	const float r2 = dot(rb, rb);
	if(MODE == 2) {
		val[k] = m_sqrt(r2);
		return;
	}
	float e = 0.f;
	bool near = false;
	if(p.btype + q.btype == 3 && float(OXM_HYDR_RCLOW) * float(OXM_HYDR_RCLOW) < r2 &&
			r2 < float(OXM_HYDR_RCHIGH) * float(OXM_HYDR_RCHIGH)) {
		const float rmod = m_sqrt(r2);
		const v3<float> rd = rb * (1.f / rmod);
		float f1, f1d, g[6], gd;
		f1_both(P, rmod, OXM_F1_HB, p.type, q.type, f1, f1d);
		f4_both(-dot(p.a1, q.a1), sin_between(p.a1, q.a1), OXM_F4_HB_T1, g[0], gd);
		f4_both(-dot(q.a1, rd), sin_between(q.a1, rd), OXM_F4_HB_T2, g[1], gd);
		f4_both(dot(p.a1, rd), sin_between(p.a1, rd), OXM_F4_HB_T2, g[2], gd);
		f4_both(dot(p.a3, q.a3), sin_between(p.a3, q.a3), OXM_F4_HB_T4, g[3], gd);
		f4_both(-dot(rd, q.a3), sin_between(q.a3, rd), OXM_F4_HB_T7, g[4], gd);
		f4_both(dot(rd, p.a3), sin_between(p.a3, rd), OXM_F4_HB_T7, g[5], gd);
		e = f1;
		int on = f1 < 0.f;
#pragma unroll
		for(int m = 0; m < 6; m++) {
			e *= g[m];
			on += g[m] > 0.f;
		}
		near = on >= 6;
	}
	if(MODE == 0) val[k] = e;
	else flag[k] = near;
}

cudaError_t launch_order_params(int mode, const float4 *poss, const float4 *quat, const int *op1, const int *op2, int n,
		const void *table, float *val, bool *flag, cudaStream_t s) {
	const int blocks = (n + 127) / 128;
	const DNA2Table<float> *t = reinterpret_cast<const DNA2Table<float> *>(table);
	if(mode == 0) k_order_params<0><<<blocks, 128, 0, s>>>(poss, quat, op1, op2, n, t, val, flag);
	else if(mode == 1) k_order_params<1><<<blocks, 128, 0, s>>>(poss, quat, op1, op2, n, t, val, flag);
	else k_order_params<2><<<blocks, 128, 0, s>>>(poss, quat, op1, op2, n, t, val, flag);
	return cudaGetLastError();
}

}  // namespace oxgb

// ====================================================================== split path
//
// A nucleotide has ~20-30 neighbours, only a few of them close enough for hydrogen bonding, cross or
// coaxial stacking.  The split path
//  * evaluates every bonded pair once, for both nucleotides, by two threads in different warps (bonded_block);
//  * evaluates hydrogen bonding, cross and coaxial stacking once per pair of the pair-term lists, for both
//    nucleotides, in stages with eight lanes per term (pair_block);
//  * runs Debye-Hueckel and the excluded volume from both ends of a pair, K lanes per nucleotide over lists of
//    their own (pairs whose sites can come into reach before the next build);
//  * gathers the bonded and pair results in the non-bonded kernel's epilogue (fixed order, no atomics).

namespace oxgb {

// the remainders of nucleotide k's a1 and backbone offset (written with the mirrors)
__device__ __forceinline__ SiteLo site_lo(const float4 *a1lo, const float4 *backlo, int k) {
	const float4 u = __ldg(a1lo + k), v = __ldg(backlo + k);
	return SiteLo{v3<float>{u.x, u.y, u.z}, v3<float>{v.x, v.y, v.z}};
}

// the refined excluded volume of a stiff bonded contact (rare): out of line, so that the kernel's
// register allocation stays that of its common path
template <int K>
__device__ __noinline__ float ev_refined_call(const float4 *a1lo, const float4 *backlo, int i, int j, Sep<float> sep,
		v3<float> ps, v3<float> pa1, int pbase, v3<float> qs, v3<float> qa1, int qbase, v3<float> *f) {
	v3<float> fo;
	const float e = ev_refined<K>(sep, ps, pa1, site_lo(a1lo, backlo, i), pbase, qs, qa1, site_lo(a1lo, backlo, j), qbase, fo);
	*f = fo;
	return e;
}

// a non-bonded pair with a site pair inside its excluded-volume cutoff, refined: force and torque
// on nucleotide i (of p) and the energy (rare; out of line, so that the non-bonded kernel's loops
// keep their register allocation)
__device__ __noinline__ float4 ev_pair_refined_call(const float4 *a1lo, const float4 *backlo, int i, int j, float4 sh,
		float4 sl, float4 pb, float4 pk, float4 pa, float4 qb, float4 qk, float4 qa, float3 *T) {
	Nuc<float> p, q;
	p.back = v3<float>{pb.x, pb.y, pb.z}, p.base = v3<float>{pk.x, pk.y, pk.z}, p.a1 = v3<float>{pa.x, pa.y, pa.z};
	q.back = v3<float>{qb.x, qb.y, qb.z}, q.base = v3<float>{qk.x, qk.y, qk.z}, q.a1 = v3<float>{qa.x, qa.y, qa.z};
	const Sep<float> sep{v3<float>{sh.x, sh.y, sh.z}, v3<float>{sl.x, sl.y, sl.z}};
	v3<float> F{0.f, 0.f, 0.f}, t{0.f, 0.f, 0.f};
	const float e = pair_ev_refined(sep, p, site_lo(a1lo, backlo, i), q, site_lo(a1lo, backlo, j), F, t);
	*T = make_float3(t.x, t.y, t.z);
	return make_float4(F.x, F.y, F.z, e);
}

// refines the FP32 engine path for pair (i, j): the site offsets' remainders for the stiff
// radial factors, and the stiff excluded-volume contacts
struct StoredLo {
	static constexpr bool on = true;
	const float4 *a1lo, *backlo;
	int i, j;
	__device__ __forceinline__ SiteLo lo(int which) const { return site_lo(a1lo, backlo, which ? j : i); }
	template <int K>
	__device__ __forceinline__ float ev(const Sep<float> &sep, v3<float> ps, v3<float> pa1, int pbase, v3<float> qs,
			v3<float> qa1, int qbase, v3<float> &f) const {
		return ev_refined_call<K>(a1lo, backlo, i, j, sep, ps, pa1, pbase, qs, qa1, qbase, &f);
	}
};

struct SplitMixed {
	const float4 *hi, *lo, *fa1, *fa3, *fback;
	const float4 *a1lo, *backlo;  // remainders of fa1 / fback (StoredLo)
	__device__ __forceinline__ StoredLo refine(int i, int j) const { return StoredLo{a1lo, backlo, i, j}; }
	__device__ __forceinline__ void full(int j, Nuc<float> &n, float4 &h, float4 &l) const {
		h = __ldg(hi + j);
		l = __ldg(lo + j);
		const float4 x1 = __ldg(fa1 + j), x3 = __ldg(fa3 + j), bk = __ldg(fback + j);
		n.a1 = v3<float>{x1.x, x1.y, x1.z};
		n.a3 = v3<float>{x3.x, x3.y, x3.z};
		n.a2 = cross(n.a3, n.a1);
		n.back = v3<float>{bk.x, bk.y, bk.z};
		n.stack = n.a1 * float(OXM_POS_STACK);
		n.base = n.a1 * float(OXM_POS_BASE);
		n.btype = __float_as_int(h.w) >> 22;
		n.type = __float_as_int(l.w) & 7;
		n.is_end = bk.w != 0.f;
	}
	// position, axes a1 and a3, base site and types: what the pair terms read
	__device__ __forceinline__ void axes(int j, Nuc<float> &n, float4 &h, float4 &l) const {
		h = __ldg(hi + j);
		l = __ldg(lo + j);
		const float4 x1 = __ldg(fa1 + j), x3 = __ldg(fa3 + j);
		n.a1 = v3<float>{x1.x, x1.y, x1.z};
		n.a3 = v3<float>{x3.x, x3.y, x3.z};
		n.base = n.a1 * float(OXM_POS_BASE);
		n.btype = __float_as_int(h.w) >> 22;
		n.type = __float_as_int(l.w) & 7;
	}
	__device__ __forceinline__ void dh(int j, Nuc<float> &n, float4 &h, float4 &l) const {
		h = __ldg(hi + j);
		l = __ldg(lo + j);
		const float4 bk = __ldg(fback + j);
		n.back = v3<float>{bk.x, bk.y, bk.z};
		n.is_end = bk.w != 0.f;
	}
	__device__ __forceinline__ Sep<float> sep(const float4 &ph, const float4 &pl, const float4 &qh, const float4 &ql,
			const DNA2Table<float> &P) const {
		return LoadMixed{}.sep(ph, pl, qh, ql, P);
	}
	__device__ __forceinline__ Sep<float> sep_soft(const float4 &ph, const float4 &pl, const float4 &qh, const float4 &ql,
			const DNA2Table<float> &P) const {
		return LoadMixed{}.sep_soft(ph, pl, qh, ql, P);
	}
	__device__ __forceinline__ Sep<float> diff(const float4 &ph, const float4 &pl, const float4 &qh, const float4 &ql) const {
		return LoadMixed{}.diff(ph, pl, qh, ql);
	}
};

// The FP64 engine.  Its kernels are bound by the FP64 pipe (one warp instruction in some 16 cycles), so
// what they need in FP64 is read, not made: the frames are kept (write_frame64; made by every reader, a
// frame was 40 of the 180 FP64 operations of a Debye-Hueckel pair), the periodic image is picked by a
// product and a rounding addition instead of a division per axis (45 operations of a pair, now 12: the
// same integer but for separations within an ulp of half a box, twice the range of any listed pair), and
// pairs that a conservative test can dismiss are dismissed in FP32, on the mirrors that the list build uses.
// 4,000 duplex nucleotides, k_bonded_pairs and k_nonbonded_split: 68.7 and 46.1 us with frames and
// quotients per reader, 55.7 and 27.8 us so (526,000 and 497,000 FP64 warp instructions, then 380,000 and
// 267,000).
struct SplitDouble {
	const double4_32a *pos, *frame;
	long long N;
	SplitMixed screen;  // the FP32 mirrors
	__device__ __forceinline__ NoRefine refine(int, int) const { return NoRefine{}; }
	__device__ __forceinline__ Sep<double> sep(const double4_32a &p, const double4_32a &, const double4_32a &q,
			const double4_32a &, const DNA2Table<double> &P) const {
		double d[3] = {q.x - p.x, q.y - p.y, q.z - p.z};
		const double L = P.box_hi + P.box_lo;
#pragma unroll
		for(int k = 0; k < 3; k++) {
			constexpr double magic = 6755399441055744.0;  // 1.5 * 2^52
			const double m = __dsub_rn(__fma_rn(d[k], P.inv_box, magic), magic);
			d[k] = __fma_rn(-m, L, d[k]);
		}
		return Sep<double>{v3<double>{d[0], d[1], d[2]}, v3<double>{0., 0., 0.}};
	}
	__device__ __forceinline__ Sep<double> sep_soft(const double4_32a &p, const double4_32a &, const double4_32a &q,
			const double4_32a &, const DNA2Table<double> &P) const {
		return sep(p, p, q, q, P);
	}
	__device__ __forceinline__ Sep<double> diff(const double4_32a &p, const double4_32a &, const double4_32a &q,
			const double4_32a &) const {
		return Sep<double>{v3<double>{q.x - p.x, q.y - p.y, q.z - p.z}, v3<double>{0., 0., 0.}};
	}
	__device__ __forceinline__ void types(int j, Nuc<double> &n) const {
		n.btype = __float_as_int(screen.hi[j].w) >> 22;
		n.type = __float_as_int(screen.lo[j].w) & 7;
	}
	__device__ __forceinline__ void back(int j, Nuc<double> &n, double4_32a &h) const {
		h = pos[j];
		const double4_32a b = frame[3 * N + j];
		n.back = v3<double>{b.x, b.y, b.z};
		n.is_end = b.w != 0.0;
	}
	__device__ __forceinline__ void axes(int j, Nuc<double> &n, double4_32a &h) const {
		h = pos[j];
		const double4_32a x1 = frame[j], x3 = frame[2 * N + j];
		n.a1 = v3<double>{x1.x, x1.y, x1.z};
		n.a3 = v3<double>{x3.x, x3.y, x3.z};
		n.stack = n.a1 * double(OXM_POS_STACK);
		n.base = n.stack * ((double) OXM_POS_BASE / (double) OXM_POS_STACK);
		types(j, n);
	}
	__device__ __forceinline__ void full(int j, Nuc<double> &n, double4_32a &h) const {
		axes(j, n, h);
		back(j, n, h);
		const double4_32a x2 = frame[N + j];
		n.a2 = v3<double>{x2.x, x2.y, x2.z};
	}
	// the box as the FP32 separation reads it
	__device__ __forceinline__ static DNA2Table<float> screen_box(const DNA2Table<double> &P) {
		DNA2Table<float> f;
		const double L = P.box_hi + P.box_lo;
		f.box_hi = (float) L, f.box_lo = (float) (L - (double) f.box_hi), f.inv_box = 1.f / f.box_hi;
		return f;
	}
};

template <class Loader, typename R>
__device__ __forceinline__ void load_full(const Loader &ld, int j, const DNA2Table<R> &P, Nuc<R> &n,
		typename Vec4Of<R>::T &h, typename Vec4Of<R>::T &l);
template <>
__device__ __forceinline__ void load_full<SplitMixed, float>(const SplitMixed &ld, int j, const DNA2Table<float> &, Nuc<float> &n,
		float4 &h, float4 &l) {
	ld.full(j, n, h, l);
}
template <>
__device__ __forceinline__ void load_full<SplitDouble, double>(const SplitDouble &ld, int j, const DNA2Table<double> &,
		Nuc<double> &n, double4_32a &h, double4_32a &) {
	ld.full(j, n, h);
}
template <class Loader, typename R>
__device__ __forceinline__ void load_dh(const Loader &ld, int j, const DNA2Table<R> &P, Nuc<R> &n, typename Vec4Of<R>::T &h,
		typename Vec4Of<R>::T &l);
template <>
__device__ __forceinline__ void load_dh<SplitMixed, float>(const SplitMixed &ld, int j, const DNA2Table<float> &, Nuc<float> &n,
		float4 &h, float4 &l) {
	ld.dh(j, n, h, l);
}
template <>
__device__ __forceinline__ void load_dh<SplitDouble, double>(const SplitDouble &ld, int j, const DNA2Table<double> &, Nuc<double> &n,
		double4_32a &h, double4_32a &) {
	ld.back(j, n, h);
}

template <class Loader, typename R>
__device__ __forceinline__ void load_axes(const Loader &ld, int j, const DNA2Table<R> &P, Nuc<R> &n, typename Vec4Of<R>::T &h,
		typename Vec4Of<R>::T &l);
template <>
__device__ __forceinline__ void load_axes<SplitDouble, double>(const SplitDouble &ld, int j, const DNA2Table<double> &, Nuc<double> &n,
		double4_32a &h, double4_32a &) {
	ld.axes(j, n, h);
}
template <>
__device__ __forceinline__ void load_axes<SplitMixed, float>(const SplitMixed &ld, int j, const DNA2Table<float> &, Nuc<float> &n,
		float4 &h, float4 &l) {
	ld.axes(j, n, h, l);
}

template <>
__device__ __forceinline__ void load_axes<LoadRef, float>(const LoadRef &ld, int j, const DNA2Table<float> &P, Nuc<float> &n,
		float4 &h, float4 &l) {
	ld.load(j, P, make_int2(0, 0), n, h, l);
}

// A term's energies of a warp (0: none) into system sy's sum.  All terms of all nucleotides meet at eight
// addresses per system, where atomics go one after the other: a warp in one system, nearly all of them, adds
// up first.  The whole warp calls.  (An atomic per bond and lane made an upload and evaluation of 10,000
// nucleotides 481 us long, 399 so.)
__device__ __forceinline__ void add_split(double *esplit, int sy, int term, double e) {
	if(__all_sync(0xffffffffu, sy == __shfl_sync(0xffffffffu, sy, 0))) {
#pragma unroll
		for(int off = 16; off > 0; off >>= 1) e += __shfl_xor_sync(0xffffffffu, e, off);
		if((threadIdx.x & 31) != 0) return;
	}
	if(e != 0.0) atomicAdd(esplit + 8 * sy + term, e);
}

// Bonded block b of TPB threads: TPB / 2 bonds (owner p, partner q = n3[p]), a pair of threads each, in different warps:
// the first half of the block evaluates the stacking, the second half FENE and the bonded excluded
// volume, joined through shared memory.  One thread for all of a bond is a dependent chain twice as
// long, and as long as that chain is what a launch lasts where the chip is not full.

template <typename R, class Loader, bool SPLIT, bool ENERGY, int TPB>
__device__ __forceinline__ void bonded_block(const ForceArgs &a, const Loader &ld, int b) {
	constexpr int BONDS_PER_BLOCK = TPB / 2;
	using V4 = typename Vec4Of<R>::T;
	__shared__ R part[BONDS_PER_BLOCK][11];  // force, torques, energy of the backbone part (an odd number of words)
	const int t = threadIdx.x & (BONDS_PER_BLOCK - 1);
	const bool backbone = threadIdx.x >= BONDS_PER_BLOCK;  // warp-uniform
	// an MD step: from here on its second half kick is pending (the first step has read the mark)
	if(a.th.open_step && b == 0 && threadIdx.x == 0) *a.th.open_step = *a.th.step_base + a.th.step_offset;
	const int p = b * BONDS_PER_BLOCK + t;
	const int q = p < a.N ? a.bonds[p].x : -1;
	BondOut<R> o;
	o.f = o.tp = o.tq = v3<R>{R(0), R(0), R(0)};
	o.split[0] = o.split[1] = o.split[2] = R(0);
	if(q >= 0) {
		const int sy = a.sys ? a.sys[p] : 0;
		const DNA2Table<R> &P = table_of<R>(a, sy);
		Nuc<R> np, nq;
		V4 ph, pl, qh, ql;
		load_full<Loader, R>(ld, p, P, np, ph, pl);
		load_full<Loader, R>(ld, q, P, nq, qh, ql);
		if(backbone) {
			if(!bonded_backbone(P, np, nq, ld.diff(ph, pl, qh, ql), o, ld.refine(p, q))) atomicOr(a.status, OXGB_ERR_FENE);
			const R v[10] = {o.f.x, o.f.y, o.f.z, o.tp.x, o.tp.y, o.tp.z, o.tq.x, o.tq.y, o.tq.z, o.split[0] + o.split[1]};
#pragma unroll
			for(int k = 0; k < (ENERGY ? 10 : 9); k++) part[t][k] = v[k];
		}
		else {
			bonded_stacking(P, np, nq, ld.diff(ph, pl, qh, ql), o, ld.refine(p, q));
		}
	}
	if(SPLIT) {
		const int sy = a.sys ? a.sys[min(p, a.N - 1)] : 0;
		if(backbone) {
			add_split(a.esplit, sy, T_FENE, (double) o.split[0]);
			add_split(a.esplit, sy, T_BEXC, (double) o.split[1]);
		}
		else add_split(a.esplit, sy, T_STCK, (double) o.split[2]);
	}
	__syncthreads();
	if(q >= 0 && !backbone) {
		const R *v = part[t];
		V4 f, tp, tq;
		f.x = v[0] + o.f.x, f.y = v[1] + o.f.y, f.z = v[2] + o.f.z, f.w = ENERGY ? v[9] + o.split[2] : R(0);
		tp.x = v[3] + o.tp.x, tp.y = v[4] + o.tp.y, tp.z = v[5] + o.tp.z, tp.w = R(0);
		tq.x = v[6] + o.tq.x, tq.y = v[7] + o.tq.y, tq.z = v[8] + o.tq.z, tq.w = R(0);
		reinterpret_cast<V4 *>(a.bond_f)[p] = f;
		reinterpret_cast<V4 *>(a.bond_tp)[p] = tp;
		reinterpret_cast<V4 *>(a.bond_tq)[p] = tq;
	}
}

// per-lane compensated sums of a nucleotide's pair terms; ENERGY = false leaves the energies out
// (an MD step needs only forces and torques: the energy arithmetic of the pair functions is then
// dead code)
template <typename R, bool SPLIT, bool ENERGY = true>
struct SplitAcc {
	KahanV<R> F, T;
	R E, Ec, Eh, Ehc;
	R split[N_TERMS];
	__device__ __forceinline__ void add(const PairOut<R> &o) {
		F.add(o.F);
		T.add(o.T);
		if(ENERGY) {
			KahanV<R>::kadd(E, Ec, o.E);
			KahanV<R>::kadd(Eh, Ehc, o.Ehb);
		}
		if(SPLIT) {
#pragma unroll
			for(int k = 0; k < N_TERMS; k++) split[k] += o.split[k];
		}
	}
};

__device__ __forceinline__ void atomic_add_v4(float4 *p, const float4 &v) { atomicAdd(p, v); }
__device__ __forceinline__ void atomic_add_v4(double4_32a *p, const double4_32a &v) {
	atomicAdd(&p->x, v.x);
	atomicAdd(&p->y, v.y);
	atomicAdd(&p->z, v.z);
	atomicAdd(&p->w, v.w);
}

// ---------------------------------------------------------------- pair terms
//
// Hydrogen bonding, cross and coaxial stacking are products of a radial factor F(r) and up to six
// angular factors g_k(cos theta_k).  The six angles are the same for all three terms (only the
// sites differ: base sites, or stacking sites for coaxial stacking), each between a unit vector u
// and a unit vector v:
//     lane   u   v   cos      factors of HB, CRST, CXST
//      0     a1  b1  -u.v     theta1
//      1     b1  rd  -u.v     theta2, theta2, none
//      2     a1  rd  +u.v     theta3, theta3, none
//      3     a3  b3  +u.v     theta4
//      4     b3  rd  -u.v     theta7, theta7, theta6
//      5     a3  rd  +u.v     theta8, theta8, theta5
// (a: axes of p, b: axes of q, rd: unit vector from p's site to q's; coaxial stacking has theta5 on
// lane 4 and theta6 on lane 5).  With D = dg/dcos, a factor's share of the forces is F D prod g, the
// product over the other factors, along a vector of its own: on p's axis it turns, X = u x v; between
// the sites, u less its part along rd, over r.  So a term's angular factors are evaluated by eight
// lanes, one factor each by the same instructions, which hand each other their g.
//
// A block takes its pairs through four stages, each dealt to as many threads as it has work for, with
// what they pass on in shared memory:
//   1  screening: a thread per owned entry; pairs with live terms are queued, an item per term;
//   2  a thread per item: separation, site distance, radial factor;
//   3  eight lanes per item: the angular factors, each lane's vectors and their coefficients;
//   4  a thread per pair: the sums, forces and torques of both nucleotides into the pair's two slots.
// Why: one lane per pair was a chain of some 1,500 dependent instructions (nine angles one after the
// other), and since a chip full of such warps has nothing else to issue, the launch lasted as long as
// that chain.
template <typename R>
struct __align__(16) Angular {
	R a, b, t0, ts, tc;  // f4 (see f4_both); a = b = 0 with a support that covers every angle: 1
	R both;              // 1: f4(theta) + f4(pi - theta)
	R harm;              // strength of the coaxial theta1 harmonic beyond sb
	R pad;
};
template <typename R>
struct AngularTable {
	Angular<R> t[3][8];  // [term: 0 HB, 1 CRST, 2 CXST][lane]
};
template <typename R>
constexpr AngularTable<R> angular_table() {
	constexpr float A[OXM_N_F4] = OXM_F4_TABLE_A, B[OXM_N_F4] = OXM_F4_TABLE_B, T0[OXM_N_F4] = OXM_F4_TABLE_T0,
			TS[OXM_N_F4] = OXM_F4_TABLE_TS, TC[OXM_N_F4] = OXM_F4_TABLE_TC;
	// the f4 set of every factor (-1: none) and whether it enters as f4(theta) + f4(pi - theta)
	const int set[3][6] = {{OXM_F4_HB_T1, OXM_F4_HB_T2, OXM_F4_HB_T2, OXM_F4_HB_T4, OXM_F4_HB_T7, OXM_F4_HB_T7},
			{OXM_F4_CR_T1, OXM_F4_CR_T2, OXM_F4_CR_T2, OXM_F4_CR_T4, OXM_F4_CR_T7, OXM_F4_CR_T7},
			{OXM_F4_CX_T1, -1, -1, OXM_F4_CX_T4, OXM_F4_CX_T5, OXM_F4_CX_T5}};
	const int both[3][6] = {{0, 0, 0, 0, 0, 0}, {0, 0, 0, 1, 1, 1}, {0, 0, 0, 0, 1, 1}};
	AngularTable<R> r{};
	for(int m = 0; m < 3; m++)
		for(int l = 0; l < 8; l++) {
			const int i = l < 6 ? set[m][l] : -1;
			if(i < 0) r.t[m][l] = Angular<R>{R(0), R(0), R(0), R(16), R(32), R(0), R(0), R(0)};
			else
				r.t[m][l] = Angular<R>{R(A[i]), R(B[i]), R(T0[i]), R(TS[i]), R(TC[i]), R(both[m][l]),
						i == OXM_F4_CX_T1 ? R(OXM_CXST_THETA1_SA) : R(0), R(0)};
		}
	return r;
}
__device__ const AngularTable<float> g_angular_f = angular_table<float>();
__device__ const AngularTable<double> g_angular_d = angular_table<double>();
__device__ __forceinline__ const Angular<float> &angular_of(int term, int lane, float) { return g_angular_f.t[term][lane]; }
__device__ __forceinline__ const Angular<double> &angular_of(int term, int lane, double) { return g_angular_d.t[term][lane]; }

// f4_both (its FP32 form, theta = atan2(sin, cos)) with the factor's constants as values
template <typename R>
__device__ __forceinline__ void angular_factor(const Angular<R> &k, R c, R sn, R &f, R &fd) {
	const R t = m_atan2(sn, c), s2 = sn * sn;
	R tt0 = t - k.t0;
	const R m = tt0 < R(0) ? R(-1) : R(1);
	tt0 = m_fabs(tt0);
	R dsin;
	if(tt0 > k.ts) {
		f = k.b * (k.tc - tt0) * (k.tc - tt0);
		dsin = m * (R(2) * k.b) * (tt0 - k.tc) / sn;
	}
	else {
		f = R(1) - k.a * tt0 * tt0;
		dsin = s2 > R(1e-8) ? -m * (R(2) * k.a) * tt0 / sn : -m * (R(2) * k.a);
	}
	if(!(tt0 < k.tc)) f = dsin = R(0);
	if(k.harm != R(0)) {
		const R h = t - R(OXM_CXST_THETA1_SB);
		if(h >= R(0)) {
			f += k.harm * h * h;
			dsin += s2 > R(1e-8) ? R(2) * k.harm * h / sn : R(2) * k.harm;
		}
	}
	fd = -dsin;
}

// the same in FP64 at angle t, with the sine's square and inverse
__device__ __forceinline__ void angular_factor_fp64(const Angular<double> &k, double t, double s2, double inv, double &f, double &fd) {
	const double tt0 = t - k.t0, ad = fabs(tt0), far = k.tc - ad, at = s2 > 1e-8 ? inv : 1.0;
	double dsin = 0.0;  // -df/dt / sin
	f = 0.0;
	if(ad < k.tc) {
		const bool outer = ad > k.ts;
		f = outer ? k.b * far * far : 1.0 - k.a * ad * ad;
		// (on the axis itself |t - t0| / sin is 1 where t0 is 0 or pi)
		const double lin = 2.0 * (outer ? k.b * far * inv : k.a * (s2 > 1e-8 ? ad : 1.0) * at);
		dsin = copysign(lin, tt0);
	}
	if(k.harm != 0.0) {
		const double h = t - (double) OXM_CXST_THETA1_SB;
		if(h >= 0.0) {
			f += k.harm * h * h;
			dsin -= 2.0 * k.harm * (s2 > 1e-8 ? h : 1.0) * at;
		}
	}
	fd = dsin;
}

// Which terms of pair (p, q) can be non-zero: 1 hydrogen bonding, 2 cross stacking, 4 coaxial stacking.
// Distance windows (a little wider than the terms' own, for the plain FP32 separation) and the support
// of every angular factor in its cosine; the terms themselves are zero outside them.
template <typename R>
__device__ __forceinline__ int live_terms(const Nuc<R> &p, const Nuc<R> &q, const v3<R> &r) {
	constexpr R lo = R(0.9999), hi = R(1.0001);
	const v3<R> da = q.a1 - p.a1;
	const v3<R> rb = r + da * R(OXM_POS_BASE), rk = r + da * R(OXM_POS_STACK);
	const R b2 = dot(rb, rb), k2 = dot(rk, rk);
	const bool hb = p.btype + q.btype == 3 && b2 > lo * R(OXM_HYDR_RCLOW * OXM_HYDR_RCLOW) && b2 < hi * R(OXM_HYDR_RCHIGH * OXM_HYDR_RCHIGH);
	const bool cr = b2 > lo * R(OXM_CRST_RCLOW * OXM_CRST_RCLOW) && b2 < hi * R(OXM_CRST_RCHIGH * OXM_CRST_RCHIGH);
	const bool cx = k2 > lo * R(OXM_CXST_RCLOW * OXM_CXST_RCLOW) && k2 < hi * R(OXM_CXST_RCHIGH * OXM_CXST_RCHIGH);
	if(!(hb || cr || cx)) return 0;
	const R c1 = -dot(p.a1, q.a1), c4 = dot(p.a3, q.a3);
	int m = 0;
	if(hb || cr) {
		const v3<R> rd = rb * (R(1) / m_sqrt(b2));
		const R c2 = -dot(q.a1, rd), c3 = dot(p.a1, rd), c7 = -dot(q.a3, rd), c8 = dot(p.a3, rd);
		if(hb && f4_may(c1, OXM_F4_HB_T1) && f4_may(c2, OXM_F4_HB_T2) && f4_may(c3, OXM_F4_HB_T2) && f4_may(c4, OXM_F4_HB_T4) &&
				f4_may(c7, OXM_F4_HB_T7) && f4_may(c8, OXM_F4_HB_T7))
			m |= 1;
		// theta4, theta7, theta8 of cross stacking enter through f4(theta) + f4(pi - theta)
		if(cr && f4_may(c1, OXM_F4_CR_T1) && f4_may(c2, OXM_F4_CR_T2) && f4_may(c3, OXM_F4_CR_T2) &&
				(f4_may(c4, OXM_F4_CR_T4) || f4_may(-c4, OXM_F4_CR_T4)) && (f4_may(c7, OXM_F4_CR_T7) || f4_may(-c7, OXM_F4_CR_T7)) &&
				(f4_may(c8, OXM_F4_CR_T7) || f4_may(-c8, OXM_F4_CR_T7)))
			m |= 2;
	}
	if(cx && f4_may(c1, OXM_F4_CX_T1) && f4_may(c4, OXM_F4_CX_T4)) {
		const v3<R> rd = rk * (R(1) / m_sqrt(k2));
		const R c5 = dot(p.a3, rd), c6 = -dot(q.a3, rd);
		if((f4_may(c5, OXM_F4_CX_T5) || f4_may(-c5, OXM_F4_CX_T5)) && (f4_may(c6, OXM_F4_CX_T5) || f4_may(-c6, OXM_F4_CX_T5))) m |= 4;
	}
	return m;
}

constexpr int PAIR_CHUNK = 64;             // items taken through stages 2 to 4 at a time

// one item between the stages (an odd number of words apart: no bank conflicts)
template <typename R>
struct PairItem {
	R axes[12];            // a1, a3 of p; a1, a3 of q
	R rd[3], r, F, FD;     // site direction and distance (FP64: its inverse), radial factor and its derivative
	R d[6];                // centre separation, hi and lo
	R g[6];                // the angular factors
	// a vector and its coefficient: the torque axes X of lanes 0 and 3, the force directions of lanes
	// 1, 2, 4, 5, and the torque axes rd x u of the two of them that turn p
	R turn[2][4], push[4][4], twist[2][4];
	R pad;
};
static_assert(sizeof(PairItem<float>) == 63 * 4, "an odd number of words");

// stage 2 of item m of pair (i, j), term 0 hydrogen bonding, 1 cross stacking, 2 coaxial stacking
template <typename R, class Loader>
__device__ __forceinline__ void pair_radial(const DNA2Table<R> &P, const Loader &ld, int i, int j, int term, PairItem<R> &m) {
	using V4 = typename Vec4Of<R>::T;
	Nuc<R> p, q;
	V4 ph, pl, qh, ql;
	load_axes<Loader, R>(ld, i, P, p, ph, pl);
	load_axes<Loader, R>(ld, j, P, q, qh, ql);
	const Sep<R> d = ld.sep(ph, pl, qh, ql, P);
	const bool stack = term == 2;
	p.stack = p.a1 * R(OXM_POS_STACK), q.stack = q.a1 * R(OXM_POS_STACK);
	const v3<R> rs = stack ? site_vec(d, q.stack, p.stack) : site_vec(d, q.base, p.base);
	const R r = m_sqrt(dot(rs, rs));
	const R ir = R(1) / r;
	const v3<R> rd = rs * ir;
	R rl = R(0);
	const auto x = ld.refine(i, j);
	if constexpr(decltype(x)::on) rl = site_dist_remainder(d, p, x.lo(0), q, x.lo(1), stack, r);
	R F, FD;
	if(term == 0) {
		const R hbm = (abs(q.btype) >= 300 && abs(p.btype) >= 300) ? P.hb_multiplier : R(1);
		f1_both(P, r, OXM_F1_HB, q.type, p.type, F, FD, rl);
		F *= hbm;
		FD *= hbm;
	}
	else if(term == 1) f2_both(r, OXM_F2_CRST, F, FD, rl);
	else f2_both(r, OXM_F2_CXST, F, FD, rl);
	const v3<R> ax[4] = {p.a1, p.a3, q.a1, q.a3};
#pragma unroll
	for(int k = 0; k < 4; k++) m.axes[3 * k] = ax[k].x, m.axes[3 * k + 1] = ax[k].y, m.axes[3 * k + 2] = ax[k].z;
	m.rd[0] = rd.x, m.rd[1] = rd.y, m.rd[2] = rd.z;
	m.r = sizeof(R) == 8 ? ir : r, m.F = F, m.FD = FD;
	m.d[0] = d.hi.x, m.d[1] = d.hi.y, m.d[2] = d.hi.z, m.d[3] = d.lo.x, m.d[4] = d.lo.y, m.d[5] = d.lo.z;
}

// stage 3: eight lanes (the last two idle), this one the factor of its lane; the whole warp takes part
template <typename R>
__device__ __forceinline__ void pair_angles(int term, PairItem<R> &m) {
	const int sub = threadIdx.x & 7;
	const bool v_rd = sub != 0 && sub != 3;                                  // v is the site direction
	const bool u_q = sub == 1 || sub == (term == 2 ? 5 : 4);                 // u is an axis of q
	const R s = (u_q || sub == 0) ? R(-1) : R(1);
	const Angular<R> c = angular_of(term, sub, R(0));
	// u: a1 b1 a1 a3 b3 a3 (coaxial stacking: a3 b3 at the end); v: b1 rd rd b3 rd rd
	const R *pu = m.axes + (sub < 3 ? 0 : 3) + (u_q ? 6 : 0);
	const R *pv = v_rd ? m.rd : m.axes + (sub == 3 ? 9 : 6);
	const v3<R> u{pu[0], pu[1], pu[2]}, v{pv[0], pv[1], pv[2]};
	const v3<R> X = cross(u, v);
	const R cs = s * dot(u, v);
	R g, D;
	if constexpr(sizeof(R) == 8) {
		// one reciprocal square root for the sine and its inverse, and one angle for both directions: the
		// divisions and the second arctangent are half of a factor's operations on the FP64 pipe
		const R s2 = dot(X, X), inv = m_rsqrt(s2), theta = m_atan2(s2 > R(0) ? s2 * inv : R(0), cs);
		angular_factor_fp64(c, theta, s2, inv, g, D);
		if(c.both != R(0)) {
			R g2, D2;
			angular_factor_fp64(c, R(3.14159265358979323846) - theta, s2, inv, g2, D2);
			g += g2;
			D -= D2;
		}
	}
	else {
		const R sn = m_sqrt(dot(X, X));
		angular_factor(c, cs, sn, g, D);
		if(c.both != R(0)) {
			R g2, D2;
			angular_factor(c, -cs, sn, g2, D2);
			g += g2;
			D -= D2;
		}
	}
	// F g0 .. g5 with this lane's D in the place of its g, a product from the left
	R z = m.F;
#pragma unroll
	for(int l = 0; l < 6; l++) {
		const R gl = __shfl_sync(0xffffffffu, g, l, 8);
		z *= l == sub ? D : gl;
	}
	if(sub >= 6) return;
	m.g[sub] = g;
	if(!v_rd) {
		R *o = m.turn[sub == 0 ? 0 : 1];
		o[0] = X.x, o[1] = X.y, o[2] = X.z, o[3] = sub == 0 ? z : -z;
		return;
	}
	const v3<R> w = u_q ? u + v * cs : u - v * cs;
	R *o = m.push[sub < 3 ? sub - 1 : sub - 2];
	o[0] = w.x, o[1] = w.y, o[2] = w.z, o[3] = sizeof(R) == 8 ? (u_q ? z : -z) * m.r : (u_q ? z : -z) / m.r;
	if(!u_q) {
		const v3<R> y = cross(v, u);
		R *t = m.twist[sub < 3 ? 0 : 1];
		t[0] = y.x, t[1] = y.y, t[2] = y.z, t[3] = z;
	}
}

// The force on q's site and the torque on p (without its lever arm) of an evaluated item, and its
// energy: the sums in the order of hb_term, crst_term and cxst_term
template <typename R>
__device__ __forceinline__ R pair_sums(int term, const PairItem<R> &m, v3<R> &f, v3<R> &t) {
	R e = m.F, ed = m.FD;
#pragma unroll
	for(int l = 0; l < 6; l++) e *= m.g[l], ed *= m.g[l];
	auto vec = [](const R *o) { return v3<R>{o[0], o[1], o[2]}; };
	f = v3<R>{m.rd[0], m.rd[1], m.rd[2]} * -ed;
	// hydrogen bonding sums the torque of a3, b3 first, the others that of a1, b1
	const R *t0 = m.turn[term == 0 ? 1 : 0], *t1 = m.turn[term == 0 ? 0 : 1];
	t = vec(t0) * t0[3];
	if(term != 1) t += vec(t1) * t1[3];
	if(term != 2) {
#pragma unroll
		for(int k = 0; k < 2; k++) f += vec(m.push[k]) * m.push[k][3];
		t += vec(m.twist[0]) * m.twist[0][3];
	}
	if(term == 1) t += vec(t1) * t1[3];
#pragma unroll
	for(int k = 2; k < 4; k++) f += vec(m.push[k]) * m.push[k][3];
	t += vec(m.twist[1]) * m.twist[1][3];
	return e;
}

// Blocks of a group of 32 nucleotides: in FP64, where the groups of the systems it is used for do not
// fill the chip's pipes evenly, two (about 32 items each, the least that fills a warp of stages 2 and 4).
// With angular_factor_fp64, 4,000 duplex nucleotides: 55.7 -> 34.8 us.
template <typename R>
constexpr int PAIR_PARTS = sizeof(R) == 8 ? 2 : 1;

// Pair block b (TPB threads): the entries owned by G groups of 32 nucleotides, or its part of one group's,
// in the four stages above
template <typename R, class Loader, bool SPLIT, bool ENERGY, int G, int TPB>
__device__ __forceinline__ void pair_block(const ForceArgs &a, const Loader &ld, int b) {
	constexpr int PAIR_QUEUE = 7 * TPB;  // items waiting (a round of screening adds at most 3 x TPB)
	using V4 = typename Vec4Of<R>::T;
	__shared__ int2 queue[PAIR_QUEUE];  // partner; k | m << 8 | term << 16 | further term of the pair << 18 | i - first << 19
	__shared__ PairItem<R> item[PAIR_CHUNK];
	__shared__ int wcount[TPB / 32];
	const long long N = a.N;
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	constexpr int PARTS = PAIR_PARTS<R>;
	static_assert(PARTS == 1 || G == 1, "parts of one group");
	const int g0 = b / PARTS * G, first = g0 * PAIR_GROUP, groups = (a.N + PAIR_GROUP - 1) / PAIR_GROUP;
	int start[G + 1];  // the groups' entries, one after the other
	start[0] = 0;
#pragma unroll
	for(int g = 0; g < G; g++) start[g + 1] = start[g] + (g0 + g < groups ? a.own_n[g0 + g] : 0);
	V4 *res = reinterpret_cast<V4 *>(a.pt_res);
	const int lo = start[G] * (b % PARTS) / PARTS, hi = start[G] * (b % PARTS + 1) / PARTS;
	int n = 0;  // queued items (block-uniform)
	bool more = hi > lo;
	for(int r0 = lo; more; r0 += TPB) {
		// stage 1
		int mask = 0, i0 = 0;
		int2 it = make_int2(0, 0);
		const int r = r0 + (int) threadIdx.x;
		if(r < hi) {
			int g = 0;
#pragma unroll
			for(int u = 1; u < G; u++) g += r >= start[u];
			int base = 0;
#pragma unroll
			for(int u = 1; u < G; u++)
				if(g == u) base = start[u];
			it = a.own[(long long) (g0 + g) * PAIR_GROUP * a.pt_cap + (r - base)];
			i0 = first + g * PAIR_GROUP + (it.y >> 16);
			it.y &= 0xffff;
			const DNA2Table<R> &P = table_of<R>(a, a.sys ? a.sys[i0] : 0);
			Nuc<float> p, q;
			float4 ph, pl, qh, ql;
			if constexpr(sizeof(R) == 8) {
				const DNA2Table<float> B = ld.screen_box(P);
				ld.screen.axes(i0, p, ph, pl);
				ld.screen.axes(it.x, q, qh, ql);
				mask = live_terms(p, q, ld.screen.sep(ph, pl, qh, ql, B).plain());
			}
			else {
				load_axes<Loader, R>(ld, i0, P, p, ph, pl);
				load_axes<Loader, R>(ld, it.x, P, q, qh, ql);
				mask = live_terms(p, q, ld.sep(ph, pl, qh, ql, P).plain());
			}
		}
		int incl = __popc(mask);
#pragma unroll
		for(int off = 1; off < 32; off <<= 1) {
			const int u = __shfl_up_sync(0xffffffffu, incl, off);
			if(lane >= off) incl += u;
		}
		if(lane == 31) wcount[warp] = incl;
		__syncthreads();
		more = r0 + TPB < hi;
		int at = n + incl - __popc(mask);
#pragma unroll
		for(int w = 0; w < TPB / 32; w++) {
			if(w < warp) at += wcount[w];
			n += wcount[w];
		}
		for(int left = mask, k = 0; left; left &= left - 1, k++)
			queue[at + k] = make_int2(it.x, it.y | (__ffs(left) - 1) << 16 | (k > 0 ? 1 << 18 : 0) | (i0 - first) << 19);
		__syncthreads();
		if(more && n <= PAIR_QUEUE - 3 * TPB) continue;
		for(int c0 = 0; c0 < n;) {
			// the next chunk ends with a whole pair
			int c1 = min(n, c0 + PAIR_CHUNK);
			while(c1 < n && (queue[c1].y & (1 << 18))) c1--;
			for(int m = threadIdx.x; m < c1 - c0; m += TPB) {
				const int2 w = queue[c0 + m];
				const int i = first + (w.y >> 19);
				pair_radial<R, Loader>(table_of<R>(a, a.sys ? a.sys[i] : 0), ld, i, w.x, (w.y >> 16) & 3, item[m]);
			}
			__syncthreads();
			for(int m0 = warp * 4; m0 < c1 - c0; m0 += TPB / 8) {  // warp-uniform: four items at a time
				// (lanes without an item repeat the last one: the same values, written again)
				const int m = min(m0 + lane / 8, c1 - c0 - 1);
				pair_angles<R>((queue[c0 + m].y >> 16) & 3, item[m]);
			}
			__syncthreads();
			for(int m = threadIdx.x; m < c1 - c0; m += TPB) {
				const int2 w = queue[c0 + m];
				if(w.y & (1 << 18)) continue;  // taken with the pair's first item
				const int i = first + (w.y >> 19), j = w.x, k = w.y & 255, mj = (w.y >> 8) & 255;
				V4 fi, ti, fj, tj;
				fi.x = fi.y = fi.z = fi.w = ti.x = ti.y = ti.z = ti.w = R(0);
				fj = tj = fi;
				bool any = false;
				for(int v = m;;) {
					const PairItem<R> &x = item[v];
					const int term = (queue[c0 + v].y >> 16) & 3;
					v3<R> f, t;
					const R e = pair_sums<R>(term, x, f, t);
					if(e != R(0)) {
						any = true;
						const v3<R> a1{x.axes[0], x.axes[1], x.axes[2]};
						// the lever arm as the loaders form it
						const v3<R> arm = term == 2 ? a1 * R(OXM_POS_STACK) : sizeof(R) == 4 ? a1 * R(OXM_POS_BASE) :
								a1 * R(OXM_POS_STACK) * R((double) OXM_POS_BASE / (double) OXM_POS_STACK);
						const v3<R> T = t - cross(arm, f);
						// the potential is invariant under rigid rotations, so the torques balance:
						// T_j = -T_i + (r_j - r_i) x F_i, the cross product with error-free products
						const v3<R> c = cross_accurate(Sep<R>{v3<R>{x.d[0], x.d[1], x.d[2]}, v3<R>{x.d[3], x.d[4], x.d[5]}}, -f);
						fi.x -= f.x, fi.y -= f.y, fi.z -= f.z;
						fj.x += f.x, fj.y += f.y, fj.z += f.z;
						ti.x += T.x, ti.y += T.y, ti.z += T.z;
						tj.x += c.x - T.x, tj.y += c.y - T.y, tj.z += c.z - T.z;
						if(ENERGY) {
							fi.w += e;
							if(term == 0) ti.w += e;
						}
						if(SPLIT) atomicAdd(a.esplit + 8 * (a.sys ? a.sys[i] : 0) + (term == 0 ? T_HB : term == 1 ? T_CRST : T_CXST), (double) e);
					}
					if(++v >= c1 - c0 || !(queue[c0 + v].y & (1 << 18))) break;
				}
				if(!any) continue;
				fj.w = fi.w, tj.w = ti.w;
				res[2 * ((long long) k * N + i)] = fi;
				res[2 * ((long long) k * N + i) + 1] = ti;
				atomicOr(a.pt_live + (long long) (k >> 6) * N + i, 1ull << (k & 63));
				if(mj < 255) {  // (a missing position is flagged by the list build)
					res[2 * ((long long) mj * N + j)] = fj;
					res[2 * ((long long) mj * N + j) + 1] = tj;
					atomicOr(a.pt_live + (long long) (mj >> 6) * N + j, 1ull << (mj & 63));
				}
			}
			__syncthreads();
			c0 = c1;
		}
		n = 0;
	}
}

// Minimum resident blocks per SM asked of the register allocator for the bonded/pair kernel (80 registers).
// Its warps wait for one another's stages, so residency pays until registers spill.  5, 6, 7, 8 blocks, us per
// step at the blocks' sizes of launch_md_shape: 40,000 duplex nucleotides 40.9, 39.7, 40.5, 40.8; 160,000
// 128, 123.3, 124.6, 128.0; 250,000 strand nucleotides 105, 101.0, 99.2, 102.4; batch of 96 systems 88, 81.7, 84.7,
// 88.5.
// (with the edge blocks, whose registers would spill, 5)
constexpr int PAIR_MINB = 6;


// compensated sum over the K lanes of a group (TwoSum at every level); every lane of the group
// receives it
template <typename R, int K>
__device__ __forceinline__ R group_sum_comp(R s, R c) {
	R err = -c;
#pragma unroll
	for(int off = K / 2; off > 0; off >>= 1) {
		const R so = __shfl_xor_sync(0xffffffffu, s, off, K);
		const R eo = __shfl_xor_sync(0xffffffffu, err, off, K);
		const R t = s + so;
		const R bp = t - s;
		const R e2 = (s - (t - bp)) + (so - bp);
		s = t;
		err += eo + e2;
	}
	return s + err;
}

// Edge block b (use_edge): K lanes per nucleotide i take the entries of its full row and of its
// excluded-volume list whose partner j lies above i (by slot), so every unordered pair is
// evaluated once -- the pair-parallel scheme of the reference's use_edge kernels
// (CUDA_DNA.cuh:727-775), with a nucleotide's pairs kept on one lane group.  The partner's
// share goes to edge_acc[j] by atomic vector adds (force with energy, lab torque), the
// nucleotide's own share to edge_acc[i] after a compensated group sum; the non-bonded kernel
// gathers edge_acc.  The partner's Debye-Hueckel torque is its backbone offset times its force;
// the excluded volume's follows from the rigid-rotation balance T_j = -T_i + d x F_i (error-free
// products).  Atomic adds make the summation order, and so the last bits, vary from run to run.
template <typename R, class Loader, bool SPLIT, bool ENERGY, int K>
__device__ __forceinline__ void edge_block(const ForceArgs &a, const Loader &ld, int b) {
	using V4 = typename Vec4Of<R>::T;
	const long long N = a.N;
	const int sub = threadIdx.x % K;
	const int per_block = blockDim.x / K;
	const int first = b * per_block;
	const int i_raw = first + (int) threadIdx.x / K;
	const bool live = i_raw < a.N;
	const int i = live ? i_raw : a.N - 1;
	const int sy = a.sys ? a.sys[i] : 0;
	const DNA2Table<R> &P = table_of<R>(a, sy);
	Nuc<R> p;
	V4 ph, pl;
	load_full<Loader, R>(ld, i, P, p, ph, pl);
	SplitAcc<R, SPLIT, ENERGY> acc{};
	V4 *out = reinterpret_cast<V4 *>(a.edge_acc);
	auto partner = [&](int j, const v3<R> &fj, const v3<R> &tj, R e) {
		V4 f, t;
		f.x = fj.x, f.y = fj.y, f.z = fj.z, f.w = ENERGY ? e : R(0);
		t.x = tj.x, t.y = tj.y, t.z = tj.z, t.w = R(0);
		atomic_add_v4(out + 2 * (long long) j, f);
		atomic_add_v4(out + 2 * (long long) j + 1, t);
	};
	// Debye-Hueckel over the owned entries of the full row
	const int ndh = live ? min(a.nnb[i], a.max_nb) : 0;
	for(int k = sub; k < ndh; k += K) {
		const int j = a.nb[(long long) k * N + i];
		if(j < i) continue;
		Nuc<R> q;
		V4 qh, ql;
		load_dh<Loader, R>(ld, j, P, q, qh, ql);
		PairOut<R> o{};
		pair_dh<R, SPLIT>(P, p, q, ld.sep_soft(ph, pl, qh, ql, P).plain(), o);
		acc.add(o);
		if(o.F.x != R(0) || o.F.y != R(0) || o.F.z != R(0)) partner(j, -o.F, cross(q.back, -o.F), o.E);
	}
	// excluded volume over the owned centre-close pairs
	const int nev = live ? min(a.ev_n[i], a.ev_cap) : 0;
	for(int k = sub; k < nev; k += K) {
		const int j = a.ev_nb[(long long) k * N + i];
		if(j < i) continue;
		Nuc<R> q;
		V4 qh, ql;
		load_full<Loader, R>(ld, j, P, q, qh, ql);
		PairOut<R> o{};
		const Sep<R> sp = ld.sep(ph, pl, qh, ql, P);
		if constexpr(decltype(ld.refine(0, 0))::on) {
			if(!ev_contact(p, q, sp.plain())) continue;
			float3 t;
			const float4 fe = ev_pair_refined_call(ld.a1lo, ld.backlo, i, j, make_float4(sp.hi.x, sp.hi.y, sp.hi.z, 0.f),
					make_float4(sp.lo.x, sp.lo.y, sp.lo.z, 0.f), make_float4(p.back.x, p.back.y, p.back.z, 0.f),
					make_float4(p.base.x, p.base.y, p.base.z, 0.f), make_float4(p.a1.x, p.a1.y, p.a1.z, 0.f),
					make_float4(q.back.x, q.back.y, q.back.z, 0.f), make_float4(q.base.x, q.base.y, q.base.z, 0.f),
					make_float4(q.a1.x, q.a1.y, q.a1.z, 0.f), &t);
			o.F = v3<R>{fe.x, fe.y, fe.z};
			o.T = v3<R>{t.x, t.y, t.z};
			add_e<R, SPLIT>(o, T_NEXC, fe.w);
		}
		else {
			pair_ev<R, SPLIT>(p, q, sp, o);
		}
		if(o.F.x == R(0) && o.F.y == R(0) && o.F.z == R(0) && o.E == R(0)) continue;
		acc.add(o);
		partner(j, -o.F, cross_accurate(sp, o.F) - o.T, o.E);
	}
	if(SPLIT) {
#pragma unroll
		for(int k = 0; k < N_TERMS; k++) add_split(a.esplit, sy, k, live ? (double) acc.split[k] : 0.0);
	}
	const R fx = group_sum_comp<R, K>(acc.F.s.x, acc.F.c.x), fy = group_sum_comp<R, K>(acc.F.s.y, acc.F.c.y),
			fz = group_sum_comp<R, K>(acc.F.s.z, acc.F.c.z);
	const R tx = group_sum_comp<R, K>(acc.T.s.x, acc.T.c.x), ty = group_sum_comp<R, K>(acc.T.s.y, acc.T.c.y),
			tz = group_sum_comp<R, K>(acc.T.s.z, acc.T.c.z);
	const R e = ENERGY ? group_sum_comp<R, K>(acc.E, acc.Ec) : R(0);
	if(sub == 0 && live) partner(i, v3<R>{fx, fy, fz}, v3<R>{tx, ty, tz}, e);
}

// The bonded and the pair-term work are independent (both read the mirrors, each writes its own
// result buffers), so they share one launch: blocks 0 .. pair_blocks - 1 are pair blocks (the
// costliest, dispatched first), then the bonded blocks, which fill the tail, and with use_edge the
// edge blocks.  G: groups of 32 nucleotides per pair block.
template <typename R, class Loader, bool SPLIT, bool ENERGY, int G, int TPB = 128, bool EDGE = false, int K = 4>
__global__ void __launch_bounds__(TPB, sizeof(R) == 4 ? (EDGE ? 5 : PAIR_MINB) * 128 / TPB : 1) k_bonded_pairs(ForceArgs a, Loader ld, int pair_blocks) {
	// launched programmatically after the list build, it reads nothing before that is complete; nor may
	// the non-bonded kernel start before (it reads the lists and mirrors at once, and waits only for
	// these results)
	pdl_wait();
	pdl_trigger();
	const int b = blockIdx.x;
	const int bonded_blocks = (a.N + TPB / 2 - 1) / (TPB / 2);
	if(b < pair_blocks) pair_block<R, Loader, SPLIT, ENERGY, G, TPB>(a, ld, b);
	else if(!EDGE || b < pair_blocks + bonded_blocks) bonded_block<R, Loader, SPLIT, ENERGY, TPB>(a, ld, b - pair_blocks);
	else if constexpr(EDGE) edge_block<R, Loader, SPLIT, ENERGY, K>(a, ld, b - pair_blocks - bonded_blocks);
}

// What the bonded and pair blocks (and with use_edge the edge blocks) left for nucleotide i, added to
// acc by the K lanes of its group: the live pair slots dealt to the lanes, the 3' bond to lane 0 and the
// 5' bond to the next one.  (One group per nucleotide; the whole warp calls.)
template <typename R, bool ENERGY, int K, bool EDGE, class Acc>
__device__ __forceinline__ void gather_results(const ForceArgs &a, int i, int sub, bool live, int2 bonds, Acc &acc) {
	using V4 = typename Vec4Of<R>::T;
	const long long N = a.N;
	V4 bf, bt;
	const int lane5 = K > 1 ? 1 : 0;
	const bool three = sub == 0 && live && bonds.x >= 0, five = sub == lane5 && live && bonds.y >= 0;
	const V4 *bond_f = reinterpret_cast<const V4 *>(a.bond_f);
	auto add = [&](const V4 &f, const V4 &t, R s) {
		acc.F.add(v3<R>{s * f.x, s * f.y, s * f.z});
		acc.T.add(v3<R>{t.x, t.y, t.z});
		if(ENERGY) KahanV<R>::kadd(acc.E, acc.Ec, f.w);
	};
	// (issued before the mask is waited for)
	if(three) bf = bond_f[i], bt = reinterpret_cast<const V4 *>(a.bond_tp)[i];
	else if(five) bf = bond_f[bonds.y], bt = reinterpret_cast<const V4 *>(a.bond_tq)[bonds.y];
	for(int w = 0; w < (a.pt_cap + 63) / 64; w++) {
		unsigned long long m = 0ull;
		if(sub == 0 && live) {
			unsigned long long *at = a.pt_live + (long long) w * N + i;
			m = *at;
			if(m) *at = 0ull;  // for the next evaluation
		}
		m = __shfl_sync(0xffffffffu, m, 0, K);
		// lane l takes the live slots l, l + K, ..., the next one loaded before the current one
		// is added
		for(int u = 0; u < sub; u++) m &= m - 1ull;
		const V4 *base = reinterpret_cast<const V4 *>(a.pt_res) + 2 * ((long long) w * 64 * N + i);
		V4 f, t;
		auto next = [&]() {
			const V4 *q = base + 2 * (long long) (__ffsll((long long) m) - 1) * N;
			f = q[0];
			t = q[1];
#pragma unroll
			for(int u = 0; u < K; u++) m &= m - 1ull;
		};
		bool have = m != 0ull;
		if(have) next();
		while(have) {
			const V4 cf = f, ct = t;
			have = m != 0ull;
			if(have) next();
			add(cf, ct, R(1));
			if(ENERGY) KahanV<R>::kadd(acc.Eh, acc.Ehc, ct.w);
		}
	}
	if(three) add(bf, bt, R(-1));
	if(five) {
		if(lane5 == 0 && three) bf = bond_f[bonds.y], bt = reinterpret_cast<const V4 *>(a.bond_tq)[bonds.y];
		add(bf, bt, R(1));
	}
	if constexpr(EDGE) {
		// the Debye-Hueckel and excluded-volume sums, cleared for the next evaluation
		if(sub == 0 && live) {
			V4 *ea = reinterpret_cast<V4 *>(a.edge_acc) + 2 * (long long) i;
			add(ea[0], ea[1], R(1));
			V4 z;
			z.x = z.y = z.z = z.w = R(0);
			ea[0] = z;
			ea[1] = z;
		}
	}
}

// K lanes per nucleotide: lane l of a group takes entries l, l + K, ... of every term list, so a
// warp holds 32 / K nucleotides and all its lanes run the same term loop
// minimum resident blocks per SM asked of the register allocator for the non-bonded kernel
#ifndef OXGB_NB_MINB
#define OXGB_NB_MINB 8
#endif

template <typename R, class Loader, bool SPLIT, bool ENERGY, int K, bool EDGE = false>
__global__ void __launch_bounds__(128, 1) k_nonbonded_split(ForceArgs a, Loader ld) {
	using V4 = typename Vec4Of<R>::T;
	const long long N = a.N;
	const int sub = threadIdx.x % K;
	// one nucleotide per group of K lanes: the grid covers every nucleotide (nonbonded_blocks);
	// the lanes of a group past the last nucleotide still take part in the shuffles
	const int i_raw = (blockIdx.x * blockDim.x + threadIdx.x) / K;
	{
		const bool live = i_raw < a.N;
		const int i = live ? i_raw : a.N - 1;
		const int sy = a.sys ? a.sys[i] : 0;
		const DNA2Table<R> &P = table_of<R>(a, sy);
		Nuc<R> p;
		V4 ph, pl;
		load_full<Loader, R>(ld, i, P, p, ph, pl);
		SplitAcc<R, SPLIT, ENERGY> acc{};

		// Debye-Hueckel over the full Verlet row (use_edge: the edge blocks did it).  The lever
		// arm of every pair's torque on i is i's backbone offset, so the forces are summed
		// (compensated) and the torque is taken once from the sum.
		// (the engine's Debye-Hueckel rows where built: the full rows' entries whose backbone sites
		// are within the cutoff plus twice the skin)
		const int *dhr = a.dh_nb ? a.dh_nb : a.nb;
		const int ndh = (live && !EDGE) ? min(a.dh_nb ? a.dh_n[i] : a.nnb[i], a.max_nb) : 0;
		{
			KahanV<R> fdh{};
			// the next partner's data is loaded before this partner's arithmetic, and the index
			// after it one iteration earlier still: two gathers in flight per lane (measured with
			// the torque taken from the sum: -3.6 % per MD step at 40k, -4.7 % at 250k)
			Nuc<R> qn;
			V4 qhn, qln;
			int k = sub;
			if(k < ndh) load_dh<Loader, R>(ld, dhr[(long long) k * N + i], P, qn, qhn, qln);
			int jnn = (k + K < ndh) ? dhr[(long long) (k + K) * N + i] : 0;
			for(; k < ndh; k += K) {
				const v3<R> qback = qn.back;
				const bool qend = qn.is_end;
				const V4 qh = qhn, ql = qln;
				if(k + K < ndh) load_dh<Loader, R>(ld, jnn, P, qn, qhn, qln);
				if(k + 2 * K < ndh) jnn = dhr[(long long) (k + 2 * K) * N + i];
				v3<R> f;
				R e;
				if(dh_sites(P, ld.sep_soft(ph, pl, qh, ql, P).plain() + qback - p.back, p.is_end, qend, f, e)) {
					fdh.add(f);
					if(ENERGY) KahanV<R>::kadd(acc.E, acc.Ec, e);
					if(SPLIT) acc.split[T_DH] += e;
				}
			}
			const v3<R> fs{fdh.s.x - fdh.c.x, fdh.s.y - fdh.c.y, fdh.s.z - fdh.c.z};
			acc.F.add(fs);
			acc.T.add(cross(p.back, fs));
		}
		// excluded volume over centre-close pairs (use_edge: the edge blocks did it)
		const int nev = (live && !EDGE) ? min(a.ev_n[i], a.ev_cap) : 0;
		const DNA2Table<float> B = ld.screen_box(P);
		Nuc<float> sp;
		float4 sph, spl;
		ld.screen.full(i, sp, sph, spl);
		for(int k = sub; k < nev; k += K) {
			const int j = a.ev_nb[(long long) k * N + i];
			Nuc<float> sq;
			float4 sqh, sql;
			ld.screen.full(j, sq, sqh, sql);
			if(!ev_contact(sp, sq, ld.screen.sep(sph, spl, sqh, sql, B).plain())) continue;
			Nuc<R> q;
			V4 qh, ql;
			load_full<Loader, R>(ld, j, P, q, qh, ql);
			PairOut<R> o{};
			pair_ev<R, SPLIT>(p, q, ld.sep(ph, pl, qh, ql, P), o);
			acc.add(o);
		}
		// hydrogen bonding, cross and coaxial stacking: evaluated by the pair blocks of
		// k_bonded_pairs, the slots they wrote gathered here (the terms above read only the mirrors
		// and lists, complete before k_bonded_pairs started)
		pdl_wait();
		pdl_trigger();
		gather_results<R, ENERGY, K, EDGE>(a, i, sub, live, a.bonds[i], acc);
		if(SPLIT) {
#pragma unroll
			for(int k = 0; k < N_TERMS; k++) add_split(a.esplit, sy, k, live ? 0.5 * (double) acc.split[k] : 0.0);
		}

		const R fx = group_sum_comp<R, K>(acc.F.s.x, acc.F.c.x), fy = group_sum_comp<R, K>(acc.F.s.y, acc.F.c.y),
				fz = group_sum_comp<R, K>(acc.F.s.z, acc.F.c.z);
		const v3<R> tl{group_sum_comp<R, K>(acc.T.s.x, acc.T.c.x), group_sum_comp<R, K>(acc.T.s.y, acc.T.c.y),
				group_sum_comp<R, K>(acc.T.s.z, acc.T.c.z)};
		const R e = ENERGY ? group_sum_comp<R, K>(acc.E, acc.Ec) : R(0);
		const R eh = ENERGY ? group_sum_comp<R, K>(acc.Eh, acc.Ehc) : R(0);
		if(sub == 0 && live) {
			V4 fo, to;
			fo.x = fx;
			fo.y = fy;
			fo.z = fz;
			fo.w = e;
			to.x = dot(p.a1, tl);
			to.y = dot(p.a2, tl);
			to.z = dot(p.a3, tl);
			to.w = eh;
			reinterpret_cast<V4 *>(a.forces)[i] = fo;
			reinterpret_cast<V4 *>(a.torques)[i] = to;
		}
	}
}

// The FP32 engine's non-bonded kernel, K lanes per nucleotide as above.  Debye-Hueckel and the
// excluded-volume screen read the fixed-point sites: one 16-byte gather per Debye-Hueckel partner where
// the position pair and the backbone offset took three, two per excluded-volume entry instead of five,
// and an integer subtraction in the place of a compensated difference and its periodic image.  The
// separation is good to one unit, box / 2^32 (5e-8 in a box of 230, where the FP32 difference of the
// hi parts is off by up to 3.8e-6): Debye-Hueckel's force slope is below 0.1, and the screen's margin
// is 1e-4.  Contacts are evaluated from the mirrors, refined, as everywhere.
// A nucleotide's backbone site, as fixed point, or (FIXED = false), for boxes above FIXED_BOX_MAX, where the
// unit is coarser than FP32 separations, as hi + lo position and offset, as good at any size of the box.
template <bool FIXED>
struct Partner {
	int4 s;
	__device__ __forceinline__ void load(const ForceArgs &a, const SplitMixed &, int j) { s = __ldg(a.site_back + j); }
	__device__ __forceinline__ bool end() const { return s.w != 0; }
	__device__ __forceinline__ float3 sep(const SplitMixed &, const Partner &q, const DNA2Table<float> &) const {
		return make_float3((float) fixed_sep(q.s.x, s.x), (float) fixed_sep(q.s.y, s.y), (float) fixed_sep(q.s.z, s.z));
	}
};
template <>
struct Partner<false> {
	float4 h, l, b;
	__device__ __forceinline__ void load(const ForceArgs &, const SplitMixed &ld, int j) {
		h = __ldg(ld.hi + j), l = __ldg(ld.lo + j), b = __ldg(ld.fback + j);
	}
	__device__ __forceinline__ bool end() const { return b.w != 0.f; }
	__device__ __forceinline__ float3 sep(const SplitMixed &ld, const Partner &q, const DNA2Table<float> &P) const {
		const v3<float> d = ld.sep(h, l, q.h, q.l, P).plain();
		return make_float3(d.x + q.b.x - b.x, d.y + q.b.y - b.y, d.z + q.b.z - b.z);
	}
};

template <bool SPLIT, bool ENERGY, int K, int MINB = OXGB_NB_MINB, bool EDGE = false, bool FIXED = true>
__global__ void __launch_bounds__(128, MINB) k_nonbonded_mixed(ForceArgs a, SplitMixed ld) {
	const long long N = a.N;
	const int sub = threadIdx.x % K;
	const int i_raw = (blockIdx.x * blockDim.x + threadIdx.x) / K;
	const bool live = i_raw < a.N;  // (the lanes past the last nucleotide still take part in the shuffles)
	const int i = live ? i_raw : a.N - 1;
	const int sy = a.sys ? a.sys[i] : 0;
	const DNA2Table<float> &P = table_of<float>(a, sy);
	SplitAcc<float, SPLIT, ENERGY> acc{};
	const int2 bi = a.bonds[i];
	const float4 back = __ldg(ld.fback + i);
	if(!EDGE) {
		const float unit = P.fix_unit, unit_lo = P.fix_unit_lo, u2 = P.fix_unit2, u2_lo = P.fix_unit2_lo;
		Partner<FIXED> p;
		p.load(a, ld, i);
		// Debye-Hueckel (dh_sites) over its rows: the next partner's site is loaded before this
		// partner's arithmetic, and the index after it one iteration earlier still.  The lever arm of
		// every pair's torque on i is i's backbone offset, so the forces are summed (compensated) and
		// the torque is taken once from the sum.
		const int ndh = live ? min(a.dh_n[i], a.max_nb) : 0;
		{
			const DebyeF D(P);
			const float pcut = back.w != 0.f ? D.half : 1.f;
			KahanV<float> f{};
			Partner<FIXED> qn = p;
			int k = sub;
			if(k < ndh) qn.load(a, ld, a.dh_nb[(long long) k * N + i]);
			int jn = k + K < ndh ? a.dh_nb[(long long) (k + K) * N + i] : 0;
			for(; k < ndh; k += K) {
				const Partner<FIXED> q = qn;
				if(k + K < ndh) qn.load(a, ld, jn);
				if(k + 2 * K < ndh) jn = a.dh_nb[(long long) (k + 2 * K) * N + i];
				const float3 d = p.sep(ld, q, P);
				const float x = d.x, y = d.y, z = d.z, d2 = x * x + y * y + z * z, r2 = FIXED ? fmaf(d2, u2, d2 * u2_lo) : d2;
				if(r2 < D.rc2) {
					float e;
					const float s = D.force(r2, pcut * (q.end() ? D.half : 1.f), e);  // (fixed point: per unit, scaled after the sum)
					f.add(v3<float>{x * s, y * s, z * s});
					if(ENERGY) {
						KahanV<float>::kadd(acc.E, acc.Ec, e);
						if(SPLIT) acc.split[T_DH] += e;
					}
				}
			}
			const v3<float> fs{f.s.x - f.c.x, f.s.y - f.c.y, f.s.z - f.c.z};
			auto scaled = [&](const v3<float> &v) {
				return FIXED ? v3<float>{fmaf(v.x, unit, v.x * unit_lo), fmaf(v.y, unit, v.y * unit_lo), fmaf(v.z, unit, v.z * unit_lo)} : v;
			};
			acc.F.add(scaled(fs));
			acc.T.add(scaled(cross(v3<float>{back.x, back.y, back.z}, fs)));
		}
		// Excluded volume over its list: each window of 64 of the lane's entries is screened (a site
		// pair inside its cutoff, ev_contact: a few in a thousand entries); the pairs found are
		// evaluated refined after the window, and the others contribute nothing
		const int nev = live ? min(a.ev_n[i], a.ev_cap) : 0;
		const int4 pb = FIXED ? __ldg(a.site_base + i) : make_int4(0, 0, 0, 0);
		constexpr float m = 1.0001f;
		const float iu2 = 1.f / u2;
		const float t1 = float(EVc<1>::RC * EVc<1>::RC) * m * iu2, t2 = float(EVc<2>::RC * EVc<2>::RC) * m * iu2,
					t3 = float(EVc<3>::RC * EVc<3>::RC) * m * iu2;
		static_assert(EVc<3>::RC == EVc<4>::RC, "one threshold for backbone-base");
		auto sq = [](const int4 &p, const int4 &q) {
			const float x = (float) fixed_sep(q.x, p.x), y = (float) fixed_sep(q.y, p.y), z = (float) fixed_sep(q.z, p.z);
			return x * x + y * y + z * z;
		};
		for(int w0 = 0; w0 < nev; w0 += 64 * K) {
			const int wend = min(nev, w0 + 64 * K);
			unsigned long long stiff = 0ull;
			int n = 0;
			for(int k = w0 + sub; k < wend; k += K, n++) {
				const int j = a.ev_nb[(long long) k * N + i];
				if constexpr(FIXED) {
					const int4 qk = __ldg(a.site_back + j), qb = __ldg(a.site_base + j);
					if(sq(pb, qb) < t2 || sq(p.s, qb) < t3 || sq(pb, qk) < t3 || sq(p.s, qk) < t1) stiff |= 1ull << n;
				}
				else {
					Nuc<float> ni, nj;
					float4 h, l, qh, ql;
					ld.full(i, ni, h, l);
					ld.full(j, nj, qh, ql);
					if(ev_contact(ni, nj, ld.sep(h, l, qh, ql, P).plain())) stiff |= 1ull << n;
				}
			}
			while(stiff) {
				const int nn = __ffsll((long long) stiff) - 1;
				stiff &= stiff - 1ull;
				const int j = a.ev_nb[(long long) (w0 + sub + nn * K) * N + i];
				Nuc<float> p, q;
				float4 ph, pl, qh, ql;
				ld.full(i, p, ph, pl);
				ld.full(j, q, qh, ql);
				PairOut<float> o{};
				const Sep<float> sp = ld.sep(ph, pl, qh, ql, P);
				float3 t;
				const float4 fe = ev_pair_refined_call(
						ld.a1lo, ld.backlo, i, j, make_float4(sp.hi.x, sp.hi.y, sp.hi.z, 0.f), make_float4(sp.lo.x, sp.lo.y, sp.lo.z, 0.f),
						make_float4(p.back.x, p.back.y, p.back.z, 0.f), make_float4(p.base.x, p.base.y, p.base.z, 0.f),
						make_float4(p.a1.x, p.a1.y, p.a1.z, 0.f), make_float4(q.back.x, q.back.y, q.back.z, 0.f),
						make_float4(q.base.x, q.base.y, q.base.z, 0.f), make_float4(q.a1.x, q.a1.y, q.a1.z, 0.f), &t);
				o.F = v3<float>{fe.x, fe.y, fe.z};
				o.T = v3<float>{t.x, t.y, t.z};
				add_e<float, SPLIT>(o, T_NEXC, fe.w);
				acc.add(o);
			}
		}
		if(SPLIT) {
#pragma unroll
			for(int k = 0; k < N_TERMS; k++) add_split(a.esplit, sy, k, live ? 0.5 * (double) acc.split[k] : 0.0);
		}
	}
	// the axes of the body frame, before the wait for the pair and bond results
	const float4 x1 = __ldg(ld.fa1 + i), x3 = __ldg(ld.fa3 + i);
	pdl_wait();
	pdl_trigger();
	gather_results<float, ENERGY, K, EDGE>(a, i, sub, live, bi, acc);
	const float fx = group_sum_comp<float, K>(acc.F.s.x, acc.F.c.x), fy = group_sum_comp<float, K>(acc.F.s.y, acc.F.c.y),
			fz = group_sum_comp<float, K>(acc.F.s.z, acc.F.c.z);
	const v3<float> tl{group_sum_comp<float, K>(acc.T.s.x, acc.T.c.x), group_sum_comp<float, K>(acc.T.s.y, acc.T.c.y),
			group_sum_comp<float, K>(acc.T.s.z, acc.T.c.z)};
	const float e = ENERGY ? group_sum_comp<float, K>(acc.E, acc.Ec) : 0.f;
	const float eh = ENERGY ? group_sum_comp<float, K>(acc.Eh, acc.Ehc) : 0.f;
	if(sub == 0 && live) {
		const v3<float> a1{x1.x, x1.y, x1.z}, a3{x3.x, x3.y, x3.z};
		reinterpret_cast<float4 *>(a.forces)[i] = make_float4(fx, fy, fz, e);
		reinterpret_cast<float4 *>(a.torques)[i] = make_float4(dot(a1, tl), dot(cross(a3, a1), tl), dot(a3, tl), eh);
	}
}

// lanes per nucleotide in the non-bonded kernel
#ifndef OXGB_NB_LANES
#define OXGB_NB_LANES 4
#endif

int nonbonded_blocks(int N, int lanes) {
	const long long threads = (long long) (N > 0 ? N : 1) * lanes;
	return (int) ((threads + 127) / 128);
}

// The shapes of the MD step's force kernels (engine, mixed and float precision) the autotuner
// chooses among: the pair blocks' size (npw 32: three groups, 16: six, from PAIR_WIDE_N nucleotides on; below it one
// either way, see launch_md_shape), lanes per nucleotide in the non-bonded
// kernel and the resident blocks per SM its register cap asks for.  Shape 0 is the default, the
// best of hand sweeps on the 40k and 250k workloads.
struct ForceShapeDef {
	int npw, lanes, minb;
};
constexpr ForceShapeDef FORCE_SHAPES[] = {{32, 4, 8}, {16, 4, 8}, {32, 8, 6}, {16, 8, 6}, {32, 2, 8}, {16, 2, 8}};
constexpr int N_FORCE_SHAPES = sizeof(FORCE_SHAPES) / sizeof(FORCE_SHAPES[0]);

int force_shape_count() { return N_FORCE_SHAPES; }

void force_shape_of(int k, int *npw, int *lanes, int *minb) {
	const ForceShapeDef &d = FORCE_SHAPES[k >= 0 && k < N_FORCE_SHAPES ? k : 0];
	if(npw) *npw = d.npw;
	if(lanes) *lanes = d.lanes;
	if(minb) *minb = d.minb;
}

// External forces (CUDA_MD.cuh:97-555): one thread per nucleotide that has some, its records
// in order (deterministic), added to the force the pair kernels left; FP64 positions.
template <typename V4>
__global__ void k_external(ForceArgs a) {
	pdl_wait();
	pdl_trigger();
	const int k = blockIdx.x * blockDim.x + threadIdx.x;
	if(k >= a.ext_n) return;
	// records name caller's indices
	const int i = a.slot ? a.slot[a.ext_nuc[k]] : a.ext_nuc[k];
	const long long step = a.th.step_base ? *a.th.step_base + a.th.step_offset : 0;
	const double st = (double) step;
	const oxgb_ext_force *rec = reinterpret_cast<const oxgb_ext_force *>(a.ext_rec);
	const double4_32a r = a.posd[i];
	double fx = 0, fy = 0, fz = 0;
	for(int m = a.ext_off[k]; m < a.ext_off[k + 1]; m++) {
		const oxgb_ext_force &e = rec[m];
		switch(e.type) {
		case OXGB_FORCE_CONSTANT: {
			const double in = e.F0 + st * e.rate;
			double dx = e.dir[0], dy = e.dir[1], dz = e.dir[2];
			if(e.flags & 1) {
				dx -= r.x, dy -= r.y, dz -= r.z;
				const double n = sqrt(dx * dx + dy * dy + dz * dz);
				dx /= n, dy /= n, dz /= n;
			}
			fx += dx * in, fy += dy * in, fz += dz * in;
			break;
		}
		case OXGB_FORCE_MUTUAL_TRAP: {
			const double4_32a q = a.posd[a.slot ? a.slot[e.ref_particle] : e.ref_particle];
			double dx = q.x - r.x, dy = q.y - r.y, dz = q.z - r.z;
			if(e.flags & 1) {
				const double L = a.sys_box ? (double) a.sys_box[a.sys ? a.sys[i] : 0] : (double) a.box;
				dx -= rint(dx / L) * L, dy -= rint(dy / L) * L, dz -= rint(dz / L) * L;
			}
			const double d = sqrt(dx * dx + dy * dy + dz * dz);
			const double c = (d - (e.r0 + e.rate * st)) * (e.stiff + st * e.stiff_rate) / d;
			fx += dx * c, fy += dy * c, fz += dz * c;
			break;
		}
		case OXGB_FORCE_MOVING_TRAP:
		case OXGB_FORCE_LOWDIM_TRAP: {
			const double tx = e.pos0[0] + e.rate * st * e.dir[0], ty = e.pos0[1] + e.rate * st * e.dir[1],
						 tz = e.pos0[2] + e.rate * st * e.dir[2];
			const bool all = e.type == OXGB_FORCE_MOVING_TRAP;
			if(all || (e.flags & 2)) fx += -e.stiff * (r.x - tx);
			if(all || (e.flags & 4)) fy += -e.stiff * (r.y - ty);
			if(all || (e.flags & 8)) fz += -e.stiff * (r.z - tz);
			break;
		}
		case OXGB_FORCE_REPULSION_PLANE: {
			double p = e.position + e.rate * st;
			if(e.r0 > e.position && p > e.r0) p = e.r0;
			if(e.r0 < e.position && p < e.r0) p = e.r0;
			const double d = e.dir[0] * r.x + e.dir[1] * r.y + e.dir[2] * r.z + p;
			if(d < 0.0) fx += -d * e.stiff * e.dir[0], fy += -d * e.stiff * e.dir[1], fz += -d * e.stiff * e.dir[2];
			break;
		}
		case OXGB_FORCE_ATTRACTION_PLANE: {
			const double d = e.dir[0] * r.x + e.dir[1] * r.y + e.dir[2] * r.z + e.position;
			if(d < 0.0) fx += -d * e.stiff * e.dir[0], fy += -d * e.stiff * e.dir[1], fz += -d * e.stiff * e.dir[2];
			else fx += -e.stiff * e.dir[0], fy += -e.stiff * e.dir[1], fz += -e.stiff * e.dir[2];
			break;
		}
		case OXGB_FORCE_SPHERE:
		case OXGB_FORCE_SPHERE_SMOOTH: {
			// RepulsiveSphere / RepulsiveSphereSmooth::force (src/Forces/RepulsiveSphere*.cpp):
			// minimum image of r - centre
			const double L = a.sys_box ? (double) a.sys_box[a.sys ? a.sys[i] : 0] : (double) a.box;
			double dx = r.x - e.pos0[0], dy = r.y - e.pos0[1], dz = r.z - e.pos0[2];
			dx -= rint(dx / L) * L, dy -= rint(dy / L) * L, dz -= rint(dz / L) * L;
			const double m = sqrt(dx * dx + dy * dy + dz * dz);
			double c = 0.0;
			if(e.type == OXGB_FORCE_SPHERE) {
				const double R = e.r0 + e.rate * st;
				if(m > R && m < e.cutoff) c = -e.stiff * (1.0 - R / m);
			}
			else if(!(m < e.r0 || m > e.cutoff)) {
				if(m >= e.p1) c = -(e.stiff * 0.5 * exp((m - e.p1) / e.sigma)) / m;
				else c = -(e.stiff * m - e.stiff * 0.5 * exp(-(m - e.p1) / e.sigma)) / m;
			}
			fx += dx * c, fy += dy * c, fz += dz * c;
			break;
		}
		case OXGB_FORCE_LJ_WALL: {
			// LJWall::force (src/Forces/LJWall.cpp)
			const double x = e.dir[0] * r.x + e.dir[1] * r.y + e.dir[2] * r.z + e.position;
			const double y = x / e.sigma;
			if(y <= e.cutoff) {
				const double lj = pow(y, (double) -e.n);
				const double c = 4.0 * e.n * e.stiff * (2.0 * lj * lj - lj) / x;
				fx += e.dir[0] * c, fy += e.dir[1] * c, fz += e.dir[2] * c;
			}
			break;
		}
		case OXGB_FORCE_CENTRAL: {
			// GenericCentralForce::force, force_type = gravity (src/Forces/GenericCentralForce.cpp)
			const double dx = e.pos0[0] - r.x, dy = e.pos0[1] - r.y, dz = e.pos0[2] - r.z;
			const double d2 = dx * dx + dy * dy + dz * dz;
			if(!(d2 < e.p1 * e.p1) && !(e.p2 > 0.0 && d2 > e.p2 * e.p2)) {
				const double c = e.F0 / sqrt(d2);
				fx += dx * c, fy += dy * c, fz += dz * c;
			}
			break;
		}
		case OXGB_FORCE_REPULSION_PLANE_MOVING: {
			// RepulsionPlaneMoving::force (src/Forces/RepulsionPlaneMoving.cpp), one reference particle
			const double4_32a q = a.posd[a.slot ? a.slot[e.ref_particle] : e.ref_particle];
			const double x = (r.x - q.x) * e.dir[0] + (r.y - q.y) * e.dir[1] + (r.z - q.z) * e.dir[2];
			const double c = -e.stiff * fmin(x, 0.0);
			fx += e.dir[0] * c, fy += e.dir[1] * c, fz += e.dir[2] * c;
			break;
		}
		case OXGB_FORCE_LJ_CONE: {
			// LJCone::force (src/Forces/LJCone.cpp): apex pos0, axis dir, half-angle p1
			const double vx = r.x - e.pos0[0], vy = r.y - e.pos0[1], vz = r.z - e.pos0[2];
			const double along = vx * e.dir[0] + vy * e.dir[1] + vz * e.dir[2];
			const double wx = e.dir[0] * along - vx, wy = e.dir[1] * along - vy, wz = e.dir[2] * along - vz;
			const double from_axis = sqrt(wx * wx + wy * wy + wz * wz);
			const double x = along * sin(e.p1) - from_axis * cos(e.p1);
			const double y = x / e.sigma;
			if(y <= e.cutoff) {
				const double C = from_axis * tan(e.p1);
				double nx = (along + C) * e.dir[0] - vx, ny = (along + C) * e.dir[1] - vy, nz = (along + C) * e.dir[2] - vz;
				const double nn = sqrt(nx * nx + ny * ny + nz * nz);
				nx /= nn, ny /= nn, nz /= nn;
				const double lj = pow(y, (double) -e.n);
				const double c = 4.0 * e.n * e.stiff * (2.0 * lj * lj - lj) / x;
				fx += nx * c, fy += ny * c, fz += nz * c;
			}
			break;
		}
		case OXGB_FORCE_TWIST: {
			// ConstantRateTorque::force (src/Forces/ConstantRateTorque.cpp): the trap pos0 rotated
			// about the axis dir through the centre v1 by F0 + rate step radians (Rodrigues'
			// matrix), the pull masked component-wise by v2
			const double t = e.F0 + e.rate * st;
			const double sn = sin(t), cs = cos(t), oc = 1.0 - cs;
			const double ax = e.dir[0], ay = e.dir[1], az = e.dir[2];
			const double ux = e.pos0[0] - e.v1[0], uy = e.pos0[1] - e.v1[1], uz = e.pos0[2] - e.v1[2];
			const double tx = (ax * ax * oc + cs) * ux + (ax * ay * oc - az * sn) * uy + (ax * az * oc + ay * sn) * uz + e.v1[0];
			const double ty = (ax * ay * oc + az * sn) * ux + (ay * ay * oc + cs) * uy + (ay * az * oc - ax * sn) * uz + e.v1[1];
			const double tz = (ax * az * oc - ay * sn) * ux + (ay * az * oc + ax * sn) * uy + (az * az * oc + cs) * uz + e.v1[2];
			fx += -e.stiff * (r.x - tx) * e.v2[0];
			fy += -e.stiff * (r.y - ty) * e.v2[1];
			fz += -e.stiff * (r.z - tz) * e.v2[2];
			break;
		}
		case OXGB_FORCE_ELLIPSOID: {
			// RepulsiveEllipsoid::force (src/Forces/RepulsiveEllipsoid.cpp): pushed towards the
			// centre unless inside r_2 and outside r_1
			const double L = a.sys_box ? (double) a.sys_box[a.sys ? a.sys[i] : 0] : (double) a.box;
			double dx = r.x - e.pos0[0], dy = r.y - e.pos0[1], dz = r.z - e.pos0[2];
			dx -= rint(dx / L) * L, dy -= rint(dy / L) * L, dz -= rint(dz / L) * L;
			const double in = dx * dx / (e.v2[0] * e.v2[0]) + dy * dy / (e.v2[1] * e.v2[1]) + dz * dz / (e.v2[2] * e.v2[2]);
			const double out = dx * dx / (e.v1[0] * e.v1[0]) + dy * dy / (e.v1[1] * e.v1[1]) + dz * dz / (e.v1[2] * e.v1[2]);
			if(!(in < 1.0 && out > 1.0)) {
				const double m = sqrt(dx * dx + dy * dy + dz * dz);
				fx += -e.stiff * dx / m, fy += -e.stiff * dy / m, fz += -e.stiff * dz / m;
			}
			break;
		}
		case OXGB_FORCE_COM: {
			// COMForce::force (src/Forces/COMForce.cpp): centres of mass of group n (com_list) and
			// of group ref_particle (ref_list) from the unwrapped FP64 positions
			double c[2][3] = {{0, 0, 0}, {0, 0, 0}};
			int cnt[2];
			const int gs[2] = {e.n, e.ref_particle};
			for(int w = 0; w < 2; w++) {
				const int g0 = a.grp_off[gs[w]], g1 = a.grp_off[gs[w] + 1];
				cnt[w] = g1 - g0;
				for(int u = g0; u < g1; u++) {
					const double4_32a q = a.posd[a.slot ? a.slot[a.grp_mem[u]] : a.grp_mem[u]];
					c[w][0] += q.x, c[w][1] += q.y, c[w][2] += q.z;
				}
				for(int d = 0; d < 3; d++) c[w][d] /= (double) cnt[w];
			}
			const double dx = c[1][0] - c[0][0], dy = c[1][1] - c[0][1], dz = c[1][2] - c[0][2];
			const double m = sqrt(dx * dx + dy * dy + dz * dz);
			const double f = (m - (e.r0 + e.rate * st)) * e.stiff / (double) cnt[0] / m;
			fx += dx * f, fy += dy * f, fz += dz * f;
			break;
		}
		case OXGB_FORCE_YUKAWA_SPHERE: {
			// YukawaSphere::force (src/Forces/YukawaSphere.cpp): screened repulsion from the inside
			// of a sphere of radius r0, with a WCA core near its surface
			const double L = a.sys_box ? (double) a.sys_box[a.sys ? a.sys[i] : 0] : (double) a.box;
			double dx = r.x - e.pos0[0], dy = r.y - e.pos0[1], dz = r.z - e.pos0[2];
			dx -= rint(dx / L) * L, dy -= rint(dy / L) * L, dz -= rint(dz / L) * L;
			const double m = sqrt(dx * dx + dy * dy + dz * dz);
			const double sd = e.r0 - m;
			if(sd < e.cutoff) {
				double c = e.F0 * exp(-sd / e.p2) * (1.0 / (sd * e.p2) + 1.0 / (sd * sd));
				if(sd < e.p1) {
					const double w = pow(e.sigma / sd, 6.0);
					c += 4.0 * e.stiff * e.n * (2.0 * w * w - w) / sd;
				}
				fx += -dx / m * c, fy += -dy / m * c, fz += -dz / m * c;
			}
			break;
		}
		case OXGB_FORCE_SPHERE_MOVING: {
			// RepulsiveSphereMoving::force (src/Forces/RepulsiveSphereMoving.cpp): WCA (the
			// 2x-x form with x = 2, sigma = 1, eps = stiff) of the gap to a growing sphere whose
			// centre moves from v1 to v2 over p1 steps
			double t = 0.0;
			if(e.p1 > 0.0) t = fmin(fmax(st / floor(e.p1), 0.0), 1.0);
			const double cx = e.v1[0] + (e.v2[0] - e.v1[0]) * t, cy = e.v1[1] + (e.v2[1] - e.v1[1]) * t,
						 cz = e.v1[2] + (e.v2[2] - e.v1[2]) * t;
			const double L = a.sys_box ? (double) a.sys_box[a.sys ? a.sys[i] : 0] : (double) a.box;
			double dx = r.x - cx, dy = r.y - cy, dz = r.z - cz;
			dx -= rint(dx / L) * L, dy -= rint(dy / L) * L, dz -= rint(dz / L) * L;
			const double m = sqrt(dx * dx + dy * dy + dz * dz);
			const double g = m - (e.r0 + e.rate * st);
			if(!(g >= e.cutoff) && m > 0.0 && g < 1.4142135623730951) {
				const double gs = g > 1e-9 ? g : 1e-9;
				const double A = 1.0 / (gs * gs);
				const double c = 8.0 * e.stiff * (2.0 * A - 1.0) * A / gs / m;
				fx += dx * c, fy += dy * c, fz += dz * c;
			}
			break;
		}
		default:
			break;
		}
	}
	V4 *F = reinterpret_cast<V4 *>(a.forces);
	V4 f = F[i];
	f.x += fx;
	f.y += fy;
	f.z += fz;
	F[i] = f;
}

// ====================================================================== reference layout
//
// K lanes per nucleotide over its row of the neighbour matrix, every pair from both ends (the rows are
// full, and a partner's share would need atomics).  A lane builds its partner's frame from the quaternion
// (two 16-byte gathers per partner), evaluates Debye-Hueckel, screens the excluded volume (evaluated in
// the rare case of a contact) and the pair terms; pairs with live terms go to the warp's queue, an item
// per term, which the warp takes through the stages of the pair blocks: a lane per item, then eight lanes
// per item.  The block's bonds, both sides of each nucleotide, are evaluated by two full warps, stacking by
// one and FENE with the excluded volume by the other.  Sums are compensated and their order is fixed.
//
// Latency of the dependent chains bounds it.  40,000 duplex nucleotides: 65 us per call, 43 M warp
// instructions; with a warp per nucleotide, each pair's terms on the lane that found it and the two bonds
// on two lanes, where most lanes waited for the few on a long branch, 371 us.  Error of the forces against
// 64 bits (24 states of 12,000 duplex nucleotides): 1.350e-6, that kernel's 1.353e-6.
constexpr int REF_QUEUE = 64 + 3 * 32, REF_CHUNK = 16;

// the plain excluded volume of a pair with a site pair in contact: force and torque on p, energy (rare,
// out of line: the loop keeps its registers)
__device__ __noinline__ float4 ev_pair_call(v3<float> r, v3<float> pa1, v3<float> pback, v3<float> qa1, v3<float> qback, float3 *T) {
	Nuc<float> p, q;
	p.base = pa1 * float(OXM_POS_BASE), p.back = pback;
	q.base = qa1 * float(OXM_POS_BASE), q.back = qback;
	PairOut<float> o{};
	pair_ev<float, false>(p, q, Sep<float>{r, v3<float>{0.f, 0.f, 0.f}}, o);
	*T = make_float3(o.T.x, o.T.y, o.T.z);
	return make_float4(o.F.x, o.F.y, o.F.z, o.E);
}

template <int K>
__global__ void __launch_bounds__(128, 4) k_forces_reference(RefArgs a) {
	constexpr int NB = 128 / K, NW = 32 / K;  // nucleotides of a block, of a warp
	__shared__ int2 queues[4][REF_QUEUE];      // partner; term | nucleotide of the warp << 2
	__shared__ PairItem<float> items[4][REF_CHUNK];
	__shared__ float bond[2][2 * NB][7];       // [stacking, backbone][nucleotide and side]: force, torque, energy
	const LoadRef ld{a.pos, a.quat};
	const DNA2Table<float> &P = *a.table;
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = threadIdx.x % K;
	const int first = blockIdx.x * NB, wfirst = first + warp * NW;
	const int i_raw = first + (int) threadIdx.x / K;
	const bool live = i_raw < a.N;
	const int i = live ? i_raw : a.N - 1;

	// the block's bonds: side 0 of nucleotide u its 3' bond (u is p), side 1 its 5' bond (u is q)
	if(warp < 2 && lane < 2 * NB) {
		const int u = first + (lane >> 1), side = lane & 1;
		const int2 bu = u < a.N ? a.bonds[u] : make_int2(-1, -1);
		const int p = side ? bu.y : u, q = side ? u : bu.x;
		float *out = bond[warp][lane];
#pragma unroll
		for(int k = 0; k < 7; k++) out[k] = 0.f;
		if(p >= 0 && q >= 0) {
			Nuc<float> np, nq;
			float4 ph, pl, qh, ql;
			ld.load(p, P, make_int2(0, 0), np, ph, pl);
			ld.load(q, P, make_int2(0, 0), nq, qh, ql);
			BondOut<float> o;
			o.f = o.tp = o.tq = v3<float>{0.f, 0.f, 0.f};
			o.split[0] = o.split[1] = o.split[2] = 0.f;
			if(warp == 0) bonded_stacking(P, np, nq, ld.diff(ph, pl, qh, ql), o);
			else if(!bonded_backbone(P, np, nq, ld.diff(ph, pl, qh, ql), o)) atomicOr(a.status, OXGB_ERR_FENE);
			const float s = side ? 1.f : -1.f;
			const v3<float> t = side ? o.tq : o.tp;
			out[0] = s * o.f.x, out[1] = s * o.f.y, out[2] = s * o.f.z;
			out[3] = t.x, out[4] = t.y, out[5] = t.z;
			out[6] = o.split[0] + o.split[1] + o.split[2];
		}
	}

	Nuc<float> p;
	float4 ph, pl;
	const int2 bi = a.bonds[i];
	ld.load(i, P, bi, p, ph, pl);
	SplitAcc<float, false, true> acc{};
	KahanV<float> dh{};
	const DebyeF D(P);
	const float pcut = p.is_end ? D.half : 1.f;
	int2 *queue = queues[warp];
	PairItem<float> *item = items[warp];
	int n = 0;  // queued items (warp-uniform)
	// stages 2 to 4 of all queued items; the first lane of a nucleotide adds its items in order
	auto drain = [&]() {
		__syncwarp();
		for(int c0 = 0; c0 < n; c0 += REF_CHUNK) {
			const int m = min(n - c0, REF_CHUNK);
			if(lane < m) {
				const int2 w = queue[c0 + lane];
				pair_radial<float, LoadRef>(P, ld, wfirst + (w.y >> 2), w.x, w.y & 3, item[lane]);
			}
			__syncwarp();
			for(int m0 = 0; m0 < m; m0 += 4) {
				const int v = min(m0 + lane / 8, m - 1);
				pair_angles<float>(queue[c0 + v].y & 3, item[v]);
				__syncwarp();
			}
			// the sums of an item by a lane, over the item's first words
			if(lane < m) {
				const int term = queue[c0 + lane].y & 3;
				PairItem<float> &x = item[lane];
				v3<float> f, t;
				const float e = pair_sums<float>(term, x, f, t);
				const v3<float> T = t - cross(v3<float>{x.axes[0], x.axes[1], x.axes[2]} * (term == 2 ? float(OXM_POS_STACK) : float(OXM_POS_BASE)), f);
				const bool on = e != 0.f;
				float *o = x.axes;
				o[0] = on ? -f.x : 0.f, o[1] = on ? -f.y : 0.f, o[2] = on ? -f.z : 0.f;
				o[3] = on ? T.x : 0.f, o[4] = on ? T.y : 0.f, o[5] = on ? T.z : 0.f;
				o[6] = e;
			}
			__syncwarp();
			for(int v = 0; v < m; v++) {
				const int2 w = queue[c0 + v];
				if((w.y >> 2) == lane / K && sub == v % K) {
					const float *o = item[v].axes;
					acc.F.add(v3<float>{o[0], o[1], o[2]});
					acc.T.add(v3<float>{o[3], o[4], o[5]});
					KahanV<float>::kadd(acc.E, acc.Ec, o[6]);
					if((w.y & 3) == 0) KahanV<float>::kadd(acc.Eh, acc.Ehc, o[6]);
				}
			}
			__syncwarp();
		}
		n = 0;
	};
	const int nn = live ? a.nnb[i] : 0;
	if(nn > a.max_nb && sub == 0) atomicOr(a.status, OXGB_ERR_NEIGH_OVERFLOW);
	const int nlim = min(nn, a.max_nb);
	const long long row = (long long) i * a.nb_stride_i;
	int longest = nlim;
#pragma unroll
	for(int off = 16; off >= K; off >>= 1) longest = max(longest, __shfl_xor_sync(0xffffffffu, longest, off));
	for(int k0 = 0; k0 < longest; k0 += K) {  // warp-uniform
		const int k = k0 + sub;
		int j = -1, mask = 0;
		if(k < nlim) j = a.nb[row + (long long) k * a.nb_stride_k];
		if(j >= 0 && j != i && j != bi.x && j != bi.y) {
			Nuc<float> q;
			float4 qh, ql;
			// (only Debye-Hueckel's end charges need a partner's bonds)
			ld.load(j, P, a.bonds[j], q, qh, ql);
			const v3<float> r = ld.sep(ph, pl, qh, ql, P).hi;
			if(dot(r, r) < P.rcut2) {
				const v3<float> rb = r + q.back - p.back;
				const float rb2 = dot(rb, rb);
				if(rb2 < D.rc2) {
					float e;
					dh.add(rb * D.force(rb2, pcut * (q.is_end ? D.half : 1.f), e));
					KahanV<float>::kadd(acc.E, acc.Ec, e);
				}
				if(ev_contact(p, q, r)) {
					float3 t;
					const float4 fe = ev_pair_call(r, p.a1, p.back, q.a1, q.back, &t);
					acc.F.add(v3<float>{fe.x, fe.y, fe.z});
					acc.T.add(v3<float>{t.x, t.y, t.z});
					KahanV<float>::kadd(acc.E, acc.Ec, fe.w);
				}
				mask = live_terms(p, q, r);
			}
		}
		// the round's items, in the lanes' order
		if(__any_sync(0xffffffffu, mask != 0)) {
			int incl = __popc(mask);
#pragma unroll
			for(int off = 1; off < 32; off <<= 1) {
				const int u = __shfl_up_sync(0xffffffffu, incl, off);
				if(lane >= off) incl += u;
			}
			int at = n + incl - __popc(mask);
			for(int left = mask; left; left &= left - 1) queue[at++] = make_int2(j, (__ffs(left) - 1) | (lane / K) << 2);
			n += __shfl_sync(0xffffffffu, incl, 31);
			if(n > REF_QUEUE - 3 * 32) drain();
		}
	}
	drain();
	const v3<float> fs{dh.s.x - dh.c.x, dh.s.y - dh.c.y, dh.s.z - dh.c.z};
	acc.F.add(fs);
	acc.T.add(cross(p.back, fs));
	__syncthreads();
	if(sub < 2) {
#pragma unroll
		for(int part = 0; part < 2; part++) {
			const float *o = bond[part][2 * ((int) threadIdx.x / K) + sub];
			acc.F.add(v3<float>{o[0], o[1], o[2]});
			acc.T.add(v3<float>{o[3], o[4], o[5]});
			KahanV<float>::kadd(acc.E, acc.Ec, o[6]);
		}
	}
	const float fx = group_sum_comp<float, K>(acc.F.s.x, acc.F.c.x), fy = group_sum_comp<float, K>(acc.F.s.y, acc.F.c.y),
			fz = group_sum_comp<float, K>(acc.F.s.z, acc.F.c.z);
	const v3<float> tl{group_sum_comp<float, K>(acc.T.s.x, acc.T.c.x), group_sum_comp<float, K>(acc.T.s.y, acc.T.c.y),
			group_sum_comp<float, K>(acc.T.s.z, acc.T.c.z)};
	const float e = group_sum_comp<float, K>(acc.E, acc.Ec), eh = group_sum_comp<float, K>(acc.Eh, acc.Ehc);
	if(sub == 0 && live) {
		float4 fo = a.forces[i], to = a.torques[i];
		fo.x += fx, fo.y += fy, fo.z += fz, fo.w += e;
		// body frame: components along a1, a2, a3
		to.x += dot(p.a1, tl), to.y += dot(p.a2, tl), to.z += dot(p.a3, tl), to.w = eh;
		a.forces[i] = fo;
		a.torques[i] = to;
	}
}

cudaError_t launch_forces_reference_layout(const RefArgs &a, cudaStream_t s) {
	// as many lanes per nucleotide as one resident wave of blocks holds (4 of 128 threads on each of 152
	// SMs): more lanes shorten the row loops, a second wave doubles the time.  32 / 16 / 8 lanes, us per
	// call: 1,000 nucleotides 10.3 / 12.3 / 12.3, 2,400: 12.3 / 12.3 / 14.3, 4,000: 18.5 / 14.4 / 14.4,
	// 6,000: 26.6 / 22.1 / 16.4, 40,000: 137 / 101 / 65.
	constexpr int wave = 152 * 4 * 128;
	if((long long) a.N * 32 <= wave) k_forces_reference<32><<<(a.N + 3) / 4, 128, 0, s>>>(a);
	else if((long long) a.N * 16 <= wave) k_forces_reference<16><<<(a.N + 7) / 8, 128, 0, s>>>(a);
	else k_forces_reference<8><<<(a.N + 15) / 16, 128, 0, s>>>(a);
	return cudaGetLastError();
}

template <typename R, class Loader, bool SPLIT, bool ENERGY, int G = 1, int K = OXGB_NB_LANES, int NBMINB = OXGB_NB_MINB,
		bool EDGE = false, int TPB = 128>
static void launch_split_t(const ForceArgs &a, Loader ld, cudaStream_t s) {
	const int tpb = 128;
	const int blocks = a.N > 0 ? (a.N + TPB / 2 - 1) / (TPB / 2) : 1;
	// pair blocks of G groups of 32 nucleotides, then one bonded block per TPB / 2 nucleotides, then
	// (use_edge) one edge block per TPB / K nucleotides
	const int pair_blocks = (a.N + PAIR_GROUP * G - 1) / (PAIR_GROUP * G) * PAIR_PARTS<R>;
	const int edge_blocks = EDGE ? (int) (((long long) a.N * K + TPB - 1) / TPB) : 0;
	launch_after(k_bonded_pairs<R, Loader, SPLIT, ENERGY, G, TPB, EDGE, EDGE ? K : 4>, dim3(pair_blocks + blocks + edge_blocks), dim3(TPB), 0, s, a, ld,
			pair_blocks);
	// the non-bonded kernel starts its Debye-Hueckel and excluded-volume work while the tail of
	// the bonded and pair blocks runs; the external forces follow it the same way
	auto nonbonded = [&] {
		if constexpr(sizeof(R) == 4 && EDGE) return &k_nonbonded_mixed<SPLIT, ENERGY, K, NBMINB, EDGE>;
		else if constexpr(sizeof(R) == 4)
			return a.site_back ? &k_nonbonded_mixed<SPLIT, ENERGY, K, NBMINB> : &k_nonbonded_mixed<SPLIT, ENERGY, K, NBMINB, false, false>;
		else return &k_nonbonded_split<R, Loader, SPLIT, ENERGY, K, EDGE>;
	}();
	launch_after(nonbonded, dim3(nonbonded_blocks(a.N, K)), dim3(tpb), 0, s, a, ld);
	if(a.ext_n > 0) launch_after(k_external<typename Vec4Of<R>::T>, dim3((a.ext_n + tpb - 1) / tpb), dim3(tpb), 0, s, a);
}

// The MD step's kernels (mixed / float engine) in shape k of FORCE_SHAPES.  A pair block takes one group of
// 32 nucleotides while that leaves the chip a few blocks per SM, three (shapes of 32) or six (16) where there
// are more groups than run at a time: strands have few live pairs, and a block with a handful is all latency;
// duplexes lose little, since three groups' items still go through the stages together.  1, 2, 3, 4, 6 groups, us
// per step: 40,000 duplex nucleotides 39.7, 41.8, 49.5, 55.1, 69.1, 80,000: 64.8, 68.2, 65.9, 68.8, 83.0, 160,000: 126.5,
// 125.2, 123.3, 126.8, 121.9; strands, 60,000: 32.5, 31.3, 30.0, 30.0, 30.2, 250,000: 111.0, 103.6, 101.0, 99.5, 98.2; batch
// of 96 systems (70,000) 85.1, 86.1, 81.7, 88.9, 102.3.
constexpr int PAIR_WIDE_N = 65000;
// Blocks of 256 threads instead of 128 where one resident wave (three per SM) holds them all: a group's
// stages are then half as many rounds long, which is what the launch lasts where the chip is not full.  64, 128,
// 256 threads, us per step: 24 nucleotides 18.1, 16.7, 14.9, 1,000 duplex nucleotides 20.4, 17.0, 15.6; 128 and 256: 5,000:
// 22.4, 19.3, 8,000: 22.8, 20.1, 12,000: 24.1, 23.4, 16,000: 25.2, 27.8; 10,000 strand nucleotides 17.4, 17.6.
constexpr bool pair_small(int N) { return N / 32 + N / 128 <= 3 * 152; }
// the three ranges of N in which a shape stands for different kernels, and whether shape k's differ there from
// those of the shapes before it (below PAIR_WIDE_N the groups are one whatever npw)
int force_shape_range(int N) { return pair_small(N) ? 0 : N < PAIR_WIDE_N ? 1 : 2; }
bool force_shape_distinct(int k, int N) {
	if(N >= PAIR_WIDE_N) return true;
	for(int u = 0; u < k; u++)
		if(FORCE_SHAPES[u].lanes == FORCE_SHAPES[k].lanes && FORCE_SHAPES[u].minb == FORCE_SHAPES[k].minb) return false;
	return true;
}
template <int k>
static void launch_md_shape(const ForceArgs &a, const SplitMixed &ld, cudaStream_t s) {
	constexpr ForceShapeDef d = FORCE_SHAPES[k];
	if(pair_small(a.N)) launch_split_t<float, SplitMixed, false, false, 1, d.lanes, d.minb, false, 256>(a, ld, s);
	else if(a.N < PAIR_WIDE_N) launch_split_t<float, SplitMixed, false, false, 1, d.lanes, d.minb>(a, ld, s);
	else launch_split_t<float, SplitMixed, false, false, d.npw == 32 ? 3 : 6, d.lanes, d.minb>(a, ld, s);
}

// use_edge: the default shape with the edge blocks
template <typename R, class Loader>
static void launch_edge(const ForceArgs &a, Loader ld, bool split, bool energy, cudaStream_t s) {
	constexpr int G = 1, K = OXGB_NB_LANES, MB = OXGB_NB_MINB;
	if(split) launch_split_t<R, Loader, true, true, G, K, MB, true>(a, ld, s);
	else if(energy) launch_split_t<R, Loader, false, true, G, K, MB, true>(a, ld, s);
	else launch_split_t<R, Loader, false, false, G, K, MB, true>(a, ld, s);
}

static SplitDouble double_loader(const ForceArgs &a) {
	return SplitDouble{a.posd, a.frame64, a.N, SplitMixed{a.pos_hi, a.pos_lo, a.fa1, a.fa3, a.fback, nullptr, nullptr}};
}

cudaError_t launch_forces_split(const ForceArgs &a, bool dbl, bool split, bool energy, cudaStream_t s) {
	if(a.edge) {
		if(dbl) launch_edge<double, SplitDouble>(a, double_loader(a), split, energy, s);
		else launch_edge<float, SplitMixed>(a, SplitMixed{a.pos_hi, a.pos_lo, a.fa1, a.fa3, a.fback, a.fa1lo, a.fbacklo}, split, energy, s);
		return cudaGetLastError();
	}
	if(dbl) {
		const SplitDouble ld = double_loader(a);
		if(split) launch_split_t<double, SplitDouble, true, true>(a, ld, s);
		else if(energy) launch_split_t<double, SplitDouble, false, true>(a, ld, s);
		else launch_split_t<double, SplitDouble, false, false>(a, ld, s);
	}
	else {
		SplitMixed ld{a.pos_hi, a.pos_lo, a.fa1, a.fa3, a.fback, a.fa1lo, a.fbacklo};
		if(split) launch_split_t<float, SplitMixed, true, true>(a, ld, s);
		else if(energy) launch_split_t<float, SplitMixed, false, true>(a, ld, s);
		else {
			static_assert(N_FORCE_SHAPES == 6, "one case per shape");
			switch(a.shape) {
			case 1: launch_md_shape<1>(a, ld, s); break;
			case 2: launch_md_shape<2>(a, ld, s); break;
			case 3: launch_md_shape<3>(a, ld, s); break;
			case 4: launch_md_shape<4>(a, ld, s); break;
			case 5: launch_md_shape<5>(a, ld, s); break;
			default: launch_md_shape<0>(a, ld, s); break;
			}
		}
	}
	return cudaGetLastError();
}

}  // namespace oxgb
