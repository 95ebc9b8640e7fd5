// Velocity-Verlet integration in FP64 and the Brownian ("john") and Bussi thermostats.
//
// Replaces first_step_mixed / second_step_mixed (src/CUDA/Backends/CUDA_mixed.cuh:8-93) and the
// CUDA thermostats (src/CUDA/Thermostats/CUDABrownianThermostat.cu:15-51,
// CUDABussiThermostat.cu:55-122 with the host kinetic-energy update of
// src/Backends/Thermostats/BussiThermostat.cpp:44-160).  Differences by design: positions,
// velocities, angular momenta and quaternions stay FP64 throughout (the half kicks convert the
// FP32 forces to double before multiplying by dt), the quaternion is renormalised every step,
// random numbers come from a counter-based Philox-4x32-10 stream keyed by (seed, step,
// particle) so that runs are reproducible and graph-replayable, and the Bussi kinetic-energy
// update runs on the device (its gamma deviate uses the same algorithm as the reference).
// The second half kick of a step and its thermostat are deferred to the next first step (or
// to the flush at the end of a run), where they run one thread per nucleotide next to the
// first half kick; the Bussi sums run after the forces (k_bussi_sums, with the update), and its draws, those of
// all steps of a graph at once, on a parallel branch of the step graph (k_bussi_noise).  No FP64 work is
// left in the mixed engine's force kernels, whose lanes are mostly idle at the epilogue.
#include "split.cuh"
#include "thermo.cuh"

namespace oxgb {

// ---------------------------------------------------------------- FP32 mirrors

// The FP32 mirrors of nucleotide i from its FP64 state: the position as hi + lo, the body
// axes a1, a3 and the grooved backbone offset (src/Particles/DNANucleotide.cpp:79), each
// rounded once (to within an ulp) from exact values; conversions and products on the FP32 and
// integer pipes (split.cuh).  Each part returns what the staleness test needs.
__device__ __forceinline__ void mirror_position(const StepArgs &a, int i, const double4_32a &r, float3 &rh, float3 &rl) {
	float4 hi = a.pos_hi[i], lo = a.pos_lo[i];
	split_rn(r.x, hi.x, lo.x);
	split_rn(r.y, hi.y, lo.y);
	split_rn(r.z, hi.z, lo.z);
	a.pos_hi[i] = hi;
	a.pos_lo[i] = lo;
	rh = make_float3(hi.x, hi.y, hi.z);
	rl = make_float3(lo.x, lo.y, lo.z);
}

// what the fixed-point sites need of a system's table
struct FixedBox {
	float box_hi, box_lo, inv_box, s_hi, s_lo;
};

__device__ __forceinline__ FixedBox fixed_box(const StepArgs &a, int sy) {
	const DNA2Table<float> &P = reinterpret_cast<const DNA2Table<float> *>(a.table)[sy];
	return FixedBox{P.box_hi, P.box_lo, P.inv_box, P.fix_hi, P.fix_lo};
}

// a position (hi + lo) in fixed point
__device__ __forceinline__ uint3 fixed_centre(const FixedBox &b, float3 hi, float3 lo) {
	return make_uint3(fixed_coord(hi.x, lo.x, b.box_hi, b.box_lo, b.inv_box, b.s_hi, b.s_lo),
			fixed_coord(hi.y, lo.y, b.box_hi, b.box_lo, b.inv_box, b.s_hi, b.s_lo),
			fixed_coord(hi.z, lo.z, b.box_hi, b.box_lo, b.inv_box, b.s_hi, b.s_lo));
}

// the fixed-point backbone and base sites of nucleotide i, from its position, its FP32 backbone offset
// and a1 (base site at 0.4 a1)
__device__ __forceinline__ void mirror_sites(const StepArgs &a, int i, const FixedBox &b, uint3 c, float3 a1, float4 back) {
	const float s2 = 2.f * b.s_hi, sb = 0.4f * s2;
	a.site_back[i] = make_int4(fixed_site(c.x, back.x * s2), fixed_site(c.y, back.y * s2), fixed_site(c.z, back.z * s2),
			back.w != 0.f);
	a.site_base[i] = make_int4(fixed_site(c.x, a1.x * sb), fixed_site(c.y, a1.y * sb), fixed_site(c.z, a1.z * sb), 0);
}

// returns a1 and the backbone offset (w: the strand-end flag) and with F64 keeps the FP64 engine's frame;
// with a.fa1lo also the remainders of a1 and the backbone offset (exact value = mirror + remainder to ~2^-46), which the force kernels use for the stiff
// radial factors and excluded-volume contacts
template <bool F64>
__device__ __forceinline__ void mirror_frame(const StepArgs &a, int i, const double4_32a &q, float3 &a1o, float4 &backo) {
	float qh[4], ql[4], a1[3], a3[3], bk[3], a1l[3], bkl[3];
	split_rn(q.x, qh[0], ql[0]);
	split_rn(q.y, qh[1], ql[1]);
	split_rn(q.z, qh[2], ql[2]);
	split_rn(q.w, qh[3], ql[3]);
	if(a.fa1lo) {
		frame_mirror_rem(qh, ql, OXM_POS_MM_BACK1, OXM_POS_MM_BACK2, a1, a3, bk, a1l, bkl);
		a.fa1lo[i] = make_float4(a1l[0], a1l[1], a1l[2], 0.f);
		a.fbacklo[i] = make_float4(bkl[0], bkl[1], bkl[2], 0.f);
	}
	else frame_mirror(qh, ql, OXM_POS_MM_BACK1, OXM_POS_MM_BACK2, a1, a3, bk);
	a.fa1[i] = make_float4(a1[0], a1[1], a1[2], 0.f);
	a.fa3[i] = make_float4(a3[0], a3[1], a3[2], 0.f);
	// the strand-end flag rides in w
	const int2 bd = a.bonds[i];
	backo = make_float4(bk[0], bk[1], bk[2], (bd.x < 0 || bd.y < 0) ? 1.f : 0.f);
	if(F64 && a.frame64) write_frame64(a.frame64, a.N, i, q, bd.x < 0 || bd.y < 0);
	a.fback[i] = backo;
	a1o = make_float3(a1[0], a1[1], a1[2]);
}

// true if the centre or any interaction site moved more than the skin since the last list build
// (lp, la1, lbk: centre, a1 and backbone offset at the last build; r: the new centre in FP32,
// a1 and back: the new axis and backbone offset)
__device__ __forceinline__ bool list_stale(const StepArgs &a, const float4 &lp, const float4 &la1, const float4 &lbk, float3 r,
		float3 a1, float4 bk) {
	const float dx = r.x - lp.x, dy = r.y - lp.y, dz = r.z - lp.z;
	if(dx * dx + dy * dy + dz * dz > a.skin2) return true;
	if(!a.list_a1) return false;
	const float ex = a1.x - la1.x, ey = a1.y - la1.y, ez = a1.z - la1.z;
	float sx = dx + 0.4f * ex, sy = dy + 0.4f * ey, sz = dz + 0.4f * ez;  // base site
	if(sx * sx + sy * sy + sz * sz > a.skin2) return true;
	sx = dx + 0.34f * ex, sy = dy + 0.34f * ey, sz = dz + 0.34f * ez;  // stacking site
	if(sx * sx + sy * sy + sz * sz > a.skin2) return true;
	sx = dx + (bk.x - lbk.x), sy = dy + (bk.y - lbk.y), sz = dz + (bk.z - lbk.z);  // backbone site
	return sx * sx + sy * sy + sz * sz > a.skin2;
}

__global__ void k_make_mirrors(StepArgs a) {
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if(i >= a.N) return;
	float3 a1, hi, lo;
	float4 bk;
	mirror_position(a, i, a.pos[i], hi, lo);
	mirror_frame<true>(a, i, a.quat[i], a1, bk);
	if(a.site_back) {
		const FixedBox b = fixed_box(a, a.th.sys[i]);
		mirror_sites(a, i, b, fixed_centre(b, hi, lo), a1, bk);
	}
}

// ---------------------------------------------------------------- first half step

__device__ __forceinline__ long long step_of(const ThermoArgs &t) { return *t.step_base + t.step_offset; }

// completes step sp of nucleotide i (system sy): its second half kick (CUDA_mixed.cuh:71-93)
// and its thermostat (Brownian redraw or Bussi rescaling)
template <typename V4>
__device__ __forceinline__ void complete_step(const ThermoArgs &t, int i, int sy, long long sp, const V4 &F, const V4 &T,
		double4_32a &v, double4_32a &L) {
	// the half kicks are written as FMAs here and in the first step, so that a step completed at
	// the end of a run and one completed by the next first step are the same
	const double hdt = 0.5 * t.dt;
	v.x = fma(widen(F.x), hdt, v.x);
	v.y = fma(widen(F.y), hdt, v.y);
	v.z = fma(widen(F.z), hdt, v.z);
	L.x = fma(widen(T.x), hdt, L.x);
	L.y = fma(widen(T.y), hdt, L.y);
	L.z = fma(widen(T.z), hdt, L.z);
	if(t.thermostat == 1 && sp % t.newtonian_steps == 0) brownian_redraw(t, sy, (t.id ? t.id[i] : i) - t.sys_off[sy], sp, v, L);
	else if(t.thermostat == 2 && *t.bussi_stamp == sp) bussi_rescale(t, sy, v, L);
}

// the orientation after a step of dt with angular momentum L (body frame):
// q <- q * (sin(th/2) L^, cos(th/2)), th = dt |L|, then renormalised
__device__ __forceinline__ void rotate(double4_32a &q, const double4_32a &L, double dt) {
	const double L2 = L.x * L.x + L.y * L.y + L.z * L.z;
	if(!(L2 > 0.0)) return;
	const double hd = 0.5 * dt, x2 = hd * hd * L2;  // x = th / 2
	double k, ch;
	if(x2 < 1e-5) {
		// sin(x) / x and cos(x) as Taylor series in x^2: no square root, range reduction or
		// division, which are slow in FP64.  The first omitted terms, x^6/5040 and x^8/40320,
		// are below 2e-19 for x^2 < 1e-5 (a typical step has x^2 ~ 1e-6)
		k = hd * (1.0 - x2 * (1.0 / 6.0) * (1.0 - x2 * (1.0 / 20.0)));
		ch = 1.0 - x2 * 0.5 * (1.0 - x2 * (1.0 / 12.0) * (1.0 - x2 * (1.0 / 30.0)));
	}
	else if(x2 < 1e-2) {
		// the same series to x^10 (truncation below 1e-20 for |x| < 0.1)
		k = hd * (1.0 - x2 * (1.0 / 6.0) * (1.0 - x2 * (1.0 / 20.0) * (1.0 - x2 * (1.0 / 42.0) * (1.0 - x2 * (1.0 / 72.0) * (1.0 - x2 * (1.0 / 110.0))))));
		ch = 1.0 - x2 * 0.5 * (1.0 - x2 * (1.0 / 12.0) * (1.0 - x2 * (1.0 / 30.0) * (1.0 - x2 * (1.0 / 56.0) * (1.0 - x2 * (1.0 / 90.0)))));
	}
	else {
		const double norm = sqrt(L2);
		double sh;
		sincos(hd * norm, &sh, &ch);
		k = sh / norm;
	}
	const double rx = L.x * k, ry = L.y * k, rz = L.z * k, rw = ch;
	double4_32a n;
	n.w = q.w * rw - q.x * rx - q.y * ry - q.z * rz;
	n.x = q.w * rx + q.x * rw + q.y * rz - q.z * ry;
	n.y = q.w * ry - q.x * rz + q.y * rw + q.z * rx;
	n.z = q.w * rz + q.x * ry - q.y * rx + q.z * rw;
	const double nn = n.x * n.x + n.y * n.y + n.z * n.z + n.w * n.w;
	const double d = nn - 1.0;
	// |n|^2 = 1 + d with |d| at the rounding level: 1/sqrt(1 + d) = 1 - d/2 + 3d^2/8 - ...
	const double inv = fabs(d) < 1e-6 ? 1.0 - d * (0.5 - 0.375 * d) : 1.0 / sqrt(nn);
	q = make_double4_32a(n.x * inv, n.y * inv, n.z * inv, n.w * inv);
}

// The FP32 rotation of backend_precision = float (CUDA_MD.cuh:11-25): q <- q * (sin(th/2) L^,
// cos(th/2)), th = dt |L|, in FP32; renormalised in FP32 as well (the reference's float path
// lets the norm drift)
__device__ __forceinline__ void rotate_f32(float4 &q, float3 L, float dt) {
	const float L2 = L.x * L.x + L.y * L.y + L.z * L.z;
	if(!(L2 > 0.f)) return;
	const float norm = sqrtf(L2);
	float sh, ch;
	sincosf(0.5f * dt * norm, &sh, &ch);
	const float k = sh / norm;
	const float rx = L.x * k, ry = L.y * k, rz = L.z * k, rw = ch;
	float4 n;
	n.w = q.w * rw - q.x * rx - q.y * ry - q.z * rz;
	n.x = q.w * rx + q.x * rw + q.y * rz - q.z * ry;
	n.y = q.w * ry - q.x * rz + q.y * rw + q.z * rx;
	n.z = q.w * rz + q.x * ry - q.y * rx + q.z * rw;
	const float inv = rsqrtf(n.x * n.x + n.y * n.y + n.z * n.z + n.w * n.w);
	q = make_float4(n.x * inv, n.y * inv, n.z * inv, n.w * inv);
}

__device__ __forceinline__ double4_32a widen4(float x, float y, float z, float w) {
	return make_double4_32a(widen(x), widen(y), widen(z), widen(w));
}

// a state vector rounded to FP32 (backend_precision = float keeps the state FP32-representable)
__device__ __forceinline__ double4_32a round4(const double4_32a &v) {
	return widen4(narrow(v.x), narrow(v.y), narrow(v.z), narrow(v.w));
}

// First half of step s, two warps per 32 nucleotides: the first the translation (second
// half kick and thermostat of step s - 1, half kick, drift, position mirror), the second the
// rotation (the same for the angular momentum, rotation, frame mirror).  The chains of FP64
// operations are half as long and twice as many warps hide them; a warp never diverges on the
// kind of motion.  What needs both, the sites and the staleness test, is done by the translation warp,
// whose own chain is the shorter one.
// (capped at 64 registers, 16 blocks per SM: measured in alternating runs, the 250k MD step
// 138.7 -> 136.9 us and the 256-system batch 263.4 -> 261.3 us against the uncapped 80)
// Named barrier 1 + pair of W pairs of warps: arrive or, with WAIT, wait too.  The numbers are immediates: with
// a computed one a block takes all 16 barriers, and the SM has them for half of the blocks only.
template <int W, bool WAIT>
__device__ __forceinline__ void pair_barrier(int pair) {
	if constexpr(W > 1) {
		if(pair != W - 1) {
			pair_barrier<W - 1, WAIT>(pair);
			return;
		}
	}
	if(WAIT) asm volatile("bar.sync %0, 64;" ::"n"(W) : "memory");
	else asm volatile("bar.arrive %0, 64;" ::"n"(W) : "memory");
}

// W: pairs of warps per block, which share their Brownian redraws (launch_first_step)
template <typename V4, bool F32, bool BROWNIAN, int W>
__global__ void __launch_bounds__(64 * W, 16 / W) k_first_step(StepArgs a) {
	__shared__ float3 s_a1[W][32];
	__shared__ float4 s_back[W][32];
	const int lane = threadIdx.x & 31, pair = (threadIdx.x >> 5) % W;
	const bool rot = threadIdx.x >= 32 * W;
	const int i = (blockIdx.x * W + pair) * 32 + lane;
	const bool live = i < a.N;
	float3 r32 = make_float3(0.f, 0.f, 0.f), r32l = r32, fa1 = r32;
	float4 fbk = make_float4(0.f, 0.f, 0.f, 0.f);
	int sy = 0;
	double4_32a x, y;  // (v, r) on the translation warp, (L, q) on the rotation warp
	float4 lp, la1, lbk;
	constexpr bool SITES = sizeof(V4) == sizeof(float4);  // (the double engine has no fixed-point sites)
	FixedBox fb{};
	uint3 centre = make_uint3(0, 0, 0);
	auto load_state = [&]() {
		if(live) {
			sy = a.th.sys[i];
			x = rot ? a.angmom[i] : a.vel[i];
			y = rot ? a.quat[i] : a.pos[i];
			if(!rot) {
				if(SITES) fb = fixed_box(a, sy);
				lp = a.list_pos[i];
				if(a.list_a1) la1 = a.list_a1[i], lbk = a.list_back[i];
			}
		}
	};
	// Inside a graph of steps (offset > 0) the kernel before this one is the previous step's
	// last, launched after the FP64 state and the list build's positions were written: they are
	// read before waiting for it, and only its outputs (the forces, the Bussi update) after.
	// Otherwise (the first step of a graph or a single step, which may follow any kernel that
	// writes the state) everything is read after the wait.
	// The previous step's redraws depend on nothing but the seed, the step and the caller's index.
	const bool early = a.th.step_offset > 0;
	bool redraw = false;
	double4_32a fresh;
	auto draws = [&]() {
		__shared__ RedrawPool<W> pool;
		const long long sp = step_of(a.th) - 1;
		if(sp % a.th.newtonian_steps == 0)
			redraw = brownian_redraws(a.th, pool, sy, live ? (a.th.id ? a.th.id[i] : i) - a.th.sys_off[sy] : 0, sp, rot, live, fresh);
	};
	if(early) {
		load_state();
		if(BROWNIAN) draws();
	}
	pdl_wait();
	pdl_trigger();
	if(!early) {
		load_state();
		if(BROWNIAN) draws();
	}
	if constexpr(F32) {
		if(live) {
		// backend_precision = float (CUDA_MD.cuh:11-60,556-578): the kicks, the drift and the
		// rotation in FP32 arithmetic on the FP32-representable state (exact conversions); the
		// thermostats act in FP64 on the completed momenta, rounded back to FP32
		const long long s = step_of(a.th);
		const float dt = (float) a.dt, hdt = 0.5f * dt;
		const bool complete = *a.th.open_step == s - 1;
		const long long sp = s - 1;
		const bool bussi = complete && a.th.thermostat == 2 && *a.th.bussi_stamp == sp;
		const V4 G = reinterpret_cast<const V4 *>(rot ? a.torques : a.forces)[i];
		const float gx = (float) G.x, gy = (float) G.y, gz = (float) G.z;
		float3 u = make_float3(narrow(x.x), narrow(x.y), narrow(x.z));
		if(complete) {
			u.x += gx * hdt;
			u.y += gy * hdt;
			u.z += gz * hdt;
			if(redraw || bussi) {
				x = widen4(u.x, u.y, u.z, 0.f);
				if(redraw) x = fresh;
				else bussi_rescale_part(a.th, sy, rot ? 1 : 0, x);
				u = make_float3(narrow(x.x), narrow(x.y), narrow(x.z));
			}
		}
		u.x += gx * hdt;
		u.y += gy * hdt;
		u.z += gz * hdt;
		x = widen4(u.x, u.y, u.z, 0.f);
		if(!rot) {
			float3 r = make_float3(narrow(y.x), narrow(y.y), narrow(y.z));
			r.x += u.x * dt;
			r.y += u.y * dt;
			r.z += u.z * dt;
			const double4_32a rd = widen4(r.x, r.y, r.z, 0.f);
			a.vel[i] = x;
			a.pos[i] = rd;
			mirror_position(a, i, rd, r32, r32l);
		}
		else {
			float4 q = make_float4(narrow(y.x), narrow(y.y), narrow(y.z), narrow(y.w));
			rotate_f32(q, u, dt);
			const double4_32a qd = widen4(q.x, q.y, q.z, q.w);
			a.angmom[i] = x;
			a.quat[i] = qd;
			mirror_frame<!SITES>(a, i, qd, fa1, fbk);
		}
		}
	}
	else if(live) {
		const long long s = step_of(a.th);
		const double hdt = 0.5 * a.dt;
		// the previous step's second half kick and thermostat (kept as a separate half kick, so
		// that a state is the same whether or not a run ended at that step)
		const bool complete = *a.th.open_step == s - 1;
		const long long sp = s - 1;
		const bool bussi = complete && a.th.thermostat == 2 && *a.th.bussi_stamp == sp;
		const V4 G = reinterpret_cast<const V4 *>(rot ? a.torques : a.forces)[i];
		const double gx = widen(G.x), gy = widen(G.y), gz = widen(G.z);
		if(complete) {
			x.x = fma(gx, hdt, x.x);
			x.y = fma(gy, hdt, x.y);
			x.z = fma(gz, hdt, x.z);
			if(redraw) x = fresh;
			else if(bussi) bussi_rescale_part(a.th, sy, rot ? 1 : 0, x);
		}
		x.x = fma(gx, hdt, x.x);
		x.y = fma(gy, hdt, x.y);
		x.z = fma(gz, hdt, x.z);
		if(!rot) {
			double4_32a r = y;
			r.x += x.x * a.dt;
			r.y += x.y * a.dt;
			r.z += x.z * a.dt;
			a.vel[i] = x;
			a.pos[i] = r;
			mirror_position(a, i, r, r32, r32l);
		}
		else {
			double4_32a q = y;
			// mixed precision: the small rotation as an FP64 sum of an FP32-pair correction (as
			// accurate, far fewer FP64 operations); double precision, or a large step: FP64
			if(!(sizeof(V4) == sizeof(float4) && rotate_small(q.x, q.y, q.z, q.w, x.x, x.y, x.z, 0.5 * a.dt))) rotate(q, x, a.dt);
			a.angmom[i] = x;
			a.quat[i] = q;
			mirror_frame<!SITES>(a, i, q, fa1, fbk);
		}
	}
	// (ahead of the wait for the frame)
	if(SITES && live && !rot) centre = fixed_centre(fb, r32, r32l);
	// the rotation warp posts its frame and leaves (named barrier 1 + pair: arrive, no wait)
	if(rot) {
		s_a1[pair][lane] = fa1;
		s_back[pair][lane] = fbk;
		pair_barrier<W, false>(pair);
		return;
	}
	pair_barrier<W, true>(pair);
	if(!live) return;
	fa1 = s_a1[pair][lane];
	fbk = s_back[pair][lane];
	if(SITES) mirror_sites(a, i, fb, centre, fa1, fbk);
	// Verlet list staleness (CUDA_mixed.cuh:68, extended to the interaction sites for the term
	// lists), per system
	if(list_stale(a, lp, la1, lbk, r32, fa1, fbk)) {
		a.sys_stale[sy] = 1;
		atomicOr(a.flag, 1);
	}
}

// ---------------------------------------------------------------- thermostats

// the Bussi draws of one system and step (step after step from this one on, systems together; one dimension, as
// the grid's others hold 65,535): warp 0 translational (channel 0), warp 1 rotational (channel 1)
__global__ void k_bussi_noise(StepArgs a) {
	const int k = blockIdx.x / a.th.n_systems, sy = blockIdx.x % a.th.n_systems;
	const long long s = step_of(a.th) + k;
	if(s % a.th.newtonian_steps != 0 || (threadIdx.x & 31) != 0) return;
	const int w = threadIdx.x >> 5;
	if(w > 1) return;
	const int n = a.th.sys_off[sy + 1] - a.th.sys_off[sy];
	Stream rs;
	rs.init(a.th.sys_seed[sy], s, (unsigned) w);
	double sum, rr;
	bussi_draws(rs, w == 0 ? 3 * (n - 1) : 3 * n, sum, rr);
	double *to = a.th.bussi_draws + 4 * ((size_t) k * a.th.n_systems + sy) + 2 * w;
	to[0] = sum;
	to[1] = rr;
}

// ---------------------------------------------------------------- Bussi kinetic sums
//
// The update of step s needs, per system, the sums of v, |v|^2 and |L|^2 over the completed
// momenta v + h F and L + h T (h = dt / 2).  They are split as
//   sum (v + h F)^2 = sum v^2 + 2 h sum v.F + h^2 sum F^2   (and likewise for L, T):
// the FP64 sums of the half-kicked state depend only on the first step; the force terms are FP32 products of the
// FP32 forces with the FP32-rounded momenta, summed with compensation, a correction of relative
// size h |F| / |v| to sums that stay FP64.  Both sums run over the same chunks (up to 256
// nucleotides of one system, aligned to the system's first nucleotide), so a system reduces the
// same way in a batch as alone.

__device__ __forceinline__ double shfl_xor(double v, int m) { return __shfl_xor_sync(0xffffffffu, v, m); }

// a float sum with its running error (TwoSum at every addition)
struct CompF {
	float s, e;
};
__device__ __forceinline__ CompF shfl_xor(CompF v, int m) {
	return CompF{__shfl_xor_sync(0xffffffffu, v.s, m), __shfl_xor_sync(0xffffffffu, v.e, m)};
}
__device__ __forceinline__ CompF comp_add(CompF a, CompF b) {
	const float t = a.s + b.s, bp = t - a.s;
	return CompF{t, a.e + b.e + ((a.s - (t - bp)) + (b.s - bp))};
}

// sum over a warp of 8 values per lane by a transposed butterfly (9 additions where 8
// separate reductions take 40); every lane returns the total of value (lane >> 2) & 7.  The
// order is fixed.
template <typename T, typename Add>
__device__ __forceinline__ T warp_transpose_sum8(const T (&x)[8], Add add) {
	const int lane = threadIdx.x & 31;
	const bool h16 = lane & 16, h8 = lane & 8, h4 = lane & 4;
	T w[4], u[2];
#pragma unroll
	for(int k = 0; k < 4; k++) w[k] = add(h16 ? x[k + 4] : x[k], shfl_xor(h16 ? x[k] : x[k + 4], 16));
#pragma unroll
	for(int k = 0; k < 2; k++) u[k] = add(h8 ? w[k + 2] : w[k], shfl_xor(h8 ? w[k] : w[k + 2], 8));
	T t = add(h4 ? u[1] : u[0], shfl_xor(h4 ? u[0] : u[1], 4));
	t = add(t, shfl_xor(t, 2));
	return add(t, shfl_xor(t, 1));
}

// the 8 per-thread values of a block's first nw warps summed in a fixed order into red[0..7] (a 256-thread
// block)
__device__ __forceinline__ void block_sum8(const double (&x)[8], double *red, int nw = 8) {
	__shared__ double part[8][8];
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
	if(w < nw) {
		const double t = warp_transpose_sum8(x, [](double p, double q) { return p + q; });
		if((lane & 3) == 0) part[lane >> 2][w] = t;
	}
	__syncthreads();
	if(threadIdx.x < 8) {
		double r = 0;
		for(int u = 0; u < nw; u++) r += part[threadIdx.x][u];
		red[threadIdx.x] = r;
	}
}

__device__ __forceinline__ CompF block_sum8_comp(const CompF (&x)[8]) {
	__shared__ CompF part[8][8];
	const CompF t = warp_transpose_sum8(x, comp_add);
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
	if((lane & 3) == 0) part[lane >> 2][w] = t;
	__syncthreads();
	CompF r{0.f, 0.f};
	if(threadIdx.x < 8)
		for(int u = 0; u < nw; u++) r = comp_add(r, part[threadIdx.x][u]);
	return r;
}

// the block's compensated sums of 8 values as float pairs (written by threads 0..7)
__device__ __forceinline__ void block_sum8f(const CompF (&x)[8], float2 *out) {
	const CompF r = block_sum8_comp(x);
	if(threadIdx.x < 8) out[threadIdx.x] = make_float2(r.s, r.e);
}

// The rescaling of system sy from its chunks' sums, reduced by the block in a fixed chunk order (the result
// does not depend on which block runs it); translation on thread 0 and rotation on thread 32 (two warps: the
// chains overlap).  Every step waits for this, so it is one load of the chunks and one reduction, of the five
// completed sums, over the warps that have chunks.
__device__ __forceinline__ void bussi_system_update(const StepArgs &a, int sy) {
	__shared__ double kin[8];
	const int c0 = a.th.sys_chunk0[sy], nc = a.th.sys_chunk0[sy + 1] - c0;
	const int which = threadIdx.x >> 5;
	double root = 0.0, inv_n = 0.0, n = 0.0;
	if(threadIdx.x == 0 || threadIdx.x == 32) {
		root = __ldcg(a.th.bussi_state + 16 * sy + 8 + which);
		inv_n = a.th.sys_par[sy * SP_STRIDE + SP_INVN];
		n = (double) (a.th.sys_off[sy + 1] - a.th.sys_off[sy]);
	}
	const double h = 0.5 * a.dt;
	double x[8] = {0, 0, 0, 0, 0, 0, 0, 0};
	for(int b = threadIdx.x; b < nc; b += blockDim.x) {
		const double *q = a.th.bussi_partials + 8 * (c0 + b);
		const float2 *p = a.th.bussi_fpart + 8 * (c0 + b);
		double k[5], f[7];
#pragma unroll
		for(int u = 0; u < 5; u++) k[u] = __ldcg(q + u);
#pragma unroll
		for(int u = 0; u < 7; u++) {
			const float2 v = __ldcg(p + u);
			f[u] = widen(v.x) + widen(v.y);
		}
#pragma unroll
		for(int u = 0; u < 3; u++) x[u] += k[u] + h * f[u];
		x[3] += k[3] + 2.0 * h * f[3] + h * h * f[4];
		x[4] += k[4] + 2.0 * h * f[5] + h * h * f[6];
	}
	__syncthreads();  // the block's scratch is reused
	block_sum8(x, kin, min((nc + 31) >> 5, 8));
	__syncthreads();
	if(threadIdx.x == 0 || threadIdx.x == 32) bussi_factor(a.th, sy, which, kin, root, inv_n, n);
}

// Bussi step s, after its forces.  Before it waits for them: per chunk, the FP64 sums of the half-kicked
// v, |v|^2 and |L|^2 and the system's new kinetic energies, beside the tail of the force kernels.  Then the sums of F, v.F, |F|^2, L.T and |T|^2
// (FP32 products with the FP32-rounded momenta, compensated sums; FP64 in double precision).  The block that
// brings a system's last chunk (a per-system arrival counter) makes that system's update, so there is no
// separate update launch.
//
// What bounds it is the chain from the forces to the rescaling: 40,000 nucleotides, 1 us for the chunks'
// sums, 0.8 for the arrivals, 4.1 for the last block's (5.2 with the kinetic energies' update and a reduction of
// force terms apart from it; the arithmetic is a chain of FP64 operations).  The FP64 sums were a kernel on a
// side branch of the step graph, joined before this one in every step: 57.2 us per step, 56.1 so; a batch of
// 96 systems 108.7 and 107.1.
template <typename V4>
__global__ void __launch_bounds__(256) k_bussi_sums(StepArgs a) {
	const long long s = step_of(a.th);
	const bool due = s % a.th.newtonian_steps == 0;
	const int c = blockIdx.x;
	const int sy = a.th.chunk_sys[c];
	const int i = a.th.chunk_first[c] + threadIdx.x;
	const bool live = due && i < a.th.sys_off[sy + 1];
	double4_32a v = make_double4_32a(0., 0., 0., 0.), L = v;
	if(live) v = a.vel[i], L = a.angmom[i];  // (the first step's, complete before the force kernels began)
	if(due) {
		if(c == a.th.sys_chunk0[sy] && (threadIdx.x == 0 || threadIdx.x == 32)) bussi_advance(a.th, sy, threadIdx.x >> 5);
		const double x[8] = {v.x, v.y, v.z, v.x * v.x + v.y * v.y + v.z * v.z, L.x * L.x + L.y * L.y + L.z * L.z, 0, 0, 0};
		block_sum8(x, a.th.bussi_partials + 8 * c);
	}
	pdl_wait();  // launched after the force kernels
	pdl_trigger();
	if(!due) return;
	if(sizeof(V4) == sizeof(float4)) {
		CompF x[8];
#pragma unroll
		for(int k = 0; k < 8; k++) x[k] = CompF{0.f, 0.f};
		if(live) {
			const float4 F = reinterpret_cast<const float4 *>(a.forces)[i], T = reinterpret_cast<const float4 *>(a.torques)[i];
			const float3 vf = make_float3(narrow(v.x), narrow(v.y), narrow(v.z)), Lf = make_float3(narrow(L.x), narrow(L.y), narrow(L.z));
			x[0].s = F.x;
			x[1].s = F.y;
			x[2].s = F.z;
			x[3].s = vf.x * F.x + vf.y * F.y + vf.z * F.z;
			x[4].s = F.x * F.x + F.y * F.y + F.z * F.z;
			x[5].s = Lf.x * T.x + Lf.y * T.y + Lf.z * T.z;
			x[6].s = T.x * T.x + T.y * T.y + T.z * T.z;
		}
		block_sum8f(x, a.th.bussi_fpart + 8 * c);
	}
	else {
		double x[8] = {0, 0, 0, 0, 0, 0, 0, 0};
		if(live) {
			const double4_32a F = reinterpret_cast<const double4_32a *>(a.forces)[i],
							  T = reinterpret_cast<const double4_32a *>(a.torques)[i];
			x[0] = F.x;
			x[1] = F.y;
			x[2] = F.z;
			x[3] = v.x * F.x + v.y * F.y + v.z * F.z;
			x[4] = F.x * F.x + F.y * F.y + F.z * F.z;
			x[5] = L.x * T.x + L.y * T.y + L.z * T.z;
			x[6] = T.x * T.x + T.y * T.y + T.z * T.z;
		}
		// FP64 sums, kept as float pairs like the mixed-precision ones (hi + lo carries 48 bits)
		__shared__ double red[8];
		__syncthreads();  // (the block's scratch is reused)
		block_sum8(x, red);
		__syncthreads();
		if(threadIdx.x < 8) {
			float hi, lo;
			split_rn(red[threadIdx.x], hi, lo);
			a.th.bussi_fpart[8 * c + threadIdx.x] = make_float2(hi, lo);
		}
	}
	__shared__ int last;
	__syncthreads();
	if(threadIdx.x == 0) {
		const unsigned nc = (unsigned) (a.th.sys_chunk0[sy + 1] - a.th.sys_chunk0[sy]);
		// released after and acquired before the block's barriers: the partials of every chunk that
		// arrived are visible to the block that arrives last
		unsigned old;
		asm volatile("atom.add.acq_rel.gpu.u32 %0, [%1], 1;" : "=r"(old) : "l"(a.th.bussi_done + sy) : "memory");
		last = old == nc - 1u;
		if(last) {
			a.th.bussi_done[sy] = 0u;  // every chunk has arrived: ready for the next step
			// the next first step applies the rescaling of step s (every system updates at the same steps)
			if(sy == 0) *a.th.bussi_stamp = s;
		}
	}
	__syncthreads();
	if(!last) return;
	bussi_system_update(a, sy);
}

__global__ void k_step_advance(StepArgs a, int K) {
	if(threadIdx.x == 0 && blockIdx.x == 0) *a.th.step_base += K;
}

// end of a run: the last step's second half kick and thermostat ...
template <typename V4>
__global__ void k_step_flush(StepArgs a) {
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	const long long sp = *a.th.step_base - 1;
	if(i >= a.N || *a.th.open_step != sp) return;
	const V4 F = reinterpret_cast<const V4 *>(a.forces)[i];
	const V4 T = reinterpret_cast<const V4 *>(a.torques)[i];
	double4_32a v = a.vel[i], L = a.angmom[i];
	complete_step(a.th, i, a.th.sys[i], sp, F, T, v, L);
	a.vel[i] = a.f32 ? round4(v) : v;
	a.angmom[i] = a.f32 ? round4(L) : L;
}

// ... after which nothing is pending
__global__ void k_step_flush_clear(StepArgs a) {
	if(threadIdx.x == 0 && blockIdx.x == 0) {
		*a.th.open_step = OXGB_NO_STEP;
		*a.th.bussi_stamp = OXGB_NO_STEP;
	}
}

// The caller's state arrays (positions, quaternions, velocities, angular momenta: 3, 4, 3 and 3
// doubles per nucleotide, the four arrays one after the other in `in`) into the FP64 state, each
// quaternion normalised (sums and products rounded in a fixed order); the lowest nucleotide whose
// quaternion cannot be normalised is kept in *bad.  With check_only nothing is written but *bad.
__global__ void k_unpack_state(StepArgs a, const double *in, int *bad, int check_only) {
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if(i >= a.N) return;
	const long long N = a.N;
	const double *p = in + 3 * (long long) i, *q = in + 3 * N + 4 * (long long) i, *v = in + 7 * N + 3 * (long long) i,
				 *l = in + 10 * N + 3 * (long long) i;
	const double n2 = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(q[0], q[0]), __dmul_rn(q[1], q[1])), __dmul_rn(q[2], q[2])),
			__dmul_rn(q[3], q[3]));
	double n = sqrt(n2);
	if(!(n > 0.5)) {
		atomicMin(bad, i);
		n = 1.0;
	}
	if(check_only) return;
	if(i == 0) *a.th.open_step = *a.th.bussi_stamp = OXGB_NO_STEP;  // nothing is pending in a new state
	double4_32a P = make_double4_32a(p[0], p[1], p[2], 0.0);
	double4_32a Q = make_double4_32a(__ddiv_rn(q[0], n), __ddiv_rn(q[1], n), __ddiv_rn(q[2], n), __ddiv_rn(q[3], n));
	double4_32a V = make_double4_32a(v[0], v[1], v[2], 0.0), M = make_double4_32a(l[0], l[1], l[2], 0.0);
	if(a.f32) {  // backend_precision = float: the state FP32 from the start
		P = round4(P);
		Q = round4(Q);
		V = round4(V);
		M = round4(M);
	}
	a.pos[i] = P;
	a.quat[i] = Q;
	a.vel[i] = V;
	a.angmom[i] = M;
}

// the FP64 state into the caller's layout and order (the reverse of k_unpack_state)
__global__ void k_pack_state(StepArgs a, double *out) {
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if(i >= a.N) return;
	const long long N = a.N;
	const long long c = a.th.id ? a.th.id[i] : i;  // the caller's index
	double *p = out + 3 * c, *q = out + 3 * N + 4 * c, *v = out + 7 * N + 3 * c, *l = out + 10 * N + 3 * c;
	const double4_32a r = a.pos[i], o = a.quat[i], u = a.vel[i], m = a.angmom[i];
	p[0] = r.x, p[1] = r.y, p[2] = r.z;
	q[0] = o.x, q[1] = o.y, q[2] = o.z, q[3] = o.w;
	v[0] = u.x, v[1] = u.y, v[2] = u.z;
	l[0] = m.x, l[1] = m.y, l[2] = m.z;
}

// velocities and angular momenta of nucleotides lo .. hi - 1 times f (a replica exchange)
__global__ void k_scale_momenta(StepArgs a, int lo, int hi, double f) {
	const int i = lo + blockIdx.x * blockDim.x + threadIdx.x;
	if(i >= hi) return;
	double4_32a v = a.vel[i], L = a.angmom[i];
	v.x *= f;
	v.y *= f;
	v.z *= f;
	L.x *= f;
	L.y *= f;
	L.z *= f;
	a.vel[i] = v;
	a.angmom[i] = L;
}

// per-chunk FP64 sums: potential energy (F.w / 2), translational and rotational kinetic energy
template <typename V4>
__global__ void __launch_bounds__(256) k_system_sums(StepArgs a, double *out) {
	const int c = blockIdx.x;
	const int sy = a.th.chunk_sys[c];
	const int i = a.th.chunk_first[c] + threadIdx.x;
	double acc[3] = {0, 0, 0};
	if(i < a.th.sys_off[sy + 1]) {
		const V4 F = reinterpret_cast<const V4 *>(a.forces)[i];
		const double4_32a v = a.vel[i], L = a.angmom[i];
		acc[0] = 0.5 * (double) F.w;
		acc[1] = 0.5 * (v.x * v.x + v.y * v.y + v.z * v.z);
		acc[2] = 0.5 * (L.x * L.x + L.y * L.y + L.z * L.z);
	}
	__shared__ double red[3][8];
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
	for(int k = 0; k < 3; k++) {
		double x = acc[k];
		for(int off = 16; off > 0; off >>= 1) x += __shfl_down_sync(0xffffffffu, x, off);
		if(lane == 0) red[k][w] = x;
	}
	__syncthreads();
	if(threadIdx.x < 3) {
		double x = 0;
		for(int u = 0; u < nw; u++) x += red[threadIdx.x][u];
		out[c * 4 + threadIdx.x] = x;
	}
}

// ---------------------------------------------------------------- launchers

static inline int blocks_for(int N, int tpb) { return N > 0 ? (N + tpb - 1) / tpb : 1; }

cudaError_t launch_first_step(const StepArgs &a, bool double_forces, cudaStream_t s) {
	const bool brownian = a.th.thermostat == 1;
	// double and float engines: two-warp blocks of 32 nucleotides, so that the FP64 work (1/64 of the FP32
	// rate) spreads evenly over the SMs
	const dim3 grid(blocks_for(a.N, 32)), block(64);
	if(double_forces)
		return brownian ? launch_after(k_first_step<double4_32a, false, true, 1>, grid, block, 0, s, a) :
				launch_after(k_first_step<double4_32a, false, false, 1>, grid, block, 0, s, a);
	if(a.f32)
		return brownian ? launch_after(k_first_step<float4, true, true, 1>, grid, block, 0, s, a) :
				launch_after(k_first_step<float4, true, false, 1>, grid, block, 0, s, a);
	// mixed engine: two pairs of warps per block.  One, two, four, us per step: 40,000 duplex nucleotides 53.8,
	// 52.6, 53.4, 250,000 strand nucleotides 106.8, 104.7, 105.8, a batch of 96 systems 109.3, 108.2, 108.1,
	// 1,000 duplex nucleotides 17.2, 17.2, 18.3.
	const dim3 grid2(blocks_for(a.N, 64)), block2(128);
	if(!brownian) return launch_after(k_first_step<float4, false, false, 2>, grid2, block2, 0, s, a);
	// Where redraws come in (nearly) every step, the FP64 pipes they load want the blocks spread evenly, but
	// blocks launched ahead pile up on the SMs that the kernel before leaves first.  If one wave holds the
	// grid, a block asks for as much shared memory as leaves room for no more than an even share: 32,000
	// nucleotides, a tenth redrawn in every step, 30.6 -> 26.8 us per step.  (Without redraws, 40,000 nucleotides, it
	// costs 1.5 us: changing the split of the SM's memory between kernels is not free.)
	const int share = (int) (grid2.x + 151) / 152;
	size_t room = 0;
	if(a.th.newtonian_steps <= 2 && share < 8) {
		room = ((228 * 1024 / (share + 1) - 8192) / 128 + 1) * 128;  // (8 KB: its static memory)
		const cudaError_t e = cudaFuncSetAttribute(k_first_step<float4, false, true, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
				227 * 1024 - 16384);
		if(e != cudaSuccess) return e;
	}
	return launch_after(k_first_step<float4, false, true, 2>, grid2, block2, room, s, a);
}

cudaError_t launch_bussi_noise(const StepArgs &a, int steps, cudaStream_t s) {
	k_bussi_noise<<<a.th.n_systems * steps, 64, 0, s>>>(a);
	return cudaGetLastError();
}

cudaError_t launch_bussi_reduce(const StepArgs &a, int n_chunks, bool double_forces, cudaStream_t s) {
	if(double_forces) return launch_after(k_bussi_sums<double4_32a>, dim3(n_chunks), dim3(256), 0, s, a);
	return launch_after(k_bussi_sums<float4>, dim3(n_chunks), dim3(256), 0, s, a);
}

cudaError_t launch_step_advance(const StepArgs &a, int K, cudaStream_t s) {
	k_step_advance<<<1, 32, 0, s>>>(a, K);
	return cudaGetLastError();
}

cudaError_t launch_step_flush(const StepArgs &a, bool double_forces, cudaStream_t s) {
	if(double_forces) k_step_flush<double4_32a><<<blocks_for(a.N, 256), 256, 0, s>>>(a);
	else k_step_flush<float4><<<blocks_for(a.N, 256), 256, 0, s>>>(a);
	k_step_flush_clear<<<1, 32, 0, s>>>(a);
	return cudaGetLastError();
}

cudaError_t launch_make_mirrors(const StepArgs &a, cudaStream_t s) {
	k_make_mirrors<<<blocks_for(a.N, 256), 256, 0, s>>>(a);
	return cudaGetLastError();
}

cudaError_t launch_unpack_state(const StepArgs &a, const double *in, int *bad, bool check_only, cudaStream_t s) {
	k_unpack_state<<<blocks_for(a.N, 256), 256, 0, s>>>(a, in, bad, check_only ? 1 : 0);
	return cudaGetLastError();
}

__global__ void k_identity_order(int *id, int *slot, int N) {
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if(i >= N) return;
	id[i] = i;
	slot[i] = i;
}

cudaError_t launch_identity_order(int *id, int *slot, int N, cudaStream_t s) {
	k_identity_order<<<blocks_for(N, 256), 256, 0, s>>>(id, slot, N);
	return cudaGetLastError();
}

cudaError_t launch_pack_state(const StepArgs &a, double *out, cudaStream_t s) {
	k_pack_state<<<blocks_for(a.N, 256), 256, 0, s>>>(a, out);
	return cudaGetLastError();
}

cudaError_t launch_scale_momenta(const StepArgs &a, int lo, int hi, double f, cudaStream_t s) {
	if(hi > lo) k_scale_momenta<<<blocks_for(hi - lo, 256), 256, 0, s>>>(a, lo, hi, f);
	return cudaGetLastError();
}

cudaError_t launch_system_sums(const StepArgs &a, int n_chunks, bool double_forces, double *out, cudaStream_t s) {
	if(double_forces) k_system_sums<double4_32a><<<n_chunks, 256, 0, s>>>(a, out);
	else k_system_sums<float4><<<n_chunks, 256, 0, s>>>(a, out);
	return cudaGetLastError();
}

}  // namespace oxgb
