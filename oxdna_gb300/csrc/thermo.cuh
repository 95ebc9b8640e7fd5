// Random streams and thermostat arithmetic of the integrator kernels (integrate.cu).
//
// Random numbers come from a counter-based Philox-4x32-10 stream keyed by (seed, step,
// particle), so runs are reproducible and graph-replayable; the oracle (oracle/dna2_oracle.c,
// oxo_philox) draws the same numbers.  The Bussi kinetic-energy update follows
// src/Backends/Thermostats/BussiThermostat.cpp:44-160 and the Brownian ("john") redraw
// src/CUDA/Thermostats/CUDABrownianThermostat.cu:15-51.
#pragma once

#include "kernels.h"

namespace oxgb {

// ---------------------------------------------------------------- Philox-4x32-10

static __device__ __forceinline__ void philox(unsigned k0, unsigned k1, unsigned c0, unsigned c1, unsigned c2, unsigned c3,
		unsigned out[4]) {
	const unsigned M0 = 0xD2511F53u, M1 = 0xCD9E8D57u, W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
#pragma unroll
	for(int r = 0; r < 10; r++) {
		const unsigned hi0 = __umulhi(M0, c0), lo0 = M0 * c0;
		const unsigned hi1 = __umulhi(M1, c2), lo1 = M1 * c2;
		const unsigned n0 = hi1 ^ c1 ^ k0, n2 = hi0 ^ c3 ^ k1;
		c0 = n0;
		c1 = lo1;
		c2 = n2;
		c3 = lo0;
		k0 += W0;
		k1 += W1;
	}
	out[0] = c0;
	out[1] = c1;
	out[2] = c2;
	out[3] = c3;
}

static __device__ __forceinline__ double u01(unsigned x) { return ((double) x + 1.0) * (1.0 / 4294967296.0); }

// (one compiled copy, so that a redraw has the same bits wherever it is made)
static __device__ __noinline__ double2 box_muller(unsigned ua, unsigned ub) {
	const double r = sqrt(-2.0 * log(u01(ua)));
	double s, c;
	sincospi(2.0 * u01(ub), &s, &c);
	return make_double2(r * c, r * s);
}

#define RNG_BROWNIAN 0x42524f57u
#define RNG_BUSSI 0x42555353u

struct Stream {
	unsigned k0, k1, s0, s1, c, blk, idx;
	unsigned buf[4];
	__device__ void init(unsigned long long seed, long long s, unsigned channel) {
		k0 = (unsigned) seed;
		k1 = (unsigned) (seed >> 32);
		s0 = (unsigned) s;
		s1 = (unsigned) ((unsigned long long) s >> 32);
		c = RNG_BUSSI ^ channel;
		blk = 0;
		idx = 4;
	}
	__device__ double u() {
		if(idx == 4) {
			philox(k0, k1, s0, s1, c, blk++, buf);
			idx = 0;
		}
		return u01(buf[idx++]);
	}
	__device__ double gauss() {
		const double a = u(), b = u();
		return sqrt(-2.0 * log(a)) * cos(6.283185307179586 * b);
	}
};

// gamma deviate of integer order (the Numerical Recipes algorithm the reference uses)
static __device__ double gamdev(Stream &st, int ia) {
	if(ia < 6) {
		double x = 1.0;
		for(int j = 1; j <= ia; j++) x *= st.u();
		return -log(x);
	}
	const double am = ia - 1, s = sqrt(2.0 * am + 1.0);
	double x = am, e, y = 0.0, v1, v2;
	// every rejection loop is bounded; each accepts with probability > 0.5, so the bounds are
	// never reached by a working random stream
	for(int guard = 0; guard < 1000; guard++) {
		bool got = false;
		for(int g2 = 0; g2 < 1000 && !got; g2++) {
			for(int g1 = 0; g1 < 1000; g1++) {
				v1 = st.u();
				v2 = 2.0 * st.u() - 1.0;
				if(v1 * v1 + v2 * v2 <= 1.0) break;
			}
			y = v2 / v1;
			x = s * y + am;
			got = x > 0.0;
		}
		if(!got) return am;
		e = (1.0 + y * y) * exp(am * log(x / am) - s * y);
		if(st.u() <= e) return x;
	}
	return am;
}

static __device__ double sum_noises(Stream &st, int nn) {
	if(nn == 0) return 0.0;
	if(nn == 1) {
		const double r = st.gauss();
		return r * r;
	}
	if(nn % 2 == 0) return 2.0 * gamdev(st, nn / 2);
	const double r = st.gauss();
	return 2.0 * gamdev(st, (nn - 1) / 2) + r * r;
}

// the two draws of one kinetic-energy update (BussiThermostat::_update_K, BussiThermostat.cpp:
// 55-65): the Gaussian r, then the sum of dof - 1 squared Gaussians; they do not depend on the
// state, so they are drawn apart from (and concurrently with) the force evaluation
static __device__ void bussi_draws(Stream &st, int dof, double &sum, double &rr) {
	rr = st.gauss();
	sum = sum_noises(st, dof - 1);
}

// K <- K + (1 - c) (K_target (sum + rr^2) / dof - K) + 2 rr sqrt(K K_target / dof (1 - c) c) with
// K_target = dof T / 2 (BussiThermostat::_update_K), written with the host-side constants
// a = (1 - c) T / 2 and b = sqrt(2 T (1 - c) c), so that the device chain is short
static __device__ __forceinline__ void update_K(double &K, double one_minus_c, double a, double b, double sum, double rr) {
	K += a * (sum + rr * rr) - one_minus_c * K + b * rr * sqrt(K);
}

// Brownian ("john") thermostat: every newtonian_steps steps each nucleotide redraws its
// velocity with probability pt and its angular momentum with probability pr from the
// Maxwell-Boltzmann distribution at T (unit mass and moment of inertia).  Keyed by the
// system's seed, the step and the index within the system.
static __device__ __noinline__ void brownian_redraw(const ThermoArgs &t, int sy, int i_local, long long s, double4_32a &v,
		double4_32a &L) {
	const double *par = t.sys_par + sy * SP_STRIDE;
	const unsigned long long seed = t.sys_seed[sy];
	unsigned o0[4], o1[4];
	const unsigned k0 = (unsigned) seed, k1 = (unsigned) (seed >> 32);
	const unsigned s0 = (unsigned) s, s1 = (unsigned) ((unsigned long long) s >> 32);
	philox(k0, k1, s0, s1, RNG_BROWNIAN, (unsigned) (2 * i_local), o0);
	philox(k0, k1, s0, s1, RNG_BROWNIAN, (unsigned) (2 * i_local + 1), o1);
	const double sT = par[SP_SQRTT];
	const bool dv = drawn(o0[0], par[SP_PT]), dL = drawn(o0[1], par[SP_PR]);
	if(!(dv || dL)) return;
	const double2 b = box_muller(o1[0], o1[1]);
	if(dv) {
		const double2 c = box_muller(o0[2], o0[3]);
		v = make_double4_32a(c.x * sT, c.y * sT, b.x * sT, 0.0);
	}
	if(dL) {
		const double2 c = box_muller(o1[2], o1[3]);
		L = make_double4_32a(b.y * sT, c.x * sT, c.y * sT, 0.0);
	}
}

// The redraws of a block of W pairs of warps, warp w < W the velocities of 32 nucleotides and warp w + W
// their angular momenta (`rot`), with the same draws as brownian_redraw: whether this lane's is redrawn, and
// to what (g).  A redraw takes two pairs of normal deviates, each a logarithm, a square root, a sine and a
// cosine on the slow FP64 pipe, some 150 operations that take as long for one lane as for all: so the pairs of
// the lanes that redraw (a tenth of them at most, commonly a hundredth) are dealt to all threads.  The whole
// block calls, ahead of its wait for the forces.  Measured for 32,000 nucleotides of which a tenth is redrawn
// in every step, us per step: dealt over a warp and after the wait 45.1, over one pair of warps and before it
// 35.4, over two pairs 30.6, four 31.0.
template <int W>
struct RedrawPool {
	uint2 key[128 * W];
	double2 dev[128 * W];
	int count[2 * W];
};

template <int W>
static __device__ __noinline__ bool brownian_redraws(const ThermoArgs &t, RedrawPool<W> &y, int sy, int i_local, long long s, bool rot,
		bool live, double4_32a &g) {
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	unsigned o0[4], o1[4];
	bool redraw = false;
	if(live) {
		const double *par = t.sys_par + sy * SP_STRIDE;
		const unsigned long long seed = t.sys_seed[sy];
		const unsigned k0 = (unsigned) seed, k1 = (unsigned) (seed >> 32);
		const unsigned s0 = (unsigned) s, s1 = (unsigned) ((unsigned long long) s >> 32);
		philox(k0, k1, s0, s1, RNG_BROWNIAN, (unsigned) (2 * i_local), o0);
		redraw = rot ? drawn(o0[1], par[SP_PR]) : drawn(o0[0], par[SP_PT]);
		if(redraw) philox(k0, k1, s0, s1, RNG_BROWNIAN, (unsigned) (2 * i_local + 1), o1);
	}
	const unsigned who = __ballot_sync(0xffffffffu, redraw);
	if(lane == 0) y.count[warp] = __popc(who);
	__syncthreads();
	int total = 0, at = 0;
#pragma unroll
	for(int w = 0; w < 2 * W; w++) {
		if(w == warp) at = total;
		total += y.count[w];
	}
	if(total == 0) return false;  // (block-uniform)
	at = 2 * (at + __popc(who & ((1u << lane) - 1u)));
	// the two pairs of a nucleotide: velocity g0 g1 | g2 -, angular momentum - g3 | g4 g5
	if(redraw) {
		y.key[at] = rot ? make_uint2(o1[0], o1[1]) : make_uint2(o0[2], o0[3]);
		y.key[at + 1] = rot ? make_uint2(o1[2], o1[3]) : make_uint2(o1[0], o1[1]);
	}
	__syncthreads();
	for(int q = threadIdx.x; q < 2 * total; q += 64 * W) y.dev[q] = box_muller(y.key[q].x, y.key[q].y);
	__syncthreads();
	if(!redraw) return false;
	const double sT = t.sys_par[sy * SP_STRIDE + SP_SQRTT];
	const double2 p0 = y.dev[at], p1 = y.dev[at + 1];
	g = rot ? make_double4_32a(p0.y * sT, p1.x * sT, p1.y * sT, 0.0) : make_double4_32a(p0.x * sT, p0.y * sT, p1.x * sT, 0.0);
	return true;
}

// Bussi: the new running kinetic energy of one kind of motion of system sy (which = 0 translation, 1
// rotation) from this step's draws, and its square root.  It needs no sums, so it is off the chain from the
// forces to the rescaling.
static __device__ void bussi_advance(const ThermoArgs &t, int sy, int which) {
	const double *par = t.sys_par + sy * SP_STRIDE;
	double *st = t.bussi_state + 16 * sy;
	const double *dr = t.bussi_draws + 4 * ((size_t) t.step_offset * t.n_systems + sy) + 2 * which;
	update_K(st[which], par[SP_1MC], par[SP_A], par[SP_B], __ldcg(dr), __ldcg(dr + 1));
	st[8 + which] = sqrt(st[which]);
}

// the rescaling factor of one kind of motion (translation: about the centre-of-mass velocity) from the sums
// of v, |v|^2 and |L|^2 over system sy; root: bussi_advance's, inv_n: 1 / n
static __device__ __forceinline__ void bussi_factor(const ThermoArgs &t, int sy, int which, const double sum[5], double root,
		double inv_n, double n) {
	double *st = t.bussi_state + 16 * sy;
	if(which == 0) {
		const double vc[3] = {sum[0] * inv_n, sum[1] * inv_n, sum[2] * inv_n};
		const double Kt_now = 0.5 * (sum[3] - n * (vc[0] * vc[0] + vc[1] * vc[1] + vc[2] * vc[2]));
		st[2] = root * rsqrt(Kt_now);
		st[4] = vc[0];
		st[5] = vc[1];
		st[6] = vc[2];
	}
	else st[3] = root * rsqrt(0.5 * sum[4]);
}

// one kind of motion of bussi_rescale (which = 0: the velocity, 1: the angular momentum)
static __device__ __forceinline__ void bussi_rescale_part(const ThermoArgs &t, int sy, int which, double4_32a &x) {
	const double *st = t.bussi_state + 16 * sy;
	if(which == 0) {
		const double ft = __ldcg(st + 2), cx = __ldcg(st + 4), cy = __ldcg(st + 5), cz = __ldcg(st + 6);
		x.x = (x.x - cx) * ft + cx;
		x.y = (x.y - cy) * ft + cy;
		x.z = (x.z - cz) * ft + cz;
	}
	else {
		const double fr = __ldcg(st + 3);
		x.x *= fr;
		x.y *= fr;
		x.z *= fr;
	}
}

// the rescaling of the last Bussi update of system sy, applied to one nucleotide
static __device__ __forceinline__ void bussi_rescale(const ThermoArgs &t, int sy, double4_32a &v, double4_32a &L) {
	const double *st = t.bussi_state + 16 * sy;
	const double ft = __ldcg(st + 2), fr = __ldcg(st + 3), cx = __ldcg(st + 4), cy = __ldcg(st + 5), cz = __ldcg(st + 6);
	v.x = (v.x - cx) * ft + cx;
	v.y = (v.y - cy) * ft + cy;
	v.z = (v.z - cz) * ft + cz;
	L.x *= fr;
	L.y *= fr;
	L.z *= fr;
}

}  // namespace oxgb
