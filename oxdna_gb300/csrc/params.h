// Host-side derivation of the oxDNA2 parameter tables from the user settings.
//
// Restates DNAInteraction::DNAInteraction + init and DNA2Interaction::DNA2Interaction +
// get_settings + init (src/Interactions/DNAInteraction.cpp:12-213,290-380,
// src/Interactions/DNA2Interaction.cpp:5-21,62-155) with the reference's mixed float/double
// arithmetic: model constants are floats, so float-only sub-expressions are evaluated in float
// (the Morse-shift exponent, the Debye-Hueckel T / 0.1f, the salt read as a float) while the
// math functions are double.
#pragma once

#include <cmath>
#include <cstddef>
#include <cstring>

#include "../../include/oxgb.h"
#include "dna2_pair.cuh"

namespace oxgb {

inline void default_settings(oxgb_dna2_settings *s, double T, double salt) {
	std::memset(s, 0, sizeof(*s));
	s->T = T;
	s->salt = salt;
	s->average = 1;
	s->hb_multiplier = 1.0;
	s->dh_half_charged_ends = 1;
	s->dh_lambda = OXM_DH_LAMBDA_DEFAULT;
	s->dh_strength = OXM_DH_STRENGTH_DEFAULT;
	s->mbf_finf = 0.04;
}

// returns 0, or -1 for invalid settings
inline int build_table(const oxgb_dna2_settings &s, double box, DNA2Table<double> &P, double &rcut) {
	static const float f1a[2] = OXM_F1_TABLE_A, f1rc[2] = OXM_F1_TABLE_RC, f1r0[2] = OXM_F1_TABLE_R0;
	if(!(s.T > 0) || !(s.salt > 0) || !(box > 0)) return -1;
	std::memset(&P, 0, sizeof(P));
	const double T = s.T;
	// exponent in float arithmetic on the float constants, exp in double
	const double st_x = 1 - std::exp((double) (-(f1rc[1] - f1r0[1]) * f1a[1]));
	const double hb_x = 1 - std::exp((double) (-(f1rc[0] - f1r0[0]) * f1a[0]));
	const double st_shift = st_x * st_x, hb_shift = hb_x * hb_x;
	const bool oxdna2_avg = s.average && !s.reference_cuda_eps;
	for(int i = 0; i < 5; i++) {
		for(int j = 0; j < 5; j++) {
			P.f1_eps[1][i][j] = oxdna2_avg ? OXM_STCK_BASE_EPS_OXDNA2 + OXM_STCK_FACT_EPS_OXDNA2 * T
										   : OXM_STCK_BASE_EPS_OXDNA + OXM_STCK_FACT_EPS_OXDNA * T;
			P.f1_eps[0][i][j] = oxdna2_avg ? OXM_HYDR_EPS_OXDNA2 : OXM_HYDR_EPS_OXDNA;
		}
	}
	if(!s.average) {
		const float fe = (float) s.seq_stck_fact_eps;
		float last = 0.f;
		for(int i = 0; i < 4; i++) {
			for(int j = 0; j < 4; j++) {
				last = (float) s.seq_stck[i][j];
				P.f1_eps[1][i][j] = last * (1.0 - fe + (T * 9.0 * fe));
			}
		}
		// entries of the dummy base keep the last value read when the file has none of them
		for(int i = 0; i < 5; i++)
			for(int j = 0; j < 5; j++)
				if(i == 4 || j == 4) P.f1_eps[1][i][j] = last * (1.0 - fe + (T * 9.0 * fe));
		const float at = (float) s.seq_hydr_at, gc = (float) s.seq_hydr_gc;
		P.f1_eps[0][0][3] = P.f1_eps[0][3][0] = at;
		P.f1_eps[0][1][2] = P.f1_eps[0][2][1] = gc;
	}
	for(int i = 0; i < 5; i++) {
		for(int j = 0; j < 5; j++) {
			P.f1_shift[1][i][j] = P.f1_eps[1][i][j] * st_shift;
			P.f1_shift[0][i][j] = P.f1_eps[0][i][j] * hb_shift;
		}
	}
	P.hb_multiplier = s.hb_multiplier;

	P.use_mbf = s.use_mbf ? 1 : 0;
	if(s.use_mbf) {
		if(!(s.mbf_fmax > 0) || s.mbf_finf < 0) return -1;
		P.mbf_fmax = s.mbf_fmax;
		P.mbf_finf = s.mbf_finf;
		P.mbf_xmax = (-OXM_FENE_EPS + std::sqrt(OXM_FENE_EPS * OXM_FENE_EPS + 4.f * s.mbf_fmax * s.mbf_fmax * OXM_FENE_DELTA2)) /
				(2.f * s.mbf_fmax);
		P.mbf_fene_xmax = -(OXM_FENE_EPS / 2.f) * std::log(1.f - P.mbf_xmax * P.mbf_xmax / OXM_FENE_DELTA2);
		P.mbf_long_xmax = (P.mbf_fmax - P.mbf_finf) * P.mbf_xmax * std::log(P.mbf_xmax) + P.mbf_finf * P.mbf_xmax;
	}

	P.dh_half_charged_ends = s.dh_half_charged_ends ? 1 : 0;
	P.dh_prefactor = s.dh_strength;
	const double salt = (double) (float) s.salt;
	const double lambda_rhigh = s.dh_lambda * std::sqrt(T / 0.1f) / std::sqrt(salt);
	P.dh_rhigh = 3.0 * lambda_rhigh;
	const double lambda = s.dh_lambda * std::sqrt(T / 0.1) / std::sqrt(salt);
	P.dh_minus_kappa = -1.0 / lambda;
	const double x = P.dh_rhigh, q = P.dh_prefactor, l = lambda;
	P.dh_b = -(std::exp(-x / l) * q * q * (x + l) * (x + l)) / (-4. * x * x * x * l * l * q);
	P.dh_rc = x * (q * x + 3. * q * l) / (q * (x + l));

	const double rcutback = 2 * std::sqrt((double) ((OXM_POS_MM_BACK1) * (OXM_POS_MM_BACK1) + (OXM_POS_MM_BACK2) * (OXM_POS_MM_BACK2))) + OXM_EXCL_RC1;
	const double rcutbase = 2 * std::fabs(OXM_POS_BASE) + OXM_HYDR_RCHIGH;
	rcut = std::fmax(rcutback, rcutbase);
	const double debyecut = 2.0 * std::sqrt((double) (OXM_POS_MM_BACK1 * OXM_POS_MM_BACK1 + OXM_POS_MM_BACK2 * OXM_POS_MM_BACK2)) + P.dh_rc;
	if(debyecut > rcut) rcut = debyecut;
	P.rcut2 = rcut * rcut;
	P.box_hi = box;
	P.box_lo = 0.0;
	P.inv_box = 1.0 / box;
	P.fix_hi = 2147483648.0 / box;
	P.fix_lo = 0.0;
	P.fix_unit = box / 4294967296.0;
	P.fix_unit2 = P.fix_unit * P.fix_unit;
	return 0;
}

// FP32 copy of a table; the box side is split into a float and the float of the remainder
inline void to_float(const DNA2Table<double> &d, double box, DNA2Table<float> &f) {
	const double *src = reinterpret_cast<const double *>(&d);
	float *dst = reinterpret_cast<float *>(&f);
	// every member before the int fields is a double / float, in the same order
	const size_t nreal = offsetof(DNA2Table<double>, dh_half_charged_ends) / sizeof(double);
	for(size_t k = 0; k < nreal; k++) dst[k] = (float) src[k];
	f.dh_half_charged_ends = d.dh_half_charged_ends;
	f.use_mbf = d.use_mbf;
	f.box_hi = (float) box;
	f.box_lo = (float) (box - (double) f.box_hi);
	f.inv_box = (float) (1.0 / (double) f.box_hi);
	f.fix_lo = (float) (2147483648.0 / box - (double) f.fix_hi);
	f.fix_unit_lo = (float) (d.fix_unit - (double) f.fix_unit);
	f.fix_unit2_lo = (float) (d.fix_unit2 - (double) f.fix_unit2);
}

// pair-distance bounds of the force kernel's term lists: a term can only act within these
// distances (model constants), widened by twice the skin so that a list built now stays complete
// until the next rebuild.  ev: centre-centre (excluded volume), base: base-base (hydrogen bonding,
// cross stacking), stk: stack-stack (coaxial stacking); evs: the excluded volume's four site
// pairs, of which one must be within its bound for a pair to enter the excluded-volume list.
// Squared, FP32.
struct TermRadii {
	float ev2, base2, stk2;
	float evs2[3];  // site pairs of the excluded volume: backbone-backbone, base-base, backbone-base
};

inline TermRadii term_radii(double skin) {
	const double back = std::sqrt((double) OXM_POS_MM_BACK1 * OXM_POS_MM_BACK1 + (double) OXM_POS_MM_BACK2 * OXM_POS_MM_BACK2);
	const double base = OXM_POS_BASE;
	double ev = OXM_EXCL_RC1 + 2 * back;                     // back-back
	ev = std::fmax(ev, (double) OXM_EXCL_RC2 + 2 * base);     // base-base
	ev = std::fmax(ev, (double) OXM_EXCL_RC3 + base + back);  // base-back
	const double hb = std::fmax((double) OXM_HYDR_RCHIGH, (double) OXM_CRST_RCHIGH);
	const double margin = 1e-3;
	TermRadii t;
	t.ev2 = (float) ((ev + 2 * skin + margin) * (ev + 2 * skin + margin));
	t.base2 = (float) ((hb + 2 * skin + margin) * (hb + 2 * skin + margin));
	t.stk2 = (float) (((double) OXM_CXST_RCHIGH + 2 * skin + margin) * ((double) OXM_CXST_RCHIGH + 2 * skin + margin));
	const double rc[3] = {OXM_EXCL_RC1, OXM_EXCL_RC2, std::fmax((double) OXM_EXCL_RC3, (double) OXM_EXCL_RC4)};
	for(int k = 0; k < 3; k++) t.evs2[k] = (float) ((rc[k] + 2 * skin + margin) * (rc[k] + 2 * skin + margin));
	return t;
}

// cells per side, CUDASimpleVerletList::_compute_N_cells_side
// (src/CUDA/Lists/CUDASimpleVerletList.cu:96-110), with the min-3 clamp applied last
inline int cells_per_side(int N, float L, float rverlet, bool auto_opt) {
	const float V3 = L * L * L;
	const float max_factor = (float) std::pow(2. * N / V3, 1. / 3.);
	const float min_cell = std::sqrt(rverlet * rverlet);
	int n = (int) (std::floor((double) L / (double) min_cell) + 0.1);
	if(auto_opt && n > std::ceil(max_factor * L)) n = (int) std::ceil(max_factor * L);
	if(n < 3) n = 3;
	return n;
}

}  // namespace oxgb
