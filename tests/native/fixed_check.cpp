// fixed_coord against extended precision, and draw_threshold's test on integers against the division it stands
// for; prints what failed and returns 1.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "split.cuh"

using namespace oxgb;

static double threshold(double p) {  // (the rule of kernels.h, which needs CUDA's headers)
	const double c = std::ceil(p * 4294967296.0) - 1.0;
	return c > 0.0 ? c : 0.0;
}

int main(int argc, char **argv) {
	const int n = argc > 1 ? atoi(argv[1]) : 100000;
	std::mt19937_64 rng(3);
	std::uniform_real_distribution<double> u(0, 1);
	double worst = 0;
	for(int k = 0; k < n; k++) {
		const double L = std::exp(std::log(4.0) + u(rng) * std::log(500.0)), s = 2147483648.0 / L;  // (fixed_coord takes 2^31 / box)
		const float box_hi = (float) L, box_lo = (float) (L - (double) box_hi), inv = 1.f / box_hi;
		const float s_hi = (float) s, s_lo = (float) (s - (double) s_hi);
		double x = (u(rng) - 0.5) * 40.0 * L;  // unwrapped, many boxes away
		if(k % 4 == 0) x = (k % 8 ? 0.5 : -0.5) * L * (1.0 + 1e-7 * (u(rng) - 0.5));  // at the faces
		if(k % 16 == 1) x = 0.0;
		const float hi = (float) x, lo = (float) (x - (double) hi);
		const unsigned got = fixed_coord(hi, lo, box_hi, box_lo, inv, s_hi, s_lo);
		const long double t = ((long double) hi + lo) / L, frac = t - floorl(t);
		long double d = (long double) got - frac * 4294967296.0L;
		d -= 4294967296.0L * roundl(d / 4294967296.0L);
		// two roundings of half a unit, the FP32 products' remainders (2^-47 of 2^31), and hi + lo's own
		// rounding (2^-48 of the coordinate, up to 20 boxes) with the box's (2^-48 per box)
		const long double bound = 1.25L + fabsl(t) * 4294967296.0L * ldexpl(1, -46);
		if(fabsl(d) > bound) {
			printf("fixed_coord(%.17g, L %.17g): off by %Lg units, bound %Lg\n", x, L, d, bound);
			return 1;
		}
		if(fabsl(d) > worst) worst = (double) fabsl(d);
	}
	for(int k = 0; k < n; k++) {
		double p = k % 3 == 0 ? u(rng) : k % 3 == 1 ? std::exp(-30 * u(rng)) : (double) (rng() >> 32) / 4294967296.0;
		if(k == 0) p = 0;
		if(k == 3) p = 1;
		const double c = threshold(p);
		for(long long x : {(long long) c - 1, (long long) c, (long long) c + 1, (long long) (rng() >> 32)}) {
			if(x < 0 || x > 4294967295LL) continue;
			const bool want = ((double) x + 1.0) / 4294967296.0 < p, got = (double) x < c;
			if(want != got) {
				printf("threshold(%.17g): draw %lld\n", p, x);
				return 1;
			}
		}
	}
	printf("fixed_coord within %.3f units\n", worst);
	return 0;
}
