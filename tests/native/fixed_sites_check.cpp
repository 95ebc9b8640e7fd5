// The separation of two fixed-point sites against the minimum image in extended precision, pairs on both sides of a
// face of the box among them; prints what failed and returns 1.  Built with checks for undefined arithmetic.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "split.cuh"

using namespace oxgb;

int main(int argc, char **argv) {
	const int n = argc > 1 ? atoi(argv[1]) : 100000;
	std::mt19937_64 rng(5);
	std::uniform_real_distribution<double> u(0, 1);
	double worst = 0;
	int across = 0;
	for(int k = 0; k < n; k++) {
		const double L = std::exp(std::log(8.0) + u(rng) * std::log(100.0)), s = 2147483648.0 / L;
		const float box_hi = (float) L, box_lo = (float) (L - (double) box_hi), inv = 1.f / box_hi;
		const float s_hi = (float) s, s_lo = (float) (s - (double) s_hi), s2 = 2.f * s_hi;
		// centres up to 3 apart, in any images; offsets of a site
		double x[2];
		x[0] = k % 3 == 0 ? 0.5 * L * (1.0 - 2e-8 * u(rng)) : k % 3 == 1 ? -1e-6 * u(rng) : (u(rng) - 0.5) * 20.0 * L;
		x[1] = x[0] + 6.0 * (u(rng) - 0.5) + (k % 5 ? 0.0 : L * std::floor(10.0 * (u(rng) - 0.5)));
		int site[2];
		unsigned c[2];
		long double t[2];
		for(int m = 0; m < 2; m++) {
			const float hi = (float) x[m], lo = (float) (x[m] - (double) hi), off = (float) (1.1 * (u(rng) - 0.5));
			c[m] = fixed_coord(hi, lo, box_hi, box_lo, inv, s_hi, s_lo);
			site[m] = fixed_site(c[m], off * s2);
			t[m] = ((long double) hi + lo + off) / L * 4294967296.0L;
		}
		long double d = t[1] - t[0];
		d -= 4294967296.0L * roundl(d / 4294967296.0L);
		across += ((site[1] ^ site[0]) < 0) && fabsl(d) < 1e9L;
		// a site: fixed_coord's error (tests/native/fixed_check.cpp), half a unit of its own and the offset's
		// FP32 product and scale (2^-23 of 0.55 / L 2^32)
		long double bound = 0;
		for(int m = 0; m < 2; m++) bound += 1.75L + fabsl(t[m]) * ldexpl(1, -46) + 0.56L / L * ldexpl(1, 9);
		const long double e = fabsl((long double) fixed_sep(site[1], site[0]) - d);
		if(e > bound) {
			printf("separation of %.17g and %.17g in a box of %.17g: off by %Lg units, bound %Lg\n", x[0], x[1], L, e, bound);
			return 1;
		}
		if(e > worst) worst = (double) e;
	}
	if(across < n / 10) {
		printf("only %d pairs across a face\n", across);
		return 1;
	}
	printf("separations within %.2f units, %d across a face\n", worst, across);
	return 0;
}
