// drawn with draw_threshold's value (an integer in the bits of a double) against the division of the draw that it
// stands for, at the draws next to the threshold, the ends of their range and random ones; prints what failed and
// returns 1.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "split.cuh"

using namespace oxgb;

int main(int argc, char **argv) {
	const int n = argc > 1 ? atoi(argv[1]) : 100000;
	std::mt19937_64 rng(11);
	std::uniform_real_distribution<double> u(0, 1);
	const double ends[] = {0.0, -0.25, 1.0, 1.5, 1e300, 1.0 / 4294967296.0, 2.0 / 4294967296.0, 0.5, 4294967295.0 / 4294967296.0,
			std::nan(""), 5e-324, 1e-12, std::nextafter(1.0, 0.0), std::nextafter(1.0, 2.0)};
	const int m = (int) (sizeof ends / sizeof ends[0]);
	for(int k = 0; k < n; k++) {
		const double p = k < m ? ends[k] : k % 3 == 0 ? u(rng) : k % 3 == 1 ? std::exp(-30 * u(rng)) : (double) (rng() >> 32) / 4294967296.0;
		const double t = draw_threshold(p);
		const double at = p > 0 ? std::fmin(p, 2.0) * 4294967296.0 : 0.0;
		long long x[9] = {0, 1, 4294967294LL, 4294967295LL, (long long) (rng() >> 32)};
		for(int d = 0; d < 4; d++) x[5 + d] = (long long) at - 2 + d;
		for(long long v : x) {
			if(v < 0 || v > 4294967295LL) continue;
			const bool want = ((double) v + 1.0) * (1.0 / 4294967296.0) < p, got = drawn((unsigned) v, t);
			if(want != got) {
				printf("p %.17g, draw %lld: drawn %d, want %d\n", p, v, (int) got, (int) want);
				return 1;
			}
		}
	}
	return 0;
}
