// The device arithmetic of qpc_fixed.cuh on its own: prints the largest error of quant, of to_double in both forms and of
// reciprocal, each in units of what it may be off.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>
#include "qpc_fixed.cuh"

using namespace qpc;

struct item {
	long long h, m;
	int s, E;
	double v, x;
	double wide, narrow, rec;	// out
	int2 q;
};

__global__ void k_check(item* t, int n)
{
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n) return;
	t[i].wide = to_double<true>(t[i].h, t[i].m, t[i].s, false);
	t[i].narrow = to_double<false>(t[i].h >> 2, t[i].m, t[i].s, false);	// |h| < 2^61
	t[i].rec = reciprocal(t[i].x);
	t[i].q = quant(t[i].v, t[i].E);
}

// |y - (h + m 2^-28) 2^s| over 2^(s - 2) (what is cut off below the 64 bits kept) + 2^-53 |y| (one rounding).  Both
// sides as integers of 2^(s - 62): h and m exactly, y exactly where it is no smaller than that.
static double off(double y, long long h, long long m, int s)
{
	const long double v = ((long double)h + std::ldexp((long double)m, -28));	// exact, or to 2^-64 of h
	const long double got = std::ldexp((long double)y, -s);
	return (double)(std::fabs(got - v) / (0.25L + std::ldexp(std::fabs(v), -53) * (1.0L + 1.0L / 256)));
}

int main()
{
	const int n = 1 << 16;
	std::vector<item> t(n);
	std::mt19937_64 g(7);
	for (int i = 0; i < n; ++i) {
		item& a = t[i];
		const int bits = 1 + (int)(g() % 63);	// magnitudes of every size up to 2^63
		a.h = (long long)(g() >> (64 - bits));
		if (i % 16 == 0) a.h = (1ll << (bits - 1)) - 1 + (long long)(g() % 3);	// beside the powers of two
		if (a.h < 0) a.h = 0x7fffffffffffffffll;
		if (g() & 1) a.h = -a.h;
		a.m = (long long)(g() >> 36);
		a.s = (int)(g() % 1600) - 900;
		a.E = 200 + (int)(g() % 1700);
		const double f = std::ldexp((double)(g() >> 11) * std::ldexp(1.0, -53), -(int)(g() % 70));	// [0, 1) of every size
		a.v = std::ldexp((g() & 1) ? f : -f, a.E - 1022);
		a.x = std::ldexp(1.0 + (double)(g() >> 12) * std::ldexp(1.0, -52), (int)(g() % 130));
		if (i % 16 == 1) a.x = std::nextafter(std::ldexp(1.0, (int)(g() % 99) + 1), (g() & 1) ? 0.0 : 1e300);
		if (i == 2) a.x = 1.0;
	}
	item* d = nullptr;
	if (cudaMalloc(&d, sizeof(item) * n) != cudaSuccess || cudaMemcpy(d, t.data(), sizeof(item) * n, cudaMemcpyHostToDevice) != cudaSuccess) return 1;
	k_check<<<(n + 255) / 256, 256>>>(d, n);
	if (cudaMemcpy(t.data(), d, sizeof(item) * n, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
	cudaFree(d);
	double wide = 0, narrow = 0, rec = 0, qu = 0;
	for (const item& a : t) {
		wide = std::fmax(wide, off(a.wide, a.h, a.m, a.s));
		narrow = std::fmax(narrow, off(a.narrow, a.h >> 2, a.m, a.s));
		rec = std::fmax(rec, std::fabs(a.rec * 1.0L * a.x - 1.0L) * 4503599627370496.0);	// of 2^-52
		const long long x = (long long)a.q.x * (1ll << 28) + a.q.y;
		const bool limbs = std::abs((long long)a.q.x) <= (1ll << 28) && a.q.y >= -(1 << 27) && a.q.y < (1 << 27);
		qu = std::fmax(qu, limbs ? 2.0 * std::fabs((double)((long double)x - std::ldexp((long double)a.v, 1078 - a.E))) : 1e9);	// of half a unit
	}
	std::printf("quant %.17g\nto_double_wide %.17g\nto_double %.17g\nreciprocal %.17g\n", qu, wide, narrow, rec);
	return 0;
}
