// Fixed-point products of FP64 vectors with fixed real or complex matrices, as the kernels of qpc_radial.cu,
// qpc_pos.cu and qpc_vpos.cu form them (the arithmetic and its error: qpc_radial.cu): limbs, sums and the one
// rounding back.
#pragma once
#include <cuda_runtime.h>

namespace qpc {

constexpr int TM = 32;		// rows (positions) of a tile, one per lane
constexpr int KC = 16;		// k per chunk of the stored operators
constexpr int TE = 8;		// rows that share a recorded exponent
constexpr int EPT = TM / TE;
// largest exponent of a column whose product is formed: a sum of 2^5 units stays finite.  Beyond (5.6e306, infinities, NaN)
// the product is NaN, which a run reports
constexpr int EMAX = 2041;

__device__ __forceinline__ int bexp(double v) { return (__double2hiint(v) >> 20) & 0x7ff; }

// v as limbs (hi, lo), v = (hi 2^28 + lo) 2^(E - 1078), |hi| <= 2^28, -2^27 <= lo < 2^27; E >= bexp(v)
__device__ __forceinline__ int2 quant(double v, int E)
{
	const int h = __double2hiint(v);
	const int ex = (h >> 20) & 0x7ff;
	const int d = E - ex;
	unsigned long long m = ((unsigned long long)(unsigned)((h & 0xfffff) | 0x100000) << 32) | (unsigned)__double2loint(v);
	m <<= 3;
	m = (d > 57 || ex == 0) ? 0ull : (m + ((1ull << d) >> 1)) >> d;
	long long x = h < 0 ? -(long long)m : (long long)m;
	const int hi = (int)((x + (1ll << 27)) >> 28);
	return make_int2(hi, (int)(x - ((long long)hi << 28)));
}

// (h + m 2^-28) 2^s rounded to double, m in [0, 2^28), |h| < 2^61, or 2^63 if WIDE (infinite from 2^1024 on: an operator may
// grow its column); nf: the operand's exponent was above EMAX.  Two
// bits of m beside h, or from |h| = 2^61 on h alone, whose 62 bits leave m below the rounding.  2^61 is a sum of 32 in
// units of the column's power of two: rows of a dense orthogonal matrix reach sqrt(N), k_angle 8, k_couple 21, F~ 27 (where
// WIDE would cost 0.5 % of a step)
template <bool WIDE>
__device__ __forceinline__ double to_double(long long h, long long m, int s, bool nf)
{
	const bool wide = WIDE && (unsigned long long)(h + (1ll << 61)) >> 62;
	long long q = wide ? h : (h << 2) | (m >> 26);
	unsigned long long a = q < 0 ? 0ull - (unsigned long long)q : (unsigned long long)q;
	const int lz = __clzll((long long)a);
	const int e = 1023 + 63 - lz + s - (wide ? 0 : 2);
	a <<= (lz & 63);
	unsigned long long b = ((unsigned long long)(unsigned)(e - 1) << 52) + (a >> 11) + ((a >> 10) & 1ull);
	b |= (unsigned long long)q & 0x8000000000000000ull;
	if (WIDE && e > 2046) b = 0x7ff0000000000000ull;
	if (q == 0 || e < 1) b = 0ull;
	if (nf) b = 0x7ff8000000000000ull;
	return __longlong_as_double((long long)b);
}

// Kernels of a step follow each other on one stream by programmatic dependent launch (launch_after): a block may become
// resident and read what no kernel of a run writes (operators, tables) before the previous kernel has ended; prev_wait()
// holds it until that kernel, and so every one before it, is complete and its writes are visible.  Every block calls it
// before it reads or writes a state and before it can return, so a kernel never ends before the previous one.
// One wavefunction of 400 x 21, 120 steps of two kernels: 2.39 -> 1.77 ms; four with own potentials 1.57 -> 1.24 ms.
// Launches of many waves start in the usual order (256 wavefunctions: 13.6 against 13.8 ms).
__device__ __forceinline__ void prev_wait()
{
	asm volatile("griddepcontrol.wait;" ::: "memory");
	asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <class... P, class... A>
void launch_after(void (*k)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, A... a)
{
	cudaLaunchConfig_t c{};
	c.gridDim = grid; c.blockDim = dim3(threads); c.dynamicSmemBytes = smem; c.stream = st;
	cudaLaunchAttribute at[1];
	at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
	at[0].val.programmaticStreamSerializationAllowed = 1;
	c.attrs = at; c.numAttrs = (long)grid.x * grid.y <= 2000 ? 1 : 0;
	cudaLaunchKernelEx(&c, k, P(a)...);	// errors: the caller's cudaGetLastError
}

// the largest of e over each group of TE lanes
__device__ __forceinline__ int group_max(int e)
{
#pragma unroll
	for (int o = 1; o < TE; o <<= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
	return e;
}

__device__ __forceinline__ long long madw(int a, int b, long long c) { return c + (long long)a * b; }
__device__ __forceinline__ void flush(long long& h, long long& m) { h += m >> 28; m &= (1ll << 28) - 1; }

// v in [-1, 1] as limbs of unit 2^-56 (host side)
inline int2 limbs_of(double v)
{
	const long long x = __builtin_llrint(v * 72057594037927936.0);
	const int hi = (int)((x + (1ll << 27)) >> 28);
	return make_int2(hi, (int)(x - ((long long)hi << 28)));
}

// 1 / x, x >= 1: two Newton steps from the fp32 approximation (relative error 2^-23 -> 2^-46 -> rounding)
__device__ __forceinline__ double reciprocal(double x)
{
	if (!(x < 1e30)) return 1.0 / x;
	float r0;
	asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(__int_as_float(((__double2hiint(x) - 0x38000000) << 3) | (int)((unsigned)__double2loint(x) >> 29))));
	const int b = __float_as_int(r0);
	double r = __hiloint2double((b >> 3) + 0x38000000, b << 29);
	r = fma(r, fma(-x, r, 1.0), r);
	return fma(r, fma(-x, r, 1.0), r);
}

// G outputs of a real matrix, A = [k][G] limbs, times the column at x[k * XK]; the mixed sums hold 64 k (128 products
// below 2^55): LONG carries them into the high ones that often
template <int G, int XK, bool LONG>
__device__ __forceinline__ void task_product(const int2* __restrict__ A, int nk, const int4* __restrict__ x, long long (&h)[G][2], long long (&m)[G][2])
{
#pragma unroll
	for (int g = 0; g < G; ++g) h[g][0] = h[g][1] = m[g][0] = m[g][1] = 0;
	for (int k0 = 0; k0 < nk; k0 += LONG ? 64 : nk) {
		const int k1 = LONG ? min(nk, k0 + 64) : nk;
#pragma unroll 4
		for (int k = k0; k < k1; ++k) {
			const int4 y = x[k * XK];
#pragma unroll
			for (int g = 0; g < G; ++g) {
				const int2 a = __ldg(A + k * G + g);
				h[g][0] = madw(a.x, y.x, h[g][0]); h[g][1] = madw(a.x, y.z, h[g][1]);
				m[g][0] = madw(a.x, y.y, m[g][0]); m[g][0] = madw(a.y, y.x, m[g][0]);
				m[g][1] = madw(a.x, y.w, m[g][1]); m[g][1] = madw(a.y, y.z, m[g][1]);
			}
		}
#pragma unroll
		for (int g = 0; g < G; ++g) { flush(h[g][0], m[g][0]); flush(h[g][1], m[g][1]); }
	}
}

} // namespace qpc
