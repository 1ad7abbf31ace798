// The length-gauge Crank-Nicolson step in the position basis.
//
// One step is C(f) F C(f) with C(f) = P^T M(f) P, M = (S + i b R)^-1 (S - i b R) on every eigen-channel of
// Y10, b = lambda f dt/4, and F = (S + i dt/2 H_l)^-1 (S - i dt/2 H_l) per l (cn_propagate_kernel_avx1 and
// cn_hc_propagate0, spherical/propagator/propagate.hpp:3-98, 311-331).  With X the eigenvectors of the pencil
// (R, S), X^T S X = 1, X^T R X = diag(r_j), and c = X y:
//   * M(f) is diagonal: the phase ((1 - i b r_j)/(1 + i b r_j)) of channel k at position j.  No coupling
//     factorisation and no recurrence is left;
//   * F~_l = X^T S F_l X is one fixed unitary matrix per l.  Its entries fall off the diagonal by a constant
//     factor per row (0.70 at p = 6), so a band of ~110 either side holds it to 2^-57.
// A step is two kernels: k_angle (l transform, phases, l transform back, everything local in j) and
// k_band_apply (the banded products, everything local in l).
//
// Arithmetic.  GB300 issues 2 FP64 FMAs per cycle and SM (1.6 measured) and 20-25 wide integer multiply-adds
// (32 x 32 + 64 bits, distinct operands, measured).  Both products have fixed matrices with entries of magnitude
// <= 1 and vectors whose largest element is known, so they are formed in fixed point: 56 bits under the vector's
// largest exponent (matrix: under 1), as two balanced 28-bit limbs; hi*hi and the two mixed products are summed
// exactly in 64-bit integers (three multiply-adds per product: ~4 times the DFMA rate, and without its 64-cycle
// latency), lo*lo lies at 2^-56 of the unit and is left out; one rounding to FP64 at the end.  The quantisation is
// 2^-57 of the largest element of the ~250 a sum covers, below the FP64 rounding of the sum itself.  Entries of
// F~ below 2^-29 have no hi limb: the outer part of the band costs one multiply-add and half the bytes.
// Against the banded solves (GB300, per step): one wavefunction of 800 x 41 with its dipole 1340 -> 60 us,
// 400 x 21 287 -> 26 us, 24 wavefunctions of 517 x 30 1120 -> 200 us, 256 of 800 x 41 8.0 -> 3.3 ms; error against
// extended precision after 60 steps 3.3e-13 against 4.7e-13.
#include "qpc_pos.cuh"
#include "qpc_cuda_util.cuh"
#include <cstring>
#include <cmath>
#include <vector>
#include <cstdio>

namespace qpc {

namespace {

constexpr int TM = 32;		// rows of an output tile (one per lane)
constexpr int KC = 16;		// k per chunk of the stored operators
constexpr int WMAX = 176;	// widest band (either side of the diagonal) the path takes
constexpr int LMAX = 128;	// most l channels (the l transform's 64-bit sums)
constexpr int SEEDW = 40;	// half-width of the windows the starting vectors are found in

// ------------------------------------------------------------------ fixed point

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

// (h + m 2^-28) 2^s rounded to double, m in [0, 2^28), |h| < 2^61; nf: the operand was not finite
__device__ __forceinline__ double to_double(long long h, long long m, int s, bool nf)
{
	long long q = (h << 2) | (m >> 26);
	unsigned long long a = q < 0 ? 0ull - (unsigned long long)q : (unsigned long long)q;
	const int lz = __clzll((long long)a);
	const int e = 1023 + 63 - lz + s - 2;
	a <<= (lz & 63);
	unsigned long long b = ((unsigned long long)(unsigned)(e - 1) << 52) + (a >> 11) + ((a >> 10) & 1ull);
	b |= (unsigned long long)q & 0x8000000000000000ull;
	if (q == 0 || e < 1) b = 0ull;
	if (nf) b = 0x7ff8000000000000ull;
	return __longlong_as_double((long long)b);
}

__device__ __forceinline__ long long madw(int a, int b, long long c) { return c + (long long)a * b; }
__device__ __forceinline__ void flush(long long& h, long long& m) { h += m >> 28; m &= (1ll << 28) - 1; }

// ------------------------------------------------------------------ banded products
// dst[col][row] = sum_k A_l[row][k] src[col][k] for every channel l and column (wavefunction).  A block owns
// TM rows of one channel and COLS = NB * 8/KS columns; each warp NB columns (lane = row), KS warps share a
// column and split its k.  The operator is stored per tile as chunks of KC k x TM rows, so that a warp's load is
// 32 consecutive elements; the columns are quantised into shared memory once per block and read as broadcasts.
// Bound by the integer multiply-adds from ~8 columns on (12 NB per k and lane against one 16-byte load), by the
// operator's bytes below.
struct band_args {
	const char* A;		// operators, [set][nlh] of astride bytes
	long astride, set_stride;
	const int4* td;		// per tile: first chunk, first and end chunk with hi limbs, end chunk
	const long* toff;	// per tile: byte offset
	const int* lmap;	// channel -> operator of a set
	const int* amap;	// destination slot -> set (NULL: one set)
	int ea;			// |A| <= 2^ea
	int N, ntile, nchan, ncols;
	const double2 *s0, *s1;	// [slot][nchan][N]; s1 where par[slot] is odd
	const int *e0, *e1;	// largest biased exponent per [slot][nchan][tile]
	const int64_t* par;
	const int* smap;	// slot -> source slot (NULL: the same)
	const int* dmap;	// slot -> destination slot (NULL: the same)
	double2* dst;
	int* edst;
	const int64_t* nta;	// slots with step < nta[slot] take part (NULL: all)
	long step;
	int tile0;		// first tile of the launch
};

template <int NB, int KS, bool CX>
__global__ void __launch_bounds__(256, 2) k_band_apply(const band_args p)
{
	constexpr int CG = 8 / KS, COLS = NB * CG, SK = 32 * KS, XS = COLS | 1;
	constexpr int FB = KC * TM * (CX ? 16 : 8), TB = FB / 2;
	constexpr int UN = NB <= 1 ? 16 : (NB <= 2 ? 8 : (NB <= 4 ? 4 : 2));
	constexpr size_t XBYTES = sizeof(int4) * SK * XS, RBYTES = KS > 1 ? sizeof(long long) * 8 * NB * 4 * 32 : 0;
	constexpr size_t QBYTES = XBYTES > RBYTES ? XBYTES : RBYTES;
	extern __shared__ __align__(16) char smem[];
	double2* raw = reinterpret_cast<double2*>(smem + QBYTES);
	__shared__ int sE[COLS];
	__shared__ const double2* sp[COLS];
	int4* xs = reinterpret_cast<int4*>(smem);
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const int ncg = (p.ncols + COLS - 1) / COLS;
	const int cg = blockIdx.x % ncg, tile = p.tile0 + blockIdx.x / ncg, ch = blockIdx.y;
	const int col0 = cg * COLS;
	if (p.nta && KS == 8 && NB == 1 && !(p.step < p.nta[col0])) return;
	const int4 td = p.td[tile];
	const int t0 = td.x * KC / TM, t1 = min(p.ntile, (td.w * KC + TM - 1) / TM);
	if (threadIdx.x < COLS) {
		const int c = col0 + threadIdx.x;
		int e = 0;
		const double2* src = nullptr;
		if (c < p.ncols && (!p.nta || p.step < p.nta[c])) {
			const bool odd = p.par && (p.par[c] & 1);
			const long v = (long)(p.smap ? p.smap[c] : c) * p.nchan + ch;
			const int* ex = (odd ? p.e1 : p.e0) + v * p.ntile;
			for (int t = t0; t < t1; ++t) e = max(e, ex[t]);
			src = (odd ? p.s1 : p.s0) + v * p.N;
		}
		sE[threadIdx.x] = e;
		sp[threadIdx.x] = src;
	}
	// the stage's raw values arrive by cp.async in the order they are converted in (this thread's own elements)
	const int lk = threadIdx.x % SK;
	const int kend = min(p.N, td.w * KC);
	auto load = [&](int k) {
#pragma unroll
		for (int j = 0; j < NB; ++j) {
			const double2* s = sp[threadIdx.x / SK + j * (256 / SK)];
			const bool in = s && k < kend;
			const unsigned d = (unsigned)__cvta_generic_to_shared(raw + j * 256 + threadIdx.x);
			asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(in ? s + k : p.s0), "r"(in ? 16 : 0) : "memory");
		}
		asm volatile("cp.async.commit_group;" ::: "memory");
	};
	__syncthreads();
	load(td.x * KC + lk);
	const int ks = warp % KS, wc = (warp / KS) * NB;
	const int set = p.amap ? p.amap[p.dmap ? p.dmap[col0] : col0] : 0;
	const char* A = p.A + set * p.set_stride + (long)p.lmap[ch] * p.astride + p.toff[tile];
	const long tl = (long)(td.y - td.x) * TB, tf = tl + (long)(td.z - td.y) * FB;
	long long rh[NB], rm[NB], ih[NB], im[NB];
#pragma unroll
	for (int j = 0; j < NB; ++j) rh[j] = rm[j] = ih[j] = im[j] = 0;
	for (int c0 = td.x; c0 < td.w; c0 += 2 * KS) {
		asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
		for (int j = 0; j < NB; ++j) {
			const int c = threadIdx.x / SK + j * (256 / SK);
			const int E = sE[c];
			const double2 v = raw[j * 256 + threadIdx.x];
			const int2 a = quant(v.x, E), b = quant(v.y, E);
			xs[lk * XS + c] = make_int4(a.x, a.y, b.x, b.y);
		}
		__syncthreads();
		if (c0 + 2 * KS < td.w) load((c0 + 2 * KS) * KC + lk);
#pragma unroll
		for (int half = 0; half < 2; ++half) {
			const int c = c0 + 2 * ks + half;
			if (c >= td.w) break;
			const int4* x = xs + (ks * 32 + half * KC) * XS + wc;
			if (c >= td.y && c < td.z) {
				const char* a0 = A + tl + (long)(c - td.y) * FB;
				if (CX) {
					const int4* ap = reinterpret_cast<const int4*>(a0) + lane;
#pragma unroll UN
					for (int k = 0; k < KC; ++k) {
						const int4 a = __ldg(ap + k * TM);
						const int nz = -a.z, nw = -a.w;
#pragma unroll
						for (int j = 0; j < NB; ++j) {
							const int4 y = x[k * XS + j];
							rh[j] = madw(a.x, y.x, rh[j]); rh[j] = madw(nz, y.z, rh[j]);
							ih[j] = madw(a.x, y.z, ih[j]); ih[j] = madw(a.z, y.x, ih[j]);
							rm[j] = madw(a.x, y.y, rm[j]); rm[j] = madw(a.y, y.x, rm[j]);
							rm[j] = madw(nz, y.w, rm[j]); rm[j] = madw(nw, y.z, rm[j]);
							im[j] = madw(a.x, y.w, im[j]); im[j] = madw(a.y, y.z, im[j]);
							im[j] = madw(a.z, y.y, im[j]); im[j] = madw(a.w, y.x, im[j]);
						}
					}
				} else {
					const int2* ap = reinterpret_cast<const int2*>(a0) + lane;
#pragma unroll UN
					for (int k = 0; k < KC; ++k) {
						const int2 a = __ldg(ap + k * TM);
#pragma unroll
						for (int j = 0; j < NB; ++j) {
							const int4 y = x[k * XS + j];
							rh[j] = madw(a.x, y.x, rh[j]); ih[j] = madw(a.x, y.z, ih[j]);
							rm[j] = madw(a.x, y.y, rm[j]); rm[j] = madw(a.y, y.x, rm[j]);
							im[j] = madw(a.x, y.w, im[j]); im[j] = madw(a.y, y.z, im[j]);
						}
					}
				}
			} else {
				const char* a0 = A + (c < td.y ? (long)(c - td.x) * TB : tf + (long)(c - td.z) * TB);
				if (CX) {
					const int2* ap = reinterpret_cast<const int2*>(a0) + lane;
#pragma unroll UN
					for (int k = 0; k < KC; ++k) {
						const int2 a = __ldg(ap + k * TM);
						const int nb = -a.y;
#pragma unroll
						for (int j = 0; j < NB; ++j) {
							const int4 y = x[k * XS + j];
							rm[j] = madw(a.x, y.x, rm[j]); rm[j] = madw(nb, y.z, rm[j]);
							im[j] = madw(a.x, y.z, im[j]); im[j] = madw(a.y, y.x, im[j]);
						}
					}
				} else {
					const int* ap = reinterpret_cast<const int*>(a0) + lane;
#pragma unroll UN
					for (int k = 0; k < KC; ++k) {
						const int a = __ldg(ap + k * TM);
#pragma unroll
						for (int j = 0; j < NB; ++j) {
							const int4 y = x[k * XS + j];
							rm[j] = madw(a, y.x, rm[j]); im[j] = madw(a, y.z, im[j]);
						}
					}
				}
			}
		}
		// at most 32 k since the last flush: 128 mixed products below 2^55
#pragma unroll
		for (int j = 0; j < NB; ++j) { flush(rh[j], rm[j]); flush(ih[j], im[j]); }
		__syncthreads();
	}
	const int row = tile * TM + lane;
	auto emit = [&](int cl, long long hr, long long mr, long long hi, long long mi) {
		const int c = col0 + cl;
		if (c >= p.ncols || (p.nta && !(p.step < p.nta[c]))) return;
		const int E = sE[cl], s = p.ea + E - 1078;
		const double2 y = make_double2(to_double(hr, mr, s, E == 0x7ff), to_double(hi, mi, s, E == 0x7ff));
		const long o = (long)(p.dmap ? p.dmap[c] : c) * p.nchan + ch;
		if (row < p.N) p.dst[o * p.N + row] = y;
		const int e = __reduce_max_sync(0xffffffffu, row < p.N ? max(bexp(y.x), bexp(y.y)) : 0);
		if (lane == 0) p.edst[o * p.ntile + tile] = e;
	};
	if constexpr (KS == 1) {
#pragma unroll
		for (int j = 0; j < NB; ++j) emit(wc + j, rh[j], rm[j], ih[j], im[j]);
	} else {
		long long* red = reinterpret_cast<long long*>(smem);
#pragma unroll
		for (int j = 0; j < NB; ++j) {
			long long* q = red + ((warp * NB + j) * 4) * 32 + lane;
			q[0] = rh[j]; q[32] = rm[j]; q[64] = ih[j]; q[96] = im[j];
		}
		__syncthreads();
		for (int cl = warp; cl < COLS; cl += 8) {
			long long a = 0, b = 0, c = 0, d = 0;
#pragma unroll
			for (int k = 0; k < KS; ++k) {
				const long long* q = red + ((((cl / NB) * KS + k) * NB + cl % NB) * 4) * 32 + lane;
				a += q[0]; b += q[32]; c += q[64]; d += q[96];
			}
			flush(a, b); flush(c, d);
			emit(cl, a, b, c, d);
		}
	}
}

// largest exponent of every TM-row tile of src [nvec][N]
__global__ void k_exponents(const double2* __restrict__ src, int* __restrict__ ex, int N, int ntile, long nvec)
{
	const long w = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
	const int lane = threadIdx.x & 31;
	if (w >= nvec * ntile) return;
	const long vec = w / ntile;
	const int row = (int)(w % ntile) * TM + lane;
	int e = 0;
	if (row < N) { const double2 v = src[vec * N + row]; e = max(bexp(v.x), bexp(v.y)); }
	e = __reduce_max_sync(0xffffffffu, e);
	if (lane == 0) ex[w] = e;
}

// ------------------------------------------------------------------ the local part of a step
// One block: TM positions of one (slot, m), all l; lane = position.  y -> E_k, O_k (the even-l and odd-l
// halves of the transform by the eigenvectors of Y10; +-lambda share them), phases, and back:
//   z+- = E +- O, z+' = phi z+, z-' = conj(phi) z-, s = z+' + z-' = 2 (c E + i s O), d = z+' - z-' = 2 (i s E + c O)
// with phi = c + i s.  Both transforms in fixed point under each position's largest exponent, the phases in FP64
// (28 instructions per pair and position: the kernel's largest single share).  The dipole of f(r) = r is
// sum_k lambda_k r_j (|z+|^2 - |z-|^2) = sum_k 4 lambda_k r_j Re(conj(E_k) O_k).
struct angle_args {
	double2* y;		// [slot][M][L][N], in place
	int* ex;		// [slot][M][L][ntile]
	const int2* V;		// [M][npair+1][L] limbs, |V| <= 1
	const double* lamp;	// [M][npair]
	const double* r;	// [N]
	const double* ftab;
	long ld;
	const int64_t *ntf, *ntt;
	long step;
	int cmode;
	double dt4;		// dt / 4
	int N, ntile, L, M, npair;
	double* zpart;		// [slot][M][ntile] of this step, or NULL
};

__device__ __forceinline__ int power_of(long s, long nt, int cmode)
{
	if (nt <= 0) return 0;
	if (cmode == 1) return (s >= 1 && s <= nt) ? 1 : 0;
	if (cmode == 2) return s < nt ? 1 : 0;
	if (s > nt) return 0;
	return (s == 0 || s == nt) ? 1 : 2;
}

// outputs o0 .. o0+G-1 of a real matrix (element (o, k) at V[o * so + k * sk]) times the column in x[k * xk + lane]
template <int G>
__device__ __forceinline__ void local_product(const int2* __restrict__ V, int so, int sk, int nk, int no, const int4* __restrict__ x, int xk,
	long long (&h)[G][2], long long (&m)[G][2])
{
#pragma unroll
	for (int g = 0; g < G; ++g) h[g][0] = h[g][1] = m[g][0] = m[g][1] = 0;
#pragma unroll 4
	for (int k = 0; k < nk; ++k) {
		const int4 y = x[k * xk];
#pragma unroll
		for (int g = 0; g < G; ++g) {
			const int2 a = __ldg(V + (g < no ? g : 0) * so + k * sk);
			h[g][0] = madw(a.x, y.x, h[g][0]); h[g][1] = madw(a.x, y.z, h[g][1]);
			m[g][0] = madw(a.x, y.y, m[g][0]); m[g][0] = madw(a.y, y.x, m[g][0]);
			m[g][1] = madw(a.x, y.w, m[g][1]); m[g][1] = madw(a.y, y.z, m[g][1]);
		}
	}
#pragma unroll
	for (int g = 0; g < G; ++g) { flush(h[g][0], m[g][0]); flush(h[g][1], m[g][1]); }
}

template <int G>
__global__ void __launch_bounds__(256) k_angle(const angle_args p)
{
	extern __shared__ double2 sm[];
	__shared__ int pe[8][32];
	__shared__ double zs[8][32];
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const int tile = blockIdx.x % p.ntile;
	const int im = blockIdx.x / p.ntile;	// slot * M + m
	const int m = im % p.M, slot = im / p.M;
	const int pw = power_of(p.step, p.ntf[slot], p.cmode);
	const bool obs = p.zpart && p.step < p.ntt[slot];
	if (pw == 0 && !obs) return;
	const int L = p.L, np = p.npair, N = p.N;
	double2* a = sm;		// [L][32]: y, then its limbs, then the eigen-channels' limbs
	double2* b = sm + L * 32;	// [L][32]: E_k at 2k, O_k at 2k + 1, the zero channel at 2 npair
	const int row = tile * TM + lane;
	const bool in = row < N;
	double2* y = p.y + (long)im * L * N + row;
	int e = 0;
	for (int l = warp; l < L; l += 8) {
		const double2 v = in ? y[(long)l * N] : make_double2(0.0, 0.0);
		a[l * 32 + lane] = v;
		e = max(e, max(bexp(v.x), bexp(v.y)));
	}
	pe[warp][lane] = e;
	__syncthreads();
	e = 0;
#pragma unroll
	for (int w = 0; w < 8; ++w) e = max(e, pe[w][lane]);
	for (int l = warp; l < L; l += 8) {
		const double2 v = a[l * 32 + lane];
		const int2 q0 = quant(v.x, e), q1 = quant(v.y, e);
		reinterpret_cast<int4*>(a)[l * 32 + lane] = make_int4(q0.x, q0.y, q1.x, q1.y);
	}
	__syncthreads();
	const int4* qa = reinterpret_cast<const int4*>(a) + lane;
	const int2* V = p.V + (long)m * (np + 1) * L;
	const int nE = np + (L & 1), gE = (nE + G - 1) / G, gO = (np + G - 1) / G;
	long long h[G][2], mm[G][2];
	for (int t = warp; t < gE + gO; t += 8) {
		const bool odd = t >= gE;
		const int k0 = (odd ? t - gE : t) * G, no = min(G, (odd ? np : nE) - k0);
		local_product<G>(V + k0 * L + (odd ? 1 : 0), L, 2, odd ? L / 2 : (L + 1) / 2, no, qa + (odd ? 32 : 0), 64, h, mm);
#pragma unroll
		for (int g = 0; g < G; ++g)
			if (g < no) {
				const int s = e - 1078;
				b[(2 * (k0 + g) + (odd ? 1 : 0)) * 32 + lane] =
					make_double2(to_double(h[g][0], mm[g][0], s, e == 0x7ff), to_double(h[g][1], mm[g][1], s, e == 0x7ff));
			}
	}
	__syncthreads();
	const double rj = in ? p.r[row] : 0.0;
	const double f = pw ? p.ftab[(long)slot * p.ld + p.step] * p.dt4 : 0.0;
	double z = 0.0;
	e = 0;
	for (int k = warp; k < np; k += 8) {
		const double2 E = b[(2 * k) * 32 + lane], O = b[(2 * k + 1) * 32 + lane];
		const double lam = p.lamp[m * np + k];
		if (obs) z = fma(lam, fma(E.x, O.x, E.y * O.y), z);
		if (pw) {
			const double beta = lam * f * rj;
			const double inv = 1.0 / fma(beta, beta, 1.0);
			double c = fma(-beta, beta, 1.0) * inv, s = -2.0 * beta * inv;
			if (pw == 2) {
				const double c1 = c;
				c = fma(-2.0 * s, s, 1.0);
				s = 2.0 * s * c1;
			}
			c *= 2.0; s *= 2.0;
			const double2 S = make_double2(fma(c, E.x, -s * O.y), fma(c, E.y, s * O.x));
			const double2 D = make_double2(fma(c, O.x, -s * E.y), fma(c, O.y, s * E.x));
			e = max(max(e, max(bexp(S.x), bexp(S.y))), max(bexp(D.x), bexp(D.y)));
			b[(2 * k) * 32 + lane] = S;
			b[(2 * k + 1) * 32 + lane] = D;
		}
	}
	if (obs) {
		zs[warp][lane] = 4.0 * z * rj;
		__syncthreads();
		if (warp == 0) {
			double t = 0.0;
#pragma unroll
			for (int w = 0; w < 8; ++w) t += zs[w][lane];
#pragma unroll
			for (int o = 16; o; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
			if (lane == 0) p.zpart[(long)im * p.ntile + tile] = t;
		}
	}
	if (pw == 0) return;
	if ((L & 1) && warp == 7) { const double2 Z = b[2 * np * 32 + lane]; e = max(e, max(bexp(Z.x), bexp(Z.y))); }
	pe[warp][lane] = e;
	__syncthreads();
	e = 0;
#pragma unroll
	for (int w = 0; w < 8; ++w) e = max(e, pe[w][lane]);
	for (int k = warp; k < L; k += 8) {
		const double2 v = b[k * 32 + lane];
		const int2 q0 = quant(v.x, e), q1 = quant(v.y, e);
		reinterpret_cast<int4*>(a)[k * 32 + lane] = make_int4(q0.x, q0.y, q1.x, q1.y);
	}
	__syncthreads();
	const int nl0 = (L + 1) / 2, nl1 = L / 2, g0 = (nl0 + G - 1) / G, g1 = (nl1 + G - 1) / G;
	for (int t = warp; t < g0 + g1; t += 8) {
		const int odd = t >= g0 ? 1 : 0;
		const int o0 = (odd ? t - g0 : t) * G, no = min(G, (odd ? nl1 : nl0) - o0);
		// even l: s_k (slots 2k) and, for odd n_l, the zero channel (slot 2 npair); odd l: d_k (slots 2k + 1)
		local_product<G>(V + 2 * o0 + odd, 2, L, odd ? np : nE, no, qa + odd * 32, 64, h, mm);
#pragma unroll
		for (int g = 0; g < G; ++g)
			if (g < no) {
				const int s = e - 1078, l = 2 * (o0 + g) + odd;
				const double2 v = make_double2(to_double(h[g][0], mm[g][0], s, e == 0x7ff), to_double(h[g][1], mm[g][1], s, e == 0x7ff));
				if (in) y[(long)l * N] = v;
				const int x = __reduce_max_sync(0xffffffffu, in ? max(bexp(v.x), bexp(v.y)) : 0);
				if (lane == 0) p.ex[((long)im * L + l) * p.ntile + tile] = x;
			}
	}
}

// z[slot][s] of `cnt` steps from s0: the tiles' parts in a fixed order
__global__ void k_dipole_sum(const double* __restrict__ zpart, double* __restrict__ z, long ldz, const int64_t* __restrict__ ntt, int B, int per,
	long s0, int cnt)
{
	const int t = blockIdx.x * blockDim.x + threadIdx.x;
	if (t >= B * cnt) return;
	const int slot = t % B;
	const long s = s0 + t / B;
	if (s >= ntt[slot]) return;
	const double* q = zpart + ((long)(t / B) * B + slot) * per;
	double v = 0.0;
	for (int i = 0; i < per; ++i) v += q[i];
	z[slot * ldz + s] = v;
}

// ------------------------------------------------------------------ set-up: the eigenvectors of (R, S)
// Starting vector i: inverse iteration on the pencil restricted to the 2 SEEDW + 1 rows around i (the
// eigenvectors are localised), one warp each.  The eigenvalue is isolated by its index with Sturm counts of
// the banded LDL^T, 32 shifts at a time.
template <int P>
__device__ __forceinline__ int sturm(const double* __restrict__ R, const double* __restrict__ S, int lo, int m, double sig, double* __restrict__ Lout,
	double* __restrict__ dout)
{
	constexpr int NE = P + 1;
	double Lp[P][P], di[P];		// rows r-1-q: L(r-1-q, r-1-q-1-j), 1/d
#pragma unroll
	for (int q = 0; q < P; ++q) {
		di[q] = 0.0;
#pragma unroll
		for (int j = 0; j < P; ++j) Lp[q][j] = 0.0;
	}
	int neg = 0;
	for (int r = 0; r < m; ++r) {
		double u[P], l[P];
#pragma unroll
		for (int k = P; k >= 1; --k) {	// u_k = L(r, r-k) d(r-k)
			const long o = (long)(lo + r - k) * NE + k;
			double a = r >= k ? fma(-sig, __ldg(S + o), __ldg(R + o)) : 0.0;
#pragma unroll
			for (int j = P; j > k; --j) a = fma(-u[j - 1], Lp[k - 1][j - k - 1], a);
			u[k - 1] = a;
		}
		double d = fma(-sig, __ldg(S + (long)(lo + r) * NE), __ldg(R + (long)(lo + r) * NE));
		const double sc = fabs(d);
#pragma unroll
		for (int k = 1; k <= P; ++k) {
			l[k - 1] = u[k - 1] * di[k - 1];
			d = fma(-u[k - 1], l[k - 1], d);
		}
		if (fabs(d) < 1e-14 * sc) d = 1e-14 * sc;
		if (!(d != 0.0)) d = 1e-300;
		neg += d < 0.0;
		const double dv = 1.0 / d;
		if (Lout) {
#pragma unroll
			for (int k = 0; k < P; ++k) Lout[r * P + k] = l[k];
			dout[r] = dv;
		}
#pragma unroll
		for (int q = P - 1; q > 0; --q) {
			di[q] = di[q - 1];
#pragma unroll
			for (int j = 0; j < P; ++j) Lp[q][j] = Lp[q - 1][j];
		}
		di[0] = dv;
#pragma unroll
		for (int j = 0; j < P; ++j) Lp[0][j] = l[j];
	}
	return neg;
}

template <int P>
__global__ void __launch_bounds__(32) k_seed(const double* __restrict__ R, const double* __restrict__ S, int N, double* __restrict__ Xt)
{
	constexpr int NE = P + 1, MW = 2 * SEEDW + 1;
	__shared__ double sL[MW * P], sd[MW], x[MW], y[MW];
	const int i = blockIdx.x, lane = threadIdx.x;
	int m = min(MW, N), lo = min(max(i - SEEDW, 0), N - m);
	const int t = i - lo;
	const double mu = R[(long)i * NE] / S[(long)i * NE];
	const int j = i + 1 < N ? i + 1 : i - 1;
	double w = 8.0 * fabs(R[(long)j * NE] / S[(long)j * NE] - mu);
	if (!(w > 0.0) || !isfinite(w)) return;		// the caller sees a vector of zeros
	double a = mu - w, b = mu + w;
	for (int it = 0; it < 24; ++it) {		// count(a) <= t < count(b)
		const int c = sturm<P>(R, S, lo, m, (lane & 1) ? b : a, nullptr, nullptr);
		const int ca = __shfl_sync(0xffffffffu, c, 0), cb = __shfl_sync(0xffffffffu, c, 1);
		if (ca <= t && cb > t) break;
		w *= 2.0;
		if (ca > t) a -= w;
		if (cb <= t) b += w;
	}
	for (int it = 0; it < 3; ++it) {
		const double s = a + (b - a) * (lane + 1) / 33.0;
		const int c = sturm<P>(R, S, lo, m, s, nullptr, nullptr);
		const unsigned below = __ballot_sync(0xffffffffu, c <= t);
		const int n = __popc(below);	// counts ascend with the shift: the first n shifts are below the eigenvalue
		const double na = n ? a + (b - a) * n / 33.0 : a, nb = n < 32 ? a + (b - a) * (n + 1) / 33.0 : b;
		a = na; b = nb;
	}
	// shift just below the eigenvalue: leading blocks beyond row t have no eigenvalue near it
	if (lane == 0) sturm<P>(R, S, lo, m, a, sL, sd);
	for (int r = lane; r < m; r += 32) x[r] = r == t ? 1.0 : 0.0;
	__syncwarp();
	for (int it = 0; it < 4; ++it) {
		for (int r = lane; r < m; r += 32) {	// y = S x
			double v = S[(long)(lo + r) * NE] * x[r];
			for (int k = 1; k <= P; ++k) {
				if (r - k >= 0) v = fma(S[(long)(lo + r - k) * NE + k], x[r - k], v);
				if (r + k < m) v = fma(S[(long)(lo + r) * NE + k], x[r + k], v);
			}
			y[r] = v;
		}
		__syncwarp();
		double part = 0.0;
		for (int r = lane; r < m; r += 32) part = fma(x[r], y[r], part);
		for (int o = 16; o; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
		if (it == 3) {
			const double sc = rsqrt(part);
			for (int r = lane; r < m; r += 32) Xt[(long)i * N + lo + r] = x[r] * sc;
			return;
		}
		if (lane == 0) {
			for (int r = 0; r < m; ++r)
				for (int k = 1; k <= P && k <= r; ++k) y[r] = fma(-sL[r * P + k - 1], y[r - k], y[r]);
			for (int r = 0; r < m; ++r) y[r] *= sd[r];
			for (int r = m - 1; r >= 0; --r)
				for (int k = 1; k <= P && r + k < m; ++k) y[r] = fma(-sL[(r + k) * P + k - 1], y[r + k], y[r]);
		}
		__syncwarp();
		double big = 0.0;
		for (int r = lane; r < m; r += 32) big = fmax(big, fabs(y[r]));
		for (int o = 16; o; o >>= 1) big = fmax(big, __shfl_xor_sync(0xffffffffu, big, o));
		for (int r = lane; r < m; r += 32) x[r] = y[r] / big;
		__syncwarp();
	}
}

// Yt[i] = S x_i, Zt[i] = R x_i
__global__ void k_band_vec(const double* __restrict__ S, const double* __restrict__ R, int N, int P, const double* __restrict__ Xt, double* __restrict__ Yt,
	double* __restrict__ Zt)
{
	const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
	if (t >= (long)N * N) return;
	const int r = (int)(t % N), NE = P + 1;
	const double* x = Xt + t;
	double y = S[(long)r * NE] * x[0], z = R ? R[(long)r * NE] * x[0] : 0.0;
	for (int k = 1; k <= P; ++k) {
		if (r - k >= 0) { y = fma(S[(long)(r - k) * NE + k], x[-k], y); if (R) z = fma(R[(long)(r - k) * NE + k], x[-k], z); }
		if (r + k < N) { y = fma(S[(long)r * NE + k], x[k], y); if (R) z = fma(R[(long)r * NE + k], x[k], z); }
	}
	Yt[t] = y;
	if (R) Zt[t] = z;
}

__global__ void k_ritz(const double* __restrict__ Xt, const double* __restrict__ Yt, const double* __restrict__ Zt, int N, double* __restrict__ lam)
{
	const int i = blockIdx.x, lane = threadIdx.x;
	double g = 0.0, t = 0.0;
	for (int r = lane; r < N; r += 32) { const double x = Xt[(long)i * N + r]; g = fma(x, Yt[(long)i * N + r], g); t = fma(x, Zt[(long)i * N + r], t); }
	for (int o = 16; o; o >>= 1) { g += __shfl_xor_sync(0xffffffffu, g, o); t += __shfl_xor_sync(0xffffffffu, t, o); }
	if (lane == 0) lam[i] = t / g;
}

// 32 x 32 tiles of A B^T (A, B [N][N] row-major, rows localised within WMAX + 32 of the diagonal) for tiles near
// the diagonal, in FP64.  mode 0: the correction E of Ogita and Aishima (Iterative refinement for symmetric
// eigenvalue decomposition, 2018) in the S metric, from G = X^T S X and T = X^T R X in one pass,
//   E_ij = (T_ij - lambda_j G_ij)/(lambda_j - lambda_i), E_ii = (1 - G_ii)/2,
// tiles on and above the diagonal only, stored as C[j][i] = E_ij, the largest magnitude in err; mode 1: C = A B^T.
__global__ void __launch_bounds__(256) k_outer(const double* __restrict__ A, const double* __restrict__ Bg, const double* __restrict__ Bt,
	const double* __restrict__ lam, int N, int nt, int wt, int mode, double* __restrict__ C, unsigned long long* __restrict__ err)
{
	const int ti = blockIdx.x, tj = ti + (int)blockIdx.y - wt;
	if (tj < 0 || tj >= nt || (mode == 0 && tj < ti)) return;
	__shared__ double sa[32][33], sg[32][33], st[32][33];
	const int x = threadIdx.x & 31, y0 = threadIdx.x >> 5;
	double g[4] = {0, 0, 0, 0}, t[4] = {0, 0, 0, 0};
	const int k0 = max(0, max(ti, tj) - wt) * 32, k1 = min(N, (min(ti, tj) + wt + 1) * 32);
	for (int k = k0; k < k1; k += 32) {
		for (int q = y0; q < 32; q += 8) {
			const int i = ti * 32 + q, j = tj * 32 + q;
			const bool kin = k + x < N;
			sa[q][x] = (i < N && kin) ? A[(long)i * N + k + x] : 0.0;
			sg[q][x] = (j < N && kin) ? Bg[(long)j * N + k + x] : 0.0;
			if (mode == 0) st[q][x] = (j < N && kin) ? Bt[(long)j * N + k + x] : 0.0;
		}
		__syncthreads();
#pragma unroll 8
		for (int q = 0; q < 32; ++q) {
			const double bg = sg[x][q], bt = mode == 0 ? st[x][q] : 0.0;
#pragma unroll
			for (int u = 0; u < 4; ++u) {
				const double a = sa[y0 + 8 * u][q];
				g[u] = fma(a, bg, g[u]);
				if (mode == 0) t[u] = fma(a, bt, t[u]);
			}
		}
		__syncthreads();
	}
	if (mode) {
		const int j = tj * 32 + x;
#pragma unroll
		for (int u = 0; u < 4; ++u) {
			const int i = ti * 32 + y0 + 8 * u;
			if (i < N && j < N) C[(long)i * N + j] = g[u];
		}
		return;
	}
#pragma unroll
	for (int u = 0; u < 4; ++u) { sg[y0 + 8 * u][x] = g[u]; st[y0 + 8 * u][x] = t[u]; }
	__syncthreads();
	double big = 0.0;
	for (int q = y0; q < 32; q += 8) {
		// E_ij and E_ji of one pair i < j from the same G_ij, T_ij: E + E^T = 1 - G to the last digit
		const int i = ti * 32 + q, j = tj * 32 + x;
		if (i >= N || j >= N || i > j) continue;
		const double G = sg[q][x], T = st[q][x];
		double eij, eji;
		if (i == j) eij = eji = 0.5 * (1.0 - G);
		else {
			const double a = (T - 0.5 * (lam[i] + lam[j]) * G) / (lam[j] - lam[i]);
			eij = a - 0.5 * G;
			eji = -a - 0.5 * G;
		}
		C[(long)j * N + i] = eij;
		C[(long)i * N + j] = eji;
		big = fmax(big, isfinite(eij) ? fmax(fabs(eij), fabs(eji)) : 1e300);
	}
	for (int o = 16; o; o >>= 1) big = fmax(big, __shfl_xor_sync(0xffffffffu, big, o));
	if (x == 0) atomicMax(err, (unsigned long long)__double_as_longlong(big));
}

// Xn[i][r] = Xt[i][r] + sum_j E[j][i] Xt[j][r], with Et[i][j] = E_ji
__global__ void __launch_bounds__(256) k_update(const double* __restrict__ Et, const double* __restrict__ Xt, int N, int nt, int wt, double* __restrict__ Xn)
{
	const int ti = blockIdx.x, tr = ti + (int)blockIdx.y - wt;
	if (tr < 0 || tr >= nt) return;
	__shared__ double se[32][33], sx[32][33];
	const int x = threadIdx.x & 31, y0 = threadIdx.x >> 5;
	double g[4] = {0, 0, 0, 0};
	const int k0 = max(0, max(ti, tr) - wt) * 32, k1 = min(N, (min(ti, tr) + wt + 1) * 32);
	for (int k = k0; k < k1; k += 32) {
		for (int q = y0; q < 32; q += 8) {
			const int i = ti * 32 + q, r = tr * 32 + x;
			se[q][x] = (i < N && k + x < N) ? Et[(long)i * N + k + x] : 0.0;
			sx[q][x] = (k + q < N && r < N) ? Xt[(long)(k + q) * N + r] : 0.0;
		}
		__syncthreads();
#pragma unroll 8
		for (int q = 0; q < 32; ++q) {
			const double b = sx[q][x];
#pragma unroll
			for (int u = 0; u < 4; ++u) g[u] = fma(se[y0 + 8 * u][q], b, g[u]);
		}
		__syncthreads();
	}
	const int r = tr * 32 + x;
#pragma unroll
	for (int u = 0; u < 4; ++u) {
		const int i = ti * 32 + y0 + 8 * u;
		if (i < N && r < N) Xn[(long)i * N + r] = Xt[(long)i * N + r] + g[u];
	}
}

// ------------------------------------------------------------------ set-up: the stored operators

// largest |A_ij| per distance |i - j| <= WMAX (as ordered bits); A(i, j) = A[i * si + j * sj]
__global__ void k_profile(const double* __restrict__ A, long si, long sj, int N, unsigned long long* __restrict__ prof)
{
	const int d = blockIdx.x;
	double big = 0.0;
	for (int i = threadIdx.x; i + d < N; i += blockDim.x) {
		const double a = fabs(A[i * si + (i + d) * sj]), b = fabs(A[(i + d) * si + i * sj]);
		big = fmax(big, isfinite(a) && isfinite(b) ? fmax(a, b) : 1e300);
	}
	for (int o = 16; o; o >>= 1) big = fmax(big, __shfl_xor_sync(0xffffffffu, big, o));
	if ((threadIdx.x & 31) == 0) atomicMax(prof + d, (unsigned long long)__double_as_longlong(big));
}

// columns j0 .. j0+J of F~ (G[jj][l][i]) into the band Fb[l][i][2 WMAX + 1], with the profile
__global__ void k_gather_band(const double2* __restrict__ G, int j0, int J, int N, int nlh, double2* __restrict__ Fb, unsigned long long* __restrict__ prof)
{
	__shared__ unsigned long long sp[WMAX + 1];
	for (int t = threadIdx.x; t <= WMAX; t += blockDim.x) sp[t] = 0;
	__syncthreads();
	const int jj = blockIdx.x, l = blockIdx.y, j = j0 + jj;
	for (int d = (int)threadIdx.x - WMAX; d <= WMAX; d += blockDim.x) {
		const int i = j + d;
		if (i < 0 || i >= N) continue;
		const double2 v = G[((long)jj * nlh + l) * N + i];
		Fb[((long)l * N + i) * (2 * WMAX + 1) + (j - i + WMAX)] = v;
		double b = fmax(fabs(v.x), fabs(v.y));
		if (!isfinite(v.x) || !isfinite(v.y)) b = 1e300;
		atomicMax(sp + abs(d), (unsigned long long)__double_as_longlong(b));
	}
	__syncthreads();
	for (int t = threadIdx.x; t <= WMAX; t += blockDim.x) if (sp[t]) atomicMax(prof + t, sp[t]);
}

__device__ __forceinline__ int2 fixed(double v, double scale)
{
	const long long x = __double2ll_rn(v * scale);
	const int hi = (int)((x + (1ll << 27)) >> 28);
	return make_int2(hi, (int)(x - ((long long)hi << 28)));
}

// one operator per blockIdx.y, one tile per blockIdx.x: the chunks of the tile as limbs.  CX: Fb band as above;
// else A(i, j) = A[i * si + j * sj].  scale = 2^(56 - ea).
template <bool CX>
__global__ void k_store(const double2* __restrict__ Fb, const double* __restrict__ A, long si, long sj, int N, int w, double scale, const int4* __restrict__ td,
	const long* __restrict__ toff, char* __restrict__ out, long astride)
{
	constexpr int FB = KC * TM * (CX ? 16 : 8), TB = FB / 2;
	const int tile = blockIdx.x, l = blockIdx.y;
	const int4 t = td[tile];
	char* o = out + l * astride + toff[tile];
	for (int e = threadIdx.x; e < (t.w - t.x) * KC * TM; e += blockDim.x) {
		const int c = t.x + e / (KC * TM), k = (e / TM) % KC, row = e % TM;
		const int i = tile * TM + row, j = c * KC + k;
		double2 v = make_double2(0.0, 0.0);
		if (i < N && j < N && abs(i - j) <= w) {
			if (CX) v = Fb[((long)l * N + i) * (2 * WMAX + 1) + (j - i + WMAX)];
			else v.x = A[i * si + j * sj];
		}
		const int2 a = fixed(v.x, scale), b = fixed(v.y, scale);
		const bool full = c >= t.y && c < t.z;
		char* q = o + (c < t.y ? (long)(c - t.x) * TB : (long)(t.y - t.x) * TB + (full ? (long)(c - t.y) * FB : (long)(t.z - t.y) * FB + (long)(c - t.z) * TB));
		const int at = k * TM + row;
		if (CX) {
			if (full) reinterpret_cast<int4*>(q)[at] = make_int4(a.x, a.y, b.x, b.y);
			else reinterpret_cast<int2*>(q)[at] = make_int2(a.y, b.y);
		} else {
			if (full) reinterpret_cast<int2*>(q)[at] = a;
			else reinterpret_cast<int*>(q)[at] = a.y;
		}
	}
}

// X[jj][r][l] = (x_{j0 + jj})_r for every l
__global__ void k_columns(const double* __restrict__ Xt, int j0, int N, int nlh, long total, double2* __restrict__ X)
{
	const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
	if (t >= total) return;
	X[t] = make_double2(Xt[(long)j0 * N + t / nlh], 0.0);
}

// [vec][r][l] -> [vec][l][r]
__global__ void __launch_bounds__(256) k_transpose(const double2* __restrict__ src, double2* __restrict__ dst, int N, int L)
{
	__shared__ double2 s[32][33];
	const int x = threadIdx.x & 31, y0 = threadIdx.x >> 5;
	const long base = (long)blockIdx.z * N * L;
	const int r0 = blockIdx.x * 32, l0 = blockIdx.y * 32;
	for (int q = y0; q < 32; q += 8)
		if (r0 + q < N && l0 + x < L) s[q][x] = src[base + (long)(r0 + q) * L + l0 + x];
	__syncthreads();
	for (int q = y0; q < 32; q += 8)
		if (l0 + q < L && r0 + x < N) dst[base + (long)(l0 + q) * N + r0 + x] = s[x][q];
}

} // namespace

// ------------------------------------------------------------------ host side

struct band_store {
	int w = 0, ea = 0;
	long stride = 0;		// bytes of one operator
	std::vector<int4> td;
	std::vector<long> off;
	int4* d_td = nullptr;
	long* d_off = nullptr;
	char* A = nullptr;
	size_t cap = 0;
	void release() { cudaFree(d_td); cudaFree(d_off); cudaFree(A); d_td = nullptr; d_off = nullptr; A = nullptr; }
};

struct pos_path {
	int dev = 0, N = 0, P = 0, L = 0, M = 0, m0 = 0, B = 0, nlh = 0, npair = 0, nff = 1, ntile = 0;
	double dt = 0.0;
	double *Xt = nullptr, *r = nullptr, *scratch = nullptr;	// eigenvectors [i][r], positions, [N][N] for the mask
	const double *S = nullptr;
	band_store F, W, X, K;		// F~_l, X^T S, X, the mask
	double2* buf[2] = {nullptr, nullptr};
	int* ex[2] = {nullptr, nullptr};
	int* exin = nullptr;
	int2* V = nullptr;
	double* lamp = nullptr;
	int *lmap = nullptr, *zero = nullptr;	// channel -> l, channel -> 0
	double* zpart = nullptr;
	static constexpr int ZB = 32;		// steps between two sums of the dipole's parts
	long zfirst = 0;
	int zcount = 0;
	unsigned long long* prof = nullptr;
	int angle_g = 3;
	size_t angle_smem = 0;
	std::vector<int> perm;
};

namespace {

// tiles of an operator whose entries at distance d are below 2^-57 for d > w and have no hi limb for d > wf
void lay_out(band_store& b, int N, int w, int wf, bool cx)
{
	const int nt = (N + TM - 1) / TM, nc = (N + KC - 1) / KC;
	const long FB = KC * TM * (cx ? 16 : 8), TB = FB / 2;
	b.w = w;
	b.td.resize(nt);
	b.off.resize(nt);
	long o = 0;
	for (int t = 0; t < nt; ++t) {
		auto first = [&](int d) { return std::max(0, t * TM - d) / KC; };
		auto last = [&](int d) { return std::min(nc, (std::min(N, t * TM + TM) - 1 + d) / KC + 1); };
		const int4 q = make_int4(first(w), first(std::min(w, wf)), last(std::min(w, wf)), last(w));
		b.td[t] = q;
		b.off[t] = o;
		o += (long)(q.z - q.y) * FB + (long)(q.y - q.x + q.w - q.z) * TB;
	}
	b.stride = o;
}

int upload(band_store& b, size_t bytes)
{
	const size_t nt = b.td.size();
	int rc;
	if (!b.d_td) if ((rc = dalloc(&b.d_td, nt)) || (rc = dalloc(&b.d_off, nt))) return rc;
	if (b.cap < bytes) {
		cudaFree(b.A); b.A = nullptr; b.cap = 0;
		if ((rc = dalloc(&b.A, bytes))) return rc;
		b.cap = bytes;
	}
	QPC_CUDA(cudaMemcpy(b.d_td, b.td.data(), sizeof(int4) * nt, cudaMemcpyHostToDevice));
	QPC_CUDA(cudaMemcpy(b.d_off, b.off.data(), sizeof(long) * nt, cudaMemcpyHostToDevice));
	return QPC_OK;
}

// Band of an operator from its profile: the distance where it has fallen to 2^-44 of its largest entry (well
// above the FP64 noise of its construction, ~2^-52), continued at the rate of the last 14 binary orders to 2^-57.
// false: it does not fall off within WMAX.
bool decay(const std::vector<unsigned long long>& prof, int N, double big, int& w, int& wf, int bits_hi)
{
	auto beyond = [&](double th) {	// smallest d with every entry at a larger distance below th
		int d = std::min(WMAX, N - 1);
		while (d >= 0) {
			double v;
			std::memcpy(&v, &prof[d], 8);
			if (!(v < th)) break;
			--d;
		}
		return d;
	};
	const int d30 = beyond(std::ldexp(big, -30)), d44 = beyond(std::ldexp(big, -44));
	wf = std::max(0, beyond(std::ldexp(big, -bits_hi)));
	if (N - 1 <= 64) { w = N - 1; return true; }
	if (d44 >= WMAX) return false;
	w = std::min(N - 1, d44 + ((d44 - d30) * 13 + 13) / 14 + 2);
	return w <= WMAX || N - 1 <= WMAX;
}

int read_profile(pos_path* p, cudaStream_t st, std::vector<unsigned long long>& prof)
{
	prof.resize(WMAX + 1);
	return copy_to_host(prof.data(), p->prof, sizeof(unsigned long long) * (WMAX + 1), st);
}

// quantised stage (or the reduction over the KS warps of a column) and the raw stage
template <int NB, int KS>
constexpr size_t band_smem()
{
	const size_t x = sizeof(int4) * 32 * KS * ((NB * 8 / KS) | 1), r = KS > 1 ? sizeof(long long) * 8 * NB * 4 * 32 : 0;
	return (x > r ? x : r) + sizeof(double2) * 256 * NB;
}

template <int NB, int KS, bool CX>
void band_launch(const band_args& a, int tiles, cudaStream_t st)
{
	constexpr int COLS = NB * 8 / KS;
	constexpr size_t smem = band_smem<NB, KS>();
	const int ncg = (a.ncols + COLS - 1) / COLS;
	k_band_apply<NB, KS, CX><<<dim3((unsigned)(tiles * ncg), (unsigned)a.nchan), 256, smem, st>>>(a);
}

template <int NB, int KS>
void band_attr()
{
	constexpr int smem = (int)band_smem<NB, KS>();
	cudaFuncSetAttribute(k_band_apply<NB, KS, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
	cudaFuncSetAttribute(k_band_apply<NB, KS, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
}

// columns per block by their number: 64 (8 per warp) keeps the operator's traffic lowest, fewer columns share
// their k range between warps so that a block still has eight
template <bool CX>
void band_apply(const band_args& a, int tiles, cudaStream_t st)
{
	const int n = a.ncols;
	if (a.amap || n == 1) band_launch<1, 8, CX>(a, tiles, st);
	else if (n == 2) band_launch<2, 8, CX>(a, tiles, st);
	else if (n <= 4) band_launch<4, 8, CX>(a, tiles, st);
	else if (n <= 8) band_launch<4, 4, CX>(a, tiles, st);
	else if (n <= 16) band_launch<4, 2, CX>(a, tiles, st);
	else if (n <= 32 || (n > 64 && n <= 96)) band_launch<4, 1, CX>(a, tiles, st);
	else band_launch<8, 1, CX>(a, tiles, st);
}

band_args args_of(const pos_path* p, const band_store& b, int nchan, int ncols)
{
	band_args a{};
	a.A = b.A; a.astride = b.stride; a.td = b.d_td; a.toff = b.d_off; a.ea = b.ea;
	a.N = p->N; a.ntile = p->ntile; a.nchan = nchan; a.ncols = ncols;
	a.lmap = p->zero;
	return a;
}

template <int P>
void seed(const pos_setup& in, double* Xt) { k_seed<P><<<in.N, 32, 0, in.stream>>>(in.R, in.S, in.N, Xt); }

template <int G>
void angle_launch(const pos_path* p, const angle_args& a, int slots, cudaStream_t st)
{
	k_angle<G><<<(unsigned)((long)slots * p->M * p->ntile), 256, p->angle_smem, st>>>(a);
}

// device scratch of a set-up, given back at its end
struct scratch {
	cudaStream_t st;
	std::vector<void*> ptr;
	explicit scratch(cudaStream_t s) : st(s) {}
	~scratch() { for (void* q : ptr) cudaFreeAsync(q, st); }
	template <class T> int get(T** q, size_t n)
	{
		if (cudaMallocAsync((void**)q, sizeof(T) * std::max<size_t>(n, 1), st) != cudaSuccess) {
			cudaGetLastError();
			set_error("set-up scratch of %zu bytes", sizeof(T) * n);
			return QPC_ERR_NOMEM;
		}
		ptr.push_back(*q);
		return QPC_OK;
	}
};

// the eigenvectors Xt and positions r; ok = false when the refinement does not converge
int eigenvectors(pos_path* p, const pos_setup& in, scratch& tmp, double** Yt_out, bool* ok)
{
	const int N = p->N, nt = p->ntile, wt = std::min(nt - 1, (WMAX + 31) / 32 + 1);
	const size_t nn = (size_t)N * N;
	cudaStream_t st = in.stream;
	double *Xn, *Yt, *Zt, *Et;
	unsigned long long* err;
	int rc;
	if ((rc = tmp.get(&Xn, nn)) || (rc = tmp.get(&Yt, nn)) || (rc = tmp.get(&Zt, nn)) || (rc = tmp.get(&Et, nn)) || (rc = tmp.get(&err, 3))) return rc;
	QPC_CUDA(cudaMemsetAsync(p->Xt, 0, sizeof(double) * nn, st));
	QPC_CUDA(cudaMemsetAsync(Xn, 0, sizeof(double) * nn, st));
	QPC_CUDA(cudaMemsetAsync(Et, 0, sizeof(double) * nn, st));
	QPC_CUDA(cudaMemsetAsync(err, 0, sizeof(*err) * 3, st));
	switch (p->P) {
	case 3: seed<3>(in, p->Xt); break;
	case 4: seed<4>(in, p->Xt); break;
	case 5: seed<5>(in, p->Xt); break;
	case 6: seed<6>(in, p->Xt); break;
	case 7: seed<7>(in, p->Xt); break;
	default: seed<8>(in, p->Xt); break;
	}
	const unsigned nb = (unsigned)((nn + 255) / 256);
	for (int it = 0; it < 3; ++it) {
		k_band_vec<<<nb, 256, 0, st>>>(in.S, in.R, N, p->P, p->Xt, Yt, Zt);
		k_ritz<<<N, 32, 0, st>>>(p->Xt, Yt, Zt, N, p->r);
		k_outer<<<dim3(nt, 2 * wt + 1), 256, 0, st>>>(p->Xt, Yt, Zt, p->r, N, nt, wt, 0, Et, err + it);
		k_update<<<dim3(nt, 2 * wt + 1), 256, 0, st>>>(Et, p->Xt, N, nt, wt, Xn);
		QPC_CUDA(cudaMemcpyAsync(p->Xt, Xn, sizeof(double) * nn, cudaMemcpyDeviceToDevice, st));
	}
	k_band_vec<<<nb, 256, 0, st>>>(in.S, in.R, N, p->P, p->Xt, Yt, Zt);
	k_ritz<<<N, 32, 0, st>>>(p->Xt, Yt, Zt, N, p->r);
	QPC_CUDA(cudaGetLastError());
	double e[3];
	if ((rc = copy_to_host(e, err, sizeof(e), st))) return rc;
	// the corrections shrink quadratically: the third is at the rounding level when the first two converged
	*ok = e[0] < 0.05 && e[1] < 1e-3 && e[2] < 1e-8;
	*Yt_out = Yt;
	return QPC_OK;
}

int store_real(pos_path* p, band_store& b, const double* A, long si, long sj, cudaStream_t st, bool* ok)
{
	std::vector<unsigned long long> prof;
	QPC_CUDA(cudaMemsetAsync(p->prof, 0, sizeof(unsigned long long) * (WMAX + 1), st));
	k_profile<<<std::min(WMAX, p->N - 1) + 1, 128, 0, st>>>(A, si, sj, p->N, p->prof);
	if (int rc = read_profile(p, st, prof)) return rc;
	double big = 0.0;
	for (auto u : prof) { double v; std::memcpy(&v, &u, 8); big = std::max(big, v); }
	*ok = big > 0.0 && big < 1e200;
	if (!*ok) return QPC_OK;
	int w, wf;
	std::frexp(big, &b.ea);
	*ok = decay(prof, p->N, std::ldexp(1.0, b.ea), w, wf, 29);
	if (!*ok) return QPC_OK;
	lay_out(b, p->N, w, wf, false);
	if (int rc = upload(b, (size_t)b.stride)) return rc;
	k_store<false><<<dim3(p->ntile, 1), 256, 0, st>>>(nullptr, A, si, sj, p->N, w, std::ldexp(1.0, 56 - b.ea), b.d_td, b.d_off, b.A, b.stride);
	QPC_CUDA(cudaGetLastError());
	return QPC_OK;
}

int build(pos_path* p, const pos_setup& in, bool* ok)
{
	const int N = p->N, L = p->L, M = p->M, nlh = p->nlh;
	cudaStream_t st = in.stream;
	int rc;
	const long nvec = (long)p->B * M * L;
	std::vector<int> lm(std::max(M * L, nlh)), zr(std::max(M * L, nlh), 0);
	for (int c = 0; c < M * L; ++c) lm[c] = c % L + std::abs(p->m0 + c / L);
	std::vector<int2> V((size_t)M * (p->npair + 1) * L);
	for (size_t i = 0; i < V.size(); ++i) {
		const long long x = std::llrint(std::ldexp(in.Vh[i], 56));
		const int hi = (int)((x + (1ll << 27)) >> 28);
		V[i] = make_int2(hi, (int)(x - ((long long)hi << 28)));
	}
	if ((rc = dalloc(&p->Xt, (size_t)N * N)) || (rc = dalloc(&p->r, N)) || (rc = dalloc(&p->prof, WMAX + 1)) || (rc = dalloc(&p->lmap, lm.size())) ||
		(rc = dalloc(&p->zero, zr.size())) || (rc = dalloc(&p->V, V.size())) || (rc = dalloc(&p->lamp, (size_t)M * std::max(p->npair, 1))))
		return rc;
	QPC_CUDA(cudaMemcpy(p->lmap, lm.data(), sizeof(int) * lm.size(), cudaMemcpyHostToDevice));
	QPC_CUDA(cudaMemcpy(p->zero, zr.data(), sizeof(int) * zr.size(), cudaMemcpyHostToDevice));
	QPC_CUDA(cudaMemcpy(p->V, V.data(), sizeof(int2) * V.size(), cudaMemcpyHostToDevice));
	QPC_CUDA(cudaMemcpy(p->lamp, in.lamp, sizeof(double) * M * std::max(p->npair, 1), cudaMemcpyHostToDevice));
	scratch tmp(st);
	double* Yt = nullptr;
	if ((rc = eigenvectors(p, in, tmp, &Yt, ok)) || !*ok) return rc;
	if ((rc = store_real(p, p->W, Yt, N, 1, st, ok)) || !*ok) return rc;
	if ((rc = store_real(p, p->X, p->Xt, 1, N, st, ok)) || !*ok) return rc;
	// F~_l, a set of columns at a time: the engine's field-free solve on the eigenvectors, then X^T S
	const int J = (int)std::min<long>(N, std::max<long>(32, (64l << 20) / ((long)N * nlh * 16)));
	const size_t chunk = (size_t)J * N * nlh;
	double2 *c0, *c1, *Fb;
	int *ce, *cd;
	const size_t band = (size_t)nlh * N * (2 * WMAX + 1);
	if ((rc = tmp.get(&c0, chunk)) || (rc = tmp.get(&c1, chunk)) || (rc = tmp.get(&Fb, band)) || (rc = tmp.get(&ce, (size_t)J * nlh * p->ntile)) ||
		(rc = tmp.get(&cd, (size_t)J * nlh * p->ntile)))
		return rc;
	std::vector<unsigned long long> prof;
	for (int fi = 0; fi < p->nff; ++fi) {
		QPC_CUDA(cudaMemsetAsync(Fb, 0, sizeof(double2) * band, st));
		if (fi == 0) QPC_CUDA(cudaMemsetAsync(p->prof, 0, sizeof(unsigned long long) * (WMAX + 1), st));
		for (int j0 = 0; j0 < N; j0 += J) {
			const int n = std::min(J, N - j0);
			const long total = (long)n * N * nlh, vec = (long)n * nlh;
			k_columns<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(p->Xt, j0, N, nlh, total, c0);
			if ((rc = in.fieldfree(c0, c1, n, fi))) return rc;
			k_transpose<<<dim3((N + 31) / 32, (nlh + 31) / 32, n), 256, 0, st>>>(c0, c1, N, nlh);
			k_exponents<<<(unsigned)((vec * p->ntile * 32 + 255) / 256), 256, 0, st>>>(c1, ce, N, p->ntile, vec);
			band_args a = args_of(p, p->W, nlh, n);
			a.s0 = c1; a.e0 = ce; a.dst = c0; a.edst = cd;
			a.tile0 = std::max(0, (j0 - WMAX) / TM);
			band_apply<false>(a, std::min(p->ntile, (j0 + n + WMAX + TM - 1) / TM) - a.tile0, st);
			k_gather_band<<<dim3(n, nlh), 128, 0, st>>>(c0, j0, n, N, nlh, Fb, p->prof);
			QPC_CUDA(cudaGetLastError());
		}
		if (fi == 0) {
			if ((rc = read_profile(p, st, prof))) return rc;
			int w, wf;
			if (!(*ok = decay(prof, N, 1.0, w, wf, 29))) return QPC_OK;
			if (p->nff > 1) { w = std::min(std::min(WMAX, N - 1), w + 8); wf = std::min(w, wf + 12); }	// the other potentials' bands, checked below
			lay_out(p->F, N, w, wf, true);
			if (!(*ok = (size_t)p->F.stride * nlh * p->nff <= (size_t)16 << 30)) return QPC_OK;
			if ((rc = upload(p->F, (size_t)p->F.stride * nlh * p->nff))) return rc;
		}
		k_store<true><<<dim3(p->ntile, nlh), 256, 0, st>>>(Fb, nullptr, 0, 0, N, p->F.w, std::ldexp(1.0, 56), p->F.d_td, p->F.d_off,
			p->F.A + (size_t)fi * nlh * p->F.stride, p->F.stride);
	}
	if (p->nff > 1) {
		int w, wf;
		if ((rc = read_profile(p, st, prof))) return rc;
		if (!decay(prof, N, 1.0, w, wf, 29) || w > p->F.w || wf > p->F.w) { *ok = false; return QPC_OK; }
		// entries beyond the chunks with hi limbs must have none
		int reach = N;
		for (size_t t = 0; t < p->F.td.size(); ++t) {
			const int4 q = p->F.td[t];
			if (q.y > q.x) reach = std::min(reach, (int)t * TM - q.y * KC);
			if (q.w > q.z) reach = std::min(reach, q.z * KC - 1 - ((int)t * TM + TM - 1));
		}
		if (wf > reach) { *ok = false; return QPC_OK; }
	}
	p->F.ea = 0;
	for (int i = 0; i < 2; ++i)
		if ((rc = dalloc(&p->buf[i], (size_t)nvec * N)) || (rc = dalloc(&p->ex[i], (size_t)nvec * p->ntile))) return rc;
	if ((rc = dalloc(&p->exin, (size_t)nvec * p->ntile))) return rc;
	// outputs per task of k_angle: the fewest rounds of eight warps
	int best = 1 << 30;
	for (int g = 2; g <= 4; ++g) {
		const int ne = p->npair + (L & 1), tasks = (ne + g - 1) / g + (p->npair + g - 1) / g, cost = (tasks + 7) / 8 * (g * 6 + 4);
		if (cost < best) { best = cost; p->angle_g = g; }
	}
	p->angle_smem = sizeof(double2) * 2 * 32 * L;
	return wait_on(st);
}

// the dynamic shared memory the kernels may ask for, on the current device
void set_attrs()
{
	band_attr<1, 8>(); band_attr<2, 8>(); band_attr<4, 8>(); band_attr<4, 4>(); band_attr<4, 2>(); band_attr<4, 1>(); band_attr<8, 1>();
	const int smem = (int)(sizeof(double2) * 64 * LMAX);
	cudaFuncSetAttribute(k_angle<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
	cudaFuncSetAttribute(k_angle<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
	cudaFuncSetAttribute(k_angle<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
}

} // namespace

// The path is taken when: 3 <= p <= 8, 2 <= n_l <= LMAX, the eigenvectors of (R, S) are found (S positive definite,
// eigenvalues apart), and X, X^T S and F~_l fall off within WMAX of the diagonal (their number of bytes is
// bounded too).  Everything else keeps the banded solves.
int pos_create(const pos_setup& in, pos_path** out)
{
	*out = nullptr;
	if (in.L > LMAX || in.L < 2 || in.P < 3 || in.P > 8) return QPC_OK;
	auto* p = new (std::nothrow) pos_path();
	if (!p) { set_error("host allocation"); return QPC_ERR_NOMEM; }
	p->dev = in.dev; p->N = in.N; p->P = in.P; p->L = in.L; p->M = in.M; p->m0 = in.m0; p->B = in.B; p->nlh = in.nlh; p->npair = in.npair;
	p->nff = in.nff; p->dt = in.dt; p->S = in.S; p->ntile = (in.N + TM - 1) / TM;
	set_attrs();
	bool ok = false;
	const int rc = build(p, in, &ok);
	if (rc || !ok) {
		pos_destroy(p);
		return rc;
	}
	*out = p;
	return QPC_OK;
}

void pos_destroy(pos_path* p)
{
	if (!p) return;
	cudaFree(p->Xt); cudaFree(p->r); cudaFree(p->scratch); cudaFree(p->prof); cudaFree(p->lmap); cudaFree(p->zero); cudaFree(p->V); cudaFree(p->lamp);
	for (int i = 0; i < 2; ++i) { cudaFree(p->buf[i]); cudaFree(p->ex[i]); }
	cudaFree(p->exin); cudaFree(p->zpart);
	p->F.release(); p->W.release(); p->X.release(); p->K.release();
	delete p;
}

#define POS_PROF(kind) struct prof_ { const pos_run& r; int k; prof_(const pos_run& r_, int k_) : r(r_), k(k_) { if (r.prof_begin) r.prof_begin(k, r.stream); } \
	~prof_() { if (r.prof_end) r.prof_end(k, r.stream); } } prof_scope_(r, kind)

int pos_begin(pos_path* p, const pos_run& r)
{
	const int nchan = p->M * p->L;
	const long nvec = (long)p->B * nchan;
	cudaStream_t st = r.stream;
	if (r.mask) {
		// the mask X^T (M X) in this basis (S^-1 is 1 there)
		const int N = p->N, nt = p->ntile, wt = std::min(nt - 1, (WMAX + 31) / 32 + 1);
		scratch tmp(st);
		double *Mx, *A;
		int rc;
		if ((rc = tmp.get(&Mx, (size_t)N * N)) || (rc = tmp.get(&A, (size_t)N * N))) return rc;
		QPC_CUDA(cudaMemsetAsync(A, 0, sizeof(double) * N * N, st));
		k_band_vec<<<(unsigned)(((long)N * N + 255) / 256), 256, 0, st>>>(r.mask, nullptr, N, p->P, p->Xt, Mx, nullptr);
		k_outer<<<dim3(nt, 2 * wt + 1), 256, 0, st>>>(p->Xt, Mx, nullptr, nullptr, N, nt, wt, 1, A, nullptr);
		*r.launches += 4;
		bool ok = false;
		if ((rc = store_real(p, p->K, A, N, 1, st, &ok))) return rc;
		if (!ok) { set_error("the mask does not fall off the diagonal in the position basis"); return QPC_ERR_NUMERIC; }
	}
	if (r.z && !p->zpart) if (int rc = dalloc(&p->zpart, (size_t)pos_path::ZB * p->B * p->M * p->ntile)) return rc;
	p->zcount = 0;
	POS_PROF(QPC_KERNEL_TRANSFORM_FWD);
	k_exponents<<<(unsigned)((nvec * p->ntile * 32 + 255) / 256), 256, 0, st>>>(r.state, p->exin, p->N, p->ntile, nvec);
	band_args a = args_of(p, p->W, nchan, p->B);
	a.s0 = r.state; a.e0 = p->exin; a.smap = r.perm;
	a.dst = p->buf[0]; a.edst = p->ex[0];
	band_apply<false>(a, p->ntile, st);
	*r.launches += 2;
	return QPC_OK;
}

static void sum_dipole(pos_path* p, const pos_run& r)
{
	if (!p->zcount) return;
	const int n = p->B * p->zcount;
	k_dipole_sum<<<(n + 127) / 128, 128, 0, r.stream>>>(p->zpart, r.z, r.ldz, r.ntt, p->B, p->M * p->ntile, p->zfirst, p->zcount);
	++*r.launches;
	p->zcount = 0;
}

int pos_step(pos_path* p, const pos_run& r, long s, int Bc, int Bf)
{
	// field-free steps alternate between the buffers; with a mask the state is in buf[0] before a step, and the
	// step leaves it in buf[1], from where the mask takes it back
	const int nchan = p->M * p->L;
	int cur = r.mask ? 1 : (int)(s & 1);
	cudaStream_t st = r.stream;
	auto angle = [&](int cmode, int slots, bool observe) {
		POS_PROF(QPC_KERNEL_SWEEP);
		angle_args a{};
		a.y = p->buf[cur]; a.ex = p->ex[cur]; a.V = p->V; a.lamp = p->lamp; a.r = p->r; a.ftab = r.ftab; a.ld = r.ld; a.ntf = r.ntf; a.ntt = r.ntt;
		a.step = s; a.cmode = cmode; a.dt4 = 0.25 * p->dt; a.N = p->N; a.ntile = p->ntile; a.L = p->L; a.M = p->M; a.npair = p->npair;
		if (observe) {
			if (!p->zcount) p->zfirst = s;
			a.zpart = p->zpart + (size_t)p->zcount * p->B * p->M * p->ntile;
			++p->zcount;
		}
		switch (p->angle_g) {
		case 2: angle_launch<2>(p, a, slots, st); break;
		case 3: angle_launch<3>(p, a, slots, st); break;
		default: angle_launch<4>(p, a, slots, st); break;
		}
		++*r.launches;
	};
	if (r.mask) {
		if (s > 0) {
			if (Bc > 0) angle(1, Bc, false);
			// the slots whose step s - 1 has just ended
			POS_PROF(QPC_KERNEL_TRANSFORM_BWD);
			band_args a = args_of(p, p->K, nchan, p->B);
			a.s0 = p->buf[1]; a.e0 = p->ex[1]; a.dst = p->buf[0]; a.edst = p->ex[0];
			a.nta = r.ntt; a.step = s - 1;
			band_apply<false>(a, p->ntile, st);
			++*r.launches;
		}
		cur = 0;
		if (Bc > 0) angle(2, Bc, false);
	} else if (r.z) {
		if (std::max(Bc, Bf) > 0) angle(0, std::max(Bc, Bf), true);
		if (p->zcount == pos_path::ZB) sum_dipole(p, r);
	} else if (Bc > 0) angle(0, Bc, false);
	if (Bf > 0) {
		POS_PROF(QPC_KERNEL_FIELDFREE);
		band_args a = args_of(p, p->F, nchan, Bf);
		a.lmap = p->lmap;
		a.set_stride = (long)p->nlh * p->F.stride;
		if (p->nff > 1) a.amap = r.perm;
		a.s0 = p->buf[cur]; a.e0 = p->ex[cur]; a.dst = p->buf[1 - cur]; a.edst = p->ex[1 - cur];
		a.nta = r.ntt; a.step = s;
		band_apply<true>(a, p->ntile, st);
		++*r.launches;
	}
	QPC_CUDA(cudaGetLastError());
	return QPC_OK;
}

int pos_end(pos_path* p, const pos_run& r)
{
	if (r.z) sum_dipole(p, r);
	POS_PROF(QPC_KERNEL_TRANSFORM_BWD);
	const int nchan = p->M * p->L;
	band_args a = args_of(p, p->X, nchan, p->B);
	a.s0 = p->buf[0]; a.e0 = p->ex[0]; a.s1 = p->buf[1]; a.e1 = p->ex[1]; a.par = r.mask ? nullptr : r.ntt; a.dmap = r.perm;
	a.dst = r.state; a.edst = p->exin;
	band_apply<false>(a, p->ntile, r.stream);
	++*r.launches;
	QPC_CUDA(cudaGetLastError());
	return QPC_OK;
}

} // namespace qpc
