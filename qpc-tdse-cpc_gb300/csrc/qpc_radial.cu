// Radial operators in a localised orthonormal basis, and their products in fixed point.
//
// With X the eigenvectors of a pencil (R, S) of banded radial matrices (R = <B|r|B> or -<B|1/r|B>), X^T S X = 1,
// every function of the position is diagonal, and any banded operator, S^-1 times one, or the Crank-Nicolson step
// F~_l = X^T S (S + i dt/2 H_l)^-1 (S - i dt/2 H_l) X is a fixed matrix whose entries fall off the diagonal by a
// constant factor per row (0.70 at p = 6): a band of ~110 either side holds F~_l to 2^-57.
//
// Arithmetic.  GB300 issues 2 FP64 FMAs per cycle and SM (1.6 measured) and 20-25 wide integer multiply-adds
// (32 x 32 + 64 bits, distinct operands, measured).  Both products have fixed matrices with entries of magnitude
// <= 1 and vectors whose largest element is known, so they are formed in fixed point: 56 bits under the vector's
// largest exponent (matrix: under 1), as two balanced 28-bit limbs; hi*hi and the two mixed products are summed
// exactly in 64-bit integers (three multiply-adds per product: ~4 times the DFMA rate, and without its 64-cycle
// latency), lo*lo lies at 2^-56 of the unit and is left out; one rounding to FP64 at the end.  The quantisation is
// 2^-57 of the largest element of the ~250 a sum covers, below the FP64 rounding of the sum itself.  Entries of
// F~ below 2^-29 have no hi limb: the outer part of the band costs one multiply-add and half the bytes.
#include "qpc_radial.cuh"
#include "qpc_tcband.cuh"
#include <cstring>
#include <cstdlib>
#include <cmath>
#include <type_traits>

namespace qpc {

namespace {

constexpr int SEEDW = 40;	// half-width of the windows the starting vectors are found in

// ------------------------------------------------------------------ banded products
// dst[col][row] = sum_k A_l[row][k] src[col][k] for every channel l and column (wavefunction).  A block owns
// TM rows of one channel and COLS = NB * 8/KS columns; each warp NB columns (lane = row), KS warps share a
// column and split its k.  The operator is stored per tile as chunks of KC k x TM rows, so that a warp's load is
// 32 consecutive elements; the columns are quantised into shared memory once per block and read as broadcasts.
// Bound by the integer multiply-adds from ~8 columns on (12 NB per k and lane against one 16-byte load), by the
// operator's bytes below.
template <int NB, int KS, bool CX>
__global__ void __launch_bounds__(256, 2) k_band_apply(const band_args p)
{
	constexpr int CG = 8 / KS, COLS = NB * CG, SK = 32 * KS, XS = COLS | 1;
	constexpr int FB = KC * TM * (CX ? 16 : 8), TB = FB / 2;
	constexpr int UN = NB <= 2 ? 8 : (NB <= 4 ? 4 : 2);
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
	const int4 td = p.td[tile];
	prev_wait();
	// every column's largest exponent over the tile's k range, one warp per column
	const int nex = p.ntile * EPT, x0 = td.x * KC / TE, x1 = td.w * KC / TE;
	for (int cl = warp; cl < COLS; cl += 8) {
		const int c = col0 + cl;
		int e = 0;
		const double2* src = nullptr;
		if (c < p.ncols && (!p.nta || p.step < p.nta[c])) {
			const bool odd = p.par && (p.par[c] & 1);
			const long v = (long)(p.smap ? p.smap[c] : c) * p.nchan + ch;
			const int* ex = (odd ? p.e1 : p.e0) + v * nex;
			for (int t = x0 + lane; t < x1; t += 32) e = max(e, ex[t]);
			src = (odd ? p.s1 : p.s0) + v * p.N;
		}
		e = __reduce_max_sync(0xffffffffu, e);
		if (lane == 0) { sE[cl] = e; sp[cl] = src; }
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
	const char* A = p.A + (long)p.lmap[ch] * p.astride + p.toff[tile];
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
		// the stage's chunks before, with and after the hi limbs.  Of every chunk a warp takes KC / KS k, so that the
		// warps of a column have equal work whatever the kind of a chunk; with eight warps to a column (few columns,
		// bound by the latency of the operator's loads) two whole chunks, all their loads in flight
		constexpr int KW = KS == 8 ? KC : KC / KS;
		const int k0 = KS == 8 ? 0 : ks * KW;
		const int ce = min(c0 + 2 * KS, td.w);
		auto span = [&](int ca, int cb, const char* seg, auto full) {
			constexpr bool FULL = decltype(full)::value;
			const int n = (cb - ca) * KW;
			const int4* x = xs + ((ca - c0) * KC + k0) * XS + wc;
			using elem = std::conditional_t<CX, std::conditional_t<FULL, int4, int2>, std::conditional_t<FULL, int2, int>>;
			const elem* src = reinterpret_cast<const elem*>(seg) + k0 * TM + lane;
			// UN loads in flight, then their products (elements past the end: zero)
			for (int i0 = 0; i0 < n; i0 += UN) {
				elem av[UN];
#pragma unroll
				for (int u = 0; u < UN; ++u) {
					const int i = i0 + u;
					if constexpr (KW % UN == 0) av[u] = __ldg(src + ((i / KW) * KC + i % KW) * TM);
					else av[u] = i < n ? __ldg(src + ((i / KW) * KC + i % KW) * TM) : elem{};
				}
#pragma unroll
				for (int u = 0; u < UN; ++u) {
					const int i = KW % UN == 0 ? i0 + u : min(i0 + u, n - 1);
					const int4* y0 = x + ((i / KW) * KC + i % KW) * XS;
					if constexpr (CX && FULL) {
						const int4 A4 = av[u];
						const int nz = -A4.z, nw = -A4.w;
#pragma unroll
						for (int j = 0; j < NB; ++j) {
							const int4 y = y0[j];
							rh[j] = madw(A4.x, y.x, rh[j]); ih[j] = madw(A4.x, y.z, ih[j]); rm[j] = madw(A4.x, y.y, rm[j]); im[j] = madw(A4.x, y.w, im[j]);
							rh[j] = madw(nz, y.z, rh[j]); ih[j] = madw(A4.z, y.x, ih[j]); rm[j] = madw(nz, y.w, rm[j]); im[j] = madw(A4.z, y.y, im[j]);
							rm[j] = madw(A4.y, y.x, rm[j]); im[j] = madw(A4.y, y.z, im[j]);
							rm[j] = madw(nw, y.z, rm[j]); im[j] = madw(A4.w, y.x, im[j]);
						}
					} else if constexpr (CX) {
						const int2 A2 = av[u];
						const int nb = -A2.y;
#pragma unroll
						for (int j = 0; j < NB; ++j) {
							const int4 y = y0[j];
							rm[j] = madw(A2.x, y.x, rm[j]); im[j] = madw(A2.x, y.z, im[j]);
							rm[j] = madw(nb, y.z, rm[j]); im[j] = madw(A2.y, y.x, im[j]);
						}
					} else if constexpr (FULL) {
						const int2 A2 = av[u];
#pragma unroll
						for (int j = 0; j < NB; ++j) {
							const int4 y = y0[j];
							rh[j] = madw(A2.x, y.x, rh[j]); ih[j] = madw(A2.x, y.z, ih[j]); rm[j] = madw(A2.x, y.y, rm[j]); im[j] = madw(A2.x, y.w, im[j]);
							rm[j] = madw(A2.y, y.x, rm[j]); im[j] = madw(A2.y, y.z, im[j]);
						}
					} else {
						const int A1 = av[u];
#pragma unroll
						for (int j = 0; j < NB; ++j) {
							const int4 y = y0[j];
							rm[j] = madw(A1, y.x, rm[j]); im[j] = madw(A1, y.z, im[j]);
						}
					}
				}
			}
		};
		auto spans = [&](int from, int to) {
			if (from < td.y) span(from, min(to, td.y), A + (long)(from - td.x) * TB, std::false_type());
			if (from < td.z && to > td.y) {
				const int ca = max(from, td.y);
				span(ca, min(to, td.z), A + tl + (long)(ca - td.y) * FB, std::true_type());
			}
			if (to > td.z) {
				const int ca = max(from, td.z);
				span(ca, to, A + tf + (long)(ca - td.z) * TB, std::false_type());
			}
		};
		if constexpr (KS == 8) {
			if (c0 + ks < td.w) spans(c0 + ks, c0 + ks + 1);
			if (c0 + ks + 8 < td.w) spans(c0 + ks + 8, c0 + ks + 9);
		} else spans(c0, ce);
		// at most 32 k since the last flush: 128 mixed products below 2^55
#pragma unroll
		for (int j = 0; j < NB; ++j) { flush(rh[j], rm[j]); flush(ih[j], im[j]); }
		__syncthreads();
	}
	const int row = tile * TM + lane;
	auto emit = [&](int cl, long long hr, long long mr, long long hi, long long mi) {
		const int c = col0 + cl;
		if (c >= p.ncols || (p.nta && !(p.step < p.nta[c]))) return;
		const int E = sE[cl], s = p.ea + E - 1078 + (!CX && p.er && row < p.N ? p.er[row] : 0);
		const double2 y = make_double2(to_double<!CX>(hr, mr, s, E > EMAX), to_double<!CX>(hi, mi, s, E > EMAX));
		const long o = (long)(p.dmap ? p.dmap[c] : c) * p.nchan + ch;
		if (row < p.N) p.dst[o * p.N + row] = y;
		const int e = group_max(row < p.N ? max(bexp(y.x), bexp(y.y)) : 0);
		if (lane % TE == 0) p.edst[o * nex + tile * EPT + lane / TE] = e;
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

// The same for one column per block (one wavefunction, or an operator of its own for each): eight warps split k by whole
// chunks.  Bound by the latency of its loads and the operator's bytes, so a warp's first eight k of the operator are on
// their way before the column is, four blocks share an SM, and only one barrier stands between the loads and the
// products.  F~ of 800 x 41 (105 MB) 30 -> 24 us, 4 x (400 x 21) with own potentials 30 -> 25 us against k_band_apply<1, 8>
// (two blocks, 16 k in flight after two barriers); what comes before prev_wait() then overlaps the kernel before.
template <bool CX>
__global__ void __launch_bounds__(256, 4) k_band_one(const band_args p)
{
	constexpr int FB = KC * TM * (CX ? 16 : 8), TB = FB / 2, UN = 8, RC = 32;	// RC: chunks of a round
	__shared__ int4 xs[RC * KC];
	__shared__ long long red[8][4][32];
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const int c = blockIdx.x % p.ncols, tile = p.tile0 + blockIdx.x / p.ncols, ch = blockIdx.y;
	const int4 td = p.td[tile];
	const long toff = p.toff[tile];
	const bool on = !p.nta || p.step < p.nta[c];
	const int nex = p.ntile * EPT;
	const bool odd = p.par && (p.par[c] & 1);
	const long v = (long)(p.smap ? p.smap[c] : c) * p.nchan + ch;
	const int set = p.amap ? p.amap[p.dmap ? p.dmap[c] : c] : 0;
	const char* A = p.A + set * p.set_stride + (long)p.lmap[ch] * p.astride + toff;
	const long tl = (long)(td.y - td.x) * TB, tf = tl + (long)(td.z - td.y) * FB;
	using full_t = std::conditional_t<CX, int4, int2>;
	using tail_t = std::conditional_t<CX, int2, int>;
	int4 av[UN];
	auto fetch = [&](int k, int half) {	// eight k of chunk k
		if (k >= td.y && k < td.z) {
			const full_t* q = reinterpret_cast<const full_t*>(A + tl + (long)(k - td.y) * FB) + half * UN * TM + lane;
#pragma unroll
			for (int u = 0; u < UN; ++u) {
				const full_t a = __ldg(q + u * TM);
				if constexpr (CX) av[u] = a; else av[u] = make_int4(a.x, a.y, 0, 0);
			}
		} else {
			const tail_t* q = reinterpret_cast<const tail_t*>(A + (k < td.y ? (long)(k - td.x) * TB : tf + (long)(k - td.z) * TB)) + half * UN * TM + lane;
#pragma unroll
			for (int u = 0; u < UN; ++u) {
				const tail_t a = __ldg(q + u * TM);
				if constexpr (CX) av[u] = make_int4(a.x, a.y, 0, 0); else av[u] = make_int4(a, 0, 0, 0);
			}
		}
	};
	const double2* src = (odd ? p.s1 : p.s0) + v * p.N;
	const int* ex = (odd ? p.e1 : p.e0) + v * nex;
	const int kend = min(p.N, td.w * KC);
	long long rh = 0, rm = 0, ih = 0, im = 0;
	int E = 0;
	for (int c0 = td.x; c0 < td.w; c0 += RC) {
		if (on && c0 + warp < td.w) fetch(c0 + warp, 0);
		if (c0 == td.x) {
			prev_wait();
			if (!on) return;
		}
		double2 raw[RC * KC / 256];
#pragma unroll
		for (int i = 0; i < RC * KC / 256; ++i) {
			const int k = c0 * KC + i * 256 + threadIdx.x;
			raw[i] = k < kend ? src[k] : make_double2(0.0, 0.0);
		}
		if (c0 == td.x) {	// the column's largest exponent over the tile's k range
			for (int t = td.x * KC / TE + lane; t < td.w * KC / TE; t += 32) E = max(E, ex[t]);
			E = __reduce_max_sync(0xffffffffu, E);
		} else __syncthreads();
#pragma unroll
		for (int i = 0; i < RC * KC / 256; ++i) {
			const int2 a = quant(raw[i].x, E), b = quant(raw[i].y, E);
			xs[i * 256 + threadIdx.x] = make_int4(a.x, a.y, b.x, b.y);
		}
		__syncthreads();
		const int ce = min(c0 + RC, td.w);
		for (int k = c0 + warp; k < ce; k += 8) {
#pragma unroll
			for (int half = 0; half < 2; ++half) {
				const int4* x = xs + (k - c0) * KC + half * UN;
				if (half || k >= c0 + 8) fetch(k, half);
				if (k >= td.y && k < td.z) {
#pragma unroll
					for (int u = 0; u < UN; ++u) {
						const int4 y = x[u], a = av[u];
						rh = madw(a.x, y.x, rh); ih = madw(a.x, y.z, ih); rm = madw(a.x, y.y, rm); im = madw(a.x, y.w, im);
						rm = madw(a.y, y.x, rm); im = madw(a.y, y.z, im);
						if constexpr (CX) {
							const int nz = -a.z, nw = -a.w;
							rh = madw(nz, y.z, rh); ih = madw(a.z, y.x, ih); rm = madw(nz, y.w, rm); im = madw(a.z, y.y, im);
							rm = madw(nw, y.z, rm); im = madw(a.w, y.x, im);
						}
					}
				} else {
#pragma unroll
					for (int u = 0; u < UN; ++u) {
						const int4 y = x[u], a = av[u];
						rm = madw(a.x, y.x, rm); im = madw(a.x, y.z, im);
						if constexpr (CX) { rm = madw(-a.y, y.z, rm); im = madw(a.y, y.x, im); }
					}
				}
			}
			flush(rh, rm); flush(ih, im);	// every 16 k: 64 mixed products below 2^55
		}
	}
	red[warp][0][lane] = rh; red[warp][1][lane] = rm; red[warp][2][lane] = ih; red[warp][3][lane] = im;
	__syncthreads();
	if (warp) return;
#pragma unroll
	for (int w = 1; w < 8; ++w) { rh += red[w][0][lane]; rm += red[w][1][lane]; ih += red[w][2][lane]; im += red[w][3][lane]; }
	flush(rh, rm); flush(ih, im);
	const int row = tile * TM + lane, s = p.ea + E - 1078 + (!CX && p.er && row < p.N ? p.er[row] : 0);
	const double2 y = make_double2(to_double<!CX>(rh, rm, s, E > EMAX), to_double<!CX>(ih, im, s, E > EMAX));
	const long o = (long)(p.dmap ? p.dmap[c] : c) * p.nchan + ch;
	if (row < p.N) p.dst[o * p.N + row] = y;
	const int e = group_max(row < p.N ? max(bexp(y.x), bexp(y.y)) : 0);
	if (lane % TE == 0) p.edst[o * nex + tile * EPT + lane / TE] = e;
}

// largest exponent of every TE rows of src [nvec][N]
__global__ void k_exponents(const double2* __restrict__ src, int* __restrict__ ex, int N, int ntile, long nvec)
{
	const long w = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
	const int lane = threadIdx.x & 31;
	if (w >= nvec * ntile) return;
	const long vec = w / ntile;
	const int row = (int)(w % ntile) * TM + lane;
	int e = 0;
	if (row < N) { const double2 v = src[vec * N + row]; e = max(bexp(v.x), bexp(v.y)); }
	e = group_max(e);
	if (lane % TE == 0) ex[w * EPT + lane / TE] = e;
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

// Yt[i] = S x_i, Zt[i] = R x_i (R may be NULL); sgn = -1: S anti-symmetric, given by its upper entries
__global__ void k_band_vec(const double* __restrict__ S, const double* __restrict__ R, int N, int P, const double* __restrict__ Xt, double* __restrict__ Yt,
	double* __restrict__ Zt, double sgn = 1.0)
{
	const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
	if (t >= (long)N * N) return;
	const int r = (int)(t % N), NE = P + 1;
	const double* x = Xt + t;
	double y = S[(long)r * NE] * x[0], z = R ? R[(long)r * NE] * x[0] : 0.0;
	for (int k = 1; k <= P; ++k) {
		if (r - k >= 0) { y = fma(sgn * S[(long)(r - k) * NE + k], x[-k], y); if (R) z = fma(R[(long)(r - k) * NE + k], x[-k], z); }
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
// tiles on and above the diagonal only, stored as C[j][i] = E_ij, the largest magnitude in err; mode 1: C = A B^T;
// mode 2 (A = B): C = (1 - A A^T)/2, its largest magnitude in err.
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
		double big = 0.0;
#pragma unroll
		for (int u = 0; u < 4; ++u) {
			const int i = ti * 32 + y0 + 8 * u;
			if (i >= N || j >= N) continue;
			const double v = mode == 1 ? g[u] : 0.5 * ((i == j ? 1.0 : 0.0) - g[u]);
			C[(long)i * N + j] = v;
			big = fmax(big, isfinite(v) ? fabs(v) : 1e300);
		}
		if (mode == 2) {
			for (int o = 16; o; o >>= 1) big = fmax(big, __shfl_xor_sync(0xffffffffu, big, o));
			if (x == 0) atomicMax(err, (unsigned long long)__double_as_longlong(big));
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

// each row under its own power of two: A(i, j) = out[i][j] 2^er[i], |out| < 1
__global__ void __launch_bounds__(128) k_scale_rows(const double* __restrict__ A, long si, long sj, int N, double* __restrict__ out, int* __restrict__ er)
{
	const int i = blockIdx.x;
	__shared__ double part[4];
	double big = 0.0;
	for (int j = threadIdx.x; j < N; j += 128) big = fmax(big, fabs(A[i * si + j * sj]));
	for (int o = 16; o; o >>= 1) big = fmax(big, __shfl_xor_sync(0xffffffffu, big, o));
	if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = big;
	__syncthreads();
	big = fmax(fmax(part[0], part[1]), fmax(part[2], part[3]));
	const int e = big > 0.0 && big < 1e200 ? ilogb(big) + 1 : 0;
	if (threadIdx.x == 0) er[i] = e;
	for (int j = threadIdx.x; j < N; j += 128) out[(long)i * N + j] = ldexp(A[i * si + j * sj], -e);
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

// X[jj][r][l] (r-major) or X[jj][l][r] = (x_{j0 + jj})_r for every l
__global__ void k_columns(const double* __restrict__ Xt, int j0, int N, int nlh, bool rmajor, long total, double2* __restrict__ X)
{
	const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
	if (t >= total) return;
	X[t] = make_double2(Xt[(long)j0 * N + (rmajor ? t / nlh : t / ((long)nlh * N) * N + t % N)], 0.0);
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

// ------------------------------------------------------------------ host side

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

int upload(band_store& b, size_t bytes, cudaStream_t st)
{
	const size_t nt = b.td.size();
	int rc;
	if (!b.d_td) if ((rc = dalloc(&b.d_td, nt)) || (rc = dalloc(&b.d_off, nt))) return rc;
	if (b.cap < bytes) {
		cudaFree(b.A); b.A = nullptr; b.cap = 0;
		if ((rc = dalloc(&b.A, bytes))) return rc;
		b.cap = bytes;
	}
	QPC_CUDA(cudaMemcpyAsync(b.d_td, b.td.data(), sizeof(int4) * nt, cudaMemcpyHostToDevice, st));
	QPC_CUDA(cudaMemcpyAsync(b.d_off, b.off.data(), sizeof(long) * nt, cudaMemcpyHostToDevice, st));
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

int read_profile(radial_ops* p, cudaStream_t st, std::vector<unsigned long long>& prof)
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
	launch_after(k_band_apply<NB, KS, CX>, dim3((unsigned)(tiles * ncg), (unsigned)a.nchan), 256, smem, st, a);
}

template <int NB, int KS>
void band_attr()
{
	constexpr int smem = (int)band_smem<NB, KS>();
	cudaFuncSetAttribute(k_band_apply<NB, KS, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
	cudaFuncSetAttribute(k_band_apply<NB, KS, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
}

// Columns per block: 64 (8 per warp) keeps the operator's traffic lowest; fewer where 64 or 32 would leave SMs
// without a second block (two fit), and, for few columns, warps that share a column and split its k so that a
// block still has eight.
template <bool CX>
int dispatch(const band_args& a, int tiles, cudaStream_t st)
{
	const int n = a.ncols;
	const long per = (long)tiles * a.nchan;
	auto blocks = [&](int cols) { return per * ((n + cols - 1) / cols); };
	if (a.amap || n == 1) {
		launch_after(k_band_one<CX>, dim3((unsigned)(tiles * n), (unsigned)a.nchan), 256, 0, st, a);
		return QPC_PRODUCT_ONE;
	}
	if (n == 2) band_launch<2, 8, CX>(a, tiles, st);
	else if (n <= 4) band_launch<4, 8, CX>(a, tiles, st);
	else if (n <= 8) band_launch<4, 4, CX>(a, tiles, st);
	else if (n <= 16 || blocks(32) < 304) band_launch<4, 2, CX>(a, tiles, st);
	else if (n <= 32 || (n > 64 && n <= 96) || blocks(64) < 608) band_launch<4, 1, CX>(a, tiles, st);
	else band_launch<8, 1, CX>(a, tiles, st);
	return QPC_PRODUCT_MADD;
}

template <int P>
void seed(const radial_setup& in, double* Xt) { k_seed<P><<<in.N, 32, 0, in.stream>>>(in.R, in.S, in.N, Xt); }

// the eigenvectors Xt and positions r; ok = false when the refinement does not converge
int eigenvectors(radial_ops* p, const radial_setup& in, scratch& tmp, double** Yt_out, bool* ok)
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


std::vector<double> as_doubles(const std::vector<unsigned long long>& prof)
{
	std::vector<double> d(prof.size());
	std::memcpy(d.data(), prof.data(), 8 * d.size());
	return d;
}

// scale and profile of a real operator; ok as in decay()
int store_banded_impl(radial_ops* p, band_store& b, const double* A, long si, long sj, cudaStream_t st, bool dense, bool* ok)
{
	double big = 0.0;
	int w = p->N - 1, wf = p->N - 1;
	*ok = true;
	if (dense) {	// orthogonal matrices
		b.ea = 0;
		*ok = p->N <= DENSE_MAX;
		if (!*ok) return QPC_OK;
	}
	else {
		std::vector<unsigned long long> prof;
		QPC_CUDA(cudaMemsetAsync(p->prof, 0, sizeof(unsigned long long) * (WMAX + 1), st));
		k_profile<<<std::min(WMAX, p->N - 1) + 1, 128, 0, st>>>(A, si, sj, p->N, p->prof);
		if (int rc = read_profile(p, st, prof)) return rc;
		for (auto u : prof) { double v; std::memcpy(&v, &u, 8); big = std::max(big, v); }
		*ok = big == 0.0 || (big > 1e-200 && big < 1e200);	// its power of two and the limbs' in FP64
		if (!*ok) return QPC_OK;
		b.ea = 0;	// of zeros
		if (big > 0.0) std::frexp(big, &b.ea);
		*ok = decay(prof, p->N, std::ldexp(1.0, b.ea), w, wf, 29);
		if (!*ok) return QPC_OK;
		double sum = -big;	// at least any row's sum of magnitudes
		for (int d = 0; d <= std::min(w, WMAX); ++d) { double v; std::memcpy(&v, &prof[d], 8); sum += 2.0 * v; }
		*ok = sum <= std::ldexp(SUM_MAX, b.ea);
		if (!*ok) return QPC_OK;
		b.prof = as_doubles(prof);
	}
	lay_out(b, p->N, w, wf, false);
	if (int rc = upload(b, (size_t)b.stride, st)) return rc;
	k_store<false><<<dim3(p->ntile, 1), 256, 0, st>>>(nullptr, A, si, sj, p->N, w, std::ldexp(1.0, 56 - b.ea), b.d_td, b.d_off, b.A, b.stride);
	QPC_CUDA(cudaGetLastError());
	return QPC_OK;
}

int build(radial_ops* p, const radial_setup& in, int nmap, bool* ok)
{
	const int N = p->N, nlh = p->nlh;
	cudaStream_t st = in.stream;
	int rc;
	const size_t nz = (size_t)std::max(nmap, nlh);
	if ((rc = dalloc(&p->Xt, (size_t)N * N)) || (rc = dalloc(&p->r, N)) || (rc = dalloc(&p->prof, WMAX + 1)) || (rc = dalloc(&p->zero, nz))) return rc;
	QPC_CUDA(cudaMemsetAsync(p->zero, 0, sizeof(int) * nz, st));
	scratch tmp(st);
	double* Yt = nullptr;
	if ((rc = eigenvectors(p, in, tmp, &Yt, ok)) || !*ok) return rc;
	// The rows of W = X^T S go with sqrt(h) and those of X with 1 / sqrt(h), h the grid's local spacing: one power of two for
	// all would leave the rows of a graded grid's fine end log2 sqrt(h_max / h_min) bits fewer.  W also forms F~ below.
	double *Ws, *Xs;
	if ((rc = dalloc(&p->W.er, N)) || (rc = dalloc(&p->X.er, N)) || (rc = tmp.get(&Ws, (size_t)N * N)) || (rc = tmp.get(&Xs, (size_t)N * N))) return rc;
	k_scale_rows<<<N, 128, 0, st>>>(Yt, N, 1, N, Ws, p->W.er);
	k_scale_rows<<<N, 128, 0, st>>>(p->Xt, 1, N, N, Xs, p->X.er);
	QPC_CUDA(cudaGetLastError());
	if ((rc = store_banded(p, p->W, Ws, N, 1, st, ok)) || !*ok) return rc;
	if ((rc = store_banded(p, p->X, Xs, N, 1, st, ok)) || !*ok) return rc;
	const char* mode = std::getenv("QPC_POS_TC");	// 0: multiply-adds only, 1: tensor cores wherever they can
	const bool always = mode && mode[0] == '1';
	p->F.tc_always = p->W.tc_always = p->X.tc_always = always;
	const bool tcp = p->nff == 1 && (always || (in.batch >= TC_MIN && N >= 128 && !(mode && mode[0] == '0')));
	if (tcp) {
		if ((rc = tc_make(p->W.tc, nullptr, Ws, 0, N, 1, N, N, 1, p->W.w, p->W.prof.data(), p->W.ea, false, st, &p->W.has_tc))) return rc;
		if ((rc = tc_make(p->X.tc, nullptr, Xs, 0, N, 1, N, N, 1, p->X.w, p->X.prof.data(), p->X.ea, false, st, &p->X.has_tc))) return rc;
	}
	// F~_l, a set of columns at a time: the engine's field-free solve on the eigenvectors, then X^T S
	const int J = (int)std::min<long>(N, std::max<long>(32, (64l << 20) / ((long)N * nlh * 16)));
	const size_t chunk = (size_t)J * N * nlh;
	double2 *c0, *c1, *Fb;
	int *ce, *cd;
	const size_t band = (size_t)nlh * N * (2 * WMAX + 1);
	if ((rc = tmp.get(&c0, chunk)) || (rc = tmp.get(&c1, chunk)) || (rc = tmp.get(&Fb, band)) || (rc = tmp.get(&ce, (size_t)J * nlh * p->ntile * EPT)) ||
		(rc = tmp.get(&cd, (size_t)J * nlh * p->ntile * EPT)))
		return rc;
	std::vector<unsigned long long> prof;
	for (int fi = 0; fi < p->nff; ++fi) {
		QPC_CUDA(cudaMemsetAsync(Fb, 0, sizeof(double2) * band, st));
		if (fi == 0) QPC_CUDA(cudaMemsetAsync(p->prof, 0, sizeof(unsigned long long) * (WMAX + 1), st));
		for (int j0 = 0; j0 < N; j0 += J) {
			const int n = std::min(J, N - j0);
			const long total = (long)n * N * nlh, vec = (long)n * nlh;
			if (in.rmajor) {
				k_columns<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(p->Xt, j0, N, nlh, true, total, c0);
				if ((rc = in.fieldfree(c0, c1, n, fi))) return rc;
				k_transpose<<<dim3((N + 31) / 32, (nlh + 31) / 32, n), 256, 0, st>>>(c0, c1, N, nlh);
			} else {
				k_columns<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(p->Xt, j0, N, nlh, false, total, c1);
				if ((rc = in.fieldfree(c1, c0, n, fi))) return rc;
			}
			exponents(c1, ce, N, p->ntile, vec, st);
			band_args a = band_args_of(p, p->W, nlh, n);
			a.s0 = c1; a.e0 = ce; a.dst = c0; a.edst = cd;
			a.tile0 = std::max(0, (j0 - WMAX) / TM);
			band_apply(a, false, std::min(p->ntile, (j0 + n + WMAX + TM - 1) / TM) - a.tile0, st);
			k_gather_band<<<dim3(n, nlh), 128, 0, st>>>(c0, j0, n, N, nlh, Fb, p->prof);
			QPC_CUDA(cudaGetLastError());
		}
		if (fi == 0) {
			if ((rc = read_profile(p, st, prof))) return rc;
			int w, wf;
			if (!(*ok = decay(prof, N, 1.0, w, wf, 29))) return QPC_OK;
			if (p->nff > 1) { w = std::min(std::min(WMAX, N - 1), w + 8); wf = std::min(w, wf + 12); }	// the other potentials' bands, checked below
			lay_out(p->F, N, w, wf, true);
			// resident for the handle's life: at most 16 GB, and a quarter of what is free (more handles and the caller's own data share the card)
			if (!(*ok = (size_t)p->F.stride * nlh * p->nff <= std::min<size_t>((size_t)16 << 30, free_bytes() / 4))) return QPC_OK;
			if ((rc = upload(p->F, (size_t)p->F.stride * nlh * p->nff, st))) return rc;
		}
		k_store<true><<<dim3(p->ntile, nlh), 256, 0, st>>>(Fb, nullptr, 0, 0, N, p->F.w, std::ldexp(1.0, 56), p->F.d_td, p->F.d_off,
			p->F.A + (size_t)fi * nlh * p->F.stride, p->F.stride);
		if (tcp) {
			const std::vector<double> pd = as_doubles(prof);
			if ((rc = tc_make(p->F.tc, Fb, nullptr, 0, 0, 0, N, N, nlh, p->F.w, pd.data(), 0, false, st, &p->F.has_tc))) return rc;
		}
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
	return wait_on(st);
}

void set_attrs()
{
	band_attr<2, 8>(); band_attr<4, 8>(); band_attr<4, 4>(); band_attr<4, 2>(); band_attr<4, 1>(); band_attr<8, 1>();
}

} // namespace

void exponents(const double2* src, int* ex, int N, int ntile, long nvec, cudaStream_t st)
{
	k_exponents<<<(unsigned)((nvec * ntile * 32 + 255) / 256), 256, 0, st>>>(src, ex, N, ntile, nvec);
}

band_args band_args_of(const radial_ops* p, const band_store& b, int nchan, int ncols)
{
	band_args a{};
	a.A = b.A; a.astride = b.stride; a.td = b.d_td; a.toff = b.d_off; a.ea = b.ea; a.er = b.er;
	a.N = p->N; a.ntile = p->ntile; a.nchan = nchan; a.ncols = ncols;
	a.lmap = p->zero;
	return a;
}

// Microseconds of k_band_apply: its multiply-adds at 8e12 a second (26 per cycle and SM), 6 us of latency.  Measured against
// the tensor cores (F~, us): 800 x 41, 4 columns 56 to 76, 8 98 to 78, 48 613 to 131; 400 x 21, 8 30 to 41, 12 50 to 41,
// 48 164 to 56; 250 x 30 (p = 7), 8 30 to 33, 16 50 to 34.  The two estimates cross where these do
static double madd_cost(const band_store& b, bool cx, int nchan, int ncols)
{
	double k = 0.0;
	for (const int4& t : b.td) k += KC * ((t.z - t.y) * (cx ? 12.0 : 6.0) + (t.y - t.x + t.w - t.z) * (cx ? 4.0 : 2.0));
	return 6.0 + k * TM * nchan * ((ncols + 7) & ~7) / 8e6;
}

int band_apply(const band_args& a, bool cx, int tiles, cudaStream_t st, const band_store* b, int* status, int stbit)
{
	if (b && b->has_tc && !a.amap && (b->tc_always || tc_cost(b->tc, a.nchan, a.ncols) < madd_cost(*b, cx, a.nchan, a.ncols))) {
		tc_apply(b->tc, a, status, stbit, st);
		return QPC_PRODUCT_DIGITS;
	}
	return cx ? dispatch<true>(a, tiles, st) : dispatch<false>(a, tiles, st);
}

int store_banded(radial_ops* p, band_store& b, const double* A, long si, long sj, cudaStream_t st, bool* ok)
{
	return store_banded_impl(p, b, A, si, sj, st, false, ok);
}

int store_dense(radial_ops* p, band_store& b, const double* A, long si, long sj, int ncols, cudaStream_t st, bool* ok)
{
	if (int rc = store_banded_impl(p, b, A, si, sj, st, true, ok)) return rc;
	if (!*ok) return QPC_OK;
	const char* mode = std::getenv("QPC_POS_TC");
	b.tc_always = mode && mode[0] == '1';
	if (ncols < TC_MIN || (mode && mode[0] == '0')) return QPC_OK;
	return tc_make(b.tc, nullptr, A, 0, si, sj, p->N, p->N, 1, -1, nullptr, 0, true, st, &b.has_tc);
}

int project_band(const radial_ops* p, const double* B, bool anti, double* Bx, double* A, cudaStream_t st)
{
	const int N = p->N, nt = p->ntile, wt = std::min(nt - 1, (WMAX + 31) / 32 + 1);
	QPC_CUDA(cudaMemsetAsync(A, 0, sizeof(double) * N * N, st));
	k_band_vec<<<(unsigned)(((long)N * N + 255) / 256), 256, 0, st>>>(B, nullptr, N, p->P, p->Xt, Bx, nullptr, anti ? -1.0 : 1.0);
	k_outer<<<dim3(nt, 2 * wt + 1), 256, 0, st>>>(p->Xt, Bx, nullptr, nullptr, N, nt, wt, 1, A, nullptr);
	QPC_CUDA(cudaGetLastError());
	return QPC_OK;
}

// Newton-Schulz, Q <- Q (3 - Q^T Q)/2 twice (rows of Qt); the second correction is at the rounding level
int orthonormalise(double* Qt, int N, double* E, double* T, cudaStream_t st, bool* ok)
{
	const int nt = (N + TM - 1) / TM;
	scratch tmp(st);
	unsigned long long* err;
	int rc;
	if ((rc = tmp.get(&err, 2))) return rc;
	QPC_CUDA(cudaMemsetAsync(err, 0, sizeof(*err) * 2, st));
	for (int it = 0; it < 2; ++it) {
		k_outer<<<dim3(nt, 2 * nt + 1), 256, 0, st>>>(Qt, Qt, nullptr, nullptr, N, nt, nt, 2, E, err + it);
		k_update<<<dim3(nt, 2 * nt + 1), 256, 0, st>>>(E, Qt, N, nt, nt, T);
		QPC_CUDA(cudaMemcpyAsync(Qt, T, sizeof(double) * N * N, cudaMemcpyDeviceToDevice, st));
	}
	QPC_CUDA(cudaGetLastError());
	double e[2];
	if ((rc = copy_to_host(e, err, sizeof(e), st))) return rc;
	*ok = e[0] < 1e-3 && e[1] < 1e-6;
	return QPC_OK;
}

int radial_create(radial_ops* p, const radial_setup& in, int nmap, bool* ok)
{
	p->N = in.N; p->P = in.P; p->nlh = in.nlh; p->nff = in.nff; p->ntile = (in.N + TM - 1) / TM;
	set_attrs();
	*ok = false;
	return build(p, in, nmap, ok);
}

void radial_destroy(radial_ops* p)
{
	cudaFree(p->Xt); cudaFree(p->r); cudaFree(p->prof); cudaFree(p->zero);
	p->F.release(); p->W.release(); p->X.release();
}

} // namespace qpc
