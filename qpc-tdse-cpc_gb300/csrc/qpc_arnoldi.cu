// GB300 (sm_103a) engine for the QPC-TDSE Arnoldi (Lanczos) propagator in the
// length gauge: propagator_arnoldi::propagate1 driven by propagator_hc_lgwz
// (spherical/propagator/la_1e.hpp:312-335, 390-444).  One step maps
// w -> exp(-i dt S^-1 H) w in a Krylov space of at most kmax vectors built in
// the S metric, H = H_l (x) 1 + ez R (x) Y10.
//
// A batch holds B wavefunctions on one radial grid; each may carry its own
// Hamiltonian (its own potential) and its own field table and step count.
// Per step and per instance the kernels are
//   k_ar_snorm   |w|_S (and, inside the loop, |v|_S with the breakdown test)
//   k_ar_expand  u_k = v_k / |v_k|_S, v_{k+1} = H u_k, x_i = <u_i|v_{k+1}>
//   k_ar_sinv    v = S^-1 v, forward and backward banded Cholesky sweeps
//   k_ar_orth    v -= x_i u_i (i = k always, others when |x_i|^2 > 4e-27)
//   k_ar_small   exp(-i dt T) e1 b0 for the m x m tridiagonal T (implicit QL)
//   k_ar_combine w = sum_i x_i u_i
// in the reference's order of operations (la_1e.hpp:132-240).  Reductions are
// deterministic: each block writes a partial, and the last block of the
// instance to finish adds the partials in a fixed order.
//
// The state is kept r-major inside the engine, [inst][r][ch] with ch = im n_l + il,
// so that one warp reads 32 consecutive doubles: consecutive channels at one r
// for the band products, and the real and imaginary parts of consecutive
// channels for the S^-1 recurrences (one real recurrence per lane).
// All arithmetic is complex FP64.
#include "qpc_internal.h"
#include "qpc_cuda_util.cuh"
#include <cuda_runtime.h>
#include <cmath>
#include <vector>
#include <algorithm>
#include <cstdlib>

namespace qpc {
namespace {

constexpr int AR_THREADS = 256;
// elements per thread of the element-wise kernels: 4, or 1 for batches whose blocks would leave SMs idle
constexpr int AR_KMAX = 32;                          // largest Krylov dimension accepted
constexpr int CH_THREADS = 32;                       // real recurrences per block of k_ar_sinv

// per-instance state of the expansion within one step
enum : int { AR_LIVE = 0, AR_BROKEN = 1, AR_IDLE = 2 };
// device status bits (never a trap)
enum : int { ARS_NONFINITE = 2, ARS_NOCONV = 4, ARS_ZERO = 8 };

struct ar_args {
	int N, P, L, M, m0, nch, nlh, B, kmax, nbe;
	int b0;       // first instance of the group a launch covers (blockIdx.y / blockIdx.x offset)
	long n;       // complex elements per instance
	long hstride; // doubles between the Hamiltonians of consecutive instances (0: shared)
	double dt, emin, emax;
	const double *S, *R, *Lrow, *Lcol, *dinv, *H, *y10;
	const double *SM, *SN, *SI;	// block substitution (k_ar_sinv_blk): M_t, N_t, L11^-1 per block [P][P]
	const double *SF, *SB;		// products of -M, -N from the start of a segment
	double2 *X, *U, *V0, *V1;
	double2* partX;
	double* partN;
	unsigned* cnt;
	double2* xfin;
	double *a, *b, *sfac, *nu0;
	int *msub, *flag;
	double2* xc;
	const double* ez;
	long ld;
	const long long* nt;
	int8_t *crit, *msub_out;
	int* status;
};

__device__ __forceinline__ double2 cmul(double2 x, double2 y)
{
	return make_double2(fma(y.x, x.x, -(y.y * x.y)), fma(y.x, x.y, y.y * x.x));
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 rmul(double2 x, double s) { return make_double2(x.x * s, x.y * s); }
// conj(u) v
__device__ __forceinline__ double2 cdot(double2 u, double2 v)
{
	return make_double2(fma(u.x, v.x, u.y * v.y), fma(u.x, v.y, -(u.y * v.x)));
}

// deterministic block sum (fixed shuffle tree, then warp 0 over the warp sums); valid in thread 0
__device__ double2 block_sum(double2 v, double2* sm)
{
	for (int o = 16; o; o >>= 1) {
		v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
		v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
	}
	const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
	__syncthreads();
	if (l == 0) sm[w] = v;
	__syncthreads();
	double2 r = make_double2(0.0, 0.0);
	if (w == 0) {
		r = l < nw ? sm[l] : make_double2(0.0, 0.0);
		for (int o = 16; o; o >>= 1) {
			r.x += __shfl_xor_sync(0xffffffffu, r.x, o);
			r.y += __shfl_xor_sync(0xffffffffu, r.y, o);
		}
	}
	return r;
}

// after thread 0 wrote this block's partial: true in every thread of the block that
// arrives last among the instance's nb blocks (threadFenceReduction pattern)
__device__ bool arrive_last(unsigned* cnt, int nb)
{
	__shared__ bool last;
	if (threadIdx.x == 0) {
		__threadfence();
		unsigned t = atomicAdd(cnt, 1u);
		last = (t == (unsigned)nb - 1u);
	}
	__syncthreads();
	return last;
}

// ---------------------------------------------------------------- layout
__global__ void k_ar_to_rmajor(const double2* __restrict__ src, double2* __restrict__ dst, int N, int nch, long total)
{
	long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= total) return;
	long n = (long)N * nch, b = i / n, e = i - b * n;
	int r = (int)(e / nch), ch = (int)(e - (long)r * nch);
	dst[i] = src[b * n + (long)ch * N + r];
}
__global__ void k_ar_to_lmajor(const double2* __restrict__ src, double2* __restrict__ dst, int N, int nch, long total)
{
	long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= total) return;
	long n = (long)N * nch, b = i / n, e = i - b * n;
	int ch = (int)(e / N), r = (int)(e - (long)ch * N);
	dst[i] = src[b * n + (long)r * nch + ch];
}

// ---------------------------------------------------------------- S-norm and breakdown test
// Re sum_e conj(x_e) (S x)_e per instance (operator_rsym::observe, operators/1e.hpp:69-79).
// k < 0: start of a step (construct_sub, la_1e.hpp:132-151): sfac = 1/|w|_S, b[0] = |w|_S,
//        or the instance idles this step (step >= nt).
// k >= 0: end of iteration k (orthogonalize_ip, la_1e.hpp:221-238): nu < 1e-13 ends the
//        expansion with m = k+1; else sfac = 1/sqrt(nu), b[k+1] = sqrt(nu).
template <int PT>
__global__ void __launch_bounds__(AR_THREADS) k_ar_snorm(ar_args g, const double2* __restrict__ src, int k, long step)
{
	const int b = g.b0 + blockIdx.y;
	if (k < 0) {
		if (step >= g.nt[b]) {
			if (blockIdx.x == 0 && threadIdx.x == 0) g.flag[b] = AR_IDLE;
			return;
		}
	} else if (g.flag[b] != AR_LIVE) return;
	__shared__ double2 sm[32];
	const int P = g.P, nch = g.nch, N = g.N;
	const double2* x = src + (long)b * g.n;
	double acc = 0.0;
	for (int j = 0; j < PT; ++j) {
		long e = (long)blockIdx.x * (AR_THREADS * PT) + j * AR_THREADS + threadIdx.x;
		if (e >= g.n) break;
		int r = (int)(e / nch);
		double2 t = make_double2(0.0, 0.0);
		for (int q = 1; q <= P && q <= r; ++q) {
			double s = g.S[(long)(r - q) * (P + 1) + q];
			double2 v = x[e - (long)q * nch];
			t.x = fma(s, v.x, t.x); t.y = fma(s, v.y, t.y);
		}
		for (int q = 0; q <= P && r + q < N; ++q) {
			double s = g.S[(long)r * (P + 1) + q];
			double2 v = x[e + (long)q * nch];
			t.x = fma(s, v.x, t.x); t.y = fma(s, v.y, t.y);
		}
		double2 c = x[e];
		acc = fma(c.x, t.x, fma(c.y, t.y, acc));
	}
	double2 tot = block_sum(make_double2(acc, 0.0), sm);
	if (threadIdx.x == 0) g.partN[(long)b * g.nbe + blockIdx.x] = tot.x;
	if (!arrive_last(g.cnt + b, g.nbe)) return;
	if (threadIdx.x < 32) {
		double s = 0.0;
		for (int j = threadIdx.x; j < g.nbe; j += 32) s += __ldcg(g.partN + (long)b * g.nbe + j);
		for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
		if (threadIdx.x == 0) {
			g.cnt[b] = 0u;
			const long bb = (long)b * (g.kmax + 1);
			if (k < 0) {
				g.nu0[b] = s;
				if (!(s > 0.0) || !isfinite(s)) {
					atomicOr(g.status, ARS_ZERO);
					g.flag[b] = AR_IDLE;
				} else {
					double nrm = sqrt(s);
					g.sfac[b] = 1.0 / nrm;
					g.b[bb] = nrm;
					g.flag[b] = AR_LIVE;
					g.msub[b] = g.kmax;
				}
			} else if (s < 1e-13) {
				g.b[bb + k + 1] = 0.0;
				g.flag[b] = AR_BROKEN;
				g.msub[b] = k + 1;
			} else {
				double nrm = sqrt(s);
				g.sfac[b] = 1.0 / nrm;
				g.b[bb + k + 1] = nrm;
			}
		}
	}
}

// ---------------------------------------------------------------- expansion
// u_k = sfac * src (stored as U[k]); dst = H u_k (multiply, la_1e.hpp:420-434:
// symb_mul_vecd of H_l, then + (R u_{l-1}) ez y10(m,l-1), + (R u_{l+1}) ez y10(m,l));
// x_i = <u_i|dst> for i <= k (orthogonalize_ip, la_1e.hpp:204-209), a[k] = Re x_k.
// The band sums run on the unscaled src and are scaled once, H (s x) = s (H x): the
// same value to rounding, for a third of the FP64 instructions.
template <int PT>
__global__ void __launch_bounds__(AR_THREADS) k_ar_expand(ar_args g, const double2* __restrict__ src, double2* __restrict__ dst,
	int k, long step)
{
	const int b = g.b0 + blockIdx.y;
	if (g.flag[b] != AR_LIVE) return;
	const int P = g.P, nch = g.nch, N = g.N, L = g.L;
	const long n = g.n;
	const double s = g.sfac[b];
	const double ez = g.ez[(long)b * g.ld + step];
	const double2* __restrict__ x = src + (long)b * n;
	double2* y = dst + (long)b * n;
	double2* Uk = g.U + ((long)b * g.kmax + k) * n;
	const double* __restrict__ H = g.H + (long)b * g.hstride;
	const double* __restrict__ Rb = g.R;
	double2 yv[PT], uv[PT];
#pragma unroll
	for (int j = 0; j < PT; ++j) {
		yv[j] = uv[j] = make_double2(0.0, 0.0);
		long e = (long)blockIdx.x * (AR_THREADS * PT) + j * AR_THREADS + threadIdx.x;
		if (e >= n) continue;
		int r = (int)(e / nch), ch = (int)(e - (long)r * nch);
		int im = ch / L, il = ch - im * L;
		int l = il + abs(g.m0 + im);
		double2 ue = rmul(x[e], s);
		Uk[e] = ue;
		uv[j] = ue;
		// H_l band: lower neighbours q ascending, then the row itself and the upper ones
		double2 t = make_double2(0.0, 0.0);
		for (int q = 1; q <= P && q <= r; ++q) {
			double h = H[((long)(r - q) * (P + 1) + q) * g.nlh + l];
			double2 v = x[e - (long)q * nch];
			t.x = fma(v.x, h, t.x); t.y = fma(v.y, h, t.y);
		}
		for (int q = 0; q <= P && r + q < N; ++q) {
			double h = H[((long)r * (P + 1) + q) * g.nlh + l];
			double2 v = x[e + (long)q * nch];
			t.x = fma(v.x, h, t.x); t.y = fma(v.y, h, t.y);
		}
		// R band on the l-1 and l+1 channels of the same m
		double2 t2 = make_double2(0.0, 0.0), t3 = make_double2(0.0, 0.0);
		const bool lo = il > 0, hi = il < L - 1;
		for (int q = 1; q <= P && q <= r; ++q) {
			double rq = Rb[(long)(r - q) * (P + 1) + q];
			long o = e - (long)q * nch;
			if (lo) { double2 v = x[o - 1]; t2.x = fma(v.x, rq, t2.x); t2.y = fma(v.y, rq, t2.y); }
			if (hi) { double2 v = x[o + 1]; t3.x = fma(v.x, rq, t3.x); t3.y = fma(v.y, rq, t3.y); }
		}
		for (int q = 0; q <= P && r + q < N; ++q) {
			double rq = Rb[(long)r * (P + 1) + q];
			long o = e + (long)q * nch;
			if (lo) { double2 v = x[o - 1]; t2.x = fma(v.x, rq, t2.x); t2.y = fma(v.y, rq, t2.y); }
			if (hi) { double2 v = x[o + 1]; t3.x = fma(v.x, rq, t3.x); t3.y = fma(v.y, rq, t3.y); }
		}
		const double clo = lo ? ez * g.y10[im * L + il - 1] : 0.0;
		const double chi = hi ? ez * g.y10[im * L + il] : 0.0;
		double2 acc;
		acc.x = fma(t3.x, chi, fma(t2.x, clo, t.x)) * s;
		acc.y = fma(t3.y, chi, fma(t2.y, clo, t.y)) * s;
		y[e] = acc;
		yv[j] = acc;
	}
	// projections x_i = <u_i|v>, i <= k: eight at a time, every thread's part to shared memory, one warp per sum (a
	// block-wide sum each had two barriers and a shuffle tree of its own: 4.5 us per projection)
	constexpr int ND = 8;
	__shared__ double2 sp[ND][AR_THREADS + 1];
	double2* part = g.partX + ((long)b * g.nbe + blockIdx.x) * g.kmax;
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	for (int i0 = 0; i0 <= k; i0 += ND) {
		const int ni = min(ND, k + 1 - i0);
		for (int i = 0; i < ni; ++i) {
			const double2* Ui = g.U + ((long)b * g.kmax + i0 + i) * n;
			double2 acc = make_double2(0.0, 0.0);
#pragma unroll
			for (int j = 0; j < PT; ++j) {
				const long e = (long)blockIdx.x * (AR_THREADS * PT) + j * AR_THREADS + threadIdx.x;
				if (e >= n) break;
				acc = cadd(acc, cdot(i0 + i == k ? uv[j] : Ui[e], yv[j]));
			}
			sp[i][threadIdx.x] = acc;
		}
		__syncthreads();
		if (warp < ni) {
			double2 t = make_double2(0.0, 0.0);
#pragma unroll
			for (int j = 0; j < AR_THREADS / 32; ++j) t = cadd(t, sp[warp][j * 32 + lane]);
			for (int o = 16; o; o >>= 1) { t.x += __shfl_xor_sync(0xffffffffu, t.x, o); t.y += __shfl_xor_sync(0xffffffffu, t.y, o); }
			if (lane == 0) part[i0 + warp] = t;
		}
		__syncthreads();
	}
	// the barrier above orders the warps' partials before thread 0's fence
	if (!arrive_last(g.cnt + b, g.nbe)) return;
	for (int i = warp; i <= k; i += AR_THREADS / 32) {
		double2 t = make_double2(0.0, 0.0);
		const double2* q = g.partX + (long)b * g.nbe * g.kmax + i;
		for (int j = lane; j < g.nbe; j += 32) t = cadd(t, __ldcg(q + (long)j * g.kmax));
		for (int o = 16; o; o >>= 1) { t.x += __shfl_xor_sync(0xffffffffu, t.x, o); t.y += __shfl_xor_sync(0xffffffffu, t.y, o); }
		if (lane == 0) {
			g.xfin[(long)b * g.kmax + i] = t;
			if (i == k) g.a[(long)b * g.kmax + k] = t.x;
		}
	}
	if (threadIdx.x == 0) g.cnt[b] = 0u;
}

// ---------------------------------------------------------------- S^-1
// v = (L L^T)^-1 v per (m,l) channel: ltrb_inv_vecd then utrb_inv_vecd
// (utilities/blas2.hpp:421-433, 1006-1040), the per-channel solve of
// operator_sc::inverse_sub (operators/1e.hpp:1247-1251).  One lane per real
// recurrence (channel, real or imaginary part); the previous P values of each
// sweep stay in registers.  Lrow[r][j-1] = L(r, r-j), Lcol[r][k-1] = L(r+k, r)
// (zero outside the matrix), dinv[r] = 1/L(r,r).  The rows advance in tiles of
// SV_D: the next tile's values are loaded while the current one is solved, and
// the factor rows of the next tile are staged in shared memory by the block.
constexpr int SV_D = 8;

template <int P, bool FWD>
__device__ __forceinline__ void sinv_sweep(const ar_args& g, double* v, long stride, bool act,
	double (*Lt)[SV_D][P + 1])
{
	const int N = g.N;
	const double* __restrict__ Lf = FWD ? g.Lrow : g.Lcol;
	const int ntile = (N + SV_D - 1) / SV_D;
	auto row = [&](int t, int j) { return FWD ? t * SV_D + j : N - 1 - (t * SV_D + j); };
	auto stage = [&](int t, int buf) {
		for (int i = threadIdx.x; i < SV_D * (P + 1); i += blockDim.x) {
			int j = i / (P + 1), c = i - j * (P + 1);
			int r = row(t, j);
			double val = 0.0;
			if (t * SV_D + j < N) val = c < P ? Lf[(long)r * P + c] : g.dinv[r];
			Lt[buf][j][c] = val;
		}
	};
	double w[P];
#pragma unroll
	for (int j = 0; j < P; ++j) w[j] = 0.0;
	double cur[SV_D], nxt[SV_D];
#pragma unroll
	for (int j = 0; j < SV_D; ++j) cur[j] = (act && j < N) ? v[(long)row(0, j) * stride] : 0.0;
	stage(0, 0);
	__syncthreads();
	for (int t = 0; t < ntile; ++t) {
		const int buf = t & 1;
		if (t + 1 < ntile) {
#pragma unroll
			for (int j = 0; j < SV_D; ++j) nxt[j] = (act && (t + 1) * SV_D + j < N) ? v[(long)row(t + 1, j) * stride] : 0.0;
			stage(t + 1, buf ^ 1);
		}
#pragma unroll
		for (int j = 0; j < SV_D; ++j) {
			if (t * SV_D + j < N) {
				double x = cur[j];
#pragma unroll
				for (int q = 0; q < P; ++q) x = fma(-w[q], Lt[buf][j][q], x);
				x *= Lt[buf][j][P];
#pragma unroll
				for (int q = P - 1; q > 0; --q) w[q] = w[q - 1];
				w[0] = x;
				if (act) v[(long)row(t, j) * stride] = x;
			}
		}
		__syncthreads();
#pragma unroll
		for (int j = 0; j < SV_D; ++j) cur[j] = nxt[j];
	}
}

template <int P>
__global__ void __launch_bounds__(CH_THREADS) k_ar_sinv(ar_args g, double2* __restrict__ vbuf)
{
	const int b = g.b0 + blockIdx.y;
	if (g.flag[b] != AR_LIVE) return;
	__shared__ double Lt[2][SV_D][P + 1];
	const int c = blockIdx.x * CH_THREADS + threadIdx.x;
	const bool act = c < 2 * g.nch;
	const long stride = 2L * g.nch;
	double* v = reinterpret_cast<double*>(vbuf + (long)b * g.n) + (act ? c : 0);
	sinv_sweep<P, true>(g, v, stride, act, Lt);
	sinv_sweep<P, false>(g, v, stride, act, Lt);
}

// The same solve for batches too small to occupy the GPU one lane per recurrence: block substitution in blocks of
// P rows, P lanes per recurrence.  With L21(t) the factor's block left of the diagonal block L11(t),
//   a(t) = v(t) - M_t a(t-1),  M_t = L21(t) L11(t-1)^-1      y(t) = L11(t)^-1 a(t)
//   b(t) = y(t) - N_t b(t+1),  N_t = (L11(t+1)^-1 L21(t+1))^T    x(t) = L11(t)^-T b(t):
// only a and b are sequences, P rows per link of a few dependent FMAs, the rest is done by the whole block.  The sequences
// are cut into four segments, a warp each, started from zero; what a segment should have started from then adds
// Phi_t a(end of the segment before), Phi_t the product of -M (or -N) from the segment's start to t.
// The vector stays in shared memory in between.  Bound by the latency of the sequences (P FMAs of 64 cycles per P
// rows); measured at groups of 4 wavefunctions of 400 x 21: 38 us (68 with one segment, ~270 for one dependent chain
// of three FP64 instructions and two shuffles per row).
constexpr int SB_THREADS = 128;
constexpr int SB_SEG = SB_THREADS / 32;
constexpr size_t SB_SMEM = 200 * 1024;	// longest vectors it takes: 5 recurrences of 5 000 rows at p = 6
template <int P>
__global__ void __launch_bounds__(SB_THREADS) k_ar_sinv_blk(ar_args g, double2* __restrict__ vbuf)
{
	const int b = g.b0 + blockIdx.y;
	if (g.flag[b] != AR_LIVE) return;
	constexpr int CPW = 32 / P, PP = P * P;
	extern __shared__ double xs[];	// [CPW][nt P]
	__shared__ double carry[SB_SEG][CPW * P];	// what enters each segment
	const int N = g.N, nt = (N + P - 1) / P, np = nt * P;
	const long stride = 2L * g.nch;
	const int c0 = blockIdx.x * CPW, nc = min(CPW, 2 * g.nch - c0);
	double* v = reinterpret_cast<double*>(vbuf + (long)b * g.n) + c0;
	for (int i = threadIdx.x; i < np * CPW; i += SB_THREADS) {
		const int r = i / CPW, c = i - r * CPW;
		xs[c * np + r] = (r < N && c < nc) ? v[(long)r * stride + c] : 0.0;
	}
	__syncthreads();
	const int lane = threadIdx.x & 31, seg = threadIdx.x >> 5, cs = lane / P, j = lane - cs * P;
	const int sl = (nt + SB_SEG - 1) / SB_SEG;	// blocks of a segment
	auto sequence = [&](const double* __restrict__ C, const double* __restrict__ Phi, bool fwd) {
		const bool act = cs < CPW;
		const int ib = seg * sl, ie = min(nt, ib + sl);
		double* x = xs + (act ? cs : 0) * np;
		const int base = (act ? cs : 0) * P;
		auto blk = [&](int i) { return fwd ? i : nt - 1 - i; };
		// coefficients of the next D - 1 blocks on their way (a read from L2 takes two links)
		constexpr int D = 4;
		double cf[D][P], vl[D];
		auto fetch = [&](int i, double* c, double& w) {
#pragma unroll
			for (int k = 0; k < P; ++k) c[k] = (act && i < ie) ? __ldg(C + (long)blk(i) * PP + j * P + k) : 0.0;
			w = (act && i < ie) ? x[blk(i) * P + j] : 0.0;
		};
		double a = (act && ib < ie) ? x[blk(ib) * P + j] : 0.0;
#pragma unroll
		for (int d = 0; d < D - 1; ++d) fetch(ib + 1 + d, cf[d], vl[d]);
		for (int i0 = ib + 1; i0 < ie; i0 += D) {
#pragma unroll
			for (int d = 0; d < D; ++d) {
				const int i = i0 + d;
				if (i >= ie) break;
				fetch(i + D - 1, cf[(d + D - 1) % D], vl[(d + D - 1) % D]);
				double p = vl[d], q = 0.0;
#pragma unroll
				for (int k = 0; k < P; ++k) {
					const double ak = __shfl_sync(0xffffffffu, a, base + k);
					if (k & 1) q = fma(-cf[d][k], ak, q); else p = fma(-cf[d][k], ak, p);
				}
				a = p + q;
				if (act) x[blk(i) * P + j] = a;
			}
		}
		if (act) carry[seg][lane] = a;	// the segment's end; turned into what enters it
		__syncthreads();
		if (seg) return;
		double in = 0.0;
		for (int s = 0; s < SB_SEG; ++s) {
			const int e = min(nt, (s + 1) * sl) - 1;
			double out = act ? carry[s][lane] : 0.0;
#pragma unroll
			for (int k = 0; k < P; ++k) {
				const double ik = __shfl_sync(0xffffffffu, in, base + k);
				if (s && act && s * sl < nt) out = fma(__ldg(Phi + (long)blk(e) * PP + j * P + k), ik, out);
			}
			if (act) carry[s][lane] = in;
			in = out;
		}
	};
	auto blocks = [&](bool trans) {	// every block, with what entered its segment, times L11^-1 or its transpose
		const double* __restrict__ Phi = trans ? g.SB : g.SF;
		for (int i = threadIdx.x; i < nt * CPW; i += SB_THREADS) {
			const int t = i / CPW, c = i - t * CPW;
			double* x = xs + c * np + t * P;
			const double* Li = g.SI + (long)t * PP;
			double in[P], out[P];
#pragma unroll
			for (int k = 0; k < P; ++k) in[k] = x[k];
			const int s = (trans ? nt - 1 - t : t) / sl;
			if (s) {
#pragma unroll
				for (int k = 0; k < P; ++k)
#pragma unroll
					for (int q = 0; q < P; ++q) in[k] = fma(__ldg(Phi + (long)t * PP + k * P + q), carry[s][c * P + q], in[k]);
			}
#pragma unroll
			for (int r = 0; r < P; ++r) {
				double s = 0.0;
#pragma unroll
				for (int k = 0; k < P; ++k)
					if (trans ? k >= r : k <= r) s = fma(__ldg(Li + (trans ? k * P + r : r * P + k)), in[k], s);
				out[r] = s;
			}
#pragma unroll
			for (int k = 0; k < P; ++k) x[k] = out[k];
		}
	};
	sequence(g.SM, g.SF, true);
	__syncthreads();
	blocks(false);
	__syncthreads();
	sequence(g.SN, g.SB, false);
	__syncthreads();
	blocks(true);
	__syncthreads();
	for (int i = threadIdx.x; i < N * CPW; i += SB_THREADS) {
		const int r = i / CPW, c = i - r * CPW;
		if (c < nc) v[(long)r * stride + c] = xs[c * np + r];
	}
}

// The same solve with P lanes per real recurrence, column-oriented (for batches too small to occupy the GPU one lane
// per recurrence whose vectors are too long for the shared memory of k_ar_sinv_blk; bound by its dependent chain per
// row): lane j of a recurrence holds the pending sum
// of one of the next P rows; when row r is complete its owner's sum is broadcast, every lane
// computes x_r, and each lane adds L(row_j, r) x_r to its own row's sum.  Three FP64
// instructions per row instead of P + 1, on P times as many warps.
template <int P>
__global__ void __launch_bounds__(128) k_ar_sinv_sys(ar_args g, double2* __restrict__ vbuf)
{
	const int b = g.b0 + blockIdx.y;
	if (g.flag[b] != AR_LIVE) return;
	constexpr int CPW = 32 / P;
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const int cs = lane / P, j = lane - cs * P;
	const int c = (blockIdx.x * (int)(blockDim.x >> 5) + warp) * CPW + cs;
	const bool act = cs < CPW && c < 2 * g.nch;
	const int base = (cs < CPW ? cs : 0) * P;
	const long stride = 2L * g.nch;
	const int N = g.N;
	double* v = reinterpret_cast<double*>(vbuf + (long)b * g.n) + (act ? c : 0);
	const double* __restrict__ Lcol = g.Lcol;
	const double* __restrict__ Lrow = g.Lrow;
	const double* __restrict__ dinv = g.dinv;
	// forward: rows r ascending, owner o = r mod P
	{
		double acc = 0.0, cur[SV_D], nxt[SV_D];
		const int ntile = (N + SV_D - 1) / SV_D;
#pragma unroll
		for (int q = 0; q < SV_D; ++q) cur[q] = (act && q < N) ? v[(long)q * stride] : 0.0;
		int o = 0;
		for (int t = 0; t < ntile; ++t) {
#pragma unroll
			for (int q = 0; q < SV_D; ++q) {
				int r = (t + 1) * SV_D + q;
				nxt[q] = (act && r < N) ? v[(long)r * stride] : 0.0;
			}
#pragma unroll
			for (int q = 0; q < SV_D; ++q) {
				const int r = t * SV_D + q;
				if (r < N) {
					double ao = __shfl_sync(0xffffffffu, acc, base + o);
					double x = (cur[q] - ao) * dinv[r];
					if (j == o) acc = 0.0;
					int k = (j - o - 1 + P) % P + 1;
					acc = fma(Lcol[(long)r * P + k - 1], x, acc);
					if (act && j == o) v[(long)r * stride] = x;
					o = (o + 1 == P) ? 0 : o + 1;
				}
			}
#pragma unroll
			for (int q = 0; q < SV_D; ++q) cur[q] = nxt[q];
		}
	}
	__syncwarp();
	// backward: rows s = N-1-i descending, owner o = i mod P
	{
		double acc = 0.0, cur[SV_D], nxt[SV_D];
		const int ntile = (N + SV_D - 1) / SV_D;
#pragma unroll
		for (int q = 0; q < SV_D; ++q) cur[q] = (act && q < N) ? v[(long)(N - 1 - q) * stride] : 0.0;
		int o = 0;
		for (int t = 0; t < ntile; ++t) {
#pragma unroll
			for (int q = 0; q < SV_D; ++q) {
				int i = (t + 1) * SV_D + q;
				nxt[q] = (act && i < N) ? v[(long)(N - 1 - i) * stride] : 0.0;
			}
#pragma unroll
			for (int q = 0; q < SV_D; ++q) {
				const int i = t * SV_D + q;
				if (i < N) {
					const int sr = N - 1 - i;
					double ao = __shfl_sync(0xffffffffu, acc, base + o);
					double x = (cur[q] - ao) * dinv[sr];
					if (j == o) acc = 0.0;
					int k = (j - o - 1 + P) % P + 1;
					acc = fma(Lrow[(long)sr * P + k - 1], x, acc);
					if (act && j == o) v[(long)sr * stride] = x;
					o = (o + 1 == P) ? 0 : o + 1;
				}
			}
#pragma unroll
			for (int q = 0; q < SV_D; ++q) cur[q] = nxt[q];
		}
	}
}

// ---------------------------------------------------------------- Gram-Schmidt
// v -= u_i x_i for i <= k with i == k or |x_i|^2 > 4e-27, i ascending (la_1e.hpp:212-219)
template <int PT>
__global__ void __launch_bounds__(AR_THREADS) k_ar_orth(ar_args g, double2* __restrict__ vbuf, int k)
{
	const int b = g.b0 + blockIdx.y;
	if (g.flag[b] != AR_LIVE) return;
	__shared__ double2 xs[AR_KMAX];
	__shared__ int use[AR_KMAX];
	if (threadIdx.x <= k) {
		double2 xi = g.xfin[(long)b * g.kmax + threadIdx.x];
		xs[threadIdx.x] = xi;
		use[threadIdx.x] = ((int)threadIdx.x == k) || (xi.x * xi.x + xi.y * xi.y > 4e-27);
	}
	__syncthreads();
	const long n = g.n;
	double2* v = vbuf + (long)b * n;
	for (int j = 0; j < PT; ++j) {
		long e = (long)blockIdx.x * (AR_THREADS * PT) + j * AR_THREADS + threadIdx.x;
		if (e >= n) break;
		double2 t = v[e];
		for (int i = 0; i <= k; ++i)
			if (use[i]) t = csub(t, cmul(g.U[((long)b * g.kmax + i) * n + e], xs[i]));
		v[e] = t;
	}
}

// ---------------------------------------------------------------- Krylov-space propagation
// propagate_sub (la_1e.hpp:153-174) and criterion (la_1e.hpp:296-310), one warp per
// instance.  The m x m tridiagonal (a[0..m), b[1..m)) is diagonalised by the implicit
// QL iteration with Wilkinson shifts (Bowdler, Martin, Reinsch and Wilkinson, Numer.
// Math. 11 (1968) 293-306).  Every lane runs the same scalar recurrence on its own
// copy of (d, e); lane j applies the rotations to row j of the eigenvector matrix.
// Then x_j = b0 sum_i z_i[0] exp(-i dt d_i) z_i[j].
__global__ void __launch_bounds__(32) k_ar_small(ar_args g, long step)
{
	const int b = g.b0 + blockIdx.x, lane = threadIdx.x;
	const int fl = g.flag[b];
	if (fl == AR_IDLE) return;
	const int m = fl == AR_BROKEN ? g.msub[b] : g.kmax;
	double d[AR_KMAX], e[AR_KMAX], z[AR_KMAX];
	for (int i = 0; i < m; ++i) {
		d[i] = g.a[(long)b * g.kmax + i];
		e[i] = i + 1 < m ? g.b[(long)b * (g.kmax + 1) + i + 1] : 0.0;
		z[i] = (i == lane) ? 1.0 : 0.0;
	}
	// scaled by the largest entry, so that sums of squares neither overflow nor lose what matters
	double big = 0.0;
	for (int i = 0; i < m; ++i) big = fmax(big, fmax(fabs(d[i]), fabs(e[i])));
	const double up = big > 0.0 ? big : 1.0, down = 1.0 / up;
	for (int i = 0; i < m; ++i) { d[i] *= down; e[i] *= down; }
	bool ok = true;
	for (int l = 0; l < m && ok; ++l) {
		int iter = 0, mm;
		for (;;) {
			for (mm = l; mm < m - 1; ++mm) {
				double dd = fabs(d[mm]) + fabs(d[mm + 1]);
				if (fabs(e[mm]) <= 1e-300 || fabs(e[mm]) + dd == dd) break;
			}
			if (mm == l) break;
			if (iter++ == 60) { ok = false; break; }
			double gg = (d[l + 1] - d[l]) / (2.0 * e[l]);
			double r = sqrt(fma(gg, gg, 1.0));
			gg = d[mm] - d[l] + e[l] / (gg + (gg >= 0 ? r : -r));
			double s = 1.0, c = 1.0, pp = 0.0;
			int i;
			bool underflow = false;
			for (i = mm - 1; i >= l; --i) {
				double f = s * e[i], bb = c * e[i];
				// one reciprocal root in place of a hypot and two divisions (m = 12: 325 -> 210 us)
				const double rr = fma(f, f, gg * gg), ri = rsqrt(rr);
				r = rr * ri;
				if (!(rr > 0.0)) r = 0.0;
				e[i + 1] = r;
				if (r == 0.0) {
					d[i + 1] -= pp;
					e[mm] = 0.0;
					underflow = true;
					break;
				}
				s = f * ri;
				c = gg * ri;
				gg = d[i + 1] - pp;
				r = (d[i] - gg) * s + 2.0 * c * bb;
				pp = s * r;
				d[i + 1] = gg + pp;
				gg = c * r - bb;
				double zf = z[i + 1];
				z[i + 1] = s * z[i] + c * zf;
				z[i] = c * z[i] - s * zf;
			}
			if (underflow) continue;
			d[l] -= pp;
			e[l] = gg;
			e[mm] = 0.0;
		}
	}
	if (!ok) {
		if (lane == 0) atomicOr(g.status, ARS_NOCONV);
		return;
	}
	// lane j holds z[i] = component j of eigenvector i
	const double b0 = g.b[(long)b * (g.kmax + 1)];
	double2 xj = make_double2(0.0, 0.0);
	for (int i = 0; i < m; ++i) {
		double z0 = __shfl_sync(0xffffffffu, z[i], 0);
		double sn, cs;
		sincos(-(g.dt * (d[i] * up)), &sn, &cs);
		double2 wi = make_double2(z0 * cs, z0 * sn);
		xj = i == 0 ? rmul(wi, z[i]) : cadd(xj, rmul(wi, z[i]));
	}
	xj = rmul(xj, b0);
	if (lane < m) g.xc[(long)b * g.kmax + lane] = xj;
	double2 xl = make_double2(__shfl_sync(0xffffffffu, xj.x, m - 1), __shfl_sync(0xffffffffu, xj.y, m - 1));
	if (lane == 0 && step < g.ld) {
		double eps = m > 1 ? xl.x * xl.x + xl.y * xl.y : 0.0;
		if (g.crit) g.crit[(long)b * g.ld + step] = (int8_t)(eps > g.emax ? 0 : eps > g.emin ? 1 : 2);
		if (g.msub_out) g.msub_out[(long)b * g.ld + step] = (int8_t)m;
	}
}

// w = sum_{i<m} u_i x_i (eliminate_sub, la_1e.hpp:176-193)
template <int PT>
__global__ void __launch_bounds__(AR_THREADS) k_ar_combine(ar_args g)
{
	const int b = g.b0 + blockIdx.y;
	const int fl = g.flag[b];
	if (fl == AR_IDLE) return;
	const int m = fl == AR_BROKEN ? g.msub[b] : g.kmax;
	__shared__ double2 xs[AR_KMAX];
	if (threadIdx.x < m) xs[threadIdx.x] = g.xc[(long)b * g.kmax + threadIdx.x];
	__syncthreads();
	const long n = g.n;
	bool bad = false;
	for (int j = 0; j < PT; ++j) {
		long e = (long)blockIdx.x * (AR_THREADS * PT) + j * AR_THREADS + threadIdx.x;
		if (e >= n) break;
		const double2* U = g.U + (long)b * g.kmax * n + e;
		double2 w = cmul(U[0], xs[0]);
		for (int i = 1; i < m; ++i) w = cadd(w, cmul(U[(long)i * n], xs[i]));
		g.X[(long)b * n + e] = w;
		bad |= !isfinite(w.x) || !isfinite(w.y);
	}
	if (bad) atomicOr(g.status, ARS_NONFINITE);
}

} // namespace

} // namespace qpc

using namespace qpc;

struct qpc_arnoldi {
	int dev = 0;
	qpc_dims d{};
	int P = 0, nch = 0, nlh = 0, kmax = 0, nbe = 0, hper = 0, pt = 4;
	long n = 0;
	double dt = 0, emin = 0, emax = 0;
	cudaStream_t stream = nullptr, stream2 = nullptr;	// stream2: second instance group (n_inst >= 2)
	cudaEvent_t ev0 = nullptr, ev1 = nullptr, ev2 = nullptr;
	double *S = nullptr, *R = nullptr, *Lrow = nullptr, *Lcol = nullptr, *SM = nullptr, *SN = nullptr, *SI = nullptr, *SF = nullptr, *SB = nullptr, *dinv = nullptr, *H = nullptr, *y10 = nullptr;
	double2 *X = nullptr, *U = nullptr, *V0 = nullptr, *V1 = nullptr, *tmp = nullptr;
	double2* partX = nullptr;
	double* partN = nullptr;
	unsigned* cnt = nullptr;
	double2 *xfin = nullptr, *xc = nullptr;
	double *a = nullptr, *b = nullptr, *sfac = nullptr, *nu0 = nullptr;
	int *msub = nullptr, *flag = nullptr, *status = nullptr;
	double* ez = nullptr;
	long ez_cap = 0;
	long long* nt = nullptr;
	int8_t *crit = nullptr, *msub_out = nullptr;
	long crit_cap = 0;
	float last_ms = 0.f;
	long launches = 0;
};

namespace {

void ar_free(qpc_arnoldi* h)
{
	if (!h) return;
	cudaSetDevice(h->dev);
	void* ptrs[] = {h->S, h->R, h->Lrow, h->Lcol, h->SM, h->SN, h->SI, h->SF, h->SB, h->dinv, h->H, h->y10, h->X, h->U, h->V0, h->V1, h->tmp, h->partX, h->partN,
		h->cnt, h->xfin, h->xc, h->a, h->b, h->sfac, h->nu0, h->msub, h->flag, h->status, h->ez, h->nt, h->crit, h->msub_out};
	for (void* p : ptrs)
		if (p) cudaFree(p);
	if (h->ev0) cudaEventDestroy(h->ev0);
	if (h->ev1) cudaEventDestroy(h->ev1);
	if (h->ev2) cudaEventDestroy(h->ev2);
	if (h->stream) cudaStreamDestroy(h->stream);
	if (h->stream2) cudaStreamDestroy(h->stream2);
	delete h;
}

ar_args make_args(qpc_arnoldi* h)
{
	ar_args g{};
	g.N = h->d.n_r; g.P = h->P; g.L = h->d.n_l; g.M = h->d.n_m; g.m0 = h->d.m0; g.nch = h->nch; g.nlh = h->nlh;
	g.B = h->d.n_inst; g.kmax = h->kmax; g.nbe = h->nbe; g.n = h->n; g.b0 = 0;
	g.hstride = h->hper ? (long)h->d.n_r * (h->P + 1) * h->nlh : 0;
	g.dt = h->dt; g.emin = h->emin; g.emax = h->emax;
	g.S = h->S; g.R = h->R; g.Lrow = h->Lrow; g.Lcol = h->Lcol; g.SM = h->SM; g.SN = h->SN; g.SI = h->SI; g.SF = h->SF; g.SB = h->SB; g.dinv = h->dinv; g.H = h->H; g.y10 = h->y10;
	g.X = h->X; g.U = h->U; g.V0 = h->V0; g.V1 = h->V1;
	g.partX = h->partX; g.partN = h->partN; g.cnt = h->cnt; g.xfin = h->xfin;
	g.a = h->a; g.b = h->b; g.sfac = h->sfac; g.nu0 = h->nu0; g.msub = h->msub; g.flag = h->flag; g.xc = h->xc;
	g.ez = h->ez; g.nt = h->nt; g.crit = h->crit; g.msub_out = h->msub_out; g.status = h->status;
	return g;
}

void launch_sinv(const ar_args& g, int Bg, double2* v, cudaStream_t st)
{
	// one lane per recurrence when that fills the GPU, else block substitution, or P lanes per recurrence where its vectors
	// do not fit the shared memory (four steps of 8 vectors, one lane / P lanes: 8000 x 21, p = 6, two wavefunctions 167 / 112 ms;
	// 3000 x 21, p = 3 41 / 40; 1603 x 21, p = 2 20 / 23, so not there)
	const long chains = 2L * g.nch * Bg;
	const char* e = getenv("QPC_AR_SINV");
	const bool blk = e ? atoi(e) == 2 : chains < 32L * 304;
	if (blk && g.P >= 2) {
		const int cpw = 32 / g.P;
		const size_t smem = sizeof(double) * cpw * ((g.N + g.P - 1) / g.P) * g.P;
		if (smem <= SB_SMEM) {
			const dim3 gs((unsigned)((2 * g.nch + cpw - 1) / cpw), Bg);
			switch (g.P) {
			case 2: k_ar_sinv_blk<2><<<gs, SB_THREADS, smem, st>>>(g, v); return;
			case 3: k_ar_sinv_blk<3><<<gs, SB_THREADS, smem, st>>>(g, v); return;
			case 4: k_ar_sinv_blk<4><<<gs, SB_THREADS, smem, st>>>(g, v); return;
			case 5: k_ar_sinv_blk<5><<<gs, SB_THREADS, smem, st>>>(g, v); return;
			case 6: k_ar_sinv_blk<6><<<gs, SB_THREADS, smem, st>>>(g, v); return;
			case 7: k_ar_sinv_blk<7><<<gs, SB_THREADS, smem, st>>>(g, v); return;
			default: k_ar_sinv_blk<8><<<gs, SB_THREADS, smem, st>>>(g, v); return;
			}
		}
		const dim3 gs((unsigned)((2 * g.nch + 4 * cpw - 1) / (4 * cpw)), Bg);
		switch (g.P) {
		case 2: break;
		case 3: k_ar_sinv_sys<3><<<gs, 128, 0, st>>>(g, v); return;
		case 4: k_ar_sinv_sys<4><<<gs, 128, 0, st>>>(g, v); return;
		case 5: k_ar_sinv_sys<5><<<gs, 128, 0, st>>>(g, v); return;
		case 6: k_ar_sinv_sys<6><<<gs, 128, 0, st>>>(g, v); return;
		case 7: k_ar_sinv_sys<7><<<gs, 128, 0, st>>>(g, v); return;
		default: k_ar_sinv_sys<8><<<gs, 128, 0, st>>>(g, v); return;
		}
	}
	dim3 grid((2 * g.nch + CH_THREADS - 1) / CH_THREADS, Bg);
	switch (g.P) {
	case 1: k_ar_sinv<1><<<grid, CH_THREADS, 0, st>>>(g, v); break;
	case 2: k_ar_sinv<2><<<grid, CH_THREADS, 0, st>>>(g, v); break;
	case 3: k_ar_sinv<3><<<grid, CH_THREADS, 0, st>>>(g, v); break;
	case 4: k_ar_sinv<4><<<grid, CH_THREADS, 0, st>>>(g, v); break;
	case 5: k_ar_sinv<5><<<grid, CH_THREADS, 0, st>>>(g, v); break;
	case 6: k_ar_sinv<6><<<grid, CH_THREADS, 0, st>>>(g, v); break;
	case 7: k_ar_sinv<7><<<grid, CH_THREADS, 0, st>>>(g, v); break;
	default: k_ar_sinv<8><<<grid, CH_THREADS, 0, st>>>(g, v); break;
	}
}

// one Arnoldi step of instances [g.b0, g.b0 + Bg) on stream st: 4 kmax launches
template <int PT>
long launch_step_t(qpc_arnoldi* h, const ar_args& g, int Bg, cudaStream_t st, long step)
{
	dim3 ge(g.nbe, Bg);
	long nl = 0;
	k_ar_snorm<PT><<<ge, AR_THREADS, 0, st>>>(g, h->X, -1, step); ++nl;
	double2* src = h->X;
	for (int k = 0; k < g.kmax; ++k) {
		double2* dst = (k & 1) ? h->V1 : h->V0;
		k_ar_expand<PT><<<ge, AR_THREADS, 0, st>>>(g, src, dst, k, step); ++nl;
		if (k == g.kmax - 1) break; // u_kmax is never used (eliminate_sub sums i < m)
		launch_sinv(g, Bg, dst, st); ++nl;
		k_ar_orth<PT><<<ge, AR_THREADS, 0, st>>>(g, dst, k); ++nl;
		k_ar_snorm<PT><<<ge, AR_THREADS, 0, st>>>(g, dst, k, step); ++nl;
		src = dst;
	}
	k_ar_small<<<Bg, 32, 0, st>>>(g, step); ++nl;
	k_ar_combine<PT><<<ge, AR_THREADS, 0, st>>>(g); ++nl;
	return nl;
}

long launch_step(qpc_arnoldi* h, const ar_args& g, int Bg, cudaStream_t st, long step)
{
	return h->pt == 1 ? launch_step_t<1>(h, g, Bg, st, step) : launch_step_t<4>(h, g, Bg, st, step);
}

int read_status(qpc_arnoldi* h)
{
	int st = 0;
	if (int rc = copy_to_host(&st, h->status, sizeof(int), h->stream)) return rc;
	QPC_CUDA(cudaMemsetAsync(h->status, 0, sizeof(int), h->stream));
	if (int rc = wait_on(h->stream)) return rc;
	if (st & ARS_ZERO) { set_error("a wavefunction has zero or non-finite S-norm"); return QPC_ERR_NUMERIC; }
	if (st & ARS_NOCONV) { set_error("Krylov-space eigenproblem did not converge"); return QPC_ERR_NUMERIC; }
	if (st & ARS_NONFINITE) { set_error("non-finite value in the state"); return QPC_ERR_NUMERIC; }
	return QPC_OK;
}

} // namespace

extern "C" {

int qpc_arnoldi_create(const qpc_dims* dims, const double* S, const double* R, const double* H, int32_t h_per_instance,
	const double* y10, double dt, int32_t kmax, double emin, double emax, qpc_arnoldi** out)
{
	if (!out) { set_error("out is NULL"); return QPC_ERR_ARGS; }
	*out = nullptr;
	if (!dims || !S || !R || !H || !y10) { set_error("NULL argument"); return QPC_ERR_ARGS; }
	const qpc_dims d = *dims;
	if (d.p < 1 || d.p > QPC_MAX_RANK || d.n_r < 2 * d.p + 2 || d.n_l < 1 || d.n_m < 1 || d.n_inst < 1 || d.n_inst > 65535) {
		set_error("bad dims n_r=%d p=%d n_l=%d n_m=%d n_inst=%d", d.n_r, d.p, d.n_l, d.n_m, d.n_inst);
		return QPC_ERR_ARGS;
	}
	if (kmax < 1 || kmax > AR_KMAX) { set_error("kmax=%d outside [1, %d]", kmax, AR_KMAX); return QPC_ERR_ARGS; }
	// arnoldi_workspace's constructor check (la_1e.hpp:58-61)
	if (!(emin <= emax) || !(emin > 0) || !(emax > 0)) { set_error("invalid parameters for arnoldi propagator (emin=%g emax=%g)", emin, emax); return QPC_ERR_ARGS; }
	if (!(dt > 0) || !std::isfinite(dt)) { set_error("dt=%g", dt); return QPC_ERR_ARGS; }
	int dev = 0;
	if (int rc = check_device(&dev)) return rc;
	qpc_arnoldi* h = new (std::nothrow) qpc_arnoldi;
	if (!h) { set_error("host allocation"); return QPC_ERR_NOMEM; }
	auto fail = [&](int rc) { ar_free(h); return rc; };
	h->dev = dev;
	h->d = d;
	h->P = d.p;
	h->nch = d.n_m * d.n_l;
	const int mmax = std::max(std::abs(d.m0), std::abs(d.m0 + d.n_m - 1));
	h->nlh = mmax + d.n_l;
	h->kmax = kmax;
	h->n = (long)h->nch * d.n_r;
	h->pt = h->n * d.n_inst < 4L * AR_THREADS * 608 ? 1 : 4;
	h->nbe = (int)((h->n + AR_THREADS * h->pt - 1) / (AR_THREADS * h->pt));
	h->hper = h_per_instance ? 1 : 0;
	h->dt = dt; h->emin = emin; h->emax = emax;
	const int N = d.n_r, P = d.p, NE = P + 1, B = d.n_inst;
	// Cholesky factor of S in both sweep orders
	std::vector<double> Lc((size_t)N * NE);
	int bad = qpc_cholesky_band(N, P, S, Lc.data());
	if (bad) { set_error("S is not positive definite (pivot %d)", bad); return fail(QPC_ERR_SINGULAR); }
	std::vector<double> lrow((size_t)N * P, 0.0), lcol((size_t)N * P, 0.0), di(N);
	for (int r = 0; r < N; ++r) {
		di[r] = 1.0 / Lc[(size_t)r * NE];
		for (int j = 1; j <= P; ++j) {
			if (r - j >= 0) lrow[(size_t)r * P + j - 1] = Lc[(size_t)(r - j) * NE + j];
			if (r + j < N) lcol[(size_t)r * P + j - 1] = Lc[(size_t)r * NE + j];
		}
	}
	// the tables of the block substitution, blocks of P rows (rows past the last: the identity)
	const int nt = (N + P - 1) / P;
	auto Lat = [&](int r, int c) -> double {	// L(r, c)
		if (r >= N || c >= N) return r == c ? 1.0 : 0.0;
		return (c > r || r - c > P) ? 0.0 : Lc[(size_t)c * NE + (r - c)];
	};
	std::vector<double> sM((size_t)nt * P * P, 0.0), sN((size_t)nt * P * P, 0.0), sI((size_t)nt * P * P, 0.0);
	for (int t = 0; t < nt; ++t) {
		double* I = sI.data() + (size_t)t * P * P;
		for (int c = 0; c < P; ++c)
			for (int r = c; r < P; ++r) {
				double x = r == c ? 1.0 : 0.0;
				for (int k = c; k < r; ++k) x -= Lat(t * P + r, t * P + k) * I[k * P + c];
				I[r * P + c] = x / Lat(t * P + r, t * P + r);
			}
	}
	for (int t = 1; t < nt; ++t)
		for (int r = 0; r < P; ++r)
			for (int c = 0; c < P; ++c) {
				const double *Ip = sI.data() + (size_t)(t - 1) * P * P, *It = sI.data() + (size_t)t * P * P;
				double x = 0.0, y = 0.0;
				for (int k = 0; k < P; ++k) {
					x += Lat(t * P + r, (t - 1) * P + k) * Ip[k * P + c];
					y += It[r * P + k] * Lat(t * P + k, (t - 1) * P + c);
				}
				sM[((size_t)t * P + r) * P + c] = x;
				sN[((size_t)(t - 1) * P + c) * P + r] = y;
			}
	// Phi of the segments (zero in the first, where nothing enters)
	std::vector<double> sF((size_t)nt * P * P, 0.0), sB((size_t)nt * P * P, 0.0);
	const int sl = (nt + SB_SEG - 1) / SB_SEG;
	for (int back = 0; back < 2; ++back)
		for (int i = sl; i < nt; ++i) {
			const int t = back ? nt - 1 - i : i, prev = back ? t + 1 : t - 1;
			const double* C = (back ? sN : sM).data() + (size_t)t * P * P;
			double* F = (back ? sB : sF).data();
			for (int r = 0; r < P; ++r)
				for (int c = 0; c < P; ++c) {
					double x = 0.0;
					if (i % sl == 0) x = -C[r * P + c];
					else for (int k = 0; k < P; ++k) x -= C[r * P + k] * F[((size_t)prev * P + k) * P + c];
					F[((size_t)t * P + r) * P + c] = x;
				}
		}
	// Hamiltonian bands r-major: Hr[hs][r][k][l]
	const int nhs = h->hper ? B : 1;
	std::vector<double> Hr((size_t)nhs * N * NE * h->nlh);
	for (int hs = 0; hs < nhs; ++hs)
		for (int l = 0; l < h->nlh; ++l)
			for (int r = 0; r < N; ++r)
				for (int k = 0; k < NE; ++k) {
					double v = H[(((size_t)hs * h->nlh + l) * N + r) * NE + k];
					if (!std::isfinite(v)) { set_error("non-finite H"); return fail(QPC_ERR_ARGS); }
					Hr[(((size_t)hs * N + r) * NE + k) * h->nlh + l] = v;
				}
	int rc = 0;
	if ((cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking)) != cudaSuccess) { set_error("cudaStreamCreateWithFlags failed"); return fail(QPC_ERR_CUDA); }
	if ((cudaEventCreate(&h->ev0)) != cudaSuccess) { set_error("cudaEventCreate failed"); return fail(QPC_ERR_CUDA); }
	if ((cudaEventCreate(&h->ev1)) != cudaSuccess) { set_error("cudaEventCreate failed"); return fail(QPC_ERR_CUDA); }
	if ((cudaEventCreateWithFlags(&h->ev2, cudaEventDisableTiming)) != cudaSuccess) { set_error("cudaEventCreateWithFlags failed"); return fail(QPC_ERR_CUDA); }
	if (B >= 2 && !(getenv("QPC_STREAMS") && atoi(getenv("QPC_STREAMS")) == 1))
		if ((cudaStreamCreateWithFlags(&h->stream2, cudaStreamNonBlocking)) != cudaSuccess) { set_error("cudaStreamCreateWithFlags failed"); return fail(QPC_ERR_CUDA); }
	const long nst = (long)B * h->n;
	if ((rc = dalloc(&h->S, (size_t)N * NE)) || (rc = dalloc(&h->R, (size_t)N * NE)) || (rc = dalloc(&h->Lrow, (size_t)N * P)) ||
		(rc = dalloc(&h->Lcol, (size_t)N * P)) || (rc = dalloc(&h->SM, sM.size())) || (rc = dalloc(&h->SN, sN.size())) || (rc = dalloc(&h->SI, sI.size())) || (rc = dalloc(&h->SF, sF.size())) || (rc = dalloc(&h->SB, sB.size())) || (rc = dalloc(&h->dinv, (size_t)N)) || (rc = dalloc(&h->H, Hr.size())) ||
		(rc = dalloc(&h->y10, (size_t)d.n_m * d.n_l)) || (rc = dalloc(&h->X, nst)) || (rc = dalloc(&h->U, nst * kmax)) ||
		(rc = dalloc(&h->V0, nst)) || (rc = dalloc(&h->V1, nst)) || (rc = dalloc(&h->tmp, nst)) ||
		(rc = dalloc(&h->partX, (size_t)B * h->nbe * kmax)) || (rc = dalloc(&h->partN, (size_t)B * h->nbe)) ||
		(rc = dalloc(&h->cnt, (size_t)B)) || (rc = dalloc(&h->xfin, (size_t)B * kmax)) || (rc = dalloc(&h->xc, (size_t)B * kmax)) ||
		(rc = dalloc(&h->a, (size_t)B * kmax)) || (rc = dalloc(&h->b, (size_t)B * (kmax + 1))) || (rc = dalloc(&h->sfac, (size_t)B)) || (rc = dalloc(&h->nu0, (size_t)B)) ||
		(rc = dalloc(&h->msub, (size_t)B)) || (rc = dalloc(&h->flag, (size_t)B)) || (rc = dalloc(&h->status, 1)) ||
		(rc = dalloc(&h->nt, (size_t)B)))
		return fail(rc);
	if (cudaMemcpyAsync(h->S, S, sizeof(double) * N * NE, cudaMemcpyHostToDevice, h->stream) != cudaSuccess ||
		cudaMemcpyAsync(h->R, R, sizeof(double) * N * NE, cudaMemcpyHostToDevice, h->stream) != cudaSuccess ||
		cudaMemcpyAsync(h->Lrow, lrow.data(), sizeof(double) * lrow.size(), cudaMemcpyHostToDevice, h->stream) != cudaSuccess ||
		cudaMemcpyAsync(h->Lcol, lcol.data(), sizeof(double) * lcol.size(), cudaMemcpyHostToDevice, h->stream) != cudaSuccess ||
		cudaMemcpyAsync(h->SM, sM.data(), sizeof(double) * sM.size(), cudaMemcpyHostToDevice, h->stream) != cudaSuccess ||
		cudaMemcpyAsync(h->SN, sN.data(), sizeof(double) * sN.size(), cudaMemcpyHostToDevice, h->stream) != cudaSuccess ||
		cudaMemcpyAsync(h->SI, sI.data(), sizeof(double) * sI.size(), cudaMemcpyHostToDevice, h->stream) != cudaSuccess ||
		cudaMemcpyAsync(h->SF, sF.data(), sizeof(double) * sF.size(), cudaMemcpyHostToDevice, h->stream) != cudaSuccess ||
		cudaMemcpyAsync(h->SB, sB.data(), sizeof(double) * sB.size(), cudaMemcpyHostToDevice, h->stream) != cudaSuccess ||
		cudaMemcpyAsync(h->dinv, di.data(), sizeof(double) * N, cudaMemcpyHostToDevice, h->stream) != cudaSuccess ||
		cudaMemcpyAsync(h->H, Hr.data(), sizeof(double) * Hr.size(), cudaMemcpyHostToDevice, h->stream) != cudaSuccess ||
		cudaMemcpyAsync(h->y10, y10, sizeof(double) * d.n_m * d.n_l, cudaMemcpyHostToDevice, h->stream) != cudaSuccess ||
		cudaMemsetAsync(h->X, 0, sizeof(double2) * nst, h->stream) != cudaSuccess || cudaMemsetAsync(h->cnt, 0, sizeof(unsigned) * B, h->stream) != cudaSuccess ||
		cudaMemsetAsync(h->status, 0, sizeof(int), h->stream) != cudaSuccess) {
		set_error("device upload failed");
		return fail(QPC_ERR_CUDA);
	}
	auto attr = [](auto kern) { cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SB_SMEM); };
	attr(k_ar_sinv_blk<2>); attr(k_ar_sinv_blk<3>); attr(k_ar_sinv_blk<4>); attr(k_ar_sinv_blk<5>); attr(k_ar_sinv_blk<6>); attr(k_ar_sinv_blk<7>);
	attr(k_ar_sinv_blk<8>);
	if ((rc = wait_on(h->stream))) return fail(rc);
	*out = h;
	return QPC_OK;
}

int qpc_arnoldi_destroy(qpc_arnoldi* h)
{
	ar_free(h);
	return QPC_OK;
}

static int ar_transfer(qpc_arnoldi* h, const double* src, double* dst, bool put, cudaMemcpyKind kind)
{
	cudaSetDevice(h->dev);
	const long nst = (long)h->d.n_inst * h->n;
	const int tb = 256;
	const unsigned nb = (unsigned)((nst + tb - 1) / tb);
	// host buffers are copied with the stream idle (bounded wait first): such a copy then
	// never waits for queued work, and a wait that runs out leaves no copy pending
	if (put) {
		if (kind == cudaMemcpyHostToDevice) if (int rc = wait_on(h->stream)) return rc;
		QPC_CUDA(cudaMemcpyAsync(h->tmp, src, sizeof(double2) * nst, kind, h->stream));
		k_ar_to_rmajor<<<nb, tb, 0, h->stream>>>(h->tmp, h->X, h->d.n_r, h->nch, nst);
	} else {
		k_ar_to_lmajor<<<nb, tb, 0, h->stream>>>(h->X, h->tmp, h->d.n_r, h->nch, nst);
		QPC_CUDA(cudaGetLastError());
		if (kind == cudaMemcpyDeviceToHost) return copy_to_host(dst, h->tmp, sizeof(double2) * nst, h->stream);
		QPC_CUDA(cudaMemcpyAsync(dst, h->tmp, sizeof(double2) * nst, kind, h->stream));
	}
	QPC_CUDA(cudaGetLastError());
	return wait_on(h->stream);
}

int qpc_arnoldi_put(qpc_arnoldi* h, const double* coef)
{
	if (!h || !coef) { set_error("NULL argument"); return QPC_ERR_ARGS; }
	return ar_transfer(h, coef, nullptr, true, cudaMemcpyHostToDevice);
}

int qpc_arnoldi_get(qpc_arnoldi* h, double* coef)
{
	if (!h || !coef) { set_error("NULL argument"); return QPC_ERR_ARGS; }
	return ar_transfer(h, nullptr, coef, false, cudaMemcpyDeviceToHost);
}

int qpc_arnoldi_put_device(qpc_arnoldi* h, const double* dev_coef)
{
	if (!h || !dev_coef) { set_error("NULL argument"); return QPC_ERR_ARGS; }
	return ar_transfer(h, dev_coef, nullptr, true, cudaMemcpyDeviceToDevice);
}

int qpc_arnoldi_get_device(qpc_arnoldi* h, double* dev_coef)
{
	if (!h || !dev_coef) { set_error("NULL argument"); return QPC_ERR_ARGS; }
	return ar_transfer(h, nullptr, dev_coef, false, cudaMemcpyDeviceToDevice);
}

int qpc_arnoldi_run(qpc_arnoldi* h, const double* ez, int64_t ld, const int64_t* nt, int8_t* crit, int8_t* msub)
{
	if (!h || !ez || !nt) { set_error("NULL argument"); return QPC_ERR_ARGS; }
	cudaSetDevice(h->dev);
	const int B = h->d.n_inst;
	long ntmax = 0;
	for (int k = 0; k < B; ++k) {
		if (nt[k] < 0 || nt[k] > ld) { set_error("instance %d: nt=%lld outside [0, ld=%lld]", k, (long long)nt[k], (long long)ld); return QPC_ERR_ARGS; }
		for (long s = 0; s < nt[k]; ++s)
			if (!std::isfinite(ez[(size_t)k * ld + s])) { set_error("non-finite field value, instance %d step %ld", k, s); return QPC_ERR_ARGS; }
		ntmax = std::max<long>(ntmax, nt[k]);
	}
	if (ntmax == 0) return QPC_OK;
	const long cap = (long)B * ld;
	if (cap > h->ez_cap) {
		if (h->ez) cudaFree(h->ez);
		h->ez = nullptr; h->ez_cap = 0;
		if (int rc = dalloc(&h->ez, cap)) return rc;
		h->ez_cap = cap;
	}
	if ((crit || msub) && cap > h->crit_cap) {
		// (re)allocated below; filled with -1 for the steps an instance does not take
		if (h->crit) cudaFree(h->crit);
		if (h->msub_out) cudaFree(h->msub_out);
		h->crit = h->msub_out = nullptr; h->crit_cap = 0;
		if (int rc = dalloc(&h->crit, cap)) return rc;
		if (int rc = dalloc(&h->msub_out, cap)) return rc;
		h->crit_cap = cap;
	}
	std::vector<long long> ntl(nt, nt + B);
	if (int rc = wait_on(h->stream)) return rc;
	QPC_CUDA(cudaMemcpyAsync(h->ez, ez, sizeof(double) * cap, cudaMemcpyHostToDevice, h->stream));
	QPC_CUDA(cudaMemcpyAsync(h->nt, ntl.data(), sizeof(long long) * B, cudaMemcpyHostToDevice, h->stream));
	ar_args g = make_args(h);
	g.ld = ld;
	if (crit || msub) {
		QPC_CUDA(cudaMemsetAsync(h->crit, 0xff, cap, h->stream));
		QPC_CUDA(cudaMemsetAsync(h->msub_out, 0xff, cap, h->stream));
	} else g.crit = g.msub_out = nullptr;
	long nl = 0;
	// two instance groups on two streams: the latency-bound S^-1 sweeps of one group
	// overlap the band products of the other (instances never interact)
	const int ng = h->stream2 ? 2 : 1;
	int gb[3] = {0, ng == 2 ? (B + 1) / 2 : B, B};
	cudaStream_t gs[2] = {h->stream, h->stream2};
	QPC_CUDA(cudaEventRecord(h->ev0, h->stream));
	if (ng == 2) QPC_CUDA(cudaStreamWaitEvent(h->stream2, h->ev0, 0));
	for (long s = 0; s < ntmax; ++s)
		for (int q = 0; q < ng; ++q) {
			ar_args gq = g;
			gq.b0 = gb[q];
			nl += launch_step(h, gq, gb[q + 1] - gb[q], gs[q], s);
		}
	QPC_CUDA(cudaGetLastError());
	if (ng == 2) {
		QPC_CUDA(cudaEventRecord(h->ev2, h->stream2));
		QPC_CUDA(cudaStreamWaitEvent(h->stream, h->ev2, 0));
	}
	QPC_CUDA(cudaEventRecord(h->ev1, h->stream));
	if (int rc = wait_on(h->stream)) return rc;
	cudaEventElapsedTime(&h->last_ms, h->ev0, h->ev1);
	h->launches = nl;
	if (crit) if (int rc = copy_to_host(crit, h->crit, cap, h->stream)) return rc;
	if (msub) if (int rc = copy_to_host(msub, h->msub_out, cap, h->stream)) return rc;
	return read_status(h);
}

int qpc_arnoldi_propagate(qpc_arnoldi* h, const double* ez, int8_t* crit)
{
	if (!h || !ez) { set_error("NULL argument"); return QPC_ERR_ARGS; }
	std::vector<int64_t> ones(h->d.n_inst, 1);
	return qpc_arnoldi_run(h, ez, 1, ones.data(), crit, nullptr);
}

int qpc_arnoldi_norm(qpc_arnoldi* h, double* norm)
{
	if (!h || !norm) { set_error("NULL argument"); return QPC_ERR_ARGS; }
	cudaSetDevice(h->dev);
	const int B = h->d.n_inst;
	// one S-norm pass with every instance live at "step 0" of a one-step table
	std::vector<long long> one(B, 1);
	if (int rc = wait_on(h->stream)) return rc;
	QPC_CUDA(cudaMemcpyAsync(h->nt, one.data(), sizeof(long long) * B, cudaMemcpyHostToDevice, h->stream));
	ar_args g = make_args(h);
	if (h->pt == 1) k_ar_snorm<1><<<dim3(h->nbe, B), AR_THREADS, 0, h->stream>>>(g, h->X, -1, 0);
	else k_ar_snorm<4><<<dim3(h->nbe, B), AR_THREADS, 0, h->stream>>>(g, h->X, -1, 0);
	QPC_CUDA(cudaGetLastError());
	std::vector<double> nu(B);
	if (int rc = copy_to_host(nu.data(), h->nu0, sizeof(double) * B, h->stream)) return rc;
	QPC_CUDA(cudaMemsetAsync(h->status, 0, sizeof(int), h->stream));
	if (int rc = wait_on(h->stream)) return rc;
	for (int k = 0; k < B; ++k) norm[k] = nu[k];
	return QPC_OK;
}

int qpc_arnoldi_last_run(qpc_arnoldi* h, float* ms, int64_t* launches)
{
	if (!h || !ms || !launches) { set_error("NULL argument"); return QPC_ERR_ARGS; }
	*ms = h->last_ms;
	*launches = h->launches;
	return QPC_OK;
}

} // extern "C"
