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
// Both products run in fixed point (qpc_radial.cu), for batches on the tensor cores (qpc_tcband.cu).
// Against the banded solves (GB300, per step): one wavefunction of 800 x 41 with its dipole 1340 -> 37 us,
// 400 x 21 287 -> 15 us, 24 wavefunctions of 517 x 30 1120 -> 77 us, 256 of 800 x 41 8.0 -> 1.13 ms; error against
// extended precision after 60 steps 3.3e-13 against 4.7e-13.
#include "qpc_pos.cuh"
#include "qpc_radial.cuh"
#include <cmath>
#include <vector>

namespace qpc {

namespace {

constexpr int LMAX = 128;	// most l channels
constexpr int GRID_Y = 65535;	// most channels of a launch

// ------------------------------------------------------------------ the local part of a step
// One block: PT positions of one (slot, m), all l; PT lanes of a warp hold the positions, the 32 / PT groups of lanes
// work as so many warps.  y -> E_k, O_k (the even-l and odd-l halves of the transform by the eigenvectors of Y10;
// +-lambda share them), phases, and back:
//   z+- = E +- O, z+' = phi z+, z-' = conj(phi) z-, s = z+' + z-' = 2 (c E + i s O), d = z+' - z-' = 2 (i s E + c O)
// with phi = c + i s.  Both transforms in fixed point under each position's largest exponent, the phases in FP64
// (28 instructions per pair and position).  The dipole of f(r) = r is sum_k lambda_k r_j (|z+|^2 - |z-|^2) =
// sum_k 4 lambda_k r_j Re(conj(E_k) O_k).  PT = 32 is bound by the multiply-adds; with too few blocks to fill the
// SMs a block's own latency counts, and PT = 8 cuts it (four times the blocks, a quarter of the serial products).
// Three or four blocks per SM (80 or 64 registers, a few spilled), coefficients stored in the order a task reads them:
// 256 wavefunctions of 800 x 41 570 -> 438 us (multiply-adds alone 270), 24 of 517 x 30 36 -> 28 us.
struct angle_args {
	double2* y;		// [slot][M][L][N], in place
	int* ex;		// [slot][M][L][ntile * EPT]
	const int2 *V, *W;	// limbs of the transform and of its transpose, [M][task][k][G] (|V| <= 1)
	int nV, nW;		// of one m
	const double* lamp;	// [M][npair]
	const double* r;	// [N]
	const double* ftab;
	long ld;
	const int64_t *ntf, *ntt;
	long step;
	int cmode;
	double dt4;		// dt / 4
	int N, ntile, L, M, npair;
	double* zpart;		// one per block, [slot][M][.], of this step, or NULL
};

__device__ __forceinline__ int power_of(long s, long nt, int cmode)
{
	if (nt <= 0) return 0;
	if (cmode == 1) return (s >= 1 && s <= nt) ? 1 : 0;
	if (cmode == 2) return s < nt ? 1 : 0;
	if (s > nt) return 0;
	return (s == 0 || s == nt) ? 1 : 2;
}

template <int G, int PT, int BPS>
__global__ void __launch_bounds__(256, BPS) k_angle(const angle_args p)
{
	constexpr int NV = 8 * 32 / PT, TPT = TM / PT;	// virtual warps; blocks per tile
	extern __shared__ double2 sm[];
	__shared__ int pe[NV][PT];
	__shared__ double zs[NV][PT];
	const int lane = threadIdx.x % PT, warp = threadIdx.x / PT;
	const int tile = blockIdx.x % (p.ntile * TPT);
	const int im = blockIdx.x / (p.ntile * TPT);	// slot * M + m
	const int m = im % p.M, slot = im / p.M;
	const int pw = power_of(p.step, p.ntf[slot], p.cmode);
	const bool obs = p.zpart && p.step < p.ntt[slot];
	prev_wait();
	if (pw == 0 && !obs) return;
	const int L = p.L, np = p.npair, N = p.N;
	double2* a = sm;		// [L][PT]: y, then its limbs, then the eigen-channels' limbs
	double2* b = sm + L * PT;	// [L][PT]: E_k at 2k, O_k at 2k + 1, the zero channel at 2 npair
	const int row = tile * PT + lane;
	const bool in = row < N;
	double2* y = p.y + (long)im * L * N + row;
	int e = 0;
	for (int l = warp; l < L; l += NV) {
		const double2 v = in ? y[(long)l * N] : make_double2(0.0, 0.0);
		a[l * PT + lane] = v;
		e = max(e, max(bexp(v.x), bexp(v.y)));
	}
	pe[warp][lane] = e;
	__syncthreads();
	e = 0;
#pragma unroll
	for (int w = 0; w < NV; ++w) e = max(e, pe[w][lane]);
	for (int l = warp; l < L; l += NV) {
		const double2 v = a[l * PT + lane];
		const int2 q0 = quant(v.x, e), q1 = quant(v.y, e);
		reinterpret_cast<int4*>(a)[l * PT + lane] = make_int4(q0.x, q0.y, q1.x, q1.y);
	}
	__syncthreads();
	const int4* qa = reinterpret_cast<const int4*>(a) + lane;
	const int2* V = p.V + (long)m * p.nV;
	const int nl0 = (L + 1) / 2, nl1 = L / 2;	// even and odd l
	const int nE = np + (L & 1), gE = (nE + G - 1) / G, gO = (np + G - 1) / G;
	long long h[G][2], mm[G][2];
	for (int t = warp; t < gE + gO; t += NV) {
		const bool odd = t >= gE;
		const int k0 = (odd ? t - gE : t) * G, no = min(G, (odd ? np : nE) - k0);
		task_product<G, 2 * PT, false>(V + t * G * nl0, odd ? nl1 : nl0, qa + (odd ? PT : 0), h, mm);
#pragma unroll
		for (int g = 0; g < G; ++g)
			if (g < no) {
				const int s = e - 1078;
				b[(2 * (k0 + g) + (odd ? 1 : 0)) * PT + lane] =
					make_double2(to_double<false>(h[g][0], mm[g][0], s, e > EMAX), to_double<false>(h[g][1], mm[g][1], s, e > EMAX));
			}
	}
	__syncthreads();
	const double rj = in ? p.r[row] : 0.0;
	const double f = pw ? p.ftab[(long)slot * p.ld + p.step] * p.dt4 * rj : 0.0;
	double z = 0.0;
	e = 0;
	for (int k = warp; k < np; k += NV) {
		const double2 E = b[(2 * k) * PT + lane], O = b[(2 * k + 1) * PT + lane];
		const double lam = p.lamp[m * np + k];
		if (obs) z = fma(lam, fma(E.x, O.x, E.y * O.y), z);
		if (pw) {
			// 2 (c + i s), c + i s = ((1 - i beta) / (1 + i beta))^pw
			const double beta = lam * f, inv = reciprocal(fma(beta, beta, 1.0));
			double s = -4.0 * beta * inv, c = fma(s, beta, 2.0);	// a rounding of inv moves |c + i s| by beta^2 of it
			if (pw == 2) {
				const double s1 = s;
				s *= c;
				c = fma(-s1, s1, 2.0);
			}
			const double2 S = make_double2(fma(c, E.x, -s * O.y), fma(c, E.y, s * O.x));
			const double2 D = make_double2(fma(c, O.x, -s * E.y), fma(c, O.y, s * E.x));
			e = max(max(e, max(bexp(S.x), bexp(S.y))), max(bexp(D.x), bexp(D.y)));
			b[(2 * k) * PT + lane] = S;
			b[(2 * k + 1) * PT + lane] = D;
		}
	}
	if (obs) {
		zs[warp][lane] = 4.0 * z * rj;
		__syncthreads();
		if (threadIdx.x < 32) {
			double t = 0.0;
#pragma unroll
			for (int w = 0; w < NV; w += 32 / PT) t += zs[w + warp][lane];
#pragma unroll
			for (int o = 16; o; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
			if (threadIdx.x == 0) p.zpart[(long)im * p.ntile * TPT + tile] = t;
		}
	}
	if (pw == 0) return;
	if ((L & 1) && warp == NV - 1) { const double2 Z = b[2 * np * PT + lane]; e = max(e, max(bexp(Z.x), bexp(Z.y))); }
	pe[warp][lane] = e;
	__syncthreads();
	e = 0;
#pragma unroll
	for (int w = 0; w < NV; ++w) e = max(e, pe[w][lane]);
	for (int k = warp; k < L; k += NV) {
		const double2 v = b[k * PT + lane];
		const int2 q0 = quant(v.x, e), q1 = quant(v.y, e);
		reinterpret_cast<int4*>(a)[k * PT + lane] = make_int4(q0.x, q0.y, q1.x, q1.y);
	}
	__syncthreads();
	const int g0 = (nl0 + G - 1) / G, g1 = (nl1 + G - 1) / G;
	V = p.W + (long)m * p.nW;
	const unsigned grp = PT == 32 ? 0xffffffffu : ((1u << PT) - 1) << (threadIdx.x & 31 & ~(PT - 1));
	for (int t = warp; t < g0 + g1; t += NV) {
		const int odd = t >= g0 ? 1 : 0;
		const int o0 = (odd ? t - g0 : t) * G, no = min(G, (odd ? nl1 : nl0) - o0);
		// even l: s_k (slots 2k) and, for odd n_l, the zero channel (slot 2 npair); odd l: d_k (slots 2k + 1)
		task_product<G, 2 * PT, false>(V + t * G * nE, odd ? np : nE, qa + odd * PT, h, mm);
#pragma unroll
		for (int g = 0; g < G; ++g)
			if (g < no) {
				const int s = e - 1078, l = 2 * (o0 + g) + odd;
				const double2 v = make_double2(to_double<false>(h[g][0], mm[g][0], s, e > EMAX), to_double<false>(h[g][1], mm[g][1], s, e > EMAX));
				if (in) y[(long)l * N] = v;
				int x = in ? max(bexp(v.x), bexp(v.y)) : 0;
#pragma unroll
				for (int o = 1; o < TE; o <<= 1) x = max(x, __shfl_xor_sync(grp, x, o));
				if (lane % TE == 0) p.ex[((long)im * L + l) * p.ntile * EPT + row / TE] = x;
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

} // namespace

struct pos_path {
	int N = 0, P = 0, L = 0, M = 0, m0 = 0, B = 0, nlh = 0, npair = 0, nff = 1, ntile = 0;
	double dt = 0.0;
	radial_ops ops;
	band_store K;			// the mask of the run
	double2* buf[2] = {nullptr, nullptr};
	int* ex[2] = {nullptr, nullptr};
	int* exin = nullptr;
	int2 *V = nullptr, *W = nullptr;
	int nV = 0, nW = 0;
	double* lamp = nullptr;
	int* lmap = nullptr;		// channel -> l
	double* zpart = nullptr;
	static constexpr int ZB = 32;		// steps between two sums of the dipole's parts
	long zfirst = 0;
	int zcount = 0;
	int angle_g = 3;		// outputs per task of k_angle, PT = 32
	bool angle_small = false;	// PT = 8, one output per task
	bool angle_many = false;	// four blocks per SM
	int product = QPC_PRODUCT_NONE;	// kernel of the last run's first field-free product
};


namespace {

template <int G, int BPS>
void angle_launch(const pos_path* p, const angle_args& a, int slots, cudaStream_t st)
{
	launch_after(k_angle<G, 32, BPS>, dim3((unsigned)((long)slots * p->M * p->ntile)), 256, sizeof(double2) * 2 * 32 * p->L, st, a);
}

int build(pos_path* p, const pos_setup& in, bool* ok)
{
	const int N = p->N, L = p->L, M = p->M;
	int rc;
	const long nvec = (long)p->B * M * L;
	if ((rc = radial_create(&p->ops, radial_setup{N, p->P, p->nlh, p->nff, in.S, in.R, true, in.fieldfree, in.stream, p->B}, M * L, ok)) || !*ok) return rc;
	std::vector<int> lm(M * L);
	for (int c = 0; c < M * L; ++c) lm[c] = c % L + std::abs(p->m0 + c / L);
	// outputs per task of k_angle: the fewest rounds of eight warps
	int best = 1 << 30;
	for (int g = 2; g <= 4; ++g) {
		const int ne = p->npair + (L & 1), tasks = (ne + g - 1) / g + (p->npair + g - 1) / g, cost = (tasks + 7) / 8 * (g * 6 + 4);
		if (cost < best) { best = cost; p->angle_g = g; }
	}
	// fewer blocks than SMs with 32 positions each: 8
	p->angle_small = (long)p->B * M * p->ntile <= 304;
	// more than three per SM: four, with two outputs per task (256 wavefunctions of 800 x 41 460 -> 438 us, 48 108 -> 98;
	// 24 of 517 x 30, where three hold every block at once, 28 -> 29.6)
	p->angle_many = (long)p->B * M * p->ntile > 456;
	if (p->angle_many) p->angle_g = 2;
	// the transforms' limbs as the tasks read them; a task's outputs beyond the last are zero
	const int np = p->npair, nE = np + (L & 1), nl0 = (L + 1) / 2, nl1 = L / 2, G = p->angle_small ? 1 : p->angle_g;
	const int gE = (nE + G - 1) / G, gO = (np + G - 1) / G, g0 = (nl0 + G - 1) / G, g1 = (nl1 + G - 1) / G;
	p->nV = (gE + gO) * nl0 * G;
	p->nW = (g0 + g1) * nE * G;
	std::vector<int2> V((size_t)M * p->nV, make_int2(0, 0)), W((size_t)M * p->nW, make_int2(0, 0));
	for (int m = 0; m < M; ++m)
		for (int odd = 0; odd < 2; ++odd)
			for (int k = 0; k < (odd ? np : nE); ++k)
				for (int l = 0; l < (odd ? nl1 : nl0); ++l) {
					const int2 v = limbs_of(in.Vh[((size_t)m * (np + 1) + k) * L + 2 * l + odd]);
					V[(size_t)m * p->nV + (((odd ? gE : 0) + k / G) * nl0 + l) * G + k % G] = v;
					W[(size_t)m * p->nW + (((odd ? g0 : 0) + l / G) * nE + k) * G + l % G] = v;
				}
	if ((rc = dalloc(&p->lmap, lm.size())) || (rc = dalloc(&p->V, V.size())) || (rc = dalloc(&p->W, std::max<size_t>(W.size(), 1))) || (rc = dalloc(&p->lamp, (size_t)M * std::max(p->npair, 1)))) return rc;
	QPC_CUDA(cudaMemcpyAsync(p->lmap, lm.data(), sizeof(int) * lm.size(), cudaMemcpyHostToDevice, in.stream));
	QPC_CUDA(cudaMemcpyAsync(p->V, V.data(), sizeof(int2) * V.size(), cudaMemcpyHostToDevice, in.stream));
	QPC_CUDA(cudaMemcpyAsync(p->W, W.data(), sizeof(int2) * W.size(), cudaMemcpyHostToDevice, in.stream));
	QPC_CUDA(cudaMemcpyAsync(p->lamp, in.lamp, sizeof(double) * M * std::max(p->npair, 1), cudaMemcpyHostToDevice, in.stream));
	for (int i = 0; i < 2; ++i)
		if ((rc = dalloc(&p->buf[i], (size_t)nvec * N)) || (rc = dalloc(&p->ex[i], (size_t)nvec * p->ntile * EPT))) return rc;
	if ((rc = dalloc(&p->exin, (size_t)nvec * p->ntile * EPT))) return rc;
	const int smem = (int)(sizeof(double2) * 64 * LMAX);
	cudaFuncSetAttribute(k_angle<2, 32, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
	cudaFuncSetAttribute(k_angle<3, 32, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
	cudaFuncSetAttribute(k_angle<2, 32, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
	cudaFuncSetAttribute(k_angle<4, 32, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
	return wait_on(in.stream);	// the tables' copies
}

} // namespace

// The path is taken when 3 <= p <= 8, 2 <= n_l <= LMAX, the channels fit the second dimension of a grid and radial_create finds the operators to suit it.
// Everything else keeps the banded solves.
int pos_create(const pos_setup& in, pos_path** out)
{
	*out = nullptr;
	if (in.L > LMAX || in.L < 2 || in.P < 3 || in.P > 8 || (long)in.M * in.L > GRID_Y || in.nlh > GRID_Y) return QPC_OK;
	auto* p = new (std::nothrow) pos_path();
	if (!p) { set_error("host allocation"); return QPC_ERR_NOMEM; }
	p->N = in.N; p->P = in.P; p->L = in.L; p->M = in.M; p->m0 = in.m0; p->B = in.B; p->nlh = in.nlh; p->npair = in.npair;
	p->nff = in.nff; p->dt = in.dt; p->ntile = (in.N + TM - 1) / TM;
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
	cudaFree(p->lmap); cudaFree(p->V); cudaFree(p->W); cudaFree(p->lamp);
	for (int i = 0; i < 2; ++i) { cudaFree(p->buf[i]); cudaFree(p->ex[i]); }
	cudaFree(p->exin); cudaFree(p->zpart);
	p->K.release();
	radial_destroy(&p->ops);
	delete p;
}

void pos_buffers(const pos_path* p, double2* out[2])
{
	out[0] = p->buf[0]; out[1] = p->buf[1];
}

void pos_report(const pos_path* p, int32_t out[4])
{
	out[0] = p->ops.F.has_tc; out[1] = p->ops.W.has_tc; out[2] = p->ops.X.has_tc;
	out[3] = p->product;
}

#define POS_PROF(kind) struct prof_ { const pos_run& r; int k; prof_(const pos_run& r_, int k_) : r(r_), k(k_) { if (r.prof_begin) r.prof_begin(k, r.stream); } \
	~prof_() { if (r.prof_end) r.prof_end(k, r.stream); } } prof_scope_(r, kind)

// X^T (M X): S^-1 is 1 in this basis
int pos_mask(pos_path* p, const double* mask, int64_t* launches, cudaStream_t st, bool* ok)
{
	const size_t nn = (size_t)p->N * p->N;
	scratch tmp(st);
	double *Mx, *A;
	int rc;
	if ((rc = tmp.get(&Mx, nn)) || (rc = tmp.get(&A, nn)) || (rc = project_band(&p->ops, mask, false, Mx, A, st))) return rc;
	*launches += 4;
	return store_banded(&p->ops, p->K, A, p->N, 1, st, ok);
}

int pos_begin(pos_path* p, const pos_run& r)
{
	const int nchan = p->M * p->L;
	const long nvec = (long)p->B * nchan;
	cudaStream_t st = r.stream;
	if (r.z && !p->zpart) if (int rc = dalloc(&p->zpart, (size_t)pos_path::ZB * p->B * p->M * p->ntile * EPT)) return rc;
	p->zcount = 0;
	POS_PROF(QPC_KERNEL_TRANSFORM_FWD);
	exponents(r.state, p->exin, p->N, p->ntile, nvec, st);
	band_args a = band_args_of(&p->ops, p->ops.W, nchan, p->B);
	a.s0 = r.state; a.e0 = p->exin; a.smap = r.perm;
	a.dst = p->buf[0]; a.edst = p->ex[0];
	band_apply(a, false, p->ntile, st, &p->ops.W, r.status, r.stbit);
	*r.launches += 2;
	return QPC_OK;
}

static void sum_dipole(pos_path* p, const pos_run& r)
{
	if (!p->zcount) return;
	const int n = p->B * p->zcount;
	k_dipole_sum<<<(n + 127) / 128, 128, 0, r.stream>>>(p->zpart, r.z, r.ldz, r.ntt, p->B, p->M * p->ntile * (p->angle_small ? EPT : 1), p->zfirst, p->zcount);
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
		a.y = p->buf[cur]; a.ex = p->ex[cur]; a.V = p->V; a.W = p->W; a.nV = p->nV; a.nW = p->nW; a.lamp = p->lamp; a.r = p->ops.r; a.ftab = r.ftab; a.ld = r.ld; a.ntf = r.ntf; a.ntt = r.ntt;
		a.step = s; a.cmode = cmode; a.dt4 = 0.25 * p->dt; a.N = p->N; a.ntile = p->ntile; a.L = p->L; a.M = p->M; a.npair = p->npair;
		if (observe) {
			if (!p->zcount) p->zfirst = s;
			a.zpart = p->zpart + (size_t)p->zcount * p->B * p->M * p->ntile * (p->angle_small ? EPT : 1);
			++p->zcount;
		}
		if (p->angle_small) launch_after(k_angle<1, 8, 3>, dim3((unsigned)((long)slots * p->M * p->ntile * EPT)), 256, sizeof(double2) * 2 * 8 * p->L, st, a);
		else switch (p->angle_g) {
		case 2:
			if (p->angle_many) angle_launch<2, 4>(p, a, slots, st);
			else angle_launch<2, 3>(p, a, slots, st);
			break;
		case 3: angle_launch<3, 3>(p, a, slots, st); break;
		default: angle_launch<4, 3>(p, a, slots, st); break;
		}
		++*r.launches;
	};
	if (r.mask) {
		if (s > 0) {
			if (Bc > 0) angle(1, Bc, false);
			// the slots whose step s - 1 has just ended
			POS_PROF(QPC_KERNEL_TRANSFORM_BWD);
			band_args a = band_args_of(&p->ops, p->K, nchan, p->B);
			a.s0 = p->buf[1]; a.e0 = p->ex[1]; a.dst = p->buf[0]; a.edst = p->ex[0];
			a.nta = r.ntt; a.step = s - 1;
			band_apply(a, false, p->ntile, st);
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
		band_args a = band_args_of(&p->ops, p->ops.F, nchan, Bf);
		a.lmap = p->lmap;
		a.set_stride = (long)p->nlh * p->ops.F.stride;
		if (p->nff > 1) a.amap = r.perm;
		a.s0 = p->buf[cur]; a.e0 = p->ex[cur]; a.dst = p->buf[1 - cur]; a.edst = p->ex[1 - cur];
		a.nta = r.ntt; a.step = s;
		const int product = band_apply(a, true, p->ntile, st, &p->ops.F, r.status, r.stbit);
		if (s == 0) p->product = product;
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
	band_args a = band_args_of(&p->ops, p->ops.X, nchan, p->B);
	a.s0 = p->buf[0]; a.e0 = p->ex[0]; a.s1 = p->buf[1]; a.e1 = p->ex[1]; a.par = r.mask ? nullptr : r.ntt; a.dmap = r.perm;
	a.dst = r.state; a.edst = p->exin;
	a.nta = r.ntt; a.step = 0;	// a slot without steps stays as it is
	band_apply(a, false, p->ntile, r.stream, &p->ops.X, r.status, r.stbit);
	++*r.launches;
	QPC_CUDA(cudaGetLastError());
	return QPC_OK;
}

} // namespace qpc
