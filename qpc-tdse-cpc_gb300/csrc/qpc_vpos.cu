// The velocity-gauge elliptical step (qpc_vgwr.cu) with every radial coupling diagonal.
//
// Per eigen-channel of an angular coupling the step applies (S + e O)^-1 (S - e O) with O = 1/r (x2, y2) or d/dr
// (x1, y1).  In the basis I that is orthonormal in S and diagonalises 1/r the first is a phase; there d/dr is a real
// anti-symmetric matrix, Q^T A Q = blocks omega [[0, -1], [1, 0]], and in the basis D = I Q the second is a rotation
// of position pairs.  Radial transforms commute with the angular ones, so a step is a chain of
//   k_couple: coupling of one component, then its merged angular transform (both local in position), and
//   k_band_apply: the dense real Q or Q^T on every channel (from ~200 columns on tensor cores, qpc_tcband.cu), or the
//   banded F~_l in the basis I,
// with no factorisation and no recurrence.  The pairing of the angular eigenvectors (u, +-v)/sqrt 2 folds into the
// coupling: with a, b the two m-parity halves, M+- = c +- i s (phase) or c -+ s J (rotation),
//   a' = c a + i s kappa b, b' = c b + i s conj(kappa) a   or   a' = c a - s kappa J b, b' = c b - s conj(kappa) J a,
// kappa = conj(g_A) g_B.  Between two steps the closing and the opening x1 coupling (same field) are one of power 2.
// All products in fixed point (qpc_radial.cu).  The banded solves cost the latency of eight recurrences over N rows
// (4.85 us per row, whatever the batch, until ~10^4 chains fill the FP64 pipe); this form costs 8 N^2 products per
// channel.  Measured on GB300 at 400 x (25 x 13), two wavefunctions: 22.6 -> 1.07 ms per step (1.7 with Q on the
// multiply-adds: 136 -> 40 us each).
#include "qpc_vpos.cuh"
#include "qpc_radial.cuh"
#include <cusolverDn.h>
#include <cmath>
#include <vector>

namespace qpc {

namespace {

constexpr int AG = 3;		// outputs per task of k_couple
constexpr int CW = 16;		// its warps
constexpr int NBMAX = 452;	// most channels of a parity block (its 32-position tile sits in shared memory)

struct set_args {
	const double2* in;	// [slot][nch][N]
	double2* out;
	int* eout;		// [slot][nch][ntile * EPT]
	const int2* A[2][2];	// real matrices of the angular transform, [block][set], limbs as [task][k][AG]
	int off[2], na[2], ns[2];
	int kind;		// 0: no coupling, 1: phase, 2: rotation of position pairs
	int power;
	const double* sig;	// eigenvalue of row k by engine channel
	double2 kap[2];
	const double* rad;	// per position: 1/r_j or omega
	const double* atab;
	long ld, at;		// atab[(perm[slot] ld + at) 2 + axis]
	int axis;
	double scale;		// e = sig * A * scale * rad
	const int* perm;
	int N, ntile, nch, slices;
};

// One block: TM positions of one parity block of one slot, an interleaved share of the outputs; lane = position.
// Bound by the integer multiply-adds of the two real products (6 n per output) and the FP64 of the coupling (35 per pair
// and position, in every share): 16 warps, two blocks per SM, shares to give every SM a block once.  400 x 325 channels,
// two wavefunctions 96 -> 76 us, 800 x 861 channels 440 -> 275 us (8 warps, an IEEE division per phase, row-major
// coefficients before).
__global__ void __launch_bounds__(CW * 32, 2) k_couple(const set_args p)
{
	extern __shared__ double2 sm[];
	__shared__ int pe[2][32];
	constexpr int G = AG;
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const int tile = blockIdx.x, blk = blockIdx.y & 1, slot = blockIdx.y >> 1, slice = blockIdx.z;
	const int na = p.na[blk], ns = p.ns[blk], n = na + ns, N = p.N;
	const int row = tile * TM + lane;
	const bool in = row < N;
	const long base = ((long)slot * p.nch + p.off[blk]) * N + row;
	if (warp < 2) pe[warp][lane] = 0;
	for (int q = warp; q < n; q += CW) sm[q * 32 + lane] = in ? p.in[base + (long)q * N] : make_double2(0.0, 0.0);
	__syncthreads();
	if (p.kind) {
		const double f = p.atab[((long)p.perm[slot] * p.ld + p.at) * 2 + p.axis] * p.scale * (in ? p.rad[row] : 0.0);
		const double2 kp = p.kap[blk];
		for (int k = warp; k < ns; k += CW) {
			const double2 a = sm[k * 32 + lane], b = sm[(na + k) * 32 + lane];
			const double x = p.sig[p.off[blk] + k] * f;
			double s = -2.0 * x * reciprocal(fma(x, x, 1.0)), c = fma(s, x, 1.0);
			if (p.power == 2) {
				const double s1 = 2.0 * s;
				s = s1 * c;
				c = fma(-0.5 * s1, s1, 1.0);
			}
			double2 u = b, v = a, g;	// a' = c a + s g u, b' = c b + s h v with g = i kappa, h = i conj(kappa), or kappa
			double2 h;
			if (p.kind == 1) {
				g = make_double2(-kp.y, kp.x);
				h = make_double2(kp.y, kp.x);
			} else {
				const double sg = (lane & 1) ? 1.0 : -1.0;	// (J v)_2j = -v_2j+1, (J v)_2j+1 = v_2j
				u = make_double2(sg * __shfl_xor_sync(0xffffffffu, b.x, 1), sg * __shfl_xor_sync(0xffffffffu, b.y, 1));
				v = make_double2(sg * __shfl_xor_sync(0xffffffffu, a.x, 1), sg * __shfl_xor_sync(0xffffffffu, a.y, 1));
				g = kp;
				h = make_double2(kp.x, -kp.y);
			}
			const double2 gu = make_double2(g.x * u.x - g.y * u.y, g.x * u.y + g.y * u.x), hv = make_double2(h.x * v.x - h.y * v.y, h.x * v.y + h.y * v.x);
			sm[k * 32 + lane] = make_double2(fma(c, a.x, s * gu.x), fma(c, a.y, s * gu.y));
			sm[(na + k) * 32 + lane] = make_double2(fma(c, b.x, s * hv.x), fma(c, b.y, s * hv.y));
		}
		__syncthreads();
	}
	int e0 = 0, e1 = 0;
	for (int q = warp; q < n; q += CW) {
		const double2 v = sm[q * 32 + lane];
		const int e = max(bexp(v.x), bexp(v.y));
		if (q < na) e0 = max(e0, e); else e1 = max(e1, e);
	}
	atomicMax(&pe[0][lane], e0);
	atomicMax(&pe[1][lane], e1);
	__syncthreads();
	e0 = pe[0][lane];
	e1 = pe[1][lane];
	for (int q = warp; q < n; q += CW) {
		const double2 v = sm[q * 32 + lane];
		const int e = q < na ? e0 : e1;
		const int2 x = quant(v.x, e), y = quant(v.y, e);
		reinterpret_cast<int4*>(sm)[q * 32 + lane] = make_int4(x.x, x.y, y.x, y.y);
	}
	__syncthreads();
	const int4* qs = reinterpret_cast<const int4*>(sm) + lane;
	const int ga = (na + G - 1) / G, gb = (ns + G - 1) / G;
	long long h[G][2], m[G][2];
	for (int t = warp + CW * slice; t < ga + gb; t += CW * p.slices) {
		const int set = t >= ga ? 1 : 0;
		const int o0 = (set ? t - ga : t) * G, nn = set ? ns : na, no = min(G, nn - o0);
		task_product<G, 32, true>(p.A[blk][set] + (long)o0 * nn, nn, qs + (set ? na : 0) * 32, h, m);
		const int e = set ? e1 : e0;
#pragma unroll
		for (int g = 0; g < G; ++g)
			if (g < no) {
				const double2 v = make_double2(to_double<false>(h[g][0], m[g][0], e - 1078, e > EMAX), to_double<false>(h[g][1], m[g][1], e - 1078, e > EMAX));
				const int ch = (set ? na : 0) + o0 + g;
				if (in) p.out[base + (long)ch * N] = v;
				const int x = group_max(in ? max(bexp(v.x), bexp(v.y)) : 0);
				if (lane % TE == 0) p.eout[(((long)slot * p.nch + p.off[blk] + ch) * p.ntile + tile) * EPT + lane / TE] = x;
			}
	}
}

// i A as a column-major Hermitian matrix
__global__ void k_hermitian(const double* __restrict__ A, int N, cuDoubleComplex* __restrict__ H)
{
	const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
	if (t >= (long)N * N) return;
	const long j = t / N, i = t % N;
	H[t] = make_cuDoubleComplex(0.0, 0.5 * (A[i * N + j] - A[j * N + i]));
}

// rows 2j, 2j+1 of Qt: sqrt 2 (Re, Im) of the eigenvector of the j-th largest omega; for odd N the last row: the
// null vector, turned real.  om: omega per row.  i A u = omega u gives A Re u = omega Im u, A Im u = -omega Re u.
__global__ void k_pairs(const cuDoubleComplex* __restrict__ U, const double* __restrict__ w, int N, double* __restrict__ Qt, double* __restrict__ om)
{
	const int j = blockIdx.x;
	if (2 * j + 1 < N) {
		const cuDoubleComplex* u = U + (long)(N - 1 - j) * N;
		const double r2 = 1.41421356237309504880;
		for (int i = threadIdx.x; i < N; i += blockDim.x) { Qt[(long)(2 * j) * N + i] = r2 * u[i].x; Qt[(long)(2 * j + 1) * N + i] = r2 * u[i].y; }
		if (threadIdx.x == 0) om[2 * j] = om[2 * j + 1] = w[N - 1 - j];
	} else if (threadIdx.x == 0) {
		const cuDoubleComplex* u = U + (long)((N - 1) / 2) * N;
		double re = 0.0, im = 0.0;
		for (int i = 0; i < N; ++i) { re += u[i].x * u[i].x - u[i].y * u[i].y; im += 2.0 * u[i].x * u[i].y; }
		const double ph = -0.5 * atan2(im, re), c = cos(ph), s = sin(ph);
		for (int i = 0; i < N; ++i) Qt[(long)(N - 1) * N + i] = c * u[i].x - s * u[i].y;
		om[N - 1] = 0.0;
	}
}

// limbs of op(A), row-major n x n, as [task][k][AG]
__global__ void k_limbs(const double* __restrict__ A, int n, int trans, int2* __restrict__ out)
{
	const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
	if (t >= (long)n * n) return;
	const long i = t / n, k = t % n;
	const long long x = __double2ll_rn((trans ? A[k * n + i] : A[t]) * 72057594037927936.0);
	const int hi = (int)((x + (1ll << 27)) >> 28);
	out[(i / AG * n + k) * AG + i % AG] = make_int2(hi, (int)(x - ((long long)hi << 28)));
}

__global__ void k_negate(const double* __restrict__ a, double* __restrict__ b, int n)
{
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i < n) b[i] = -a[i];
}

} // namespace

struct vpos_path {
	int N = 0, nch = 0, B = 0, ntile = 0;
	double dt = 0.0;
	int off[2], na[2], ns[2];
	double2 kap[4][2];
	radial_ops ops;
	band_store TD, TI;		// basis I -> D, D -> I
	double *om = nullptr, *rinv = nullptr;	// per position
	const double* lam[4];
	int2* tab = nullptr;		// angular matrices, [mat][block][set][trans]
	const int2* A[5][2][2][2] = {};
	int* lmap = nullptr;
	double2* buf[2] = {nullptr, nullptr};
	int* ex[2] = {nullptr, nullptr};
	int* exin = nullptr;
	size_t smem = 0;
	int *status = nullptr, *hstatus = nullptr;	// a tensor-core wait ran out (device, pinned)
	bool on_tensor_cores() const { return TD.has_tc || TI.has_tc; }	// either transform may have planes without the other
	cudaStream_t stream = nullptr;
};

namespace {

// the basis D: Q from the Hermitian eigenproblem of i X^T D X (cuSOLVER, set-up only), orthonormal to rounding
int momentum_basis(vpos_path* p, const vpos_setup& in, bool* ok)
{
	const int N = p->N;
	const size_t nn = (size_t)N * N;
	cudaStream_t st = in.stream;
	scratch tmp(st);
	double *A, *T, *w, *Qt;
	cuDoubleComplex *H, *work = nullptr;
	int* info;
	int rc;
	if ((rc = tmp.get(&A, nn)) || (rc = tmp.get(&T, nn)) || (rc = tmp.get(&w, N)) || (rc = tmp.get(&Qt, nn)) || (rc = tmp.get(&H, nn)) || (rc = tmp.get(&info, 1)))
		return rc;
	if ((rc = project_band(&p->ops, in.D, true, T, A, st))) return rc;
	k_hermitian<<<(unsigned)((nn + 255) / 256), 256, 0, st>>>(A, N, H);
	cusolverDnHandle_t sol = nullptr;
	// without room for its handle or work space: as any allocation that fails
	if (cusolverDnCreate(&sol) != CUSOLVER_STATUS_SUCCESS) { cudaGetLastError(); set_error("cusolverDnCreate failed"); return QPC_ERR_NOMEM; }
	struct guard { cusolverDnHandle_t s; ~guard() { cusolverDnDestroy(s); } } g{sol};
	int lwork = 0;
	if (cusolverDnSetStream(sol, st) != CUSOLVER_STATUS_SUCCESS ||
		cusolverDnZheevd_bufferSize(sol, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER, N, H, N, w, &lwork) != CUSOLVER_STATUS_SUCCESS) {
		set_error("heevd buffer size failed");
		return QPC_ERR_CUDA;
	}
	if ((rc = tmp.get(&work, (size_t)std::max(lwork, 1)))) return rc;
	const cusolverStatus_t cs = cusolverDnZheevd(sol, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER, N, H, N, w, work, lwork, info);
	if (cs != CUSOLVER_STATUS_SUCCESS) {
		set_error("heevd failed");
		if (cs == CUSOLVER_STATUS_ALLOC_FAILED) { cudaGetLastError(); return QPC_ERR_NOMEM; }
		return QPC_ERR_CUDA;
	}
	k_pairs<<<(N + 1) / 2, 128, 0, st>>>(H, w, N, Qt, p->om);
	QPC_CUDA(cudaGetLastError());
	int hinfo = 0;
	if ((rc = copy_to_host(&hinfo, info, sizeof(int), st))) return rc;
	*ok = hinfo == 0;
	if (!*ok) return QPC_OK;
	if ((rc = orthonormalise(Qt, N, A, T, st, ok)) || !*ok) return rc;
	if ((rc = store_dense(&p->ops, p->TD, Qt, N, 1, p->B * p->nch, st, ok)) || !*ok) return rc;
	if ((rc = store_dense(&p->ops, p->TI, Qt, 1, N, p->B * p->nch, st, ok)) || !*ok) return rc;
	return wait_on(st);
}

int build(vpos_path* p, const vpos_setup& in, bool* ok)
{
	const int N = p->N, nch = p->nch, nb = N * (in.P + 1);
	cudaStream_t st = in.stream;
	int rc;
	// -1/r ascends with the row
	std::vector<double> neg(in.Ri, in.Ri + nb);
	for (double& v : neg) v = -v;
	double* R = nullptr;
	if ((rc = dalloc(&R, nb))) return rc;
	struct guard { double* p; ~guard() { cudaFree(p); } } g{R};
	QPC_CUDA(cudaMemcpyAsync(R, neg.data(), sizeof(double) * nb, cudaMemcpyHostToDevice, st));
	if ((rc = radial_create(&p->ops, radial_setup{N, in.P, in.nlh, 1, in.S, R, false, in.fieldfree, st, 0}, nch, ok)) || !*ok) return rc;
	if ((rc = dalloc(&p->om, N)) || (rc = dalloc(&p->rinv, N))) return rc;
	k_negate<<<(N + 255) / 256, 256, 0, st>>>(p->ops.r, p->rinv, N);
	if ((rc = momentum_basis(p, in, ok)) || !*ok) return rc;
	// angular tables
	size_t tot = 0;
	auto room = [](int n) { return (size_t)((n + AG - 1) / AG) * AG * n; };	// a task's outputs beyond the last are zero
	for (int b = 0; b < 2; ++b) tot += room(p->na[b]) + room(p->ns[b]);
	if ((rc = dalloc(&p->tab, tot * 10))) return rc;
	QPC_CUDA(cudaMemsetAsync(p->tab, 0, sizeof(int2) * tot * 10, st));
	size_t o = 0;
	for (int m = 0; m < 5; ++m)
		for (int b = 0; b < 2; ++b)
			for (int s = 0; s < 2; ++s) {
				const int n = s ? p->ns[b] : p->na[b];
				for (int t = 0; t < 2; ++t) {
					p->A[m][b][s][t] = p->tab + o;
					if (n) k_limbs<<<(unsigned)(((long)n * n + 255) / 256), 256, 0, st>>>(in.tm[m][b][s], n, t, p->tab + o);
					o += room(n);
				}
			}
	for (int c = 0; c < 4; ++c) {
		p->lam[c] = in.lam[c];
		for (int b = 0; b < 2; ++b) {
			const double2 ga = in.gam[c][b][0], gb = in.gam[c][b][1];
			p->kap[c][b] = make_double2(ga.x * gb.x + ga.y * gb.y, ga.x * gb.y - ga.y * gb.x);
		}
	}
	std::vector<int> lm(nch);
	for (int t = 0; t < nch; ++t) lm[t] = in.chmap[t] % in.n_l + std::abs(in.m0 + in.chmap[t] / in.n_l);
	if ((rc = dalloc(&p->lmap, nch))) return rc;
	QPC_CUDA(cudaMemcpyAsync(p->lmap, lm.data(), sizeof(int) * nch, cudaMemcpyHostToDevice, st));
	const long nvec = (long)p->B * nch;
	for (int i = 0; i < 2; ++i) {
		p->buf[i] = in.buf[i];
		if ((rc = dalloc(&p->ex[i], (size_t)nvec * p->ntile * EPT))) return rc;
	}
	if ((rc = dalloc(&p->exin, (size_t)nvec * p->ntile * EPT)) || (rc = dalloc(&p->status, 1))) return rc;
	QPC_CUDA(cudaMemsetAsync(p->status, 0, sizeof(int), st));
	QPC_CUDA(cudaMallocHost(&p->hstatus, sizeof(int)));
	*p->hstatus = 0;
	p->smem = sizeof(double2) * 32 * std::max(in.nb[0], in.nb[1]);
	QPC_CUDA(cudaFuncSetAttribute(k_couple, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(sizeof(double2) * 32 * NBMAX)));
	QPC_CUDA(cudaGetLastError());
	return wait_on(st);
}

} // namespace

// Taken for parity blocks of at most NBMAX channels, 3 <= p <= 8, and sizes where the products are cheaper than
// the recurrences: per step 8 N^2 * 6 multiply-adds per channel at 6e12 a second (plus ~0.2 ms of launches), against
// the larger of 8 * 4.85 us N (latency) and 8 * 240 N FP64 instructions per channel at 6e11 a second.
int vpos_create(const vpos_setup& in, vpos_path** out)
{
	*out = nullptr;
	if (in.P < 3 || in.P > 8 || in.N > DENSE_MAX || std::max(in.nb[0], in.nb[1]) > NBMAX) return QPC_OK;
	const double cols = (double)in.B * in.nch, N = in.N;
	const double here = 2e-4 + cols * N * (48.0 * N + 30.0 * in.nch) / 6e12, there = std::max(38.8e-6 * N, cols * N * 1920.0 / 6e11);
	if (here > there) return QPC_OK;
	auto* p = new (std::nothrow) vpos_path();
	if (!p) { set_error("host allocation"); return QPC_ERR_NOMEM; }
	p->N = in.N; p->nch = in.nch; p->B = in.B; p->dt = in.dt; p->ntile = (in.N + TM - 1) / TM; p->stream = in.stream;
	for (int b = 0; b < 2; ++b) { p->off[b] = in.off[b]; p->na[b] = in.na[b]; p->ns[b] = in.nb[b] - in.na[b]; }
	bool ok = false;
	const int rc = build(p, in, &ok);
	if (rc || !ok) {
		vpos_destroy(p);
		return rc;
	}
	*out = p;
	return QPC_OK;
}

void vpos_destroy(vpos_path* p)
{
	if (!p) return;
	cudaFree(p->om); cudaFree(p->rinv); cudaFree(p->tab); cudaFree(p->lmap);
	for (int i = 0; i < 2; ++i) cudaFree(p->ex[i]);
	cudaFree(p->exin); cudaFree(p->status);
	if (p->hstatus) cudaFreeHost(p->hstatus);
	p->TD.release(); p->TI.release();
	radial_destroy(&p->ops);
	delete p;
}

void vpos_report(const vpos_path* p, int32_t out[2])
{
	out[0] = p->TD.has_tc; out[1] = p->TI.has_tc;
}

namespace {

struct prof_scope {
	const vpos_run& r; int k;
	prof_scope(const vpos_run& r_, int k_) : r(r_), k(k_) { if (r.prof_begin) r.prof_begin(k); }
	~prof_scope() { if (r.prof_end) r.prof_end(k); }
};

// coupling of component c (-1: none) with the field at atab index `at`, then the angular matrix mat: buf[src] -> buf[1 - src]
void couple(vpos_path* p, const vpos_run& r, int src, int c, long at, int power, int mat, int trans, int nlive)
{
	prof_scope ps(r, c < 0 ? 0 : 1);
	set_args a{};
	a.in = p->buf[src]; a.out = p->buf[1 - src]; a.eout = p->ex[1 - src];
	for (int b = 0; b < 2; ++b) {
		for (int s = 0; s < 2; ++s) a.A[b][s] = p->A[mat][b][s][trans];
		a.off[b] = p->off[b]; a.na[b] = p->na[b]; a.ns[b] = p->ns[b];
	}
	if (c >= 0) {
		const bool anti = c == 0 || c == 2;
		a.kind = anti ? 2 : 1;
		a.power = power;
		a.sig = p->lam[c];
		for (int b = 0; b < 2; ++b) a.kap[b] = p->kap[c][b];
		a.rad = anti ? p->om : p->rinv;
		a.atab = r.atab; a.ld = r.ld; a.at = at; a.axis = c < 2 ? 0 : 1;
		// e = lam * (sgn A/2) * (-+ dt/4), cn_1e.hpp:911-914
		a.scale = 0.5 * (c == 1 ? 1.0 : -1.0) * (0.25 * p->dt) * (anti ? -1.0 : 1.0);
	}
	a.perm = r.perm;
	a.N = p->N; a.ntile = p->ntile; a.nch = p->nch;
	a.slices = std::max(1, std::min(4, 152 / std::max(1, 2 * nlive * p->ntile)));
	// not launch_after: two blocks would share an SM beside the previous kernel's last ones, the others stay empty (4.3 -> 5.6 ms)
	k_couple<<<dim3(p->ntile, 2 * nlive, a.slices), CW * 32, p->smem, p->stream>>>(a);
	++*r.launches;
}

// every channel of the live slots through the dense radial transform b
void radial(vpos_path* p, const vpos_run& r, int src, const band_store& b, int nlive)
{
	prof_scope ps(r, 0);
	band_args a = band_args_of(&p->ops, b, 1, nlive * p->nch);
	a.s0 = p->buf[src]; a.e0 = p->ex[src]; a.dst = p->buf[1 - src]; a.edst = p->ex[1 - src];
	band_apply(a, false, p->ntile, p->stream, &b, p->status, 1);
	++*r.launches;
}

void fieldfree(vpos_path* p, const vpos_run& r, int src, long s, int k0, int n)
{
	prof_scope ps(r, 2);
	band_args a = band_args_of(&p->ops, p->ops.F, p->nch, n);
	a.lmap = p->lmap;
	const long o = (long)k0 * p->nch;
	a.s0 = p->buf[src] + o * p->N; a.e0 = p->ex[src] + o * p->ntile * EPT;
	a.dst = p->buf[1 - src] + o * p->N; a.edst = p->ex[1 - src] + o * p->ntile * EPT;
	a.nta = r.ntt + k0; a.step = s;
	band_apply(a, true, p->ntile, p->stream);
	++*r.launches;
}

} // namespace

int vpos_begin(vpos_path* p, const vpos_run& r)
{
	prof_scope ps(r, 0);
	if (p->on_tensor_cores()) QPC_CUDA(cudaMemsetAsync(p->status, 0, sizeof(int), p->stream));
	exponents(r.X, p->exin, p->N, p->ntile, (long)p->B * p->nch, p->stream);
	band_args a = band_args_of(&p->ops, p->ops.W, p->nch, p->B);
	a.s0 = r.X; a.e0 = p->exin; a.dst = p->buf[0]; a.edst = p->ex[0];
	band_apply(a, false, p->ntile, p->stream);
	*r.launches += 2;
	QPC_CUDA(cudaGetLastError());
	return QPC_OK;
}

int vpos_step(vpos_path* p, const vpos_run& r, long s, int nlive, int nff, bool open, bool close)
{
	// the state of every running slot is in buf[s & 1] and ends in the other one; `at` is where the live ones are
	const int in = (int)(s & 1);
	int at = in;
	auto c = [&](int comp, long t, int power, int mat, int trans) { couple(p, r, at, comp, t, power, mat, trans, nlive); at = 1 - at; };
	auto to = [&](const band_store& b) { radial(p, r, at, b, nlive); at = 1 - at; };
	if (nff > nlive) fieldfree(p, r, in, s, nlive, nff - nlive);
	if (nlive > 0) {
		if (open) { c(-1, 0, 0, 0, 1); to(p->TD); }
		c(0, s, open ? 1 : 2, 2, 0); to(p->TI);
		c(1, s, 1, 3, 0); to(p->TD);
		c(2, s, 1, 4, 0); to(p->TI);
		c(3, s, 1, 1, 0);
		fieldfree(p, r, at, s, 0, nlive);
		at = 1 - at;
		c(-1, 0, 0, 1, 1);
		c(3, s + 1, 1, 4, 1); to(p->TD);
		c(2, s + 1, 1, 3, 1); to(p->TI);
		c(1, s + 1, 1, 2, 1); to(p->TD);
		if (close) { c(0, s + 1, 1, 0, 0); to(p->TI); }
	}
	QPC_CUDA(cudaGetLastError());
	return QPC_OK;
}

int vpos_peek(vpos_path* p, const vpos_run& r, long s, int n)
{
	prof_scope ps(r, 0);
	band_args a = band_args_of(&p->ops, p->ops.X, p->nch, n);
	a.s0 = p->buf[s & 1]; a.e0 = p->ex[s & 1]; a.dst = r.X; a.edst = p->exin;
	a.nta = r.ntt; a.step = s;
	band_apply(a, false, p->ntile, p->stream);
	++*r.launches;
	QPC_CUDA(cudaGetLastError());
	return QPC_OK;
}

int vpos_end(vpos_path* p, const vpos_run& r)
{
	prof_scope ps(r, 0);
	band_args a = band_args_of(&p->ops, p->ops.X, p->nch, p->B);
	a.s0 = p->buf[0]; a.e0 = p->ex[0]; a.s1 = p->buf[1]; a.e1 = p->ex[1]; a.par = r.ntt;
	a.dst = r.X; a.edst = p->exin;
	a.nta = r.ntt; a.step = 0;	// a slot without steps stays as it is
	band_apply(a, false, p->ntile, p->stream);
	++*r.launches;
	QPC_CUDA(cudaGetLastError());
	if (p->on_tensor_cores()) QPC_CUDA(cudaMemcpyAsync(p->hstatus, p->status, sizeof(int), cudaMemcpyDeviceToHost, p->stream));
	return QPC_OK;
}

int vpos_check(const vpos_path* p)
{
	if (*p->hstatus == 0) return QPC_OK;
	set_error("a tensor-core wait ran out");
	return QPC_ERR_TIMEOUT;
}

} // namespace qpc
