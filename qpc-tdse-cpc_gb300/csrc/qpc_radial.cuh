// The radial operators of a grid in a localised orthonormal basis, stored for fixed-point banded products
// (qpc_radial.cu).
#pragma once
#include "qpc_internal.h"
#include "qpc_cuda_util.cuh"
#include "qpc_fixed.cuh"
#include <functional>
#include <vector>

namespace qpc {

constexpr int WMAX = 176;	// widest band (either side of the diagonal) the products take
// a product's sum is held in 63 bits, less than 128 in units of the column's and the operator's powers of two.  F~ is
// unitary and stays below 27; the entries of any other band are added up at set-up, and a dense orthogonal matrix has rows
// of norm 1, so at most sqrt(N)
constexpr double SUM_MAX = 126.0;
constexpr int DENSE_MAX = 15876;	// SUM_MAX^2

struct band_args {
	const char* A;		// operators, [set][nlh] of astride bytes
	long astride, set_stride;
	const int4* td;		// per tile: first chunk, first and end chunk with hi limbs, end chunk
	const long* toff;	// per tile: byte offset
	const int* lmap;	// channel -> operator of a set
	const int* amap;	// destination slot -> set (NULL: one set)
	int ea;			// |A| <= 2^ea
	const int* er;		// times 2^er of the row (real operators; NULL: 1)
	int N, ntile, nchan, ncols;
	const double2 *s0, *s1;	// [slot][nchan][N]; s1 where par[slot] is odd
	const int *e0, *e1;	// largest biased exponent of every TE rows, [slot][nchan][ntile * EPT]
	const int64_t* par;
	const int* smap;	// slot -> source slot (NULL: the same)
	const int* dmap;	// slot -> destination slot (NULL: the same)
	double2* dst;
	int* edst;
	const int64_t* nta;	// slots with step < nta[slot] take part (NULL: all)
	long step;
	int tile0;		// first tile of the launch
};

// digit planes of a set of operators (one per l) for k_tc_apply; made from the FP64 entries
struct tc_store {
	bool cx = false;
	int ea = 0;			// |A| <= 2^ea
	int* ear = nullptr;		// per operator and row instead, or NULL
	int db = 8;			// bits of a digit
	int N = 0, ntile = 0;		// columns, 128-row tiles
	int nrow = 0;
	size_t stride = 0;		// bytes of one operator
	int2* d_list = nullptr;		// per tile: its (first k, first digit) stages, those with every digit first
	int4* d_first = nullptr;	// per tile: its entries of d_list, the k they cover
	size_t* d_off = nullptr;	// per tile: byte offset of its first plane
	char* A = nullptr;
	std::vector<int> work;		// per tile: cycles of tensor-core math
	void release();
};

// an operator (or one per l and set) in the layout k_band_apply reads: per tile of TM rows the chunks of KC columns
// td = (first, first with hi limbs, end of those, end) at byte off
struct band_store {
	int w = 0, ea = 0;
	int* er = nullptr;		// the rows' own powers of two (device [N]), or NULL
	long stride = 0;		// bytes of one operator
	std::vector<int4> td;
	std::vector<long> off;
	int4* d_td = nullptr;
	long* d_off = nullptr;
	char* A = nullptr;
	size_t cap = 0;
	std::vector<double> prof;	// largest entry per distance, as laid out
	tc_store tc;			// the same for the tensor cores, for batches
	bool has_tc = false, tc_always = false;
	void release() { tc.release(); has_tc = false; cudaFree(d_td); cudaFree(d_off); cudaFree(A); cudaFree(er); d_td = nullptr; d_off = nullptr; A = nullptr; er = nullptr; }
};

// what radial_create reads: device bands S, R [N][P+1] (R: the operator the basis diagonalises, its eigenvalues
// ascending with the row), nff sets of field-free operators for l = 0..nlh-1.  fieldfree(X, wk, J, fi) applies the
// step of set fi to J vectors on `stream`: X[J][N][nlh] (r-major) when rmajor, else X[J][nlh][N]; wk the same size.
struct radial_setup {
	int N, P, nlh, nff;
	const double *S, *R;
	bool rmajor;
	std::function<int(double2*, double2*, int, int)> fieldfree;
	cudaStream_t stream;
	int batch;		// most columns of a product: from TC_MIN on the operators are kept for the tensor cores too
};
constexpr int TC_MIN = 6;	// below, the multiply-adds win at every size (16 MB to 300 MB of planes saved)

// eigenvectors x_i of (R, S): X^T S X = 1, X^T R X = diag(r); c = X y
struct radial_ops {
	int N = 0, P = 0, nlh = 0, nff = 1, ntile = 0;
	double *Xt = nullptr, *r = nullptr;	// x_i as rows, eigenvalues
	band_store F, W, X;			// X^T S F_l X, X^T S, X
	int* zero = nullptr;			// zeros [max(nlh, nmap)]
	unsigned long long* prof = nullptr;
};

// ok = false (with QPC_OK): S not positive definite, eigenvalues not apart, or an operator that does not fall off
// within WMAX of the diagonal (or takes more than 16 GB,
// or more than a quarter of the free memory)
int radial_create(radial_ops* p, const radial_setup& in, int nmap, bool* ok);
void radial_destroy(radial_ops* p);

// A (device, FP64, element (i, j) at A[i si + j sj]) into b, banded where it falls off (ok), or dense
int store_banded(radial_ops* p, band_store& b, const double* A, long si, long sj, cudaStream_t st, bool* ok);
// an orthogonal matrix (ok: N at most DENSE_MAX); ncols: most columns of a product
int store_dense(radial_ops* p, band_store& b, const double* A, long si, long sj, int ncols, cudaStream_t st, bool* ok);
// A [N][N] = X^T B X for a symmetric band B, or for an anti-symmetric one given by its upper entries (device
// [N][P+1]), zero beyond ~WMAX of the diagonal; Bx scratch [N][N]
int project_band(const radial_ops* p, const double* B, bool anti, double* Bx, double* A, cudaStream_t st);

// rows of Qt [N][N] made orthonormal to rounding from nearly so (ok); E, T scratch [N][N]
int orthonormalise(double* Qt, int N, double* E, double* T, cudaStream_t st, bool* ok);

band_args band_args_of(const radial_ops* p, const band_store& b, int nchan, int ncols);
// status, stbit: device word or-ed with stbit when a wait of the tensor-core kernel ran out; b: the store behind a (its
// planes are used where that is the faster way), or NULL
// returns the kernel it took (QPC_PRODUCT_*)
int band_apply(const band_args& a, bool cx, int tiles, cudaStream_t st, const band_store* b = nullptr, int* status = nullptr, int stbit = 0);
// largest biased exponent of every TE rows of src [nvec][N]
void exponents(const double2* src, int* ex, int N, int ntile, long nvec, cudaStream_t st);

// device scratch of a set-up, given back at its end
struct scratch {
	cudaStream_t st;
	std::vector<void*> ptr;
	explicit scratch(cudaStream_t s) : st(s) {}
	~scratch() { release(); }
	void release()
	{
		for (void* q : ptr) cudaFreeAsync(q, st);
		ptr.clear();
	}
	template <class T> int get(T** q, size_t n)
	{
		const size_t bytes = sizeof(T) * std::max<size_t>(n, 1);
		if (alloc_refused(bytes) || cudaMallocAsync((void**)q, bytes, st) != cudaSuccess) {
			cudaGetLastError();
			set_error("set-up scratch of %zu bytes", sizeof(T) * n);
			return QPC_ERR_NOMEM;
		}
		ptr.push_back(*q);
		return QPC_OK;
	}
};

} // namespace qpc
