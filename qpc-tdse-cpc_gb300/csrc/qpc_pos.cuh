// The length-gauge step in the position basis (qpc_pos.cu): the radial functions that are orthonormal in S
// and diagonalise R.  Used by the engine (qpc_engine.cu) for runs on handles whose operators fit it.
#pragma once
#include "qpc_internal.h"
#include <cuda_runtime.h>
#include <functional>

namespace qpc {

struct pos_path;

// what pos_create reads: device bands S, R [N][P+1], host eigenvector halves Vh [M][npair+1][L] and the
// positive eigenvalues lamp [M][npair]; nff sets of field-free operators (1, or one per instance).
// fieldfree(X, wk, J, fi) applies the field-free step of set fi for l = 0..nlh-1 to J vectors X[J][N][nlh]
// (r-major, wk scratch of the same size) on `stream`.
struct pos_setup {
	int dev, N, P, L, M, m0, B, nlh, npair, nff;
	double dt;
	const double *S, *R;
	const double *Vh, *lamp;
	std::function<int(double2*, double2*, int, int)> fieldfree;
	cudaStream_t stream;
};

// *out = nullptr with QPC_OK when the operators do not suit the path
int pos_create(const pos_setup& in, pos_path** out);
void pos_destroy(pos_path* p);
// its two state-sized buffers, which hold nothing between runs
void pos_buffers(const pos_path* p, double2* out[2]);
// digit planes of F~, W = X^T S and X (0 or 1), and the kernel of the last run's first field-free product (QPC_PRODUCT_*)
void pos_report(const pos_path* p, int32_t out[4]);

// one run: nothing is kept from one run to the next but buffers.
struct pos_run {
	double2* state;			// [B][M][L][N], the coefficients, in and out
	const int* perm;		// device [B]: slot k holds instance perm[k]
	const int64_t *ntf, *ntt;	// device [B], by slot
	const double* ftab;		// device [B][ld], by slot
	long ld;
	bool mask;			// the operator of pos_mask is applied after every step
	double* z;			// device [B][ldz], the dipole of f(r) = r before every step, or nullptr
	long ldz;
	int64_t* launches;
	int* status;			// device word, or-ed with stbit when a wait on the tensor cores ran out
	int stbit;
	std::function<void(int, cudaStream_t)> prof_begin, prof_end;	// per-kernel timing, or empty
	cudaStream_t stream;
};
// the operator of a run's mask (device band [N][P+1]), before pos_begin of that run; ok = false: it does not suit the
// fixed-point products
int pos_mask(pos_path* p, const double* mask, int64_t* launches, cudaStream_t st, bool* ok);
int pos_begin(pos_path* p, const pos_run& r);
// loop step s: Bc slots (a prefix) may couple, Bf slots (a prefix) may take the field-free step
int pos_step(pos_path* p, const pos_run& r, long s, int Bc, int Bf);
int pos_end(pos_path* p, const pos_run& r);

} // namespace qpc
