// The banded and dense products of qpc_radial.cu on the tensor cores (qpc_tcband.cu), for batches.
#pragma once
#include "qpc_radial.cuh"

namespace qpc {

// From the band Fb [nop][N][2 WMAX + 1] (complex), or a real matrix A(i, j) = A[op * sop + i * si + j * sj] of nrow x N;
// w: half-band, or -1 for a dense one; rows: each row under its own
// largest exponent in place of ea; kb, ke: the columns that take part (kb a multiple of 32).
// prof: largest |entry| per distance as in radial_create (NULL: every entry counts).  ok = false: an exact sum could
// exceed 2^24, the planes would take more than 4 GB or an eighth of the free memory, or there is no room for them (t is
// empty then, and the products go without).
int tc_make(tc_store& t, const double2* Fb, const double* A, long sop, long si, long sj, int nrow, int N, int nop, int w, const double* prof, int ea,
	bool rows, cudaStream_t st, bool* ok, int kb = 0, int ke = -1);

// the product of band_args a with the planes t (a.A, a.td, a.toff unused); status: device word or-ed with stbit when a
// wait ran out
void tc_apply(const tc_store& t, const band_args& a, int* status, int stbit, cudaStream_t st);
// microseconds it takes: twice the tensor-core math and 9 us of a block's own, one block per SM
double tc_cost(const tc_store& t, int nchan, int ncols);

} // namespace qpc
