// The velocity-gauge step with diagonal radial couplings (qpc_vpos.cu), used by the engine (qpc_vgwr.cu) for the
// sizes where it is the faster one.
#pragma once
#include "qpc_internal.h"
#include <cuda_runtime.h>
#include <functional>

namespace qpc {

struct vpos_path;

struct vpos_setup {
	int N, P, nch, nlh, B, n_l, m0;
	double dt;
	const double *S, *D;		// device bands
	const double *Ri;		// host band <B|1/r|B>
	const int* chmap;		// host: engine channel -> im * n_l + il
	int off[2], na[2], nb[2];	// parity blocks: larger m-parity set first
	const double* tm[5][2][2];	// device, see qpc_vgwr.cu
	const double* lam[4];		// device, engine order
	double2 gam[4][2][2];
	double2* buf[2];		// two state-sized buffers of the caller's, used within a run only
	std::function<int(double2*, double2*, int, int)> fieldfree;	// on J vectors X[J][nlh][N]
	cudaStream_t stream;
};

// *out = nullptr with QPC_OK when the sizes or operators do not suit it
int vpos_create(const vpos_setup& in, vpos_path** out);
void vpos_destroy(vpos_path* p);
// digit planes of the dense transform and of the one back (0 or 1)
void vpos_report(const vpos_path* p, int32_t out[2]);

struct vpos_run {
	double2* X;		// [slot][nch][N], engine channel order, in and out
	const double* atab;	// device [inst][ld][2]
	long ld;
	const int* perm;	// device: slot -> instance
	const int64_t* ntt;	// device, by slot
	long* launches;
	std::function<void(int)> prof_begin, prof_end;	// kinds 0 transforms, 1 couplings (with a transform), 2 field-free
};
int vpos_begin(vpos_path* p, const vpos_run& r);
// step s: the first nlive slots in their pulse, the first nff running.  open: the live slots start in the l basis
// (else the last step left them before its closing x1 coupling); close: they end there
int vpos_step(vpos_path* p, const vpos_run& r, long s, int nlive, int nff, bool open, bool close);
// the B-spline coefficients of the first n slots before step s (all of them in the l basis) into r.X
int vpos_peek(vpos_path* p, const vpos_run& r, long s, int n);
int vpos_end(vpos_path* p, const vpos_run& r);
// after the stream has been waited for: an error if a wait in a kernel of the run ran out
int vpos_check(const vpos_path* p);

} // namespace qpc
