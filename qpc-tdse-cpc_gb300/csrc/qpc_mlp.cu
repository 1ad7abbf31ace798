// Ensemble MLP for the spectra surrogate: members x (n_in -> n_layers x n_hidden GELU
// -> n_out), trained with Adam on the GPU.  No counterpart in the reference.
//
// Numerics: weights and activations enter every product as bfloat16, products are
// accumulated in fp32 on the tensor cores (mma.sync m16n8k16 bf16 -> f32), biases,
// pre-activations, GELU, the loss gradient and the Adam state are fp32, and the
// master weights are fp32 (re-rounded to bf16 after each update).
//
// Every GEMM is C[M][N] = sum_k A[m][k] B[n][k] with both operands k-contiguous:
//   forward   Z = A W^T          A = activations [M][K],  B = W   [N][K]
//   input grad  dA = G W         A = G [M][N],            B = W^T [K][N]
//   weight grad dW = G^T A       A = G^T [N][M],          B = A^T [K][M]
// so each layer keeps its activations and gradients in both orientations, written
// by the epilogue of the kernel that produces them.  One launch covers all members
// (blockIdx.z).
#include "qpc_internal.h"
#include "qpc_cuda_util.cuh"
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cmath>
#include <cstdint>
#include <vector>
#include <algorithm>

namespace qpc {
namespace {

constexpr int MT = 64;           // block tile (rows and columns)
constexpr int KT = 64;           // k of a stage
constexpr int NSTG = 4;          // stages in flight
constexpr int PITCH = KT + 8;    // of a staged row: ldmatrix without bank conflicts
constexpr int MLP_THREADS = 256; // 8 warps, 2 x 4 warp tiles of 32 x 16
constexpr int MLP_SMEM = NSTG * 2 * MT * PITCH * (int)sizeof(__nv_bfloat16);

// what becomes of a product v (bias added)
enum {
	EPI_STORE = 0,   // out = v
	EPI_HIDDEN = 1,  // out = v, outb/outt = gelu(v)
	EPI_BACK = 2,    // outb/outt = v gelu'(aux), cs = sums over the tile's rows
	EPI_LOSS = 3     // d = v - aux on valid rows: outb/outt = 2 d scale, cs as above, part = the tile's sum of d^2
};

struct gemm_args {
	const __nv_bfloat16* A; long sA;  // [M][K] per member, member stride
	const __nv_bfloat16* B; long sB;  // [N][K]
	int M, N, K, epi;
	const float* bias; long sbias;    // [N] or null
	const float* aux; long saux;      // EPI_BACK: pre-activation Z [M][N]; EPI_LOSS: targets
	float* out; long sout;            // fp32 [M][N]
	__nv_bfloat16* outb; long soutb;  // bf16 [M][N]
	__nv_bfloat16* outt; long soutt;  // bf16 [N][M]
	float* cs; long scs;              // [ceil(M / MT)][N]
	const int* idx;                   // [E][M]: rows < 0 do not count
	float scale;
	float* part;                      // [E][tiles]
	__host__ __device__ int tiles() const { return ((M + MT - 1) / MT) * ((N + MT - 1) / MT); }
};

// the last stage of a reduction, a block of a backward launch: gb[n] = sum over the row tiles, in order; and the loss
struct sum_args {
	const float* cs; long scs;
	int nt, N;
	float* gb; long sgb;
	const float* part; int npart;     // null: no loss
	float scale;
	float* loss;
};

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float z)
{
	return 0.5f * (1.0f + erff(z * 0.70710678118654752f)) + z * 0.39894228040143268f * expf(-0.5f * z * z);
}

__device__ __forceinline__ uint32_t smem_at(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t a)
{
	asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}

// rows row0.. of X [nrow][K] into a stage, zero beyond the rows and beyond K (a multiple of 8)
__device__ __forceinline__ void stage_rows(__nv_bfloat16* to, const __nv_bfloat16* X, int row0, int nrow, int K, int k0)
{
#pragma unroll
	for (int i = 0; i < MT * KT / 8 / MLP_THREADS; ++i) {
		const int q = threadIdx.x + i * MLP_THREADS, r = q / (KT / 8), k = q % (KT / 8) * 8;
		const bool in = row0 + r < nrow && k0 + k < K;
		const __nv_bfloat16* src = in ? X + (long)(row0 + r) * K + k0 + k : X;
		asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_at(to + r * PITCH + k)), "l"(src), "r"(in ? 16 : 0) : "memory");
	}
}

// One 64 x 64 tile.  The products of the surrogate (256 x 256 x 256 per member) are bound by latency, not by the tensor
// cores: the whole K = 256 is in flight at once (16 dependent rounds of loads from global memory took 12-24 us a product,
// now 7).  Sums over rows leave as partial sums of the tile, the transposed copies through shared memory.  A gradient of
// five members on 256 rows: 26 launches and 1.00 ms before, 11 and 0.31 ms now, mostly the copies to and from the host.
__device__ void gemm_tile(const gemm_args& a, int tile, int e, __nv_bfloat16* sm)
{
	const int nbx = (a.N + MT - 1) / MT, m0 = tile / nbx * MT, n0 = tile % nbx * MT;
	const __nv_bfloat16* A = a.A + e * a.sA;
	const __nv_bfloat16* B = a.B + e * a.sB;
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
	const int wm = (warp >> 2) * 32, wn = (warp & 3) * 16;
	const int nk = (a.K + KT - 1) / KT;
	auto stage = [&](int t) {
		if (t < nk) {
			__nv_bfloat16* to = sm + (t % NSTG) * 2 * MT * PITCH;
			stage_rows(to, A, m0, a.M, a.K, t * KT);
			stage_rows(to + MT * PITCH, B, n0, a.N, a.K, t * KT);
		}
		asm volatile("cp.async.commit_group;\n" ::: "memory");
	};
	for (int t = 0; t < NSTG; ++t) stage(t);
	float acc[2][2][4];
#pragma unroll
	for (int i = 0; i < 2; ++i)
#pragma unroll
		for (int j = 0; j < 2; ++j)
#pragma unroll
			for (int c = 0; c < 4; ++c) acc[i][j][c] = 0.f;
	for (int t = 0; t < nk; ++t) {
		asm volatile("cp.async.wait_group %0;\n" ::"n"(NSTG - 1) : "memory");
		__syncthreads();
		const __nv_bfloat16* As = sm + (t % NSTG) * 2 * MT * PITCH;
		const uint32_t aa = smem_at(As + (wm + (lane & 15)) * PITCH + (lane >> 4) * 8);
		const uint32_t ba = smem_at(As + (MT + wn + (lane & 7) + ((lane >> 4) << 3)) * PITCH + ((lane >> 3) & 1) * 8);
#pragma unroll
		for (int k = 0; k < KT; k += 16) {
			uint32_t af[2][4], bf[4];
			ldmatrix4(af[0], aa + k * 2);
			ldmatrix4(af[1], aa + (16 * PITCH + k) * 2);
			ldmatrix4(bf, ba + k * 2);
#pragma unroll
			for (int i = 0; i < 2; ++i)
#pragma unroll
				for (int j = 0; j < 2; ++j)
					asm volatile(
						"mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
						: "+f"(acc[i][j][0]), "+f"(acc[i][j][1]), "+f"(acc[i][j][2]), "+f"(acc[i][j][3])
						: "r"(af[i][0]), "r"(af[i][1]), "r"(af[i][2]), "r"(af[i][3]), "r"(bf[2 * j]), "r"(bf[2 * j + 1]));
		}
		__syncthreads();
		stage(t + NSTG);
	}
	// acc[i][j][c] is C(row, col) with row = m0 + wm + 16 i + gid + 8 (c >> 1), col = n0 + wn + 8 j + 2 tig + (c & 1);
	// N is a multiple of 8: a pair of columns is inside or outside
	asm volatile("cp.async.wait_group 0;\n" ::: "memory");
	__nv_bfloat16* T = sm;	// [64][PITCH], bf16 results
	float* cs = reinterpret_cast<float*>(sm + MT * PITCH);	// [2][64] column sums, then 8 sums of squares
	float sq = 0.f;
#pragma unroll
	for (int j = 0; j < 2; ++j) {
		const int lc = wn + 8 * j + 2 * tig, col = n0 + lc;
		float s0 = 0.f, s1 = 0.f;
#pragma unroll
		for (int i = 0; i < 2; ++i)
#pragma unroll
			for (int c = 0; c < 4; c += 2) {
				const int lr = wm + 16 * i + gid + 4 * c, row = m0 + lr;
				if (row >= a.M || col >= a.N) continue;
				float v0 = acc[i][j][c], v1 = acc[i][j][c + 1];
				const long o = (long)row * a.N + col;
				if (a.bias) { v0 += a.bias[e * a.sbias + col]; v1 += a.bias[e * a.sbias + col + 1]; }
				if (a.epi <= EPI_HIDDEN) *reinterpret_cast<float2*>(a.out + e * a.sout + o) = make_float2(v0, v1);
				if (a.epi == EPI_HIDDEN) { v0 = gelu(v0); v1 = gelu(v1); }
				if (a.epi >= EPI_BACK) {
					const float2 x = *reinterpret_cast<const float2*>(a.aux + e * a.saux + o);
					if (a.epi == EPI_BACK) { v0 *= gelu_grad(x.x); v1 *= gelu_grad(x.y); }
					else {
						const bool valid = a.idx[(long)e * a.M + row] >= 0;
						v0 = valid ? v0 - x.x : 0.f;
						v1 = valid ? v1 - x.y : 0.f;
						sq += v0 * v0 + v1 * v1;
						v0 = 2.f * v0 * a.scale;
						v1 = 2.f * v1 * a.scale;
					}
					s0 += v0;
					s1 += v1;
				}
				if (a.epi) *reinterpret_cast<__nv_bfloat162*>(T + lr * PITCH + lc) = __floats2bfloat162_rn(v0, v1);
			}
		if (a.epi >= EPI_BACK) {
#pragma unroll
			for (int o = 4; o < 32; o <<= 1) { s0 += __shfl_xor_sync(0xffffffffu, s0, o); s1 += __shfl_xor_sync(0xffffffffu, s1, o); }
			if (gid == 0) { cs[(warp >> 2) * 64 + lc] = s0; cs[(warp >> 2) * 64 + lc + 1] = s1; }
		}
	}
	if (a.epi == EPI_STORE) return;
	if (a.epi == EPI_LOSS) {
#pragma unroll
		for (int o = 16; o; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
		if (lane == 0) cs[128 + warp] = sq;
	}
	__syncthreads();
	for (int q = threadIdx.x; q < MT * MT / 8; q += MLP_THREADS) {
		const int r = q / (MT / 8), x = q % (MT / 8) * 8;
		if (m0 + r < a.M && n0 + x < a.N)
			*reinterpret_cast<uint4*>(a.outb + e * a.soutb + (long)(m0 + r) * a.N + n0 + x) = *reinterpret_cast<const uint4*>(T + r * PITCH + x);
		// transposed: column r of the tile, rows x .. x + 7 (M is a multiple of 64)
		if (n0 + r < a.N) {
			uint32_t w[4];
#pragma unroll
			for (int i = 0; i < 4; ++i) {
				const uint16_t lo = *reinterpret_cast<const uint16_t*>(T + (x + 2 * i) * PITCH + r), hi = *reinterpret_cast<const uint16_t*>(T + (x + 2 * i + 1) * PITCH + r);
				w[i] = lo | (uint32_t)hi << 16;
			}
			*reinterpret_cast<uint4*>(a.outt + e * a.soutt + (long)(n0 + r) * a.M + m0 + x) = make_uint4(w[0], w[1], w[2], w[3]);
		}
	}
	if (a.epi >= EPI_BACK && threadIdx.x < MT && n0 + threadIdx.x < a.N)
		a.cs[e * a.scs + (long)(m0 / MT) * a.N + n0 + threadIdx.x] = cs[threadIdx.x] + cs[64 + threadIdx.x];
	if (a.epi == EPI_LOSS && threadIdx.x == 0) {
		float t = 0.f;
		for (int w = 0; w < MLP_THREADS / 32; ++w) t += cs[128 + w];
		a.part[(long)e * a.tiles() + tile] = t;
	}
}

__global__ void __launch_bounds__(MLP_THREADS) k_mlp_gemm(const gemm_args a)
{
	extern __shared__ __align__(16) __nv_bfloat16 mlp_sm[];
	gemm_tile(a, blockIdx.x, blockIdx.z, mlp_sm);
}

// one layer backwards: the tiles of the weight gradient, those of the input gradient (na of them, 0 for the first layer),
// and the bias gradient (with the loss), none of which waits for another
__global__ void __launch_bounds__(MLP_THREADS) k_mlp_back(const gemm_args w, const gemm_args a, const sum_args s, int nw, int na)
{
	extern __shared__ __align__(16) __nv_bfloat16 mlp_sm[];
	const int e = blockIdx.z, t = blockIdx.x;
	if (t < nw) gemm_tile(w, t, e, mlp_sm);
	else if (t < nw + na) gemm_tile(a, t - nw, e, mlp_sm);
	else {
		const int n = (t - nw - na) * MLP_THREADS + threadIdx.x;
		if (n < s.N) {
			float v = 0.f;
			for (int i = 0; i < s.nt; ++i) v += s.cs[e * s.scs + (long)i * s.N + n];
			s.gb[e * s.sgb + n] = v;
		}
		if (s.part && t == nw + na && threadIdx.x < 32) {
			double v = 0.0;
			for (int i = threadIdx.x; i < s.npart; i += 32) v += s.part[(long)e * s.npart + i];
			for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
			if (threadIdx.x == 0) s.loss[e] = (float)(v * s.scale);
		}
	}
}

// rows of the dataset into the first layer's input (bf16, zero-padded to K0, both
// orientations) and the targets; idx < 0 marks a padding row (zero input, no loss)
__global__ void k_mlp_gather(const float* __restrict__ X, const float* __restrict__ Y, const int* __restrict__ idx,
	int n_in, int K0, int n_out, int M, __nv_bfloat16* A0, __nv_bfloat16* A0t, float* Yb)
{
	const int e = blockIdx.y;
	const int m = blockIdx.x;
	const int id = idx[e * M + m];
	for (int k = threadIdx.x; k < K0; k += blockDim.x) {
		float v = (id >= 0 && k < n_in) ? X[(long)id * n_in + k] : 0.f;
		__nv_bfloat16 b = __float2bfloat16_rn(v);
		A0[((long)e * M + m) * K0 + k] = b;
		A0t[((long)e * K0 + k) * M + m] = b;
	}
	if (Y)
		for (int k = threadIdx.x; k < n_out; k += blockDim.x) Yb[((long)e * M + m) * n_out + k] = id >= 0 ? Y[(long)id * n_out + k] : 0.f;
}

// Adam (Kingma & Ba 2015) on the fp32 masters of one member's parameters, then the
// bf16 copies of the weights in both orientations
struct adam_layer {
	float *W, *b, *gW, *gb, *mW, *vW, *mb, *vb;
	__nv_bfloat16 *Wb, *Wt;
	int N, K;
};

__global__ void k_mlp_adam(adam_layer L, long sW, long sb, long sg, float lr, float b1, float b2, float c1, float c2, float eps)
{
	const int e = blockIdx.y;
	const long nw = (long)L.N * L.K;
	for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < nw + L.N; i += (long)gridDim.x * blockDim.x) {
		const bool isw = i < nw;
		float* p = isw ? L.W + e * sW + i : L.b + e * sb + (i - nw);
		const float g = isw ? L.gW[e * sg + i] : L.gb[e * sg + (i - nw)];
		float* m = isw ? L.mW + e * sW + i : L.mb + e * sb + (i - nw);
		float* v = isw ? L.vW + e * sW + i : L.vb + e * sb + (i - nw);
		float mm = b1 * *m + (1.f - b1) * g;
		float vv = b2 * *v + (1.f - b2) * g * g;
		*m = mm;
		*v = vv;
		float w = *p - lr * (mm / c1) / (sqrtf(vv / c2) + eps);
		*p = w;
		if (isw) {
			int n = (int)(i / L.K), k = (int)(i - (long)n * L.K);
			__nv_bfloat16 b = __float2bfloat16_rn(w);
			L.Wb[e * sW + i] = b;
			L.Wt[e * sW + (long)k * L.N + n] = b;
		}
	}
}

__global__ void k_mlp_cast(const float* __restrict__ W, int N, int K, long sW, __nv_bfloat16* Wb, __nv_bfloat16* Wt)
{
	const int e = blockIdx.y;
	const long nw = (long)N * K;
	for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < nw; i += (long)gridDim.x * blockDim.x) {
		int n = (int)(i / K), k = (int)(i - (long)n * K);
		__nv_bfloat16 b = __float2bfloat16_rn(W[e * sW + i]);
		Wb[e * sW + i] = b;
		Wt[e * sW + (long)k * N + n] = b;
	}
}

} // namespace
} // namespace qpc

using namespace qpc;

struct qpc_mlp {
	int dev = 0;
	int n_in = 0, K0 = 0, n_hidden = 0, n_layers = 0, n_out = 0, E = 0, J = 0;
	std::vector<int> Ns, Ks;          // per linear layer j: out, in
	std::vector<long> offW, offb;     // offsets of layer j in the per-member flat arrays
	std::vector<long> goff;           // of its weights in the gradient [E][nW + nb] (W_0, b_0, W_1, ..): the caller's layout
	long nW = 0, nb = 0;              // per-member totals
	cudaStream_t st = nullptr;
	float *W = nullptr, *b = nullptr, *grad = nullptr, *mW = nullptr, *vW = nullptr, *mb = nullptr, *vb = nullptr;
	__nv_bfloat16 *Wb = nullptr, *Wt = nullptr;
	long t = 0;                       // Adam step count
	// batch work space (capacity M)
	int Mcap = 0;
	std::vector<__nv_bfloat16*> Act, ActT;  // layer inputs j = 0..J-1: [E][M][K_j] and [E][K_j][M]
	std::vector<float*> Z;                  // pre-activations of hidden layers [E][M][N_j]
	float *Yh = nullptr, *Yb = nullptr, *part = nullptr, *loss = nullptr;
	__nv_bfloat16 *Gb[2] = {}, *Gt[2] = {}; // a layer's output gradient and the one below it, in turn
	float* cs[2] = {};                      // their sums over 64 rows
	int* idx = nullptr;
	// dataset on the device
	float *dX = nullptr, *dY = nullptr;
	long dcap = 0;
};

namespace {

void mlp_free_batch(qpc_mlp* h)
{
	for (auto p : h->Act) cudaFree(p);
	for (auto p : h->ActT) cudaFree(p);
	for (auto p : h->Z) cudaFree(p);
	h->Act.clear(); h->ActT.clear(); h->Z.clear();
	void* ps[] = {h->Yh, h->Yb, h->part, h->loss, h->Gb[0], h->Gb[1], h->Gt[0], h->Gt[1], h->cs[0], h->cs[1], h->idx};
	for (void* p : ps) if (p) cudaFree(p);
	h->Yh = h->Yb = h->part = h->loss = nullptr;
	for (int i = 0; i < 2; ++i) { h->Gb[i] = h->Gt[i] = nullptr; h->cs[i] = nullptr; }
	h->idx = nullptr;
	h->Mcap = 0;
}

void mlp_free(qpc_mlp* h)
{
	if (!h) return;
	cudaSetDevice(h->dev);
	mlp_free_batch(h);
	void* ps[] = {h->W, h->b, h->grad, h->mW, h->vW, h->mb, h->vb, h->Wb, h->Wt, h->dX, h->dY};
	for (void* p : ps) if (p) cudaFree(p);
	if (h->st) cudaStreamDestroy(h->st);
	delete h;
}

// every kernel of a pass works on exactly Mcap rows (padding rows carry idx < 0)
int ensure_batch(qpc_mlp* h, int M)
{
	if (M == h->Mcap) return QPC_OK;
	mlp_free_batch(h);
	const int E = h->E, J = h->J;
	int rc = 0;
	h->Act.assign(J, nullptr); h->ActT.assign(J, nullptr); h->Z.assign(J, nullptr);
	for (int j = 0; j < J; ++j) {
		if ((rc = dalloc(&h->Act[j], (size_t)E * M * h->Ks[j])) || (rc = dalloc(&h->ActT[j], (size_t)E * M * h->Ks[j]))) return rc;
		if (j < J - 1 && (rc = dalloc(&h->Z[j], (size_t)E * M * h->Ns[j]))) return rc;
	}
	const int maxN = *std::max_element(h->Ns.begin(), h->Ns.end());
	if ((rc = dalloc(&h->Yh, (size_t)E * M * h->n_out)) || (rc = dalloc(&h->Yb, (size_t)E * M * h->n_out)) ||
		(rc = dalloc(&h->part, (size_t)E * (M / MT) * ((h->n_out + MT - 1) / MT))) || (rc = dalloc(&h->loss, (size_t)E)) ||
		(rc = dalloc(&h->idx, (size_t)E * M)))
		return rc;
	for (int i = 0; i < 2; ++i)
		if ((rc = dalloc(&h->Gb[i], (size_t)E * M * maxN)) || (rc = dalloc(&h->Gt[i], (size_t)E * M * maxN)) || (rc = dalloc(&h->cs[i], (size_t)E * (M / MT) * maxN)))
			return rc;
	h->Mcap = M;
	return QPC_OK;
}

gemm_args product(int epi, const __nv_bfloat16* A, long sA, const __nv_bfloat16* B, long sB, int M, int N, int K)
{
	gemm_args a{};
	a.A = A; a.sA = sA; a.B = B; a.sB = sB; a.M = M; a.N = N; a.K = K; a.epi = epi;
	return a;
}

// forward of the Mcap rows gathered into Act[0]; the output into Yh, or with Mvalid > 0 the loss gradient of that many
// rows into G[0] (and its partial sums)
void forward(qpc_mlp* h, int Mvalid)
{
	const int E = h->E, J = h->J, M = h->Mcap;
	const int maxN = *std::max_element(h->Ns.begin(), h->Ns.end());
	for (int j = 0; j < J; ++j) {
		const int N = h->Ns[j], K = h->Ks[j];
		const bool last = j == J - 1;
		gemm_args a = product(!last ? EPI_HIDDEN : Mvalid ? EPI_LOSS : EPI_STORE, h->Act[j], (long)M * K, h->Wb + h->offW[j], h->nW, M, N, K);
		a.bias = h->b + h->offb[j]; a.sbias = h->nb;
		a.out = last ? h->Yh : h->Z[j]; a.sout = (long)M * N;
		if (!last) {
			a.outb = h->Act[j + 1]; a.outt = h->ActT[j + 1];
			a.soutb = a.soutt = (long)M * N;
		} else {
			a.outb = h->Gb[0]; a.outt = h->Gt[0]; a.cs = h->cs[0];
			a.soutb = a.soutt = (long)M * maxN;
			a.scs = (long)(M / MT) * maxN;
			a.aux = h->Yb; a.saux = (long)M * N; a.idx = h->idx; a.part = h->part;
			a.scale = 1.0f / ((float)std::max(Mvalid, 1) * (float)h->n_out);
		}
		k_mlp_gemm<<<dim3(a.tiles(), 1, E), MLP_THREADS, MLP_SMEM, h->st>>>(a);
	}
}

// gradients and loss after forward(h, Mvalid)
void backward(qpc_mlp* h, int Mvalid)
{
	const int E = h->E, J = h->J, M = h->Mcap, nt = M / MT;
	const int maxN = *std::max_element(h->Ns.begin(), h->Ns.end());
	const long sg = (long)M * maxN, np = h->nW + h->nb;
	for (int j = J - 1, g = 0; j >= 0; --j, g = 1 - g) {
		const int N = h->Ns[j], K = h->Ks[j];
		// gW_j[n][k] = sum_m G[m][n] A_j[m][k]: A = G^T [N][M], B = A_j^T [K][M]
		gemm_args w = product(EPI_STORE, h->Gt[g], sg, h->ActT[j], (long)M * K, N, K, M), a{};
		w.out = h->grad + h->goff[j]; w.sout = np;
		if (j > 0) {
			// dA[m][k] = sum_n G[m][n] W[n][k]: A = G [M][N], B = W^T [K][N]; times gelu'(Z_{j-1})
			a = product(EPI_BACK, h->Gb[g], sg, h->Wt + h->offW[j], h->nW, M, K, N);
			a.aux = h->Z[j - 1]; a.saux = (long)M * K;
			a.outb = h->Gb[1 - g]; a.outt = h->Gt[1 - g]; a.soutb = a.soutt = sg;
			a.cs = h->cs[1 - g]; a.scs = (long)nt * maxN;
		}
		sum_args s{h->cs[g], (long)nt * maxN, nt, N, h->grad + h->goff[j] + (long)N * K, np, nullptr, 0, 0.f, h->loss};
		if (j == J - 1) {
			s.part = h->part; s.npart = nt * ((h->n_out + MT - 1) / MT);
			s.scale = 1.0f / ((float)Mvalid * (float)h->n_out);
		}
		const int nw = w.tiles(), na = j > 0 ? a.tiles() : 0;
		k_mlp_back<<<dim3(nw + na + (N + MLP_THREADS - 1) / MLP_THREADS, 1, E), MLP_THREADS, MLP_SMEM, h->st>>>(w, a, s, nw, na);
	}
}

void adam(qpc_mlp* h, float lr)
{
	const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
	h->t += 1;
	const float c1 = 1.f - powf(b1, (float)h->t), c2 = 1.f - powf(b2, (float)h->t);
	for (int j = 0; j < h->J; ++j) {
		adam_layer L{h->W + h->offW[j], h->b + h->offb[j], h->grad + h->goff[j], h->grad + h->goff[j] + (long)h->Ns[j] * h->Ks[j], h->mW + h->offW[j], h->vW + h->offW[j],
			h->mb + h->offb[j], h->vb + h->offb[j], h->Wb + h->offW[j], h->Wt + h->offW[j], h->Ns[j], h->Ks[j]};
		long n = (long)h->Ns[j] * h->Ks[j] + h->Ns[j];
		int blocks = (int)std::min<long>((n + 255) / 256, 1024);
		k_mlp_adam<<<dim3(blocks, h->E), 256, 0, h->st>>>(L, h->nW, h->nb, h->nW + h->nb, lr, b1, b2, c1, c2, eps);
	}
}

void cast_all(qpc_mlp* h)
{
	for (int j = 0; j < h->J; ++j) {
		long nw = (long)h->Ns[j] * h->Ks[j];
		k_mlp_cast<<<dim3((int)std::min<long>((nw + 255) / 256, 1024), h->E), 256, 0, h->st>>>(h->W + h->offW[j], h->Ns[j], h->Ks[j],
			h->nW, h->Wb + h->offW[j], h->Wt + h->offW[j]);
	}
}

// splitmix64 (Steele, Lea and Flood 2014) for the initial weights
uint64_t splitmix(uint64_t& s)
{
	uint64_t z = (s += 0x9E3779B97F4A7C15ull);
	z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
	z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
	return z ^ (z >> 31);
}

int upload_data(qpc_mlp* h, const float* X, const float* Y, long n)
{
	if (n > h->dcap) {
		if (h->dX) cudaFree(h->dX);
		if (h->dY) cudaFree(h->dY);
		h->dX = h->dY = nullptr; h->dcap = 0;
		int rc;
		if ((rc = dalloc(&h->dX, (size_t)n * h->n_in)) || (rc = dalloc(&h->dY, (size_t)n * h->n_out))) return rc;
		h->dcap = n;
	}
	QPC_CUDA(cudaMemcpyAsync(h->dX, X, sizeof(float) * n * h->n_in, cudaMemcpyHostToDevice, h->st));
	if (Y) QPC_CUDA(cudaMemcpyAsync(h->dY, Y, sizeof(float) * n * h->n_out, cudaMemcpyHostToDevice, h->st));
	return QPC_OK;
}

int round_m(int m) { return (m + MT - 1) / MT * MT; }

} // namespace

extern "C" {

int qpc_mlp_create(int32_t n_in, int32_t n_hidden, int32_t n_layers, int32_t n_out, int32_t n_members, uint64_t seed, qpc_mlp** out)
{
	if (!out) { set_error("out is NULL"); return QPC_ERR_ARGS; }
	*out = nullptr;
	if (n_in < 1 || n_hidden < 16 || n_hidden % 16 || n_layers < 1 || n_out < 8 || n_out % 8 || n_members < 1 || n_members > 64) {
		set_error("bad MLP shape n_in=%d n_hidden=%d n_layers=%d n_out=%d members=%d (hidden a multiple of 16, out of 8)",
			n_in, n_hidden, n_layers, n_out, n_members);
		return QPC_ERR_ARGS;
	}
	int dev = 0;
	if (int rc = check_device(&dev)) return rc;
	qpc_mlp* h = new (std::nothrow) qpc_mlp;
	if (!h) { set_error("host allocation"); return QPC_ERR_NOMEM; }
	auto fail = [&](int rc) { mlp_free(h); return rc; };
	h->dev = dev;
	h->n_in = n_in; h->K0 = (n_in + 15) / 16 * 16; h->n_hidden = n_hidden; h->n_layers = n_layers; h->n_out = n_out;
	h->E = n_members; h->J = n_layers + 1;
	for (int j = 0; j < h->J; ++j) {
		h->Ks.push_back(j == 0 ? h->K0 : n_hidden);
		h->Ns.push_back(j == h->J - 1 ? n_out : n_hidden);
		h->offW.push_back(h->nW);
		h->offb.push_back(h->nb);
		h->goff.push_back(h->nW + h->nb);
		h->nW += (long)h->Ns[j] * h->Ks[j];
		h->nb += h->Ns[j];
	}
	if ((cudaStreamCreateWithFlags(&h->st, cudaStreamNonBlocking)) != cudaSuccess) { set_error("cudaStreamCreateWithFlags failed"); return fail(QPC_ERR_CUDA); }
	const size_t tw = (size_t)h->E * h->nW, tb = (size_t)h->E * h->nb;
	int rc;
	if ((rc = dalloc(&h->W, tw)) || (rc = dalloc(&h->b, tb)) || (rc = dalloc(&h->grad, tw + tb)) ||
		(rc = dalloc(&h->mW, tw)) || (rc = dalloc(&h->vW, tw)) || (rc = dalloc(&h->mb, tb)) || (rc = dalloc(&h->vb, tb)) ||
		(rc = dalloc(&h->Wb, tw)) || (rc = dalloc(&h->Wt, tw)))
		return fail(rc);
	// He-uniform weights (bound sqrt(6 / fan_in), fan_in = the unpadded inputs), zero biases
	std::vector<float> W(tw, 0.f);
	uint64_t sd = seed;
	for (int e = 0; e < h->E; ++e)
		for (int j = 0; j < h->J; ++j) {
			const int fan = j == 0 ? n_in : h->Ks[j];
			const float bound = std::sqrt(6.0f / (float)fan);
			for (int nn = 0; nn < h->Ns[j]; ++nn)
				for (int k = 0; k < h->Ks[j]; ++k) {
					double u = (double)(splitmix(sd) >> 11) * (1.0 / 9007199254740992.0);
					W[(size_t)e * h->nW + h->offW[j] + (size_t)nn * h->Ks[j] + k] = (j == 0 && k >= n_in) ? 0.f : (float)((2.0 * u - 1.0) * bound);
				}
		}
	if (cudaMemcpyAsync(h->W, W.data(), sizeof(float) * tw, cudaMemcpyHostToDevice, h->st) != cudaSuccess ||
		cudaMemsetAsync(h->b, 0, sizeof(float) * tb, h->st) != cudaSuccess || cudaMemsetAsync(h->mW, 0, sizeof(float) * tw, h->st) != cudaSuccess ||
		cudaMemsetAsync(h->vW, 0, sizeof(float) * tw, h->st) != cudaSuccess || cudaMemsetAsync(h->mb, 0, sizeof(float) * tb, h->st) != cudaSuccess ||
		cudaMemsetAsync(h->vb, 0, sizeof(float) * tb, h->st) != cudaSuccess) {
		set_error("device upload failed");
		return fail(QPC_ERR_CUDA);
	}
	cudaFuncSetAttribute(k_mlp_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, MLP_SMEM);
	cudaFuncSetAttribute(k_mlp_back, cudaFuncAttributeMaxDynamicSharedMemorySize, MLP_SMEM);
	cast_all(h);
	if (cudaGetLastError() != cudaSuccess) { set_error("cast failed"); return fail(QPC_ERR_CUDA); }
	if (int rc2 = wait_on(h->st)) return fail(rc2);
	*out = h;
	return QPC_OK;
}

int qpc_mlp_destroy(qpc_mlp* h)
{
	mlp_free(h);
	return QPC_OK;
}

int qpc_mlp_param_count(qpc_mlp* h, int64_t* n)
{
	if (!h || !n) { set_error("NULL argument"); return QPC_ERR_ARGS; }
	*n = h->nW + h->nb;
	return QPC_OK;
}

// flat fp32 parameters of one member: W_0 [N][K0] (K0 = n_in rounded up to 16, padding
// columns ignored on set and zero on get), b_0, W_1, b_1, ...
static int params_io(qpc_mlp* h, int32_t member, float* host, bool get)
{
	if (!h || !host || member < 0 || member >= h->E) { set_error("bad arguments"); return QPC_ERR_ARGS; }
	cudaSetDevice(h->dev);
	if (int rc = wait_on(h->st)) return rc;
	std::vector<std::vector<float>> w(h->J);
	long o = 0;
	for (int j = 0; j < h->J; ++j) {
		const size_t nw = (size_t)h->Ns[j] * h->Ks[j];
		float* dW = h->W + (size_t)member * h->nW + h->offW[j];
		float* db = h->b + (size_t)member * h->nb + h->offb[j];
		if (get) {
			if (int rc = copy_to_host(host + o, dW, sizeof(float) * nw, h->st)) return rc;
			if (int rc = copy_to_host(host + o + nw, db, sizeof(float) * h->Ns[j], h->st)) return rc;
		} else {
			w[j].assign(host + o, host + o + nw);	// kept until the copies are done
			if (j == 0)
				for (int nn = 0; nn < h->Ns[j]; ++nn)
					for (int k = h->n_in; k < h->K0; ++k) w[j][(size_t)nn * h->K0 + k] = 0.f;
			QPC_CUDA(cudaMemcpyAsync(dW, w[j].data(), sizeof(float) * nw, cudaMemcpyHostToDevice, h->st));
			QPC_CUDA(cudaMemcpyAsync(db, host + o + nw, sizeof(float) * h->Ns[j], cudaMemcpyHostToDevice, h->st));
		}
		o += nw + h->Ns[j];
	}
	if (!get) {
		cast_all(h);
		QPC_CUDA(cudaGetLastError());
		if (int rc = wait_on(h->st)) return rc;
	}
	return QPC_OK;
}

int qpc_mlp_get_params(qpc_mlp* h, int32_t member, float* params) { return params_io(h, member, params, true); }
int qpc_mlp_set_params(qpc_mlp* h, int32_t member, const float* params) { return params_io(h, member, const_cast<float*>(params), false); }

// loss and gradient of every member on the same n rows (no update); grad [members][param_count]
int qpc_mlp_loss_grad(qpc_mlp* h, const float* X, const float* Y, int32_t n, float* loss, float* grad)
{
	if (!h || !X || !Y || !loss || n < 1) { set_error("bad arguments"); return QPC_ERR_ARGS; }
	cudaSetDevice(h->dev);
	const int M = round_m(n);
	if (int rc = ensure_batch(h, M)) return rc;
	if (int rc = upload_data(h, X, Y, n)) return rc;
	std::vector<int> idx((size_t)h->E * h->Mcap, -1);
	for (int e = 0; e < h->E; ++e)
		for (int m = 0; m < n; ++m) idx[(size_t)e * h->Mcap + m] = m;
	QPC_CUDA(cudaMemcpyAsync(h->idx, idx.data(), sizeof(int) * idx.size(), cudaMemcpyHostToDevice, h->st));
	k_mlp_gather<<<dim3(M, h->E), 64, 0, h->st>>>(h->dX, h->dY, h->idx, h->n_in, h->K0, h->n_out, M, h->Act[0], h->ActT[0], h->Yb);
	forward(h, n);
	backward(h, n);
	QPC_CUDA(cudaGetLastError());
	if (int rc = copy_to_host(loss, h->loss, sizeof(float) * h->E, h->st)) return rc;
	if (grad) return copy_to_host(grad, h->grad, sizeof(float) * (size_t)h->E * (h->nW + h->nb), h->st);
	return QPC_OK;
}

// epochs of Adam over n rows in batches; every member sees its own shuffle (seeded)
// of all rows.  loss_hist [epochs][members] (may be NULL): mean batch loss per epoch.
int qpc_mlp_train(qpc_mlp* h, const float* X, const float* Y, int32_t n, int32_t epochs, int32_t batch, float lr, uint64_t seed,
	float* loss_hist)
{
	if (!h || !X || !Y || n < 1 || epochs < 0 || batch < 1 || !(lr > 0)) { set_error("bad arguments"); return QPC_ERR_ARGS; }
	cudaSetDevice(h->dev);
	const int M = round_m(std::min(batch, n));
	if (int rc = ensure_batch(h, M)) return rc;
	if (int rc = upload_data(h, X, Y, n)) return rc;
	const int nbat = (n + batch - 1) / batch;
	std::vector<int> perm((size_t)h->E * n), idx((size_t)h->E * h->Mcap);
	std::vector<float> lsum(h->E), lb(h->E);
	uint64_t sd = seed;
	int rc = QPC_OK;
	for (int ep = 0; ep < epochs && !rc; ++ep) {
		for (int e = 0; e < h->E; ++e) {
			int* p = perm.data() + (size_t)e * n;
			for (int i = 0; i < n; ++i) p[i] = i;
			for (int i = n - 1; i > 0; --i) std::swap(p[i], p[splitmix(sd) % (uint64_t)(i + 1)]);
		}
		std::fill(lsum.begin(), lsum.end(), 0.f);
		for (int bi = 0; bi < nbat && !rc; ++bi) {
			const int m0 = bi * batch, mv = std::min(batch, n - m0);
			for (int e = 0; e < h->E; ++e)
				for (int m = 0; m < h->Mcap; ++m) idx[(size_t)e * h->Mcap + m] = m < mv ? perm[(size_t)e * n + m0 + m] : -1;
			if (cudaMemcpyAsync(h->idx, idx.data(), sizeof(int) * idx.size(), cudaMemcpyHostToDevice, h->st) != cudaSuccess) { rc = QPC_ERR_CUDA; break; }
			k_mlp_gather<<<dim3(M, h->E), 64, 0, h->st>>>(h->dX, h->dY, h->idx, h->n_in, h->K0, h->n_out, M, h->Act[0], h->ActT[0], h->Yb);
			forward(h, mv);
			backward(h, mv);
			adam(h, lr);
			if (loss_hist) {
				if ((rc = copy_to_host(lb.data(), h->loss, sizeof(float) * h->E, h->st))) break;
				for (int e = 0; e < h->E; ++e) lsum[e] += lb[e] / nbat;
			}
		}
		if (loss_hist) for (int e = 0; e < h->E; ++e) loss_hist[(size_t)ep * h->E + e] = lsum[e];
	}
	if (!rc && cudaGetLastError() != cudaSuccess) { rc = QPC_ERR_CUDA; set_error("training step failed on the device"); }
	if (!rc) rc = wait_on(h->st);
	return rc;
}

// every member's prediction for n rows: out [members][n][n_out]
int qpc_mlp_predict(qpc_mlp* h, const float* X, int32_t n, float* out)
{
	if (!h || !X || !out || n < 0) { set_error("bad arguments"); return QPC_ERR_ARGS; }
	if (n == 0) return QPC_OK;
	cudaSetDevice(h->dev);
	const int M = round_m(std::min(1024, n));
	if (int rc = ensure_batch(h, M)) return rc;
	if (int rc = upload_data(h, X, nullptr, n)) return rc;
	std::vector<int> idx((size_t)h->E * h->Mcap);
	std::vector<float> yh((size_t)h->E * h->Mcap * h->n_out);
	for (int m0 = 0; m0 < n; m0 += h->Mcap) {
		const int mv = std::min(h->Mcap, n - m0);
		for (int e = 0; e < h->E; ++e)
			for (int m = 0; m < h->Mcap; ++m) idx[(size_t)e * h->Mcap + m] = m < mv ? m0 + m : -1;
		QPC_CUDA(cudaMemcpyAsync(h->idx, idx.data(), sizeof(int) * idx.size(), cudaMemcpyHostToDevice, h->st));
		k_mlp_gather<<<dim3(M, h->E), 64, 0, h->st>>>(h->dX, nullptr, h->idx, h->n_in, h->K0, h->n_out, M, h->Act[0], h->ActT[0], nullptr);
		forward(h, 0);
		QPC_CUDA(cudaGetLastError());
		if (int rc = copy_to_host(yh.data(), h->Yh, sizeof(float) * yh.size(), h->st)) return rc;
		for (int e = 0; e < h->E; ++e)
			for (int m = 0; m < mv; ++m)
				std::copy(yh.begin() + ((size_t)e * h->Mcap + m) * h->n_out, yh.begin() + ((size_t)e * h->Mcap + m + 1) * h->n_out,
					out + ((size_t)e * n + m0 + m) * h->n_out);
	}
	return QPC_OK;
}

} // extern "C"
