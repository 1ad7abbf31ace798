// Products of fixed operators with batches of columns on the tcgen05 tensor cores, exactly as sums of digits.
//
// An operator entry and a column element are 56-bit integers under 2^ea and under the column's largest exponent (as in
// qpc_radial.cu), written as 7 balanced digits of 8 bits, which bf16 holds exactly.  The products of digit s of the
// operator with digit t of the column, s + t <= 6, go to the fp32 accumulator of level s + t in tensor memory: at most
// 2^24 by a bound checked at set-up, so the sums are exact (where the bound fails: 8 digits of 7 bits).  The levels of an
// output are combined as integers and rounded once to FP64.  The dropped pairs carry 2^-53 of the column's largest element
// (rms over random columns of ~250, 2^-51.5 at most in 60 of them; every digit at its largest and of one sign: 2^-46.6);
// the banded solves this replaces stood at 2^-47.
//
// One block: 128 rows of one operator, TC = 16, 24 or 32 columns (twice with the imaginary parts).  Warp 0 brings the operator's digit
// planes (16 KB: 128 rows, 32 k, real | imaginary part, or two digits of a real operator) by bulk copies into a ring;
// warp 1 issues the MMAs (M 128, K 16): digit t of the columns is rows 2 TC t .. of one tile and level l columns 2 TC l ..
// of the accumulators, so digit s meets all the digits it pairs with in one or two instructions of N <= 256 (one pair at a
// time, N = 64, took 85 cycles for 32 of math); sixteen warps split the columns into digit planes, two halves of 32 k in
// turn, and at the end read the accumulators.  For a complex operator the columns are there as (xr, xi) and (-xi, xr), so
// that Fr and Fi take one plane each.  Digits that vanish are not formed: the entries of F~ lose a leading digit every ~15
// rows off the diagonal, and the stages of a tile start at their first digit.
//
// GB300, F~ of 800 x 41 (complex, band 110): 256 columns 2.64 (multiply-adds of k_band_apply) -> 0.54 ms, 48 columns
// 613 -> 131 us, 8 columns 98 -> 78 us, 4 columns 56 against 76 us.  A block takes 72 thousand cycles: 54 of stages, held
// back by shared memory (618 KB a full stage, 3.7 of math in 5.6 thousand cycles), 8 until the first MMA, 10 of epilogue.
#include "qpc_tcband.cuh"
#include "qpc_tcgen05.cuh"
#include <algorithm>
#include <cmath>

namespace qpc {

void tc_store::release()
{
	cudaFree(d_list); cudaFree(d_first); cudaFree(d_off); cudaFree(A); cudaFree(ear);
	d_list = nullptr; d_first = nullptr; d_off = nullptr; A = nullptr; ear = nullptr;
}

namespace {

constexpr int TR = 128;			// rows of a block
constexpr int TCMAX = 32;		// most columns of a block (TC: 16, 24 or 32)
constexpr int KS = 32;			// k of a stage
constexpr int NA = 6;			// operator planes in the ring
constexpr int PLANE_A = TR * 128;
constexpr int COLUMNS = 1024;	// bytes of barriers and column data, in front
constexpr int B_MAX = 16 * 2 * TCMAX * 128, SMEM = COLUMNS + B_MAX + NA * PLANE_A + 1024;	// the last for alignment
constexpr int DROP = 9;			// bits of an output's sum that are rounded off (the dropped pairs are worth 10)
constexpr int SPLIT = 512, THREADS = 64 + SPLIT;

// DB: bits of a digit.  x = sum_s d_s 2^(DB (ND - 1 - s)) with d_s in [-HALF, HALF) (the leading one up to HALF);
// field s of x + BIAS is d_s + HALF
template <int DB>
struct digits {
	static constexpr int ND = 56 / DB, HALF = 1 << (DB - 1);
	static constexpr long long BIAS = DB == 8 ? 128ll * ((1ll << 56) - 1) / 255 : 64ll * ((1ll << 56) - 1) / 127;
};

struct tc_args {
	const char* A;
	size_t stride;
	const int2* list;
	const int4* first;
	const size_t* off;
	int nrow, ea;
	const int* ear;		// per operator and row, or NULL
	int* status;
	int stbit;
};

__device__ __forceinline__ long long fixed55(double v, int E)	// v 2^(1077 - E), rounded
{
	const int h = __double2hiint(v);
	const int ex = (h >> 20) & 0x7ff, d = E - ex;
	unsigned long long m = ((unsigned long long)(unsigned)((h & 0xfffff) | 0x100000) << 32) | (unsigned)__double2loint(v);
	m <<= 2;
	m = (d > 56 || ex == 0) ? 0ull : (m + ((1ull << d) >> 1)) >> d;
	return h < 0 ? -(long long)m : (long long)m;
}

// digit s (0 = leading) of x, from xb = x + BIAS, as the upper half of an fp32 pattern
template <int DB>
__device__ __forceinline__ unsigned digit_bits(unsigned long long xb, int s)
{
	using D = digits<DB>;
	unsigned f;	// 2^23 + field
	if (DB == 8 && s > 0) f = __byte_perm(s > 2 ? (unsigned)xb : (unsigned)(xb >> 32), 0x4b000000u, 0x7650 | ((D::ND - 1 - s) & 3));
	else f = 0x4b000000u | (s == 0 ? (unsigned)(xb >> (DB * (D::ND - 1))) : (unsigned)(xb >> (DB * (D::ND - 1 - s))) & (2 * D::HALF - 1));
	return __float_as_uint(__uint_as_float(f) - (8388608.0f + D::HALF));
}

// v 2^s rounded to double (flushed below the normal range)
__device__ __forceinline__ double int_double(long long v, int s, bool nf)
{
	const unsigned long long n = v < 0 ? -(unsigned long long)v : (unsigned long long)v;
	const int z = __clzll(n), e = 1023 + 63 - z + s;
	const unsigned long long f = n << z;	// the leading bit adds one to the exponent field; rounding may carry into it
	long long r = ((long long)(e - 1) << 52) + (long long)(f >> 11) + (long long)((f >> 10) & 1);
	if (v == 0 || e < 1) r = 0;
	if (nf || e > 2046) r = nf ? 0x7ff8000000000000ll : 0x7ff0000000000000ll;
	return __longlong_as_double(r | (v & (1ll << 63)));
}

__device__ __forceinline__ void st_shared(uint32_t a, uint32_t v) { asm volatile("st.shared.b32 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }

__device__ __forceinline__ void mbar_arrive(uint32_t a) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(a) : "memory"); }

// low word of a descriptor (tc::sw128_desc); the high word is the same for every tile
__device__ __forceinline__ uint32_t desc_lo(uint32_t a) { return (a >> 4) | (1u << 16); }
__device__ __forceinline__ uint64_t desc(uint32_t lo) { return ((tc::sw128_desc(0) >> 32) << 32) | lo; }

// every product of digit D of an operator plane (two halves of 32 k: real | imaginary, or D | D + 1) with the digits of
// the columns.  Digit t of the columns are rows 2 TC t .. of one tile and level l is tensor-memory columns
// 2 TC l .., so one instruction multiplies by up to four digits at once
template <bool CX, int ND, int TC, int D>
__device__ __forceinline__ void plane_products(uint32_t tmem, uint32_t a, uint32_t b, bool start)
{
#pragma unroll
	for (int part = 0; part < 2; ++part) {
		const int d = CX ? D : D + part, cols = (ND - d) * 2 * TC;
		const int n = cols > 256 ? (cols / 2 + 15) & ~15 : cols;	// N: a multiple of 16, at most 256
		const uint32_t o = (CX && part) ? (ND * 2 * TC * 128) >> 4 : 0u;	// Fi meets (-xi, xr), else (xr, xi)
#pragma unroll
		for (int c = 0; c < cols; c += n)
#pragma unroll
			for (int k = 0; k < 2; ++k)
				tc::mma_bf16(tmem + (uint32_t)(d * 2 * TC + c), desc(a + 4u * part + 2u * k), desc(b + o + (uint32_t)c * 8u + 2u * k),
					tc::idesc_bf16(TR, cols - c < n ? cols - c : n), (D == 0 && part == 0 && k == 0) ? (start ? 0u : 1u) : 1u);
	}
}

template <bool CX, int DB, int TC>
__global__ void __launch_bounds__(THREADS, 1) k_tc_apply(const band_args p, const tc_args t)
{
	constexpr int ND = digits<DB>::ND, PLANE_B = 2 * TC * 128;
	constexpr long long BIAS = digits<DB>::BIAS;
	extern __shared__ char dyn[];
	const uint32_t raw = tc::smem_u32(dyn), base = (raw + 1023u) & ~1023u;
	char* sm = dyn + (base - raw);
	const uint32_t fullA = base, emptyA = fullA + 8 * NA, fullB = emptyA + 8 * NA, emptyB = fullB + 16, done = emptyB + 16, tslot = done + 8;
	const uint32_t planeB = base + COLUMNS, planeA = planeB + (CX ? 2 : 1) * ND * PLANE_B;
	int* sE = reinterpret_cast<int*>(sm + 192);
	const double2** sp = reinterpret_cast<const double2**>(sm + 320);
	volatile int* bad = reinterpret_cast<volatile int*>(sm + 576);
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const int ncg = (p.ncols + TC - 1) / TC;
	const int cg = blockIdx.x % ncg, tile = blockIdx.x / ncg, ch = blockIdx.y, col0 = cg * TC;
	const int4 span = t.first[tile];	// stages, and the k they cover
	const int e0 = span.x, e1 = span.y;
	if (threadIdx.x == 0) {
		for (int i = 0; i < NA; ++i) { tc::mbar_init(fullA + 8 * i, 1); tc::mbar_init(emptyA + 8 * i, 1); }
		for (int i = 0; i < 2; ++i) { tc::mbar_init(fullB + 8 * i, SPLIT); tc::mbar_init(emptyB + 8 * i, 1); }
		tc::mbar_init(done, 1);
		*bad = 0;
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	if (warp == 0) {
		__syncwarp();
		asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tslot), "r"(512) : "memory");
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
	}
	// a splitter thread has two consecutive k of one column in every stage; a warp columns c and c + 4, whose swizzled rows
	// fall on different banks (those of columns beyond TC only take part in the waits)
	const int kq = lane & 15, c = ((warp - 2) & 3) + 4 * (lane >> 4) + 8 * ((warp - 2) >> 2);
	const double2* x = nullptr;
	int E = 0;
	double2 v[2];
	auto load = [&](int k0) {
#pragma unroll
		for (int j = 0; j < 2; ++j) { const int k = k0 + 2 * kq + j; v[j] = (x && k < p.N) ? x[k] : make_double2(0.0, 0.0); }
	};
	if (warp >= 2) {
		const int cc = col0 + c, cl = min(cc, p.ncols - 1), k0 = t.list[e0].x, nex = p.ntile * EPT;
		const bool odd = p.par && (p.par[cl] & 1);
		const long o = (long)(p.smap ? p.smap[cl] : cl) * p.nchan + ch;
		if (c < TC && cc < p.ncols && (!p.nta || p.step < p.nta[cl])) x = (odd ? p.s1 : p.s0) + o * p.N;
		prev_wait();
		load(k0);
		if (x) {
			const int* ex = (odd ? p.e1 : p.e0) + o * nex;
			for (int i = span.z / TE + kq; i < min(nex, span.w / TE); i += 16) E = max(E, ex[i]);
		}
		for (int s = 1; s < 16; s <<= 1) E = max(E, __shfl_xor_sync(0xffffffffu, E, s));
		if (kq == 0 && c < TC) { sE[c] = E; sp[c] = x; }
	}
	tc::fence_before();
	__syncthreads();
	tc::fence_after();
	uint32_t tmem;
	asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(tslot) : "memory");

	if (threadIdx.x == 0) {
		// ---- the operator's planes, in the order they are stored
		const char* src = t.A + (size_t)p.lmap[ch] * t.stride + t.off[tile];
		int n = 0;
		bool ok = true;
		for (int e = e0; e < e1 && ok; ++e) {
			const int planes = CX ? ND - t.list[e].y : (ND + 1 - t.list[e].y) / 2;
			for (int i = 0; i < planes && ok; ++i, ++n) {
				const int slot = n % NA;
				if (n >= NA && !tc::mbar_wait(emptyA + 8 * slot, (n / NA - 1) & 1)) { ok = false; break; }
				if (*bad) { ok = false; break; }
				asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(fullA + 8 * slot), "r"(PLANE_A) : "memory");
				asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(planeA + slot * PLANE_A),
					"l"(src + (size_t)n * PLANE_A), "r"(PLANE_A), "r"(fullA + 8 * slot) : "memory");
			}
		}
		if (!ok) *bad = 1;
		if (*bad)	// copies in flight end before the block does
			for (int i = max(0, n - NA); i < n; ++i) tc::mbar_wait(fullA + 8 * (i % NA), (i / NA) & 1);
	} else if (warp == 1) {
		// ---- the MMAs: the warp in step, one lane issues
		int n = 0;
		bool ok = true;
		int next = t.list[e0].y;
		for (int e = e0; e < e1 && ok; ++e) {
			const int i = e - e0, h = i & 1, s0 = __shfl_sync(0xffffffffu, next, 0);
			next = t.list[min(e + 1, e1 - 1)].y;
			if (!__all_sync(0xffffffffu, tc::mbar_wait(fullB + 8 * h, (i >> 1) & 1))) { ok = false; break; }
			const uint32_t b = desc_lo(planeB + 64u * h);
			for (int s = s0; s < ND; s += CX ? 1 : 2, ++n) {
				const int slot = n % NA;
				if (!__all_sync(0xffffffffu, tc::mbar_wait(fullA + 8 * slot, (n / NA) & 1))) { ok = false; break; }
				tc::fence_after();
				const uint32_t a = desc_lo(planeA + slot * PLANE_A);
				if (lane == 0) {
					switch (s) {	// the first stage has every digit: all levels start there
					case 0: plane_products<CX, ND, TC, 0>(tmem, a, b, i == 0); break;
					case 1: if (CX) plane_products<CX, ND, TC, 1>(tmem, a, b, false); break;
					case 2: plane_products<CX, ND, TC, 2>(tmem, a, b, false); break;
					case 3: if (CX) plane_products<CX, ND, TC, 3>(tmem, a, b, false); break;
					case 4: plane_products<CX, ND, TC, 4>(tmem, a, b, false); break;
					case 5: if (CX) plane_products<CX, ND, TC, 5>(tmem, a, b, false); break;
					case 6: plane_products<CX, ND, TC, 6>(tmem, a, b, false); break;
					case 7: if (CX && ND == 8) plane_products<CX, ND, TC, ND - 1>(tmem, a, b, false); break;
					}
					tc::commit(emptyA + 8 * slot);
				}
				__syncwarp();
			}
			if (ok && lane == 0) tc::commit(emptyB + 8 * h);
		}
		if (lane == 0) {
			if (!ok) *bad = 1;
			tc::commit(done);
		}
		__syncwarp();
	} else if (warp >= 2) {
		// ---- the columns' digits
		uint32_t at[2];
#pragma unroll
		for (int h = 0; h < 2; ++h)	// 128-byte swizzle; rows c and c + TC alike
			at[h] = planeB + (uint32_t)c * 128u + (((uint32_t)(4 * h + (kq >> 2)) ^ (uint32_t)(c & 7)) << 4) + 4u * (kq & 3);
		int2 at_e = t.list[e0], next = t.list[min(e0 + 1, e1 - 1)];
		bool ok = true;
		for (int e = e0; e < e1; ++e) {
			const int i = e - e0, h = i & 1;
			unsigned long long re[2], im[2];
#pragma unroll
			for (int j = 0; j < 2; ++j) {
				re[j] = (unsigned long long)(fixed55(v[j].x, E) + BIAS);
				im[j] = (unsigned long long)(fixed55(v[j].y, E) + BIAS);
			}
			const int nd = ND - at_e.y;	// a stage whose operator digits start at s0 meets the columns' first ND - s0
			if (e + 1 < e1) { load(next.x); at_e = next; next = t.list[min(e + 2, e1 - 1)]; }
			if (i >= 2 && !tc::mbar_wait(emptyB + 8 * h, ((i >> 1) - 1) & 1)) { ok = false; break; }
#pragma unroll
			for (int s = 0; s < ND; ++s) {
				if (s >= nd || c >= TC) break;
				const uint32_t r = __byte_perm(digit_bits<DB>(re[0], s), digit_bits<DB>(re[1], s), 0x7632), m = __byte_perm(digit_bits<DB>(im[0], s), digit_bits<DB>(im[1], s), 0x7632);
				const uint32_t q = at[h] + (uint32_t)s * PLANE_B, half = TC * 128u;
				st_shared(q, r);
				st_shared(q + half, m);
				if (CX) {
					st_shared(q + ND * PLANE_B, m ^ 0x80008000u);
					st_shared(q + ND * PLANE_B + half, r);
				}
			}
			tc::fence_async_smem();
			mbar_arrive(fullB + 8 * h);
		}
		if (!ok) *bad = 1;
		// ---- the levels of 128 rows x 64 columns: a warp its quarter of the rows and 8 columns
		const bool fin = tc::mbar_wait(done, 0);
		tc::fence_after();
		if (__all_sync(0xffffffffu, fin && ok && !*bad) && (warp - 2) >> 2 < TC / 8) {
			const int qr = warp & 3, c8 = 8 * ((warp - 2) >> 2);
			const int row = tile * TR + qr * 32 + lane;
			const bool in = row < t.nrow;
			const uint32_t tl = tmem + ((uint32_t)(qr * 32) << 16);
			const int ea = (t.ear ? (in ? t.ear[(long)p.lmap[ch] * t.nrow + row] : 0) : t.ea) + (!CX && p.er && in ? p.er[row] : 0);
			const int nexo = (t.nrow + TM - 1) / TM * EPT;
#pragma unroll 1
			for (int b = 0; b < 2; ++b) {
				const int c0 = c8 + 4 * b;
				long long sum[2][4];
#pragma unroll
				for (int part = 0; part < 2; ++part) {
					uint32_t lv[ND][4];
#pragma unroll
					for (int l = 0; l < ND; ++l) tc::ld4(tl + (uint32_t)(l * 2 * TC + part * TC + c0), lv[l]);
					tc::wait_ld();
#pragma unroll
					for (int j = 0; j < 4; ++j) {
						long long h = 0;
						int m = 1 << (DROP - 1);
#pragma unroll
						for (int l = 0; l < ND; ++l) {
							const int f = __float2int_rn(__uint_as_float(lv[l][j])), sh = DB * (ND - 1 - l);
							if (sh >= DROP + 32) h += ((long long)f << 32) << (sh - DROP - 32);
							else if (sh >= DROP) h += (long long)f * (1ll << (sh - DROP));
							else if (sh == 0) m += f;
							else { h += f >> (DROP - sh); m += (f & ((1 << (DROP - sh)) - 1)) << sh; }
						}
						sum[part][j] = h + (m >> DROP);
					}
				}
#pragma unroll
				for (int j = 0; j < 4; ++j) {
					const int cl = c0 + j, cc = col0 + cl;
					if (cc >= p.ncols || !sp[cl]) continue;
					const int Ec = sE[cl], s = ea + Ec + DROP - (DB == 8 ? 1084 : 1083);
					const double2 y = make_double2(int_double(sum[0][j], s, Ec == 0x7ff), int_double(sum[1][j], s, Ec == 0x7ff));
					const long o = (long)(p.dmap ? p.dmap[cc] : cc) * p.nchan + ch;
					if (in) p.dst[o * t.nrow + row] = y;
					if (p.edst) {
						const int x = group_max(in ? max(bexp(y.x), bexp(y.y)) : 0);
						if (lane % TE == 0 && row / TE < nexo) p.edst[o * nexo + row / TE] = x;
					}
				}
			}
		} else if (!fin) *bad = 1;
	}
	tc::fence_before();
	__syncthreads();
	tc::fence_after();
	if (threadIdx.x == 0 && *bad) atomicOr(t.status, t.stbit);
	__syncwarp();
	if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

struct make_args {
	const double2* Fb;
	const double* A;
	long sop, si, sj;
	int nrow, N, w, ea;
	const int* ear;
	int kb, ke;		// columns that take part; kb a multiple of KS
};

__device__ __forceinline__ double2 entry(const make_args& m, int op, int i, int j)
{
	double2 v = make_double2(0.0, 0.0);
	if (i < m.nrow && j < m.ke && (m.w < 0 || abs(i - j) <= m.w)) {
		if (m.Fb) v = m.Fb[((long)op * m.N + i) * (2 * WMAX + 1) + (j - i + WMAX)];
		else v.x = m.A[op * m.sop + i * m.si + j * m.sj];
	}
	return v;
}

// the planes of one stage (blockIdx.x: entry of the list; tile: its tile) of operator blockIdx.y
template <int DB>
__global__ void k_tc_planes(const make_args m, const int2* __restrict__ list, const int* __restrict__ tile_of, const size_t* __restrict__ at, size_t stride,
	char* __restrict__ out, bool cx)
{
	constexpr int ND = digits<DB>::ND;
	constexpr long long BIAS = digits<DB>::BIAS;
	const int e = blockIdx.x, op = blockIdx.y;
	const int k0 = list[e].x, s0 = list[e].y, row0 = tile_of[e] * TR;
	char* o = out + op * stride + at[e];
	for (int q = threadIdx.x; q < TR * KS; q += blockDim.x) {
		const int r = q / KS, k = q % KS;
		const double2 v = entry(m, op, row0 + r, k0 + k);
		const int sc = 55 - ((m.ear && row0 + r < m.nrow) ? m.ear[(long)op * m.nrow + row0 + r] : m.ea);
		const unsigned long long x = (unsigned long long)(__double2ll_rn(ldexp(v.x, sc)) + BIAS), y = (unsigned long long)(__double2ll_rn(ldexp(v.y, sc)) + BIAS);
		for (int s = s0; s < ND; ++s) {
			const int plane = cx ? s - s0 : (s - s0) / 2, part = cx ? 0 : (s - s0) & 1;
			const int b = plane * PLANE_A + r * 128 + (k & 7) * 2;
			*reinterpret_cast<uint16_t*>(o + b + ((((k >> 3) + 4 * part) ^ (r & 7)) << 4)) = (uint16_t)(digit_bits<DB>(x, s) >> 16);
			if (cx) *reinterpret_cast<uint16_t*>(o + b + ((((k >> 3) + 4) ^ (r & 7)) << 4)) = (uint16_t)(digit_bits<DB>(y, s) >> 16);
		}
	}
}

// worst[0]: largest sum over a row of the digits' magnitudes (every level's sum is at most HALF times that), worst[1]: of
// the leading digits' (the first level's)
template <int DB>
__global__ void k_tc_bound(const make_args m, int* __restrict__ worst)
{
	constexpr int ND = digits<DB>::ND;
	constexpr long long BIAS = digits<DB>::BIAS;
	const int i = blockIdx.x, op = blockIdx.y;
	const int sc = 55 - (m.ear ? m.ear[(long)op * m.nrow + i] : m.ea);
	int sum = 0, lead = 0;
	const int j0 = m.w < 0 ? m.kb : max(m.kb, i - m.w), j1 = m.w < 0 ? m.ke : min(m.ke, i + m.w + 1);
	for (int j = j0 + threadIdx.x; j < j1; j += blockDim.x) {
		double2 v = entry(m, op, i, j);
		v.x = ldexp(v.x, sc); v.y = ldexp(v.y, sc);
		if (!(fabs(v.x) <= 36028797018963968.0) || !(fabs(v.y) <= 36028797018963968.0)) sum = lead = 1 << 28;	// 2^55
		else {
			const unsigned long long x = (unsigned long long)(__double2ll_rn(v.x) + BIAS), y = (unsigned long long)(__double2ll_rn(v.y) + BIAS);
			lead += abs((int)__uint_as_float(digit_bits<DB>(x, 0))) + abs((int)__uint_as_float(digit_bits<DB>(y, 0)));
			for (int s = 0; s < ND; ++s) sum += abs((int)__uint_as_float(digit_bits<DB>(x, s))) + abs((int)__uint_as_float(digit_bits<DB>(y, s)));
		}
	}
	for (int o = 16; o; o >>= 1) {
		sum = min(1 << 28, sum + __shfl_xor_sync(0xffffffffu, sum, o));
		lead = min(1 << 28, lead + __shfl_xor_sync(0xffffffffu, lead, o));
	}
	__shared__ int part[8];
	if ((threadIdx.x & 31) == 0) { part[threadIdx.x >> 5] = sum; part[4 + (threadIdx.x >> 5)] = lead; }
	__syncthreads();
	if (threadIdx.x < 2) { const int* q = part + 4 * threadIdx.x; atomicMax(worst + threadIdx.x, q[0] + q[1] + q[2] + q[3]); }
}

// |entry| <= 2^ear of each row
__global__ void k_tc_rows(const make_args m, int* __restrict__ ear)
{
	const int i = blockIdx.x, op = blockIdx.y;
	double v = 0.0;
	for (int j = m.kb + threadIdx.x; j < m.ke; j += 32) { const double2 a = entry(m, op, i, j); v = fmax(v, fmax(fabs(a.x), fabs(a.y))); }
	for (int o = 16; o; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
	if (threadIdx.x == 0) ear[(long)op * m.nrow + i] = v > 0.0 && v < 1e300 ? ilogb(v) + 1 : 0;
}

template <int DB>
int make(tc_store& t, const make_args& m, int nop, const double* prof, cudaStream_t st, bool* ok)
{
	constexpr int ND = digits<DB>::ND;
	const int nrow = m.nrow, w = m.w, ea = m.ea;
	t.cx = m.Fb != nullptr; t.ea = ea; t.N = m.N; t.nrow = nrow; t.ntile = (nrow + TR - 1) / TR; t.db = DB;
	int rc;
	scratch tmp(st);
	int* d_worst;
	if ((rc = tmp.get(&d_worst, 2))) return rc;
	QPC_CUDA(cudaMemsetAsync(d_worst, 0, 2 * sizeof(int), st));
	k_tc_bound<DB><<<dim3(nrow, nop), 128, 0, st>>>(m, d_worst);
	QPC_CUDA(cudaGetLastError());
	int worst[2];
	if ((rc = copy_to_host(worst, d_worst, sizeof(worst), st))) return rc;
	// exact fp32 sums; and the first level, 2^(48 or 49 - DROP) of the sum, within 2^62
	if (worst[0] > (1 << 24) / digits<DB>::HALF || worst[1] > (1 << (62 - DB * (ND - 1) + DROP)) / digits<DB>::HALF) return QPC_OK;
	std::vector<int2> list;
	std::vector<int4> first;
	std::vector<int> tile_of;
	std::vector<size_t> at, off;
	t.work.clear();
	size_t o = 0;
	for (int tl = 0; tl < t.ntile; ++tl) {
		const int r0 = tl * TR, r1 = std::min(nrow, r0 + TR) - 1;
		std::vector<int2> mine;
		for (int k0 = m.kb; k0 < m.ke; k0 += KS) {
			const int k1 = k0 + KS - 1, gap = w < 0 ? 0 : std::max(0, std::max(k0 - r1, r0 - k1));
			if (w >= 0 && gap > w) continue;
			int s0 = 0;
			if (prof) {
				double big = 0.0;
				for (int d = gap; d <= std::min(w, WMAX); ++d) big = std::max(big, prof[d]);
				while (s0 < ND && big < 0.98 * std::ldexp(1.0, ea - DB * (s0 + 1))) ++s0;
				if (s0 == ND) continue;
				if (!t.cx) s0 &= ~1;
			}
			mine.push_back(make_int2(k0, s0));
		}
		std::stable_sort(mine.begin(), mine.end(), [](int2 a, int2 b) { return a.y < b.y; });
		if (mine.empty() || mine[0].y != 0) return QPC_OK;	// every level starts in the first stage
		int work = 0, k0 = 1 << 30, k1 = 0;
		const int f = (int)list.size();
		off.push_back(o);
		for (int2 e : mine) {
			list.push_back(e); tile_of.push_back(tl); at.push_back(o);
			o += (size_t)(t.cx ? ND - e.y : (ND + 1 - e.y) / 2) * PLANE_A;
			work += (ND - e.y) * (ND + 1 - e.y) / 2 * (t.cx ? 128 : 64);	// tensor-core cycles: 32 for 16 k of a pair of digits
			k0 = std::min(k0, e.x); k1 = std::max(k1, e.x + KS);
		}
		first.push_back(make_int4(f, (int)list.size(), k0, k1));
		t.work.push_back(work);
	}
	t.stride = o;
	if (o * nop > std::min<size_t>((size_t)4 << 30, free_bytes() / 8)) return QPC_OK;
	int* d_tile;
	size_t* d_at;
	if ((rc = tmp.get(&d_tile, tile_of.size())) || (rc = tmp.get(&d_at, at.size()))) return rc;
	if ((rc = dalloc(&t.d_list, list.size())) || (rc = dalloc(&t.d_first, first.size())) || (rc = dalloc(&t.d_off, off.size())) || (rc = dalloc(&t.A, o * nop))) return rc;
	QPC_CUDA(cudaMemcpyAsync(t.d_list, list.data(), sizeof(int2) * list.size(), cudaMemcpyHostToDevice, st));
	QPC_CUDA(cudaMemcpyAsync(t.d_first, first.data(), sizeof(int4) * first.size(), cudaMemcpyHostToDevice, st));
	QPC_CUDA(cudaMemcpyAsync(t.d_off, off.data(), sizeof(size_t) * off.size(), cudaMemcpyHostToDevice, st));
	QPC_CUDA(cudaMemcpyAsync(d_tile, tile_of.data(), sizeof(int) * tile_of.size(), cudaMemcpyHostToDevice, st));
	QPC_CUDA(cudaMemcpyAsync(d_at, at.data(), sizeof(size_t) * at.size(), cudaMemcpyHostToDevice, st));
	k_tc_planes<DB><<<dim3((unsigned)list.size(), nop), 256, 0, st>>>(m, t.d_list, d_tile, d_at, t.stride, t.A, t.cx);
	QPC_CUDA(cudaGetLastError());
	auto attr = [](auto kern) { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM); };
	if (t.cx) {
		QPC_CUDA(attr(k_tc_apply<true, DB, 16>)); QPC_CUDA(attr(k_tc_apply<true, DB, 24>)); QPC_CUDA(attr(k_tc_apply<true, DB, 32>));
	} else {
		QPC_CUDA(attr(k_tc_apply<false, DB, 16>)); QPC_CUDA(attr(k_tc_apply<false, DB, 24>)); QPC_CUDA(attr(k_tc_apply<false, DB, 32>));
	}
	*ok = true;
	return wait_on(st);
}

} // namespace

int tc_make(tc_store& t, const double2* Fb, const double* A, long sop, long si, long sj, int nrow, int N, int nop, int w, const double* prof, int ea,
	bool rows, cudaStream_t st, bool* ok, int kb, int ke)
{
	t.release();
	*ok = false;
	make_args m{Fb, A, sop, si, sj, nrow, N, w, ea, nullptr, kb, ke < 0 ? N : ke};
	int rc;
	if (rows) {
		if (dalloc(&t.ear, (size_t)nrow * nop)) return QPC_OK;
		k_tc_rows<<<dim3(nrow, nop), 32, 0, st>>>(m, t.ear);
		QPC_CUDA(cudaGetLastError());
		m.ear = t.ear;
	}
	rc = make<8>(t, m, nop, prof, st, ok);
	if (!rc && !*ok) rc = make<7>(t, m, nop, prof, st, ok);
	if (rc || !*ok) { *ok = false; t.release(); }
	return rc == QPC_ERR_NOMEM ? QPC_OK : rc;
}

namespace {

// cycles of a launch with blocks of tc columns: twice the tensor-core math of an average tile and 18 thousand of a block's
// own, one block per SM.  (Blocks of 32 only before: 48 wavefunctions
// of 800 x 41, 20 steps 5.60 -> 5.39 ms, 24 of 517 x 30, 30 steps 2.30 -> 2.23, 8 of 640 x 25, 20 steps 2.53 -> 2.44.)
double cycles(const tc_store& t, int nchan, int ncols, int tc)
{
	double mma = 0.0;
	for (int w : t.work) mma += w;
	const double blocks = (double)t.ntile * nchan * ((ncols + tc - 1) / tc);
	return std::ceil(blocks / 152.0) * (2.0 * mma / t.ntile * tc / 32.0 + 18e3);
}

int columns(const tc_store& t, int nchan, int ncols)
{
	int best = 32;
	for (int tc : {24, 16})
		if (cycles(t, nchan, ncols, tc) < cycles(t, nchan, ncols, best)) best = tc;
	return best;
}

template <bool CX, int DB>
void launch(const tc_args& q, const tc_store& t, const band_args& a, cudaStream_t st)
{
	const int tc = columns(t, a.nchan, a.ncols);
	const dim3 g((unsigned)(t.ntile * ((a.ncols + tc - 1) / tc)), (unsigned)a.nchan);
	if (tc == 16) launch_after(k_tc_apply<CX, DB, 16>, g, THREADS, SMEM, st, a, q);
	else if (tc == 24) launch_after(k_tc_apply<CX, DB, 24>, g, THREADS, SMEM, st, a, q);
	else launch_after(k_tc_apply<CX, DB, 32>, g, THREADS, SMEM, st, a, q);
}

} // namespace

void tc_apply(const tc_store& t, const band_args& a, int* status, int stbit, cudaStream_t st)
{
	const tc_args q{t.A, t.stride, t.d_list, t.d_first, t.d_off, t.nrow, t.ea, t.ear, status, stbit};
	if (t.db == 8) {
		if (t.cx) launch<true, 8>(q, t, a, st);
		else launch<false, 8>(q, t, a, st);
	} else if (t.cx) launch<true, 7>(q, t, a, st);
	else launch<false, 7>(q, t, a, st);
}

double tc_cost(const tc_store& t, int nchan, int ncols) { return cycles(t, nchan, ncols, columns(t, nchan, ncols)) / 2000.0; }

} // namespace qpc
