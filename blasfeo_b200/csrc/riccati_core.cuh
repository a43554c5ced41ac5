// FP64 batched Riccati factorization (LQR backward pass) for both slab
// layouts: the per-problem recursion of examples/example_d_riccati_recursion.c:
// 115-143 (d_back_ric_trf_libstr),
//   L_N = chol(Q_N)                                   (blasfeo_dpotrf_l)
//   for k = N-1 .. 0:
//     W   = BAbt_k * Lxx_{k+1}                        (blasfeo_dtrmm_rlnn)
//     L_k = chol(RSQ_k + W W^T)                       (blasfeo_dsyrk_dpotrf_ln)
// with Lxx_{k+1} the lower-right nx x nx block of L_{k+1} (all of L_N),
// nu + nx <= 16.
//
// A CTA has 8 problems, a warp each, everything between the loads and the
// stores in FP64 tensor core fragments (mma m8n8k4; an 8 x 8 accumulator holds
// columns 2q and 2q + 1 of row g in lane (g, q) = (lane / 4, lane % 4)):
//   products: W as 2 x 2 blocks, then RSQ_k + W W^T.  Summing W W^T over the
//     columns in the accumulators' order makes the accumulators of W the
//     operands of the second product as they are, so W never leaves the
//     registers.  The columns 8..15 of W are taken in the order 8, 12, 9, 13,
//     .. so that nx <= 12 needs one step for them, not two;
//   factor: two 8-column panels.  Per column the pivot goes through shared
//     memory to the warp, the column is scaled in the 8 lanes that hold it and
//     subtracted from the rest of the panel as a rank-1 tensor core step (the
//     column sits in one k slot, the other three are zero); the second panel
//     gets the first one's update in two steps.  No shuffles: a 64-bit shuffle
//     occupies the SM's shuffle unit for about 8 cycles, and the quad and
//     half-warp forms of the factorization need 272 of them per warp, which
//     bounded them (4,096 problems, N = 30, 12 + 4, interleaved: quads 0.277
//     ms, 8 lanes 0.271, 16 lanes 0.275; this kernel 0.268, back to back 0.232
//     against 0.88 for a warp with FMAs and shuffles).
// The next stage's inputs arrive by cp.async under the factorization.
//
// What bounds it: latency with 7 warps per SM sub-partition, each a stage of 31
// after another.  Back to back issue slots are 60% and the FP64 pipe 53% used (ncu;
// a warp issues every 10.2 cycles: 2.9 waiting for an earlier result, 2.5 for the pipe,
// 1.3 for shared memory); interleaved 45% and 45%, with 2.8 cycles for shared memory
// and 1.4 for its queue: one 8-byte copy per element and lane instead of 16-byte
// ones, and CTA barriers in the place of warp barriers.  The bytes (BAbt, lower RSQ
// in; lower L out: 0.073 ms there) are the floor.
#pragma once

#include "chol_frag.cuh"
#include "quad.cuh"

namespace ric {

using quad::IL;
using quad::pme;

constexpr int PC = 8;       // problems per CTA
constexpr int NT = 256;     // threads per CTA
constexpr int LD = 20;      // row stride of L, column stride of BAbt: 4 mod 16, so that the
                            // 4 x 4 lanes of a fragment phase hit 16 different 8-byte banks
constexpr int L_EL = 16 * LD;
constexpr int RQ_EL = 256;  // lower RSQ: columns 0..7 with stride 20, then rows 8.. of 8..15 with stride 12

__host__ __device__ inline int prob_el(int cnx) { return L_EL + cnx * LD + RQ_EL + 32 + 2; }  // + inverse pivots, pivots; 2 mod 16

__device__ __forceinline__ int rq_idx(int i, int j) { return j < 8 ? j * LD + i : 160 + (j - 8) * 12 + (i - 8); }

struct Args {
	int batch, N, nx, nu, cnx;
	const double *BA, *RSQ;
	double *L, *Ld;          // Ld: inverse diagonal (back-to-back)
	long long sba, srsq, sl; // elements between instances (back-to-back) or groups of 16 (interleaved)
	long long bs;            // instances per stage (interleaved)
	int *info;
};

__device__ __forceinline__ void cpa8(double *dst, const double *src) {
	const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
	asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}

using frag::dmma;

// stage k's inputs of the CTA's problems, interleaved slab: thread = (problem
// t % 8, row t / 8 % 16, RSQ or BAbt), 8 bytes per copy; 8 problems of an
// element are one 64-byte run in HBM
__device__ __forceinline__ void load_il(const Args &a, int k, int b0, double *sm, int PS) {
	const int tp = threadIdx.x & 7, i = (threadIdx.x >> 3) & 15;
	if (b0 + tp >= a.batch) return;
	const long long gk = (long long)k * (a.bs / IL) + b0 / IL;
	const int sl = b0 % IL + tp;
	double *pb = sm + (size_t)tp * PS;
	if (threadIdx.x < 128) {
		const double *R = a.RSQ + gk * a.srsq + sl + pme(i, 0, 16) * IL;
		double *rq = pb + L_EL + a.cnx * LD;
#pragma unroll
		for (int j = 0; j < 16; j++)
			if (j <= i) cpa8(rq + rq_idx(i, j), R + j * 4 * IL);
	} else if (k < a.N) {
		const double *B = a.BA + gk * a.sba + sl + pme(i, 0, a.cnx) * IL;
		for (int j = 0; j < a.nx; j++) cpa8(pb + L_EL + j * LD + i, B + j * 4 * IL);
	}
}

// stage k's inputs of one problem of a back-to-back slab by one warp: 16-byte
// copies of two rows of a column (lower 4 x 4 tiles of RSQ only)
__device__ __forceinline__ void load_b2b(const Args &a, int k, long long b, double *pb, int lane) {
	const double *R = a.RSQ + a.srsq * (b * (a.N + 1) + k);
	double *rq = pb + L_EL + a.cnx * LD;
#pragma unroll
	for (int c = lane; c < 80; c += 32) {
		const int p = c < 8 ? 0 : (c < 24 ? 1 : (c < 48 ? 2 : 3));
		const int w = c - (p == 0 ? 0 : (p == 1 ? 8 : (p == 2 ? 24 : 48)));
		const int j = w >> 1, i = 4 * p + 2 * (w & 1);
		quad::cpa16(rq + rq_idx(i, j), R + 64 * p + 2 * w);
	}
	if (k < a.N) {
		const double *B = a.BA + a.sba * (b * a.N + k);
#pragma unroll
		for (int p = 0; p < 4; p++)
			for (int w = lane; w < 2 * a.cnx; w += 32)
				quad::cpa16(pb + L_EL + (w >> 1) * LD + 4 * p + 2 * (w & 1), B + 4 * p * a.cnx + 2 * w);
	}
}

// L_k (rows and columns < m, lower triangle) and its inverse diagonal, shared
// memory -> slab.  Interleaved: the CTA's problems, thread = (problem, row,
// columns 0..7 or 8..15); back to back: the warp's problem (pb), lane = (row,
// column parity)
template <bool INTER>
__device__ __forceinline__ void store_l(const Args &a, int k, int b0, const double *pb, int PS) {
	const int m = k == a.N ? a.nx : a.nx + a.nu;
	if (INTER) {
		const int tp = threadIdx.x & 7, i = (threadIdx.x >> 3) & 15, j0 = (threadIdx.x >> 7) * 8;
		if (b0 + tp >= a.batch || i >= m) return;
		pb += (size_t)tp * PS;
		double *g = a.L + ((long long)k * (a.bs / IL) + b0 / IL) * a.sl + b0 % IL + tp;
		if (j0 == 0) g[(256LL + i) * IL] = pb[L_EL + a.cnx * LD + RQ_EL + i];
		double *r = g + pme(i, j0, 16) * IL;
#pragma unroll
		for (int j = 0; j < 8; j += 2) {
			const double2 v = *(const double2 *)(pb + i * LD + j0 + j);
			if (j0 + j <= i) r[j * 4 * IL] = v.x;
			if (j0 + j + 1 <= i) r[(j + 1) * 4 * IL] = v.y;
		}
	} else {
		const int i = threadIdx.x & 15, h = (threadIdx.x >> 4) & 1;
		if (i >= m) return;
		const long long at = a.sl * ((long long)b0 * (a.N + 1) + k);
		if (h == 0) a.Ld[at + i] = pb[L_EL + a.cnx * LD + RQ_EL + i];
		double *r = a.L + at + pme(i, h, 16);
#pragma unroll
		for (int j = 0; j < 16; j += 2)
			if (j + h <= i) r[4 * j] = pb[i * LD + j + h];
	}
}

// One 8-column panel of the factorization of the 16 x 16 matrix of a warp: D
// the panel's diagonal block (finite values right of its diagonal), B (TWO)
// the block below it, columns c0.. of L to Ls (row-major) with zeros above the
// diagonal, inverse pivots to dv (0 for a pivot that is not positive), pv: 16
// entries through which the pivots reach the warp.  Valid while every number
// is finite (frag::panel).  keep: the lane's entries
// of B's factored columns 2q and 2q + 1, the operands of the next panel's
// update.
template <bool TWO>
__device__ __forceinline__ void panel(double (&D)[2], double (&B)[2], double (&keep)[2], double *Ls, double *dv, double *pv,
                                      int c0, int g, int q) {
	double *col = Ls + (c0 + g) * LD + c0 + 2 * q;
#pragma unroll
	for (int c = 0; c < 8; c++) {
		const int e = c & 1;
		const bool mine = q == c >> 1;
		if (mine && g == c) pv[c0 + c] = D[e];
		__syncwarp();
		const double p = pv[c0 + c];
		const bool ok = p > 0.0;
		const double iv = chol_rsqrt(p);
		// the column's lanes scale it; zeros elsewhere (and above the diagonal)
		// make it a rank-1 operand
		const double l0 = D[e] * (ok && mine && g >= c ? iv : 0.0);
		double l1 = 0.0;
		if (TWO) l1 = B[e] * (ok && mine ? iv : 0.0);
		if (c < 7) {
			dmma(D[0], D[1], -l0, l0);
			if (TWO) dmma(B[0], B[1], -l1, l0);
		}
		if (mine) {
			col[e] = l0;
			if (TWO) {
				col[8 * LD + e] = l1;
				keep[e] = l1;
			}
			if (g == c) dv[c0 + c] = ok ? iv : 0.0;
		}
	}
}

template <bool INTER>
__global__ void __launch_bounds__(NT, 4) k_ric_trf_dmma(Args a) {
	extern __shared__ __align__(16) double ric_sm[];
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const int g = lane >> 2, q = lane & 3;
	const int b0 = blockIdx.x * PC, b = b0 + warp;
	const int PS = prob_el(a.cnx);
	const int nx = a.nx, nu = a.nu, N = a.N, M = nu + nx;
	double *Ls = ric_sm + (size_t)warp * PS;   // this warp's problem: L, BAbt, RSQ, inverse pivots
	const double *ba = Ls + L_EL, *rq = ba + a.cnx * LD;
	double *dv = Ls + L_EL + a.cnx * LD + RQ_EL, *pv = dv + 16;
	int first = 0;

	if (!INTER && b >= a.batch) return;        // back to back: no CTA barrier follows
	auto load = [&](int k) {
		if (INTER)
			load_il(a, k, b0, ric_sm, PS);
		else
			load_b2b(a, k, b, Ls, lane);
		quad::cpa_commit();
	};
	// the problems of a CTA share only the interleaved copies
	auto sync = [&]() {
		if (INTER)
			__syncthreads();
		else
			__syncwarp();
	};
	load(N);
	for (int k = N; k >= 0; k--) {
		quad::cpa_wait_all();
		sync();  // stage k's inputs and L_{k+1} are in shared memory
		if (k < N) store_l<INTER>(a, k + 1, INTER ? b0 : b, INTER ? ric_sm : Ls, PS);
		const int m = (k == N) ? nx : M;
		const int off = (k + 1 == N) ? 0 : nu;
		// ---- products: RSQ_k + W W^T, blocks (0,0), (1,0), (1,1) ----
		double F0[2], F1[2], F2[2];
#pragma unroll
		for (int h = 0; h < 2; h++) {
			F0[h] = rq[rq_idx(g, 2 * q + h)];
			F1[h] = rq[rq_idx(8 + g, 2 * q + h)];
			F2[h] = rq[160 + (2 * q + h) * 12 + g];
		}
		if (k < N) {
			double W[2][2][2];
#pragma unroll
			for (int I = 0; I < 2; I++)
#pragma unroll
				for (int J = 0; J < 2; J++) W[I][J][0] = W[I][J][1] = 0.0;
			const int c1 = 8 + (g >> 1) + 4 * (g & 1);  // column of slot g in W's second block
#pragma unroll
			for (int ks = 0; ks < 4; ks++) {
				if (4 * ks >= nx) break;
				const int kk = 4 * ks + q;
				const bool in = kk < nx;
				const double a0 = in ? ba[kk * LD + g] : 0.0, a1 = in ? ba[kk * LD + 8 + g] : 0.0;
				const double *lr = Ls + (off + kk) * LD + off;
				const double bb0 = (in && g <= kk) ? lr[g] : 0.0;
				dmma(W[0][0][0], W[0][0][1], a0, bb0);
				dmma(W[1][0][0], W[1][0][1], a1, bb0);
				if (ks >= 2) {  // columns 8.. of the lower triangle start at row 8
					const double bb1 = (in && c1 <= kk) ? lr[c1] : 0.0;
					dmma(W[0][1][0], W[0][1][1], a0, bb1);
					dmma(W[1][1][0], W[1][1][1], a1, bb1);
				}
			}
			auto add = [&](double w0, double w1) {
				dmma(F0[0], F0[1], w0, w0);
				dmma(F1[0], F1[1], w1, w0);
				dmma(F2[0], F2[1], w1, w1);
			};
			add(W[0][0][0], W[1][0][0]);
			add(W[0][0][1], W[1][0][1]);
			if (nx > 8) add(W[0][1][0], W[1][1][0]);
			if (nx > 12) add(W[0][1][1], W[1][1][1]);
		}
		// zeros right of the diagonal; rows and columns >= m: an identity block,
		// whatever the padding holds
#pragma unroll
		for (int h = 0; h < 2; h++) {
			if (g < 2 * q + h) F0[h] = F2[h] = 0.0;
			if (m < 16) {
				if (g >= m) F0[h] = g == 2 * q + h ? 1.0 : 0.0;
				if (8 + g >= m) {
					F1[h] = 0.0;
					F2[h] = g == 2 * q + h ? 1.0 : 0.0;
				}
			}
		}
		sync();  // every read of stage k's inputs and of L_{k+1} is done
		if (k > 0) load(k - 1);
		double A0[2] = {F0[0], F0[1]}, A1[2] = {F1[0], F1[1]}, A2[2] = {F2[0], F2[1]}, keep[2] = {0.0, 0.0};
		panel<true>(A0, A1, keep, Ls, dv, pv, 0, g, q);
		dmma(A2[0], A2[1], -keep[0], keep[0]);
		dmma(A2[0], A2[1], -keep[1], keep[1]);
		panel<false>(A2, A1, keep, Ls, dv, pv, 8, g, q);
		__syncwarp();
		double iv = dv[lane & 15];
		bool odd = !(iv < __longlong_as_double(0x7ff0000000000000LL)) || !(Ls[(lane & 15) * (LD + 1)] >= 0.0);
		if (__any_sync(0xffffffffu, odd)) {
			// a pivot that panel() does not take: by rows (chol_frag.cuh)
			double G[3][2] = {{-F0[0], -F0[1]}, {-F1[0], -F1[1]}, {-F2[0], -F2[1]}};
			__syncwarp();
			frag::chol16_rows(G, dv - 16, lane);
			*(double2 *)(Ls + g * LD + 2 * q) = make_double2(G[0][0], G[0][1]);
			*(double2 *)(Ls + (8 + g) * LD + 2 * q) = make_double2(G[1][0], G[1][1]);
			*(double2 *)(Ls + (8 + g) * LD + 8 + 2 * q) = make_double2(G[2][0], G[2][1]);
			iv = dv[lane & 15];
		}
		const bool zero = lane < m && iv == 0.0;
		if (__any_sync(0xffffffffu, zero)) {
			// L_jj and 1 / L_jj of a pivot that is not positive: 0.  An infinite
			// pivot (1 / L_jj = 0, L_jj = inf * 0 = NaN) counts in info back to back,
			// where it is L_jj that must be positive, but not interleaved, where it
			// is the pivot (as in potrf_l on these slabs)
			if (zero) {
				if (!odd) Ls[lane * LD + lane] = 0.0;
				dv[lane] = 0.0;
			}
			const bool inf = INTER && zero && Ls[lane * LD + lane] != 0.0;
			const unsigned bad = __ballot_sync(0xffffffffu, zero && !inf);
			if (bad && first == 0) first = (N - k) * 16 + __ffs(bad);
			__syncwarp();
		}
	}
	sync();
	store_l<INTER>(a, 0, INTER ? b0 : b, INTER ? ric_sm : Ls, PS);
	if (lane == 0 && b < a.batch && a.info) a.info[b] = first;
}

template <bool INTER>
int launch(const Args &a, cudaStream_t s) {
	const size_t smem = (size_t)PC * prob_el(a.cnx) * sizeof(double);
	bf::smem_optin(k_ric_trf_dmma<INTER>, smem);
	k_ric_trf_dmma<INTER><<<(a.batch + PC - 1) / PC, NT, smem, s>>>(a);
	return bf::check_launch();
}

}  // namespace ric
