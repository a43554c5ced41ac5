// Cholesky panels in FP64 tensor core fragments, one warp per matrix.
//
// A matrix is a grid of 8 x 8 blocks, each an m8n8 accumulator fragment: lane
// (g, q) = (lane / 4, lane % 4) keeps row g, columns 2q and 2q + 1.  Summing a
// product L_I L_J^T over the columns in the order 0, 2, 4, 6 | 1, 3, 5, 7 makes
// these accumulators the operands of mma m8n8k4 as they are (k slot q holds
// column 2q, then 2q + 1), so factored blocks update others without a shuffle.
// A 64-bit shuffle occupies the SM's shuffle unit for about 8 cycles, which
// bounded the forms that broadcast by shuffles (n = 64: 1,200 32-bit shuffles
// per matrix, 136 of 171 us for 8,000 matrices).
#pragma once
#include "common.cuh"

#define CHOL_NB 16

// One column J of the 16x16 diagonal-block factorization; lane i holds row i
// of the block in r[] (compile-time indices only, so r stays in registers).
// The pivot is broadcast by a shuffle and every lane computes its reciprocal
// square root in FP64 (T = float: FP32 entries and updates, FP64 pivots);
// column J reaches the other rows by shuffles.  The pivot rule is applied
// without branches so the compiler can overlap the column update with the
// next pivot.  The terminal step records the first non-positive pivot
// (c0 + j + 1) in *bad by one ballot over the rows.
// WIDTH = 16 factors two independent blocks per warp, one per half-warp:
// `lane` is then the lane within the half (0..15), the shuffles stay inside
// the half, and each half records its own dinv / bad (the caller passes the
// half's pointers).  The whole warp executes the call.
template <int J, typename T = double, int WIDTH = 32>
struct DiagCol {
	static __device__ __forceinline__ void run(T (&r)[CHOL_NB], int lane, int nbk, int c0, double *dinv, int *bad) {
		const double cj = (double)__shfl_sync(0xffffffffu, r[J], J, WIDTH);
		const bool ok = cj > 0.0;
		const double inv = ok ? rsqrt(cj) : 0.0;
		r[J] = (lane == J) ? (T)(ok ? cj * inv : 0.0) : r[J] * (T)inv;
		if (lane == J && J < nbk) dinv[c0 + J] = inv;
#pragma unroll
		for (int l = J + 1; l < CHOL_NB; l++) {
			const T t = __shfl_sync(0xffffffffu, r[J], l, WIDTH);
			if (lane >= l) r[l] = fma(-r[J], t, r[l]);
		}
		DiagCol<J + 1, T, WIDTH>::run(r, lane, nbk, c0, dinv, bad);
	}
};
template <typename T, int WIDTH>
struct DiagCol<CHOL_NB, T, WIDTH> {
	static __device__ __forceinline__ void run(T (&r)[CHOL_NB], int lane, int nbk, int c0, double *, int *bad) {
		T d = T(1);
#pragma unroll
		for (int l = 0; l < CHOL_NB; l++)
			if (l == lane) d = r[l];
		unsigned m = __ballot_sync(0xffffffffu, lane < nbk && !(d > T(0)));
		if (WIDTH == 16) m = (m >> (threadIdx.x & 16)) & 0xffffu;  // this half-warp's rows
		if (m && lane == 0 && *bad == 0) *bad = c0 + __ffs(m);
	}
};

namespace frag {

__device__ __forceinline__ void dmma(double &d0, double &d1, double a, double b) {
	asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
	    : "+d"(d0), "+d"(d1)
	    : "d"(a), "d"(b));
}

// D += A B^T with A and B factored 8 x 8 blocks
__device__ __forceinline__ void update(double (&D)[2], const double (&A)[2], const double (&B)[2]) {
	dmma(D[0], D[1], A[0], B[0]);
	dmma(D[0], D[1], A[1], B[1]);
}

// Whether an inverse pivot of panel() or chol16() stands for a pivot that is not
// positive: -0 (an infinite pivot's inverse is +0)
__device__ __forceinline__ bool bad_pivot(double v) { return __double2hiint(v) < 0; }

// Whether the lane's entries of a diagonal block of L hold a NaN on the diagonal
__device__ __forceinline__ bool odd_diag(const double (&L)[2], int g, int q) {
	return (g == 2 * q && !(L[0] >= 0.0)) || (g == 2 * q + 1 && !(L[1] >= 0.0));
}

// Factor one 8-column panel: P[0] the diagonal block, P[1..] the blocks below
// it, holding -A on entry (zeros right of the diagonal) and L on return
// (undefined right of the diagonal).  Two columns (2p, 2p + 1: the lanes q = p)
// per step: their 2 x 2 pivot block reaches the warp through sc (16 entries of
// shared memory, 16-byte aligned), every lane forms both reciprocal pivots, the
// column lanes scale their rows and the rest of the panel gets two rank-1
// tensor core steps (one k slot in use: 6 steps of 15 cycles per block and
// panel, no chain through the lanes).  dv[0..7] receives the inverse pivots, -0
// for a pivot that is not positive (see bad_pivot; its L entry is then
// undefined: the caller stores 0).  Zeros as factors stand for masks, so this
// is only valid while every number is finite.  Any infinity or NaN in row i
// reaches pivot i; a pivot that is infinite, NaN or outside chol_rsqrt's range
// leaves an inverse that is not finite or a NaN on the diagonal of L (odd_diag),
// and the caller factors the matrix another way.
template <int NI>
__device__ __forceinline__ void panel(double (&P)[NI][2], double *sc, double *dv, int g, int q) {
#pragma unroll
	for (int p = 0; p < 4; p++) {
		const bool mine = q == p;
		double *s = sc + 4 * p;
		if (mine && g == 2 * p) s[0] = P[0][0];
		if (mine && g == 2 * p + 1) *(double2 *)(s + 2) = make_double2(P[0][0], P[0][1]);
		__syncwarp();
		const double d0 = -s[0];
		const double2 r1 = *(const double2 *)(s + 2);
		const double n0 = d0 > 0.0 ? -chol_rsqrt(d0) : 0.0;  // -1 / L_00
		const double l10 = r1.x * n0;
		const double d1 = -fma(l10, l10, r1.y);
		const double n1 = d1 > 0.0 ? -chol_rsqrt(d1) : 0.0;
		if (mine && (g >> 1) == p) dv[g] = (g & 1) ? -n1 : -n0;
		const double m0 = mine ? n0 : 0.0, m1 = mine ? n1 : 0.0;
		double l0[NI], l1[NI];
#pragma unroll
		for (int I = 0; I < NI; I++) {
			// rows above the pivots take no part
			l0[I] = P[I][0] * (I == 0 && g < 2 * p ? 0.0 : m0);
			l1[I] = fma(l0[I], l10, P[I][1]) * (I == 0 && g < 2 * p + 1 ? 0.0 : m1);
		}
		if (p < 3) {
			// the two steps of a block are a chain of 29 cycles each: every
			// block's first, then every block's second
#pragma unroll
			for (int I = 0; I < NI; I++) dmma(P[I][0], P[I][1], l0[I], l0[0]);
#pragma unroll
			for (int I = 0; I < NI; I++) dmma(P[I][0], P[I][1], l1[I], l1[0]);
		}
		if (mine) {
#pragma unroll
			for (int I = 0; I < NI; I++) {
				P[I][0] = l0[I];
				P[I][1] = l1[I];
			}
		}
	}
}

// chol16 by rows and shuffles (DiagCol), for matrices with a pivot that panel()
// does not take; F as there, scr + 16 receives the inverse pivots
static __device__ __noinline__ void chol16_rows(double (&F)[3][2], double *scr, int lane) {
	const int g = lane >> 2, q = lane & 3, i = lane & 15;
	double r[CHOL_NB];
#pragma unroll
	for (int j = 0; j < CHOL_NB; j++) {
		const int src = (i & 7) * 4 + ((j & 7) >> 1), h = j & 1;
		const double lo = __shfl_sync(0xffffffffu, F[j < 8 ? 0 : 2][h], src), hi = __shfl_sync(0xffffffffu, F[j < 8 ? 1 : 2][h], src);
		r[j] = j > i ? 0.0 : -(i < 8 ? lo : hi);
	}
	int bad = 0;
	DiagCol<0, double>::run(r, lane, CHOL_NB, 0, scr + 16, &bad);
	double d = 0.0;
#pragma unroll
	for (int j = 0; j < CHOL_NB; j++) {
		if (j == i) d = r[j];
		const double lo = __shfl_sync(0xffffffffu, r[j], g), hi = __shfl_sync(0xffffffffu, r[j], 8 + g);
		if ((j & 7) == 2 * q + (j & 1)) {
			if (j < 8) {
				F[0][j & 1] = lo;
				F[1][j & 1] = hi;
			} else {
				F[2][j & 1] = hi;
			}
		}
	}
	__syncwarp();
	if (lane < 16 && !(d > 0.0)) scr[16 + lane] = -0.0;
	__syncwarp();
}

// Cholesky of a 16 x 16 matrix: F its blocks (0,0), (1,0), (1,1), -A on entry
// (zeros right of the diagonal), L on return (undefined right of the diagonal,
// 0 for a pivot that is not positive).  scr: 32 entries of shared memory
// (16-byte aligned); returns lane % 16's inverse pivot (bad_pivot).  About 2,000
// cycles, against 3,700 alone and 7,500 with 8 such warps on the SM for the
// form with a row per lane and shuffles.
__device__ __forceinline__ double chol16(double (&F)[3][2], double *scr, int lane) {
	const int g = lane >> 2, q = lane & 3;
	double P[2][2] = {{F[0][0], F[0][1]}, {F[1][0], F[1][1]}}, D[1][2] = {{F[2][0], F[2][1]}};
	panel<2>(P, scr, scr + 16, g, q);
	update(D[0], P[1], P[1]);
	panel<1>(D, scr, scr + 24, g, q);
	__syncwarp();
	double v = scr[16 + (lane & 15)];
	if (__any_sync(0xffffffffu, !(v < __longlong_as_double(0x7ff0000000000000LL)) || odd_diag(P[0], g, q) ||
	                                odd_diag(D[0], g, q))) {
		double G[3][2] = {{F[0][0], F[0][1]}, {F[1][0], F[1][1]}, {F[2][0], F[2][1]}};
		chol16_rows(G, scr, lane);
#pragma unroll
		for (int b = 0; b < 3; b++) {
			F[b][0] = G[b][0];
			F[b][1] = G[b][1];
		}
		return scr[16 + (lane & 15)];
	}
	const bool z0 = bad_pivot(scr[16 + g]), z1 = bad_pivot(scr[24 + g]);
#pragma unroll
	for (int h = 0; h < 2; h++) {
		const bool dg = g == 2 * q + h;
		F[0][h] = (dg && z0) ? 0.0 : P[0][h];
		F[1][h] = P[1][h];
		F[2][h] = (dg && z1) ? 0.0 : D[0][h];
	}
	return v;
}

}  // namespace frag
