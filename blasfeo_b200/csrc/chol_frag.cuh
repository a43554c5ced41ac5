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

// Factor one 8-column panel: P[0] the diagonal block, P[1..] the blocks below
// it, holding -A on entry (finite values right of the diagonal) and L on
// return (undefined right of the diagonal).  Two columns (2p, 2p + 1: the lanes
// q = p) per step: their 2 x 2 pivot block reaches the warp through sc (16
// entries of shared memory, 16-byte aligned), every lane forms both reciprocal
// pivots, the column lanes scale their rows and the rest of the panel gets two
// rank-1 tensor core steps (one k slot in use: 6 steps of 15 cycles per block
// and panel, no chain through the lanes).  dv[0..7] receives the inverse
// pivots, 0 for a pivot that is not positive (its L entry is then 0 or
// undefined: the caller stores 0).  FAST: see chol_rsqrt; a pivot outside its
// range leaves an inverse that is not finite.
template <int NI, bool FAST>
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
		const bool ok0 = d0 > 0.0;
		const double v0 = FAST ? chol_rsqrt(d0) : rsqrt(d0);
		const double n0 = ok0 ? -v0 : 0.0;              // -1 / L_00
		const double l10 = r1.x * n0;
		const double d1 = -fma(l10, l10, r1.y);
		const bool ok1 = d1 > 0.0;
		const double v1 = FAST ? chol_rsqrt(d1) : rsqrt(d1);
		const double n1 = ok1 ? -v1 : 0.0;
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

}  // namespace frag
