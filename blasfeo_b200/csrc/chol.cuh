// CTA-level Cholesky of a matrix held in shared memory, used by potrf_l and by
// the fused factor+solve kernels.
//
// Shared-memory layout ("lower panels"): the lower triangle of an n x n matrix
// as P = ceil(n/4) row panels; panel p (rows 4p..4p+3) keeps the 4x4 tiles
// 0..p, i.e. the BLASFEO panel layout with everything right of the diagonal
// tile dropped.  Panel p starts at element 8p(p+1); tile (p,q) is 16
// contiguous elements, column-major inside the tile.  Inside a tile the
// 16-byte chunks are XOR-swizzled with (p+q): threads that read different
// tiles of one tile row or one tile column then hit different banks (every
// tile starts on a 128-byte (FP64) / 64-byte (FP32) boundary, so without the
// swizzle all of them would collide on the same banks).
// Padding rows/columns (n..4P-1) hold the identity so they factor to the
// identity and never touch real entries.
//
// Algorithm: right-looking, 16 columns (4 panels) per block step, two
// __syncthreads per step:
//   A. all threads: panel of block column K by substitution with the
//      factored diagonal block (one row per thread, the reciprocal pivots
//      multiplied in);
//   B. warp 0 (critical path): rank-16 update of the 16x16 diagonal block K+1
//      and its factorization in FP64 fragments (chol_diag; pivot rule of
//      kernel/generic/kernel_dgemm_4x4_lib4.c:5700-5710: c>0 -> sqrt(c) and its
//      reciprocal, else 0 and 0); the warps on the other three schedulers:
//      rank-16 update of the rest of the trailing matrix (8 x 4 tile blocks
//      per warp), which hides the serial diagonal work.
// With inv_diag the diagonal blocks are replaced at the end by their explicit
// inverses (FP64 arithmetic, all blocks in parallel) for the blocked
// triangular solves of the factor+solve kernels.
#pragma once
#include "chol_frag.cuh"
#include "common.cuh"

__host__ __device__ __forceinline__ int lp_off(int p) { return 8 * p * (p + 1); }
__host__ __device__ __forceinline__ int lp_size(int n) {
	int P = (n + 3) / 4;
	return 8 * P * (P + 1);
}

// physical index of element (i,j) (j <= 4*(i/4)+3) in the swizzled lower panels
template <typename T>
__device__ __forceinline__ int lp_idx(int i, int j);
template <>
__device__ __forceinline__ int lp_idx<double>(int i, int j) {
	const int p = i >> 2, q = j >> 2;
	const int e = ((j & 3) << 2) | (i & 3);
	return lp_off(p) + 16 * q + ((((e >> 1) ^ ((p + q) & 7)) << 1) | (e & 1));
}
template <>
__device__ __forceinline__ int lp_idx<float>(int i, int j) {
	const int p = i >> 2, q = j >> 2;
	return lp_off(p) + 16 * q + ((((j & 3) ^ ((p + q) & 3)) << 2) | (i & 3));
}
template <typename T>
__device__ __forceinline__ T &lp_at(T *S, int i, int j) {
	return S[lp_idx<T>(i, j)];
}
template <typename T>
__device__ __forceinline__ const T &lp_at(const T *S, int i, int j) {
	return S[lp_idx<T>(i, j)];
}

// column c (0..3) of tile (p,q): the 4 rows as a, b, c, d
template <typename T>
__device__ __forceinline__ void tile_col_ld(const T *S, int p, int q, int c, T &a0, T &a1, T &a2, T &a3);
template <>
__device__ __forceinline__ void tile_col_ld<double>(const double *S, int p, int q, int c, double &a0, double &a1,
                                                    double &a2, double &a3) {
	const double *t = S + lp_off(p) + 16 * q;
	const int s = (p + q) & 7;
	double2 v0 = *(const double2 *)(t + (((2 * c) ^ s) << 1));
	double2 v1 = *(const double2 *)(t + (((2 * c + 1) ^ s) << 1));
	a0 = v0.x; a1 = v0.y; a2 = v1.x; a3 = v1.y;
}
template <>
__device__ __forceinline__ void tile_col_ld<float>(const float *S, int p, int q, int c, float &a0, float &a1,
                                                   float &a2, float &a3) {
	const float *t = S + lp_off(p) + 16 * q;
	float4 v = *(const float4 *)(t + ((c ^ ((p + q) & 3)) << 2));
	a0 = v.x; a1 = v.y; a2 = v.z; a3 = v.w;
}
template <typename T>
__device__ __forceinline__ void tile_col_st(T *S, int p, int q, int c, T a0, T a1, T a2, T a3);
template <>
__device__ __forceinline__ void tile_col_st<double>(double *S, int p, int q, int c, double a0, double a1, double a2,
                                                    double a3) {
	double *t = S + lp_off(p) + 16 * q;
	const int s = (p + q) & 7;
	*(double2 *)(t + (((2 * c) ^ s) << 1)) = make_double2(a0, a1);
	*(double2 *)(t + (((2 * c + 1) ^ s) << 1)) = make_double2(a2, a3);
}
template <>
__device__ __forceinline__ void tile_col_st<float>(float *S, int p, int q, int c, float a0, float a1, float a2,
                                                   float a3) {
	float *t = S + lp_off(p) + 16 * q;
	*(float4 *)(t + ((c ^ ((p + q) & 3)) << 2)) = make_float4(a0, a1, a2, a3);
}

// map a linear index over the lower-triangular tile set {(ti,tj): 0<=tj<=ti<R}
__device__ __forceinline__ void tri_index(int t, int &ti, int &tj) {
	int r = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
	while ((r + 1) * (r + 2) / 2 <= t) r++;
	while (r * (r + 1) / 2 > t) r--;
	ti = r;
	tj = t - r * (r + 1) / 2;
}

// Doubles of scratch of the diagonal blocks: the row-major copy Lt (16 x 17,
// sized for FP64), then what frag::chol16 needs
constexpr int CHOL_SCR = 16 * 17 + 32;

// Warp 0: the diagonal block at column c0n (nbk <= 16 real columns; the
// padding is the identity), in FP64 tensor core fragments whatever T is.
// c0 >= 0 (look-ahead step): first its rank-16 update with the panel of block
// column c0 (already solved).  Writes L_KK back into S, 1/L_jj into
// dinv[c0n + j] (FP64), the first bad pivot (c0n + j + 1) into *bad, and for
// the panel solve a row-major 16x17 copy Lt of L_KK in the working precision
// with the reciprocal pivots in column 16.  This block is the critical path of
// the factorization; with a row per lane and shuffles it waited for the
// shared-memory / shuffle unit that the update warps keep busy (n = 256, FP32:
// 11.7k cycles per block beside a full trailing update).
template <typename T>
__device__ void chol_diag(T *S, int c0n, int nbk, int c0, double *dinv, T *Lt, int *bad) {
	const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
	double *scr = (double *)Lt + 16 * 17;
	double F[3][2];
#pragma unroll
	for (int h = 0; h < 2; h++) {
		const int j = 2 * q + h;
		const bool r0 = g < nbk, r1 = 8 + g < nbk;
		F[0][h] = r0 ? (j <= g ? -(double)lp_at(S, c0n + g, c0n + j) : 0.0) : (j == g ? -1.0 : 0.0);
		F[1][h] = r1 ? -(double)lp_at(S, c0n + 8 + g, c0n + j) : 0.0;
		F[2][h] = r1 ? (j <= g ? -(double)lp_at(S, c0n + 8 + g, c0n + 8 + j) : 0.0) : (j == g ? -1.0 : 0.0);
	}
	if (c0 >= 0) {
		double a0[4], a1[4];
#pragma unroll
		for (int ks = 0; ks < 4; ks++) {
			a0[ks] = g < nbk ? (double)lp_at(S, c0n + g, c0 + 4 * ks + q) : 0.0;
			a1[ks] = 8 + g < nbk ? (double)lp_at(S, c0n + 8 + g, c0 + 4 * ks + q) : 0.0;
		}
#pragma unroll
		for (int ks = 0; ks < 4; ks++) {
			frag::dmma(F[0][0], F[0][1], a0[ks], a0[ks]);
			frag::dmma(F[1][0], F[1][1], a1[ks], a0[ks]);
			frag::dmma(F[2][0], F[2][1], a1[ks], a1[ks]);
		}
	}
	const double v = frag::chol16(F, scr, lane);
	const unsigned m = __ballot_sync(0xffffffffu, lane < nbk && frag::bad_pivot(v));
	if (m && lane == 0 && *bad == 0) *bad = c0n + __ffs(m);
	if (lane < nbk) dinv[c0n + lane] = fabs(v);
	if (lane < 16) Lt[lane * 17 + 16] = (T)fabs(v);
#pragma unroll
	for (int h = 0; h < 2; h++) {
		const int j = 2 * q + h;
		const T l0 = j <= g ? (T)F[0][h] : T(0), l1 = (T)F[1][h], l2 = j <= g ? (T)F[2][h] : T(0);
		Lt[g * 17 + j] = l0;
		Lt[g * 17 + 8 + j] = T(0);
		Lt[(8 + g) * 17 + j] = l1;
		Lt[(8 + g) * 17 + 8 + j] = l2;
		if (g < nbk && j <= g) lp_at(S, c0n + g, c0n + j) = l0;
		if (8 + g < nbk) {
			lp_at(S, c0n + 8 + g, c0n + j) = l1;
			if (j <= g) lp_at(S, c0n + 8 + g, c0n + 8 + j) = l2;
		}
	}
	__syncwarp();
}

// panel of block column c0, rows r in [rbeg, rend): substitution with the
// diagonal block, L[r][c0+c] = (A[r][c0+c] - sum_{l<c} L[r][c0+l] L_KK[c][l]) * inv_c
template <typename T>
__device__ __forceinline__ void chol_panel_rows(T *S, int c0, int rbeg, int rend, int tid0, int nthr, const T *Lt) {
	const int kb = c0 >> 2;
	for (int r = rbeg + tid0; r < rend; r += nthr) {
		const int p = r >> 2, ri = r & 3;
		T *row = S + lp_off(p) + 16 * kb;
		int idx[CHOL_NB];
#pragma unroll
		for (int l = 0; l < CHOL_NB; l++) {
			const int qq = l >> 2, e = ((l & 3) << 2) | ri;
			idx[l] = 16 * qq + (sizeof(T) == 4 ? ((((l & 3) ^ ((p + kb + qq) & 3)) << 2) | ri)
			                                   : ((((e >> 1) ^ ((p + kb + qq) & 7)) << 1) | (e & 1)));
		}
		T a[CHOL_NB];
#pragma unroll
		for (int l = 0; l < CHOL_NB; l++) a[l] = row[idx[l]];
#pragma unroll
		for (int c = 0; c < CHOL_NB; c++) {
			T s = a[c];
#pragma unroll
			for (int l = 0; l < c; l++) s = fma(-a[l], Lt[c * 17 + l], s);
			a[c] = s * Lt[c * 17 + 16];
		}
#pragma unroll
		for (int l = 0; l < CHOL_NB; l++) row[idx[l]] = a[l];
	}
}

// Explicit inverse of diagonal block K (row-major 16x16, stored as T) from the
// factor in S and the FP64 reciprocal pivots; lane c computes column c.
template <typename T>
__device__ void chol_block_inverse(const T *S, int n, int K, const double *dinv, T *invL, int lane) {
	const int c0 = 16 * K;
	const int nbk = min(CHOL_NB, n - c0);
	const int c = lane;
	if (c >= CHOL_NB) return;
	double x[CHOL_NB];
#pragma unroll
	for (int i = 0; i < CHOL_NB; i++) {
		double s = (i == c) ? 1.0 : 0.0;
#pragma unroll
		for (int l = 0; l < i; l++) {
			const double lil = (i < nbk && l < nbk) ? (double)lp_at(S, c0 + i, c0 + l) : 0.0;
			s = fma(-lil, x[l], s);
		}
		const double di = (i < nbk) ? dinv[c0 + i] : 1.0;
		x[i] = (i < c) ? 0.0 : s * di;
	}
#pragma unroll
	for (int i = 0; i < CHOL_NB; i++) invL[i * CHOL_NB + c] = (T)x[i];
}

// Diagonal block K of the factor in S replaced by its inverse (lower
// triangular, same tiles, working precision), from the factor in S and the
// FP64 reciprocal pivots; lane c computes column c.  Only the real rows and
// columns (< n) are written; the whole warp calls it.
template <typename T>
__device__ void chol_block_inverse_inplace(T *S, int n, int K, const double *dinv, int lane) {
	const int c0 = 16 * K;
	const int nbk = min(CHOL_NB, n - c0);
	const int c = lane & 15;
	double x[CHOL_NB];
#pragma unroll
	for (int i = 0; i < CHOL_NB; i++) {
		double s = (i == c) ? 1.0 : 0.0;
#pragma unroll
		for (int l = 0; l < i; l++) {
			const double lil = (i < nbk && l < nbk) ? (double)lp_at(S, c0 + i, c0 + l) : 0.0;
			s = fma(-lil, x[l], s);
		}
		const double di = (i < nbk) ? dinv[c0 + i] : 1.0;
		x[i] = (i < c) ? 0.0 : s * di;
	}
	__syncwarp();  // every lane has read the block before any lane overwrites it
	if (lane < CHOL_NB && c < nbk) {
#pragma unroll
		for (int i = 0; i < CHOL_NB; i++)
			if (i >= c && i < nbk) lp_at(S, c0 + i, c0 + c) = (T)x[i];
	}
	__syncwarp();
}

// rank-16 update of tile (ti,tj) with the panel at block column c0
template <typename T>
__device__ __forceinline__ void chol_tile_update(T *S, int ti, int tj, int c0) {
	T acc[16];
	const int kb = c0 >> 2;
#pragma unroll
	for (int q = 0; q < 4; q++) tile_col_ld<T>(S, ti, tj, q, acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]);
	const T *pa = S + lp_off(ti) + 16 * kb;
	const T *pb = S + lp_off(tj) + 16 * kb;
#pragma unroll
	for (int qq = 0; qq < 4; qq++) {
		// tile kb+qq of row panels ti and tj; column slices with the tile swizzle
		const T *ta = pa + 16 * qq, *tb = pb + 16 * qq;
		const int sa = ti + kb + qq, sb = tj + kb + qq;
#pragma unroll
		for (int c = 0; c < 4; c++) {
			T a0, a1, a2, a3, b0, b1, b2, b3;
			if (sizeof(T) == 4) {
				float4 va = *(const float4 *)(ta + ((c ^ (sa & 3)) << 2));
				float4 vb = *(const float4 *)(tb + ((c ^ (sb & 3)) << 2));
				a0 = (T)va.x; a1 = (T)va.y; a2 = (T)va.z; a3 = (T)va.w;
				b0 = (T)vb.x; b1 = (T)vb.y; b2 = (T)vb.z; b3 = (T)vb.w;
			} else {
				double2 va0 = *(const double2 *)(ta + (((2 * c) ^ (sa & 7)) << 1));
				double2 va1 = *(const double2 *)(ta + (((2 * c + 1) ^ (sa & 7)) << 1));
				double2 vb0 = *(const double2 *)(tb + (((2 * c) ^ (sb & 7)) << 1));
				double2 vb1 = *(const double2 *)(tb + (((2 * c + 1) ^ (sb & 7)) << 1));
				a0 = (T)va0.x; a1 = (T)va0.y; a2 = (T)va1.x; a3 = (T)va1.y;
				b0 = (T)vb0.x; b1 = (T)vb0.y; b2 = (T)vb1.x; b3 = (T)vb1.y;
			}
			// acc[4*q + r] is element (row r of ti, column q of tj)
			acc[0] = fma(-a0, b0, acc[0]); acc[1] = fma(-a1, b0, acc[1]);
			acc[2] = fma(-a2, b0, acc[2]); acc[3] = fma(-a3, b0, acc[3]);
			acc[4] = fma(-a0, b1, acc[4]); acc[5] = fma(-a1, b1, acc[5]);
			acc[6] = fma(-a2, b1, acc[6]); acc[7] = fma(-a3, b1, acc[7]);
			acc[8] = fma(-a0, b2, acc[8]); acc[9] = fma(-a1, b2, acc[9]);
			acc[10] = fma(-a2, b2, acc[10]); acc[11] = fma(-a3, b2, acc[11]);
			acc[12] = fma(-a0, b3, acc[12]); acc[13] = fma(-a1, b3, acc[13]);
			acc[14] = fma(-a2, b3, acc[14]); acc[15] = fma(-a3, b3, acc[15]);
		}
	}
#pragma unroll
	for (int q = 0; q < 4; q++) tile_col_st<T>(S, ti, tj, q, acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]);
}

// Full factorization of the n x n lower-panel matrix S by the whole CTA
// (blockDim.x >= 64).  dinv: FP64 shared array of >= 4P entries; Lt: CHOL_SCR
// doubles (16-byte aligned), the row-major diagonal block first; bad: shared int (0 on entry).  With inv_diag the diagonal
// blocks of the factor are replaced at the end by their explicit inverses
// (all blocks in parallel), for the blocked triangular solves; the blocks
// below the diagonal keep L.  w (optional, shared, 16 ceil(n/16) entries, zeros
// from n on): overwritten by L^{-1} w, as one more row of each panel solve whose
// update of the entries below runs beside the trailing update, so that the
// forward substitution has no chain and no barriers of its own.
template <typename T>
__device__ void chol_smem(T *S, int n, double *dinv, T *Lt, int *bad, bool inv_diag, T *w = nullptr) {
	const int P = (n + 3) >> 2;
	const int NB = (n + 15) >> 4;
	const int tid = threadIdx.x, nt = blockDim.x;
	const int warp = tid >> 5, lane = tid & 31;
	if (warp == 0) chol_diag<T>(S, 0, min(CHOL_NB, n), -1, dinv, Lt, bad);
	__syncthreads();
	for (int K = 0; K < NB; K++) {
		const int c0 = 16 * K, k0 = 4 * K;
		// A. panel rows below the diagonal block
		chol_panel_rows<T>(S, c0, c0 + CHOL_NB, 4 * P, tid, nt, Lt);
		if (w && tid == nt - 1) {
			T a[CHOL_NB];
#pragma unroll
			for (int c = 0; c < CHOL_NB; c++) {
				T s = w[c0 + c];
#pragma unroll
				for (int l = 0; l < c; l++) s = fma(-a[l], Lt[c * 17 + l], s);
				a[c] = s * Lt[c * 17 + 16];
			}
#pragma unroll
			for (int c = 0; c < CHOL_NB; c++) w[c0 + c] = a[c];
		}
		__syncthreads();
		if (K + 1 >= NB) break;
		// B. trailing tiles (ti,tj), k0+4 <= tj <= ti < P; the 10 of the
		// diagonal block K+1 belong to warp 0, which then factors that block
		const int R = P - (k0 + 4);
		if (warp == 0) {
			chol_diag<T>(S, c0 + CHOL_NB, min(CHOL_NB, n - c0 - CHOL_NB), c0, dinv, Lt, bad);
		} else if (warp & 3) {
			// warps 4, 8, ... share warp 0's scheduler (warp w issues from
			// sub-partition w % 4): they sit the update out so that the serial
			// diagonal chain keeps its issue slots
			// A warp takes an 8 x 4 block of tiles (8 tile rows, 4 tile columns;
			// lane l: row l / 4, column l % 4): each tile column slice of the
			// panel is then read by 4 lanes and each tile row slice by 8 lanes
			// at once (broadcast), 12 distinct 16-byte loads per 32 tile
			// updates instead of 33 for 32 tiles of one tile row.  Shared-memory
			// bandwidth bounds this update, and its traffic also delays the
			// diagonal warp's loads and shuffles.  Tiles above the diagonal or
			// past the matrix are skipped; the tiles of block K+1 (rows < 4)
			// belong to warp 0.
			const int nuw = (nt >> 5) - ((nt >> 5) + 3) / 4;
			const int uw = warp - (warp >> 2) - 1;
			if (w) {
				for (int i = c0 + CHOL_NB + 32 * uw + lane; i < n; i += 32 * nuw) {
					T s = w[i];
#pragma unroll
					for (int l = 0; l < CHOL_NB; l++) s = fma(-lp_at(S, i, c0 + l), w[c0 + l], s);
					w[i] = s;
				}
			}
			const int scmax = (R + 3) >> 2, sr = (R + 7) >> 3;
			int si = 0, base = 0, cnt = scmax < 2 ? scmax : 2;
			for (int sidx = uw;; sidx += nuw) {
				while (si < sr && sidx >= base + cnt) {
					base += cnt;
					si++;
					cnt = (2 * si + 2 < scmax) ? 2 * si + 2 : scmax;
				}
				if (si >= sr) break;
				const int ti = 8 * si + (lane >> 2), tj = 4 * (sidx - base) + (lane & 3);
				if (ti < R && ti >= 4 && tj <= ti) chol_tile_update<T>(S, ti + k0 + 4, tj + k0 + 4, c0);
			}
		}
		__syncthreads();
	}
	if (inv_diag) {
		const int nw = nt >> 5;
		for (int K = warp; K < NB; K += nw) chol_block_inverse_inplace<T>(S, n, K, dinv, lane);
		__syncthreads();
	}
}

// Panel index of 4-element chunk ch of the lower panels (panel p holds
// 4(p+1) chunks; chunks before panel p: 2p(p+1)).
__device__ __forceinline__ int lp_chunk_panel(int ch) {
	int p = (int)((sqrtf(2.0f * (float)ch + 1.0f) - 1.0f) * 0.5f);
	while (2 * (p + 1) * (p + 2) <= ch) p++;
	while (2 * p * (p + 1) > ch) p--;
	return p;
}

// Load the lower triangle of an n x n panel-major matrix (row offset a
// multiple of 4: panel p of the lower triangle is the contiguous run
// src[4p*cn .. 4p*cn + 16(p+1)) ) into swizzled lower panels of type TD,
// identity in the padding.  Each thread moves 4-element column slices,
// UNR of them in flight.  slot (optional): unswizzled FP64 copy.
template <typename TD, typename TS, int UNR>
__device__ void load_lp_vec(TD *S, int n, const TS *__restrict__ src, int cn, double *slot) {
	const int P = (n + 3) >> 2;
	const int nch = 2 * P * (P + 1);
	const int tid = threadIdx.x, nt = blockDim.x;
	for (int base = tid; base < nch; base += UNR * nt) {
		TS v[UNR][4];
		int pp[UNR], cc[UNR];
#pragma unroll
		for (int u = 0; u < UNR; u++) {
			const int ch = base + u * nt;
			pp[u] = -1;
			if (ch < nch) {
				const int p = lp_chunk_panel(ch);
				const int col = ch - 2 * p * (p + 1);
				pp[u] = p;
				cc[u] = col;
				const TS *g = src + (size_t)(4 * p) * cn + 4 * col;
				if (sizeof(TS) == 8) {
					double2 x0 = __ldg((const double2 *)g), x1 = __ldg((const double2 *)g + 1);
					v[u][0] = (TS)x0.x; v[u][1] = (TS)x0.y; v[u][2] = (TS)x1.x; v[u][3] = (TS)x1.y;
				} else {
					float4 x = __ldg((const float4 *)g);
					v[u][0] = (TS)x.x; v[u][1] = (TS)x.y; v[u][2] = (TS)x.z; v[u][3] = (TS)x.w;
				}
			}
		}
#pragma unroll
		for (int u = 0; u < UNR; u++) {
			const int p = pp[u];
			if (p < 0) continue;
			const int j = cc[u];
			TD o[4];
			double d[4];
#pragma unroll
			for (int r = 0; r < 4; r++) {
				const int i = 4 * p + r;
				double x;
				if (i < n && j < n)
					x = (j <= i) ? (double)v[u][r] : 0.0;
				else
					x = (i == j) ? 1.0 : 0.0;
				d[r] = x;
				o[r] = (TD)x;
			}
			tile_col_st<TD>(S, p, j >> 2, j & 3, o[0], o[1], o[2], o[3]);
			if (slot) {
				double *sd = slot + lp_off(p) + 4 * j;
				*(double2 *)sd = make_double2(d[0], d[1]);
				*(double2 *)(sd + 2) = make_double2(d[2], d[3]);
			}
		}
	}
}

// Store the lower triangle (j <= i < n) of swizzled lower panels into a
// panel-major matrix with panel-aligned row offset (see load_lp_vec).
template <typename T, int UNR>
__device__ void store_lp_vec(const T *S, int n, T *dst, int cn) {
	const int P = (n + 3) >> 2;
	const int nch = 2 * P * (P + 1);
	const int tid = threadIdx.x, nt = blockDim.x;
	for (int base = tid; base < nch; base += UNR * nt) {
#pragma unroll
		for (int u = 0; u < UNR; u++) {
			const int ch = base + u * nt;
			if (ch >= nch) continue;
			const int p = lp_chunk_panel(ch);
			const int j = ch - 2 * p * (p + 1);
			if (j >= n) continue;
			T o0, o1, o2, o3;
			tile_col_ld<T>(S, p, j >> 2, j & 3, o0, o1, o2, o3);
			T *g = dst + (size_t)(4 * p) * cn + 4 * j;
			if (j < 4 * p && 4 * p + 3 < n) {
				if (sizeof(T) == 8) {
					*(double2 *)g = make_double2((double)o0, (double)o1);
					*((double2 *)g + 1) = make_double2((double)o2, (double)o3);
				} else {
					*(float4 *)g = make_float4((float)o0, (float)o1, (float)o2, (float)o3);
				}
			} else {
				const T o[4] = {o0, o1, o2, o3};
#pragma unroll
				for (int r = 0; r < 4; r++)
					if (4 * p + r < n && j <= 4 * p + r) g[r] = o[r];
			}
		}
	}
}
