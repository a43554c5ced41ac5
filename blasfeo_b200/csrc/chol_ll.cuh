// FP64 Cholesky of one matrix per CTA whose lower triangle does not fit in
// shared memory (the reference's dpotrf_l, blasfeo_hp_pm/d_lapack_lib4.c:918,
// for n beyond the shared-memory kernels), and the two triangular solves of
// the factor+solve chain (dtrsv_lnn / dtrsv_ltn) on the result.
//
// Left-looking by 16-column panels K (columns c0 = 16K .. c0+15):
//   update:  the panel (rows c0..n-1) starts from C and receives
//            -L(rows, 0:c0) L(c0:c0+16, 0:c0)^T on the FP64 tensor cores
//            (DMMA m8n8k4; every warp owns 8-row fragment rows, the operand
//            fragments are read from the factored columns in global memory --
//            two 128-byte runs each in the panel layout, L2-resident while the
//            CTA works on the matrix);
//   factor:  warp 0 updates and factors the 16 x 16 diagonal block in its
//            fragments (frag::chol16: pivot rule of
//            kernel/generic/kernel_dgemm_4x4_lib4.c:5700-5710) while the other
//            warps update the rows below, then the rows below solve their 16
//            entries against it (one thread per row, reciprocal-pivot multiply);
//   store:   the finished panel goes to D once, 1/L_jj to D's dA.
// The forward substitution of the solver (dtrsv_lnn) rides along: the right-hand
// side is one more row of the panel solve, and the rows below take its update
// while the panel is still in shared memory.
// Every element of L is written once and read back only by later panels'
// updates, so D may alias C.  Rows and columns n..16*ceil(n/16)-1 act as the
// identity.
#pragma once
#include "chol.cuh"
#include "common.cuh"

constexpr int LL_PSTR = 17;  // shared-memory panel row stride (doubles)

// doubles of the panel for an n x n matrix (what follows 16-byte aligned)
__host__ __device__ inline size_t ll_panel(int n) { return ((size_t)(n + 8) * LL_PSTR + 1) & ~(size_t)1; }
// shared memory of chol_ll for matrices up to max_n: the panel, whose first 16 rows
// are the diagonal factor with its reciprocal pivots in column 16, then 16x17
// entries for the factorization's scratch
__host__ __device__ inline size_t ll_smem_bytes(int max_n) { return (ll_panel(max_n) + 16 * 17) * sizeof(double); }

__device__ __forceinline__ void ll_dmma(double &d0, double &d1, double a, double b) {
	asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
	             : "+d"(d0), "+d"(d1)
	             : "d"(a), "d"(b));
}

// acc[u] += L(rows of fragment u, 0:c0) L(c0 + 0..7 | 8..15, 0:c0)^T.  ap[u]: row
// of the lane in fragment u, b0 / b1: rows c0 + lane/4 and + 8, all at column
// lane%4 of the factored columns (consecutive columns 4 elements apart).
// UNR steps of 8 columns have their loads in flight.
template <int FR, int UNR>
__device__ __forceinline__ void ll_update(double (&acc)[FR][2][2], const double *const (&ap)[FR], const double *b0,
                                          const double *b1, int c0) {
#pragma unroll
	for (int u = 0; u < FR; u++) acc[u][0][0] = acc[u][0][1] = acc[u][1][0] = acc[u][1][1] = 0.0;
#pragma unroll UNR
	for (int k = 0; k < c0; k += 8) {
		double a[FR][2], b[2][2];
#pragma unroll
		for (int h = 0; h < 2; h++) {
			b[0][h] = b0[4 * k + 16 * h];
			b[1][h] = b1[4 * k + 16 * h];
#pragma unroll
			for (int u = 0; u < FR; u++) a[u][h] = ap[u][4 * k + 16 * h];
		}
#pragma unroll
		for (int h = 0; h < 2; h++)
#pragma unroll
			for (int u = 0; u < FR; u++) {
				ll_dmma(acc[u][0][0], acc[u][0][1], a[u][h], b[0][h]);
				ll_dmma(acc[u][1][0], acc[u][1][1], a[u][h], b[1][h]);
			}
	}
}

// Factor the n x n lower triangle of c into d (lower triangle of L, 1/L_jj in
// d.d[j]); *bad (shared, zeroed by the caller) receives the first
// non-positive pivot j+1.  All NT threads of the CTA call it.  FR: fragment
// rows a warp updates at a time.  y (optional, shared memory, n doubles):
// overwritten by L^{-1} y.
template <int NT, int FR, int UNR>
__device__ void chol_ll(const PMat<double> &c, const PMat<double> &d, int n, double *smem, int *bad,
                        double *y = nullptr) {
	__shared__ int next;  // fragment rows claimed in the panel at hand
	double *pan = smem;
	double *Lt = pan;  // row stride LL_PSTR = 17
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int r = lane >> 2, q = lane & 3;
	const int NBK = (n + 15) >> 4;
	if (tid == 0) next = 2;
	__syncthreads();
	for (int K = 0; K < NBK; K++) {
		const int c0 = 16 * K;
		const int m = n - c0;
		const int nbk = m < 16 ? m : 16;
		const int R = (m + 7) >> 3;
		// rows past the matrix read its last row; what they give is never used
		auto rowp = [&](int row) { return d.addr(row < n ? row : n - 1, q); };
		const double *b0 = rowp(c0 + r), *b1 = rowp(c0 + 8 + r);
		// ---- diagonal block: its update and factorization in warp 0's fragments,
		// beside the other warps' updates of the rows below ----
		if (warp == 0) {
			double *scr = pan + ll_panel(n);
			double cv[3][2];
#pragma unroll
			for (int h = 0; h < 2; h++) {
				const int j = 2 * q + h;
				cv[0][h] = j <= r && r < m ? *c.addr(c0 + r, c0 + j) : (j == r ? 1.0 : 0.0);
				cv[1][h] = 8 + r < m ? *c.addr(c0 + 8 + r, c0 + j) : 0.0;
				cv[2][h] = j <= r && 8 + r < m ? *c.addr(c0 + 8 + r, c0 + 8 + j) : (j == r ? 1.0 : 0.0);
			}
			double acc[2][2][2];
			const double *const ap[2] = {b0, b1};
			ll_update<2, 2>(acc, ap, b0, b1, c0);
			double F[3][2];
#pragma unroll
			for (int h = 0; h < 2; h++) {
				const bool lo = 2 * q + h <= r;
				F[0][h] = (lo && r < m ? acc[0][0][h] : 0.0) - cv[0][h];
				F[1][h] = (8 + r < m ? acc[1][0][h] : 0.0) - cv[1][h];
				F[2][h] = (lo && 8 + r < m ? acc[1][1][h] : 0.0) - cv[2][h];
			}
			double v = frag::chol16(F, scr, lane);
			const unsigned z = __ballot_sync(0xffffffffu, lane < nbk && frag::bad_pivot(v));
			if (z && lane == 0 && *bad == 0) *bad = c0 + __ffs(z);
			v = fabs(v);
#pragma unroll
			for (int h = 0; h < 2; h++) {
				const int j = 2 * q + h;
				Lt[r * 17 + j] = j <= r ? F[0][h] : 0.0;
				Lt[r * 17 + 8 + j] = 0.0;
				Lt[(8 + r) * 17 + j] = F[1][h];
				Lt[(8 + r) * 17 + 8 + j] = j <= r ? F[2][h] : 0.0;
			}
			if (lane < nbk) d.d[c0 + lane] = v;
			if (lane < 16) Lt[lane * 17 + 16] = v;
		}
		// ---- panel update: FR fragment rows at a time, claimed by the warps ----
		for (;;) {
			int f = 0;
			if (lane == 0) f = atomicAdd(&next, FR);
			f = __shfl_sync(0xffffffffu, f, 0);
			if (f >= R) break;
			double cv[FR][2][2], acc[FR][2][2];
			const double *ap[FR];
#pragma unroll
			for (int u = 0; u < FR; u++) {
				const int row = c0 + 8 * (f + u) + r;
				ap[u] = rowp(row);
#pragma unroll
				for (int fc = 0; fc < 2; fc++)
#pragma unroll
					for (int h = 0; h < 2; h++)
						cv[u][fc][h] = row < n ? *c.addr(row, c0 + 8 * fc + 2 * q + h) : 0.0;
			}
			ll_update<FR, UNR>(acc, ap, b0, b1, c0);
#pragma unroll
			for (int u = 0; u < FR; u++) {
				if (f + u >= R) break;
				double *pr = pan + (8 * (f + u) + r) * LL_PSTR + 2 * q;
#pragma unroll
				for (int fc = 0; fc < 2; fc++)
#pragma unroll
					for (int h = 0; h < 2; h++) pr[8 * fc + h] = cv[u][fc][h] - acc[u][fc][h];
			}
		}
		__syncthreads();
		// ---- rows below the diagonal block (and the right-hand side): x = a L_KK^{-T} ----
		const int m1 = m > 16 ? m : 16;  // the right-hand side's place behind the rows
		for (int i = 16 + tid; i < m1 + (y ? 1 : 0); i += NT) {
			const bool rhs = i == m1;
			double x[16];
#pragma unroll
			for (int cc = 0; cc < 16; cc++) x[cc] = rhs ? (cc < nbk ? y[c0 + cc] : 0.0) : pan[i * LL_PSTR + cc];
#pragma unroll
			for (int cc = 0; cc < 16; cc++) {
				double s = x[cc];
#pragma unroll
				for (int l = 0; l < cc; l++) s = fma(-x[l], Lt[cc * 17 + l], s);
				x[cc] = s * Lt[cc * 17 + 16];
			}
#pragma unroll
			for (int cc = 0; cc < 16; cc++) {
				if (!rhs)
					pan[i * LL_PSTR + cc] = x[cc];
				else if (cc < nbk)
					y[c0 + cc] = x[cc];
			}
		}
		__syncthreads();
		if (y) {
			for (int i = 16 + tid; i < m; i += NT) {
				double s = y[c0 + i];
#pragma unroll
				for (int l = 0; l < 16; l++) s = fma(-pan[i * LL_PSTR + l], y[c0 + l], s);
				y[c0 + i] = s;
			}
		}
		if (tid == 0) next = 2;
		// ---- store the panel: 4-row x 16-column runs of the panel layout ----
		for (int e = tid; e < 16 * ((m + 3) & ~3); e += NT) {
			const int p = e >> 6, w = e & 63;
			const int i = 4 * p + (w & 3), j = w >> 2;  // panel-relative row, column
			const int gi = c0 + i, gj = c0 + j;
			if (gi < n && gj < n && (i >= 16 || j <= i))
				*d.addr(gi, gj) = pan[i * LL_PSTR + j];
		}
		__syncthreads();
	}
}

// y := L^{-T} y for the factor in d (global memory, row offset 0), y in shared
// memory (n doubles), by 16-row blocks from the last.  Every load of L is
// issued ahead of the chain that waits for it: the diagonal block (column l in
// lane l of warp 0) one block early, the 16 rows of a thread's first column
// before the block's substitution.  With the loads inside the 16-step
// substitution each step waited for L2.
template <int NT>
__device__ void trsv_ll_bwd(const PMat<double> &d, int n, double *y) {
	const int tid = threadIdx.x, lane = tid & 31;
	const bool al = ((uintptr_t)d.p & 15) == 0;  // a caller's workspace may be aligned to 8 bytes only
	// rows c0 .. c0+15 of column j, zeros beyond row n
	auto col16 = [&](int c0, int j, double(&v)[16]) {
#pragma unroll
		for (int p = 0; p < 4; p++) {
			const int i = c0 + 4 * p;
			double2 a = make_double2(0.0, 0.0), b = a;
			if (i < n) {
				const double *s = d.addr(i, j);
				if (al) {
					a = *(const double2 *)s;
					b = *(const double2 *)(s + 2);
				} else {
					a = make_double2(s[0], s[1]);
					b = make_double2(s[2], s[3]);
				}
			}
			v[4 * p] = a.x;
			v[4 * p + 1] = i + 1 < n ? a.y : 0.0;
			v[4 * p + 2] = i + 2 < n ? b.x : 0.0;
			v[4 * p + 3] = i + 3 < n ? b.y : 0.0;
		}
	};
	const int cl = (n - 1) & ~15;
	double dg[16], rcp = 0.0;
	auto diag = [&](int c0) {
		const bool in = lane < 16 && c0 + lane < n;
		col16(c0, in ? c0 + lane : c0, dg);
		rcp = in ? d.d[c0 + lane] : 0.0;
	};
	if (tid < 32) diag(cl);
	for (int c0 = cl; c0 >= 0; c0 -= 16) {
		const int nbk = n - c0 < 16 ? n - c0 : 16;
		double a[16];
		const bool has = tid < c0;
		if (has) col16(c0, tid, a);
		if (tid < 32) {
			double v = (lane < nbk) ? y[c0 + lane] : 0.0;
#pragma unroll
			for (int k = 15; k >= 0; k--) {
				const double x = v * rcp;
				const double xk = __shfl_sync(0xffffffffu, x, k);
				if (lane == k) v = x;
				if (lane < k) v = fma(-dg[k], xk, v);
			}
			if (lane < nbk) y[c0 + lane] = v;
			if (c0) diag(c0 - 16);
		}
		__syncthreads();
		for (int j = tid; j < c0; j += NT) {
			if (j != tid) col16(c0, j, a);
			double s = y[j];
#pragma unroll
			for (int k = 0; k < 16; k++) s = fma(-a[k], k < nbk ? y[c0 + k] : 0.0, s);
			y[j] = s;
		}
		__syncthreads();
	}
}
