// FP64 LU with row pivoting (getrf_rp, blasfeo_hp_pm/d_lapack_lib4.c:2396; and
// getrf_np, :2078) of matrices with up to 512 rows, one CTA per matrix, blocked
// by 16-column panels whose rows live in registers.
//
// Per panel (columns c0..c0+15):
//   a. thread t reads row c0 + t (+ NT, ..): 16 entries per row in registers,
//      with the row's position;
//   b. per column: the largest |entry| (first position on a tie,
//      kernel/generic/kernel_dgetrf_pivot_lib4.c:84-165) by three redux per
//      warp, the warp's candidate row to shared memory, ONE barrier, the
//      winner among the warps by three more; rows are not moved, the two
//      positions are exchanged (without pivoting row j goes to shared memory, no
//      search); every thread scales and updates its rows;
//   c. the rows go to their positions in D and in shared memory; the positions
//      are the panel's permutation;
//   per chunk of at most CH columns right of the panel:
//   d. the 16 pivot rows and the 16 rows they displace are read once, U12 =
//      L11^{-1} A12 (a thread per column);
//   e. A22 -= L21 U12 as 32 x 32 tensor core tiles per warp; a displaced row is
//      taken from the copy made in d, so the swaps cost no pass of their own;
// the columns left of each panel are permuted once at the end, a 16-column
// block at a time through shared memory, with the composition of the later
// panels' permutations.  The first panel's steps read C, the later ones D.
// Arithmetic and order per element are those of k_getrf_blk (lapack.cu): one
// FMA per earlier column of the panel, then rank-16 DMMA updates.
//
// Bound: the column chain (search, barrier, reciprocal, update: about 500
// cycles against 2,500 with the panel in shared memory, two barriers and a
// butterfly of 64-bit shuffles per column), then the trailing update's traffic
// to L2.  Size classes: a variable-size launch starts its CTAs largest first
// (grid = classes x batch, the CTAs of the other classes leave at once): a
// 384 x 384 matrix that starts last would otherwise run alone.  1,024 matrices,
// sizes log-uniform in 4..384: 2.39 -> 0.72 ms; uniform n = 16 x 20,000 0.38 -> 0.11,
// n = 64 x 20,000 5.39 -> 1.86, n = 256 x 2,013 7.51 -> 3.82, n = 384 x 825
// 10.7 -> 5.2 ms.  That uneven batch (512 threads, one CTA per SM; ncu): a warp issues
// every 11.6 cycles, 4.0 of them at barriers; issue slots 34%, tensor pipe 9%, DRAM
// 6%.  The 128 registers per thread spill (224 bytes of stores, 172 without
// pivoting).
#include "common.cuh"
#include "kernels.cuh"

namespace {

constexpr int PLD = 20;   // row stride of the panel in shared memory (4 mod 16: fragment reads without conflicts)
constexpr unsigned FULL = 0xffffffffu;

__device__ __forceinline__ void lu_dmma(double &d0, double &d1, double a, double b) {
	asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
	    : "+d"(d0), "+d"(d1)
	    : "d"(a), "d"(b));
}

// shared memory of a launch
struct LuPlan {
	int ch;                                   // columns per chunk (a multiple of 32)
	size_t u, t, rows, map, s, rec, total;    // byte offsets (the panel is at 0)
};
__host__ __device__ inline LuPlan lu_plan(int nt, int max_m, int max_n) {
	LuPlan p;
	p.ch = max_n < 128 ? (max_n + 31) / 32 * 32 : 128;
	const int np = ((max_m < max_n ? max_m : max_n) + 15) / 16;
	p.u = (size_t)max_m * PLD * 8;
	p.t = p.u + (size_t)16 * (p.ch + 4) * 8;
	p.rows = p.t + (size_t)16 * (p.ch + 4) * 8;
	p.map = p.rows + (size_t)2 * (nt / 32) * 16 * 8;
	p.s = p.map + (size_t)(max_m + 1) / 2 * 2 * sizeof(short);
	p.rec = p.s + (size_t)(max_m + 1) / 2 * 2 * sizeof(short);
	p.total = (p.rec + (size_t)np * 66 * sizeof(short) + 15) / 16 * 16;
	return p;
}

// sort key of an entry: larger |a| first, NaN last (never chosen before a number)
__device__ __forceinline__ unsigned long long lu_key(double a) {
	const unsigned long long b = (unsigned long long)__double_as_longlong(a) & 0x7fffffffffffffffULL;
	return b > 0x7ff0000000000000ULL ? 0ULL : b + 1;
}

// the warp's lane with the largest key, the smallest pos among equals; pos < 0x7fffffff on at least one lane
__device__ __forceinline__ void warp_best(unsigned long long &key, int &pos, bool &win) {
	const unsigned kh = (unsigned)(key >> 32), mh = __reduce_max_sync(FULL, kh);
	const unsigned kl = kh == mh ? (unsigned)key : 0u, ml = __reduce_max_sync(FULL, kl);
	const bool c = kh == mh && (unsigned)key == ml;
	const int mp = __reduce_min_sync(FULL, c ? pos : 0x7fffffff);
	win = c && pos == mp;
	key = (unsigned long long)mh << 32 | ml;
	pos = mp;
}

template <int NT, int RPT, int MINB, bool PIV>
__global__ void __launch_bounds__(NT, MINB)
    k_getrf_reg(int batch, SizeArg sz, MatArg<double> C, MatArg<double> D, int *ipiv, long long ipiv_stride, int *info,
                int max_m, int max_n, int classes) {
	constexpr int NW = NT / 32;
	extern __shared__ __align__(16) unsigned char lu_sm[];
	__shared__ unsigned long long s_key[2][NW];
	__shared__ int s_pos[2][NW], s_bad, s_nmv;
	__shared__ int s_src[16];
	const int b = blockIdx.x % batch;
	const int m = sz.M(b), n = sz.N(b);
	if (m <= 0 || n <= 0 || m > max_m || n > max_n) return;
	if (classes > 1) {
		// class 0: the largest, by quarters of the largest matrix
		const int big = m > n ? m : n, top = max_m > max_n ? max_m : max_n;
		if (classes - 1 - (big * classes - 1) / top != (int)(blockIdx.x / batch)) return;
	}
	const LuPlan pl = lu_plan(NT, max_m, max_n);
	double *P = (double *)lu_sm;                       // panel, row r at P + PLD r
	double *Us = (double *)(lu_sm + pl.u), *Ts = (double *)(lu_sm + pl.t);
	double *crow = (double *)(lu_sm + pl.rows);        // candidate rows [2][NW][16]
	short *dmap = (short *)(lu_sm + pl.map);           // displaced rows: index into Ts, else -1
	short *S = (short *)(lu_sm + pl.s);
	short *rec = (short *)(lu_sm + pl.rec);            // per panel: count, then (row, from) pairs
	const int ldu = pl.ch + 4;
	const PMat<double> c = C.get(b), d = D.get(b);
	int *piv = PIV ? ipiv + ipiv_stride * b : nullptr;
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int g = lane >> 2, q = lane & 3;
	for (int r = tid; r < m; r += NT) dmap[r] = -1;
	if (tid == 0) s_bad = 0;
	const int mn = m < n ? m : n;
	for (int c0 = 0; c0 < mn; c0 += 16) {
		const int w = mn - c0 < 16 ? mn - c0 : 16;
		const int pr = m - c0;
		const PMat<double> x = c0 ? d : c;             // where the matrix is now
		// a. rows into registers
		double a[RPT][16];
		int pos[RPT];
#pragma unroll
		for (int u = 0; u < RPT; u++) {
			const int r = tid + u * NT;
			pos[u] = r < pr ? r : 0x7fffffff;
#pragma unroll
			for (int j = 0; j < 16; j++) a[u][j] = (r < pr && j < w) ? x.at(c0 + r, c0 + j) : 0.0;
		}
		if (tid == 0) s_nmv = 0;
		// b. factor
#pragma unroll
		for (int j = 0; j < 16; j++) {
			if (j < w) {
				const double *ur;
				int ip = j;
				if (PIV) {
					// the thread's candidate: among its rows at positions >= j
					unsigned long long key = 0;
					int best = 0x7fffffff;
					double row[16];
#pragma unroll
					for (int l = j; l < 16; l++) row[l] = a[0][l];
#pragma unroll
					for (int u = 0; u < RPT; u++) {
						const bool act = pos[u] != 0x7fffffff && pos[u] >= j;
						const unsigned long long k = act ? lu_key(a[u][j]) : 0ULL;
						if (act && (k > key || best == 0x7fffffff || (k == key && pos[u] < best))) {
							key = k;
							best = pos[u];
							if (u > 0) {
#pragma unroll
								for (int l = j; l < 16; l++) row[l] = a[u][l];
							}
						}
					}
					bool win;
					warp_best(key, best, win);
					double *cr = crow + (size_t)((j & 1) * NW + warp) * 16;
					if (win && best != 0x7fffffff) {
#pragma unroll
						for (int l = j; l < 16; l++) cr[l] = row[l];
					}
					if (lane == 0) {
						s_key[j & 1][warp] = key;
						s_pos[j & 1][warp] = best;
					}
					__syncthreads();
					key = lane < NW ? s_key[j & 1][lane] : 0ULL;
					best = lane < NW ? s_pos[j & 1][lane] : 0x7fffffff;
					warp_best(key, best, win);
					ip = best;
					ur = crow + (size_t)((j & 1) * NW + __ffs(__ballot_sync(FULL, win)) - 1) * 16;
				} else {
					// row j is thread j's first
					double *cr = crow + (size_t)(j & 1) * NW * 16;
					if (tid == j) {
#pragma unroll
						for (int l = j; l < 16; l++) cr[l] = a[0][l];
					}
					__syncthreads();
					ur = cr;
				}
				const double pv = ur[j];
				// getrf_rp: a zero pivot gives inverse 0; getrf_np divides as the
				// reference does (blasfeo_ref/x_lapack_ref.c, REF_GETRF_NOPIVOT)
				const double inv = PIV ? (pv != 0.0 ? 1.0 / pv : 0.0) : 1.0 / pv;
				if (tid == 0) {
					if (PIV) piv[c0 + j] = c0 + ip;
					d.d[c0 + j] = inv;
					if (pv == 0.0 && s_bad == 0) s_bad = c0 + j + 1;
				}
				double uv[16];
#pragma unroll
				for (int l = j + 1; l < 16; l++) uv[l] = ur[l];
#pragma unroll
				for (int u = 0; u < RPT; u++) {
					const int p0 = pos[u];
					if (p0 == ip)
						pos[u] = j;
					else if (p0 == j)
						pos[u] = ip;
					if (pos[u] > j && pos[u] != 0x7fffffff) {
						const double lj = a[u][j] * inv;
						a[u][j] = lj;
#pragma unroll
						for (int l = j + 1; l < 16; l++) a[u][l] = fma(-lj, uv[l], a[u][l]);
					}
				}
			}
		}
		// c. rows to their positions
		short *rc = rec + (size_t)(c0 >> 4) * 66;
#pragma unroll
		for (int u = 0; u < RPT; u++) {
			const int r0 = tid + u * NT, p = pos[u];
			if (r0 < pr) {
#pragma unroll
				for (int j = 0; j < 16; j += 2) *(double2 *)(P + (size_t)p * PLD + j) = make_double2(a[u][j], a[u][j + 1]);
#pragma unroll
				for (int j = 0; j < 16; j++)
					if (j < w) d.at(c0 + p, c0 + j) = a[u][j];
				if (p < w) s_src[p] = r0;
				if (p != r0) {
					const int k = atomicAdd(&s_nmv, 1);
					rc[2 + 2 * k] = (short)(c0 + p);
					rc[3 + 2 * k] = (short)(c0 + r0);
					if (p >= w) dmap[c0 + p] = (short)r0;  // r0 < w: displaced from the panel's rows
				}
			}
		}
		__syncthreads();
		if (tid == 0) rc[0] = (short)s_nmv;
		// columns right of the panel, a chunk at a time
		for (int l0 = c0 + w; l0 < n; l0 += pl.ch) {
			const int nc = n - l0 < pl.ch ? n - l0 : pl.ch;
			// d. U12 (threads below) and the displaced rows' old contents
			for (int e = tid; e < 2 * nc; e += NT) {
				const int l = e < nc ? e : e - nc;
				double uu[16];
				if (e < nc) {
#pragma unroll
					for (int k = 0; k < 16; k++) uu[k] = k < w ? x.at(c0 + s_src[k < w ? k : 0], l0 + l) : 0.0;
#pragma unroll
					for (int k = 1; k < 16; k++)
#pragma unroll
						for (int kk = 0; kk < k; kk++) uu[k] = fma(-P[(size_t)k * PLD + kk], uu[kk], uu[k]);
#pragma unroll
					for (int k = 0; k < 16; k++) Us[k * ldu + l] = k < w ? uu[k] : 0.0;
				} else {
#pragma unroll
					for (int k = 0; k < 16; k++) uu[k] = k < w ? x.at(c0 + k, l0 + l) : 0.0;
#pragma unroll
					for (int k = 0; k < 16; k++) Ts[k * ldu + l] = uu[k];
				}
			}
			__syncthreads();
			// U12 to D (after every read of the rows it overwrites), and
			// e. A22 -= L21 U12
			for (int e = tid; e < 16 * nc; e += NT) {
				const int k = e & 15, l = e >> 4;
				if (k < w) d.at(c0 + k, l0 + l) = Us[k * ldu + l];
			}
			const int rows = pr - w;
			const int nct = (nc + 31) >> 5, ntile = (rows > 0 ? (rows + 31) >> 5 : 0) * nct;
			for (int t = warp; t < ntile; t += NW) {
				const int r0 = w + 32 * (t / nct), lc = 32 * (t % nct);
				double acc[4][4][2];
#pragma unroll
				for (int rb = 0; rb < 4; rb++) {
					const int row = r0 + 8 * rb + g;
					const int dm = row < pr ? dmap[c0 + row] : -1;
#pragma unroll
					for (int cb = 0; cb < 4; cb++)
#pragma unroll
						for (int h = 0; h < 2; h++) {
							const int col = lc + 8 * cb + 2 * q + h;
							double v = 0.0;
							if (row < pr && col < nc) v = dm >= 0 ? Ts[dm * ldu + col] : x.at(c0 + row, l0 + col);
							acc[rb][cb][h] = v;
						}
				}
#pragma unroll
				for (int ks = 0; ks < 4; ks++) {
					double av[4], bv[4];
#pragma unroll
					for (int rb = 0; rb < 4; rb++) {
						const int row = r0 + 8 * rb + g;
						av[rb] = row < pr ? -P[(size_t)row * PLD + 4 * ks + q] : 0.0;
					}
#pragma unroll
					for (int cb = 0; cb < 4; cb++) {
						const int col = lc + 8 * cb + g;
						bv[cb] = col < nc ? Us[(4 * ks + q) * ldu + col] : 0.0;
					}
#pragma unroll
					for (int rb = 0; rb < 4; rb++)
#pragma unroll
						for (int cb = 0; cb < 4; cb++) lu_dmma(acc[rb][cb][0], acc[rb][cb][1], av[rb], bv[cb]);
				}
#pragma unroll
				for (int rb = 0; rb < 4; rb++) {
					const int row = r0 + 8 * rb + g;
#pragma unroll
					for (int cb = 0; cb < 4; cb++)
#pragma unroll
						for (int h = 0; h < 2; h++) {
							const int col = lc + 8 * cb + 2 * q + h;
							if (row < pr && col < nc) d.at(c0 + row, l0 + col) = acc[rb][cb][h];
						}
				}
			}
			__syncthreads();
		}
		// displaced rows of this panel no longer apply
#pragma unroll
		for (int u = 0; u < RPT; u++)
			if (pos[u] != 0x7fffffff && pos[u] >= w) dmap[c0 + pos[u]] = -1;
		__syncthreads();
	}
	// columns left of the panels: block K takes the row swaps of the panels
	// after it, S[r] = the row whose content ends at r
	const int np = (mn + 15) >> 4;
	if (PIV && np > 1) {
		for (int r = tid; r < m; r += NT) {
			S[r] = (short)r;
			dmap[r] = (short)r;
		}
		__syncthreads();
		for (int K = np - 2; K >= 0; K--) {
			const short *rc = rec + (size_t)(K + 1) * 66;
			const int nm = rc[0], c1 = 16 * (K + 1);
			for (int e = tid; e < nm; e += NT) dmap[rc[2 + 2 * e]] = rc[3 + 2 * e];
			// stage rows c1.. of the block meanwhile
			for (int r = c1 + tid; r < m; r += NT) {
				double v[16];
#pragma unroll
				for (int j = 0; j < 16; j++) v[j] = d.at(r, 16 * K + j);
#pragma unroll
				for (int j = 0; j < 16; j += 2)
					*(double2 *)(P + (size_t)(r - c1) * PLD + j) = make_double2(v[j], v[j + 1]);
			}
			__syncthreads();
			for (int r = c1 + tid; r < m; r += NT) {
				const short s = dmap[S[r]];
				S[r] = s;
				if (s != r) {
#pragma unroll
					for (int j = 0; j < 16; j++) d.at(r, 16 * K + j) = P[(size_t)(s - c1) * PLD + j];
				}
			}
			__syncthreads();
			for (int e = tid; e < nm; e += NT) dmap[rc[2 + 2 * e]] = rc[2 + 2 * e];
			__syncthreads();
		}
	}
	if (info && tid == 0) info[b] = s_bad;
}

template <int NT, int RPT, int MINB>
int launch(int batch, SizeArg sz, MatArg<double> C, MatArg<double> D, int *ipiv, long long stride, int *info,
           cudaStream_t s, int max_m, int max_n, bool piv, int classes) {
	auto kern = piv ? k_getrf_reg<NT, RPT, MINB, true> : k_getrf_reg<NT, RPT, MINB, false>;
	const size_t smem = lu_plan(NT, max_m, max_n).total;
	bf::smem_optin(kern, smem);
	kern<<<(unsigned)(batch * (long long)classes), NT, smem, s>>>(batch, sz, C, D, ipiv, stride, info, max_m, max_n,
	                                                              classes);
	return bf::check_launch();
}

}  // namespace

namespace bf {

// rows beyond the register panels, or shared memory (very wide matrices)
bool dgetrf_reg_fits(int max_m, int max_n) {
	return max_m <= 512 && lu_plan(512, max_m, max_n).total + 4096 <= max_smem_optin();
}

int dgetrf_reg_launch(int batch, SizeArg sz, MatArg<double> C, MatArg<double> D, int *ipiv, long long stride, int *info,
                      cudaStream_t s, int max_m, int max_n, bool piv, int nt) {
	// size classes only where sizes differ, matrices are long enough to matter
	// and the larger grid stays in range
	const int mx = max_m > max_n ? max_m : max_n;
	const int classes = (sz.pm && mx > 64 && batch <= (1 << 28)) ? 4 : 1;
	const int need = (max_m + nt - 1) / nt;  // rows per thread
	switch (nt) {
	case 32:
		if (need <= 1) return launch<32, 1, 16>(batch, sz, C, D, ipiv, stride, info, s, max_m, max_n, piv, classes);
		nt = 64;
		// fall through
	case 64:
		if (max_m <= 64) return launch<64, 1, 8>(batch, sz, C, D, ipiv, stride, info, s, max_m, max_n, piv, classes);
		nt = 128;
		// fall through
	case 128:
		if (max_m <= 128) return launch<128, 1, 4>(batch, sz, C, D, ipiv, stride, info, s, max_m, max_n, piv, classes);
		if (max_m <= 256) return launch<128, 2, 4>(batch, sz, C, D, ipiv, stride, info, s, max_m, max_n, piv, classes);
		// fall through
	case 256:
		if (max_m <= 256) return launch<256, 1, 2>(batch, sz, C, D, ipiv, stride, info, s, max_m, max_n, piv, classes);
		return launch<256, 2, 2>(batch, sz, C, D, ipiv, stride, info, s, max_m, max_n, piv, classes);
	default: return launch<512, 1, 1>(batch, sz, C, D, ipiv, stride, info, s, max_m, max_n, piv, classes);
	}
}

}  // namespace bf
