// FP64 Householder QR (geqrf, blasfeo_hp_pm/d_lapack_lib4.c:3444) of matrices
// with up to 512 rows, one CTA per matrix, blocked by 16-column panels whose
// columns live in registers.
//
// Per panel (columns c0..c0+15):
//   a. SL = NT / 16 lanes per column hold it in registers (rows s, s + SL, ..);
//   b. column by column: its lanes form the reflector (dlarfg signs,
//      kernel/generic/kernel_dgeqrf_4_lib4.c:80-96) and pass v through shared
//      memory, ONE barrier, the later columns' lanes apply it.  Sums over the
//      lanes of a column are a tensor core step against ones and another one or
//      one or two shuffles (66 cycles; the butterfly of 64-bit shuffles takes 190
//      and occupies the SM's shuffle unit);
//   c. panel to D, V (unit lower trapezoid) to shared memory;
//   d. G = V^T V on the tensor cores, T^T from it column by column:
//      x_k = tau_k (e_k - sum_{q<k} G_qk x_q);
//   e. the columns right of the panel, 32 at a time, C -= V T^T (V^T C): each
//      warp loads its rows of C once as C^T accumulators.  Lane (g, q) =
//      (lane / 4, lane % 4) then holds rows 2q, 2q + 1 of column g, which is the
//      B operand of V^T C (rows in the order 0, 2, 4, 6 | 1, 3, 5, 7) and the
//      accumulator of C^T -= (T^T V^T C)^T V^T, so C is read and written once.
// The first panel's steps read C, the later ones D.
//
// Bound at 384 x 192 (512 threads, clock64): the column chain 40% (2,300 cycles a
// column: two sums, square root, reciprocals, v through shared memory to 16
// warps, a barrier), the chunks of 32 columns 55% (11,000 cycles each, 5,800 of
// them tensor steps at the FP64 peak, the rest waits for C and three barriers).
// Size classes as in getrf_reg.cu.  1,024 matrices 2n x n, n log-uniform in
// 4..192: 1.27 -> 0.62 ms; uniform 16 x 8 x 20,000 198 -> 151 us, 64 x 32 x
// 20,000 3.38 -> 1.35 ms, 128 x 64 x 20,000 13.0 -> 5.3, 384 x 192 x 3,791 19.8 ->
// 15.7 ms.  That uneven batch (512 threads, one CTA per SM; ncu): a warp issues every
// 14.4 cycles, 5.9 of them at barriers; issue slots 28%, tensor pipe 15%, DRAM 2%.
// The 128 registers per thread spill (bytes of stores: 284 for up to 384 rows, 560
// beyond, 152 at 256, 188 with 256 threads).  Matrices much wider than tall go to the
// blocked kernel (geqrf_wide, lapack.cu).
#include "common.cuh"
#include "kernels.cuh"

namespace {

constexpr int PLD = 20;   // row stride of V
constexpr int TLD = 17;

__device__ __forceinline__ void qr_dmma(double &d0, double &d1, double a, double b) {
	asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
	    : "+d"(d0), "+d"(d1)
	    : "d"(a), "d"(b));
}

// sum of v over the SL lanes of the lane's segment (SL = 4, 8, 16 or 32), in all of them
template <int SL>
__device__ __forceinline__ double seg_sum(double v, int g, int q) {
	double s0 = 0.0, s1 = 0.0;
	if constexpr (SL == 4) {
		qr_dmma(s0, s1, v, 1.0);  // lanes g: the sum over their four lanes
		return s0;
	}
	qr_dmma(s0, s1, 1.0, v);  // lanes q: sums over the four lanes of g = 2q and g = 2q + 1
	s0 += s1;
	if constexpr (SL == 32) {
		double r0 = 0.0, r1 = 0.0;
		qr_dmma(r0, r1, 1.0, s0);
		return r0;
	} else if constexpr (SL == 16) {
		const int src = (g << 2) | ((g >> 2) << 1);
		return __shfl_sync(0xffffffffu, s0, src) + __shfl_sync(0xffffffffu, s0, src + 1);
	} else {
		return __shfl_sync(0xffffffffu, s0, (g << 2) | (g >> 1));
	}
}

struct QrPlan {
	size_t part, vb, wraw, ws, tt, gm, total;  // byte offsets (V at 0)
};
// row stride of 16 x cw blocks (at least 16 wide for V^T V)
__host__ __device__ constexpr int qr_wld(int cw) { return cw + 4; }
__host__ __device__ inline QrPlan qr_plan(int nt, int cw, int max_m) {
	QrPlan p;
	const int WLD = qr_wld(cw);
	const int rows = (max_m + 7) / 8 * 8;
	p.part = (size_t)rows * PLD * 8;
	p.vb = p.part + (size_t)(nt / 32) * 16 * WLD * 8;
	p.wraw = p.vb + (size_t)2 * rows * 8;
	p.ws = p.wraw + (size_t)16 * WLD * 8;
	p.tt = p.ws + (size_t)16 * WLD * 8;
	p.gm = p.tt + (size_t)16 * TLD * 8;
	p.total = p.gm + (size_t)16 * TLD * 8;
	return p;
}

template <int NT, int RPT, int CW, int MINB>
__global__ void __launch_bounds__(NT, MINB)
    k_geqrf_reg(int batch, SizeArg sz, MatArg<double> C, MatArg<double> D, int max_m, int max_n, int classes) {
	constexpr int SL = NT / 16, NW = NT / 32, TB = RPT / 4, CB = CW / 8, WLD = qr_wld(CW);
	extern __shared__ __align__(16) unsigned char qr_sm[];
	__shared__ double s_tau[16], s_t[2];
	const int b = blockIdx.x % batch;
	const int m = sz.M(b), n = sz.N(b);
	if (m <= 0 || n <= 0 || m > max_m || n > max_n) return;
	if (classes > 1) {
		// class 0: the largest, by quarters of the largest matrix
		const int big = m > n ? m : n, top = max_m > max_n ? max_m : max_n;
		if (classes - 1 - (big * classes - 1) / top != (int)(blockIdx.x / batch)) return;
	}
	const QrPlan pl = qr_plan(NT, CW, max_m);
	double *V = (double *)qr_sm;
	double *part = (double *)(qr_sm + pl.part), *vb = (double *)(qr_sm + pl.vb);
	double *Wr = (double *)(qr_sm + pl.wraw), *Ws = (double *)(qr_sm + pl.ws);
	double *Tt = (double *)(qr_sm + pl.tt), *Gm = (double *)(qr_sm + pl.gm);
	const int vld = (max_m + 7) / 8 * 8;
	const PMat<double> c = C.get(b), d = D.get(b);
	double *tau = d.d + d.ri;
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int g = lane >> 2, q = lane & 3;
	const int col = tid / SL, s = tid % SL;  // panel column and first row of this thread
	const int kmax = m < n ? m : n;
	for (int c0 = 0; c0 < kmax; c0 += 16) {
		const int w = kmax - c0 < 16 ? kmax - c0 : 16;
		const int pr = m - c0;
		const PMat<double> x = c0 ? d : c;
		// a. the panel's columns into registers
		double a[RPT];
#pragma unroll
		for (int i = 0; i < RPT; i++) {
			const int r = s + SL * i;
			a[i] = (r < pr && col < w) ? x.at(c0 + r, c0 + col) : 0.0;
		}
		// b. reflectors
		for (int j = 0; j < w; j++) {
			double *v = vb + (j & 1) * vld;
			if (warp == j * SL / 32) {  // the warp that holds column j
				double p0 = 0.0, p1 = 0.0, al = 0.0;
#pragma unroll
				for (int i = 0; i < RPT; i++) {
					if (SL * i < pr) {
						const int r = s + SL * i;
						const double y = (SL * i < 16 && r <= j) ? 0.0 : a[i];
						if (SL * i < 16 && r == j) al = a[i];
						if (i & 1)
							p1 = fma(y, y, p1);
						else
							p0 = fma(y, y, p0);
					}
				}
				const double sq = seg_sum<SL>(p0 + p1, g, q);
				const double alpha = seg_sum<SL>(al, g, q);
				double t = 0.0, sc = 1.0, beta = alpha;
				// (no rows below: no reflector, whatever a NaN or an infinity has left in
				// the registers of the rows past the last)
				if (sq != 0.0 && j + 1 < pr) {
					beta = sqrt(fma(alpha, alpha, sq));
					if (alpha > 0.0) beta = -beta;
					t = (beta - alpha) / beta;
					sc = 1.0 / (alpha - beta);
				}
				if (col == j) {
#pragma unroll
					for (int i = 0; i < RPT; i++) {
						const int r = s + SL * i;
						if (r < pr) {
							if (SL * i >= 16 || r > j) {
								a[i] *= sc;
								v[r] = a[i];
							} else {
								v[r] = r == j ? 1.0 : 0.0;
								if (r == j) a[i] = beta;
							}
						}
					}
					if (s == 0) {
						s_t[j & 1] = t;
						s_tau[j] = t;
						tau[c0 + j] = t;
					}
				}
			}
			__syncthreads();
			if (warp >= (j + 1) * SL / 32) {  // warps with a later column
				const double t = s_t[j & 1];
				double y[RPT], p0 = 0.0, p1 = 0.0;
#pragma unroll
				for (int i = 0; i < RPT; i++) {
					if (SL * i < pr) {
						const int r = s + SL * i;
						y[i] = r < pr ? v[r] : 0.0;
						if (i & 1)
							p1 = fma(y[i], a[i], p1);
						else
							p0 = fma(y[i], a[i], p0);
					}
				}
				const double z = -t * seg_sum<SL>(p0 + p1, g, q);
				if (col > j && col < w) {
#pragma unroll
					for (int i = 0; i < RPT; i++)
						if (SL * i < pr && (SL * i >= 16 || s + SL * i >= j)) a[i] = fma(z, y[i], a[i]);
				}
			}
		}
		// c. panel to D, V to shared memory (zeros above the diagonal and past the
		// last row, ones on it)
		const int pr8 = (pr + 7) & ~7;
#pragma unroll
		for (int i = 0; i < RPT; i++) {
			const int r = s + SL * i;
			if (r < pr8) V[(size_t)r * PLD + col] = (r >= pr || r < col || col >= w) ? 0.0 : (r == col ? 1.0 : a[i]);
			if (r < pr && col < w) d.at(c0 + r, c0 + col) = a[i];
		}
		if (tid < 16 && tid >= w) s_tau[tid] = 0.0;
		const int l00 = c0 + w;
		if (l00 >= n) break;
		__syncthreads();
		// d. G = V^T V, blocks (0,0), (0,1), (1,1): partial sums of each warp's rows
		{
			double e[3][2] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
#pragma unroll
			for (int t = 0; t < TB; t++) {
				const int r0 = 8 * (warp + NW * t);
				if (r0 < pr) {
#pragma unroll
					for (int h = 0; h < 2; h++) {
						const double *vr = V + (size_t)(r0 + 2 * q + h) * PLD + g;
						const double v0 = vr[0], v1 = vr[8];
						qr_dmma(e[0][0], e[0][1], v0, v0);
						qr_dmma(e[1][0], e[1][1], v0, v1);
						qr_dmma(e[2][0], e[2][1], v1, v1);
					}
				}
			}
			double *pw = part + (size_t)warp * 16 * WLD;
			*(double2 *)(pw + g * WLD + 2 * q) = make_double2(e[0][0], e[0][1]);
			*(double2 *)(pw + g * WLD + 8 + 2 * q) = make_double2(e[1][0], e[1][1]);
			*(double2 *)(pw + (8 + g) * WLD + 8 + 2 * q) = make_double2(e[2][0], e[2][1]);
		}
		__syncthreads();
		for (int e = tid; e < 256; e += NT) {
			const int i = e >> 4, k = e & 15;
			if (i < k) {
				double z = 0.0;
#pragma unroll
				for (int u = 0; u < NW; u++) z += part[(size_t)u * 16 * WLD + i * WLD + k];
				Gm[i * TLD + k] = z;
			}
		}
		__syncthreads();
		if (tid < 16) {
			// T^T, column tid
			double t[16];
#pragma unroll
			for (int k = 0; k < 16; k++) t[k] = k == tid ? 1.0 : 0.0;
#pragma unroll
			for (int k = 0; k < 16; k++) {
				t[k] *= s_tau[k];
#pragma unroll
				for (int i = k + 1; i < 16; i++) t[i] = fma(-Gm[k * TLD + i], t[k], t[i]);
			}
#pragma unroll
			for (int k = 0; k < 16; k++) Tt[k * TLD + tid] = t[k];
		}
		// (the first chunk's barriers order Tt before its use)
		// e. columns right of the panel
		const bool vec = ((x.ri | d.ri) & 1) == 0 && (((uintptr_t)x.p | (uintptr_t)d.p) & 15) == 0;
		for (int l0 = l00; l0 < n; l0 += CW) {
			const int nc = n - l0 < CW ? n - l0 : CW;
			double f[TB][CB][2], wv[2][CB][2];
#pragma unroll
			for (int u = 0; u < 2; u++)
#pragma unroll
				for (int cb = 0; cb < CB; cb++) wv[u][cb][0] = wv[u][cb][1] = 0.0;
#pragma unroll
			for (int t = 0; t < TB; t++) {
				const int r = 8 * (warp + NW * t) + 2 * q;
#pragma unroll
				for (int cb = 0; cb < CB; cb++) {
					const int l = 8 * cb + g;
					double y0 = 0.0, y1 = 0.0;
					if (r < pr && l < nc) {
						const double *p = x.addr(c0 + r, l0 + l);
						if (vec) {
							const double2 y = *(const double2 *)p;
							y0 = y.x;
							y1 = r + 1 < pr ? y.y : 0.0;
						} else {
							y0 = *p;
							if (r + 1 < pr) y1 = x.at(c0 + r + 1, l0 + l);
						}
					}
					f[t][cb][0] = y0;
					f[t][cb][1] = y1;
				}
			}
#pragma unroll
			for (int t = 0; t < TB; t++) {
				const int r0 = 8 * (warp + NW * t);
				if (r0 < pr) {
#pragma unroll
					for (int h = 0; h < 2; h++) {
						const double *vr = V + (size_t)(r0 + 2 * q + h) * PLD + g;
						const double v0 = vr[0], v1 = vr[8];
#pragma unroll
						for (int cb = 0; cb < CB; cb++) {
							qr_dmma(wv[0][cb][0], wv[0][cb][1], v0, f[t][cb][h]);
							qr_dmma(wv[1][cb][0], wv[1][cb][1], v1, f[t][cb][h]);
						}
					}
				}
			}
			double *pw = part + (size_t)warp * 16 * WLD;
#pragma unroll
			for (int u = 0; u < 2; u++)
#pragma unroll
				for (int cb = 0; cb < CB; cb++)
					*(double2 *)(pw + (8 * u + g) * WLD + 8 * cb + 2 * q) = make_double2(wv[u][cb][0], wv[u][cb][1]);
			__syncthreads();
			for (int e = tid; e < 16 * CW; e += NT) {
				const int k = e / CW, l = e % CW;
				double z = 0.0;
#pragma unroll
				for (int u = 0; u < NW; u++) z += part[(size_t)u * 16 * WLD + k * WLD + l];
				Wr[k * WLD + l] = z;
			}
			__syncthreads();
			for (int e = tid; e < 16 * CW; e += NT) {
				const int k = e / CW, l = e % CW;
				double z = 0.0;
#pragma unroll
				for (int u = 0; u < 16; u++) z = fma(Tt[k * TLD + u], Wr[u * WLD + l], z);
				Ws[k * WLD + l] = z;
			}
			__syncthreads();
#pragma unroll
			for (int ks = 0; ks < 4; ks++) {
				double av[CB];
#pragma unroll
				for (int cb = 0; cb < CB; cb++) av[cb] = -Ws[(4 * ks + q) * WLD + 8 * cb + g];
#pragma unroll
				for (int t = 0; t < TB; t++) {
					const int r0 = 8 * (warp + NW * t);
					if (r0 < pr) {
						const double vv = V[(size_t)(r0 + g) * PLD + 4 * ks + q];
#pragma unroll
						for (int cb = 0; cb < CB; cb++) qr_dmma(f[t][cb][0], f[t][cb][1], av[cb], vv);
					}
				}
			}
#pragma unroll
			for (int t = 0; t < TB; t++) {
				const int r = 8 * (warp + NW * t) + 2 * q;
#pragma unroll
				for (int cb = 0; cb < CB; cb++) {
					const int l = 8 * cb + g;
					if (r < pr && l < nc) {
						double *p = d.addr(c0 + r, l0 + l);
						if (vec && r + 1 < pr) {
							*(double2 *)p = make_double2(f[t][cb][0], f[t][cb][1]);
						} else {
							*p = f[t][cb][0];
							if (r + 1 < pr) d.at(c0 + r + 1, l0 + l) = f[t][cb][1];
						}
					}
				}
			}
		}
		__syncthreads();  // the next panel's columns are in D, V and the partial sums are free
	}
}

template <int NT, int RPT, int CW, int MINB>
int launch(int batch, SizeArg sz, MatArg<double> C, MatArg<double> D, cudaStream_t s, int max_m, int max_n, int classes) {
	auto kern = k_geqrf_reg<NT, RPT, CW, MINB>;
	const size_t smem = qr_plan(NT, CW, max_m).total;
	bf::smem_optin(kern, smem);
	kern<<<(unsigned)(batch * (long long)classes), NT, smem, s>>>(batch, sz, C, D, max_m, max_n, classes);
	return bf::check_launch();
}

}  // namespace

namespace bf {

bool dgeqrf_reg_fits(int max_m) { return max_m <= 512; }

int dgeqrf_reg_launch(int batch, SizeArg sz, MatArg<double> C, MatArg<double> D, cudaStream_t s, int max_m, int max_n,
                      int nt) {
	const int mx = max_m > max_n ? max_m : max_n;
	const int classes = (sz.pm && mx > 64 && batch <= (1 << 28)) ? 4 : 1;
	// NT / 16 lanes per column with RPT rows each
	if (nt <= 128) {
		if (max_m <= 16) return launch<64, 4, 16, 8>(batch, sz, C, D, s, max_m, max_n, classes);
		if (max_m <= 32) return launch<64, 8, 16, 8>(batch, sz, C, D, s, max_m, max_n, classes);
		if (max_m <= 64) return launch<128, 8, 16, 4>(batch, sz, C, D, s, max_m, max_n, classes);
		if (max_m <= 128) return launch<128, 16, 16, 4>(batch, sz, C, D, s, max_m, max_n, classes);
	}
	if (nt <= 256) {
		if (max_m <= 128) return launch<256, 8, 32, 2>(batch, sz, C, D, s, max_m, max_n, classes);
		if (max_m <= 256) return launch<256, 16, 16, 2>(batch, sz, C, D, s, max_m, max_n, classes);
	}
	// (two CTAs of 256 threads per SM spill beyond 256 rows: m = 384, n = 192 x
	// 3,791 20.2 ms against 15.7 for one of 512)
	if (max_m <= 256) return launch<512, 8, 32, 1>(batch, sz, C, D, s, max_m, max_n, classes);
	if (max_m <= 384) return launch<512, 12, 32, 1>(batch, sz, C, D, s, max_m, max_n, classes);
	return launch<512, 16, 32, 1>(batch, sz, C, D, s, max_m, max_n, classes);
}

}  // namespace bf
