// Cholesky potrf_l (blasfeo_hp_pm/d_lapack_lib4.c:918) and syrk_potrf_ln (:1848)
// for instances with n <= 64: one warp per instance, the whole lower triangle in registers, the
// trailing updates on the FP64 tensor cores (DMMA, mma.sync m8n8k4 f64).
//
// The matrix is a grid of 8 x 8 blocks; block (I,J), J <= I, is held as an
// m8n8 accumulator fragment: lane l keeps row 8I + l/4, columns 8J + 2(l%4)
// and 8J + 2(l%4) + 1.  Unfactored blocks are kept NEGATED (F = -A), so the
// rank-8 trailing update A_IJ -= L_IK L_JK^T is a plain accumulate,
// F_IJ += L_IK L_JK^T, two m8n8k4 DMMAs per block.
//
// Right-looking by 8-column panels (chol_frag.cuh): the panel's pivots two at
// a time, then every block right of it gets two DMMAs.  Pivot rule of
// kernel/generic/kernel_dgemm_4x4_lib4.c:5700-5710: c > 0 -> L_jj = c * rsqrt(c),
// dA_j = rsqrt(c); else 0 and 0.  Everything is unrolled over the compile-time
// block grid (N8 = ceil(n/8)), so the fragments never leave registers; rows and
// columns n..8*N8-1 hold the identity.  The instance arrives through shared
// memory (16-byte cp.async copies of the lower panels, all in flight
// together).  HBM traffic: one read and one write of the lower triangle.
//
// FP32 matrices are computed in FP64 and rounded when they are stored.
// SYRK: D = chol(C + A B^T): the product is formed in the same fragments first
// (A and B in chunks of 8 columns, double buffered in the place that C's panels
// take afterwards), so the sum is never written: FP32 n = 50, k = 37 x 6,000 as
// two launches 125 + 127 us, this kernel 109.
//
// Bound: latency with the two warps per SM sub-partition that the registers allow
// (n = 64): a matrix is about 6,000 instructions, and a warp issues one every 7.6
// cycles (ncu: 2.8 of them waiting for an earlier result, 1.1 for the FP64 pipe, 0.7
// for shared memory, 0.6 for global memory, 0.5 for instructions; issue slots 26%
// used, the pipe 38%), 45,000 cycles a matrix.  The pivots themselves (two per 220
// cycles, 7,000 a matrix) and the tensor steps (384 of 15 cycles) are the smaller
// part.  8,000 matrices of n = 64: pivots, rows and columns broadcast by shuffles 171
// us, this form 156 (n = 48: 21,000 matrices 526 -> 309 us, n = 32: 40,000 198 -> 150).
// With the product the fragments of n = 41..48 spill (208 bytes of stores in FP32).
#include "chol_frag.cuh"
#include "kernels.cuh"

namespace {

constexpr unsigned FULL = 0xffffffffu;

__host__ __device__ constexpr int blk(int i, int j) { return i * (i + 1) / 2 + j; }

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
	asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// doubles of the compact lower panels of an n8 x n8 matrix (panel p keeps its
// columns 0..4p+3 at offset 8p(p+1), the global panel layout cut at the
// diagonal tile)
__host__ __device__ constexpr int lower_panels(int n8) { return 8 * (n8 / 4) * (n8 / 4 + 1); }

// shared memory of one warp in bytes: the lower panels (SYRK: or two buffers of
// 8 columns of A and B), then 64 inverse pivots and the 16 entries of frag::panel
template <typename T, bool SYRK>
__host__ __device__ constexpr int panel_bytes(int n8) {
	const int lp = lower_panels(8 * n8) * (int)sizeof(T), ab = SYRK ? 256 * n8 * (int)sizeof(T) : 0;
	return ((lp > ab ? lp : ab) + 15) / 16 * 16;
}
template <typename T, bool SYRK>
__host__ __device__ constexpr int warp_bytes(int n8) { return panel_bytes<T, SYRK>(n8) + 80 * 8; }

// The same factorization column by column in global memory by one warp, for
// matrices with a pivot that frag::panel does not take (subnormal, infinite, NaN)
template <typename T>
__device__ __noinline__ void potrf_warp(PMat<T> c, PMat<T> d, PMat<T> a, PMat<T> b, int n, int k, int *info, int lane) {
	int bad = 0;
	for (int j = 0; j < n; j++)
		for (int i = j + lane; i < n; i += 32) {
			T s = c.at(i, j);
			for (int l = 0; l < k; l++) s = fma(a.at(i, l), b.at(j, l), s);
			d.at(i, j) = s;
		}
	__syncwarp();
	for (int j = 0; j < n; j++) {
		const double p = (double)d.at(j, j);
		const bool ok = p > 0.0;
		const double iv = ok ? rsqrt(p) : 0.0;
		// info of an infinite pivot (1 / L_jj = 0, L_jj = inf * 0 = NaN): FP64 looks at
		// the pivot, FP32 at L_jj, as the FP32 kernel for n > 64 does
		if ((!ok || (sizeof(T) == 4 && !(p * iv > 0.0))) && bad == 0) bad = j + 1;
		__syncwarp();
		for (int i = j + lane; i < n; i += 32)
			d.at(i, j) = i == j ? (T)(ok ? p * iv : 0.0) : d.at(i, j) * (T)iv;
		if (lane == 0) d.d[j] = (T)iv;
		__syncwarp();
		for (int l = j + 1; l < n; l++) {
			const T t = d.at(l, j);
			for (int i = l + lane; i < n; i += 32) d.at(i, l) = fma(-d.at(i, j), t, d.at(i, l));
		}
		__syncwarp();
	}
	if (info && lane == 0) *info = bad;
}

// 8 columns k0.. of the n rows of x into dst (panel p at 32 p, column at 4 kk),
// zeros beyond column k; rows beyond n of the last panel as they are
template <typename T>
__device__ __forceinline__ void stage8(T *dst, const PMat<T> &x, int n, int k, int k0, bool fast, int lane) {
	const int P = (n + 3) >> 2;
	if (fast) {
		constexpr int E = 16 / sizeof(T), PP = 32 / E;  // elements per copy, copies per panel
		const uint32_t s = (uint32_t)__cvta_generic_to_shared(dst);
		for (int c = lane; c < P * PP; c += 32) {
			const int p = c / PP, w = c % PP * E, kk = w >> 2;
			const bool ok = k0 + kk < k;
			const T *g = ok ? x.addr(4 * p + (w & 3), k0 + kk) : x.p;
			asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s + 16u * c), "l"(g), "r"(ok ? 16u : 0u)
			             : "memory");
		}
	} else {
		for (int e = lane; e < P * 32; e += 32) {
			const int p = e >> 5, kk = (e & 31) >> 2, row = 4 * p + (e & 3);
			dst[e] = (row < n && k0 + kk < k) ? x.at(row, k0 + kk) : T(0);
		}
	}
}

// panels K.. of the factorization (compile-time K, so the fragments stay in registers)
template <int N8, int K>
__device__ __forceinline__ void factor(double (&F)[N8 * (N8 + 1) / 2][2], double *sc, double *dv, int r, int q) {
	if constexpr (K < N8) {
		double P[N8 - K][2];
#pragma unroll
		for (int I = K; I < N8; I++) {
			P[I - K][0] = F[blk(I, K)][0];
			P[I - K][1] = F[blk(I, K)][1];
		}
		frag::panel<N8 - K>(P, sc, dv + 8 * K, r, q);
		// trailing update, next panel's column first, the first step of every
		// block of a column before the second
#pragma unroll
		for (int J = K + 1; J < N8; J++)
#pragma unroll
			for (int e = 0; e < 2; e++)
#pragma unroll
				for (int I = J; I < N8; I++) frag::dmma(F[blk(I, J)][0], F[blk(I, J)][1], P[I - K][e], P[J - K][e]);
#pragma unroll
		for (int I = K; I < N8; I++) {
			F[blk(I, K)][0] = P[I - K][0];
			F[blk(I, K)][1] = P[I - K][1];
		}
		factor<N8, K + 1>(F, sc, dv, r, q);
	}
}

template <typename T, int N8, int WPC, int MINB, bool SYRK>
__global__ void __launch_bounds__(32 * WPC, MINB)
    k_potrf_dmma(int batch, SizeArg sz, MatArg<T> A, MatArg<T> B, MatArg<T> C, MatArg<T> D, int *info) {
	constexpr int NB = N8 * (N8 + 1) / 2;
	const int lane = threadIdx.x & 31;
	const int b = blockIdx.x * WPC + (threadIdx.x >> 5);
	if (b >= batch) return;
	const int n = sz.M(b);
	if (n <= 0 || n > 8 * N8) return;
	const PMat<T> c = C.get(b), d = D.get(b);
	const int r = lane >> 2, q = lane & 3;
	extern __shared__ __align__(16) unsigned char pot_smem[];
	T *S = (T *)(pot_smem + (threadIdx.x >> 5) * warp_bytes<T, SYRK>(N8));
	double *dv = (double *)((unsigned char *)S + panel_bytes<T, SYRK>(N8));

	// fragments, negated: -(A B^T) first, then -C
	double F[NB][2];
	PMat<T> xa = c, xb = c;
	int k = 0;
	if constexpr (SYRK) {
		xa = A.get(b);
		xb = B.get(b);
		k = sz.K(b);
#pragma unroll
		for (int e = 0; e < NB; e++) F[e][0] = F[e][1] = 0.0;
		const bool fa = ((xa.ri & 3) == 0) && ((((uintptr_t)xa.p) & 15) == 0);
		const bool fb = ((xb.ri & 3) == 0) && ((((uintptr_t)xb.p) & 15) == 0);
		const bool same = xa.p == xb.p && xa.ri == xb.ri && xa.cj == xb.cj && xa.cn == xb.cn;
		auto stage = [&](int k0, int buf) {
			T *dst = S + buf * 128 * N8;
			if (k0 < k) {
				stage8(dst, xa, n, k, k0, fa, lane);
				if (!same) stage8(dst + 64 * N8, xb, n, k, k0, fb, lane);
			}
			asm volatile("cp.async.commit_group;" ::: "memory");
		};
		stage(0, 0);
		for (int k0 = 0, buf = 0; k0 < k; k0 += 8, buf ^= 1) {
			stage(k0 + 8, buf ^ 1);
			asm volatile("cp.async.wait_group 1;" ::: "memory");
			__syncwarp();
			const T *sa = S + buf * 128 * N8, *sb = same ? sa : sa + 64 * N8;
#pragma unroll
			for (int ks = 0; ks < 2; ks++) {
				double av[N8];
#pragma unroll
				for (int I = 0; I < N8; I++) av[I] = -(double)sa[(2 * I + (r >> 2)) * 32 + 4 * (4 * ks + q) + (r & 3)];
#pragma unroll
				for (int J = 0; J < N8; J++) {
					const double bv = (double)sb[(2 * J + (r >> 2)) * 32 + 4 * (4 * ks + q) + (r & 3)];
#pragma unroll
					for (int I = J; I < N8; I++) frag::dmma(F[blk(I, J)][0], F[blk(I, J)][1], av[I], bv);
				}
			}
			__syncwarp();
		}
		asm volatile("cp.async.wait_all;" ::: "memory");
		__syncwarp();
	}

	// Stage the lower panels in shared memory with 16-byte asynchronous copies
	// (one wait for the whole instance: every copy is in flight at once), then
	// fill the fragments from there.  Rows not starting a panel, or panels not
	// 16-byte aligned, are read element by element from global memory.
	const bool staged = ((c.ri & 3) == 0) && ((((uintptr_t)c.p) & 15) == 0);
	if (staged) {
		constexpr int E = 16 / sizeof(T);
		const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(S);
		const int P = (n + 3) >> 2;
		for (int p = 0; p < P; p++) {
			const T *g = c.addr(4 * p, 0);
			for (int ch = lane; ch < 16 / E * (p + 1); ch += 32)
				cp_async16(sbase + (uint32_t)sizeof(T) * (uint32_t)(8 * p * (p + 1) + E * ch), g + E * ch);
		}
		asm volatile("cp.async.wait_all;" ::: "memory");
		__syncwarp();
	}
	// identity in the padding, zeros above the diagonal
#pragma unroll
	for (int I = 0; I < N8; I++)
#pragma unroll
		for (int J = 0; J <= I; J++)
#pragma unroll
			for (int h = 0; h < 2; h++) {
				const int gi = 8 * I + r, gj = 8 * J + 2 * q + h;
				double v;
				if (gi < n && gj < n) {
					if (gj > gi) {
						v = 0.0;
					} else {
						v = (double)(staged ? S[8 * (gi >> 2) * ((gi >> 2) + 1) + 4 * gj + (gi & 3)] : *c.addr(gi, gj));
						v = SYRK ? F[blk(I, J)][h] - v : -v;
					}
				} else {
					v = (gi == gj) ? -1.0 : 0.0;
				}
				F[blk(I, J)][h] = v;
			}

	factor<N8, 0>(F, dv + 64, dv, r, q);
	__syncwarp();
	const double i0 = dv[lane], i1 = N8 > 4 ? dv[N8 > 4 ? 32 + lane : 0] : 1.0;
	const double inf = __longlong_as_double(0x7ff0000000000000LL);
	bool odd = (lane < 8 * N8 && !(i0 < inf)) || (32 + lane < 8 * N8 && !(i1 < inf));
#pragma unroll
	for (int I = 0; I < N8; I++) odd |= frag::odd_diag(F[blk(I, I)], r, q);
	if (__any_sync(FULL, odd)) {
		potrf_warp<T>(c, d, xa, xb, n, k, info ? info + b : nullptr, lane);
		return;
	}
	if (lane < n) d.d[lane] = (T)fabs(i0);
	if (32 + lane < n) d.d[32 + lane] = (T)fabs(i1);
	const unsigned z0 = __ballot_sync(FULL, lane < n && frag::bad_pivot(i0)),
	               z1 = __ballot_sync(FULL, 32 + lane < n && frag::bad_pivot(i1));
	const int bad = z0 ? __ffs(z0) : (z1 ? 32 + __ffs(z1) : 0);
	if (bad) {
#pragma unroll
		for (int I = 0; I < N8; I++)
#pragma unroll
			for (int h = 0; h < 2; h++)
				if (r == 2 * q + h && frag::bad_pivot(dv[8 * I + r])) F[blk(I, I)][h] = 0.0;
	}

	// store the lower triangle of L
#pragma unroll
	for (int I = 0; I < N8; I++)
#pragma unroll
		for (int J = 0; J <= I; J++)
#pragma unroll
			for (int h = 0; h < 2; h++) {
				const int gi = 8 * I + r, gj = 8 * J + 2 * q + h;
				if (gi < n && gj <= gi) *d.addr(gi, gj) = (T)F[blk(I, J)][h];
			}
	if (info && lane == 0) info[b] = bad;
}

template <typename T, bool SYRK, int N8>
void launch_n8(int batch, SizeArg sz, MatArg<T> A, MatArg<T> B, MatArg<T> C, MatArg<T> D, int *info, cudaStream_t s) {
	constexpr int WPC = N8 <= 4 ? 4 : (N8 <= 6 ? 2 : 1);
	// resident CTAs per SM by the registers that the fragments need: 8, 12, 16,
	// 16, 20, 24, 32, 32 warps per SM for N8 = 8 .. 1 (the chain of a matrix is
	// hidden by the others; a tighter cap spills fragments)
	constexpr int MINB = N8 == 8 ? 8 : (N8 == 7 ? 12 : (N8 >= 5 ? 8 : (N8 == 4 ? 5 : (N8 == 3 ? 6 : 8))));
	const size_t smem = (size_t)WPC * warp_bytes<T, SYRK>(N8);
	auto kern = k_potrf_dmma<T, N8, WPC, MINB, SYRK>;
	bf::smem_optin(kern, smem);
	kern<<<(batch + WPC - 1) / WPC, 32 * WPC, smem, s>>>(batch, sz, A, B, C, D, info);
}

template <typename T, bool SYRK>
int launch(int batch, SizeArg sz, int max_m, MatArg<T> A, MatArg<T> B, MatArg<T> C, MatArg<T> D, int *info,
           cudaStream_t s) {
	if (max_m <= 0 || batch <= 0) return BLASFEO_B200_OK;
	switch ((max_m + 7) / 8) {
	case 1: launch_n8<T, SYRK, 1>(batch, sz, A, B, C, D, info, s); break;
	case 2: launch_n8<T, SYRK, 2>(batch, sz, A, B, C, D, info, s); break;
	case 3: launch_n8<T, SYRK, 3>(batch, sz, A, B, C, D, info, s); break;
	case 4: launch_n8<T, SYRK, 4>(batch, sz, A, B, C, D, info, s); break;
	case 5: launch_n8<T, SYRK, 5>(batch, sz, A, B, C, D, info, s); break;
	case 6: launch_n8<T, SYRK, 6>(batch, sz, A, B, C, D, info, s); break;
	case 7: launch_n8<T, SYRK, 7>(batch, sz, A, B, C, D, info, s); break;
	case 8: launch_n8<T, SYRK, 8>(batch, sz, A, B, C, D, info, s); break;
	default: return BLASFEO_B200_ENOTSUP;
	}
	return bf::check_launch();
}

}  // namespace

namespace bf {

// potrf_l, one warp per instance, for max_m <= 64
template <typename T>
int potrf_dmma_launch(int batch, SizeArg sz, int max_m, MatArg<T> C, MatArg<T> D, int *info, cudaStream_t s) {
	return launch<T, false>(batch, sz, max_m, C, C, C, D, info, s);
}
template int potrf_dmma_launch<double>(int, SizeArg, int, MatArg<double>, MatArg<double>, int *, cudaStream_t);
template int potrf_dmma_launch<float>(int, SizeArg, int, MatArg<float>, MatArg<float>, int *, cudaStream_t);

// D = chol(C + A B^T), one warp per instance, for max_m <= 64
template <typename T>
int syrk_potrf_dmma_launch(int batch, SizeArg sz, int max_m, MatArg<T> A, MatArg<T> B, MatArg<T> C, MatArg<T> D,
                           int *info, cudaStream_t s) {
	return launch<T, true>(batch, sz, max_m, A, B, C, D, info, s);
}
template int syrk_potrf_dmma_launch<double>(int, SizeArg, int, MatArg<double>, MatArg<double>, MatArg<double>,
                                            MatArg<double>, int *, cudaStream_t);
template int syrk_potrf_dmma_launch<float>(int, SizeArg, int, MatArg<float>, MatArg<float>, MatArg<float>,
                                           MatArg<float>, int *, cudaStream_t);

}  // namespace bf
