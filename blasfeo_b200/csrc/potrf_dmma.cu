// FP64 Cholesky potrf_l (blasfeo_hp_pm/d_lapack_lib4.c:918) for instances with
// n <= 64: one warp per instance, the whole lower triangle in registers, the
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
// Bound: the pivot chain (two pivots per 220 cycles) with the warps that the
// registers allow (8 per SM at n = 64), then the FP64 tensor pipe (384 steps of
// 15 cycles per SM sub-partition at n = 64).  8,000 matrices of n = 64: pivots,
// rows and columns broadcast by shuffles 171 us, this form 155 us (n = 48:
// 21,000 matrices 526 -> 309 us, n = 32: 40,000 198 -> 150 us).
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

// shared memory of one warp: the lower panels, then 64 inverse pivots and the
// 16 entries of frag::panel
__host__ __device__ constexpr int warp_doubles(int n8) { return lower_panels(8 * n8) + 80; }

// The same factorization column by column in global memory by one warp, for
// matrices with a pivot that frag::panel does not take (subnormal, infinite, NaN)
__device__ __noinline__ void potrf_warp(PMat<double> c, PMat<double> d, int n, int *info, int lane) {
	int bad = 0;
	for (int j = 0; j < n; j++)
		for (int i = j + lane; i < n; i += 32) d.at(i, j) = c.at(i, j);
	__syncwarp();
	for (int j = 0; j < n; j++) {
		const double p = d.at(j, j);
		const bool ok = p > 0.0;
		const double iv = ok ? rsqrt(p) : 0.0;
		if (!ok && bad == 0) bad = j + 1;
		__syncwarp();
		for (int i = j + lane; i < n; i += 32) d.at(i, j) = (i == j && !ok) ? 0.0 : d.at(i, j) * iv;
		if (lane == 0) d.d[j] = iv;
		__syncwarp();
		for (int l = j + 1; l < n; l++) {
			const double t = d.at(l, j);
			for (int i = l + lane; i < n; i += 32) d.at(i, l) = fma(-d.at(i, j), t, d.at(i, l));
		}
		__syncwarp();
	}
	if (info && lane == 0) *info = bad;
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

template <int N8, int WPC, int MINB>
__global__ void __launch_bounds__(32 * WPC, MINB) k_potrf_dmma(int batch, SizeArg sz, MatArg<double> C,
                                                               MatArg<double> D, int *info) {
	constexpr int NB = N8 * (N8 + 1) / 2;
	const int lane = threadIdx.x & 31;
	const int b = blockIdx.x * WPC + (threadIdx.x >> 5);
	if (b >= batch) return;
	const int n = sz.M(b);
	if (n <= 0 || n > 8 * N8) return;
	const PMat<double> c = C.get(b), d = D.get(b);
	const int r = lane >> 2, q = lane & 3;

	// Stage the lower panels in shared memory with 16-byte asynchronous copies
	// (one wait for the whole instance: every copy is in flight at once), then
	// fill the fragments from there.  Rows not starting a panel, or panels not
	// 16-byte aligned, are read element by element from global memory.
	extern __shared__ __align__(16) double pot_smem[];
	double *S = pot_smem + (threadIdx.x >> 5) * warp_doubles(N8);
	double *dv = S + lower_panels(8 * N8);
	const bool staged = ((c.ri & 3) == 0) && ((((uintptr_t)c.p) & 15) == 0);
	if (staged) {
		const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(S);
		const int P = (n + 3) >> 2;
		for (int p = 0; p < P; p++) {
			const double *g = c.addr(4 * p, 0);
			for (int ch = lane; ch < 8 * (p + 1); ch += 32)
				cp_async16(sbase + 8u * (uint32_t)(8 * p * (p + 1) + 2 * ch), g + 2 * ch);
		}
		asm volatile("cp.async.wait_all;" ::: "memory");
		__syncwarp();
	}

	// fragments (negated), identity in the padding, zeros above the diagonal
	double F[NB][2];
#pragma unroll
	for (int I = 0; I < N8; I++)
#pragma unroll
		for (int J = 0; J <= I; J++)
#pragma unroll
			for (int h = 0; h < 2; h++) {
				const int gi = 8 * I + r, gj = 8 * J + 2 * q + h;
				double v;
				if (gi < n && gj < n) {
					if (gj > gi)
						v = 0.0;
					else
						v = -(staged ? S[8 * (gi >> 2) * ((gi >> 2) + 1) + 4 * gj + (gi & 3)] : *c.addr(gi, gj));
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
		potrf_warp(c, d, n, info ? info + b : nullptr, lane);
		return;
	}
	if (lane < n) d.d[lane] = fabs(i0);
	if (32 + lane < n) d.d[32 + lane] = fabs(i1);
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
				if (gi < n && gj <= gi) *d.addr(gi, gj) = F[blk(I, J)][h];
			}
	if (info && lane == 0) info[b] = bad;
}

template <int N8>
void launch_n8(int batch, SizeArg sz, MatArg<double> C, MatArg<double> D, int *info, cudaStream_t s) {
	constexpr int WPC = N8 <= 4 ? 4 : (N8 <= 6 ? 2 : 1);
	// resident CTAs per SM by the registers that the fragments need: 8, 12, 16,
	// 16, 20, 24, 32, 32 warps per SM for N8 = 8 .. 1 (the chain of a matrix is
	// hidden by the others; a tighter cap spills fragments)
	constexpr int MINB = N8 == 8 ? 8 : (N8 == 7 ? 12 : (N8 >= 5 ? 8 : (N8 == 4 ? 5 : (N8 == 3 ? 6 : 8))));
	const size_t smem = (size_t)WPC * warp_doubles(N8) * sizeof(double);
	k_potrf_dmma<N8, WPC, MINB><<<(batch + WPC - 1) / WPC, 32 * WPC, smem, s>>>(batch, sz, C, D, info);
}

}  // namespace

namespace bf {

// FP64 potrf_l, one warp per instance, for max_m <= 64
int dpotrf_dmma_launch(int batch, SizeArg sz, int max_m, MatArg<double> C, MatArg<double> D, int *info,
                       cudaStream_t s) {
	if (max_m <= 0 || batch <= 0) return BLASFEO_B200_OK;
	switch ((max_m + 7) / 8) {
	case 1: launch_n8<1>(batch, sz, C, D, info, s); break;
	case 2: launch_n8<2>(batch, sz, C, D, info, s); break;
	case 3: launch_n8<3>(batch, sz, C, D, info, s); break;
	case 4: launch_n8<4>(batch, sz, C, D, info, s); break;
	case 5: launch_n8<5>(batch, sz, C, D, info, s); break;
	case 6: launch_n8<6>(batch, sz, C, D, info, s); break;
	case 7: launch_n8<7>(batch, sz, C, D, info, s); break;
	case 8: launch_n8<8>(batch, sz, C, D, info, s); break;
	default: return BLASFEO_B200_ENOTSUP;
	}
	return check_launch();
}

}  // namespace bf
