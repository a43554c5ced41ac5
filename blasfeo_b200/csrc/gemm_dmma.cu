// FP64 gemm_nt / syrk_ln on the FP64 tensor cores (DMMA, mma.sync m8n8k4
// f64): D = beta*C + alpha*A*B^T, syrk writing only the lower triangle
// (blasfeo_hp_pm/d_blas3_lib4.c:727 gemm_nt, :5400 syrk_ln).
//
// One CTA computes a BM x BN output tile of one instance; every warp owns a
// 32 x 32 sub-tile as 4 x 4 fragments of 8 x 8 (two FP64 accumulators per
// thread and fragment).  K is walked in BK = 16 slices through a 3-stage
// cp.async pipeline.  The staging copies BLASFEO's panel layout as it is: the
// BK columns of one 4-row panel are one contiguous run of 4*BK doubles in
// global memory and land as one contiguous run in shared memory, so every
// 16-byte copy is fully used.  An m8n8k4 operand fragment (8 rows x 4 k:
// lane l holds row l/4, k l%4) is then two 4x4 tiles of two panels, i.e. two
// contiguous 128-byte runs: conflict-free shared-memory loads.
//
// Out-of-range rows of a partial tile only feed output rows/columns that are
// never stored; columns k >= K are zero-filled in both operands.  Three modes
// (GemmMode; launch_dmma has the rule) differ in what a warp does of a partial
// tile and in how an uneven batch is spread over CTAs.  The 64 x 64 kernel is held
// to 128 registers but for WHOLE: 4 CTAs per SM hide each other's first copies
// and stores.  us, whole tiles at 3 CTAs per SM everywhere / now: 2,048 of sizes
// log-uniform up to 384 277 / 207, n = 50 x 5,000 124 / 112, n = 200 x 1,000 936 /
// 874, n = 128 x 2,000 322 / 316, n = 20 x 20,000 114 / 87, 10 x 10 x 300 x 5,000
// 153 / 108; syrk n = 128 x 2,000 246 / 240, n = 200 x 1,000 592 / 557; two stages
// at 5 CTAs spill (377 at n = 128).  C is read only when beta != 0 (as the HP
// kernels do).  Instances whose row offset is not a multiple of 4, or whose panels
// are not 16-byte aligned, are copied element by element (8-byte cp.async) with the
// same arithmetic.
#include <algorithm>

#include "common.cuh"
#include "kernels.cuh"

namespace {

constexpr int DM_BK = 16;
constexpr int DM_STAGES = 3;
constexpr int GCTAS = 4;  // CTAs per instance of an uneven batch, beside the helpers
constexpr int GHELP = 4;  // helpers per SM (as many as are resident)

// How a launch is split and what a warp multiplies of a partial tile (launch_dmma
// has the rule):
//   LIVE    a CTA per tile; the 8 x 8 fragments and 4-column steps that the output
//           needs;
//   WHOLE   a CTA per tile; everything, without a branch in copies and steps: the
//           shortest time of a single tile;
//   HELPED  a CTA for each of an instance's first tiles, the others spread over the
//           helpers; partial sub-tiles by halves, with the steps unrolled.
enum GemmMode { LIVE, WHOLE, HELPED };

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, uint32_t src_bytes) {
	asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const void *src, uint32_t src_bytes) {
	asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
	asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ void dmma(double &d0, double &d1, double a, double b) {
	asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
	             : "+d"(d0), "+d"(d1)
	             : "d"(a), "d"(b));
}

// Stage the ROWS x BK slice (rows r0.., columns k0..) of one operand into
// shared memory `dst` (panel-major: panel p at p*4*BK, column kk at 4*kk).
// Chunk c (16 bytes, two rows of one column) of the slice sits at dst + 2c.
// SKIP: panels past the last row, which feed nothing that is stored, are not
// copied (without it they are zeros, and no copy has a branch).
template <int ROWS, int NT, bool SKIP>
__device__ __forceinline__ void stage_operand(double *dst, const PMat<double> &a, int rows, int kdim, int r0,
                                              int k0, bool fast) {
	const uint32_t sdst = (uint32_t)__cvta_generic_to_shared(dst);
	if (fast) {
		constexpr int CH = ROWS * DM_BK / 2;
#pragma unroll
		for (int c = threadIdx.x; c < CH; c += NT) {
			const int p = c / (2 * DM_BK), w = c % (2 * DM_BK);
			const int kk = w >> 1;
			if (SKIP && r0 + 4 * p >= rows) continue;
			const bool ok = (SKIP || r0 + 4 * p < rows) && k0 + kk < kdim;
			const double *src = ok ? a.addr(r0 + 4 * p + 2 * (w & 1), k0 + kk) : a.p;
			cp_async16(sdst + 16u * c, src, ok ? 16u : 0u);
		}
	} else {
		constexpr int EL = ROWS * DM_BK;
		for (int e = threadIdx.x; e < EL; e += NT) {
			const int p = e / (4 * DM_BK), w = e % (4 * DM_BK);
			const int kk = w >> 2, r = r0 + 4 * p + (w & 3);
			const bool ok = (r < rows) && (k0 + kk < kdim);
			const double *src = ok ? a.addr(r, k0 + kk) : a.p;
			cp_async8(sdst + 8u * e, src, ok ? 8u : 0u);
		}
	}
}

// rows r, r + 8, .. (F of them) of column kk of a staged slice
template <int F>
__device__ __forceinline__ void ld_frag(double (&v)[4], const double *t, int r, int kk) {
#pragma unroll
	for (int i = 0; i < F; i++) v[i] = t[((r + 8 * i) >> 2) * (4 * DM_BK) + kk * 4 + (r & 3)];
}

// FI x FJ fragments of a warp's sub-tile times the 4-column steps kq < kqn of a slice
template <int FI, int FJ>
__device__ __forceinline__ void mul(double (&acc)[4][4][2], const double *tA, const double *tB, int ra, int rb, int fk,
                                    int kqn) {
#pragma unroll
	for (int kq = 0; kq < DM_BK / 4; kq++) {
		if (kq >= kqn) break;
		double av[4], bv[4];
		ld_frag<FI>(av, tA, ra, 4 * kq + fk);
		ld_frag<FJ>(bv, tB, rb, 4 * kq + fk);
#pragma unroll
		for (int i = 0; i < FI; i++)
#pragma unroll
			for (int j = 0; j < FJ; j++) dmma(acc[i][j][0], acc[i][j][1], av[i], bv[j]);
	}
}

// output tiles of an m x n instance; LOWER: those that reach the lower triangle
template <int BM, int BN, bool LOWER>
__host__ __device__ inline int tile_count(int m, int n) {
	const int tm = cdiv(m, BM), tn = cdiv(n, BN);
	if (!LOWER) return tm * tn;
	static_assert(!LOWER || BM == BN, "a triangle of square tiles");
	return tm <= tn ? tm * (tm + 1) / 2 : tn * (tn + 1) / 2 + (tm - tn) * tn;
}
// first row and column of a tile (LOWER: row by row of the triangle, then whole rows)
template <int BM, int BN, bool LOWER>
__device__ __forceinline__ void tile_origin(int tile, int n, int &i0, int &j0) {
	const int tn = cdiv(n, BN);
	int ti, tj;
	if (LOWER && tile < tn * (tn + 1) / 2) {
		ti = (int)((sqrtf(8.0f * tile + 1.0f) - 1.0f) * 0.5f);
		while (ti * (ti + 1) / 2 > tile) ti--;
		while ((ti + 1) * (ti + 2) / 2 <= tile) ti++;
		tj = tile - ti * (ti + 1) / 2;
	} else {
		const int u = LOWER ? tile - tn * (tn + 1) / 2 : tile;
		ti = u / tn + (LOWER ? tn : 0);
		tj = u % tn;
	}
	i0 = ti * BM;
	j0 = tj * BN;
}

// The tiles beyond the first `ctas` of each instance form a list, instance by
// instance; helper h takes the entries h, h + helpers, ..  NT instances are
// looked at together: s_end[t] is where those of instance b0 + t end, counted
// from `base`.
template <int NT>
struct HelpList {
	int *s_end, *s_warp;
	int b0, total;
	long long base, next;
	// the next tile of this CTA (the whole CTA calls it), false after the last
	template <int BM, int BN>
	__device__ __forceinline__ bool take(int batch, const SizeArg &sz, int ctas, int helpers, int &b, int &tile) {
		const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
		while (next >= base + total) {
			base += total;
			b0 += NT;
			if (b0 >= batch) return false;
			int x = 0;
			if (b0 + (int)threadIdx.x < batch) {
				const int m = sz.M(b0 + threadIdx.x), n = sz.N(b0 + threadIdx.x);
				if (m > 0 && n > 0) x = max(0, tile_count<BM, BN, false>(m, n) - ctas);
			}
#pragma unroll
			for (int o = 1; o < 32; o <<= 1) {
				const int y = __shfl_up_sync(0xffffffffu, x, o);
				if (lane >= o) x += y;
			}
			if (lane == 31) s_warp[warp] = x;
			__syncthreads();
			total = 0;
			int before = 0;
#pragma unroll
			for (int w = 0; w < NT / 32; w++) {
				if (w == warp) before = total;
				total += s_warp[w];
			}
			s_end[threadIdx.x] = before + x;
			__syncthreads();
		}
		const int e = (int)(next - base);
		int lo = 0, hi = NT - 1;  // the first instance that ends beyond e
		while (lo < hi) {
			const int mid = (lo + hi) >> 1;
			if (s_end[mid] > e)
				hi = mid;
			else
				lo = mid + 1;
		}
		b = b0 + lo;
		tile = ctas + e - (lo ? s_end[lo - 1] : 0);
		next += helpers;
		return true;
	}
};

// one output tile of an instance, by the whole CTA
template <int BM, int BN, bool LOWER, GemmMode MODE>
__device__ __forceinline__ void gemm_tile(int tile, int m, int n, int k, double alpha, const PMat<double> &a,
                                          const PMat<double> &bm, double beta, const PMat<double> &c,
                                          const PMat<double> &d, bool fast_a, bool fast_b, double *sA, double *sB) {
	constexpr int WN = BN / 32;
	constexpr int NT = (BM / 32) * WN * 32;
	constexpr int SA = BM * DM_BK, SB = BN * DM_BK;  // doubles per stage
	constexpr bool SKIP = MODE != WHOLE;
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const int wm0 = (warp / WN) * 32, wn0 = (warp % WN) * 32;
	const int fr = lane >> 2, fk = lane & 3;
	const int KT = (k + DM_BK - 1) / DM_BK;
	int i0, j0;
	tile_origin<BM, BN, LOWER>(tile, n, i0, j0);
	// the warp's live 8 x 8 fragments: fi x fj, none where syrk's sub-tile is above the diagonal
	int fi = min(4, max(0, (m - i0 - wm0 + 7) >> 3)), fj = min(4, max(0, (n - j0 - wn0 + 7) >> 3));
	if (LOWER && j0 + wn0 > i0 + wm0) fi = 0;
	const bool full = MODE == WHOLE ? fi > 0 && fj > 0 : fi == 4 && fj == 4;
	double acc[4][4][2];
#pragma unroll
	for (int i = 0; i < 4; i++)
#pragma unroll
		for (int j = 0; j < 4; j++) acc[i][j][0] = acc[i][j][1] = 0.0;

#pragma unroll
	for (int s = 0; s < DM_STAGES - 1; s++) {
		if (s < KT) {
			stage_operand<BM, NT, SKIP>(sA + s * SA, a, m, k, i0, s * DM_BK, fast_a);
			stage_operand<BN, NT, SKIP>(sB + s * SB, bm, n, k, j0, s * DM_BK, fast_b);
		}
		cp_async_commit();
	}
	for (int kt = 0; kt < KT; kt++) {
		cp_async_wait<DM_STAGES - 2>();
		__syncthreads();
		{
			const int ks = kt + DM_STAGES - 1;
			if (ks < KT) {
				const int buf = ks % DM_STAGES;
				stage_operand<BM, NT, SKIP>(sA + buf * SA, a, m, k, i0, ks * DM_BK, fast_a);
				stage_operand<BN, NT, SKIP>(sB + buf * SB, bm, n, k, j0, ks * DM_BK, fast_b);
			}
			cp_async_commit();
		}
		const double *tA = sA + (kt % DM_STAGES) * SA;
		const double *tB = sB + (kt % DM_STAGES) * SB;
		const int kqn = min(DM_BK / 4, (k - kt * DM_BK + 3) >> 2);
		if (full) {
			mul<4, 4>(acc, tA, tB, wm0 + fr, wn0 + fr, fk, DM_BK / 4);
		} else if (MODE == HELPED && fi > 0 && fj > 0) {
			if (fi > 2 && fj > 2)
				mul<4, 4>(acc, tA, tB, wm0 + fr, wn0 + fr, fk, kqn);
			else if (fi > 2)
				mul<4, 2>(acc, tA, tB, wm0 + fr, wn0 + fr, fk, kqn);
			else if (fj > 2)
				mul<2, 4>(acc, tA, tB, wm0 + fr, wn0 + fr, fk, kqn);
			else
				mul<2, 2>(acc, tA, tB, wm0 + fr, wn0 + fr, fk, kqn);
		} else if (MODE == LIVE && fi == 2 && fj == 2) {
			mul<2, 2>(acc, tA, tB, wm0 + fr, wn0 + fr, fk, kqn);
		} else if (MODE == LIVE && fi == 3 && fj == 3) {
			mul<3, 3>(acc, tA, tB, wm0 + fr, wn0 + fr, fk, kqn);
		} else if (MODE == LIVE && fi > 0 && fj > 0) {
			for (int kq = 0; kq < kqn; kq++) {
				double av[4], bv[4];
				ld_frag<4>(av, tA, wm0 + fr, 4 * kq + fk);
				ld_frag<4>(bv, tB, wn0 + fr, 4 * kq + fk);
#pragma unroll
				for (int i = 0; i < 4; i++)
#pragma unroll
					for (int j = 0; j < 4; j++)
						if (i < fi && j < fj) dmma(acc[i][j][0], acc[i][j][1], av[i], bv[j]);
			}
		}
	}
	cp_async_wait<0>();

	// epilogue: fragment (i,j), thread holds row 8i + lane/4, columns 8j + 2(lane%4) + {0,1}
#pragma unroll
	for (int i = 0; i < 4; i++) {
		const int gi = i0 + wm0 + 8 * i + fr;
		if (gi >= m) continue;
#pragma unroll
		for (int j = 0; j < 4; j++) {
#pragma unroll
			for (int h = 0; h < 2; h++) {
				const int gj = j0 + wn0 + 8 * j + 2 * fk + h;
				if (gj >= n) continue;
				if (LOWER && gj > gi) continue;
				double v = alpha * acc[i][j][h];
				if (beta != 0.0) v = fma(beta, c.at(gi, gj), v);
				d.at(gi, gj) = v;
			}
		}
	}
}

template <int BM, int BN, bool LOWER, GemmMode MODE>
__global__ void __launch_bounds__((BM / 32) * (BN / 32) * 32, BM == 64 ? (MODE == WHOLE ? 3 : 4) : 1)
    k_dgemm_nt_dmma(int batch, SizeArg sz, double alpha, MatArg<double> A, MatArg<double> B, double beta,
                    MatArg<double> C, MatArg<double> D, int ctas, int helpers) {
	constexpr int NT = (BM / 32) * (BN / 32) * 32;
	extern __shared__ __align__(128) double dm_smem[];
	__shared__ int s_end[MODE == HELPED ? NT : 1], s_warp[NT / 32];
	double *sA = dm_smem;
	double *sB = dm_smem + DM_STAGES * BM * DM_BK;
	// one-dimensional grid: the helpers, then instance by instance: the CTAs that
	// share an instance's A and B slices run together and meet in L2
	const bool help = MODE == HELPED && (int)blockIdx.x < helpers;
	HelpList<NT> list{s_end, s_warp, -NT, 0, 0, blockIdx.x};
	int b, tile;
	if (MODE == HELPED) {
		b = (int)((blockIdx.x - (unsigned)helpers) / (unsigned)ctas);
		tile = (int)((blockIdx.x - (unsigned)helpers) % (unsigned)ctas);
		if (help && !list.template take<BM, BN>(batch, sz, ctas, helpers, b, tile)) return;
	} else {
		b = (int)(blockIdx.x / (unsigned)ctas);
		tile = (int)(blockIdx.x % (unsigned)ctas);
	}
	for (;;) {
		const int m = sz.M(b), n = sz.N(b), k = sz.K(b);
		if (m <= 0 || n <= 0) return;
		const int tiles = tile_count<BM, BN, LOWER>(m, n);
		if (tile >= tiles) return;
		const PMat<double> a = A.get(b), bm = B.get(b), c = C.get(b), d = D.get(b);
		// the 16-byte copies need panel-aligned rows and 16-byte aligned panels
		const bool fast_a = ((a.ri & 3) == 0) && ((((uintptr_t)a.p) & 15) == 0);
		const bool fast_b = ((bm.ri & 3) == 0) && ((((uintptr_t)bm.p) & 15) == 0);
		if (MODE == HELPED) {
			gemm_tile<BM, BN, LOWER, MODE>(tile, m, n, k, alpha, a, bm, beta, c, d, fast_a, fast_b, sA, sB);
			if (!help) return;
			__syncthreads();  // the next tile's copies overwrite the stages
			if (!list.template take<BM, BN>(batch, sz, ctas, helpers, b, tile)) return;
		} else {
			// one tile, written as a loop: the compiler's schedule without it takes
			// 19% longer for one-warp CTAs (n = 32 x 20,000 140 us against 118)
			for (; tile < tiles; tile += ctas) {
				gemm_tile<BM, BN, LOWER, MODE>(tile, m, n, k, alpha, a, bm, beta, c, d, fast_a, fast_b, sA, sB);
				__syncthreads();
			}
			return;
		}
	}
}

template <int BM, int BN, bool LOWER>
int launch_dmma(int batch, SizeArg sz, int max_m, int max_n, int max_k, double alpha, MatArg<double> A,
                MatArg<double> B, double beta, MatArg<double> C, MatArg<double> D, cudaStream_t s) {
	constexpr int NT = (BM / 32) * (BN / 32) * 32;
	const size_t smem = (size_t)DM_STAGES * (BM + BN) * DM_BK * sizeof(double);
	int ctas = tile_count<BM, BN, LOWER>(max_m, max_n), helpers = 0;
	const long long all = (long long)batch * ctas, sms = bf::num_sms();
	const bool uneven = sz.pm && !LOWER;
	GemmMode mode = LIVE;
	// WHOLE where the time is that of a few tiles one after another on an SM (us,
	// LIVE / WHOLE; the sums of a K slice must be long enough to matter): few 32 x 32
	// tiles (n = 256 x 1 28.9 / 26.9, n = 400 x 1 43 / 37); 64 x 64 tiles of which
	// little is padding, up to 3 per SM, and 5 or 6, which are two rounds for 3 CTAs
	// per SM as for 4 (n = 400 x 16 127 / 104); uneven batches with no more CTAs than
	// 64 per SM, whose few large instances' tiles pile up on SMs at 4 CTAs each (64 of
	// sizes log-uniform up to 384 72 / 54, 200 up to 300 80 / 57)
	if (BM == 32 ? (max_m > 32 || max_n > 32) && max_k >= 48 : max_k >= 64) {
		const bool most = 5LL * max_m * max_n >= 3LL * cdiv(max_m, BM) * BM * cdiv(max_n, BN) * BN;
		if (BM == 32 || (most && all <= 3 * sms) || (most && !LOWER && all > 4 * sms && all <= 6 * sms) ||
		    (uneven && ctas > 8 && all > 6 * sms && all <= 64 * sms))
			mode = WHOLE;
	}
	// HELPED beyond that: a grid of max_m x max_n tiles per instance is mostly CTAs
	// that find nothing to do (2,048 of sizes log-uniform up to 384: 7,072 of 73,728),
	// and with a fixed number of CTAs per instance a large one is left to few of them
	// (one of n = 2,000 among 600 small ones: 8 CTAs 22.3 ms, a grid of tiles 1.04,
	// helpers 0.74; one of n = 384 among 2,000: 189 / 97 / 58 us; 600 log-uniform up to
	// 384 365 / 276 / 263).  Fewer CTAs per instance than this leave the helpers, which
	// hold every SM, too much (64 of n = 1,000: 4.90 ms against 4.38)
	if (uneven && ctas > 8 && all > 64 * sms) {
		ctas = std::max(GCTAS, cdiv(32 * (int)sms, batch));
		helpers = GHELP * (int)sms;
		mode = HELPED;
	}
	const long long grid = helpers + (long long)batch * ctas;
	if (grid > 0x7fffffffLL) return BLASFEO_B200_ENOTSUP;
	auto kern = mode == HELPED ? k_dgemm_nt_dmma<BM, BN, LOWER, LOWER ? LIVE : HELPED>
	            : mode == WHOLE ? k_dgemm_nt_dmma<BM, BN, LOWER, WHOLE>
	                            : k_dgemm_nt_dmma<BM, BN, LOWER, LIVE>;
	bf::smem_optin(kern, smem);
	kern<<<(unsigned)grid, NT, smem, s>>>(batch, sz, alpha, A, B, beta, C, D, ctas, helpers);
	return bf::check_launch();
}

}  // namespace

namespace bf {

// FP64 tensor-core gemm_nt / syrk_ln: tile 0 = 64 x 64 (4 warps), 1 = 32 x 32 (1 warp)
template <bool LOWER>
int dgemm_nt_dmma_launch(int batch, SizeArg sz, int max_m, int max_n, int max_k, double alpha, MatArg<double> A,
                         MatArg<double> B, double beta, MatArg<double> C, MatArg<double> D, cudaStream_t s,
                         int tile) {
	if (tile == 0) return launch_dmma<64, 64, LOWER>(batch, sz, max_m, max_n, max_k, alpha, A, B, beta, C, D, s);
	return launch_dmma<32, 32, LOWER>(batch, sz, max_m, max_n, max_k, alpha, A, B, beta, C, D, s);
}
template int dgemm_nt_dmma_launch<false>(int, SizeArg, int, int, int, double, MatArg<double>, MatArg<double>, double,
                                         MatArg<double>, MatArg<double>, cudaStream_t, int);
template int dgemm_nt_dmma_launch<true>(int, SizeArg, int, int, int, double, MatArg<double>, MatArg<double>, double,
                                        MatArg<double>, MatArg<double>, cudaStream_t, int);

}  // namespace bf
