// FP64 potrf_l for instances whose lower triangle does not fit in shared
// memory: one CTA per instance, left-looking 16-column panels with the
// updates on the FP64 tensor cores (chol_ll.cuh).
#include "chol_ll.cuh"
#include "kernels.cuh"

namespace {

// 128 threads, POTRF_LL_MINB resident CTAs per SM: the serial panel chain of
// one instance is hidden behind the other instances on the SM, so occupancy
// pays for a few spilled registers; POTRF_LL_FR fragment rows per warp in the
// panel update
#ifndef POTRF_LL_MINB
#define POTRF_LL_MINB 6
#endif
#ifndef POTRF_LL_FR
#define POTRF_LL_FR 1
#endif
constexpr int LL_NT = 128;
// Up to here the diagonal blocks are factored in tensor core fragments, beyond
// by rows and shuffles: the panel updates of longer matrices keep the tensor
// pipe busy and the diagonal chain waits for it (us for uniform batches,
// fragments / rows: n = 72 x 22,733 922 / 1,193, n = 128 x 5,394 592 / 700,
// n = 160 x 3,088 578 / 628, n = 192 x 1,957 584 / 655, n = 200 x 1,767 610 /
// 601, n = 224 x 1,331 709 / 668, n = 256 x 953 918 / 823)
constexpr int LL_FRAG_N = 192;

template <bool FRAG>
__global__ void __launch_bounds__(LL_NT, POTRF_LL_MINB)
    k_potrf_ll(SizeArg sz, MatArg<double> C, MatArg<double> D, int *info, int min_n, int max_n) {
	extern __shared__ __align__(16) double ll_smem[];
	__shared__ int s_bad;
	const int b = blockIdx.x;
	const int n = sz.M(b);
	if (n <= min_n || n > max_n) return;
	if (threadIdx.x == 0) s_bad = 0;
	__syncthreads();
	chol_ll<LL_NT, POTRF_LL_FR, FRAG>(C.get(b), D.get(b), n, ll_smem, &s_bad);
	if (info && threadIdx.x == 0) info[b] = s_bad;
}

}  // namespace

namespace bf {

// largest n the blocked global-memory kernel takes (its panel lives in shared memory)
int dpotrf_ll_max_n() {
	static int lim = 0;
	if (!lim)
		for (int v = 16; v <= 8192; v += 16)
			if (ll_smem_bytes(v) <= max_smem_optin()) lim = v;
	return lim;
}

// instances with min_n < n <= max_m
int dpotrf_ll_launch(int batch, SizeArg sz, int min_n, int max_m, MatArg<double> C, MatArg<double> D, int *info,
                     cudaStream_t s) {
	if (batch <= 0 || max_m <= min_n) return BLASFEO_B200_OK;
	if (max_m > dpotrf_ll_max_n()) return BLASFEO_B200_ENOTSUP;
	// one launch per range, each kernel skips the instances of the other (equal
	// sizes are in one range)
	if (!sz.pm && max_m > LL_FRAG_N && min_n < LL_FRAG_N) min_n = LL_FRAG_N;
	const int mid = max_m < LL_FRAG_N ? max_m : LL_FRAG_N;
	if (min_n < mid) {
		const size_t smem = ll_smem_bytes(mid);
		bf::smem_optin(k_potrf_ll<true>, smem);
		k_potrf_ll<true><<<batch, LL_NT, smem, s>>>(sz, C, D, info, min_n, mid);
	}
	if (max_m > mid) {
		const size_t smem = ll_smem_bytes(max_m);
		bf::smem_optin(k_potrf_ll<false>, smem);
		k_potrf_ll<false><<<batch, LL_NT, smem, s>>>(sz, C, D, info, min_n > mid ? min_n : mid, max_m);
	}
	return check_launch();
}

}  // namespace bf
