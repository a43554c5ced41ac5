// FP64 potrf_l for instances whose lower triangle does not fit in shared
// memory: one CTA per instance, left-looking 16-column panels with the
// updates on the FP64 tensor cores (chol_ll.cuh).
#include "chol_ll.cuh"
#include "kernels.cuh"

namespace {

// 128 threads, MINB resident CTAs per SM, FR fragment rows by UNR steps of 8
// columns in flight in a warp's panel update.  Bound by the latency of L (L2)
// and of the diagonal blocks.  Shorter matrices have few fragment rows to hand
// out and gain from more CTAs; longer ones from two fragment rows on each pair
// of operand loads.  us for uniform batches, <1, 4, 7> / <2, 2, 6> (and with
// the other warps idle during the diagonal blocks): n = 72 x 22,733 595 / 679
// (933), n = 128 x 5,394 388 / 400 (624), n = 192 x 1,957 392 / 396 (644), n =
// 200 x 1,767 446 / 370 (600), n = 256 x 953 589 / 529 (830), n = 300 x 640
// 651 / 558 (787).
constexpr int LL_NT = 128;
constexpr int LL_SHORT_N = 160;  // up to here <1, 4, 7>

template <int FR, int UNR, int MINB>
__global__ void __launch_bounds__(LL_NT, MINB)
    k_potrf_ll(SizeArg sz, MatArg<double> C, MatArg<double> D, int *info, int min_n, int max_n) {
	extern __shared__ __align__(16) double ll_smem[];
	__shared__ int s_bad;
	const int b = blockIdx.x;
	const int n = sz.M(b);
	if (n <= min_n || n > max_n) return;
	if (threadIdx.x == 0) s_bad = 0;
	__syncthreads();
	chol_ll<LL_NT, FR, UNR>(C.get(b), D.get(b), n, ll_smem, &s_bad);
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
	if (!sz.pm && max_m > LL_SHORT_N && min_n < LL_SHORT_N) min_n = LL_SHORT_N;
	const int mid = max_m < LL_SHORT_N ? max_m : LL_SHORT_N;
	if (min_n < mid) {
		const size_t smem = ll_smem_bytes(mid);
		bf::smem_optin(k_potrf_ll<1, 4, 7>, smem);
		k_potrf_ll<1, 4, 7><<<batch, LL_NT, smem, s>>>(sz, C, D, info, min_n, mid);
	}
	if (max_m > mid) {
		const size_t smem = ll_smem_bytes(max_m);
		bf::smem_optin(k_potrf_ll<2, 2, 6>, smem);
		k_potrf_ll<2, 2, 6><<<batch, LL_NT, smem, s>>>(sz, C, D, info, min_n > mid ? min_n : mid, max_m);
	}
	return check_launch();
}

}  // namespace bf
