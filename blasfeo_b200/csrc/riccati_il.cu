// Batched Riccati factorization on batch-interleaved slabs: the kernel of
// riccati_core.cuh.
//
// Slabs are stage-major so that the problems of a CTA are consecutive
// instances at every stage: stage k of problem b is instance k * bs + b,
// bs = batch rounded up to a multiple of 16.  Each element of the CTA's 8
// problems is one contiguous 64-byte run in HBM.
#include "riccati_core.cuh"

namespace {

using quad::IL;

bool il16(const struct blasfeo_dmat_batch_il *s, int n, long long need) {
	return s && s->mem && s->m == 16 && s->n == n && (long long)s->batch >= need && s->il == IL &&
	       !((uintptr_t)s->mem & 15);
}

}  // namespace

extern "C" int blasfeo_dric_trf_batch_il(int batch, int N, int nx, int nu, struct blasfeo_dmat_batch_il *sBAbt,
                                         struct blasfeo_dmat_batch_il *sRSQ, struct blasfeo_dmat_batch_il *sL,
                                         int *info, void *stream) {
	if (batch < 0 || N < 0 || nx < 1 || nu < 0) return BLASFEO_B200_EINVAL;
	if (batch == 0) return BLASFEO_B200_OK;
	if (nu + nx > 16) return BLASFEO_B200_ENOTSUP;
	const long long bs = (batch + IL - 1) / IL * IL;
	if (!il16(sRSQ, 16, (N + 1) * bs) || !il16(sL, 16, (N + 1) * bs) || sRSQ->gstride != sL->gstride)
		return BLASFEO_B200_EINVAL;
	if (N > 0 && !il16(sBAbt, nx, N * bs)) return BLASFEO_B200_EINVAL;
	ric::Args a;
	a.batch = batch;
	a.N = N;
	a.nx = nx;
	a.nu = nu;
	a.cnx = N > 0 ? sBAbt->cn : 4;
	a.BA = N > 0 ? sBAbt->mem : nullptr;
	a.RSQ = sRSQ->mem;
	a.L = sL->mem;
	a.Ld = nullptr;
	a.sba = N > 0 ? sBAbt->gstride : 0;
	a.srsq = sRSQ->gstride;
	a.sl = sL->gstride;
	a.bs = bs;
	a.info = info;
	return ric::launch<true>(a, (cudaStream_t)stream);
}
