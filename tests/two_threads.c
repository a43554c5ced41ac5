/* Two host threads, each on its own stream, that call one routine with different
 * sizes: two_threads trsm|getrf|ric n0 n1 calls.  Prints the failed calls of each
 * thread; exit code 1 if there were any. */
#include <cuda_runtime_api.h>
#include <pthread.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include "blasfeo_b200.h"

struct job {
	const char *op;
	int n, calls, failed;
};

static struct blasfeo_dmat_batch slab(int m, int n, int batch) {
	struct blasfeo_dmat_batch s;
	void *p = NULL;
	const size_t bytes = blasfeo_memsize_dmat_batch(m, n, batch);
	if (cudaMalloc(&p, bytes) != cudaSuccess || cudaMemset(p, 0, bytes) != cudaSuccess) exit(2);
	blasfeo_create_dmat_batch(m, n, batch, &s, p);
	return s;
}

static void *run(void *arg) {
	struct job *j = arg;
	const int n = j->n, batch = 160, few = 4, m = 33;
	cudaStream_t s;
	int *ipiv = NULL;
	if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess) exit(2);
	if (cudaMalloc((void **)&ipiv, sizeof(int) * few * n) != cudaSuccess) exit(2);
	struct blasfeo_dmat_batch a, b, d;
	const int ric = !strcmp(j->op, "ric"), lu = !strcmp(j->op, "getrf");
	if (ric) {
		a = slab(16, n, batch);
		b = slab(16, 16, 2 * batch);
		d = slab(16, 16, 2 * batch);
	} else {
		a = slab(n, n, batch);
		b = slab(lu ? n : m, n, batch);
		d = slab(lu ? n : m, n, batch);
	}
	cudaDeviceSynchronize();
	for (int i = 0; i < j->calls; i++) {
		int st;
		if (ric)
			st = blasfeo_dric_trf_batch(batch, 1, n, 0, &a, &b, &d, NULL, s);
		else if (lu)
			st = blasfeo_dgetrf_rp_batch(few, n, n, &b, 0, 0, &d, 0, 0, ipiv, NULL, s);
		else
			st = blasfeo_dtrsm_rltn_batch(batch, m, n, 1.0, &a, 0, 0, &b, 0, 0, &d, 0, 0, s);
		j->failed += st != 0;
		if (i % 64 == 63) cudaStreamSynchronize(s);
	}
	cudaStreamSynchronize(s);
	return NULL;
}

int main(int argc, char **argv) {
	if (argc != 5) return 2;
	struct job j[2];
	pthread_t t[2];
	cudaFree(0);
	for (int i = 0; i < 2; i++) {
		j[i].op = argv[1];
		j[i].n = atoi(argv[2 + i]);
		j[i].calls = atoi(argv[4]);
		j[i].failed = 0;
		pthread_create(&t[i], NULL, run, &j[i]);
	}
	for (int i = 0; i < 2; i++) pthread_join(t[i], NULL);
	printf("%d %d\n", j[0].failed, j[1].failed);
	return j[0].failed || j[1].failed;
}
