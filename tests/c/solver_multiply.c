/*
 * host/solve.c against a GPU that is not there: nbg_solver_multiply returns only
 * when nothing that it launched can still use the caller's vectors, also when a
 * later launch fails.
 */
#include <stdio.h>

#include "solve.c"

static int reading, fail_spmv;

int nbg_copy_in_f64(size_t n, const double *src, double *dst, void *stream)
{
	(void)n; (void)src; (void)dst; (void)stream;
	reading = 1;  /* until the stream has been waited for */
	return NBG_OK;
}
int nbg_h2d(void *dst, const void *src, size_t bytes, void *stream)
{
	(void)dst; (void)src; (void)bytes; (void)stream;
	return NBG_OK;
}
int nbg_d2h(void *dst, const void *src, size_t bytes, void *stream)
{
	return nbg_h2d(dst, src, bytes, stream);
}
int nbg_spmv_csr_f64(uint32_t N, const uint32_t *rp, const uint32_t *ci, const double *val,
		     const double *x, double *y, void *stream)
{
	(void)N; (void)rp; (void)ci; (void)val; (void)x; (void)y; (void)stream;
	return fail_spmv ? NBG_ERR_CUDA : NBG_OK;
}
int nbg_stream_sync(void *stream)
{
	(void)stream;
	reading = 0;
	return NBG_OK;
}
int main(void)
{
	nbg_solver_t s;
	double v[2];
	for (int direct = 0; direct < 2; direct++)
		for (fail_spmv = 0; fail_spmv < 2; fail_spmv++) {
			memset(&s, 0, sizeof(s));
			s.have_pattern = 1;
			s.host_direct = direct;
			s.N = 100000;
			if (nbg_solver_multiply(&s, v, v) != (fail_spmv ? NBG_ERR_CUDA : NBG_OK))
				return 1;
			if (reading)
				return 2;
		}
	printf("ok\n");
	return 0;
}
