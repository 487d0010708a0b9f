/*
 * host/solve.c against a GPU that is not there: nbg_solver_multiply hands a kernel
 * only vectors of the caller's that start on a double; others go through copies.
 */
#include <stdio.h>

#include "solve.c"

static const void *kernel_in, *kernel_out, *copied_in;
static void *copied_out;

int nbg_copy_in_f64(size_t n, const double *src, double *dst, void *stream)
{
	(void)n; (void)dst; (void)stream;
	kernel_in = src;
	return NBG_OK;
}
int nbg_h2d(void *dst, const void *src, size_t bytes, void *stream)
{
	(void)dst; (void)bytes; (void)stream;
	copied_in = src;
	return NBG_OK;
}
int nbg_d2h(void *dst, const void *src, size_t bytes, void *stream)
{
	(void)src; (void)bytes; (void)stream;
	copied_out = dst;
	return NBG_OK;
}
int nbg_spmv_csr_f64(uint32_t N, const uint32_t *rp, const uint32_t *ci, const double *val,
		     const double *x, double *y, void *stream)
{
	(void)N; (void)rp; (void)ci; (void)val; (void)x; (void)stream;
	kernel_out = y;
	return NBG_OK;
}
int nbg_stream_sync(void *stream)
{
	(void)stream;
	return NBG_OK;
}

int main(void)
{
	static double mem[8], dev[8];
	for (int k = 0; k < 64; k++) {
		/* bytes past a double of in and of out */
		const int pi = k & 7, po = k >> 3;
		const double *in = (const double *)((char *)mem + pi);
		double *out = (double *)((char *)(mem + 4) + po);
		for (uint32_t N = 100; N <= 100000; N *= 1000) {
			nbg_solver_t s;
			memset(&s, 0, sizeof(s));
			s.have_pattern = 1;
			s.host_direct = 1;
			s.N = N;
			s.b = dev;
			kernel_in = kernel_out = copied_in = copied_out = NULL;
			if (nbg_solver_multiply(&s, in, out) != NBG_OK)
				return 1;
			const int by_kernel = N == 100000 && pi == 0;
			if (kernel_in != (by_kernel ? in : NULL) || copied_in != (by_kernel ? NULL : in))
				return 2;
			if (kernel_out != (po ? dev : out) || copied_out != (po ? out : NULL))
				return 3;
		}
	}
	printf("ok\n");
	return 0;
}
