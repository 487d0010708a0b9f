/*
 * host/solve.c against a GPU that has only so much memory: where the FP64 block CG's
 * workspace with its plan cannot be had, the solve runs in the one without.
 */
#include <stdio.h>

#include "fem_internal.h"
#include "solve.c"

static size_t room, used, given;
static int allocs, solves;

size_t nbg_cg_bsr_workspace_bytes(uint32_t N)
{
	(void)N;
	return 1000;
}
size_t nbg_cg_bsr_layout_workspace_bytes(const nbg_bsr_t *A)
{
	(void)A;
	return 5000;
}
int nbg_dev_alloc(void **p, size_t bytes)
{
	allocs++;
	*p = NULL;
	if (bytes > room)
		return NBG_ERR_NOMEM;
	used = bytes;
	*p = &used;
	return NBG_OK;
}
int nbg_dev_free(void *p)
{
	if (p)
		used = 0;
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
int nbg_stream_sync(void *stream)
{
	(void)stream;
	return NBG_OK;
}
int nbg_cg_bsr_f64(const nbg_bsr_t *A, const double *b, double *x, uint32_t max_iter, double tol,
		   unsigned flags, nbg_cg_result_t *result, void *ws, size_t ws_bytes, void *stream)
{
	(void)A; (void)b; (void)x; (void)max_iter; (void)tol; (void)flags; (void)stream;
	memset(result, 0, sizeof(*result));
	given = ws ? ws_bytes : 0;
	solves++;
	return NBG_OK;
}

int main(void)
{
	/* room, then: the solve's status, the workspace it got */
	static const struct { size_t room; int rc; size_t given; } t[] = {
		{10000, NBG_OK, 5000}, {5000, NBG_OK, 5000}, {4999, NBG_OK, 1000},
		{1000, NBG_OK, 1000}, {999, NBG_ERR_NOMEM, 0}};
	double v[2] = {0.0, 0.0};
	for (int k = 0; k < 5; k++) {
		nbg_solver_t s;
		nbg_solve_info_t info;
		memset(&s, 0, sizeof(s));
		s.have_pattern = s.bsr_ok = 1;
		s.N = 2;
		room = t[k].room;
		used = given = 0;
		solves = 0;
		if (nbg_solver_solve(&s, v, v, 10, 1e-8, 0, NBG_METHOD_FP64, &info) != t[k].rc)
			return 1;
		if (given != t[k].given || used != t[k].given || s.ws_bytes != t[k].given)
			return 2;
		if (solves != (t[k].rc == NBG_OK))
			return 3;
		/* the same again allocates no more where it got all that it can use */
		allocs = 0;
		if (nbg_solver_solve(&s, v, v, 10, 1e-8, 0, NBG_METHOD_FP64, &info) != t[k].rc)
			return 4;
		if (t[k].given == 5000 && allocs)
			return 5;
	}
	/* the one without its plan is the whole of it: one try */
	void *ws = NULL;
	size_t have = 0;
	room = 10;
	allocs = 0;
	if (nbg_ws_grow(&ws, &have, 1000, 1000) != NBG_ERR_NOMEM || ws || have || allocs != 1)
		return 6;
	printf("ok\n");
	return 0;
}
