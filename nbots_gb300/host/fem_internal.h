/*
 * The device-resident FEM system shared by fem.c (elastic path) and
 * damage.c (quasi-static damage path).  Private to the host library.
 */
#ifndef NBG_FEM_INTERNAL_H
#define NBG_FEM_INTERNAL_H

#include "nbots_gb300.h"

struct nbg_fem {
	nbg_mesh_t m;
	uint32_t N;        /* dofs */
	uint64_t nnz;
	void *stream;
	/* device arrays */
	double *nod, *K, *F, *u, *strain, *stress, *E, *Ke, *Fe, *main_stress;
	double *damage;    /* per Gauss point, owned by the damage solve */
	uint32_t *conn, *row_ptr, *col_idx, *inc_ptr, *inc_elem, *distorted;
	uint8_t *inc_local, *enabled;
	unsigned long long *matched;
	int *status;
	double nu;
	int has_enabled;
	void *cg_ws;
	size_t cg_ws_bytes;
	/* 2x2-block SELL copy (bsr.cu), filled from K on demand */
	int bsr_ok;
	nbg_bsr_t bsr;
	uint32_t *slice_off, *bcol;
	double *b64, *dinv64;
	float *b32, *dinv32;
	uint16_t *blo;
	uint8_t *bxt;
	int block_order;           /* NBG_ORDER_* */
	uint32_t block_sigma;      /* SELL-C-sigma window, 0: default */
	uint32_t *perm, *iperm;    /* the block layout's node order, or NULL */
	void *bc_buf;              /* boundary-condition lists on the device, kept */
	size_t bc_bytes;
	uint32_t *ev_ptr;          /* per dof: its first event, N + 1 */
	double *simp_rho, *simp_out, *simp_e, *simp_lam;  /* nbg_fem_simp buffers */
	int borrowed_csr;          /* row_ptr, col_idx and K belong to the caller */
};

/* A FEM system on a CSR the caller owns on the device (row_ptr[N + 1],
 * col_idx, values K; not freed by nbg_fem_destroy), N = 2 N_nod: the mesh
 * arrays, F, u, strain and stress, and with need_incidence the node ->
 * element incidence that assembly needs.  No block layout.  The gather
 * assembly writes every pattern entry (those no element reaches get 0) and
 * reports a missing element pair as NBG_ERR_PATTERN. */
int nbg_fem_create_on_csr(nbg_fem_t **out, const nbg_mesh_t *m, uint64_t nnz,
			  uint32_t *row_ptr, uint32_t *col_idx, double *K, int need_incidence,
			  void *stream);

/* Assembly with an optional device array of damage per Gauss point; E NULL
 * means the moduli are already in f->E. */
int nbg_fem_assemble_dev_damage(nbg_fem_t *f, const double *E, double nu, double thickness,
				double density, int self_weight, const double gravity[2],
				const uint8_t *enabled, const double *damage);
/* Element matrices as node blocks (nbg_fem_element_bytes per element) and
 * loads (one double per element without self weight, else 2 nen N_elem), and
 * their gather, which does nothing when *distorted is set (assemble.cu). */
size_t nbg_fem_element_bytes(uint32_t nen);
int nbg_fem_element_blocks(uint32_t nen, uint32_t N_elem, const double *nod, const uint32_t *conn,
			   const double *E, double nu, double thickness, double density,
			   int self_weight, double gx, double gy, const uint8_t *enabled,
			   const double *damage, double *Ke, double *Fe, uint32_t *distorted,
			   void *stream);
int nbg_fem_gather_blocks(uint32_t nen, uint32_t N_nod, uint32_t N_elem, const uint32_t *inc_ptr,
			  const uint32_t *inc_elem, const uint8_t *inc_local,
			  const uint32_t *row_ptr, const uint32_t *col_idx, const uint32_t *conn,
			  const double *Ke, const double *Fe, int self_weight, double *K, double *F,
			  unsigned long long *matched, const uint32_t *distorted, void *stream);

/* xy[2 k] = nod of node ids[k]; ev_ptr[i] = how many of the ascending
 * ev_dof[n_ev] are below i, i = 0 .. N (device arrays, assemble.cu). */
int nbg_fem_pick_nodes(uint32_t n, const uint32_t *ids, const double *nod, double *xy,
		       void *stream);
int nbg_fem_event_ptr(uint32_t N, uint32_t n_ev, const uint32_t *ev_dof, uint32_t *ev_ptr,
		      void *stream);

/* Grow the device workspace *ws of *have bytes, whose content is lost, to `want` bytes,
 * or, where there is no memory for them, to `least` (solve.c). */
int nbg_ws_grow(void **ws, size_t *have, size_t want, size_t least);

/* Grow f's CG workspace to what nbg_cg_f64 needs for f->N dofs. */
int nbg_fem_cg_workspace(nbg_fem_t *f);

#endif
