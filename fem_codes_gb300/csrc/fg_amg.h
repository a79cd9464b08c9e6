/* Device state of the double-pairwise AMG preconditioner (host/amg.c sets it
 * up, amg.cu runs the V-cycle).  Plain C header. */
#ifndef FG_AMG_H
#define FG_AMG_H

#include <cuda_runtime_api.h>

#include "femgpu.h"

#ifdef __cplusplus
extern "C" {
#endif

/* The updates of one launch of SOR sweeps in an order in which each comes
 * after those it reads, levels padded to four: row | second << 30 (second: the update
 * belongs to the second of two sweeps run together), -1 padding. */
typedef struct { int *item; int nitem, wide; /* items of the widest level */ } fg_amg_sched;

#define FG_AMG_NW 4

typedef struct fg_amg_level {
	int n, nnz, longest;
	/* device: CSR, diagonal and its inverse (even levels: the smoothed ones) */
	int *ptr, *col;
	double *val, *diag, *rdiag;
	double *f;
	double *w[FG_AMG_NW];        /* iterates of the SOR sweeps (in the arena) */
	double *u;                   /* the current one                          */
	/* SOR schedules of the forward and reverse sweeps: [0] one sweep (nr
	 * odd), [1] two sweeps together (nr >= 2) */
	fg_amg_sched fw[2], bw[2];
	/* even l below the coarsest: restriction to level l+2 (4 fine rows per
	 * level-(l+2) row, -1 where absent) and the composite aggregate map */
	int4 *quad;
	int *agg2;
	int nc2;
	/* host copies: the level's CSR and (l below the coarsest) its matching */
	int *h_ptr, *h_col, *h_match;
	double *h_val;
} fg_amg_level;

struct femgpu_amg {
	int ncl, nr;
	double beta, omega;
	int nlevels;                 /* 2*ncl + 1 matrices */
	fg_amg_level *lv;
	double *qcopy;               /* [n0]: the input when q and z alias */
	double *arena;               /* the levels' w vectors */
	long long narena;
	void *ticket;                /* [nticket] fg_ticket, one per SOR launch of a cycle */
	int nticket;
	int *err;                    /* [2] errors of the device calls and of the
	                              * host ones (a solver passes its own word) */
	int wait1;                   /* 1 + bound of a wait, in polls; 0: default  */
	cudaStream_t stream, own_stream;
};

/* z = M^-1 q: one V-cycle (dpa_Vcycle_precond, amg_dpa.c:485-506).  Every
 * kernel is skipped while *active == 0 (active may be NULL). */
int fg_amg_vcycle(femgpu_amg *g, const double *q, double *z, const int *active, int *err);

#ifdef __cplusplus
}
#endif
#endif
