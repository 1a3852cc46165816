/* slabplan.h -- host-side plan of the slab-pipelined 3D solve. */
#ifndef FTEIK_SLABPLAN_H
#define FTEIK_SLABPLAN_H
#include "fteik_dev.h"
#include <stdbool.h>

typedef struct {
    fk_slabs3d_t dev; /* device pointers passed to fk3d_solve_slabs */
    void *mem;        /* the one device allocation behind them */
    int nwork, npass;
    const int *pairs_all; /* the source pairs (dev.pairs is this or NULL) */
    int *nxy;             /* host [2 nwork]: nx, ny of every work item */
    int *work_tiles;      /* host [nwork + 1] (dev.work_tiles) */
    void *tile_mem;       /* device allocation of the tile schedule */
    bool have_tiles;
    int tile_key;         /* precision and convergence they were prepared for */
} fk_slabplan_t;

/* Build the plan for nwork work items with the given grid sizes and grid
 * numbers (gid); npass is the most Gauss-Seidel passes a solve will run;
 * pairing (0 or 1) lets consecutive work items of one grid walk the passes
 * together (the pairs are built either way: pairs_all).  The plan's bounded waits take the library's current poll limit
 * (fteik_b200_setSpinLimit).  Returns 0 on success. */
int fk_slabplan_build(fk_slabplan_t *pl, int nwork, const int *nx, const int *ny, const int *nz,
                      const int *gid, int npass, int pairing, const char *who);
void fk_slabplan_free(fk_slabplan_t *pl);
/* Prepare the tile schedule of a built plan (once for a precision and
 * convergence setting); have_tiles tells whether every work item's tiles fit
 * the chip at once and the device had the memory for them (tens of MB; without,
 * the slabs run).  Returns 0 unless a copy failed or the host's memory ran out. */
int fk_slabplan_tiles(fk_slabplan_t *pl, int precision, int converge, const char *who);
/* Give its memory back (the slabs are in use). */
void fk_slabplan_drop_tiles(fk_slabplan_t *pl);
#endif
