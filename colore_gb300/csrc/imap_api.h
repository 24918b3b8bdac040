/*
 * imap_api.h -- launch interface of imap.cu.
 */
#ifndef CG_IMAP_API_H
#define CG_IMAP_API_H

#include <cuda_runtime.h>
#include <stdint.h>

#include "cg_dev.cuh"
#include "cg_exact.h"

/* One listed cell (16 bytes): ix | iy << 16; iz | flags << 11 | half(edrr)
 * << 16 with the flags the shell mode (2 bits, CG_SH_*), delta + 1 (2 bits)
 * and double (16: every sample decided in double); brightness; radial
 * shift.  Grids up to 2048 cells a side. */
struct __align__(16) cg_imap_rec {
  unsigned int ixy, izf;
  float temp, drr;
};

#define CG_IMAP_REC_BYTES 16
/* A bucket per shell -1 .. nr of the cells' corners and per class of
 * cg_cell_class: bucket 3 (j + 1) + class. */
#define CG_IMAP_CLASSES 3
#define CG_IMAP_CNT 32 /* stride of the rooms' counters, 256 bytes: at 128 the two busy ones of a
                          shell shared an L2 slice (listing of 12 shells on 256^3 210 -> 240 us) */
#define CG_IMAP_BUCKETS_MAX (CG_IMAP_CLASSES * 4100) /* nr <= 4096 */

struct cg_imap_params {
  cg::Box box;
  const float *phi;  /* the potential */
  cg_imap_args a;    /* tables, corners, shells (device pointers) */
  cg_imap_seg *seg;  /* the tables' segments (na - 1) and, past them, the bits of their
                        largest factor bound (all written by cg_imap_paint) */
  int nr, nbk;       /* shells; buckets nbk = CG_IMAP_CLASSES (nr + 2) */
  long long npix;
  float2 *acc;       /* nr * npix, RING: summed brightness, samples */
  int packed;        /* samples as a float (cg_imap_pixel_max below 2^24), else as int bits */
  unsigned int *err;
  unsigned long long *xstats; /* [2] cells, [3] samples decided in double */
  int force_double;
  /* cells are listed per bucket (the shell of their corner, which fixes nsub,
   * and the class, which fixes the painting loop).  Shell j has two rooms
   * (cg_imap_rooms) next to each other, w = 2 (j + 1) + (polar corner): general
   * cells on counter 2 w, the others on 2 w + 1 (CG_IMAP_CNT apart), one upwards
   * from the room's begin and one downwards from its end, at[counter].  Either
   * may exceed its cap: those cells are painted by the listing kernel */
  cg_imap_rec *recs;
  const long long *at, *cap;
  unsigned long long *cnt;
  /* set on the device: the first record of every bucket and their number, and
   * the painting pass's chunks, chunk_off[b] the first of bucket b (nbk + 1) */
  longlong2 *buckets;
  unsigned long long *chunk_off;
  /* ctr: [0] chunks taken, [1] rows taken, [2] samples drawn, [3] samples
   * painted by the listing kernel, [4] double-queue entries */
  unsigned long long *ctr;
  unsigned long long *queue; /* record << 30 | sample, for the double pass */
  long long queue_cap;
};

cudaError_t cg_imap_paint(cudaStream_t s, const float *dens, const float *phi, const cg_imap_params *p, int nsm);
/* RING pixels of n float directions (device arrays) at nside by the
 * margin-checked decision the painting uses, with coordinate error ein
 * relative to r; -1 where only double can decide. */
cudaError_t cg_pix_checked_dev(cudaStream_t s, int nside, const float *xyz, long long n, float ein, long long *pix,
                               int nsm);
/* Shared memory of the painting kernel for nr shells and nbk buckets. */
size_t cg_imap_shell_smem(int nr, int nbk);

#endif
