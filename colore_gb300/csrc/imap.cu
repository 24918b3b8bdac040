/*
 * imap.cu -- intensity-map painting (imap_set_cartesian_single,
 * imap.c:135-245).
 *
 * Every cell in the radial range of the shells carries a brightness
 * temp = T(r) bias_model(d, b(r)) norm(r) and a redshift-space shift dr_rsd;
 * it is split into nsub^3 sub-cells whose centres are placed in a shell (by
 * r + dr_rsd) and a RING pixel, where temp is added and a hit counted.  The
 * shells and pixels are decided as the reference's double arithmetic
 * decides them: in single precision where a bound on the distance to the
 * double value proves the decision, in float-float where that bound fails,
 * and in double only where the float-float bound fails too (cg_exact.h), so
 * the hit counts are those of the double arithmetic.
 *
 * nsub is fixed by the shell of the cell's corner radius and grows towards
 * the observer (from 2 at high redshift to ~20 for the nearest shells), and
 * a cell's class says which loop its samples need (cg_cell_class), so cells
 * are listed per shell and class -- one bucket each, holding cells of one
 * nsub and one loop -- and painted bucket after bucket.  The buckets of a shell
 * share two rooms from both ends (cg_imap_rooms), which no share of general
 * cells overfills:
 *
 *   k_imap_tab     The radial tables as one 32-byte record per segment.
 *   k_imap_list    Warps take groups of rows from a counter; a lane decides
 *                  one cell (listed or not, its shell, brightness, radial
 *                  shift, and whether all its samples certainly stay in one
 *                  shell or straddle one edge) from one segment record
 *                  (cg_imap_cell_seg) and appends it to its room: one atomic
 *                  per counter present in the warp, all issued together, on
 *                  counters that lie 256 bytes apart (next to each other
 *                  they sat in one L2 slice, whose atomics bounded the kernel:
 *                  65 against 54 ms of the stage at 1024^3).  Cells that the
 *                  segments leave open, and cells that find their room full
 *                  (painted by the warp), wait until the warp's rows are done.
 *                  504 thread-instructions a cell in range where a lookup with
 *                  a bound per table took 689: 20.6 -> 10.4 ms at 1024^3.
 *   k_imap_chunks  One block finds each bucket's records and cuts them into
 *                  chunks of about CHS samples: whole cells, or slices of one.
 *   k_imap_paint   Warps take chunks in bucket order, so the maps' working
 *                  set at any time is a few shells (50 MB per shell at nside
 *                  512) and the atomics stay in L2.  Each lane walks one unit
 *                  sample by sample, keeping a (key, count) run that it adds to
 *                  the maps with one two-float reduction.  Cells within one
 *                  octant, one of the two pixel regions and one shell or edge
 *                  -- all but the layers on the octants' planes, the cones
 *                  |cos theta| = 2/3, the nearest cells and those that span
 *                  several thin shells -- have these decisions taken once per
 *                  cell and walk along the line of sight, where the pixel
 *                  changes least.  Samples whose margins fail are staged per
 *                  warp in shared memory and queued in batches.  Bound by instruction issue (87 % of the slots): 91
 *                  thread-instructions a sample where deciding everything per
 *                  sample took 177, 79 -> 36 ms for the 1.3e10 samples at
 *                  1024^3; scalar atomics instead of the two-float reduction
 *                  cost 5.5 ms, a branch around it 1.7.
 *   k_imap_double  The queued samples: first in float-float, then, for the
 *                  few left, gathered per warp and decided in double 32 at a
 *                  time, the cell's radial shift computed once per run of
 *                  one record.
 */
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "cg_dev.cuh"
#include "imap_api.h"

namespace {
using namespace cg;

constexpr int IW = 4;     /* warps per block                     */
constexpr int ROWS = 2;   /* rows per fetch in k_imap_list        */
constexpr int LATE_CH = 64; /* words of 32 cells in a row: N <= 2048 */
constexpr int CHS = 4096; /* samples per painting chunk           */
constexpr int QB = 256;   /* queue entries staged per painting warp */
constexpr unsigned FULL = 0xffffffffu;
constexpr unsigned F_DOUBLE = 16u; /* flags: mode (2 bits), delta + 1 (2 bits), double */

/* Per-block copies of the species' shell tables. */
struct Sh {
  float *b; /* with two sentinels on either side */
  float *dxs;
  int *shell_of, *nsub;
  unsigned long long *chunk_off;
};

__host__ __device__ __forceinline__ size_t shell_smem(int nr, int nbk, bool chunks)
{
  size_t n = (size_t)(2 * nr + 4) * 4 + (size_t)(2 * nr + 1) * 4 + 2 * (size_t)(nr + 2) * 4;
  n = (n + 7) & ~(size_t)7;
  if (chunks) n += (size_t)(nbk + 1) * 8;
  return n;
}

/* Where the tables sit in the block's shared memory. */
__device__ __forceinline__ Sh shells_at(const cg_imap_params &p, unsigned char *raw)
{
  const int nr = p.nr;
  Sh s;
  s.b = reinterpret_cast<float *>(raw) + 2;
  s.shell_of = reinterpret_cast<int *>(s.b + 2 * nr + 2);
  s.nsub = s.shell_of + 2 * nr + 1;
  s.dxs = reinterpret_cast<float *>(s.nsub + nr + 2);
  s.chunk_off = reinterpret_cast<unsigned long long *>(raw + shell_smem(nr, p.nbk, false));
  return s;
}

/* The painting warps' queue stages follow the tables. */
__host__ __device__ __forceinline__ size_t paint_stage_off(int nr, int nbk) { return (shell_smem(nr, nbk, true) + 15) & ~(size_t)15; }
__host__ __device__ __forceinline__ size_t paint_smem(int nr, int nbk) { return paint_stage_off(nr, nbk) + (size_t)IW * (QB * 8 + 4); }
/* The double pass keeps the shells' bases where the painting keeps its
 * chunk table; its per-warp gathers (64 entries) follow. */
__host__ __device__ __forceinline__ size_t double_stage_off(int nr, int nbk) { return (shell_smem(nr, nbk, true) + 15) & ~(size_t)15; }

__device__ __forceinline__ Sh load_shells(const cg_imap_params &p, unsigned char *raw, bool chunks)
{
  const int nb = p.a.sh.nb, nr = p.nr;
  const Sh s = shells_at(p, raw);
  for (int i = (int)threadIdx.x - 2; i < nb + 2; i += blockDim.x)
    s.b[i] = i < 0 ? -3.0e38f : (i < nb ? p.a.sh.b[i] : 3.0e38f);
  for (int i = threadIdx.x; i <= nb; i += blockDim.x) s.shell_of[i] = p.a.sh.shell_of[i];
  for (int i = threadIdx.x; i < nr + 2; i += blockDim.x) {
    s.nsub[i] = p.a.nsub[i];
    s.dxs[i] = p.a.dxs[i];
  }
  if (chunks)
    for (int i = threadIdx.x; i <= p.nbk; i += blockDim.x) s.chunk_off[i] = p.chunk_off[i];
  return s;
}

__device__ __forceinline__ cg_imap_args args_with(const cg_imap_params &p, const Sh &s)
{
  cg_imap_args A = p.a;
  A.sh.b = s.b;
  A.sh.shell_of = s.shell_of;
  A.nsub = s.nsub;
  A.dxs = s.dxs;
  return A;
}

/* The counter of a listed cell: its room (shell j, polar corner or not) and the
 * end it is listed from. */
__device__ __forceinline__ int counter_of(int j, int polar, int cls)
{
  return 4 * (j + 1) + 2 * polar + (cls != CG_CELL_GENERAL);
}

/* Slot k of counter ct: the fast equatorial and the general polar cells upwards
 * from their room's begin, the others downwards from its end. */
__device__ __forceinline__ long long slot_of(const cg_imap_params &p, int ct, long long k)
{
  const int down = ((ct ^ (ct >> 1)) & 1) - 1; /* 0 or -1 */
  return p.at[ct] + (k ^ (long long)down);
}

/* Cells listed on counter ct.  None when both ends hold more than the room,
 * which bounds their sum unless the list is cut, and then the caps do. */
__device__ __forceinline__ long long listed(const cg_imap_params &p, int ct)
{
  long long n[2];
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int c = (ct & ~1) + k;
    const long long m = (long long)p.cnt[(size_t)c * CG_IMAP_CNT];
    n[k] = m < p.cap[c] ? m : p.cap[c];
  }
  const long long room = llabs(p.at[ct | 1] - p.at[ct & ~1]);
  if (n[0] + n[1] > room) {
    atomicOr(p.err, ERR_IMAP_ROOM);
    return 0;
  }
  return n[ct & 1];
}

/* A bucket's records, one after the other: the first and their number.  The
 * shell's rooms lie next to each other, with the general cells at the ends that
 * meet. */
__device__ __forceinline__ longlong2 bucket_of(const cg_imap_params &p, int b)
{
  const int s = b / CG_IMAP_CLASSES, cls = b - s * CG_IMAP_CLASSES;
  if (cls == CG_CELL_GENERAL) {
    const long long n = listed(p, 4 * s);
    return make_longlong2(p.at[4 * s + 2] - n, n + listed(p, 4 * s + 2));
  }
  const long long n = listed(p, 4 * s + 2 * cls - 1);
  return make_longlong2(cls == CG_CELL_EQ ? p.at[4 * s + 1] : p.at[4 * s + 3] - n, n);
}

static_assert(CG_CELL_GENERAL == 0 && CG_CELL_EQ == 1 && CG_CELL_POLAR == 2, "rooms by class");

template <typename K>
__device__ __forceinline__ K empty_key()
{
  return (K)~(K)0;
}

template <typename K>
__device__ __forceinline__ K key_of(const cg_imap_params &p, int s, long long pix)
{
  if (s < 0 || s >= p.nr) return empty_key<K>();
  if (sizeof(K) == 4) return (K)((unsigned)s * (unsigned)p.npix + (unsigned)pix);
  return (K)((long long)s * p.npix + pix);
}

/* n samples of summed brightness t on pixel k of the maps: one two-float
 * reduction when the counts are floats (p.packed), which halves the L2's
 * atomic operations, else a float and an integer one. */
__device__ __forceinline__ void add_to(const cg_imap_params &p, long long k, float t, float n)
{
  float2 *a = p.acc + k;
  if (p.packed) {
    asm volatile("red.relaxed.gpu.global.add.v2.f32 [%0], {%1, %2};" ::"l"(a), "f"(t), "f"(n) : "memory");
  } else {
    atomicAdd(&a->x, t);
    atomicAdd(reinterpret_cast<int *>(&a->y), (int)n);
  }
}

/* The lanes hold consecutive samples of one cell: each run of one key is added
 * to the maps once, by its first lane, with its length (sum += temp * run,
 * count += run). */
template <typename K>
__device__ __forceinline__ void add_runs(K key, float temp, int lane, const cg_imap_params &p)
{
  const K pk = __shfl_up_sync(FULL, key, 1);
  const bool valid = key != empty_key<K>();
  const bool head = valid && (lane == 0 || pk != key);
  const unsigned bnd = __ballot_sync(FULL, head || !valid);
  if (head) {
    const unsigned above = lane == 31 ? 0u : bnd & (FULL << (lane + 1));
    const int end = above ? __ffs(above) - 1 : 32;
    const float c = (float)(end - lane);
    add_to(p, (long long)key, CG_MUL(temp, c), c);
  }
}

/* Sub-cell (sx, sy, sz) of sample q < ns^3, x fastest. */
__device__ __forceinline__ void sub_of(int q, int ns, int *sx, int *sy, int *sz)
{
  const float inv_ns = 1.0f / (float)ns;
  int line, z;
  if (ns <= 128) {
    /* (q + 1/2)/ns is at least 1/(2 ns) from an integer and the float
     * product is within ns^2 2^-23 of it: exact while ns^3 < 2^22 */
    line = (int)(((float)q + 0.5f) * inv_ns);
    z = (int)(((float)line + 0.5f) * inv_ns);
  } else {
    line = q / ns;
    z = line / ns;
  }
  *sx = q - line * ns;
  *sy = line - z * ns;
  *sz = z;
}

/* Centred potential differences at a cell (get_rvel, imap.c:43-74): float
 * minus float, as the reference forms them from its float grid. */
__device__ __forceinline__ void grad_phi(const float *__restrict__ phi, int ix, int iy, int iz, int N, float v[3])
{
  v[0] = CG_SUB(__ldg(&phi[pidx(wrap(ix + 1, N), iy, iz, N)]), __ldg(&phi[pidx(wrap(ix - 1, N), iy, iz, N)]));
  v[1] = CG_SUB(__ldg(&phi[pidx(ix, wrap(iy + 1, N), iz, N)]), __ldg(&phi[pidx(ix, wrap(iy - 1, N), iz, N)]));
  v[2] = CG_SUB(__ldg(&phi[pidx(ix, iy, wrap(iz + 1, N), N)]), __ldg(&phi[pidx(ix, iy, wrap(iz - 1, N), N)]));
}

/* Brightness of a cell whose decisions were taken in double (imap.c:199,
 * 201), in single precision like every other cell's. */
__device__ __forceinline__ float temp32(const cg_imap_args &A, int ix, int iy, int iz, float d)
{
  const float x0 = A.xc[ix], y0 = A.yc[iy], z0 = A.zc[iz];
  const float r2 = CG_FMA(z0, z0, CG_FMA(y0, y0, CG_MUL(x0, x0)));
  const float rc = CG_MUL(r2, cg_rsqrt_fast(r2));
  const float tm = cg_tab_at(A.tz, A.na, A.idr, A.r, rc, 0.0f).v;
  const float b = cg_tab_at(A.bz, A.na, A.idr, A.r, rc, 0.0f).v;
  const float dn = cg_tab_at(A.norm, A.na, A.idr, A.r, rc, 0.0f).v;
  return CG_MUL(CG_MUL(tm, cg_bias_model(d, b, A.bias_model)), dn);
}

__device__ __forceinline__ cg_imap_rec pack(int ix, int iy, int iz, const cg_imap_cell &c, unsigned flags)
{
  cg_imap_rec r;
  r.ixy = (unsigned)ix | ((unsigned)iy << 16);
  const unsigned short eh = __half_as_ushort(__float2half_ru(c.edrr));
  r.izf = (unsigned)iz | (flags << 11) | ((unsigned)eh << 16);
  r.temp = c.temp;
  r.drr = c.drr;
  return r;
}

__device__ __forceinline__ cg_imap_cell unpack(const cg_imap_rec &r, int j, int *ix, int *iy, int *iz, int *dbl)
{
  cg_imap_cell c;
  *ix = (int)(r.ixy & 0xffffu);
  *iy = (int)(r.ixy >> 16);
  *iz = (int)(r.izf & 0x7ffu);
  const unsigned f = (r.izf >> 11) & 0x1fu;
  c.mode = (int)(f & 3u);
  c.delta = (int)((f >> 2) & 3u) - 1;
  *dbl = (f & F_DOUBLE) ? 1 : 0;
  c.edrr = __half2float(__ushort_as_half((unsigned short)(r.izf >> 16)));
  c.temp = r.temp;
  c.drr = r.drr;
  c.j = j;
  return c;
}

/* A sample of a cell the listing kernel paints itself: its double decision,
 * when needed, on the spot. */
template <typename K>
__device__ __noinline__ K sample_key_inline(const cg_imap_params &p, int ix, int iy, int iz,
                                            const cg_imap_cell &c, int dbl, int ns, int q)
{
  const cg_imap_args &A = p.a;
  int sx, sy, sz, s = -1;
  long long pix = 0;
  sub_of(q, ns, &sx, &sy, &sz);
  if (dbl || p.force_double || !cg_imap_sample_checked(&A, ix, iy, iz, &c, ns, sx, sy, sz, &s, &pix)) {
    float v[3];
    grad_phi(p.phi, ix, iy, iz, p.box.N, v);
    int j;
    double drr = 0;
    cgx_imap_cell(&A, ix, iy, iz, v, &j, &drr);
    cgx_imap_sample(&A, ix, iy, iz, ns, drr, sx, sy, sz, &s, &pix);
    atomicAdd(p.xstats + 3, 1ull);
  }
  return key_of<K>(p, s, pix);
}

/* The listing's table segments, with this realisation's normalisation. */
__global__ void __launch_bounds__(32) k_imap_tab(cg_imap_params p)
{
  const int i = blockIdx.x * 32 + threadIdx.x;
  float eg = 0.0f;
  if (i < p.a.na - 1) p.seg[i] = cg_imap_seg_make(&p.a, i, &eg);
  /* non-negative floats order like their bits */
  const unsigned m = __reduce_max_sync(FULL, __float_as_uint(eg));
  if (threadIdx.x == 0) atomicMax(reinterpret_cast<unsigned *>(p.seg + p.a.na - 1), m);
}

/* A cell that the segments leave open: with a bound per lookup
 * (cg_imap_cell_checked), then in double.  Out of line: rare, and long. */
struct OpenCell {
  cg_imap_cell c;
  int st, dbl, in_double;
};

__device__ __noinline__ OpenCell cell_open(const cg_imap_params &p, int ix, int iy, int iz, float d, float v0, float v1,
                                           float v2)
{
  const cg_imap_args &A = p.a;
  OpenCell o;
  const float v[3] = {v0, v1, v2};
  o.dbl = o.in_double = 0;
  o.st = cg_imap_cell_checked(&A, ix, iy, iz, d, v, &o.c);
  if (p.force_double && o.st == 1) o.st = 2;
  if (o.st == 2) {
    o.in_double = 1;
    int j;
    double drr;
    o.st = 0;
    if (cgx_imap_cell(&A, ix, iy, iz, v, &j, &drr)) {
      o.c.j = j;
      o.c.temp = temp32(A, ix, iy, iz, d);
      o.c.drr = (float)drr;
      o.c.edrr = 0.0f;
      o.c.mode = CG_SH_WALK;
      o.c.delta = 0;
      o.dbl = o.st = 1;
    }
  }
  return o;
}

/* Cells past their room (m: their lanes), painted by the warp. */
template <typename K>
__device__ __forceinline__ void paint_over(const cg_imap_params &p, unsigned m, const cg_imap_rec &rec, int ct, int lane)
{
  while (m) {
    const int l = __ffs(m) - 1;
    m &= m - 1;
    cg_imap_rec r;
    r.ixy = __shfl_sync(FULL, rec.ixy, l);
    r.izf = __shfl_sync(FULL, rec.izf, l);
    r.temp = __shfl_sync(FULL, rec.temp, l);
    r.drr = __shfl_sync(FULL, rec.drr, l);
    const int j = __shfl_sync(FULL, ct, l) / 4 - 1;
    int ix, iy, iz, dbl;
    const cg_imap_cell c = unpack(r, j, &ix, &iy, &iz, &dbl);
    const int ns = p.a.nsub[j + 1], n3 = ns * ns * ns;
    for (int q0 = 0; q0 < n3; q0 += 32) {
      const int q = q0 + lane;
      K key = empty_key<K>();
      if (q < n3) key = sample_key_inline<K>(p, ix, iy, iz, c, dbl, ns, q);
      add_runs(key, c.temp, lane, p);
    }
    if (lane == 0) atomicAdd(&p.ctr[3], (unsigned long long)n3);
  }
}

/* A warp's rows in words of 32 cells: the cells that the segments leave open,
 * and those that found their room full. */
struct Late {
  unsigned open[ROWS * LATE_CH], over[ROWS * LATE_CH];
};

/* Those cells, once per group of rows: out of the listing loop, whose registers
 * a call would spill. */
template <typename K>
__device__ __noinline__ void late_cells(const float *__restrict__ dens, const cg_imap_params &p, const Late &L, int rbeg,
                                        int rend, int lane)
{
  const int N = p.box.N, nch = N / 32, ngx = 2 * (N / 2 + 1);
  unsigned long long drawn = 0, ndbl = 0;
  __syncwarp();
  for (int g = 0; g < (rend - rbeg) * nch; g++) {
    const unsigned open = L.open[g], any = open | L.over[g];
    if (!any) continue;
    const int row = rbeg + g / nch, ix = (g % nch) * 32 + lane;
    const int iz = (int)divN(row, p.box), iy = row - iz * N;
    bool over = false;
    int ct = 0;
    cg_imap_rec rec = {0u, 0u, 0.0f, 0.0f};
    if ((any >> lane) & 1u) {
      float v[3];
      grad_phi(p.phi, ix, iy, iz, N, v);
      const OpenCell o = cell_open(p, ix, iy, iz, __ldg(dens + (long long)row * ngx + ix), v[0], v[1], v[2]);
      if (o.st == 1) {
        const int sfin = o.c.j + o.c.delta;
        const bool want = !(o.c.mode == CG_SH_SINGLE && (sfin < 0 || sfin >= p.nr));
        const float x0 = p.a.xc[ix], y0 = p.a.yc[iy], z0 = p.a.zc[iz];
        ct = counter_of(o.c.j, cg_corner_polar(z0, CG_FMA(x0, x0, CG_FMA(z0, z0, CG_MUL(y0, y0)))),
                        o.dbl ? CG_CELL_GENERAL : cg_cell_class(&p.a, &o.c, x0, y0, z0));
        rec = pack(ix, iy, iz, o.c, (unsigned)o.c.mode | ((unsigned)(o.c.delta + 1) << 2) | (o.dbl ? F_DOUBLE : 0u));
        over = want;
        if ((open >> lane) & 1u) {
          const int ns = p.a.nsub[o.c.j + 1];
          drawn += (unsigned long long)ns * ns * ns;
          if (want) {
            const long long k = (long long)atomicAdd(&p.cnt[(size_t)ct * CG_IMAP_CNT], 1ull);
            over = k >= p.cap[ct];
            if (!over) p.recs[slot_of(p, ct, k)] = rec;
          }
        }
      }
      if ((open >> lane) & 1u) ndbl += o.in_double;
    }
    paint_over<K>(p, __ballot_sync(FULL, over), rec, ct, lane);
  }
  if (drawn) atomicAdd(&p.ctr[2], drawn);
  if (ndbl) atomicAdd(p.xstats + 2, ndbl);
}

/* 12 blocks per SM: 5, 6, 8, 10 and 16 took 55.1, 53.8, 52.5, 51.2 and 50.5
 * against 50.7 ms of the stage at 1024^3 (16 loses at 256^3: 1194 against 1165
 * us).  Waiting for the reservations a step later, with the next cells decided
 * in between, cost more in registers than it hid (52.4 ms). */
template <typename K>
__global__ void __launch_bounds__(IW * 32, 12) k_imap_list(const float *__restrict__ dens, const float *__restrict__ phi,
                                                             const __grid_constant__ cg_imap_params p)
{
  extern __shared__ __align__(16) unsigned char sraw[];
  __shared__ Late late[IW];
  const Sh sh = load_shells(p, sraw, false);
  __syncthreads();
  const cg_imap_args A = args_with(p, sh);
  const int lane = threadIdx.x & 31;
  Late &L = late[threadIdx.x >> 5];
  const int N = p.box.N;
  const int nrow = N * N, nch = N / 32; /* N is a multiple of 32 */
  const float rlo = A.rmin - 1.0f, rhi = A.rmax + 1.0f;
  const float rlo2 = rlo > 0.0f ? rlo * rlo : 0.0f, rhi2 = rhi * rhi;
  const int ngx = 2 * (N / 2 + 1);
  const long long plane = (long long)ngx * N;
  const float eg = __uint_as_float(*reinterpret_cast<const unsigned *>(p.seg + A.na - 1));
  unsigned long long drawn = 0;
  for (;;) {
    int rbeg = 0;
    if (lane == 0) rbeg = (int)atomicAdd(&p.ctr[1], (unsigned long long)ROWS);
    rbeg = __shfl_sync(FULL, rbeg, 0);
    if (rbeg >= nrow) break;
    const int rend = rbeg + ROWS < nrow ? rbeg + ROWS : nrow;
    unsigned any_late = 0;
    for (int i = lane; i < ROWS * nch; i += 32) L.open[i] = L.over[i] = 0u;
    __syncwarp();
    for (int row = rbeg; row < rend; row++) {
      const int iz = (int)divN(row, p.box), iy = row - iz * N;
      const float y0 = A.yc[iy], z0 = A.zc[iz];
      const float yz2 = CG_FMA(z0, z0, CG_MUL(y0, y0));
      if (yz2 > rhi2) continue;
      const long long r0 = (long long)row * ngx;
      const int oyh = iy == N - 1 ? -(N - 1) * ngx : ngx, oyl = iy == 0 ? (N - 1) * ngx : -ngx;
      const long long ozh = iz == N - 1 ? -(N - 1) * plane : plane, ozl = iz == 0 ? (N - 1) * plane : -plane;
      for (int ch = 0; ch < nch; ch++) {
        const int ix = ch * 32 + lane;
        cg_imap_cell c;
        bool want = false, open = false; /* listed and painted; left to late_cells */
        const float x0 = A.xc[ix];
        const float r2 = CG_FMA(x0, x0, yz2);
        if (r2 >= rlo2 && r2 <= rhi2) {
          const float d = __ldg(dens + r0 + ix);
          const float *f = phi + r0 + ix;
          /* centred potential differences (get_rvel, imap.c:43-74) */
          const float v[3] = {CG_SUB(__ldg(f + (ix == N - 1 ? 1 - N : 1)), __ldg(f + (ix == 0 ? N - 1 : -1))),
                              CG_SUB(__ldg(f + oyh), __ldg(f + oyl)), CG_SUB(__ldg(f + ozh), __ldg(f + ozl))};
          const int st = p.force_double ? 2 : cg_imap_cell_seg(p.seg, eg, &A, x0, y0, z0, r2, d, v, &c);
          open = st == 2;
          if (st == 1) {
            const int ns = A.nsub[c.j + 1];
            drawn += (unsigned)(ns * ns * ns);
            const int sfin = c.j + c.delta;
            want = !(c.mode == CG_SH_SINGLE && (sfin < 0 || sfin >= p.nr));
          }
        }
        /* nothing to append (a chunk outside the shells' radial range, about
         * half of them): skip the bucket reservation */
        const unsigned om = __ballot_sync(FULL, open);
        if (om) {
          if (lane == 0) L.open[(row - rbeg) * nch + ch] = om;
          any_late = 1u;
        }
        if (!__any_sync(FULL, want)) continue;
        /* append to the rooms: one atomic per counter present in the warp,
         * issued together by each counter's first lane (one round trip) */
        int ct = -1;
        if (want) ct = counter_of(c.j, cg_corner_polar(z0, r2), cg_cell_class(&A, &c, x0, y0, z0));
        const unsigned same = __match_any_sync(FULL, ct);
        const int leader = __ffs(same) - 1;
        unsigned long long old = 0;
        if (want && lane == leader) old = atomicAdd(&p.cnt[(size_t)ct * CG_IMAP_CNT], (unsigned long long)__popc(same));
        old = __shfl_sync(FULL, old, leader);
        bool over = false;
        if (want) {
          const long long k = (long long)old + __popc(same & ((1u << lane) - 1u));
          over = k >= p.cap[ct];
          if (!over) p.recs[slot_of(p, ct, k)] = pack(ix, iy, iz, c, (unsigned)c.mode | ((unsigned)(c.delta + 1) << 2));
        }
        const unsigned vm = __ballot_sync(FULL, over);
        if (vm) {
          if (lane == 0) L.over[(row - rbeg) * nch + ch] = vm;
          any_late = 1u;
        }
      }
    }
    if (any_late) late_cells<K>(dens, p, L, rbeg, rend, lane);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) drawn += __shfl_xor_sync(FULL, drawn, o);
  if (lane == 0 && drawn) atomicAdd(&p.ctr[2], drawn);
}

/* Work units of a bucket of nsub ns: whole cells for ns <= 4 (8 to 64
 * samples), one slab of a cell for ns <= 32 (ns^2 samples), one line beyond;
 * each lane of a warp walks one unit. */
__host__ __device__ __forceinline__ long long units_per_cell(int ns)
{
  return ns <= 4 ? 1 : (ns <= 32 ? ns : (long long)ns * ns);
}

/* Unit groups of 32 per chunk so that a chunk is about CHS samples per lane
 * count: G = max(1, CHS / (32 x samples per unit)). */
__host__ __device__ __forceinline__ int groups_per_chunk(int ns)
{
  const int su = ns <= 4 ? ns * ns * ns : (ns <= 32 ? ns * ns : ns); /* samples per unit */
  const int g = CHS / (32 * su);
  return g > 1 ? g : 1;
}

/* Chunks of every bucket, 32 G units each, and their running sum: one block,
 * a bucket per thread. */
__global__ void __launch_bounds__(1024) k_imap_chunks(cg_imap_params p)
{
  __shared__ unsigned long long ws[33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned long long carry = 0;
  for (int b0 = 0; b0 < p.nbk; b0 += 1024) {
    const int b = b0 + threadIdx.x;
    unsigned long long x = 0;
    if (b < p.nbk) {
      const int ns = p.a.nsub[b / CG_IMAP_CLASSES];
      const longlong2 B = bucket_of(p, b);
      p.buckets[b] = B;
      const unsigned long long nu = (unsigned long long)B.y * (unsigned long long)units_per_cell(ns);
      const unsigned long long per = 32ull * (unsigned long long)groups_per_chunk(ns);
      x = (nu + per - 1) / per;
    }
    unsigned long long inc = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long t = __shfl_up_sync(FULL, inc, o);
      if (lane >= o) inc += t;
    }
    if (lane == 31) ws[w] = inc;
    __syncthreads();
    if (w == 0) {
      const unsigned long long y = ws[lane];
      unsigned long long yi = y;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long t = __shfl_up_sync(FULL, yi, o);
        if (lane >= o) yi += t;
      }
      ws[lane] = yi - y;
      if (lane == 31) ws[32] = yi;
    }
    __syncthreads();
    if (b < p.nbk) p.chunk_off[b] = carry + ws[w] + inc - x;
    carry += ws[32];
    __syncthreads();
  }
  if (threadIdx.x == 0) p.chunk_off[p.nbk] = carry;
}

/* One sample for the double pass, queued on its own. */
__device__ __noinline__ void queue_one(const cg_imap_params &p, long long rec, int q)
{
  const unsigned long long k = atomicAdd(&p.ctr[4], 1ull);
  if ((long long)k < p.queue_cap) p.queue[k] = ((unsigned long long)rec << 30) | (unsigned long long)q;
  else atomicOr(p.err, ERR_IMAP_QUEUE);
}

/* This warp's queue stage in the painting kernel's shared memory: QB entries
 * and their number. */
struct Stage {
  unsigned long long *e;
  int *n;
};

__device__ __forceinline__ Stage stage_of(const cg_imap_params &p)
{
  extern __shared__ __align__(16) unsigned char sraw[];
  unsigned char *b = sraw + paint_stage_off(p.nr, p.nbk);
  const int w = threadIdx.x >> 5;
  return Stage{reinterpret_cast<unsigned long long *>(b) + (size_t)w * QB,
               reinterpret_cast<int *>(b + (size_t)IW * QB * 8) + w};
}

/* One sample for the double pass: staged per warp, or queued at once when the
 * stage is full. */
__device__ __noinline__ void hold(const cg_imap_params &p, long long rec, int q)
{
  const Stage S = stage_of(p);
  const int k = atomicAdd(S.n, 1);
  if (k < QB) S.e[k] = ((unsigned long long)rec << 30) | (unsigned long long)q;
  else queue_one(p, rec, q);
}

/* The warp's stage to the queue, with one atomic, once it holds min_n.  One
 * lane reads the count and the exchange hands it on: the lanes take the same
 * way out, and none goes on to its next unit, where hold() raises the count,
 * before it has been read. */
__device__ __forceinline__ void queue_flush(const cg_imap_params &p, int min_n, int lane)
{
  const Stage S = stage_of(p);
  __syncwarp();
  int qn = 0;
  if (lane == 0) qn = *S.n;
  qn = __shfl_sync(FULL, qn, 0);
  if (qn > QB) qn = QB;
  if (qn < min_n) return;
  unsigned long long q0 = 0;
  if (lane == 0) q0 = atomicAdd(&p.ctr[4], (unsigned long long)qn);
  q0 = __shfl_sync(FULL, q0, 0);
  for (int i = lane; i < qn; i += 32) {
    if ((long long)(q0 + i) < p.queue_cap) p.queue[q0 + i] = S.e[i];
    else atomicOr(p.err, ERR_IMAP_QUEUE);
  }
  __syncwarp();
  if (lane == 0) *S.n = 0;
  __syncwarp();
}

/* Add a run of cnt samples of brightness temp to key k. */
template <typename K>
__device__ __forceinline__ void flush(const cg_imap_params &p, K k, float cnt, float temp)
{
  if (cnt > 0.0f) add_to(p, (long long)k, CG_MUL(temp, cnt), cnt);
}

/* What a lane carries through a unit: the pixel it is on and its run there.
 * (A second run slot saves a third of the reductions but costs more in
 * instructions: 67.0 against 61.7 ms of the stage at 1024^3.) */
template <typename K>
struct Lane {
  K k;
  float n; /* exact: a unit has at most 1024 samples */
};

/* One two-float reduction where c holds. */
__device__ __forceinline__ void red_if(bool c, float2 *a, float t, float n)
{
  asm volatile("{\n.reg .pred q;\nsetp.ne.u32 q, %0, 0;\n@q red.relaxed.gpu.global.add.v2.f32 [%1], {%2, %3};\n}" ::"r"(
                   (unsigned)c),
               "l"(a), "f"(t), "f"(n)
               : "memory");
}

/* A sample on key (ok), or one to hold, of index q0 + step floor(fi): another
 * key than the run's sends the run to the maps.  With packed sums (P) without a
 * branch but the rare one: some lane of a warp changes its pixel at nearly
 * every sample. */
template <typename K, bool P>
__device__ __forceinline__ void hit(const cg_imap_params &p, Lane<K> &L, K key, bool ok, float temp, long long rec,
                                    int q0, int step, float fi)
{
  const bool change = ok && key != L.k;
  if (P) {
    red_if(change && L.n > 0.0f, p.acc + L.k, CG_MUL(temp, L.n), L.n);
  } else if (change) {
    flush<K>(p, L.k, L.n, temp);
  }
  L.k = change ? key : L.k;
  L.n = change ? 1.0f : CG_ADD(L.n, 1.0f);
  if (!ok) {
    L.n = CG_SUB(L.n, 1.0f); /* exact */
    hold(p, rec, q0 + step * (int)fi);
  }
}

/* One axis of a cell: its corner as a float pair. */
struct Axis {
  float c, l;
};
__device__ __forceinline__ float at(const Axis &a, float half, float dxs) { return CG_ADD(a.c, CG_FMA(half, dxs, a.l)); }

/* A unit's samples, in rows along x, in the general form. */
template <typename K, bool P>
__device__ __forceinline__ void walk_general(const cg_imap_params &p, const cg_imap_args &A, const cg_imap_cell &c,
                                             int dbl, long long rec, const Axis &ax, const Axis &ay, const Axis &az,
                                             float dxs, int ns, int z0, int z1, int y0, int y1, Lane<K> &L)
{
  const float fns = (float)ns;
  for (int sz = z0; sz < z1; sz++) {
    const float z = at(az, CG_ADD((float)sz, 0.5f), dxs);
    for (int sy = y0; sy < y1; sy++) {
      const float y = at(ay, CG_ADD((float)sy, 0.5f), dxs);
#pragma unroll 1
      for (float fi = 0.5f; fi < fns; fi = CG_ADD(fi, 1.0f)) {
        int s = -1;
        long long pix = 0;
        const bool ok = !dbl && cg_imap_decide(&A, &c, at(ax, fi, dxs), y, z, &s, &pix);
        const K key = key_of<K>(p, s, pix);
        if (!ok || key != empty_key<K>()) hit<K, P>(p, L, key, ok, c.temp, rec, ns * (sy + ns * sz), 1, fi);
      }
    }
  }
}

/* The same for a cell of one octant, region and shell or edge
 * (cg_imap_fast_cell), along the axis nearest the line of sight, on which
 * consecutive samples keep their pixel longest: z in the polar caps, where the
 * octant angle is then the line's, the larger of x and y elsewhere.  Ranges
 * [o0, o1) and [m0, m1) of the outer and the middle axis. */
template <typename K, bool P, bool EQ>
__device__ __forceinline__ void walk_fast(const cg_imap_params &p, const cg_imap_fast &F, float temp, long long rec,
                                          const Axis &x, const Axis &y, const Axis &z, float dxs, int ns, int o0, int o1,
                                          int m0, int m1, float thr, Lane<K> &L)
{
  const int nside = p.a.nside;
  const K b0 = (K)F.s0 * (K)p.npix, b1 = (K)F.s1 * (K)p.npix;
  const float fns = (float)ns;
  Axis u, v;
  u.c = F.ymaj ? y.c : x.c;
  u.l = F.ymaj ? y.l : x.l;
  v.c = F.ymaj ? x.c : y.c;
  v.l = F.ymaj ? x.l : y.l;
  const int su = F.ymaj ? ns : 1, sv = F.ymaj ? 1 : ns, sz = ns * ns; /* strides of the sample index */
  for (int o = o0; o < o1; o++) {
    const float fo = CG_ADD((float)o, 0.5f);
    for (int m = m0; m < m1; m++) {
      const float fm = CG_ADD((float)m, 0.5f);
      const int q0 = EQ ? o * sz + m * sv : o * sv + m * su;
      if (EQ) {
        const float zs = at(z, fo, dxs), vs = at(v, fm, dxs);
        const float vz2 = CG_FMA(zs, zs, CG_MUL(vs, vs));
#pragma unroll 2
        for (float fi = 0.5f; fi < fns; fi = CG_ADD(fi, 1.0f)) {
          int up, pix;
          const bool ok = cg_fast_eq(&F, nside, thr, at(u, fi, dxs), vs, zs, vz2, &up, &pix);
          hit<K, P>(p, L, (up ? b1 : b0) + (K)pix, ok, temp, rec, q0, su, fi);
        }
      } else {
        const cg_fast_line l = cg_fast_polar_line(&F, nside, at(u, fm, dxs), at(v, fo, dxs));
#pragma unroll 2
        for (float fi = 0.5f; fi < fns; fi = CG_ADD(fi, 1.0f)) {
          int up, pix;
          const bool ok = cg_fast_polar(&F, &l, thr, at(z, fi, dxs), &up, &pix);
          hit<K, P>(p, L, (up ? b1 : b0) + (K)pix, ok, temp, rec, q0, sz, fi);
        }
      }
    }
  }
}

/* The G unit groups of one chunk of bucket b (nsub ns).  Each lane walks one
 * unit (a cell, a slab or a line) sample by sample.  The samples that only
 * double can decide are staged per warp in shared memory and queued in
 * batches. */
template <typename K, bool P>
__device__ __forceinline__ void paint_chunk(const cg_imap_params &p, const cg_imap_args &A, int b, int ns,
                                            unsigned long long u0, int G, unsigned long long nu, float dxs, int lane)
{
  const int U = (int)units_per_cell(ns);
  /* the chunk's first unit as (record, unit within it); later units are
   * within 32 G of it, so their offsets divide in 32 bits */
  const long long r0 = (long long)(u0 / (unsigned long long)U);
  const unsigned w0 = (unsigned)(u0 - (unsigned long long)r0 * (unsigned long long)U);
  for (int g = 0; g < G; g++) {
    const unsigned long long u = u0 + (unsigned long long)g * 32ull + (unsigned long long)lane;
    const bool valid = u < nu;
    /* the unit: record and its ranges of the outer and the middle axis */
    long long rl = 0;
    int o0 = 0, o1 = ns, m0 = 0, m1 = ns;
    if (valid) {
      if (U == 1) {
        rl = (long long)u;
      } else {
        const unsigned t = w0 + (unsigned)(g * 32 + lane);
        const unsigned dr = t / (unsigned)U;
        const int w = (int)(t - dr * (unsigned)U);
        rl = r0 + (long long)dr;
        if (ns <= 32) {
          o0 = w;
          o1 = w + 1;
        } else {
          o0 = w / ns;
          o1 = o0 + 1;
          m0 = w - o0 * ns;
          m1 = m0 + 1;
        }
      }
    }
    const long long rec = p.buckets[b].x + rl;
    float temp = 0.0f;
    Lane<K> L;
    L.k = empty_key<K>();
    L.n = 0.0f;
    if (valid) {
      int ix, iy, iz, dbl;
      const cg_imap_cell c = unpack(p.recs[rec], b / CG_IMAP_CLASSES - 1, &ix, &iy, &iz, &dbl);
      dbl |= p.force_double;
      temp = c.temp;
      const Axis x = {A.xc[ix], A.xl[ix]}, y = {A.yc[iy], A.yl[iy]}, z = {A.zc[iz], A.zl[iz]};
      /* the bucket's class: one loop for the whole warp */
      const int cls = dbl ? CG_CELL_GENERAL : b % CG_IMAP_CLASSES;
      if (cls == CG_CELL_GENERAL) {
        walk_general<K, P>(p, A, c, dbl, rec, x, y, z, dxs, ns, o0, o1, m0, m1, L);
      } else {
        cg_imap_fast F;
        cg_imap_fast_cell(&A, &c, cls, x.c, y.c, z.c, &F);
        if (cls == CG_CELL_EQ)
          walk_fast<K, P, true>(p, F, temp, rec, x, y, z, dxs, ns, o0, o1, m0, m1, cg_fast_eq_thr(A.nside), L);
        else
          walk_fast<K, P, false>(p, F, temp, rec, x, y, z, dxs, ns, o0, o1, m0, m1, cg_fast_polar_k0(A.nside), L);
      }
      flush<K>(p, L.k, L.n, temp);
    }
    queue_flush(p, QB / 2, lane);
  }
}

/* Warps take chunks in bucket order; paint_chunk paints one.  7 blocks per SM
 * with the samples two at a time: 5, 6 and 8 took 51.4, 48.6 and 49.0 against
 * 47.8 ms of the stage at 1024^3; one, three and four at a time 48.6, 47.9 and
 * 48.0. */
template <typename K, bool P>
__global__ void __launch_bounds__(IW * 32, 7) k_imap_paint(const __grid_constant__ cg_imap_params p)
{
  extern __shared__ __align__(16) unsigned char sraw[];
  const Sh sh = load_shells(p, sraw, true);
  __syncthreads();
  const cg_imap_args A = args_with(p, sh);
  const int lane = threadIdx.x & 31;
  const unsigned long long total = sh.chunk_off[p.nbk];
  if (lane == 0) *stage_of(p).n = 0;
  __syncwarp();
  for (;;) {
    unsigned long long ck = 0;
    if (lane == 0) ck = atomicAdd(&p.ctr[0], 1ull);
    ck = __shfl_sync(FULL, ck, 0);
    if (ck >= total) break;
    /* the bucket: last b with chunk_off[b] <= ck */
    int lo = 0, hi = p.nbk - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (sh.chunk_off[mid] <= ck) lo = mid;
      else hi = mid - 1;
    }
    const int b = lo;
    const int ns = sh.nsub[b / CG_IMAP_CLASSES];
    const unsigned long long nu = (unsigned long long)p.buckets[b].y * (unsigned long long)units_per_cell(ns);
    const int G = groups_per_chunk(ns);
    const float dxs = sh.dxs[b / CG_IMAP_CLASSES];
    const unsigned long long u0 = (ck - sh.chunk_off[b]) * 32ull * (unsigned long long)G;
    paint_chunk<K, P>(p, A, b, ns, u0, G, nu, dxs, lane);
  }
  queue_flush(p, 1, lane);
}

/* The samples of one warp batch (n <= 32 entries of the queue's form) in
 * double: the cell's radial shift (imap.c:196-198), taken by the first lane
 * of each run of one record and handed to the rest of the run, then the
 * sample's shell and pixel (imap.c:210-231). */
__device__ __forceinline__ void double_batch(const float *__restrict__ phi, const cg_imap_params &p,
                                             const cg_imap_args &A, const Sh &sh, const long long *sbase,
                                             unsigned long long e, bool valid, int lane)
{
  const long long rec = (long long)(e >> 30);
  const int q = (int)(e & ((1ull << 30) - 1));
  const long long prev = __shfl_up_sync(FULL, rec, 1);
  const bool lead = valid && (lane == 0 || prev != rec);
  const unsigned lm = __ballot_sync(FULL, lead);
  const unsigned le = lm & (lane == 31 ? FULL : ((2u << lane) - 1u));
  const int src = valid ? 31 - __clz(le) : lane;
  int lo = 0, ix = 0, iy = 0, iz = 0;
  float temp = 0.0f;
  double drr = 0;
  if (lead) {
    /* the record's shell: the last whose rooms begin at or before it */
    int hi = p.nr + 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (sbase[mid] <= rec) lo = mid;
      else hi = mid - 1;
    }
    int dbl;
    const cg_imap_cell c = unpack(p.recs[rec], lo - 1, &ix, &iy, &iz, &dbl);
    temp = c.temp;
    float v[3];
    grad_phi(phi, ix, iy, iz, p.box.N, v);
    int j;
    cgx_imap_cell(&A, ix, iy, iz, v, &j, &drr);
  }
  lo = __shfl_sync(FULL, lo, src);
  ix = __shfl_sync(FULL, ix, src);
  iy = __shfl_sync(FULL, iy, src);
  iz = __shfl_sync(FULL, iz, src);
  temp = __shfl_sync(FULL, temp, src);
  drr = __shfl_sync(FULL, drr, src);
  if (!valid) return;
  const int ns = sh.nsub[lo];
  int s = -1, sx, sy, sz;
  sub_of(q, ns, &sx, &sy, &sz);
  long long pix = 0;
  cgx_imap_sample(&A, ix, iy, iz, ns, drr, sx, sy, sz, &s, &pix);
  if (s >= 0 && s < p.nr) add_to(p, (long long)s * p.npix + pix, temp, 1.0f);
}

constexpr int DB_WARPS = 8; /* warps per block of k_imap_double */

/* The queued samples: first again in float-float (cg_imap_decide_ff), which
 * settles all but ~1e-9 of the pixels the float margins left open; the rest
 * -- shells within the float radial shift's bound of an edge, and every
 * sample of a cell listed in double -- are gathered per warp in shared
 * memory and decided in double 32 at a time, so that the FP64 work runs in
 * full warps. */
__global__ void __launch_bounds__(DB_WARPS * 32) k_imap_double(const float *__restrict__ phi, cg_imap_params p)
{
  extern __shared__ __align__(16) unsigned char sraw[];
  const Sh sh = load_shells(p, sraw, false);
  long long *sbase = reinterpret_cast<long long *>(sh.chunk_off); /* the shells' first records */
  for (int i = threadIdx.x; i < p.nr + 2; i += blockDim.x) sbase[i] = p.at[4 * i + 1];
  __syncthreads();
  const cg_imap_args A = args_with(p, sh);
  unsigned long long *db = reinterpret_cast<unsigned long long *>(sraw + double_stage_off(p.nr, p.nbk)) +
                           (size_t)(threadIdx.x >> 5) * 64;
  const unsigned long long nq0 = p.ctr[4];
  const long long nq = (long long)nq0 < p.queue_cap ? (long long)nq0 : p.queue_cap;
  const int lane = threadIdx.x & 31;
  const long long stride = (long long)gridDim.x * blockDim.x;
  int dn = 0; /* entries gathered for double (warp-uniform) */
  unsigned long long ndbl = 0;
  for (long long kb = (long long)blockIdx.x * blockDim.x + threadIdx.x - lane; kb < nq; kb += stride) {
    const long long k = kb + lane;
    const bool valid = k < nq;
    const unsigned long long e = valid ? p.queue[k] : ~0ull;
    bool need = valid;
    if (valid && !p.force_double) {
      const long long rec = (long long)(e >> 30);
      const int q = (int)(e & ((1ull << 30) - 1));
      int lo = 0, hi = p.nr + 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (sbase[mid] <= rec) lo = mid;
        else hi = mid - 1;
      }
      int ix, iy, iz, dbl;
      const cg_imap_cell c = unpack(p.recs[rec], lo - 1, &ix, &iy, &iz, &dbl);
      if (!dbl) {
        const int ns = sh.nsub[lo];
        int s = -1, sx, sy, sz;
        long long pix = 0;
        sub_of(q, ns, &sx, &sy, &sz);
        if (cg_imap_decide_ff(&A, &c, ix, iy, iz, sx, sy, sz, &s, &pix)) {
          need = false;
          if (s >= 0 && s < p.nr) add_to(p, (long long)s * p.npix + pix, c.temp, 1.0f);
        }
      }
    }
    const unsigned nm = __ballot_sync(FULL, need);
    if (!nm) continue;
    if (need) db[dn + __popc(nm & ((1u << lane) - 1u))] = e;
    dn += __popc(nm);
    ndbl += lane == 0 ? (unsigned long long)__popc(nm) : 0ull;
    __syncwarp();
    if (dn >= 32) {
      double_batch(phi, p, A, sh, sbase, db[lane], true, lane);
      __syncwarp();
      if (lane < dn - 32) db[lane] = db[lane + 32];
      dn -= 32;
      __syncwarp();
    }
  }
  if (dn > 0) double_batch(phi, p, A, sh, sbase, lane < dn ? db[lane] : ~0ull, lane < dn, lane);
  if (ndbl) atomicAdd(p.xstats + 3, ndbl);
}

template <typename K>
cudaError_t launch(cudaStream_t s, const float *dens, const float *phi, const cg_imap_params *p, int nsm)
{
  cudaError_t e = cudaMemsetAsync(p->ctr, 0, 5 * sizeof(unsigned long long), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(p->cnt, 0, (size_t)4 * (p->nr + 2) * CG_IMAP_CNT * sizeof(unsigned long long), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(p->seg + p->a.na - 1, 0, sizeof(cg_imap_seg), s);
  if (e != cudaSuccess) return e;
  const size_t sm_list = shell_smem(p->nr, p->nbk, false), sm_paint = paint_smem(p->nr, p->nbk);
  const size_t sm_double = double_stage_off(p->nr, p->nbk) + (size_t)DB_WARPS * 64 * 8;
  auto paint = p->packed ? k_imap_paint<K, true> : k_imap_paint<K, false>;
  if ((e = cudaFuncSetAttribute(k_imap_list<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_list)) ||
      (e = cudaFuncSetAttribute(paint, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_paint)) ||
      (e = cudaFuncSetAttribute(k_imap_double, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_double)))
    return e;
  int per_sm = 0;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_imap_list<K>, IW * 32, sm_list))) return e;
  const long long nrow = (long long)p->box.N * p->box.N;
  long long blocks = (nrow + IW * ROWS - 1) / (IW * ROWS);
  if (blocks > (long long)nsm * (per_sm > 0 ? per_sm : 1)) blocks = (long long)nsm * (per_sm > 0 ? per_sm : 1);
  k_imap_tab<<<(unsigned)((p->a.na + 31) / 32), 32, 0, s>>>(*p);
  k_imap_list<K><<<(unsigned)blocks, IW * 32, sm_list, s>>>(dens, phi, *p);
  k_imap_chunks<<<1, 1024, 0, s>>>(*p);
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, paint, IW * 32, sm_paint))) return e;
  paint<<<(unsigned)(nsm * (per_sm > 0 ? per_sm : 1)), IW * 32, sm_paint, s>>>(*p);
  k_imap_double<<<(unsigned)(nsm * 4), DB_WARPS * 32, sm_double, s>>>(phi, *p);
  return cudaGetLastError();
}

/* RING pixels of float directions by the margin-checked single-precision
 * decision, on the device. */
__global__ void k_pix_checked(int nside, const float *__restrict__ xyz, long long n, float ein, long long *pix)
{
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    cg_dir d = cg_dir_of(xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2], 0.0f);
    d.ecth = CG_FMA(2.0f, ein, d.ecth);
    pix[i] = cg_pix_checked(&d, nside, ein);
  }
}

} /* namespace */

cudaError_t cg_pix_checked_dev(cudaStream_t s, int nside, const float *xyz, long long n, float ein, long long *pix,
                               int nsm)
{
  long long blocks = (n + 255) / 256;
  if (blocks > (long long)nsm * 8) blocks = (long long)nsm * 8;
  if (blocks < 1) blocks = 1;
  k_pix_checked<<<(unsigned)blocks, 256, 0, s>>>(nside, xyz, n, ein, pix);
  return cudaGetLastError();
}

size_t cg_imap_shell_smem(int nr, int nbk) { return paint_smem(nr, nbk); }

cudaError_t cg_imap_paint(cudaStream_t s, const float *dens, const float *phi, const cg_imap_params *p, int nsm)
{
  if (!p->ctr || !p->recs || !p->queue) return cudaErrorInvalidValue;
  /* 32-bit keys when every (shell, pixel) index and the empty key fit */
  if ((unsigned long long)p->nr * (unsigned long long)p->npix < 0xffffffffull)
    return launch<unsigned int>(s, dens, phi, p, nsm);
  return launch<unsigned long long>(s, dens, phi, p, nsm);
}
