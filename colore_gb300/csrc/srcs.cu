/*
 * srcs.cu -- biased Poisson sources (srcs.c:120-283), their local
 * properties (srcs.c:386-416), the source count map, and the line-of-sight
 * redshift-space distortion at each source (srcs.c:425-504, 634-662).
 *
 * Sampling is count -> scan -> emit:
 *   k_pois_tab   : n(r) norm(r) and b(r) per table segment, with bounds.
 *   k_pois_count : per cell lambda and a Poisson deviate keyed by (seed,
 *                  population, cell), so the result does not depend on the
 *                  launch shape; counts are kept as uint16 and the totals of
 *                  every 2048 consecutive cells summed up.  A cell with
 *                  CG_COUNT_ESC or more sources stores the escape value and
 *                  appends (cell, count) to a short overflow list.
 *   k_scan_*     : exclusive scan of the block totals (three coalesced passes).
 *   k_emit       : re-reads the counts, scans them inside the block and writes
 *                  every source at its final catalog index, in cell order (the
 *                  order of the reference run with one thread); the block's
 *                  sources are spread evenly over its threads, each finding
 *                  its cell by binary search on the scanned offsets.  Positions,
 *                  the NGP velocity (get_rvel, srcs.c:87-118), ra/dec/z, the
 *                  base-pixel id and the count-map increment are fused.
 *
 * Along the line of sight to each source (one thread per source, a warp for
 * the skewers):
 *   k_beam_rsd    : trilinear RSD at the source.
 *   k_src_lensing : shear, convergence and deflection from the nearest-cell
 *                   tidal tensor and potential gradient at N/2 radial steps.
 *   k_src_skewers : trilinear density (or Gaussian field) and radial velocity
 *                   at every step up to the source.
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include "cg_dev.cuh"
#include "srcs_api.h"

namespace {
using namespace cg;

constexpr int CPT = 8;                 /* cells per thread */
constexpr int SB = 256;                /* threads per block */
constexpr int CPB = CPT * SB;          /* cells per block   */

__device__ __forceinline__ void cell_of(long long c, const Box &b, int &ix, int &iy, int &iz)
{
  const long long q = divN(c, b), z = divN(q, b);
  ix = (int)(c - q * b.N);
  iy = (int)(q - z * b.N);
  iz = (int)z;
}

/* True count of a cell whose stored count is the escape value. */
__device__ __forceinline__ int ovf_lookup(const cg_srcs_params &p, long long cid)
{
  int n = *p.ovf_n;
  if (n > CG_OVF_CAP) n = CG_OVF_CAP;
  for (int k = 0; k < n; k++)
    if (p.ovf_cell[k] == cid) return p.ovf_cnt[k];
  return CG_COUNT_ESC;
}

/* The count of a cell that the float margins leave open: the reference's
 * double arithmetic (out of line: rare, and long). */
__device__ __noinline__ int count_double(const cg_srcs_params &p, int ix, int iy, int iz, float d, long long cid,
                                         uint32_t w)
{
  const double lam = cgx_lambda(&p.pa.x, ix, iy, iz, d);
  if (lam > 1073741824.0) {
    atomicOr(p.err, ERR_COUNT_OVERFLOW);
    return 0;
  }
  return cgx_poisson(lam, (double)cg_u01f(w), cid, p.kp0, p.kp1);
}

/* The table segments of the counts' first tier, from the double tables and
 * this realisation's normalisation; the overflow list and the block totals
 * are cleared along the way. */
__global__ void __launch_bounds__(32) k_pois_tab(cg_srcs_params p, long long nb)
{
  const long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x, st = (long long)gridDim.x * blockDim.x;
  for (long long i = i0; i < CG_NA - 1; i += st) p.seg[i] = cg_pois_seg_make(&p.pa.x, CG_NA, (int)i);
  for (long long i = i0; i < nb; i += st) p.block_sums[i] = 0;
  if (i0 == 0) *p.ovf_n = 0;
}

/* A cell that the segment tables leave open: lambda with the per-lookup
 * bounds (cg_lambda_checked), then inversion or PTRS in single precision
 * where its margins allow, else double (bit 31 set).  Out of line: a few
 * cells in 10^4, and the cells with lambda >= 10. */
__device__ __noinline__ unsigned int count_open(const cg_srcs_params &p, const float *__restrict__ grid, long long cid)
{
  int ix, iy, iz;
  cell_of(cid, p.box, ix, iy, iz);
  const float d = __ldg(grid + pidx(ix, iy, iz, p.box.N));
  float lam, elam;
  int st = cg_lambda_checked(&p.pa, ix, iy, iz, d, &lam, &elam);
  if (p.force_double && (st == 1 || st == 3)) st = 2;
  if (st == 0) return 0;
  const uint32_t w = cg_pois_word(cid, p.kp0, p.kp1);
  int n = st == 1 ? cg_poisson_inv_checked(lam, elam, cg_u01f(w))
                  : (st == 3 ? cg_poisson_ptrs_checked(lam, elam, cid, p.kp0, p.kp1) : -1);
  if (n < 0) return (unsigned int)count_double(p, ix, iy, iz, d, cid, w) | 0x80000000u;
  return (unsigned int)n;
}

/* PTRS of a cell whose lambda >= 10 is certain (cells next to the observer,
 * dense coarse grids), out of line like the double path. */
__device__ __noinline__ int ptrs_float(float lam, float elam, long long cid, uint32_t k0, uint32_t k1)
{
  return cg_poisson_ptrs_checked(lam, elam, cid, k0, k1);
}

constexpr int CWN = 4;  /* warps per block of the count */
constexpr int CW = 128; /* cells per warp and step: four neighbours per lane */

/* A warp's cells in shared memory: from the front those to be inverted
 * (lambda, its bound, and the uniform's 24 bits with the cell's place above
 * them), from the back those for PTRS (the same without a uniform); those
 * left open by the segment tables; and the counts. */
struct alignas(16) CountWarp {
  float lam[CW], elam[CW];
  unsigned int uc[CW];
  unsigned char open[CW];
  unsigned short cnt[CW];
};

/* Counts, 128 cells per warp and step, `steps` consecutive steps per warp.
 * First tier: a lane forms lambda of four neighbouring cells of a row from
 * the segment tables (cg_lambda_seg: two 16-byte loads and about 40
 * instructions a cell), draws their Philox block when one may hold a source,
 * and settles u < 1 - lambda on the spot.  The cells left are compacted per
 * warp in shared memory and inverted (lambda < 10) or sampled by PTRS 32 at a
 * time, so that the exponential and the search run in full warps (inverted in
 * place, every warp paid for both in every step: 261 thread-instructions per
 * cell at 512^3, now 148).  Cells that the tier's bounds leave open follow in a last
 * list (count_open); every count is the reference's double decision.  Each
 * warp adds its total to the entry of its 2048 cells.  Twelve blocks per SM
 * (40 registers).  1024^3, 1000 sources per deg^2: 11.0 -> 5.3 ms; 512^3, two
 * populations: 3.04 -> 1.42 ms. */
__global__ void __launch_bounds__(CWN * 32, 12) k_pois_count(const float *__restrict__ grid, cg_srcs_params p, int steps)
{
  __shared__ CountWarp sw[CWN];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const unsigned int below = (1u << lane) - 1u;
  CountWarp &S = sw[wid];
  const int N = p.box.N;
  float rlo, rhi;
  cg_tier_limits(&p.pa, &rlo, &rhi);
  long long tot = 0;
  unsigned int nfb = 0;
  const long long wbase = ((long long)blockIdx.x * CWN + wid) * steps * CW;
#pragma unroll 1
  for (int step = 0; step < steps; step++) {
    const long long w0 = wbase + step * CW;
    const long long c0 = w0 + 4 * lane;
    int ix, iy, iz;
    cell_of(c0, p.box, ix, iy, iz);
    float lam[4], elam[4];
    /* per cell: left open, may hold a source, proper for inversion or PTRS */
    unsigned int open = 0u, may = 0u, inv = 0u, ptr = 0u;
    if (p.force_double) {
      open = 0xfu;
    } else {
      /* rows start at an even float (8-byte aligned), ix is a multiple of 4 */
      const float2 *row = reinterpret_cast<const float2 *>(grid + pidx(ix, iy, iz, N));
      const float2 da = __ldg(row), db = __ldg(row + 1);
      const float4 x4 = __ldg(reinterpret_cast<const float4 *>(p.pa.xc + ix));
      const float d4[4] = {da.x, da.y, db.x, db.y}, xs[4] = {x4.x, x4.y, x4.z, x4.w};
      const float y = __ldg(p.pa.yc + iy), z = __ldg(p.pa.zc + iz);
      const float yz2 = CG_FMA(z, z, CG_MUL(y, y));
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const float r2 = CG_FMA(xs[q], xs[q], yz2);
        float r;
        const float s = cg_seg_pos(r2, p.pa.idr, &r);
        lam[q] = elam[q] = 0.0f;
        if (r > rhi) continue;
        if (!cg_tier_inside(r2, r, rlo)) {
          open |= 1u << q;
          continue;
        }
        const int i = (int)s;
        const float4 *g4 = reinterpret_cast<const float4 *>(p.seg + i);
        const float4 ga = __ldg(g4), gb = __ldg(g4 + 1);
        const cg_pois_seg g = {ga.x, ga.y, ga.z, ga.w, gb.x, gb.y, gb.z, 0.0f};
        int pos;
        lam[q] = cg_lambda_seg(&g, CG_SUB(s, (float)i), d4[q], p.pa.bias_model, &elam[q], &pos);
        const int t = cg_tier_lambda(lam[q], elam[q], pos);
        if (t & CG_TIER_MAY) may |= 1u << q;
        if (t & CG_TIER_INV) inv |= 1u << q;
        if (t & CG_TIER_PTRS) ptr |= 1u << q;
      }
    }
    unsigned int u24[4] = {0u, 0u, 0u, 0u};
    if (may & ~ptr) {
      const unsigned long long m = (unsigned long long)c0 >> 2;
      const cg_u32x4 w = cg_philox4x32_10((uint32_t)m, (uint32_t)(m >> 32), 0u, 0u, p.kp0, p.kp1);
#pragma unroll
      for (int q = 0; q < 4; q++) {
        u24[q] = w.v[q] >> 8;
        if (cg_tier_uniform(lam[q], elam[q], CG_MUL((float)u24[q], CG_E24))) may &= ~(1u << q);
      }
    }
    open |= may & ~(inv | ptr);
    inv &= may;
    *reinterpret_cast<uint2 *>(&S.cnt[4 * lane]) = make_uint2(0u, 0u);
    int na = 0, np = 0, no = 0;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const bool a = (inv >> q) & 1u;
      const unsigned int m = __ballot_sync(0xffffffffu, a);
      if (a) {
        const int k = na + __popc(m & below);
        S.lam[k] = lam[q];
        S.elam[k] = elam[q];
        S.uc[k] = u24[q] | ((unsigned int)(4 * lane + q) << 24);
      }
      na += __popc(m);
    }
    if (__any_sync(0xffffffffu, (open | ptr) != 0u)) {
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const bool o = (open >> q) & 1u, t = (ptr >> q) & 1u;
        const unsigned int m = __ballot_sync(0xffffffffu, o), mt = __ballot_sync(0xffffffffu, t);
        if (o) S.open[no + __popc(m & below)] = (unsigned char)(4 * lane + q);
        if (t) {
          const int k = CW - 1 - np - __popc(mt & below);
          S.lam[k] = lam[q];
          S.elam[k] = elam[q];
          S.uc[k] = (unsigned int)(4 * lane + q) << 24;
        }
        no += __popc(m);
        np += __popc(mt);
      }
    }
    __syncwarp();
    /* the inversions, then the PTRS cells */
#pragma unroll 1
    for (int k0 = 0; k0 < na; k0 += 32) {
      const int k = k0 + lane;
      int n = 0, c = 0;
      if (k < na) {
        const unsigned int uc = S.uc[k];
        c = (int)(uc >> 24);
        n = cg_poisson_inv_checked(S.lam[k], S.elam[k], CG_MUL((float)(uc & 0xffffffu), CG_E24));
        if (n > 0) S.cnt[c] = (unsigned short)n; /* below 64 */
      }
      const unsigned int m = __ballot_sync(0xffffffffu, n < 0);
      if (n < 0) S.open[no + __popc(m & below)] = (unsigned char)c;
      else tot += n;
      no += __popc(m);
    }
    if (np) {
#pragma unroll 1
      for (int k0 = 0; k0 < np; k0 += 32) {
        const int k = CW - 1 - k0 - lane;
        int n = 0, c = 0;
        if (k0 + lane < np) {
          c = (int)(S.uc[k] >> 24);
          n = ptrs_float(S.lam[k], S.elam[k], w0 + c, p.kp0, p.kp1);
          if (n >= CG_COUNT_ESC) n = -1; /* the overflow list is count_open's */
          if (n > 0) S.cnt[c] = (unsigned short)n;
        }
        const unsigned int m = __ballot_sync(0xffffffffu, n < 0);
        if (n < 0) S.open[no + __popc(m & below)] = (unsigned char)c;
        else tot += n;
        no += __popc(m);
      }
    }
    if (no) {
      __syncwarp();
#pragma unroll 1
      for (int k = lane; k < no; k += 32) {
        const int c = S.open[k];
        const unsigned int o1 = count_open(p, grid, w0 + c);
        const int n = (int)(o1 & 0x7fffffffu);
        nfb += o1 >> 31;
        tot += n;
        if (n >= CG_COUNT_ESC) {
          const int o = atomicAdd(p.ovf_n, 1);
          if (o < CG_OVF_CAP) {
            p.ovf_cell[o] = w0 + c;
            p.ovf_cnt[o] = n;
          } else {
            atomicOr(p.err, ERR_COUNT_OVERFLOW);
          }
        }
        S.cnt[c] = (unsigned short)(n < CG_COUNT_ESC ? n : CG_COUNT_ESC);
      }
    }
    __syncwarp();
    *reinterpret_cast<uint2 *>(p.counts + c0) = *reinterpret_cast<const uint2 *>(&S.cnt[4 * lane]);
    __syncwarp();
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    tot += __shfl_xor_sync(0xffffffffu, tot, o);
    nfb += __shfl_xor_sync(0xffffffffu, nfb, o);
  }
  if (lane == 0) {
    if (tot) atomicAdd(reinterpret_cast<unsigned long long *>(&p.block_sums[wbase / CPB]), (unsigned long long)tot);
    if (nfb) atomicAdd(p.xstats, (unsigned long long)nfb);
  }
}

/* Exclusive scan of the n block totals in place, their sum into *total, in
 * three coalesced passes over tiles of SCAN_T values (a thread holds two
 * neighbours): each tile reduced to its sum (tsum), the tile sums scanned by
 * one block, then every tile scanned from its offset.  (One block walking
 * the whole array took 0.87 ms at 1024^3.) */
constexpr int SCAN_T = 2048;

/* Exclusive scan of x over the block's 1024 threads; *tot = the block sum. */
__device__ __forceinline__ long long block_scan(long long x, long long *ws, long long *tot)
{
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  long long inc = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const long long t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) ws[w] = inc;
  __syncthreads();
  if (w == 0) {
    long long y = ws[lane], yi = y;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const long long t = __shfl_up_sync(0xffffffffu, yi, o);
      if (lane >= o) yi += t;
    }
    ws[lane] = yi - y;
    if (lane == 31) ws[32] = yi;
  }
  __syncthreads();
  const long long ex = ws[w] + inc - x;
  *tot = ws[32];
  __syncthreads(); /* ws is reused by the next call */
  return ex;
}

__global__ void __launch_bounds__(1024) k_scan_tiles(const long long *__restrict__ v, long long n, long long *tsum,
                                                     unsigned int *err)
{
  __shared__ long long ws[33];
  const long long i = (long long)blockIdx.x * SCAN_T + 2 * (long long)threadIdx.x;
  const long long a = i < n ? v[i] : 0, b = i + 1 < n ? v[i + 1] : 0;
  if (a > 0x7fffffffLL || b > 0x7fffffffLL) atomicOr(err, ERR_COUNT_OVERFLOW); /* k_emit scans a block in int */
  long long tot;
  block_scan(a + b, ws, &tot);
  if (threadIdx.x == 0) tsum[blockIdx.x] = tot;
}

__global__ void __launch_bounds__(1024) k_scan_top(long long *tsum, long long nt, long long *total)
{
  __shared__ long long ws[33];
  long long carry = 0;
  for (long long c0 = 0; c0 < nt; c0 += 1024) {
    const long long i = c0 + threadIdx.x;
    const long long x = i < nt ? tsum[i] : 0;
    long long tot;
    const long long ex = block_scan(x, ws, &tot);
    if (i < nt) tsum[i] = carry + ex;
    carry += tot;
  }
  if (threadIdx.x == 0) *total = carry;
}

/* Block i's offset to the host when it is one of every bpc-th. */
__device__ __forceinline__ void tell_offset(long long *host, long long bpc, long long i, long long off)
{
  if (host && i % bpc == 0) host[2 + i / bpc] = off;
}

__global__ void __launch_bounds__(1024) k_scan_apply(long long *v, long long n, const long long *__restrict__ tsum,
                                                     const long long *__restrict__ total, const unsigned int *err,
                                                     long long *host, long long bpc)
{
  __shared__ long long ws[33];
  const long long i = (long long)blockIdx.x * SCAN_T + 2 * (long long)threadIdx.x;
  const long long a = i < n ? v[i] : 0, b = i + 1 < n ? v[i + 1] : 0;
  long long tot;
  const long long off = tsum[blockIdx.x] + block_scan(a + b, ws, &tot);
  if (i < n) {
    v[i] = off;
    tell_offset(host, bpc, i, off);
  }
  if (i + 1 < n) {
    v[i + 1] = off + a;
    tell_offset(host, bpc, i + 1, off + a);
  }
  if (host && blockIdx.x == 0 && threadIdx.x == 0) {
    host[0] = *total;
    host[1] = (long long)*err;
  }
}

/* The whole scan in one block, for up to SCAN_ONE totals: three launches and
 * their gaps cost more than its few tiles (128^3: 4 us against 12). */
constexpr long long SCAN_ONE = 4 * SCAN_T;

__global__ void __launch_bounds__(1024) k_scan_one(long long *v, long long n, long long *total, unsigned int *err,
                                                   long long *host, long long bpc)
{
  __shared__ long long ws[33];
  long long carry = 0;
  bool big = false;
  for (long long t0 = 0; t0 < n; t0 += SCAN_T) {
    const long long i = t0 + 2 * (long long)threadIdx.x;
    const long long a = i < n ? v[i] : 0, b = i + 1 < n ? v[i + 1] : 0;
    big |= a > 0x7fffffffLL || b > 0x7fffffffLL; /* k_emit scans a block in int */
    long long tot;
    const long long off = carry + block_scan(a + b, ws, &tot);
    if (i < n) {
      v[i] = off;
      tell_offset(host, bpc, i, off);
    }
    if (i + 1 < n) {
      v[i + 1] = off + a;
      tell_offset(host, bpc, i + 1, off + a);
    }
    carry += tot;
  }
  if (big) atomicOr(err, ERR_COUNT_OVERFLOW);
  __syncthreads();
  if (threadIdx.x == 0) {
    *total = carry;
    if (host) {
      host[0] = carry;
      host[1] = (long long)atomicOr(err, 0u);
    }
  }
}

/* Centred potential differences at a cell (get_rvel / get_element VEL): the
 * cell's address once, its neighbours at periodic offsets. */
__device__ __forceinline__ void grad_phi(const float *__restrict__ phi, int ix, int iy, int iz, int N, float v[3])
{
  const int ngx = 2 * (N / 2 + 1), my = (N - 1) * ngx;
  const long long plane = (long long)ngx * N, mz = plane * (N - 1);
  const float *c = phi + pidx(ix, iy, iz, N);
  v[0] = CG_SUB(__ldg(c + (ix == N - 1 ? 1 - N : 1)), __ldg(c + (ix == 0 ? N - 1 : -1)));
  v[1] = CG_SUB(__ldg(c + (iy == N - 1 ? -my : ngx)), __ldg(c + (iy == 0 ? my : -ngx)));
  v[2] = CG_SUB(__ldg(c + (iz == N - 1 ? -mz : plane)), __ldg(c + (iz == 0 ? mz : -plane)));
}

/* Base and count-map pixels of a source by the reference's double
 * arithmetic (vec2pix_ring, srcs.c:268; he_ang2pix of cart2sph); returns the
 * number of pixels decided here.  Out of line: rare. */
__device__ __noinline__ unsigned int pixels_double(const cg_srcs_params &p, float px, float py, float pz, long long *pr,
                                                   long long *pc)
{
  unsigned int k = 0;
  if (*pr < 0) {
    *pr = cgx_vec2pix_ring(p.nside_base, (double)px, (double)py, (double)pz);
    k++;
  }
  if (p.cmap && *pc < 0) {
    double r, cth, ph;
    cgx_cart2sph((double)px, (double)py, (double)pz, &r, &cth, &ph);
    *pc = cgx_ang2pix(p.nside_count, cth, ph);
    k++;
  }
  return k;
}

constexpr int SRC_F = 9; /* floats per source record (Src) */

/* Sources of 2048 cells (block b0 + blockIdx.x of them), the share blockIdx.y of
 * gridDim.y, a power of two: every share scans the counts again, a few per cent
 * of the work, so that small grids and dense populations spread over the chip
 * (c1 at 128^3: 1024 blocks of up to 20000 sources kept the SMs busy 59 % of
 * the time).  The share's sources are spread evenly over the threads.  STAGED:
 * records of 36 bytes are staged per warp and written as consecutive words;
 * written field by field they cost L2 ten sectors per source for 56 bytes. */
template <bool STAGED>
__global__ void __launch_bounds__(SB, 6) k_emit(const float *__restrict__ phi, cg_srcs_params p, long long b0)
{
  __shared__ int coff[CPB]; /* exclusive source offset of each cell in the block */
  __shared__ int ws[SB / 32];
  __shared__ float stage[STAGED ? SB / 32 : 1][STAGED ? 32 * SRC_F : 1];
  const int N = p.box.N;
  const long long blk = b0 + blockIdx.x, cb = blk * CPB;
  const long long c0 = cb + (long long)threadIdx.x * CPT;
  int n[CPT];
  int tot = 0;
  {
    const uint4 pk = *reinterpret_cast<const uint4 *>(p.counts + c0);
    const unsigned w4[4] = {pk.x, pk.y, pk.z, pk.w};
#pragma unroll
    for (int h = 0; h < CPT; h++) {
      int v = (int)((w4[h >> 1] >> (16 * (h & 1))) & 0xffffu);
      if (v == CG_COUNT_ESC) v = ovf_lookup(p, c0 + h);
      n[h] = v;
      tot += v;
    }
  }
  /* block exclusive scan of per-thread totals */
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int inc = tot;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) ws[wid] = inc;
  __syncthreads();
  int woff = 0, T = 0;
#pragma unroll
  for (int w = 0; w < SB / 32; w++) {
    if (w < wid) woff += ws[w];
    T += ws[w];
  }
  if (T == 0) return;
  int run = woff + inc - tot;
#pragma unroll
  for (int h = 0; h < CPT; h++) {
    coff[threadIdx.x * CPT + h] = run;
    run += n[h];
  }
  __syncthreads();
  const long long base = p.block_sums[blk];
  const float dx = p.box.dx;
  /* the block's first cell; a cell lo < 2048 further on lies lo2 / N rows
   * below, lo2 = ix0 + lo < 4096, by a product in 32 bits (mdiv / 2^24 is
   * 1/N + e with e lo2 < 2^-12 < 1/N) */
  int bx, by, bz;
  cell_of(cb, p.box, bx, by, bz);
  const unsigned mdiv = ((1u << 24) + (unsigned)N - 1u) / (unsigned)N;
  unsigned int nfb = 0; /* pixels decided in double */
  const int lg = 31 - __clz((int)gridDim.y);
  const int k1 = (int)(((long long)T * (blockIdx.y + 1)) >> lg);
  for (int kb = (int)(((long long)T * blockIdx.y) >> lg) + wid * 32; kb < k1; kb += SB) {
    const int k = kb + lane;
    const long long id = base + k;
    const bool ok = k < k1 && id < p.capacity;
    if (k < k1 && !ok) atomicOr(p.err, ERR_CATALOG_OVERFLOW);
    float *q = STAGED ? &stage[wid][lane * SRC_F] : p.src + (size_t)id * SRC_F;
    if (ok) {
      /* the cell holding source k: the last cell whose offset is <= k (cells
       * without sources share their successor's offset) */
      int lo = 0;
#pragma unroll
      for (int st = CPB / 2; st > 0; st >>= 1)
        if (coff[lo + st] <= k) lo += st;
      const int j = k - coff[lo];
      const long long cid = cb + lo;
      const unsigned lo2 = (unsigned)(bx + lo), dr = (lo2 * mdiv) >> 24;
      const int ix = (int)(lo2 - dr * (unsigned)N);
      int iy = by + (int)dr, iz = bz;
      if (iy >= N) {
        iy -= N;
        iz++;
      }
      const float x0 = cg_cell_coord(ix, dx, p.box.p0);
      const float y0 = cg_cell_coord(iy, dx, p.box.p1), z0 = cg_cell_coord(iz, dx, p.box.p2);
      const float rr = cg_norm3(x0, y0, z0);
      float v[3];
      grad_phi(phi, ix, iy, iz, N, v);
      const float rvel = CG_MUL(p.factor_vel, cg_rvel(v[0], v[1], v[2], x0, y0, z0, rr, p.box.idx));
      const float dz_rsd = CG_MUL(rvel, bg(p.v1, p.g, rr));
      cg_u32x4 u = cg_philox4x32_10((uint32_t)cid, (uint32_t)(cid >> 32), (uint32_t)j, 0u, p.kq0, p.kq1);
      /* the position of the double arithmetic, stored as float (srcs.c:261-263):
       * in single precision where its rounding is certain, else in double */
      float px, py, pz;
      if (p.force_double || !cg_src_offset_checked(p.pa.xc[ix], p.cl[0][ix], p.dxh, p.dxl, u.v[0], &px))
        px = cgx_src_offset(cgx_coord(ix, p.dx64, p.p64[0]), p.dx64, u.v[0]);
      if (p.force_double || !cg_src_offset_checked(p.pa.yc[iy], p.cl[1][iy], p.dxh, p.dxl, u.v[1], &py))
        py = cgx_src_offset(cgx_coord(iy, p.dx64, p.p64[1]), p.dx64, u.v[1]);
      if (p.force_double || !cg_src_offset_checked(p.pa.zc[iz], p.cl[2][iz], p.dxh, p.dxl, u.v[2], &pz))
        pz = cgx_src_offset(cgx_coord(iz, p.dx64, p.p64[2]), p.dx64, u.v[2]);
      p.pos[id] = make_float4(px, py, pz, dz_rsd);
      /* the base pixel and the count-map pixel: the reference's double
       * decisions, in single precision where the margins allow */
      float ph;
      const cg_dir dr3 = cg_dir_phi(px, py, pz, &ph);
      long long pr = -1, pc = -1;
      if (!p.force_double) {
        pr = cg_pix_checked(&dr3, (int)p.nside_base, 0.0f);
        if (p.cmap) pc = cg_pix_checked(&dr3, (int)p.nside_count, 0.0f);
      }
      if (pr < 0 || (p.cmap && pc < 0)) nfb += pixels_double(p, px, py, pz, &pr, &pc);
      /* ring2nest costs several 64-bit divisions; nside_base is small, so its
       * table (built on the host with the same function) replaces them */
      p.ipix[id] = p.base_r2n ? __ldg(p.base_r2n + pr) : (int)cg_ring2nest(p.nside_base, pr);
      if (p.cmap) atomicAdd(&p.cmap[pc], 1);
      cg_radec(px, py, pz, ph, &q[0], &q[1]);              /* ra, dec */
      q[2] = bg(p.zt, p.g, cg_norm3(px, py, pz));          /* z0  */
      q[3] = p.need_beaming ? 0.0f : dz_rsd;               /* dz_rsd */
      q[4] = p.need_beaming ? 0.0f : -1.0f;                /* e1  */
      q[5] = p.need_beaming ? 0.0f : -1.0f;                /* e2  */
      q[6] = 0.0f;
      q[7] = 0.0f;
      q[8] = 0.0f;
    }
    if (!STAGED) continue;
    __syncwarp();
    const int nw = __popc(__ballot_sync(0xffffffffu, ok)) * SRC_F;
    float *dst = p.src + (size_t)(base + kb) * SRC_F;
#pragma unroll
    for (int h = 0; h < SRC_F; h++)
      if (h * 32 + lane < nw) dst[h * 32 + lane] = stage[wid][h * 32 + lane];
    __syncwarp();
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) nfb += __shfl_xor_sync(0xffffffffu, nfb, o);
  if (lane == 0 && nfb) atomicAdd(p.xstats + 1, (unsigned long long)nfb);
}

/* Trilinear potential gradient at a point with corner cells i0/i1 (i1 the
 * periodic neighbour above i0) and weights h0/h1 (interpolate_from_grid
 * RETURN_VEL, beaming.c:183-265): per z plane the four corners' central
 * differences weighted and summed with FMAs, then the two planes added.  The
 * eight corners' differences share points: 32 loads instead of 48, at offsets
 * from one cell's address.  The RSD waits for these loads (L1 wavefronts and
 * latency): 4.1e7 sources on 256^3 984 -> 791 us, 1.07e8 on 512^3 2.94 ->
 * 2.14 ms. */
__device__ __forceinline__ void cic_grad(const float *__restrict__ phi, const int i0[3], const int i1[3],
                                         const float h0[3], const float h1[3], int N, float v[3])
{
  const int ngx = 2 * (N / 2 + 1);
  const int xm = wrap(i0[0] - 1, N) - i0[0], x1 = i1[0] - i0[0], xp = wrap(i1[0] + 1, N) - i0[0];
  const int ym = (wrap(i0[1] - 1, N) - i0[1]) * ngx, y1 = (i1[1] - i0[1]) * ngx, yp = (wrap(i1[1] + 1, N) - i0[1]) * ngx;
  const long long plane = (long long)ngx * N;
  const long long zm = (wrap(i0[2] - 1, N) - i0[2]) * plane, z1 = (i1[2] - i0[2]) * plane,
                  zp = (wrap(i1[2] + 1, N) - i0[2]) * plane;
  const float *c = phi + pidx(i0[0], i0[1], i0[2], N);
  float in[2][4], zo[2][4]; /* [z][y, x]: the corners, and those one plane out */
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int o = ((k & 2) ? y1 : 0) + ((k & 1) ? x1 : 0);
    in[0][k] = __ldg(c + o);
    in[1][k] = __ldg(c + z1 + o);
    zo[0][k] = __ldg(c + zm + o);
    zo[1][k] = __ldg(c + zp + o);
  }
  v[0] = v[1] = v[2] = 0.0f;
#pragma unroll
  for (int hz = 0; hz < 2; hz++) {
    const float *r = c + (hz ? z1 : 0);
    const float wz = hz ? h0[2] : h1[2];
    const float xo[4] = {__ldg(r + xm), __ldg(r + xp), __ldg(r + y1 + xm), __ldg(r + y1 + xp)};
    const float yo[4] = {__ldg(r + ym), __ldg(r + ym + x1), __ldg(r + yp), __ldg(r + yp + x1)};
    float acc[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const float w = CG_MUL(CG_MUL(wz, (k & 2) ? h0[1] : h1[1]), (k & 1) ? h0[0] : h1[0]);
      const float gx = (k & 1) ? CG_SUB(xo[k], in[hz][k - 1]) : CG_SUB(in[hz][k + 1], xo[k]);
      const float gy = (k & 2) ? CG_SUB(yo[k], in[hz][k - 2]) : CG_SUB(in[hz][k + 2], yo[k]);
      const float gz = hz ? CG_SUB(zo[1][k], in[0][k]) : CG_SUB(in[1][k], zo[0][k]);
      acc[0] = CG_FMA(gx, w, acc[0]);
      acc[1] = CG_FMA(gy, w, acc[1]);
      acc[2] = CG_FMA(gz, w, acc[2]);
    }
#pragma unroll
    for (int a = 0; a < 3; a++) v[a] = CG_ADD(v[a], acc[a]);
  }
}

/* radial projection 0.5 idx (v . u), srcs.c:503 */
__device__ __forceinline__ float los_vel(const float v[3], const float u[3], float idx)
{
  return CG_MUL(CG_MUL(0.5f, idx), CG_ADD(CG_ADD(CG_MUL(v[0], u[0]), CG_MUL(v[1], u[1])), CG_MUL(v[2], u[2])));
}

/* Line-of-sight RSD at each source: trilinear gradient of the potential
 * (interpolate_from_grid CIC branch, beaming.c:183-265) projected on the
 * line of sight (srcs.c:500-504), then scaled by V1(r(z0)) * factor_vel
 * (srcs.c:657-662). */
__device__ __forceinline__ long long src_count(long long n, const long long *n_dev)
{
  if (n_dev) {
    const long long d = *n_dev;
    if (d < n) n = d;
  }
  return n;
}

__global__ void __launch_bounds__(256) k_beam_rsd(const float *__restrict__ phi, cg_srcs_params p, long long nsrc,
                                                  const long long *nsrc_dev)
{
  const int N = p.box.N;
  nsrc = src_count(nsrc, nsrc_dev);
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < nsrc;
       i += (long long)gridDim.x * blockDim.x) {
    float4 q = p.pos[i];
    float pos[3] = {q.x, q.y, q.z};
    const float po[3] = {p.box.p0, p.box.p1, p.box.p2};
    float r = cg_norm3(pos[0], pos[1], pos[2]);
    float ir = CG_DIV(1.0f, r > 0.001f ? r : 0.001f);
    float u[3];
    int i0[3], i1[3];
    float h0[3], h1[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
      float xn = CG_MUL(CG_ADD(pos[a], po[a]), p.box.idx);
      u[a] = CG_MUL(pos[a], ir);
      i0[a] = (int)xn;
      h0[a] = CG_SUB(xn, (float)i0[a]);
      h1[a] = CG_SUB(1.0f, h0[a]);
      i1[a] = wrap(i0[a] + 1, N);
      i0[a] = wrap(i0[a], N);
    }
    float v[3];
    cic_grad(phi, i0, i1, h0, h1, N, v);
    const float vr = los_vel(v, u, p.box.idx);
    float *s = p.src + (size_t)i * 9;
    float z0 = s[2];
    float rz = r_of_z(p.a_a2r, p.r_a2r, p.na, z0);
    s[3] = CG_MUL(vr, CG_MUL(bg(p.v1, p.g, rz), p.factor_vel));
  }
}

/* Direction, distance and last radial step of a source (srcs.c:485-493,
 * 583): r = |pos|, u = pos / max(r, 0.001), i_r_max = min((int)(r/dr + 0.5), nr - 1). */
__device__ __forceinline__ int los_setup(float4 q, const cg_los_params &p, float *r, float u[3])
{
  *r = cg_norm3(q.x, q.y, q.z);
  const float ir = CG_DIV(1.0f, *r > 0.001f ? *r : 0.001f);
  u[0] = CG_MUL(q.x, ir);
  u[1] = CG_MUL(q.y, ir);
  u[2] = CG_MUL(q.z, ir);
  const int k = (int)CG_ADD(CG_MUL(*r, p.idr), 0.5f);
  return k < p.nr - 1 ? k : p.nr - 1;
}

/* Lensing at each source (srcs.c:536-625 without _USE_FAST_LENSING): at
 * each step up to the source the nearest cell's tidal tensor and potential
 * gradient, projected with the source's rotation, weighted by
 * rm pg dr (r - rm) (shear, convergence) and 2 pg dr (r - rm) (deflection),
 * summed with Kahan compensation; the deflections are turned to degrees
 * (srcs.c:721-722). */
__global__ void __launch_bounds__(256) k_src_lensing(const float *__restrict__ phi, cg_los_params p)
{
  extern __shared__ float lsh[];
  for (int i = threadIdx.x; i < 2 * p.nr; i += blockDim.x) lsh[i] = p.lfac[i];
  __syncthreads();
  const float *f0 = lsh, *f1 = lsh + p.nr;
  const int N = p.box.N;
  const float po[3] = {p.box.p0, p.box.p1, p.box.p2};
  const float idx = p.box.idx;
  const long long nsrc = src_count(p.nsrc, p.nsrc_dev);
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < nsrc;
       i += (long long)gridDim.x * blockDim.x) {
    float r, u[3];
    const int kmax = los_setup(p.pos[i], p, &r, u);
    const float ir = CG_DIV(1.0f, r > 0.001f ? r : 0.001f);
    float ux[3], uy[3], rk[6], re1[6], re2[6];
    cg_lens_rot(u, CG_MUL(CG_MUL(idx, idx), ir), CG_MUL(CG_MUL(0.5f, idx), ir), ux, uy, rk, re1, re2);
    float a[5] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f}, c[5] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    for (int k = 0; k <= kmax; k++) {
      const float rm = CG_MUL(CG_ADD((float)k, 0.5f), p.dr);
      const int x0 = cg_ngp_cell(rm, u[0], po[0], idx, N);
      const int y0 = cg_ngp_cell(rm, u[1], po[1], idx, N);
      const int z0 = cg_ngp_cell(rm, u[2], po[2], idx, N);
      float f[19], t[6];
      stencil19(phi, x0, y0, z0, N, f);
      cg_tidal(f, t);
      const float v[3] = {CG_SUB(f[1], f[2]), CG_SUB(f[3], f[4]), CG_SUB(f[5], f[6])};
      const float dd = CG_SUB(r, rm);
      const float fr = CG_MUL(f1[k], dd), frm = CG_MUL(f0[k], dd);
      cg_kahan_add(&a[0], &c[0], CG_MUL(cg_dot6(re1, t), fr));
      cg_kahan_add(&a[1], &c[1], CG_MUL(cg_dot6(re2, t), fr));
      cg_kahan_add(&a[2], &c[2], CG_MUL(cg_dot6(rk, t), fr));
      cg_kahan_add(&a[3], &c[3], CG_MUL(cg_dot3(ux, v), frm));
      cg_kahan_add(&a[4], &c[4], CG_MUL(cg_dot3(uy, v), frm));
    }
    float *s = p.src + (size_t)i * 9;
    s[4] = a[0];
    s[5] = a[1];
    s[6] = a[2];
    s[7] = CG_MUL(a[4], 57.2957795f); /* dra  = RTOD * dty */
    s[8] = CG_MUL(a[3], 57.2957795f); /* ddec = RTOD * dtx */
  }
}

/* Skewers (srcs.c:509-536, 725-733): at each step up to the source the
 * trilinear density, or the Gaussian field of the eight corner cells, and
 * the trilinear radial velocity times V1(rm) factor_vel; 0 beyond.  A warp per
 * source and a lane per step: the steps are independent, and neighbouring ones
 * read neighbouring cells and write one row (a thread per source left most of
 * the chip idle and wrote one float per row: 225 -> 56 us for 1.6e4 sources of 96
 * steps at 192^3). */
__global__ void __launch_bounds__(256) k_src_skewers(const float *__restrict__ dens, const float *__restrict__ phi,
                                                      cg_los_params p)
{
  extern __shared__ float ssh[];
  for (int i = threadIdx.x; i < p.nr; i += blockDim.x) ssh[i] = p.vfac[i];
  __syncthreads();
  const int N = p.box.N;
  const float po[3] = {p.box.p0, p.box.p1, p.box.p2};
  const float idx = p.box.idx;
  const float s2 = p.skw_gauss ? *p.sigma2 : 0.0f;
  const long long nsrc = src_count(p.nsrc, p.nsrc_dev);
  const int lane = threadIdx.x & 31;
  for (long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < nsrc;
       i += ((long long)gridDim.x * blockDim.x) >> 5) {
    float r, u[3];
    const int kmax = los_setup(p.pos[i], p, &r, u);
    float *sd = p.skw_d + (size_t)i * p.nr, *sv = p.skw_v + (size_t)i * p.nr;
    for (int k = lane; k < p.nr; k += 32) {
      if (k > kmax) {
        sd[k] = 0.0f;
        sv[k] = 0.0f;
        continue;
      }
      const float rm = CG_MUL(CG_ADD((float)k, 0.5f), p.dr);
      int i0[3], i1[3];
      float h0[3], h1[3];
#pragma unroll
      for (int a = 0; a < 3; a++) cg_cic_axis(rm, u[a], po[a], idx, N, &i0[a], &i1[a], &h0[a], &h1[a]);
      float d;
      if (p.skw_gauss) {
        float gv[8];
#pragma unroll
        for (int b = 0; b < 8; b++) {
          const int ix = (b & 1) ? i1[0] : i0[0], iy = (b & 2) ? i1[1] : i0[1], iz = (b & 4) ? i1[2] : i0[2];
          const float rc = cg_norm3(cg_cell_coord(ix, p.box.dx, p.box.p0), cg_cell_coord(iy, p.box.dx, p.box.p1),
                                    cg_cell_coord(iz, p.box.dx, p.box.p2));
          gv[b] = cg_gauss_of_dens(__ldg(&dens[pidx(ix, iy, iz, N)]), bg(p.d1, p.g, rc), s2);
        }
        d = cg_cic_combine(gv, h0, h1);
      } else {
        d = cg_cic_value(dens, i0, i1, h0, h1, N);
      }
      float v[3];
      cic_grad(phi, i0, i1, h0, h1, N, v);
      sd[k] = d;
      sv[k] = CG_MUL(los_vel(v, u, idx), ssh[k]);
    }
  }
}

} /* namespace */

long long cg_srcs_nblocks(int N) { return ((long long)N * N * N + CPB - 1) / CPB; }
long long cg_srcs_scan_room(long long nb) { return (nb + SCAN_T - 1) / SCAN_T; }

cudaError_t cg_srcs_count(cudaStream_t s, const float *grid, const cg_srcs_params *p, long long *total, long long *host,
                          long long bpc)
{
  const long long nb = cg_srcs_nblocks(p->box.N);
  k_pois_tab<<<(CG_NA + 31) / 32, 32, 0, s>>>(*p, nb);
  /* steps per warp: four where the grid has many times the warps that the chip
   * holds (384^3 308 us, with two and one 317 and 342; 1024^3 5.2, 5.5 and
   * 6.1 ms), one on small grids, whose dense cells near the observer would leave
   * the last warps alone (128^3 77 us, with two and four 88 and 119; 256^3 with
   * 1000 sources per deg^2 347, 361 and 369) */
  const int steps = p->box.N > 256 ? 4 : 1;
  k_pois_count<<<(unsigned)(nb * CPB / (CWN * CW * steps)), CWN * 32, 0, s>>>(grid, *p, steps);
  if (nb <= SCAN_ONE) {
    k_scan_one<<<1, 1024, 0, s>>>(p->block_sums, nb, total, p->err, host, bpc);
    return cudaGetLastError();
  }
  const long long nt = cg_srcs_scan_room(nb);
  long long *tsum = p->block_sums + nb; /* the tile sums, just past the block totals */
  k_scan_tiles<<<(unsigned)nt, 1024, 0, s>>>(p->block_sums, nb, tsum, p->err);
  k_scan_top<<<1, 1024, 0, s>>>(tsum, nt, total);
  k_scan_apply<<<(unsigned)nt, 1024, 0, s>>>(p->block_sums, nb, tsum, total, p->err, host, bpc);
  return cudaGetLastError();
}

cudaError_t cg_srcs_emit(cudaStream_t s, const float *phi, const cg_srcs_params *p, long long b0, long long b1,
                         int nsm)
{
  if (b1 <= b0) return cudaSuccess;
  /* shares per block: until there are 64 blocks per SM, ten times those it
   * holds, while a share keeps a source per thread (the capacity is the total
   * with an eighth of slack).  c1 at 128^3 with 1 and 16 shares: 244 and
   * 169 us; 192^3 with 240 sources per block: 74 and 127 us with 1 and 4. */
  const long long nb = b1 - b0, all = cg_srcs_nblocks(p->box.N);
  int sh = 1;
  while (sh < 16 && nb * sh < 64ll * nsm && p->capacity >= all * sh * 2 * SB) sh *= 2;
  /* records written directly and staged, by sources per block of cells: 13
   * (512^3) 187 and 264 us, 79 (1024^3) 2.62 and 2.85 ms, 118 (1024^3) 3.29 and
   * 3.34 ms, 151 (256^3) 74 and 71 us, 197 (1024^3) 4.60 and 4.40 ms */
  const auto k = p->capacity < 144 * all ? k_emit<false> : k_emit<true>;
  k<<<dim3((unsigned)nb, (unsigned)sh), SB, 0, s>>>(phi, *p, b0);
  return cudaGetLastError();
}

cudaError_t cg_srcs_lensing(cudaStream_t s, const float *phi, const cg_los_params *p, int nsm)
{
  if (p->nsrc <= 0) return cudaSuccess;
  long long blocks = (p->nsrc + 255) / 256;
  if (blocks > (long long)nsm * 8) blocks = (long long)nsm * 8;
  k_src_lensing<<<(unsigned)blocks, 256, 2 * p->nr * sizeof(float), s>>>(phi, *p);
  return cudaGetLastError();
}

cudaError_t cg_srcs_skewers(cudaStream_t s, const float *dens, const float *phi, const cg_los_params *p, int nsm)
{
  if (p->nsrc <= 0) return cudaSuccess;
  long long blocks = (p->nsrc + 7) / 8; /* a warp per source */
  if (blocks > (long long)nsm * 8) blocks = (long long)nsm * 8;
  k_src_skewers<<<(unsigned)blocks, 256, p->nr * sizeof(float), s>>>(dens, phi, *p);
  return cudaGetLastError();
}

cudaError_t cg_srcs_beam_rsd(cudaStream_t s, const float *phi, const cg_srcs_params *p, long long nsrc,
                             const long long *nsrc_dev, int nsm)
{
  if (nsrc <= 0) return cudaSuccess;
  long long blocks = (nsrc + 255) / 256;
  if (blocks > (long long)nsm * 16) blocks = (long long)nsm * 16;
  k_beam_rsd<<<(unsigned)blocks, 256, 0, s>>>(phi, *p, nsrc, nsrc_dev);
  return cudaGetLastError();
}
