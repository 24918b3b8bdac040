/*
 * dens.cu -- physical density field (density.c:1034-1126) and the
 * redshift-bin sums of the bias normalisation (density.c:1128-1211).
 *
 *  k_moments_final : fixed-order FP64 sum of the per-block (sum d, sum d^2)
 *                    partials of the x pass -> <d>, sigma^2 (fourier.c:24-79).
 *  k_dens_bins     : one streaming pass over the grid that applies the
 *                    lognormal (or clipped, or 1LPT "rho-1") transform in
 *                    place and accumulates, per redshift bin, the cell count,
 *                    the summed redshift and the summed bias_model of every
 *                    tracer.  A warp owns 32 consecutive cells of a row;
 *                    lanes sharing a bin are reduced with shuffles (one pass
 *                    when the 32 cells share a bin) and one lane per value
 *                    adds the sums to the warp's private bins in shared
 *                    memory: integer counts and compensated (Kahan) FP32
 *                    sums, since FP64 arithmetic is scarce on this GPU.  Each
 *                    block combines its warps' bins in FP64 in a fixed order
 *                    and adds them to global 128-bit fixed-point
 *                    accumulators with integer atomics, whose sum does not
 *                    depend on the order the blocks arrive in.
 *  k_bins_finish   : the accumulators back to FP64 sums, the same bits on
 *                    every run.
 *  k_lpt_deposit   : 1LPT particle positions (density.c:473-501) and their
 *                    NGP, CIC or TSC deposit (density.c:37-187), staged per
 *                    tile of particles in shared memory.
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include "cg_dev.cuh"
#include "dens_api.h"

namespace {
using namespace cg;

/* The sums of k_moments_final's 1024 threads, in their order, by 32 blocks into
 * the first 1024 entries (each read by the thread that writes it only): one SM
 * adds about two doubles a clock, 81 us for the 131072 entries of 1024^3, both
 * kernels now 25. */
__global__ void __launch_bounds__(32) k_moments_part(double2 *part, size_t n)
{
  const size_t t = blockIdx.x * 32 + threadIdx.x;
  double a = 0.0, b = 0.0;
#pragma unroll 8
  for (size_t i = t; i < n; i += 1024) {
    const double2 v = part[i];
    a += v.x;
    b += v.y;
  }
  part[t] = make_double2(a, b);
}

__global__ void k_moments_final(const double2 *__restrict__ part, size_t n, double inv_ncell,
                                double *stats, float *s2f)
{
  __shared__ double sa[1024], sb[1024];
  double a = 0.0, b = 0.0;
  for (size_t i = threadIdx.x; i < n; i += blockDim.x) {
    double2 v = part[i];
    a += v.x;
    b += v.y;
  }
  sa[threadIdx.x] = a;
  sb[threadIdx.x] = b;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if ((int)threadIdx.x < s) {
      sa[threadIdx.x] += sa[threadIdx.x + s];
      sb[threadIdx.x] += sb[threadIdx.x + s];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    double mean = sa[0] * inv_ncell;
    double s2 = sb[0] * inv_ncell - mean * mean;
    stats[0] = sa[0];
    stats[1] = sb[0];
    stats[2] = mean;
    stats[3] = s2;
    *s2f = (float)s2;
  }
}

constexpr int MAXT = 8;      /* tracers per bins launch */
constexpr int BINS_WARPS = 8; /* warps per block at most  */

/* Sums of V values (a power of two) over the warp.  While several values are
 * left, a step exchanges them in pairs: each half of the lanes keeps one value
 * of a pair and gives the other away; then the plain butterfly.  Every value
 * is summed over the offsets 16, 8, 4, 2, 1 in this order, as one butterfly
 * per value would, in 4 (V - 1) + 2 (5 - log2 V) instructions instead of
 * 10 V.  Lane l returns the sum of value (the bits of l from the top, log2 V
 * of them). */
template <int V>
__device__ __forceinline__ float warp_sums(float *v, int lane)
{
  int o = 16;
#pragma unroll
  for (int n = V; n > 1; n >>= 1, o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int k = 0; k < n / 2; k++) {
      const float give = up ? v[k] : v[k + n / 2], keep = up ? v[k + n / 2] : v[k];
      v[k] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
#pragma unroll
  for (; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
  return v[0];
}

__host__ __device__ constexpr int pow2_at_least(int n) { return n <= 1 ? 1 : 2 * pow2_at_least((n + 1) / 2); }

/* Compensated FP32 accumulation s += v (c holds the running correction). */
__device__ __forceinline__ void kahan_add(float &s, float &c, float v)
{
  const float y = __fsub_rn(v, c);
  const float t = __fadd_rn(s, y);
  c = __fsub_rn(__fsub_rn(t, s), y);
  s = t;
}

/* 128-bit two's-complement fixed point with FIX_FRAC fraction bits, as a
 * (low, high) pair of u64: integer additions commute, so the total of the
 * blocks' FP64 partials is the same whatever order they arrive in.  A
 * partial x (|x| < 2^(127 - FIX_FRAC)) is rounded to the nearest multiple
 * of 2^-FIX_FRAC: |x| 2^(FIX_FRAC - 64) splits exactly into its integer part
 * (the high word) and its fraction, which scaled by 2^64 is the low word. */
constexpr int FIX_FRAC = 60;
constexpr double FIX_HI = 16.0;                                        /* 2^(64 - FIX_FRAC) */
constexpr double FIX_LO = 1.0 / 1152921504606846976.0;                 /* 2^-FIX_FRAC */
constexpr double FIX_TO_HI = 1.0 / 16.0;                               /* 2^(FIX_FRAC - 64) */
constexpr double TWO64 = 18446744073709551616.0;

__device__ __forceinline__ void fix_add(unsigned long long *a, double x)
{
  const bool neg = x < 0.0;
  const double y = __dmul_rn(fabs(x), FIX_TO_HI);
  const double h = floor(y);
  const double f = __dsub_rn(y, h); /* exact: y >= 0 */
  unsigned long long hi = __double2ull_rn(h), lo = __double2ull_rn(__dmul_rn(f, TWO64));
  if (neg) {
    lo = ~lo + 1ull;
    hi = ~hi + (lo == 0ull ? 1ull : 0ull);
  }
  const unsigned long long old = atomicAdd(a, lo);
  const unsigned long long carry = (old + lo < old) ? 1ull : 0ull;
  if (hi + carry) atomicAdd(a + 1, hi + carry);
}

/* Shared-memory bytes of one warp's bins: u32 count, then (sum, correction)
 * for the redshift and every tracer. */
__host__ __device__ inline size_t bins_warp_bytes(int nz, int nt) { return (size_t)nz * (4 + 8 * (1 + nt)); }

/* Up to three tracers eight blocks per SM (32 registers), more tracers two.
 * Bound by instruction issue (12 % of DRAM peak at 1024^3 with two tracers),
 * so row quantities are formed once per row, and a warp's sums take one
 * exchange for all values (warp_sums) and one compensated addition by as many
 * lanes as there are values: 10.8 -> 8.5 ms at 1024^3 with two tracers, 2.43
 * -> 1.74 ms at 512^3 with three. */
template <int NT>
__global__ void __launch_bounds__(BINS_WARPS * 32, NT <= 3 ? 8 : 2) k_dens_bins(float *grid, cg_bins_params p)
{
  extern __shared__ unsigned char sbins[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nwb = blockDim.x >> 5;
  constexpr int nt = NT, W = 1 + nt, V = pow2_at_least(W);
  const int nz = p.nz;
  unsigned int *cnt = reinterpret_cast<unsigned int *>(sbins + (size_t)wid * bins_warp_bytes(nz, nt));
  float *acc = reinterpret_cast<float *>(cnt + nz); /* [nz][W] sums, then [nz][W] corrections */
  float *cor = acc + (size_t)nz * W;
  for (int i = lane; i < nz; i += 32) cnt[i] = 0u;
  for (int i = lane; i < 2 * nz * W; i += 32) acc[i] = 0.0f;
  __syncwarp();
  const int N = p.box.N;
  const int nrow = N * N;
  const float s2 = p.sigma2f ? *p.sigma2f : 0.0f;
  const bool need_d1 = (p.mode == CG_DMODE_LGNR || p.mode == CG_DMODE_CLIP);
  const int gw = blockIdx.x * nwb + wid;
  const int nw = gridDim.x * nwb;
  /* the value whose sum this lane ends up with: 0 the redshift, 1 + t the
   * bias of tracer t; one lane of each adds it to the bins */
  const int mine_v = V > 1 ? lane / (32 / V) : 0;
  const bool adds = lane % (32 / V) == 0 && mine_v < W;
  /* a warp takes whole rows (N is a multiple of 32), 32 cells at a time */
  for (int row = gw; row < nrow; row += nw) {
    const int iz = (int)divN(row, p.box), iy = row - iz * N;
    const float y0 = cg_cell_coord(iy, p.box.dx, p.box.p1), z0 = cg_cell_coord(iz, p.box.dx, p.box.p2);
    const float yy = CG_MUL(y0, y0), zz2 = CG_MUL(z0, z0);
    float *ptr = grid + pidx(lane, iy, iz, N);
    for (int ix = lane; ix < N; ix += 32, ptr += 32) {
      float d = *ptr;
      const float x0 = cg_cell_coord(ix, p.box.dx, p.box.p0);
      const float r = CG_SQRT(CG_ADD(CG_ADD(CG_MUL(x0, x0), yy), zz2)); /* cg_norm3 */
      const BgAt at = bg_at(p.g, r);
      if (p.mode != CG_DMODE_NONE) {
        if (p.mode == CG_DMODE_RHO) {
          /* the particle deposit's fixed-point mass (never negative unless
           * a cell overflowed) */
          const int m = __float_as_int(d);
          if (m < 0 && p.err) atomicOr(p.err, ERR_DEPOSIT_OVERFLOW);
          d = CG_MUL((float)m, DEPOSIT_UNIT);
        }
        d = cg_dens_transform(p.mode, d, need_d1 ? bgv(p.d1, at) : 0.0f, s2);
        *ptr = d;
      }
      if (nz == 0) continue;
      float v[V];
#pragma unroll
      for (int k = 0; k < V; k++) v[k] = 0.0f;
      const float z = bgv(p.zt, at);
      int bin = (int)CG_MUL(z, p.idz) + 1;
      if (bin >= 0 && bin < nz) {
        v[0] = z;
#pragma unroll
        for (int t = 0; t < nt; t++) v[1 + t] = cg_bias_model(d, bgv(p.bz[t], at), p.bias_model);
      } else {
        bin = -1;
      }
      /* segmented reduction by bin; one pass when the 32 cells share a bin */
      unsigned todo = __ballot_sync(0xffffffffu, bin >= 0);
      while (todo) {
        const int lb = __shfl_sync(0xffffffffu, bin, __ffs(todo) - 1);
        const unsigned grp = __ballot_sync(0xffffffffu, bin == lb);
        float m[V];
#pragma unroll
        for (int k = 0; k < V; k++) m[k] = k < W && bin == lb ? v[k] : 0.0f;
        const float sum = warp_sums<V>(m, lane);
        if (adds) {
          float *a = acc + (size_t)lb * W + mine_v, *c = cor + (size_t)lb * W + mine_v;
          kahan_add(*a, *c, sum);
          if (lane == 0) cnt[lb] += (unsigned)__popc(grp);
        }
        todo &= ~grp;
      }
    }
  }
  __syncthreads();
  /* combine the warps' bins in FP64 in fixed order, one global update each */
  const size_t wb = bins_warp_bytes(nz, nt);
  for (int i = threadIdx.x; i < nz * (1 + W); i += blockDim.x) {
    const int b = i / (1 + W), k = i - b * (1 + W);
    if (k == 0) {
      unsigned long long n = 0;
      for (int w = 0; w < nwb; w++) n += reinterpret_cast<const unsigned int *>(sbins + (size_t)w * wb)[b];
      if (n) atomicAdd(&p.ncount[b], n);
    } else {
      double sum = 0.0;
      for (int w = 0; w < nwb; w++) {
        const unsigned int *cw = reinterpret_cast<const unsigned int *>(sbins + (size_t)w * wb);
        const float *aw = reinterpret_cast<const float *>(cw + nz);
        sum += (double)aw[(size_t)b * W + k - 1] - (double)aw[(size_t)nz * W + (size_t)b * W + k - 1];
      }
      if (sum != 0.0) fix_add(p.acc + 2 * ((size_t)(k - 1) * nz + b), sum);
    }
  }
}

/* Accumulator value v -> FP64: redshift sums v = b, bias sums of tracer t at
 * v = (1 + t) nz + b.  One rounding from the exact 128-bit sum (the high
 * part holds at most 2^53 in magnitude for any realistic grid). */
__global__ void __launch_bounds__(256) k_bins_finish(const unsigned long long *__restrict__ acc, int nz, int nt,
                                                    double *__restrict__ zsum, double *__restrict__ bsum)
{
  const int nv = nz * (1 + nt);
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += gridDim.x * blockDim.x) {
    unsigned long long lo = acc[2 * (size_t)v], hi = acc[2 * (size_t)v + 1];
    const bool neg = (long long)hi < 0;
    if (neg) { /* two's complement of the 128-bit pair */
      lo = ~lo + 1ull;
      hi = ~hi + (lo == 0ull ? 1ull : 0ull);
    }
    /* value = hi 2^(64 - FIX_FRAC) + lo 2^-FIX_FRAC */
    double d = __dadd_rn(__dmul_rn(__ull2double_rn(hi), FIX_HI), __dmul_rn(__ull2double_rn(lo), FIX_LO));
    if (neg) d = -d;
    if (v < nz) zsum[v] = d;
    else bsum[v - nz] = d;
  }
}

/* 1LPT: x = q + D(r) Psi (wrapped into the box), then the mass assignment of
 * pos_2_dens (density.c:178-187): NGP (S = 0, density.c:37-62), CIC (S = 1,
 * density.c:64-105) or TSC (S = 2, density.c:107-176).  A block takes a tile
 * of CT_X x CT_Y x CT_Z particles (lattice cells), a thread one column of it
 * along z, and deposits into a shared-memory box that extends the tile by
 * CT_H cells on every side; the box is added to the grid at the end, down its
 * columns, with one atomic per non-zero cell.  Deposits that fall outside the
 * box (particles displaced by more than about CT_H - 1 cells) go straight to
 * the grid.  Masses are fixed point (DEPOSIT_ONE per particle, integer atomics;
 * the grid holds the int32 bits until the density pass turns them into
 * rho - 1), so the result does not depend on the order of the atomic additions.
 * Bound by instruction issue (238 issue slots a particle at 512^3; the box's
 * flush found every cell's place by divisions before): 12.5 -> 7.9 ms
 * at 1024^3 with the grid's clearing, 207 -> 143 us at 256^3.  Tiles of 8 x 8,
 * 8 x 16, 16 x 8 and 4 x 32 in y and z took 9.8, 9.1, 10.3 and 10.9 against
 * 8.4 ms of 4 x 16 before the flush went by columns; 10 and 12 blocks per SM
 * (registers cut to 48 and 40) 8.1 and 8.3 against 7.9 ms. */
constexpr int CT_X = 32, CT_Y = 4, CT_Z = 16, CT_H = 2;
constexpr int CB_X = CT_X + 2 * CT_H, CB_Y = CT_Y + 2 * CT_H, CB_Z = CT_Z + 2 * CT_H;
constexpr int CT_THREADS = CT_X * CT_Y;
static_assert(CB_X * CB_Y * CB_Z % 4 == 0, "the box is cleared 16 bytes at a time");

/* A particle's first stencil cell per axis, its weights there, and whether
 * they are those of a position in the box (no weight above 1). */
template <int S>
struct Stencil {
  int i0[3];
  float w[3][S + 1];
  bool plain;
};

template <int S>
__device__ __forceinline__ void stencil_axis(Stencil<S> &t, int a, float q, float po, float L, float iag)
{
  constexpr int K = S + 1;
  q = CG_ADD(q, po);
  if (q < 0.0f) q = CG_ADD(q, L);
  if (q >= L) q = CG_SUB(q, L);
  const float u = CG_MUL(q, iag);
  t.plain = t.plain && u >= 0.0f;
  if (S == 0) {
    t.i0[a] = (int)CG_ADD(u, 0.5f);
    t.w[a][0] = 1.0f;
  } else if (S == 1) {
    t.i0[a] = (int)u;
    const float a1 = CG_SUB(u, (float)t.i0[a]);
    t.w[a][0] = CG_SUB(1.0f, a1);
    t.w[a][K - 1] = a1;
  } else {
    const int i0 = (int)floorf(CG_ADD(u, 0.5f));
    const float a0 = CG_SUB(u, (float)i0);
    const float hm = CG_SUB(0.5f, a0), hp = CG_ADD(0.5f, a0);
    t.w[a][0] = CG_MUL(0.5f, CG_MUL(hm, hm));
    t.w[a][1] = CG_SUB(0.75f, CG_MUL(a0, a0));
    t.w[a][K - 1] = CG_MUL(0.5f, CG_MUL(hp, hp));
    t.i0[a] = i0 - 1; /* the stencil starts one cell below the nearest */
  }
}

/* A particle that leaves its block's box: straight to the grid. */
template <int S>
__device__ __noinline__ void deposit_far(int *grid, int N, Stencil<S> t)
{
  constexpr int K = S + 1;
#pragma unroll
  for (int a = 0; a < 3; a++)
    /* q is in [0, L) unless the displacement exceeds the box: then a full
     * modulo keeps the cell index inside the grid */
    if ((unsigned)t.i0[a] >= (unsigned)N) t.i0[a] = ((t.i0[a] % N) + N) % N;
#pragma unroll
  for (int cz = 0; cz < K; cz++)
#pragma unroll
    for (int cy = 0; cy < K; cy++)
#pragma unroll
      for (int cx = 0; cx < K; cx++) {
        const int v = __float2int_rn(CG_MUL(CG_MUL(CG_MUL(t.w[0][cx], t.w[1][cy]), t.w[2][cz]), DEPOSIT_ONE));
        const int gx = t.i0[0] + cx >= N ? t.i0[0] + cx - N : t.i0[0] + cx;
        const int gy = t.i0[1] + cy >= N ? t.i0[1] + cy - N : t.i0[1] + cy;
        const int gz = t.i0[2] + cz >= N ? t.i0[2] + cz - N : t.i0[2] + cz;
        atomicAdd(&grid[pidx(gx, gy, gz, N)], v);
      }
}

template <int S, bool TWO>
__global__ void __launch_bounds__(CT_THREADS, 8) k_lpt_deposit(int *grid, const float *__restrict__ dx_,
                                                            const float *__restrict__ dy_,
                                                            const float *__restrict__ dz_,
                                                            const __grid_constant__ cg_lpt_params p)
{
  constexpr int K = S + 1; /* cells per axis of the stencil */
  __shared__ __align__(16) int box[CB_Z * CB_Y * CB_X];
  const int N = p.box.N;
  const int ntx = (N + CT_X - 1) / CT_X, nty = (N + CT_Y - 1) / CT_Y;
  const int t = blockIdx.x, tx = t % ntx, tyz = t / ntx;
  const int tx0 = tx * CT_X, ty0 = (tyz % nty) * CT_Y, tz0 = (tyz / nty) * CT_Z;
  for (int i = threadIdx.x; i < CB_X * CB_Y * CB_Z / 4; i += CT_THREADS)
    reinterpret_cast<int4 *>(box)[i] = make_int4(0, 0, 0, 0);
  __syncthreads();
  const int lane = threadIdx.x & 31, wy = threadIdx.x >> 5;
  const int ix = tx0 + lane, iy = ty0 + wy;
  const long long plane = (long long)(2 * (N / 2 + 1)) * N;
  if (ix < N && iy < N) {
    const float iag = CG_DIV((float)N, p.box.L);
    const float po[3] = {p.box.p0, p.box.p1, p.box.p2};
    const int org[3] = {tx0 - CT_H, ty0 - CT_H, tz0 - CT_H};
    const int last[3] = {CB_X - K, CB_Y - K, CB_Z - K};
    float xv[3] = {cg_cell_coord(ix, p.box.dx, p.box.p0), cg_cell_coord(iy, p.box.dx, p.box.p1), 0.0f};
    long long id = pidx(ix, iy, tz0, N);
    const int nz = N - tz0 < CT_Z ? N - tz0 : CT_Z;
    /* the next plane's displacements are loaded a step ahead */
    float nx[3] = {__ldg(&dx_[id]), __ldg(&dy_[id]), __ldg(&dz_[id])};
#pragma unroll 1
    for (int kz = 0; kz < nz; kz++, id += plane) {
      xv[2] = cg_cell_coord(tz0 + kz, p.box.dx, p.box.p2);
      const float dsp[3] = {nx[0], nx[1], nx[2]};
      if (kz + 1 < nz) {
        nx[0] = __ldg(&dx_[id + plane]);
        nx[1] = __ldg(&dy_[id + plane]);
        nx[2] = __ldg(&dz_[id + plane]);
      }
      const float r = cg_norm3(xv[0], xv[1], xv[2]);
      const float dg = bg(p.d1, p.g, r);
      Stencil<S> st;
      st.plain = true;
      if (TWO) { /* 2LPT: x = q + D1 Psi1 + D2 Psi2 (density.c:890) */
        const float ds2[3] = {__ldg(&p.d2x[id]), __ldg(&p.d2y[id]), __ldg(&p.d2z[id])};
        const float d2g = bg(p.d2, p.g, r);
#pragma unroll
        for (int a = 0; a < 3; a++)
          stencil_axis<S>(st, a, CG_FMA(d2g, ds2[a], CG_FMA(dg, dsp[a], xv[a])), po[a], p.box.L, iag);
      } else {
#pragma unroll
        for (int a = 0; a < 3; a++) stencil_axis<S>(st, a, CG_FMA(dg, dsp[a], xv[a]), po[a], p.box.L, iag);
      }
      /* the first stencil cell in the box: the box may reach over the grid's
       * end, by less than a period */
      int at = 0;
      bool in = st.plain;
#pragma unroll
      for (int a = 2; a >= 0; a--) {
        int d = st.i0[a] - org[a];
        if ((unsigned)d >= (unsigned)N) d += d < 0 ? N : -N;
        in = in && (unsigned)d <= (unsigned)last[a];
        at = at * (a == 1 ? CB_Y : CB_X) + d;
      }
      if (!in) {
        deposit_far<S>(grid, N, st);
        continue;
      }
#pragma unroll
      for (int cz = 0; cz < K; cz++)
#pragma unroll
        for (int cy = 0; cy < K; cy++)
#pragma unroll
          for (int cx = 0; cx < K; cx++) {
            /* the weight in units of 2^-20, rounded to nearest: the scaling by
             * a power of two is exact, and 1.5 2^23 added to 0 .. 2^20 rounds
             * to a whole number in the low bits */
            const float v = CG_MUL(CG_MUL(st.w[0][cx], st.w[1][cy]), CG_MUL(st.w[2][cz], DEPOSIT_ONE));
            atomicAdd(&box[at + (cz * CB_Y + cy) * CB_X + cx], __float_as_int(CG_ADD(v, 12582912.0f)) - 0x4b400000);
          }
    }
  }
  __syncthreads();
  /* the box's tile columns, a lane each, down the planes; then the halo
   * columns */
  const int gx = ix >= N ? ix - N : ix, gz0 = tz0 < CT_H ? tz0 - CT_H + N : tz0 - CT_H;
  for (int by = wy; by < CB_Y; by += CT_THREADS / 32) {
    int gy = ty0 - CT_H + by;
    gy = gy < 0 ? gy + N : (gy >= N ? gy - N : gy);
    int *g = grid + pidx(gx, gy, gz0, N);
    const int *from = box + by * CB_X + CT_H + lane;
    int up = N - gz0; /* planes to the grid's end */
#pragma unroll 4
    for (int bz = 0; bz < CB_Z; bz++) {
      if (bz == up) g -= N * plane;
      const int v = from[bz * (CB_Y * CB_X)];
      if (v != 0) atomicAdd(g, v);
      g += plane;
    }
  }
  for (int i = threadIdx.x; i < 2 * CT_H * CB_Y * CB_Z; i += CT_THREADS) {
    const int row = i / (2 * CT_H), c = i - row * 2 * CT_H, bx = c < CT_H ? c : c + CT_X;
    const int v = box[row * CB_X + bx];
    if (v == 0) continue;
    const int bz = row / CB_Y, by = row - bz * CB_Y;
    int gx = tx0 - CT_H + bx, gy = ty0 - CT_H + by, gz = tz0 - CT_H + bz;
    gx = gx < 0 ? gx + N : (gx >= N ? gx - N : gx);
    gy = gy < 0 ? gy + N : (gy >= N ? gy - N : gy);
    gz = gz < 0 ? gz + N : (gz >= N ? gz - N : gz);
    atomicAdd(&grid[pidx(gx, gy, gz, N)], v);
  }
}

template <int S>
void deposit(unsigned tiles, cudaStream_t s, int *mass, const float *dx, const float *dy, const float *dz,
             const cg_lpt_params &p)
{
  if (p.d2x) k_lpt_deposit<S, true><<<tiles, CT_THREADS, 0, s>>>(mass, dx, dy, dz, p);
  else k_lpt_deposit<S, false><<<tiles, CT_THREADS, 0, s>>>(mass, dx, dy, dz, p);
}

/* compute_density_normalization after the bin sums (density.c:1272-1355):
 * mean redshift and count / sum(bias) per bin, the first and last bins
 * copied from their neighbours, then the linear spline in z evaluated at
 * z(r_i) with GSL's bracketing (largest bin centre <= z).  blockIdx.y: the
 * tracer; every block forms the bins' values again and takes 256 of the r_i
 * (one block per tracer walked all 5001: 20 us); every double operation is an explicitly rounded one, in the order
 * of the host restatement, so the tables do not depend on contraction. */
__global__ void __launch_bounds__(256) k_norm_tables(const unsigned long long *__restrict__ ncount,
                                                     const double *__restrict__ zsum,
                                                     const double *__restrict__ bsum, int nz, double zlast,
                                                     const double *__restrict__ zr, float *out, double *out64)
{
  extern __shared__ double nsh[];
  double *zz = nsh, *y = nsh + nz;
  const int t = blockIdx.y;
  for (int iz = threadIdx.x; iz < nz; iz += blockDim.x) {
    const unsigned long long n = ncount[iz];
    const double b = bsum[(size_t)t * nz + iz];
    zz[iz] = n > 0 ? __ddiv_rn(zsum[iz], __ull2double_rn(n)) : zsum[iz];
    y[iz] = n > 0 ? __ddiv_rn(__ull2double_rn(n), b) : b;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    zz[0] = 0;
    zz[nz - 1] = zlast;
    y[0] = y[1];
    y[nz - 1] = y[nz - 2];
  }
  __syncthreads();
  float *o = out + (size_t)t * (CG_NA + 2);
  double *o64 = out64 ? out64 + (size_t)t * (CG_NA + 2) : nullptr;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < CG_NA; i += gridDim.x * blockDim.x) {
    const double z = zr[i];
    double nm;
    if (z < zz[0]) {
      nm = y[0];
    } else if (z >= zz[nz - 1]) {
      nm = y[nz - 1];
    } else {
      int lo = 0, hi = nz - 1;
      while (hi > lo + 1) {
        const int mid = (lo + hi) / 2;
        if (zz[mid] > z) hi = mid;
        else lo = mid;
      }
      nm = __dadd_rn(y[lo], __ddiv_rn(__dmul_rn(__dsub_rn(z, zz[lo]), __dsub_rn(y[hi], y[lo])), __dsub_rn(zz[hi], zz[lo])));
    }
    o[i] = (float)nm;
    if (o64) o64[i] = nm;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    o[CG_NA] = (float)y[0];
    o[CG_NA + 1] = (float)y[nz - 1];
    if (o64) {
      o64[CG_NA] = y[0];
      o64[CG_NA + 1] = y[nz - 1];
    }
  }
}

} /* namespace */

cudaError_t cg_norm_tables(cudaStream_t s, const unsigned long long *ncount, const double *zsum, const double *bsum,
                           int nz, int nt, double zlast, const double *zr, float *out, double *out64)
{
  if (nz < 2 || nz > CG_NORM_NZ_MAX || nt < 1) return cudaErrorInvalidValue;
  const size_t smem = 2 * sizeof(double) * (size_t)nz;
  if (smem > 48 * 1024) {
    static bool set[CG_MAX_DEVICES]; /* opt-in above 48 KiB, once per device */
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= CG_MAX_DEVICES) return cudaErrorInvalidDevice;
    if (!set[dev]) {
      cudaError_t e = cudaFuncSetAttribute(k_norm_tables, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           2 * (int)sizeof(double) * CG_NORM_NZ_MAX);
      if (e != cudaSuccess) return e;
      set[dev] = true;
    }
  }
  k_norm_tables<<<dim3((CG_NA + 255) / 256, nt), 256, smem, s>>>(ncount, zsum, bsum, nz, zlast, zr, out, out64);
  return cudaGetLastError();
}

cudaError_t cg_moments_final(cudaStream_t s, double2 *part, size_t n, double inv_ncell, double *stats,
                             float *s2f)
{
  if (n > 8192) { /* below, the second launch costs what it saves */
    k_moments_part<<<32, 32, 0, s>>>(part, n);
    n = 1024;
  }
  k_moments_final<<<1, 1024, 0, s>>>(part, n, inv_ncell, stats, s2f);
  return cudaGetLastError();
}

cudaError_t cg_dens_bins(cudaStream_t s, float *grid, const cg_bins_params *p, int nsm)
{
  if (p->nt < 0 || p->nt > MAXT || p->nz < 0) return cudaErrorInvalidValue;
  /* as many warps per block (up to 8) as the bins of each fit in 200 KiB */
  const size_t wb = bins_warp_bytes(p->nz, p->nt);
  int nwb = BINS_WARPS;
  while (nwb > 1 && (size_t)nwb * wb > 200u * 1024u) nwb--;
  if ((size_t)nwb * wb > 200u * 1024u) return cudaErrorInvalidValue;
  const size_t smem = (size_t)nwb * wb;
  if (smem > 48u * 1024u) {
    static bool set[CG_MAX_DEVICES]; /* raised once per device to the largest size a launch asks for */
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= CG_MAX_DEVICES) return cudaErrorInvalidDevice;
    if (!set[dev]) {
      cudaError_t e = cudaSuccess;
#define X(k) \
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_dens_bins<k>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
      X(0) X(1) X(2) X(3) X(4) X(5) X(6) X(7) X(8)
#undef X
      if (e != cudaSuccess) return e;
      set[dev] = true;
    }
  }
  long long nrow = (long long)p->box.N * p->box.N;
  long long blocks = (nrow + nwb - 1) / nwb;
  long long cap = (long long)nsm * 8;
  if (blocks > cap) blocks = cap;
  switch (p->nt) { /* one instantiation per tracer count: loops of exact length */
#define X(k)                                                           \
  case k:                                                              \
    k_dens_bins<k><<<(unsigned)blocks, nwb * 32, smem, s>>>(grid, *p); \
    break;
    X(0) X(1) X(2) X(3) X(4) X(5) X(6) X(7) X(8)
#undef X
  }
  if (p->nz > 0) {
    const int nv = p->nz * (1 + p->nt);
    k_bins_finish<<<(nv + 255) / 256, 256, 0, s>>>(p->acc, p->nz, p->nt, p->zsum, p->bsum);
  }
  return cudaGetLastError();
}

int cg_dens_bins_max_tracers(void) { return MAXT; }

/* Scratch of the allocation-free bins entry: u64 counts [CG_BINS_STATIC_NZ],
 * redshift sums [CG_BINS_STATIC_NZ], bias sums [MAXT][nz] (doubles), then
 * the 128-bit accumulators [1 + MAXT][nz][2] (u64).  A module-scope array
 * costs no allocation call at run time: it exists in every context that
 * loads this module. */
static_assert(CG_BINS_STATIC_BYTES == (size_t)CG_BINS_STATIC_NZ * ((2 + MAXT) + 2 * (1 + MAXT)) * 8,
              "static bins scratch layout");
static __device__ __align__(256) unsigned char g_bins_scratch[CG_BINS_STATIC_BYTES];

cudaError_t cg_dens_bins_static_scratch(void **ptr, size_t *bytes)
{
  *bytes = sizeof(g_bins_scratch);
  return cudaGetSymbolAddress(ptr, g_bins_scratch);
}

cudaError_t cg_lpt_cic(cudaStream_t s, float *grid, const float *dx, const float *dy, const float *dz,
                       const cg_lpt_params *p, int nsm)
{
  (void)nsm;
  const long long N = p->box.N;
  const long long tiles = ((N + CT_X - 1) / CT_X) * ((N + CT_Y - 1) / CT_Y) * ((N + CT_Z - 1) / CT_Z);
  /* the grid (zeroed by the caller) holds int32 fixed-point masses until
   * the density pass of mode CG_DMODE_RHO */
  int *mass = reinterpret_cast<int *>(grid);
  if (p->interp == 0) deposit<0>((unsigned)tiles, s, mass, dx, dy, dz, *p);
  else if (p->interp == 2) deposit<2>((unsigned)tiles, s, mass, dx, dy, dz, *p);
  else deposit<1>((unsigned)tiles, s, mass, dx, dy, dz, *p);
  return cudaGetLastError();
}
