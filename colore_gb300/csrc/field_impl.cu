/*
 * field_impl.cu -- Gaussian field (fourier.c:285-423) and 1LPT displacement
 * transforms (density.c:376-445) for one grid size N = CG_N.
 *
 * This file is compiled once per supported grid size with -DCG_N=<N>; the
 * dispatcher in capi.cu selects the instantiation.  Three passes make the
 * 3-D c2r transform of the half spectrum H[kz][ky][kx] (kx in [0, N/2],
 * fastest) into the padded real grid, in place:
 *
 *   1. fill + z : a block owns TX consecutive kx at one ky and all kz.  It
 *                 generates the modes of every output field from one set of
 *                 Philox draws, kz and -kz together, parks them in shared
 *                 memory, transforms along z and writes the result.  The
 *                 spectrum is never read back from HBM.
 *   2. y        : the same column transform along y, read-modify-write.
 *   3. x (c2r)  : a group of threads owns one row of N/2+1 complex values;
 *                 the Hermitian even/odd split turns the length-N real
 *                 inverse into a length-N/2 complex one.  The block's rows
 *                 (contiguous in HBM) are staged into shared memory by one
 *                 bulk copy of the copy engine.  The normalisation
 *                 (sqrt(2 pi)/L)^3 (fourier.c:383-398) and the partial sums
 *                 of <d> and <d^2> (fourier.c:24-79) are fused here.
 *
 * FFTW's c2r semantics for the kx = 0 and kx = N/2 planes (the imaginary
 * parts of each row's DC and Nyquist terms are ignored after the y and z
 * transforms) are reproduced by dropping those imaginary parts in pass 3.
 *
 * 2LPT (density.c:646-1031) adds the forward transform of the second-order
 * source: an r2c row pass along x, the forward y pass, and a z pass that
 * transforms forward, forms Psi2_a = -i k_a S_k / (N^3 k^2) for the three
 * axes and transforms each back along z; the inverse y and x passes follow.
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include "cg_dev.cuh"
#include "cg_tma.cuh"
#include "fft.cuh"
#include "field_api.h"
#include "fft_plans.h"

#ifndef CG_N
#error "compile with -DCG_N=<grid size>"
#endif

namespace {

using namespace cg;


constexpr int N = CG_N;
constexpr int NH = N / 2 + 1;
using PL = Plan<N>;
constexpr int P = N / PL::CR;       /* threads per column transform (y pass)      */
constexpr int PF = N / PL::FR;      /* threads per column transform (fill + z)    */
constexpr int LH = N / 2;           /* row transform length         */
constexpr int PR = LH / PL::RR;     /* threads per row transform    */
/* Exchange slots (fft.cuh).  The fills and the x pass are padded against
 * bank conflicts; the y pass is not: it waits for HBM, and the padding takes
 * shared memory from the L1 that holds its loads in flight (512^3, tiles of
 * 16 columns: 0.406 ms without, 0.546 ms with). */
constexpr int fill_sh(int TX) { return TX >= 16 ? cgfft::NO_PAD : cgfft::pad_shift(PL::F0); }
template <int TX>
constexpr int FSH = fill_sh(TX);
constexpr int SHX = cgfft::pad_shift(PL::R0);
constexpr int EXX = cgfft::pad_len(LH, SHX);
constexpr int ROWS = NH > EXX ? NH : EXX; /* smem per row */
/* Stage tables of the column, fill and row transforms, one after the other. */
constexpr int TW_C = 0, TW_F = TW_C + cgfft::tw_len<PL::C0, PL::C1, PL::C2>;
constexpr int TW_R = TW_F + cgfft::tw_len<PL::F0, PL::F1, PL::F2>;
constexpr int TW_LEN = TW_R + cgfft::tw_len<PL::R0, PL::R1, PL::R2>;
template <int TX>
constexpr int EXF = cgfft::pad_len(N, fill_sh(TX)); /* exchange slots per column of the fills */

/* P(k) at log10 k, pk_linear0 (cosmo.c:291-308).  The interpolation branch
 * stops at numk-2: the reference also takes it for ik = numk-1 and then
 * reads one element past the table. */
__device__ __forceinline__ float pk_lin(const FillParams &p, float lgk)
{
  const int ik = (int)((lgk - p.logkmin) * p.idlogk);
  if (ik < 0) return __ldg(&p.pk[0]).y * exp10f(p.n_scal * (lgk - p.logkmin));
  if (ik < p.numk - 1) {
    const float4 q = __ldg(&p.pk[ik]); /* log10 k_ik, P_ik, P_ik+1 - P_ik */
    return q.y + (lgk - q.x) * q.z * p.idlogk;
  }
  return __ldg(&p.pk[p.numk - 1]).y * exp10f(-3.0f * (lgk - p.logkmax));
}

__device__ __forceinline__ float kcomp(int i, int n, float dk) { return (float)(2 * i <= n ? i : i - n) * dk; }

/* What a mode's value needs besides its random draw: |k|^2, P(k)/dk^3, the
 * smoothing factor and num/|k|^2.  They depend on the components of k through their squares
 * only, so modes (kx, ky, kz) and (kx, ky, -kz) share one evaluation. */
struct KAmp {
  float k2, s2, sm, ik2;
};

__device__ __forceinline__ KAmp k_amp(const FillParams &p, float num, int kx, int ky, int kz)
{
  const float kxf = (float)kx * p.dk, kyf = kcomp(ky, N, p.dk), kzf = kcomp(kz, N, p.dk);
  KAmp a;
  a.k2 = kxf * kxf + kyf * kyf + kzf * kzf;
  a.sm = 1.0f;
  a.s2 = a.ik2 = 0.0f;
  if (!(a.k2 > 0.0f)) return a;
  a.ik2 = num / a.k2;
  const float lgk = 0.5f * log10f(a.k2);
  a.s2 = pk_lin(p, lgk) * p.idk3;
  if (p.do_smooth) a.sm = expf(-0.5f * p.r2s * a.k2);
  return a;
}

/* Unsmoothed Gaussian mode (rng_delta_gauss, common.c:191-201, with
 * sigma^2 = P(k)/dk^3, fourier.c:343), k != 0. */
__device__ __forceinline__ float2 k_draw(const FillParams &p, float s2, int kx, int ky, int kz)
{
  uint32_t lo, hi = 0u;
  if constexpr ((uint64_t)NH * N * N <= 0x100000000ull) { /* the mode number fits 32 bits */
    lo = (uint32_t)kx + (uint32_t)NH * ((uint32_t)ky + (uint32_t)N * (uint32_t)kz);
  } else {
    const uint64_t m = (uint64_t)kx + (uint64_t)NH * ((uint64_t)ky + (uint64_t)N * (uint64_t)kz);
    lo = (uint32_t)m;
    hi = (uint32_t)(m >> 32);
  }
  /* words 0 and 1 of Philox4x32-10 at counter (lo, hi, 0, 0): cg_philox4x32_10
   * with the round keys read from the parameters */
  uint32_t c0 = lo, c1 = hi, c2 = 0u, c3 = 0u;
#pragma unroll
  for (int r = 0; r < 10; r++) {
    uint32_t h0, l0, h1, l1;
    cg_mulhilo32(0xD2511F53u, c0, &h0, &l0);
    cg_mulhilo32(0xCD9E8D57u, c2, &h1, &l1);
    c0 = h1 ^ c1 ^ p.rk0[r];
    c1 = l1;
    c2 = h0 ^ c3 ^ p.rk1[r];
    c3 = l0;
  }
  const float u1 = cg_u01f(c0), u2 = cg_u01f(c1);
  float s, c;
  sincospif(2.0f * u1, &s, &c);
  const float mod = sqrtf(-s2 * logf(1.0f - u2));
  return make_float2(mod * c, mod * s);
}

/* The modes of column (kx, ky) by pairs: put(kz, amplitude) for every kz, the
 * pair (kz, N - kz) from one amplitude (kz = 0 and N/2 pair up, each with its
 * own).  Thread t of the PF that share a column takes kz = t, t + PF, ...
 * below N/2.  Rolled: one copy of the generator in the instruction stream
 * (inlined per element it overflowed the instruction cache).  The fills wait
 * for issue slots and for the transform's exchanges, not for HBM (20 % of DRAM
 * peak at 1024^3; with the generation left out 5.4 of 6.5 ms, at 512^3 0.42 of
 * 0.68).  One amplitude for two modes, round
 * keys and the P(k) table's differences formed on the host, and exchange slots
 * free of conflicts: 7.25 -> 6.58 ms for the two-field fill at 1024^3,
 * 374 -> 334 us at 384^3. */
template <class Put>
__device__ __forceinline__ void k_pairs(const FillParams &p, float num, int kx, int ky, int t, Put put)
{
  static_assert(PL::FR % 2 == 0, "an even number of modes per thread");
#pragma unroll 1
  for (int e = 0; e < PL::FR / 2; e++) {
    const int kz = t + PF * e;
    KAmp a;
#pragma unroll 1
    for (int h = 0; h < 2; h++) {
      const int z = h == 0 ? kz : (kz == 0 ? N / 2 : N - kz);
      if (h == 0 || kz == 0) a = k_amp(p, num, kx, ky, z);
      put(z, a);
    }
  }
}

/* Pass 1: fill + z transform of delta_k and phi_k (fourier.c:337-352).
 * grid = (ceil(NH/TX), N).  The modes of the block's columns are generated by
 * pairs and parked in shared memory; delta's slot is also the exchange buffer
 * of the transforms, safe because a transform reads all its inputs before its
 * first exchange write. */
template <int TX>
__global__ void __launch_bounds__(TX *PF) k_fill_z(float2 *o0, float2 *o1, FillParams p,
                                                  const float4 *__restrict__ tw)
{
  extern __shared__ float2 smem[];
  const int c = threadIdx.x % TX, t = threadIdx.x / TX;
  const int kx = blockIdx.x * TX + c, ky = blockIdx.y;
  const bool ok = kx < NH;
  float2 *s0 = smem, *s1 = smem + (size_t)EXF<TX> * TX;
  if (ok)
    k_pairs(p, -p.prefac, kx, ky, t, [&](int kz, const KAmp &a) {
      float2 d = make_float2(0.0f, 0.0f), phi = d;
      if (a.k2 > 0.0f) {
        d = k_draw(p, a.s2, kx, ky, kz);
        phi = make_float2(a.ik2 * d.x, a.ik2 * d.y);
        if (p.do_smooth) {
          d.x *= a.sm;
          d.y *= a.sm;
          if (p.smooth_pot) {
            phi.x *= a.sm;
            phi.y *= a.sm;
          }
        }
      }
      s0[kz * TX + c] = d;
      s1[kz * TX + c] = phi;
    });
  __syncthreads();
  auto sm = [&](int slot) -> float2 & { return smem[slot * TX + c]; };
#pragma unroll
  for (int j = 0; j < 2; j++) {
    const float2 *in = j == 0 ? s0 : s1;
    auto ld = [&](int pos) -> float2 { return ok ? in[pos * TX + c] : make_float2(0.0f, 0.0f); };
    float2 *o = j == 0 ? o0 : o1;
    auto st = [&](int pos, float2 v) {
      if (ok) o[((size_t)pos * N + ky) * NH + kx] = v;
    };
    cgfft::transform<N, PL::FR, PL::F0, PL::F1, PL::F2, 1, FSH<TX>>(t, tw + TW_F, ld, st, sm);
    __syncthreads();
  }
}

/* The three-field fills: 1LPT displacements i k_a delta'_k / (N^3 k^2)
 * (density.c:430-436), where delta'_k = r2c(delta_G) = N^3 norm H(delta_k)
 * and H is the Hermitian projection that the c2r applied on the kx = 0 and
 * kx = N/2 planes; of kind 1 and 2 the second derivatives
 * i k_i (i k_j delta'_k / (N^3 k^2)) of 2LPT (density.c:704-709), xx xy xz
 * and yy yz zz.  One value per mode is kept, b = delta'_k / (N^3 k^2) with
 * the smoothing (0 at k = 0), and each field is formed from it as the
 * transform loads it.  The projection's partner -k has the same amplitude. */
__device__ __forceinline__ float2 lpt_base(const FillParams &p, const KAmp &a, int kx, int ky, int kz)
{
  if (!(a.k2 > 0.0f)) return make_float2(0.0f, 0.0f);
  float2 d = k_draw(p, a.s2, kx, ky, kz);
  d.x *= a.sm;
  d.y *= a.sm;
  if (kx == 0 || kx == N / 2) {
    const int ky2 = ky == 0 ? 0 : N - ky, kz2 = kz == 0 ? 0 : N - kz;
    float2 e = k_draw(p, a.s2, kx, ky2, kz2);
    e.x *= a.sm;
    e.y *= a.sm;
    d = make_float2(0.5f * (d.x + e.x), 0.5f * (d.y - e.y));
  }
  return make_float2(a.ik2 * d.x, a.ik2 * d.y);
}

__device__ __forceinline__ float2 lpt_field(const FillParams &p, int kind, int j, int kx, int ky, int kz, float2 b)
{
  const float kv[3] = {(float)kx * p.dk, kcomp(ky, N, p.dk), kcomp(kz, N, p.dk)};
  if (kind == 0) return make_float2(-kv[j] * b.y, kv[j] * b.x);
  const float ki[3] = {kind == 1 ? kv[0] : kv[1], kind == 1 ? kv[0] : kv[1], kind == 1 ? kv[0] : kv[2]};
  const float kj[3] = {kind == 1 ? kv[0] : kv[1], kind == 1 ? kv[1] : kv[2], kv[2]};
  const float g = -ki[j] * kj[j];
  return make_float2(g * b.x, g * b.y);
}

/* Grids of a three-field fill: Psi, then for 2LPT the six second derivatives. */
struct Lpt9 {
  float2 *o[9];
};

/* Pass 1 of the three-field fills: as k_fill_z, but one value per mode
 * (lpt_base) is parked, in the slot after the exchange buffer, and the first
 * stage of each transform forms the field from it (lpt_field).  Two slots
 * instead of three per block, so three blocks fit on an SM.  SETS 1 the
 * displacements, 3 the second derivatives too: the modes are drawn once for
 * all nine grids (a third of the time of a three-field fill). */
template <int TX, int SETS>
__global__ void __launch_bounds__(TX *PF, 3) k_fill_z3(Lpt9 out, FillParams p, const float4 *__restrict__ tw)
{
  extern __shared__ float2 smem[];
  const int c = threadIdx.x % TX, t = threadIdx.x / TX;
  const int kx = blockIdx.x * TX + c, ky = blockIdx.y;
  const bool ok = kx < NH;
  float2 *base = smem + (size_t)EXF<TX> * TX;
  if (ok) k_pairs(p, p.lpt_norm, kx, ky, t, [&](int kz, const KAmp &a) { base[kz * TX + c] = lpt_base(p, a, kx, ky, kz); });
  __syncthreads();
  auto sm = [&](int slot) -> float2 & { return smem[slot * TX + c]; };
#pragma unroll 1
  for (int kind = 0; kind < SETS; kind++) {
#pragma unroll
    for (int j = 0; j < 3; j++) {
      auto ld = [&](int pos) -> float2 {
        return ok ? lpt_field(p, SETS == 1 ? 0 : kind, j, kx, ky, pos, base[pos * TX + c]) : make_float2(0.0f, 0.0f);
      };
      float2 *o = out.o[3 * kind + j];
      auto st = [&](int pos, float2 v) {
        if (ok) o[((size_t)pos * N + ky) * NH + kx] = v;
      };
      cgfft::transform<N, PL::FR, PL::F0, PL::F1, PL::F2, 1, FSH<TX>>(t, tw + TW_F, ld, st, sm);
      __syncthreads();
    }
  }
}

/* Pass 2: in-place column transform along y (inverse, S = 1, or forward,
 * S = -1).  grid = (ceil(NH/TX), N, nf). */
template <int TX, int S>
__global__ void __launch_bounds__(TX *P) k_col_y(float2 *f0, float2 *f1, float2 *f2,
                                                 const float4 *__restrict__ tw)
{
  extern __shared__ float2 smem[];
  const int c = threadIdx.x % TX, t = threadIdx.x / TX;
  const int kx = blockIdx.x * TX + c, z = blockIdx.y;
  const bool ok = kx < NH;
  float2 *f = blockIdx.z == 0 ? f0 : (blockIdx.z == 1 ? f1 : f2);
  float2 *base = f + (size_t)z * N * NH + kx;
  auto sm = [&](int slot) -> float2 & { return smem[slot * TX + c]; };
  auto ld = [&](int pos) -> float2 { return ok ? base[(size_t)pos * NH] : make_float2(0.0f, 0.0f); };
  auto st = [&](int pos, float2 v) {
    if (ok) base[(size_t)pos * NH] = v;
  };
  cgfft::transform<N, PL::CR, PL::C0, PL::C1, PL::C2, S, cgfft::NO_PAD>(t, tw + TW_C, ld, st, sm);
}

/* Forward pass 1 of the 2LPT source (density.c:739-759): row r2c along x of
 *   xx yy + xx zz + yy zz - xy^2 - xz^2 - yz^2,
 * formed as the rows of the six second derivatives (d: xx xy xz yy yz zz) are
 * loaded, into the rows of zz (a block reads its rows before it writes them).
 * A row's N reals are read as N/2 complex z_j = x_2j + i x_2j+1, transformed
 * forward, and split into the N/2 + 1 modes
 *   X_k = (E_k - i e^{-2 pi i k/N} O_k) / 2,  E_k = Z_k + conj Z_{N/2-k},
 *   O_k = Z_k - conj Z_{N/2-k}  (Z_{N/2} = Z_0).
 * The half-length spectrum goes to its own shared buffer: the exchange
 * buffer may still be read by other threads when the last stage stores.
 * Bound by the six reads: 106 us at 256^3, 115 with the source in a kernel of
 * its own. */
struct Lpt6 {
  float2 *d[6];
};

__device__ __forceinline__ float lpt2_source(float a, float e, float f, float b, float g, float d)
{
  const float v = CG_ADD(CG_ADD(CG_MUL(a, b), CG_MUL(a, d)), CG_MUL(b, d));
  return CG_SUB(CG_SUB(CG_SUB(v, CG_MUL(e, e)), CG_MUL(f, f)), CG_MUL(g, g));
}

__global__ void __launch_bounds__(PL::RB *PR) k_row_r2c(Lpt6 in, const float2 *__restrict__ twN,
                                                        const float4 *__restrict__ tw)
{
  extern __shared__ __align__(16) float2 smem[];
  float2 *zb = smem + PL::RB * ROWS;
  const int t = threadIdx.x % PR, rl = threadIdx.x / PR;
  /* the block's rows are contiguous: their source at a stride of NH, as the c2r
   * rows of k_row_c2r, before the transform exchanges at the stride ROWS */
  const size_t b0 = (size_t)blockIdx.x * PL::RB * NH;
#pragma unroll 2
  for (int i = threadIdx.x; i < PL::RB * NH; i += PL::RB * PR) {
    const float2 a = in.d[0][b0 + i], e = in.d[1][b0 + i], f = in.d[2][b0 + i];
    const float2 b = in.d[3][b0 + i], g = in.d[4][b0 + i], d = in.d[5][b0 + i];
    smem[i] = make_float2(lpt2_source(a.x, e.x, f.x, b.x, g.x, d.x), lpt2_source(a.y, e.y, f.y, b.y, g.y, d.y));
  }
  __syncthreads();
  const float2 *rin = smem + rl * NH;
  float2 *row = smem + rl * ROWS;
  float2 *z = zb + rl * LH;
  auto ld = [&](int j) -> float2 { return rin[j]; };
  auto sm = [&](int slot) -> float2 & { return row[slot]; };
  auto st = [&](int n, float2 v) { z[n] = v; };
  cgfft::transform<LH, PL::RR, PL::R0, PL::R1, PL::R2, -1, SHX>(t, tw + TW_R, ld, st, sm);
  __syncthreads();
  float2 *dst = in.d[5] + b0 + (size_t)rl * NH;
  for (int k = t; k <= LH; k += PR) {
    const float2 a = z[k == LH ? 0 : k], b = z[k == 0 ? 0 : LH - k];
    const float2 e = make_float2(a.x + b.x, a.y - b.y), o = make_float2(a.x - b.x, a.y + b.y);
    const float2 w = __ldg(&twN[k]); /* exp(+2 pi i k/N); the split takes its conjugate */
    const float2 wo = make_float2(w.x * o.x + w.y * o.y, w.x * o.y - w.y * o.x);
    dst[k] = make_float2(0.5f * (e.x + wo.y), 0.5f * (e.y - wo.x));
  }
}

/* Forward z pass of the 2LPT source with the second-order displacement
 * fill (density.c:764-809): per column (kx, ky) the forward transform along
 * z into shared memory, then for each axis a the product
 * -i k_a S_k / (N^3 k^2) (0 at k = 0) transformed back along z.
 * grid = (ceil(NH/TX), N). */
template <int TX>
__global__ void __launch_bounds__(TX *PF) k_z_lpt2(const float2 *__restrict__ src, float2 *o0, float2 *o1,
                                                   float2 *o2, float dk, float inv_n3,
                                                   const float4 *__restrict__ tw)
{
  extern __shared__ float2 smem[];
  float2 *X = smem + (size_t)EXF<TX> * TX;
  const int c = threadIdx.x % TX, t = threadIdx.x / TX;
  const int kx = blockIdx.x * TX + c, ky = blockIdx.y;
  const bool ok = kx < NH;
  auto sm = [&](int slot) -> float2 & { return smem[slot * TX + c]; };
  auto ld = [&](int pos) -> float2 { return ok ? src[((size_t)pos * N + ky) * NH + kx] : make_float2(0.0f, 0.0f); };
  auto stx = [&](int pos, float2 v) { X[pos * TX + c] = v; };
  cgfft::transform<N, PL::FR, PL::F0, PL::F1, PL::F2, -1, FSH<TX>>(t, tw + TW_F, ld, stx, sm);
  __syncthreads();
  float2 *outs[3] = {o0, o1, o2};
  const float kxf = (float)kx * dk, kyf = kcomp(ky, N, dk);
#pragma unroll 1
  for (int a = 0; a < 3; a++) {
    auto ld2 = [&](int pos) -> float2 {
      const float kzf = kcomp(pos, N, dk);
      const float k2 = kxf * kxf + kyf * kyf + kzf * kzf;
      if (!(k2 > 0.0f)) return make_float2(0.0f, 0.0f);
      const float ka = a == 0 ? kxf : (a == 1 ? kyf : kzf);
      const float g = ka * inv_n3 / k2;
      const float2 v = X[pos * TX + c];
      return make_float2(g * v.y, -g * v.x); /* -i g v */
    };
    float2 *o = outs[a];
    auto st = [&](int pos, float2 v) {
      if (ok) o[((size_t)pos * N + ky) * NH + kx] = v;
    };
    cgfft::transform<N, PL::FR, PL::F0, PL::F1, PL::F2, 1, FSH<TX>>(t, tw + TW_F, ld2, st, sm);
    __syncthreads();
  }
}

/* Pass 3: row c2r along x with normalisation and optional moment sums of the
 * first field, RB rows per block.  grid = (N*N/RB, nf).  partials[blockIdx.x] =
 * (sum d, sum d^2). */
template <bool STATS, int RB>
__global__ void __launch_bounds__(RB *PR) k_row_c2r(float2 *f0, float2 *f1, float2 *f2, float norm,
                                                        double2 *partials, const float2 *__restrict__ twN,
                                                        const float4 *__restrict__ tw, unsigned int *err)
{
  extern __shared__ __align__(16) float2 smem[];
  __shared__ uint64_t bar;
  const int t = threadIdx.x % PR, rl = threadIdx.x / PR;
  float2 *f = blockIdx.y == 0 ? f0 : (blockIdx.y == 1 ? f1 : f2);
  const size_t row0 = (size_t)blockIdx.x * RB;
  /* the block's rows, contiguous in HBM (RB NH float2, a multiple of 16
   * bytes at a 16-byte boundary since RB is even), in one bulk copy; they
   * land at a stride of NH and the transform then exchanges through the
   * same buffer at the padded stride ROWS, once every input is loaded */
  if (!cgtma::stage_rows(smem, f + row0 * NH, (unsigned)(RB * NH * sizeof(float2)), &bar, err)) return;
  const float2 *rin = smem + rl * NH;
  float2 *row = smem + rl * ROWS;
  float2 *dst = f + (row0 + rl) * NH;
  auto ld = [&](int j) -> float2 {
    float2 a = rin[j], b = rin[LH - j];
    if (j == 0) {
      a.y = 0.0f;
      b.y = 0.0f;
    }
    float2 e = make_float2(a.x + b.x, a.y - b.y);
    float2 o = make_float2(a.x - b.x, a.y + b.y);
    float2 w = __ldg(&twN[j]);
    float2 ow = make_float2(o.x * w.x - o.y * w.y, o.x * w.y + o.y * w.x);
    return make_float2(e.x - ow.y, e.y + ow.x);
  };
  auto sm = [&](int slot) -> float2 & { return row[slot]; };
  float s1 = 0.0f, s2 = 0.0f;
  auto st = [&](int n, float2 v) {
    float2 r = make_float2(v.x * norm, v.y * norm);
    dst[n] = r;
    if (STATS) {
      s1 += r.x + r.y;
      s2 += r.x * r.x + r.y * r.y;
    }
  };
  cgfft::transform<LH, PL::RR, PL::R0, PL::R1, PL::R2, 1, SHX>(t, tw + TW_R, ld, st, sm);
  if (STATS && blockIdx.y == 0) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      s1 += __shfl_xor_sync(0xffffffffu, s1, o);
      s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    }
    __shared__ double red[2][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) {
      red[0][wid] = (double)s1;
      red[1][wid] = (double)s2;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      double a = 0.0, b = 0.0;
      for (int w = 0; w < (RB * PR + 31) / 32; w++) {
        a += red[0][w];
        b += red[1][w];
      }
      partials[blockIdx.x] = make_double2(a, b);
    }
  }
}

template <class K>
cudaError_t prep(K kern, size_t smem)
{
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

/* ---- tile candidates of the autotuner ----------------------------------
 * Each pass has up to three tile widths: variant 0 is the plan's (fft_plans.h),
 * 1 half of it, 2 twice it.  A variant is valid when its shared memory fits
 * in 200 KiB and its block in 1024 threads (x pass: an even row count, for
 * the 16-byte bulk copy).  Only the block shape changes: every column and
 * row goes through the same transform, so all variants give the same bits.
 * The x pass that also sums the moments keeps the plan's RB, since the
 * per-block partial sums depend on it. */
constexpr size_t SMEM_MAX = 200u * 1024u;
constexpr int tile_of(int def, int v) { return v == 1 ? def / 2 : (v == 2 ? def * 2 : def); }
constexpr size_t fill_smem(int T) { return (size_t)(cgfft::pad_len(N, fill_sh(T)) + N) * T * sizeof(float2); }
constexpr size_t y_smem(int T) { return (size_t)N * T * sizeof(float2); }
constexpr bool fill_ok(int T) { return T >= 1 && fill_smem(T) <= SMEM_MAX && T * PF <= 1024; }
constexpr bool y_ok(int T) { return T >= 1 && y_smem(T) <= SMEM_MAX && T * P <= 1024; }
constexpr bool x_ok(int R)
{
  return R >= 2 && R % 2 == 0 && ((size_t)N * N) % R == 0 && (size_t)R * ROWS * sizeof(float2) <= SMEM_MAX &&
         R * PR <= 1024;
}
static_assert(fill_ok(PL::TX2) && fill_ok(PL::TX3) && y_ok(PL::TXY) && x_ok(PL::RB), "plan out of limits");

template <int T>
cudaError_t fill2(const cg_field_launch *L)
{
  if constexpr (!fill_ok(T)) {
    return cudaErrorInvalidValue;
  } else {
    const size_t sm = fill_smem(T);
    cudaError_t e = prep(k_fill_z<T>, sm);
    if (e != cudaSuccess) return e;
    dim3 g((NH + T - 1) / T, N);
    k_fill_z<T><<<g, T * PF, sm, L->stream>>>(L->f[0], L->f[1], L->fill, L->tws);
    return cudaGetLastError();
  }
}

template <int T, int SETS>
cudaError_t fill3(const cg_field_launch *L)
{
  if constexpr (!fill_ok(T)) {
    return cudaErrorInvalidValue;
  } else {
    const size_t sm = fill_smem(T); /* one value per mode + the exchange buffer */
    cudaError_t e = prep(k_fill_z3<T, SETS>, sm);
    if (e != cudaSuccess) return e;
    dim3 g((NH + T - 1) / T, N);
    Lpt9 o;
    for (int j = 0; j < 9; j++) o.o[j] = j < 3 ? L->f[j] : L->f2[j - 3];
    k_fill_z3<T, SETS><<<g, T * PF, sm, L->stream>>>(o, L->fill, L->tws);
    return cudaGetLastError();
  }
}

template <int T, int S>
cudaError_t ypass(const cg_field_launch *L, float2 *a, float2 *b, float2 *c, int nf)
{
  if constexpr (!y_ok(T)) {
    return cudaErrorInvalidValue;
  } else {
    const size_t sm = y_smem(T);
    cudaError_t e = prep(k_col_y<T, S>, sm);
    if (e != cudaSuccess) return e;
    dim3 g((NH + T - 1) / T, N, nf);
    k_col_y<T, S><<<g, T * P, sm, L->stream>>>(a, b, c, L->tws);
    return cudaGetLastError();
  }
}

template <bool STATS, int R>
cudaError_t xpass(const cg_field_launch *L, float2 *a, float2 *b, float2 *c, int nf, float norm, double2 *part)
{
  if constexpr (!x_ok(R)) {
    return cudaErrorInvalidValue;
  } else {
    const size_t sm = (size_t)R * ROWS * sizeof(float2);
    cudaError_t e = prep(k_row_c2r<STATS, R>, sm);
    if (e != cudaSuccess) return e;
    dim3 g((unsigned)((size_t)N * N / R), nf);
    k_row_c2r<STATS, R><<<g, R * PR, sm, L->stream>>>(a, b, c, norm, part, L->twN, L->tws, L->err);
    return cudaGetLastError();
  }
}

cudaError_t fill2_v(const cg_field_launch *L, int v)
{
  switch (v) {
    case 1: return fill2<tile_of(PL::TX2, 1)>(L);
    case 2: return fill2<tile_of(PL::TX2, 2)>(L);
    default: return fill2<PL::TX2>(L);
  }
}

template <int SETS>
cudaError_t fill3_v(const cg_field_launch *L, int v)
{
  switch (v) {
    case 1: return fill3<tile_of(PL::TX3, 1), SETS>(L);
    case 2: return fill3<tile_of(PL::TX3, 2), SETS>(L);
    default: return fill3<PL::TX3, SETS>(L);
  }
}

template <int S>
cudaError_t ypass_v(const cg_field_launch *L, int v, float2 *a, float2 *b, float2 *c, int nf)
{
  switch (v) {
    case 1: return ypass<tile_of(PL::TXY, 1), S>(L, a, b, c, nf);
    case 2: return ypass<tile_of(PL::TXY, 2), S>(L, a, b, c, nf);
    default: return ypass<PL::TXY, S>(L, a, b, c, nf);
  }
}

cudaError_t xpass_v(const cg_field_launch *L, int v, float2 *a, float2 *b, float2 *c, int nf)
{
  switch (v) {
    case 1: return xpass<false, tile_of(PL::RB, 1)>(L, a, b, c, nf, L->norm, nullptr);
    case 2: return xpass<false, tile_of(PL::RB, 2)>(L, a, b, c, nf, L->norm, nullptr);
    default: return xpass<false, PL::RB>(L, a, b, c, nf, L->norm, nullptr);
  }
}

} /* namespace */

#define CG_CAT2(a, b) a##b
#define CG_CAT(a, b) CG_CAT2(a, b)

/* Gaussian density and potential: passes 1-3 on both grids. */
extern "C" cudaError_t CG_CAT(cg_field_gauss_, CG_N)(const cg_field_launch *L)
{
  using namespace cg;
  cudaError_t e;
  if ((e = fill2_v(L, L->var[CG_PASS_FILL2])) != cudaSuccess) return e;
  if (L->ev) cudaEventRecord(L->ev[0], L->stream);
  if ((e = ypass_v<1>(L, L->var[CG_PASS_Y], L->f[0], L->f[1], nullptr, 2)) != cudaSuccess) return e;
  if (L->ev) cudaEventRecord(L->ev[1], L->stream);
  /* the moments' pass, which keeps the plan's rows, takes the potential along
   * up to 512^3, where a launch's fill and drain cost more than the tuned row
   * count gives: both 10.6 -> 7.6 us at 64^3, 60 -> 54 at 256^3, 330 -> 321 at
   * 512^3, but 2.76 -> 2.79 ms at 1024^3.  A width forced for the potential's
   * pass keeps that pass to itself. */
  const int nf = N <= CG_FIELD_X_BOTH && !L->x_own ? 2 : 1;
  if ((e = xpass<true, PL::RB>(L, L->f[0], L->f[1], nullptr, nf, L->norm, L->partials)) != cudaSuccess) return e;
  if (nf == 1 && (e = xpass_v(L, L->var[CG_PASS_X], L->f[1], nullptr, nullptr, 1)) != cudaSuccess) return e;
  if (L->ev) cudaEventRecord(L->ev[2], L->stream);
  return cudaGetLastError();
}

/* 1LPT displacement fields Psi_x,y,z: passes 1-3 on three grids; with L->f2[0]
 * set, pass 1 also of the second derivatives in L->f2 (cg_field_lpt2_). */
extern "C" cudaError_t CG_CAT(cg_field_lpt_, CG_N)(const cg_field_launch *L)
{
  using namespace cg;
  cudaError_t e;
  /* nine fields from one draw are tuned apart from three: the half tile that
   * wins with three loses with nine (256^3: 303 against 248 us, three fills 312) */
  e = L->f2[0] ? fill3_v<3>(L, L->var[CG_PASS_FILL9]) : fill3_v<1>(L, L->var[CG_PASS_FILL3]);
  if (e != cudaSuccess) return e;
  if (L->ev) cudaEventRecord(L->ev[0], L->stream);
  if ((e = ypass_v<1>(L, L->var[CG_PASS_Y], L->f[0], L->f[1], L->f[2], 3)) != cudaSuccess) return e;
  if (L->ev) cudaEventRecord(L->ev[1], L->stream);
  if ((e = xpass_v(L, L->var[CG_PASS_X], L->f[0], L->f[1], L->f[2], 3)) != cudaSuccess) return e;
  if (L->ev) cudaEventRecord(L->ev[2], L->stream);
  return cudaGetLastError();
}

/* 2LPT second-order displacements from the second derivatives L->f2, which
 * cg_field_lpt_ has filled (xx xy xz yy yz zz, destroyed): their y and x passes,
 * the source with its r2c along x, forward y, the fused z pass into L->f2[0..2],
 * then the inverse y and x passes of those three grids. */
extern "C" cudaError_t CG_CAT(cg_field_lpt2_, CG_N)(const cg_field_launch *L)
{
  using namespace cg;
  constexpr int TX3 = PL::TX3;
  size_t smr = (size_t)PL::RB * (ROWS + LH) * sizeof(float2);
  size_t smz = fill_smem(TX3);
  cudaError_t e;
  if ((e = prep(k_row_r2c, smr)) != cudaSuccess) return e;
  if ((e = prep(k_z_lpt2<TX3>, smz)) != cudaSuccess) return e;
  dim3 gr((unsigned)((size_t)N * N / PL::RB), 1);
  cg_field_launch L1 = *L;
  L1.norm = 1.0f;
  const int vy = L->var[CG_PASS_Y], vx = L->var[CG_PASS_X];
  Lpt6 in;
  for (int a = 0; a < 6; a++) in.d[a] = L->f2[a];
  float2 **f = in.d, *src = in.d[5];
  for (int a = 0; a < 6; a += 3)
    if ((e = ypass_v<1>(L, vy, f[a], f[a + 1], f[a + 2], 3)) != cudaSuccess ||
        (e = xpass_v(&L1, vx, f[a], f[a + 1], f[a + 2], 3)) != cudaSuccess)
      return e;
  k_row_r2c<<<gr, PL::RB * PR, smr, L->stream>>>(in, L->twN, L->tws);
  if ((e = ypass_v<-1>(L, vy, src, nullptr, nullptr, 1)) != cudaSuccess) return e;
  dim3 gz((NH + TX3 - 1) / TX3, N);
  const float inv_n3 = 1.0f / ((float)N * (float)N * (float)N);
  k_z_lpt2<TX3><<<gz, TX3 * PF, smz, L->stream>>>(src, f[0], f[1], f[2], L->fill.dk, inv_n3, L->tws);
  if ((e = ypass_v<1>(L, vy, f[0], f[1], f[2], 3)) != cudaSuccess) return e;
  if ((e = xpass_v(&L1, vx, f[0], f[1], f[2], 3)) != cudaSuccess) return e;
  return cudaGetLastError();
}

/* The transforms' stage tables (cg_field_launch.tws) from the roots of unity of
 * orders N and N/2; out may be NULL.  Returns their number of float4. */
extern "C" int CG_CAT(cg_field_tables_, CG_N)(const float2 *twN, const float2 *twH, float4 *out)
{
  if (out) {
    cgfft::tw_build<N, PL::C0, PL::C1, PL::C2>(twN, out + TW_C);
    cgfft::tw_build<N, PL::F0, PL::F1, PL::F2>(twN, out + TW_F);
    cgfft::tw_build<LH, PL::R0, PL::R1, PL::R2>(twH, out + TW_R);
  }
  return TW_LEN;
}

/* Number of blocks of the moment-sum pass (size of the partials array). */
extern "C" size_t CG_CAT(cg_field_npartials_, CG_N)(void) { return (size_t)N * N / PL::RB; }

/* Tile width of variant v of a pass (CG_PASS_*), or 0 when the variant is
 * not valid at this size. */
extern "C" int CG_CAT(cg_field_tile_, CG_N)(int pass, int v)
{
  if (v < 0 || v > 2) return 0;
  switch (pass) {
    case CG_PASS_FILL2: return fill_ok(tile_of(PL::TX2, v)) ? tile_of(PL::TX2, v) : 0;
    case CG_PASS_FILL3:
    case CG_PASS_FILL9: return fill_ok(tile_of(PL::TX3, v)) ? tile_of(PL::TX3, v) : 0;
    case CG_PASS_Y: return y_ok(tile_of(PL::TXY, v)) ? tile_of(PL::TXY, v) : 0;
    case CG_PASS_X: return x_ok(tile_of(PL::RB, v)) ? tile_of(PL::RB, v) : 0;
  }
  return 0;
}

/* One pass alone with variant v, for timing: the fills write f[0..1] (two
 * fields), f[0..2] (three) or these and f2[0..5] (nine); the y and x passes transform f[0..nf-1] in
 * place (inverse, no moment sums). */
extern "C" cudaError_t CG_CAT(cg_field_pass_, CG_N)(const cg_field_launch *L, int pass, int v, int nf)
{
  switch (pass) {
    case CG_PASS_FILL2: return fill2_v(L, v);
    case CG_PASS_FILL3: return fill3_v<1>(L, v);
    case CG_PASS_FILL9: return fill3_v<3>(L, v);
    case CG_PASS_Y: return ypass_v<1>(L, v, L->f[0], nf > 1 ? L->f[1] : nullptr, nf > 2 ? L->f[2] : nullptr, nf);
    case CG_PASS_X: return xpass_v(L, v, L->f[0], nf > 1 ? L->f[1] : nullptr, nf > 2 ? L->f[2] : nullptr, nf);
  }
  return cudaErrorInvalidValue;
}
