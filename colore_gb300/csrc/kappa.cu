/*
 * kappa.cu -- lensing convergence on source planes
 * (kappa_get_beam_properties, kappa.c:78-175).
 *
 * One thread per HEALPix pixel (NEST id, as listed by hp_shell_alloc,
 * common.c:505-552) marches the N/2 radial steps of the line of sight,
 * samples the tidal tensor of the potential at the nearest grid cell
 * (get_element, beaming.c:84-116; interpolate_from_grid NGP branch,
 * beaming.c:148-182), projects it on the transverse directions and
 * accumulates the two radial moments.  At each source-plane boundary it
 * writes kappa_1 - kappa_2 / r_plane straight into RING order (the
 * nest-to-ring reordering of write_kappa, io.c:826-873).  Threads of a warp
 * hold neighbouring NEST pixels, so their rays stay close and the 19-point
 * stencil reads hit L1/L2.  The radial sums use Kahan compensation.
 * k_isw integrates the ISW maps along the same rays, k_cstm the custom maps.
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include "cg_dev.cuh"
#include "kappa_api.h"

namespace {
using namespace cg;

/* Nearest grid cell of step radius rm along axis a, before the periodic wrap
 * (cg_ngp_cell). */
__device__ __forceinline__ int step_cell(float rm, float u, float po, float idx)
{
  return (int)CG_ADD(CG_MUL(CG_ADD(CG_MUL(rm, u), po), idx), 0.5f);
}

/* The 19 potentials around a cell away from the box faces, in the order
 * cg_tidal takes them.  IDX32: the cell's byte offset fits 32 bits, so one
 * register addresses all nine rows from uniform bases. */
template <bool IDX32>
__device__ __forceinline__ void stencil_inside(const float *__restrict__ phi, int x, int y, int z, int ngx, int N,
                                               float f[19])
{
  const long long plane = (long long)ngx * N;
  if (IDX32) {
    const unsigned o = ((unsigned)z * (unsigned)plane + (unsigned)y * (unsigned)ngx + (unsigned)x) * 4u;
    const char *b = reinterpret_cast<const char *>(phi);
    const long long py = (long long)ngx * 4, pz = plane * 4;
#define CG_AT(base, dx) __ldg(reinterpret_cast<const float *>((b + (base)) + o) + (dx))
    f[0] = CG_AT(0, 0);
    f[1] = CG_AT(0, 1);
    f[2] = CG_AT(0, -1);
    f[3] = CG_AT(py, 0);
    f[4] = CG_AT(-py, 0);
    f[5] = CG_AT(pz, 0);
    f[6] = CG_AT(-pz, 0);
    f[7] = CG_AT(py, 1);
    f[8] = CG_AT(-py, -1);
    f[9] = CG_AT(-py, 1);
    f[10] = CG_AT(py, -1);
    f[11] = CG_AT(pz, 1);
    f[12] = CG_AT(-pz, -1);
    f[13] = CG_AT(-pz, 1);
    f[14] = CG_AT(pz, -1);
    f[15] = CG_AT(pz + py, 0);
    f[16] = CG_AT(-pz - py, 0);
    f[17] = CG_AT(-pz + py, 0);
    f[18] = CG_AT(pz - py, 0);
#undef CG_AT
  } else {
    const float *c = phi + (long long)z * plane + ((long long)y * ngx + x);
    const float *yp = c + ngx, *ym = c - ngx, *zp = c + plane, *zm = c - plane;
    f[0] = __ldg(c);
    f[1] = __ldg(c + 1);
    f[2] = __ldg(c - 1);
    f[3] = __ldg(yp);
    f[4] = __ldg(ym);
    f[5] = __ldg(zp);
    f[6] = __ldg(zm);
    f[7] = __ldg(yp + 1);
    f[8] = __ldg(ym - 1);
    f[9] = __ldg(ym + 1);
    f[10] = __ldg(yp - 1);
    f[11] = __ldg(zp + 1);
    f[12] = __ldg(zm - 1);
    f[13] = __ldg(zm + 1);
    f[14] = __ldg(zp - 1);
    f[15] = __ldg(zp + ngx);
    f[16] = __ldg(zm - ngx);
    f[17] = __ldg(zm + ngx);
    f[18] = __ldg(zp - ngx);
  }
}

/* Convergence along the ray of each NEST pixel.  Bound by instruction issue
 * where the rays are dense (nside 1024 on 512^3: 87 % issue-active) and by L1
 * wavefronts where they lie a cell apart (nside 512 on 1024^3: 81 % of the L1
 * data pipe).  Steps whose cells lie off the box faces take no bounds test and
 * no wrap, the step's radius and factors come in one shared-memory load: 13.4
 * -> 11.5 ms for the former, the latter unchanged (12.9 ms). */
template <bool IDX32, int KT>
__global__ void __launch_bounds__(KT, 1024 / KT) k_kappa(const float *__restrict__ phi, cg_kappa_params p)
{
  extern __shared__ float4 kst[]; /* per step: radius and the two radial factors */
  for (int i = threadIdx.x; i < p.nr; i += blockDim.x)
    kst[i] = make_float4(CG_MUL(CG_ADD((float)i, 0.5f), p.dr), p.fac1[i], p.fac2[i], 0.0f);
  __syncthreads();
  const long long ip = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (ip >= p.npix) return;
  const int N = p.box.N, ngx = 2 * (N / 2 + 1);
  float u[3], rot[6];
  cg_pix2vec_nest(p.nside, ip, u);
  cg_kappa_rot(u, CG_MUL(p.box.idx, p.box.idx), rot);
  /* the factor 1/4 of the mixed derivatives (cg_tidal), exact in either place */
  const float r4[6] = {rot[0], CG_MUL(0.25f, rot[1]), CG_MUL(0.25f, rot[2]), rot[3], CG_MUL(0.25f, rot[4]), rot[5]};
  const float po[3] = {p.box.p0, p.box.p1, p.box.p2};
  const float idx = p.box.idx;
  /* Along a ray each cell index moves one way, so when the first and the
   * in'th step's cells lie off the box faces, all between them do. */
  auto inside = [&](int k) {
    bool ok = true;
    const float rm = kst[k].x;
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const int i = step_cell(rm, u[a], po[a], idx);
      ok = ok && i > 0 && i < N - 1;
    }
    return ok;
  };
  int in = p.ir_max[p.nplanes - 1];
  if (!inside(0)) in = -1;
  while (in >= 0 && !inside(in)) in--;
  float k1 = 0.0f, k1c = 0.0f, k2 = 0.0f, k2c = 0.0f;
  for (int pl = 0; pl < p.nplanes; pl++) {
    const int irmax = p.ir_max[pl];
    int irr = p.ir_min[pl];
    const int e = min(irmax, in);
    for (; irr <= e; irr++) {
      const float4 s = kst[irr];
      float f[19];
      stencil_inside<IDX32>(phi, step_cell(s.x, u[0], po[0], idx), step_cell(s.x, u[1], po[1], idx),
                            step_cell(s.x, u[2], po[2], idx), ngx, N, f);
      const float two0 = CG_MUL(2.0f, f[0]);
      const float t[6] = {CG_SUB(CG_ADD(f[1], f[2]), two0), CG_SUB(CG_SUB(CG_ADD(f[7], f[8]), f[9]), f[10]),
                          CG_SUB(CG_SUB(CG_ADD(f[11], f[12]), f[13]), f[14]), CG_SUB(CG_ADD(f[3], f[4]), two0),
                          CG_SUB(CG_SUB(CG_ADD(f[15], f[16]), f[17]), f[18]), CG_SUB(CG_ADD(f[5], f[6]), two0)};
      const float dot = cg_dot6(r4, t);
      cg_kahan_add(&k1, &k1c, CG_MUL(dot, s.y));
      cg_kahan_add(&k2, &k2c, CG_MUL(dot, s.z));
    }
    for (; irr <= irmax; irr++) { /* at the box faces */
      const float4 s = kst[irr];
      float f[19], t[6];
      stencil19(phi, cg_ngp_cell(s.x, u[0], po[0], idx, N), cg_ngp_cell(s.x, u[1], po[1], idx, N),
                cg_ngp_cell(s.x, u[2], po[2], idx, N), N, f);
      cg_tidal(f, t);
      const float dot = cg_dot6(rot, t);
      cg_kahan_add(&k1, &k1c, CG_MUL(dot, s.y));
      cg_kahan_add(&k2, &k2c, CG_MUL(dot, s.z));
    }
    p.map[(long long)pl * p.npix + cg_nest2ring(p.nside, ip)] = CG_SUB(k1, CG_MUL(p.inv_r_max[pl], k2));
  }
}

/* isw_get_beam_properties (isw.c:78-147): the same rays, the potential at the
 * nearest cell (RETURN_PDOT, beaming.c:81-82, 145-180) weighted by
 * fac1 = 2 PD(r) dr, cumulative over the sorted planes. */
__global__ void __launch_bounds__(256) k_isw(const float *__restrict__ phi, cg_kappa_params p)
{
  extern __shared__ float ksh[];
  float *f1 = ksh;
  for (int i = threadIdx.x; i < p.nr; i += blockDim.x) f1[i] = p.fac1[i];
  __syncthreads();
  const long long ip = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (ip >= p.npix) return;
  const int N = p.box.N;
  const int ngx = 2 * (N / 2 + 1);
  const size_t plane = (size_t)ngx * N;
  float u[3];
  cg_pix2vec_nest(p.nside, ip, u);
  const float po[3] = {p.box.p0, p.box.p1, p.box.p2};
  const long long ring = cg_nest2ring(p.nside, ip);
  float acc = 0.0f, cmp = 0.0f;
  for (int pl = 0; pl < p.nplanes; pl++) {
    const int irmin = p.ir_min[pl], irmax = p.ir_max[pl];
    for (int irr = irmin; irr <= irmax; irr++) {
      const float rm = CG_MUL(CG_ADD((float)irr, 0.5f), p.dr);
      const int x0 = cg_ngp_cell(rm, u[0], po[0], p.box.idx, N);
      const int y0 = cg_ngp_cell(rm, u[1], po[1], p.box.idx, N);
      const int z0 = cg_ngp_cell(rm, u[2], po[2], p.box.idx, N);
      const float pd = __ldg(phi + (size_t)z0 * plane + y0 * ngx + x0);
      cg_kahan_add(&acc, &cmp, CG_MUL(pd, f1[irr]));
    }
    p.map[(long long)pl * p.npix + ring] = acc;
  }
}

/* cstm_get_beam_properties (cstm.c:68-145): one NEST pixel per thread, the
 * density interpolated trilinearly at each step centre of the kernel's
 * support, written back in NEST order as write_cstm stores it
 * (io.c:754-800 copies the shell data without reordering). */
__global__ void __launch_bounds__(256) k_cstm(const float *__restrict__ dens, cg_cstm_params p)
{
  extern __shared__ float csh[];
  const int ns = p.ir_max - p.ir_min + 1;
  float *kz = csh, *bz = csh + ns, *nm = csh + 2 * ns;
  for (int i = threadIdx.x; i < ns; i += blockDim.x) {
    const int irr = p.ir_min + i;
    kz[i] = p.kz[irr];
    bz[i] = p.bz[irr];
    nm[i] = bgn(p.norm, p.g, CG_MUL(CG_ADD((float)irr, 0.5f), p.dr));
  }
  __syncthreads();
  const long long ip = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (ip >= p.npix) return;
  const int N = p.box.N;
  float u[3];
  cg_pix2vec_nest(p.nside, ip, u);
  const float po[3] = {p.box.p0, p.box.p1, p.box.p2};
  float acc = 0.0f, cmp = 0.0f;
  for (int i = 0; i < ns; i++) {
    const float rm = CG_MUL(CG_ADD((float)(p.ir_min + i), 0.5f), p.dr);
    int i0[3], i1[3];
    float h0[3], h1[3];
#pragma unroll
    for (int a = 0; a < 3; a++) cg_cic_axis(rm, u[a], po[a], p.box.idx, N, &i0[a], &i1[a], &h0[a], &h1[a]);
    const float d = cg_cic_value(dens, i0, i1, h0, h1, N);
    cg_kahan_add(&acc, &cmp, CG_MUL(kz[i], CG_SUB(CG_MUL(cg_bias_model(d, bz[i], p.bias_model), nm[i]), 1.0f)));
  }
  p.map[ip] = CG_MUL(acc, p.dr);
}

} /* namespace */

cudaError_t cg_cstm_integrate(cudaStream_t s, const float *dens, const cg_cstm_params *p)
{
  long long blocks = (p->npix + 255) / 256;
  const size_t smem = 3 * sizeof(float) * (size_t)(p->ir_max - p->ir_min + 1);
  k_cstm<<<(unsigned)blocks, 256, smem, s>>>(dens, *p);
  return cudaGetLastError();
}

cudaError_t cg_isw_integrate(cudaStream_t s, const float *phi, const cg_kappa_params *p)
{
  size_t smem = (size_t)p->nr * sizeof(float);
  cudaError_t e = cudaFuncSetAttribute(k_isw, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  long long blocks = (p->npix + 255) / 256;
  k_isw<<<(unsigned)blocks, 256, smem, s>>>(phi, *p);
  return cudaGetLastError();
}

template <int KT>
static cudaError_t kappa_launch(cudaStream_t s, const float *phi, const cg_kappa_params *p)
{
  const size_t smem = (size_t)p->nr * sizeof(float4);
  const long long N = p->box.N, bytes = (2 * (N / 2 + 1)) * N * N * 4;
  auto k = bytes < 0x100000000ll ? k_kappa<true, KT> : k_kappa<false, KT>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k<<<(unsigned)((p->npix + KT - 1) / KT), KT, smem, s>>>(phi, *p);
  return cudaGetLastError();
}

cudaError_t cg_kappa_integrate(cudaStream_t s, const float *phi, const cg_kappa_params *p, int nsm)
{
  /* blocks of 256 neighbouring pixels share rows in L1 (nside 512 on 1024^3:
   * 12.9 ms, with 64 13.8 ms); maps of less than two waves of them (1024 rays
   * an SM), whose rays are bound by latency, take 64 for the balance (nside 128
   * on 256^3: 271 and 246 us) */
  return p->npix <= 2ll * nsm * 1024 ? kappa_launch<64>(s, phi, p) : kappa_launch<256>(s, phi, p);
}
