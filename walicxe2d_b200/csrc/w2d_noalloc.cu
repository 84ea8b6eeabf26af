// w2d_noalloc.cu -- the allocation-free CFL time step (w2d_timestep_noalloc).
//
// Some hosts cannot allocate device memory themselves: a Fortran program
// whose device arrays are owned by an OpenACC/OpenMP-offload runtime, or a
// code that runs the time loop under a memory manager that forbids
// cudaMalloc/cudaFree between its own set-up and tear-down.  They still own
// the block data on the device and want the CFL limit of timestep
// (src/timestep.f90:21-48) without a context (w2d_create allocates a pool).
//
// This entry point computes it with the same arithmetic as w2d_timestep: a
// per-block partial min(dx/(|u|+cs), dy/(|v|+cs)) over the interior cells,
// then dt = min(cfl*min(partials), 0.4*1e30*Psc/tsc).  The running minimum
// lives in a file-scope device array of W2D_NOALLOC_MAX_BLOCKS doubles (512 KB,
// held by every GPU that loads the library until the process exits); nothing
// is allocated per call.  Built with --fmad=false like the FP64 kernels.
#include <cuda_runtime.h>

#include <algorithm>

#include "../../include/w2d.h"
#include "w2d_phys.cuh"

namespace {

// [0] the complement of the least partial's bits, [1] of the first block (1
// based) with a level outside 1..nlevs, [2] CTAs done (64-bit words, all zero
// between calls); the results at W2D_NOALLOC_MAX_BLOCKS and the next index.
static __device__ __align__(256) double g_noalloc_scratch[W2D_NOALLOC_MAX_BLOCKS + 32];

struct Spacing {
  double dx[W2D_MAXLEV_NOALLOC + 1];
  double dy[W2D_MAXLEV_NOALLOC + 1];
};

__device__ __forceinline__ float sqrt_near(float x)
{
  float y;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// |u|+cs and |v|+cs of one cell, as k_dt's partials take them (NaN where the
// cell's values give NaN)
template <int NEQ>
__device__ __forceinline__ void cell_speeds(const double* __restrict__ ub, int c, const w2d::Phys<double>& ph,
                                            double& au, double& av)
{
  double uu[NEQ], q[NEQ], T;
#pragma unroll
  for (int k = 0; k < NEQ; ++k) uu[k] = ub[k * W2D_CELLS + c];
  w2d::uprim<NEQ>(ph, q, uu, T);
  const double cs = w2d::sound(ph, q[3], q[0]);
  au = fabs(q[1]) + cs;
  av = fabs(q[2]) + cs;
}

// Bounds of the same two speeds in FP32 (lo <= exact <= hi): the conversions,
// products and roots below err by less than 1e-6 relative each, and the pressure
// by less than 2e-6 of the energies it is the difference of.  Values whose
// ranges or NaNs void that give (0, inf).
struct Bounds {
  float ulo, uhi, vlo, vhi;
};
template <bool H>
__device__ __forceinline__ Bounds cell_bounds(double d0, double d1, double d2, double d3, double d4,
                                              const w2d::Phys<double>& ph)
{
  const float r = fmaxf((float)d0, 1e-15f), mx = (float)d1, my = (float)d2, E = (float)d3;
  const float inv = __fdividef(1.f, r), u = fabsf(mx * inv), v = fabsf(my * inv);
  const float ke = 0.5f * (fabsf(mx) * u + fabsf(my) * v), er = 2e-6f * (fabsf(E) + ke);
  const float icv = 1.f / (float)ph.cv, g = (float)ph.gamma * inv;
  float plo = fmaxf((E - ke - er) * icv, 0.f), phi = fmaxf((E - ke + er) * icv, 1.1e-15f);
  // coolingh: the pressure of T >= 1 (uprim).  Its density 2 rho - u5 can cancel:
  // three roundings of 2^-24 of the terms, not of the difference
  if (H) {
    const float n = (float)d4, dent = 2.f * r - n + 2.5e-7f * (2.f * r + fabsf(n));
    phi = fmaxf(phi, 1.00001f * fmaxf(dent, 1e-15f) / (float)ph.tempsc);
  }
  const float clo = sqrt_near(g * plo) * (1.f - 4e-6f), chi = sqrt_near(g * phi) * (1.f + 4e-6f);
  const bool fit = ph.cv > 1e-3 && ph.cv < 1e3 && ph.gamma > 1e-3 && ph.gamma < 1e3 &&
                   (!H || (ph.tempsc > 1e-12 && ph.tempsc < 1e30)) && r <= 1e15f && fabsf(E) <= 1e15f && fabsf(E) >= 1e-12f && fabsf(mx) <= 1e15f && fabsf(my) <= 1e15f &&
                   (!H || fabs(d4) <= 1e15);
  if (!fit) return {0.f, INFINITY, 0.f, INFINITY};
  return {u * (1.f - 4e-6f) + clo, u * (1.f + 4e-6f) + chi, v * (1.f - 4e-6f) + clo, v * (1.f + 4e-6f) + chi};
}

// A CTA's minimum and first bad block into the words; the last CTA of the grid
// writes the results and leaves the words zero.  One thread of a CTA.
__device__ __forceinline__ void cfl_finish(double m, int bad, double courant, double psc, double tsc,
                                           unsigned long long* __restrict__ work, double* __restrict__ out)
{
  // complements: zero is the neutral value of the maximum, and what the last
  // CTA leaves behind (the partials are positive, so their bits order as they do)
  atomicMax(&work[0], ~(unsigned long long)__double_as_longlong(m));
  if (bad) atomicMax(&work[1], ~(unsigned long long)bad);
  __threadfence();
  if (atomicAdd(&work[2], 1ull) + 1ull != gridDim.x) return;
  __threadfence();
  m = __longlong_as_double((long long)~atomicExch(&work[0], 0ull));
  const unsigned long long wb = atomicExch(&work[1], 0ull);
  work[2] = 0ull;
  const double a = courant * m;
  const double c = 0.4 * 1e30 * psc / tsc;
  out[0] = (a < c) ? a : c;
  out[1] = wb ? (double)~wb : 0.;   // a block ID with a bad level, or 0
}

// One block per CTA, a thread per cell, every cell in FP64: the shorter chain
// (one load, no bounds to rank) where the CTAs of the whole call are resident at
// once.  500 blocks are 26 us a call, of which the launch and the copy of the
// result are nearly all (28 with a second kernel for the minimum).
template <int NEQ>
__global__ void __launch_bounds__(256) k_cfl_few(const double* __restrict__ u, const int32_t* __restrict__ lev,
                                                 int nlevs, Spacing sp, w2d::Phys<double> ph, double courant,
                                                 double psc, double tsc, unsigned long long* __restrict__ work,
                                                 double* __restrict__ out)
{
  __shared__ double red[2][8];
  const int b = blockIdx.x, t = threadIdx.x;
  const int l = lev[b];
  double au, av;
  cell_speeds<NEQ>(u + (size_t)b * NEQ * W2D_CELLS, (2 + t / 16) * W2D_W + 2 + t % 16, ph, au, av);
  au = w2d::warp_max0(fmax(au, 0.));   // (NaN: left out)
  av = w2d::warp_max0(fmax(av, 0.));
  if ((t & 31) == 0) {
    red[0][t >> 5] = au;
    red[1][t >> 5] = av;
  }
  __syncthreads();
  if (t != 0) return;
  for (int w = 1; w < 8; ++w) {
    au = fmax(au, red[0][w]);
    av = fmax(av, red[1][w]);
  }
  double m = 1.e30;
  int bad = b + 1;
  if (l >= 1 && l <= nlevs) {
    const double part = fmin(sp.dx[l] / au, sp.dy[l] / av);
    if (!(part < 0.)) {   // (a negative spacing)
      m = fmin(m, part + 0.);
      bad = 0;
    }
  }
  cfl_finish(m, bad, courant, psc, tsc, work, out);
}

// The minimum of the partials of the blocks this grid walks, a warp per block,
// lane l taking cells 2 (l % 8) and the next of rows l / 8, 4 + l / 8, ... .
// For a positive x, RN(dx/x) falls with x, so a block's partial needs only the
// largest |u|+cs and |v|+cs.  FP32 bounds find the few cells that can hold
// them; those alone are computed in FP64, and of a lane's cells with the same
// values, which the bounds cannot rank, one (20,011 uniform blocks 80 -> 55 us a
// call, of 5 equations with coolingh 128 -> 68: what blocks of any values take).
// Where every block is flat to below 1e-6 and its cells yet differ, all are
// computed (82 us; with coolingh 117, a thread per cell took 96).
// Bound by the blocks' bytes: 205 MB of sectors for 20,011 blocks of 4 equations
// (every cell in FP64 with its own divisions, one CTA per block, a second kernel
// for the minimum: 86 us a call; so 60, the kernel 41.5).  VEC: 16-byte loads (u on a 16-byte
// boundary).
template <int NEQ, bool H, bool VEC>
__global__ void __launch_bounds__(256) k_cfl_min(const double* __restrict__ u, const int32_t* __restrict__ lev,
                                                 int nblocks, int nlevs, Spacing sp, w2d::Phys<double> ph,
                                                 double courant, double psc, double tsc,
                                                 unsigned long long* __restrict__ work, double* __restrict__ out)
{
  __shared__ double red[8];
  __shared__ int redb[8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int at = (2 + lane / 8) * W2D_W + 2 + 2 * (lane % 8);   // first of the lane's cells in its first row
  double m = 1.e30;
  int bad = 0;                     // first block (1-based) with a bad level
  for (int b = blockIdx.x * 8 + warp; b < nblocks; b += gridDim.x * 8) {
    const double* ub = u + (size_t)b * NEQ * W2D_CELLS;
    constexpr int NL = H && NEQ > 4 ? 5 : 4;   // (uprim takes the density where there is no fifth equation)
    double x[4][NL][2];
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int e = 0; e < NL; ++e) {
        const double* p = ub + e * W2D_CELLS + at + k * 4 * W2D_W;
        if (VEC) {
          const double2 t = *reinterpret_cast<const double2*>(p);
          x[k][e][0] = t.x;
          x[k][e][1] = t.y;
        } else {
          x[k][e][0] = p[0];
          x[k][e][1] = p[1];
        }
      }
    const int l = lev[b];
    if (l < 1 || l > nlevs) {
      if (bad == 0) bad = b + 1;
      continue;
    }
    // cells with the values of the lane's cell before them, whose speeds they share
    unsigned rep = 0;
#pragma unroll
    for (int c = 1; c < 8; ++c) {
      long long d = 0;
#pragma unroll
      for (int e = 0; e < NL; ++e)
        d |= __double_as_longlong(x[c >> 1][e][c & 1]) ^ __double_as_longlong(x[(c - 1) >> 1][e][(c - 1) & 1]);
      rep |= (unsigned)(d == 0) << c;
    }
    float uhi[8], vhi[8], ulo = 0.f, vlo = 0.f;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const double(*y)[2] = x[c >> 1];
      const int h = c & 1;
      const Bounds z = cell_bounds<H>(y[0][h], y[1][h], y[2][h], y[3][h], H ? y[NL == 5 ? 4 : 0][h] : 0., ph);
      uhi[c] = z.uhi;
      vhi[c] = z.vhi;
      ulo = fmaxf(ulo, z.ulo);
      vlo = fmaxf(vlo, z.vlo);
    }
    ulo = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(ulo)));
    vlo = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(vlo)));
    unsigned cand = 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) cand |= (unsigned)(!(uhi[c] < ulo) || !(vhi[c] < vlo)) << c;   // (NaN: a candidate)
    cand &= ~rep;
    double mu = 0., mv = 0.;
    while (__any_sync(0xffffffffu, cand != 0)) {
      if (cand) {
        const int c = __ffs(cand) - 1;
        cand &= cand - 1;
        double au, av;
        cell_speeds<NEQ>(ub, at + (c >> 1) * 4 * W2D_W + (c & 1), ph, au, av);
        mu = fmax(mu, au);
        mv = fmax(mv, av);
      }
    }
    mu = w2d::warp_max0(mu);
    mv = w2d::warp_max0(mv);
    const double part = fmin(sp.dx[l] / mu, sp.dy[l] / mv);
    if (part < 0.) {   // (a negative spacing)
      if (bad == 0) bad = b + 1;
      continue;
    }
    m = fmin(m, part + 0.);
  }
  if (lane == 0) {
    red[warp] = m;
    redb[warp] = bad;
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int w = 1; w < 8; ++w) {
    m = fmin(m, red[w]);
    if (redb[w] && (!bad || redb[w] < bad)) bad = redb[w];
  }
  cfl_finish(m, bad, courant, psc, tsc, work, out);
}

template <int NEQ, bool H>
void launch_cfl(const double* u, const int32_t* lev, int nblocks, const W2dParams* p, const Spacing& sp,
                const w2d::Phys<double>& ph, double* scratch)
{
  int dev = 0, nsm = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  auto* work = reinterpret_cast<unsigned long long*>(scratch);
  double* out = scratch + W2D_NOALLOC_MAX_BLOCKS;
  // Up to four CTAs per SM of one block each.  A call in us, k_cfl_few and
  // k_cfl_min: 500 blocks 26 and 32, 1,000 and 2,500 33 and 32 each, 5,000 35
  // and 33, 20,011 72 and 61.
  if (nblocks <= 4 * nsm) {
    k_cfl_few<NEQ><<<nblocks, 256>>>(u, lev, p->nlevs, sp, ph, p->cfl, p->psc, p->tsc, work, out);
    return;
  }
  // Three CTAs of 80 registers per SM, with coolingh two of up to 112 (20,011
  // blocks of 5 equations: on three per SM, one and a half waves, 75 us, so 68;
  // capped to three of 84 registers 83)
  const int grid = std::min((nblocks + 7) / 8, (H ? 2 : 3) * nsm);
  if (((uintptr_t)u & 15) == 0)
    k_cfl_min<NEQ, H, true><<<grid, 256>>>(u, lev, nblocks, p->nlevs, sp, ph, p->cfl, p->psc, p->tsc, work, out);
  else
    k_cfl_min<NEQ, H, false><<<grid, 256>>>(u, lev, nblocks, p->nlevs, sp, ph, p->cfl, p->psc, p->tsc, work, out);
}

// Device address of the scratch array in the caller's current device and
// context.  Looked up on every call (the lookup allocates nothing): after a
// device reset, or when an offload runtime tears its context down and builds
// a new one, the module is loaded again and the array can move, so an
// address kept from an earlier call could point at freed memory.
int scratch_for_current_device(double** out)
{
  void* ptr = nullptr;
  if (cudaGetSymbolAddress(&ptr, g_noalloc_scratch) != cudaSuccess || !ptr) return W2D_ERR_CUDA;
  *out = static_cast<double*>(ptr);
  return W2D_OK;
}

}  // namespace

extern "C" int w2d_timestep_noalloc(const W2dParams* p, const double* u, const int32_t* lev, int nblocks,
                                    const double* dx, const double* dy, double* dt)
{
  if (!p || !u || !lev || !dx || !dy || !dt) return W2D_ERR_ARG;
  if (nblocks < 1 || nblocks > W2D_NOALLOC_MAX_BLOCKS) return W2D_ERR_CAPACITY;
  if (p->neq < 4 || p->neq > 6 || p->precision != 64 || p->cooling == W2D_COOLINGDMC || p->nlevs < 1 ||
      p->nlevs > W2D_MAXLEV_NOALLOC || p->nx != W2D_NX || p->ny != W2D_NX)
    return W2D_ERR_ARG;
  double* scratch = nullptr;
  int rc = scratch_for_current_device(&scratch);
  if (rc) return rc;
  Spacing sp;
  for (int l = 0; l <= W2D_MAXLEV_NOALLOC; ++l) sp.dx[l] = sp.dy[l] = 0.0;
  for (int l = 1; l <= p->nlevs; ++l) {
    sp.dx[l] = dx[l - 1];
    sp.dy[l] = dy[l - 1];
  }
  w2d::Phys<double> ph;
  ph.cv = p->cv;
  ph.gamma = p->gamma;
  ph.tempsc = p->tempsc;
  ph.cooling = p->cooling;
  ph.hllc_compat = 0;
  ph.solver = p->solver;
  ph.limiter = p->limiter;
  ph.cvh = ph.cvl = 0.0;
  ph.cv_split = w2d::cv_split(p->cv, &ph.cvh, &ph.cvl) ? 1 : 0;
  const bool h = p->cooling == W2D_COOLINGH;
  switch (p->neq) {
    case 4:
      if (h) launch_cfl<4, true>(u, lev, nblocks, p, sp, ph, scratch);
      else launch_cfl<4, false>(u, lev, nblocks, p, sp, ph, scratch);
      break;
    case 5:
      if (h) launch_cfl<5, true>(u, lev, nblocks, p, sp, ph, scratch);
      else launch_cfl<5, false>(u, lev, nblocks, p, sp, ph, scratch);
      break;
    default:
      if (h) launch_cfl<6, true>(u, lev, nblocks, p, sp, ph, scratch);
      else launch_cfl<6, false>(u, lev, nblocks, p, sp, ph, scratch);
      break;
  }
  if (cudaGetLastError() != cudaSuccess) return W2D_ERR_CUDA;
  double res[2];
  if (cudaMemcpy(res, scratch + W2D_NOALLOC_MAX_BLOCKS, sizeof(res), cudaMemcpyDeviceToHost) != cudaSuccess)
    return W2D_ERR_CUDA;
  if (res[1] != 0.0) return W2D_ERR_TOPOLOGY;   // a level outside 1..nlevs
  *dt = res[0];
  return W2D_OK;
}
