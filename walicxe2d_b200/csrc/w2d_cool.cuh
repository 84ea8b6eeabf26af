// w2d_cool.cuh -- radiative cooling source terms on the device.
//
//   coolingh   src/coolingh.f90:5-259 (atomic, ALOSS, alpha, colf, betah)
//   coolingdmc src/coolingdmc.f90:6-54 with cooldmc, src/dmc_module.f90:14-32
//
// Same operation order as the reference, always in FP64; exp/pow/log/log10
// are CUDA's own (they differ from glibc by a few ulp), so these kernels
// agree with the reference to a relative tolerance, not bit for bit.
#pragma once

#include "w2d_kernels.cuh"

namespace w2d {

// The powers of coolingh (src/coolingh.f90:5-259) in forms equal to them
// as real functions that share one logarithm per cell: x**y as
// exp(y*log(x)), with log(c*x) = log(c) + log(x) for the constant factors;
// x**0.5 as sqrt(x).  The products y*log(x) are below ~20 in magnitude here,
// so their rounding moves a power by < 5e-15 relative, far inside the
// path's tolerance against the CPU restatement (relative L1 1e-12 per
// field).
constexpr double kLn1e3 = 6.907755278982137;      // log(1000)
constexpr double kLn1e4 = 9.210340371976184;      // log(10000)
constexpr double kLn1e5 = 11.512925464970229;     // log(100000)
constexpr double kLn157890 = 11.969653867015934;  // log(157890)
constexpr double kRs157890 = 0.0025166492284451372;  // 1/sqrt(157890)
constexpr double kSqrt1e3 = 31.622776601683793;   // sqrt(1000)

// Exponentials of several arguments at once.  The routine is bound by
// instruction issue (about 1,450 instructions per cell, a third of them FP64,
// at 20 warps per SM): one call of exp per argument loads its constants into
// registers anew and waits for one chain at a time, so N independent
// arguments go through the textbook scheme together (n = round(x/ln 2) in
// FP64, r = x - n ln 2 with ln 2 in two parts, W. J. Cody and W. Waite, 1980;
// e^r = 1 + r (1 + r g(r)) with g a Chebyshev fit of (e^r - 1 - r)/r^2 on
// |r| <= ln(2)/2, error 2^-61, made for this file), its constants operands in
// constant memory.  Arguments outside (-700, 700) and NaN take CUDA's exp.
// Cooling kernel, FP32 ensemble of 6,641 leaves: 150 -> 137 us (CUDA's calls
// with every exponential evaluated: 158).  Errors within 0.8 units in the last
// place, of 10^x 0.9 (tests/test_exp_cpu.py).
static __constant__ double kExp[16] = {
    1.4426950408889634,   // 1/ln 2
    6755399441055744.0,   // 1.5 2^52: adding it rounds to an integer
    0x1.62e42fefa39efp-1, 0x1.abc9e3b39803fp-56,   // ln 2 in two parts
    2.0914717341716378e-09, 2.5105259538448494e-08, 2.755727357010214e-07, 2.7557255297969643e-06,
    2.4801587325605324e-05, 0.0001984126987490126, 0.001388888888888373, 0.008333333333326112,
    0.04166666666666667, 0.1666666666666667, 0.5, 1.0};
static __constant__ double kExp10[5] = {
    3.321928094887362,    // log2(10)
    0x1.34413509f79ffp-2, -0x1.9dc1da994fd21p-59,  // log10(2) in two parts
    0x1.26bb1bbb55516p+1, -0x1.f48ad494ea3e9p-53}; // ln 10 in two parts

// e^r 2^n for |r| <= ln(2)/2, t = 1.5 2^52 + n, |n| < 1023
template <int N>
__device__ __forceinline__ void exp_scale(const double (&r)[N], const double (&t)[N], double (&p)[N])
{
#pragma unroll
  for (int i = 0; i < N; ++i) p[i] = kExp[4];
#pragma unroll
  for (int k = 5; k < 15; ++k)
#pragma unroll
    for (int i = 0; i < N; ++i) p[i] = fma(p[i], r[i], kExp[k]);
#pragma unroll
  for (int k = 0; k < 2; ++k)
#pragma unroll
    for (int i = 0; i < N; ++i) p[i] = fma(p[i], r[i], kExp[15]);
#pragma unroll
  for (int i = 0; i < N; ++i) p[i] *= __hiloint2double((__double2loint(t[i]) + 1023) << 20, 0);
}
static __device__ __noinline__ double exp_far(double x) { return exp(x); }
template <int N>
__device__ __forceinline__ void exp_n(double (&x)[N])
{
  double r[N], t[N], p[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    t[i] = fma(x[i], kExp[0], kExp[1]);
    const double n = t[i] - kExp[1];
    r[i] = fma(-n, kExp[3], fma(-n, kExp[2], x[i]));
  }
  exp_scale<N>(r, t, p);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    if (fabs(x[i]) < 700.) x[i] = p[i];
    else x[i] = x[i] < -746. ? 0. : exp_far(x[i]);
  }
}
// 10^x the same way: n = round(x log2(10)), r = (x - n log10(2)) ln 10
template <int N>
__device__ __forceinline__ void exp10_n(double (&x)[N])
{
  double r[N], t[N], p[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    t[i] = fma(x[i], kExp10[0], kExp[1]);
    const double n = t[i] - kExp[1];
    const double z = fma(-n, kExp10[2], fma(-n, kExp10[1], x[i]));
    r[i] = fma(z, kExp10[3], z * kExp10[4]);
  }
  exp_scale<N>(r, t, p);
#pragma unroll
  for (int i = 0; i < N; ++i) x[i] = fabs(x[i]) < 300. ? p[i] : exp10(x[i]);
}

// What ALOSS needs of a temperature te0 >= 1: te = max(te0, 1000) with its
// reciprocal (in two parts: hi + lo is 1/te to 2^-100), root and logarithm
struct CoolTe {
  double te, rhi, rlo, root, log;
};

// src/coolingh.f90:88-165 (ALOSS); eq: exp(-118409/te), ei: exp(-157900/te)
__device__ __forceinline__ double d_aloss(double x1, double den, double dh0, const CoolTe& k, double eq, double ei)
{
  const double XO = 1.e-3, XION = 2.179e-11;
  const double C0 = 0.5732, C1 = 1.8288e-5, C2 = -1.15822e-10, C3 = 9.4288e-16;
  const double D0 = 0.5856, D1 = 1.55083e-5, D2 = -9.669e-12, D3 = 5.716e-19;
  const double EN = 1.634E-11;
  const double te = k.te;
  double dh = den;
  double dhp = (1. - x1) * dh;
  double de = dhp + 1.E-4 * dh;
  double doi = XO * dh0;
  double doii = XO * dhp;
  double omega = 0.;
  if (te <= 55000.) omega = C0 + te * (C1 + te * (C2 + te * C3));
  if (te >= 72000.) omega = D0 + te * (D1 + te * (D2 + te * D3));
  if (te > 55000. && te < 72000.) {
    double omegal = C0 + te * (C1 + te * (C2 + te * C3));
    double omegah = D0 + te * (D1 + te * (D2 + te * D3));
    double frac = (te - 55000.) / 17000.;
    omega = (1. - frac) * omegal + frac * omegah;
  }
  // 8.6287E-6/(2 sqrt(te)), the root's reciprocal as root/te
  double qla = 4.31435E-6 * fma(k.root, k.rhi, k.root * k.rlo) * omega * eq;
  double ecoll = fmaxr(de * dh0 * qla * EN, 0.);
  double cion = 5.834E-11 * k.root * ei;
  double eion = de * dh0 * cion * XION;
  // the low-temperature terms weigh 1 - fr, the equilibrium curve fr; fr is 0
  // up to 44770 K and 1 from 54770 K on, so that each side's exponentials are
  // only evaluated where they count
  double fr = 0.;
  if (te >= 54770.) fr = 1.;
  if (te > 44770. && te < 54770.) {
    double ex2 = exp(-2. * (te - 49770.) / 500.);
    double th = (1. - ex2) / (1. + ex2);
    fr = 0.5 * (1. + th);
  }
  double sum = ecoll + eion;
  if (te < 54770.) {
    // betah: a = 157890/te, 1.133e-24/sqrt(a) (-0.0713 + 0.5 log a + 0.640 a**(-0.33333))
    const double la = kLn157890 - k.log;
    double xb[1] = {-0.33333 * la};
    exp_n(xb);
    const double betah = 1.133e-24 * (k.root * kRs157890) * (-0.0713 + 0.5 * la + 0.640 * xb[0]);
    double erec = fmaxr(de * dhp * betah, 0.);
    double tm = k.rhi;
    double t2 = tm * tm;
    double xo[2] = {1381465. * t2 - 12328.69 * tm - 19.82621, -2061075. * t2 - 14596.24 * tm - 19.01402};
    exp10_n(xo);
    double eoi = fmaxr(de * doi * xo[0], 0.);
    double eoii = fmaxr(de * doii * xo[1], 0.);
    sum = sum + (erec + 7.033 * (eoi + eoii)) * (1. - fr);
  }
  if (te > 44770.) {
    double betaf = 1.3 * 1.42E-27 * k.root;
    double hiicool = de * dhp * betaf;
    double xe[2] = {-0.63 * k.log, 1.63 * (k.log - kLn1e5)};
    exp_n(xe);
    double x2[1] = {-xe[1]};
    exp_n(x2);
    double equil = (1.0455E-18 * xe[0]) * (1. - x2[0]) * de * den + hiicool;
    sum = sum + equil * fr;
  }
  return sum;
}

// src/coolingh.f90:171-254 (atomic) in FP64 on one cell: from the
// temperature T, neutral fraction y0, density dh and dt (s), the new
// neutral fraction y1, the cooling rate ce of the temperature relaxation
// t1 = 10 + (T - 10) exp(-ce dt) and the clamped new temperature t1.
__device__ __forceinline__ void d_atomic_core(double T, double y0, double dh, double dt, double& y1, double& ce,
                                              double& t1)
{
  const double xi = 1.e-4, boltzm = 1.3807e-16;
  const double lT = log(T), root = sqrt(T), rhi = 1. / T;
  const double rlo = fma(-T, rhi, 1.) * rhi;
  CoolTe k = {T, rhi, rlo, root, lT};
  if (!(T > 1000.)) k = {1000., 1e-3, fma(-1000., 1e-3, 1.) * 1e-3, kSqrt1e3, kLn1e3};
  // colf's exp(-157828/T), alpha's (1e4/T)**0.79 and ALOSS's two
  double x[4] = {-fma(157828., rhi, 157828. * rlo), 0.79 * (kLn1e4 - lT), -fma(118409., k.rhi, 118409. * k.rlo),
                 -fma(1.579E5, k.rhi, 1.579E5 * k.rlo)};
  exp_n(x);
  double col = 5.83e-11 * root * x[0];
  double rec = 2.55e-13 * x[1];
  double a = rec + col;
  double b = -((2. + xi) * rec + (1. + xi) * col);
  double c = (1. + xi) * rec;
  double d = sqrt(b * b - 4. * a * c);
  double g0 = (2. * a * y0 + b + d) / (2. * a * y0 + b - d);
  double xd[1] = {-d * dh * dt};
  exp_n(xd);
  double e = xd[0];
  y1 = (-b - d * (1. + g0 * e) / (1. - g0 * e)) / (2. * a);
  y1 = fminr(y1, 1.);
  y1 = fmaxr(y1, 0.0001);
  double dh0 = y1 * dh;
  double al = d_aloss(y0, dh, dh0, k, x[2], x[3]) / (dh * dh);
  double tprime = 10.;
  ce = (2. * dh * al) / (3. * boltzm * T);
  double xc[1] = {-ce * dt};
  exp_n(xc);
  t1 = tprime + (T - tprime) * xc[0];
  t1 = fmaxr(t1, 0.1 * T);
  t1 = fminr(t1, 10. * T);
  t1 = fmaxr(t1, tprime);
}

template <int NEQ>
__device__ __forceinline__ void d_atomic(const Phys<double>& ph, double dt, double* uu)
{
  double prim[NEQ], T;
  uprim<NEQ>(ph, prim, uu, T);
  double y1, ce, t1;
  d_atomic_core(T, uu[4] / uu[0], uu[0], dt, y1, ce, t1);
  uu[4] = y1 * uu[0];
  uu[3] = ph.cv * (2. * uu[0] - uu[4]) * t1 / ph.tempsc + 0.5 * prim[0] * (prim[1] * prim[1] + prim[2] * prim[2]);
}

// Cooling of cells 0..17 of every leaf (after the fill of layer 0), then
// the per-block CFL partial, DMC cooling-time limit and criteria maximum of
// the cooled state.  pa.cooling selects coolingh or coolingdmc.
template <typename R, int NEQ>
__host__ __device__ constexpr size_t smem_cool()
{
  return 128 + sizeof(R) * NEQ * W2D_CELLS + 64 * sizeof(double);
}

// Threads of the cooling kernel: one per cell 0..17 x 0..17 of a block
// without its four corners (320), so the FP64 routine runs in one round;
// the block statistics use the first 256, and warp 8 combines them.
constexpr int W2D_COOL_THREADS = 320;

template <typename R, int NEQ, bool P>
__global__ void __launch_bounds__(W2D_COOL_THREADS, 3) k_cool(KArgs a, PhysArgs pa, double dt_s)
{
  uint64_t* bar = reinterpret_cast<uint64_t*>(w2d_smem);
  R(*st)[W2D_W][W2D_W] = reinterpret_cast<R(*)[W2D_W][W2D_W]>(w2d_smem + 128);
  double* sred = reinterpret_cast<double*>(w2d_smem + 128 + sizeof(R) * NEQ * W2D_CELLS);
  const Phys<R> ph = make_phys<R, -1, -1>(pa);
  const Phys<double> phd = make_phys<double, -1, -1>(pa);
  const int tid = threadIdx.x;
  const size_t bs = (size_t)NEQ * W2D_CELLS;
  bar_init_once(bar);
  pdl_begin();
  if (queue_ended<P>(a)) return;
  uint32_t par = 0;
  const double dt_arg = dt_s;
  for (LeafRange lr = leaf_range<P>(a); lr.li < lr.end; lr.li += lr.step, par ^= 1u) {
  const int b = a.leaves[lr.li];
  R* __restrict__ u = (R*)a.u + (size_t)b * bs;
  R* __restrict__ pb = (pa.cooling == COOL_DMC) ? (R*)a.prim + (size_t)b * bs : nullptr;
  if (tid == 0) tile_issue<R, NEQ>(&st[0][0][0], u, bar);
  // dt*tsc of the block's run, of the device dt, or the argument
  dt_s = a.run_of ? a.dt_run[a.run_of[b]] * a.tsc : (a.dt_dev ? *a.dt_dev * a.tsc : dt_arg);
  if (!wait_tiles_p(bar, a.err, b, par)) return;
  if (a.jet && a.jetblk[lr.li]) {   // impose_jet of boundaryI, before cooling
    jet_interior_fn<R, NEQ>(st, a, b, u);
    __syncthreads();
  }
  for (int t = tid; t < 320; t += W2D_COOL_THREADS) {
    // the t-th of cells 0..17 x 0..17 without the corners c = 0, 17, 306, 323
    int c = t + 1;
    c += (c >= 17);
    c += (c >= 306);
    const int i = c % 18, j = c / 18;
    double uu[NEQ];
#pragma unroll
    for (int k = 0; k < NEQ; ++k) uu[k] = (double)st[k][j + 1][i + 1];
    if (pa.cooling == COOL_H) {
      d_atomic<NEQ>(phd, dt_s, uu);
      u[3 * W2D_CELLS + cidx(i, j)] = R(uu[3]);
      u[4 * W2D_CELLS + cidx(i, j)] = R(uu[4]);
      R ur[NEQ], q[NEQ], T;
#pragma unroll
      for (int k = 0; k < NEQ; ++k) ur[k] = R(uu[k]);
      uprim<NEQ>(ph, q, ur, T);
#pragma unroll
      for (int k = 0; k < NEQ; ++k) st[k][j + 1][i + 1] = q[k];
    } else {
      double q[NEQ], T;
      uprim<NEQ>(phd, q, uu, T);
      if (T > 1.e4) {                                  // coolingdmc.f90:30-40
        double eth0 = phd.cv * q[3];
        double aloss = d_cooldmc(a.cooltab, T);
        double dens = q[0];
        double ce = (aloss * (dens * dens)) / (eth0 * a.psc);
        q[3] = q[3] * exp(-ce * dt_s);
        u[3 * W2D_CELLS + cidx(i, j)] = R(uu[3] - eth0 + phd.cv * q[3]);
      }
#pragma unroll
      for (int k = 0; k < NEQ; ++k) {
        pb[k * W2D_CELLS + cidx(i, j)] = R(q[k]);
        st[k][j + 1][i + 1] = R(q[k]);
      }
    }
  }
  __syncthreads();
  block_stats<R, NEQ>(st, ph, a, pa, sred);
  leaf_end();
  stats_finish<R>(sred, a, b, pa.cooling == COOL_DMC);
  }
}

// primitives of whole blocks into a staging buffer (w2d_get_primit when
// the pool does not store them)
// Conserved totals in FP64 (the FP32 path keeps its state in FP32, its
// totals in FP64): CTA k sums u_q dV over the 256 interior cells of block
// ids[k] into out[k*NEQ + q], dV = dx dy of the block's level, times the
// cell's radius r = (j + icoord(nb,2) - 0.5) dy in cylindrical geometry
// (volume per radian).  The sum runs in a fixed order (warp trees, then the
// warps in order), so the partials do not depend on scheduling.
template <typename R, int NEQ>
__global__ void __launch_bounds__(256) k_totals(KArgs a, int cyl, const int* __restrict__ ids,
                                                double* __restrict__ out)
{
  __shared__ double red[8][NEQ];
  const int b = ids[blockIdx.x];
  const int t = threadIdx.x, i = 1 + t % 16, j = 1 + t / 16;
  const int lev = a.lev[b];
  const double dy = geo_dy(a, b, lev);
  double dv = geo_dx(a, b, lev) * dy;
  if (cyl) dv = dv * (((double)(j + a.icoord[2 * b + 1]) - 0.5) * dy);
  const R* ub = (const R*)a.u + (size_t)b * NEQ * W2D_CELLS;
  double v[NEQ];
#pragma unroll
  for (int q = 0; q < NEQ; ++q) {
    v[q] = (double)ub[q * W2D_CELLS + cidx(i, j)] * dv;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
  }
  if ((t & 31) == 0) {
#pragma unroll
    for (int q = 0; q < NEQ; ++q) red[t >> 5][q] = v[q];
  }
  __syncthreads();
  if (t < NEQ) {
    double s = 0.;
    for (int w = 0; w < 8; ++w) s += red[w][t];
    out[(size_t)blockIdx.x * NEQ + t] = s;
  }
}

template <typename R, int NEQ>
__global__ void k_to_prim(PhysArgs pa, const R* __restrict__ u, double* __restrict__ out,
                          const int* __restrict__ ids)
{
  const Phys<R> ph = make_phys<R, -1, -1>(pa);
  const size_t bs = (size_t)NEQ * W2D_CELLS;
  const R* ub = u + (size_t)ids[blockIdx.x] * bs;
  double* ob = out + (size_t)blockIdx.x * bs;
  for (int c = threadIdx.x; c < W2D_CELLS; c += blockDim.x) {
    R uu[NEQ], q[NEQ], T;
#pragma unroll
    for (int k = 0; k < NEQ; ++k) uu[k] = ub[k * W2D_CELLS + c];
    uprim<NEQ>(ph, q, uu, T);
#pragma unroll
    for (int k = 0; k < NEQ; ++k) ob[k * W2D_CELLS + c] = q[k];
  }
}

}  // namespace w2d
