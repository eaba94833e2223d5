// exact_f64.cu -- FP64 Step, CalcHydro and InitFromHydro in the reference's
// operation order (LBSWIM_COMPAT_EXACT_F64).
//
// The reference transforms the 15 distributions to modes and back with dense
// 15x15 products (lb.cu:72-218) and reads rho, u from the first four modes
// (lb.cu:250-295); InitFromHydro projects the equilibrium modes (lb.cu:314-371).
// These kernels perform the same operations in the same order, each rounded on
// its own (__dadd_rn / __dmul_rn / __ddiv_rn never fuse), so an FP64 lattice
// reproduces the reference's host build bit for bit.
//
// The kernels are bound by GB300's FP64 pipe (two operations per clock and SM), so
// they leave out what changes no bit: products with the transforms' zeros (half
// of the entries; a sum that starts at +0 is never -0, and adding a zero of either
// sign leaves it as it is), products with 1 and -1, and products that differ only
// in sign are formed once.  That holds while the values are finite; a site with
// one that is not takes the dense loops, with the tables of the lattice's
// LBParams in constant memory.  128^3: step 3.59 -> 1.57 ms, CalcHydro 0.61 -> 0.31 ms.
#include <cuda_runtime.h>

#include <mutex>

#include "lbswim_device.cuh"
#include "lbswim_internal.h"

namespace lbswim {

__constant__ double c_mm[15][15];
__constant__ double c_mmi[15][15];

static void upload_tables(const lbswim_lbparams& P) {
  // the tables do not depend on tau: one upload per device
  static std::mutex mu;
  static bool done[64] = {};
  int dev = 0;
  LB_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  if (dev < 64 && done[dev]) return;
  LB_CUDA(cudaMemcpyToSymbol(c_mm, P.mm, sizeof(P.mm)));
  LB_CUDA(cudaMemcpyToSymbol(c_mmi, P.mmi, sizeof(P.mmi)));
  if (dev < 64) done[dev] = true;
}

// ---- the transforms' entries at compile time -----------------------------------
// Three times mode m on velocity p (d3q15.h:13-28), an integer, ...
__host__ __device__ constexpr int mode3(int m, int p) {
  const int x = cx_of(p), y = cy_of(p), z = cz_of(p), c2 = x * x + y * y + z * z;
  const int chi1 = c2 == 1 ? 1 : -2;
  return m == 0   ? 3
         : m == 1 ? 3 * x
         : m == 2 ? 3 * y
         : m == 3 ? 3 * z
         : m == 4 ? 3 * x * x - 1
         : m == 5 ? 3 * x * y
         : m == 6 ? 3 * x * z
         : m == 7 ? 3 * y * y - 1
         : m == 8 ? 3 * y * z
         : m == 9 ? 3 * z * z - 1
         : m == 10 ? 3 * chi1
         : m == 11 ? 3 * chi1 * x
         : m == 12 ? 3 * chi1 * y
         : m == 13 ? 3 * chi1 * z
                   : 3 * x * y * z;
}
// ... 72 times the weight, and 648 times the squared norm of the mode.
__host__ __device__ constexpr int weight72(int p) { return p == 0 ? 16 : p <= 6 ? 8 : 1; }
__host__ __device__ constexpr int norm648(int m) {
  int s = 0;
  for (int p = 0; p < 15; ++p) s += weight72(p) * mode3(m, p) * mode3(m, p);
  return s;
}
// |mm[m][p]| and |mmi[p][m]| as the tables hold them (one rounding of the rational).
__host__ __device__ constexpr double mm_abs(int m, int p) {
  const int v = mode3(m, p) < 0 ? -mode3(m, p) : mode3(m, p);
  return v % 3 == 0 ? (double)(v / 3) : (double)v / 3.0;
}
__host__ __device__ constexpr double mmi_abs(int p, int m) {
  const int v = mode3(m, p) < 0 ? -mode3(m, p) : mode3(m, p);
  return (double)(3 * weight72(p) * v) / (double)norm648(m);
}

struct ExactRelax {
  double tau_s, tau_b, omega_s, omega_b;
};

__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double ddiv(double a, double b) { return __ddiv_rn(a, b); }

// acc + x c for an entry of magnitude c and the sign of `three`.
__device__ __forceinline__ double add_entry(double acc, double x, int three, double c) {
  if (three == 0) return acc;
  const double t = c == 1.0 ? x : dmul(x, c);
  return three > 0 ? dadd(acc, t) : dsub(acc, t);
}
__device__ __forceinline__ bool finite_bits(double x) {
  return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000;
}

// Modes [0, M) of finite distributions.
template <int M>
__device__ __forceinline__ void modes_of(const double fo[15], double mode[15]) {
#pragma unroll
  for (int m = 0; m < M; ++m) {
    double acc = 0.0;
#pragma unroll
    for (int p = 0; p < 15; ++p) acc = add_entry(acc, fo[p], mode3(m, p), mm_abs(m, p));
    mode[m] = acc;
  }
}
// The same of any distributions.
template <int M>
__device__ __noinline__ void modes_dense(const double* fo, double* mode) {
  for (int m = 0; m < M; ++m) {
    double acc = 0.0;
    for (int p = 0; p < 15; ++p) acc = dadd(acc, dmul(fo[p], c_mm[m][p]));
    mode[m] = acc;
  }
}
// Distribution p of finite modes 0 to 9, the others zero.
__device__ __forceinline__ double from_modes(const double mode[15], int p) {
  double acc = 0.0;
#pragma unroll
  for (int m = 0; m < 10; ++m) acc = add_entry(acc, mode[m], mode3(m, p), mmi_abs(p, m));
  return acc;
}
__device__ __noinline__ double from_modes_dense(const double* mode, int p) {
  double acc = 0.0;
  for (int m = 0; m < 15; ++m) acc = dadd(acc, dmul(mode[m], c_mmi[p][m]));
  return acc;
}
__device__ __forceinline__ bool finite_modes(const double mode[15]) {
  bool ok = true;
#pragma unroll
  for (int m = 0; m < 10; ++m) ok = ok && finite_bits(mode[m]);
  return ok;
}

// DoStep, lb.cu:72-218: modes, relaxation with forcing, back-projection,
// push-stream with periodic wrap.  A thread takes site blockIdx.x * EXACT_THREADS +
// threadIdx.x of x plane blockIdx.y.
constexpr int EXACT_THREADS = 128;
__global__ void __launch_bounds__(EXACT_THREADS) k_step_exact_f64(
    const double* __restrict__ f, const double* __restrict__ F, double* __restrict__ fn, int nx,
    int ny, int nz, FastDiv by_nz, long long N, ExactRelax k) {
  const unsigned plane = (unsigned)ny * (unsigned)nz;
  const unsigned t = blockIdx.x * EXACT_THREADS + threadIdx.x;
  if (t >= plane) return;
  const int x = blockIdx.y, y = (int)div_by(t, by_nz), z = (int)(t - (unsigned)y * nz);
  const long long nynz = plane, s = (long long)x * nynz + t;
  double fo[15], mode[15];
#pragma unroll
  for (int p = 0; p < 15; ++p) fo[p] = f[p * N + s];
  // a non-finite distribution makes their sum, mode 0, non-finite
  modes_of<10>(fo, mode);
  if (!finite_bits(mode[0])) {
    double any[15], dense[10];
    for (int p = 0; p < 15; ++p) any[p] = fo[p];
    modes_dense<10>(any, dense);
    for (int m = 0; m < 10; ++m) mode[m] = dense[m];
  }
  double Fv[3], u[3], usq = 0.0, uDOTf = 0.0;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const double Fa = F ? F[a * N + s] : 0.0;
    Fv[a] = Fa;
    u[a] = ddiv(dadd(mode[1 + a], dmul(0.5, Fa)), mode[0]);
    mode[1 + a] = dadd(mode[1 + a], Fa);
    usq = dadd(usq, dmul(u[a], u[a]));
    uDOTf = dadd(uDOTf, dmul(u[a], Fa));
  }
  double S[3][3] = {{mode[4], mode[5], mode[6]}, {mode[5], mode[7], mode[8]},
                    {mode[6], mode[8], mode[9]}};
  double TrS = 0.0;
#pragma unroll
  for (int a = 0; a < 3; ++a) TrS = dadd(TrS, S[a][a]);
#pragma unroll
  for (int a = 0; a < 3; ++a) S[a][a] = dsub(S[a][a], ddiv(TrS, 3.0));
  TrS = dsub(TrS, dmul(k.omega_b, dsub(TrS, dmul(mode[0], usq))));
  TrS = dadd(TrS, dmul(dmul(dmul(2.0, k.omega_b), k.tau_b), uDOTf));
#pragma unroll
  for (int a = 0; a < 3; ++a) {
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const double d = (a == b) ? 1.0 : 0.0;
      S[a][b] = dsub(S[a][b],
                     dmul(k.omega_s, dsub(S[a][b], dmul(mode[0], dsub(dmul(u[a], u[b]), dmul(usq, d))))));
      S[a][b] = dadd(S[a][b], dmul(dmul(dmul(2.0, k.omega_s), k.tau_s),
                                   dsub(dadd(dmul(u[a], Fv[b]), dmul(Fv[a], u[b])),
                                        dmul(dmul(2.0, uDOTf), d))));
    }
    S[a][a] = dadd(S[a][a], ddiv(TrS, 3.0));
  }
  mode[4] = S[0][0];
  mode[5] = S[0][1];
  mode[6] = S[0][2];
  mode[7] = S[1][1];
  mode[8] = S[1][2];
  mode[9] = S[2][2];
#pragma unroll
  for (int m = 10; m < 15; ++m) mode[m] = 0.0;
  double out[15];
  if (finite_modes(mode)) {
#pragma unroll
    for (int p = 0; p < 15; ++p) out[p] = from_modes(mode, p);
  } else {
    double any[15];
    for (int m = 0; m < 15; ++m) any[m] = mode[m];
    for (int p = 0; p < 15; ++p) out[p] = from_modes_dense(any, p);
  }
  const int xm = wrap_once(x - 1, nx), xp = wrap_once(x + 1, nx);
  const int ym = wrap_once(y - 1, ny), yp = wrap_once(y + 1, ny);
  const int zm = wrap_once(z - 1, nz), zp = wrap_once(z + 1, nz);
#pragma unroll
  for (int p = 0; p < 15; ++p) {
    const int dx = cx_of(p), dy = cy_of(p), dz = cz_of(p);
    const long long X = dx > 0 ? xp : (dx < 0 ? xm : x);
    const long long Y = dy > 0 ? yp : (dy < 0 ? ym : y);
    const long long Z = dz > 0 ? zp : (dz < 0 ? zm : z);
    fn[p * N + X * nynz + Y * nz + Z] = out[p];
  }
}

// DoCalcHydro, lb.cu:250-295.
__global__ void k_calc_hydro_exact_f64(const double* __restrict__ f, const double* __restrict__ F,
                                       double* __restrict__ rho, double* __restrict__ u,
                                       long long N, unsigned* status) {
  for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < N;
       s += (long long)gridDim.x * blockDim.x) {
    double fo[15], mode[15];
#pragma unroll
    for (int p = 0; p < 15; ++p) fo[p] = f[p * N + s];
    modes_of<4>(fo, mode);
    if (!finite_bits(mode[0])) {
      double any[15], dense[4];
      for (int p = 0; p < 15; ++p) any[p] = fo[p];
      modes_dense<4>(any, dense);
      for (int m = 0; m < 4; ++m) mode[m] = dense[m];
    }
    rho[s] = mode[0];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const double Fa = F ? F[a * N + s] : 0.0;
      u[a * N + s] = ddiv(dadd(mode[1 + a], dmul(0.5, Fa)), mode[0]);
    }
    if (!finite_d(mode[0] + mode[1] + mode[2] + mode[3]))
      raise_status(status, LBSWIM_STATUS_NONFINITE);
  }
}

// DoInitFromHydro, lb.cu:314-371 (compat_sxz reproduces lb.cu:356).
__global__ void k_init_exact_f64(const double* __restrict__ rho, const double* __restrict__ u,
                                 double* __restrict__ f, long long N, int compat_sxz) {
  for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < N;
       s += (long long)gridDim.x * blockDim.x) {
    const double r = rho[s], ux = u[s], uy = u[N + s], uz = u[2 * N + s];
    double mode[15];
#pragma unroll
    for (int m = 0; m < 15; ++m) mode[m] = 0.0;
    mode[0] = r;
    mode[1] = dmul(r, ux);
    mode[2] = dmul(r, uy);
    mode[3] = dmul(r, uz);
    mode[4] = dmul(dmul(r, ux), ux);
    mode[5] = dmul(dmul(r, ux), uy);
    mode[6] = compat_sxz ? dmul(dmul(r, ux), uy) : dmul(dmul(r, ux), uz);
    mode[7] = dmul(dmul(r, uy), uy);
    mode[8] = dmul(dmul(r, uy), uz);
    mode[9] = dmul(dmul(r, uz), uz);
    if (finite_modes(mode)) {
#pragma unroll
      for (int p = 0; p < 15; ++p) f[p * N + s] = from_modes(mode, p);
    } else {
      double any[15];
      for (int m = 0; m < 15; ++m) any[m] = mode[m];
      for (int p = 0; p < 15; ++p) f[p * N + s] = from_modes_dense(any, p);
    }
  }
}

static int grid_1d(long long n) {
  long long g = (n + 255) / 256;
  return (int)(g < 1 ? 1 : (g > 152LL * 16 ? 152LL * 16 : g));
}

void exact_step_f64(Lattice* L) {
  upload_tables(L->params);
  const int nx = L->size[0], ny = L->size[1], nz = L->size[2];
  ExactRelax k;
  k.tau_s = L->tau_s;
  k.tau_b = L->tau_b;
  k.omega_s = 1.0 / (L->tau_s + 0.5);
  k.omega_b = 1.0 / (L->tau_b + 0.5);
  const dim3 grid((unsigned)(((long long)ny * nz + EXACT_THREADS - 1) / EXACT_THREADS), nx);
  k_step_exact_f64<<<grid, EXACT_THREADS, 0, L->stream>>>(
      (const double*)L->f[L->cur], L->force_zero_pending ? nullptr : (const double*)L->force,
      (double*)L->f[L->cur ^ 1], nx, ny, nz, fast_div((unsigned)nz), L->n, k);
  LB_CHECK_LAUNCH(1);
}

void exact_calc_hydro_f64(Lattice* L) {
  upload_tables(L->params);
  k_calc_hydro_exact_f64<<<grid_1d(L->n), 256, 0, L->stream>>>(
      (const double*)L->f[L->cur], L->force_zero_pending ? nullptr : (const double*)L->force,
      (double*)L->rho, (double*)L->u, L->n, L->status);
  LB_CHECK_LAUNCH(1);
}

void exact_init_from_hydro_f64(Lattice* L) {
  upload_tables(L->params);
  const int compat = (L->compat & LBSWIM_COMPAT_INIT_SXZ) ? 1 : 0;
  k_init_exact_f64<<<grid_1d(L->n), 256, 0, L->stream>>>((const double*)L->rho,
                                                         (const double*)L->u,
                                                         (double*)L->f[L->cur], L->n, compat);
  LB_CHECK_LAUNCH(1);
}

}  // namespace lbswim
