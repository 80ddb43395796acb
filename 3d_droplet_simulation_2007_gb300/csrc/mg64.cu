// mg64.cu -- FP64 multigrid kernels of the variable-density pressure Poisson
// solve (main.f:3765-3997, 4298-4329, 4432-4494) and the deterministic
// reductions used by the solver.
//
// Ghost handling: bc_scalar's final ghost values are a closed-form function of
// the interior (x ghost 1 = cell 2, x ghost nx = 0, y/z ghosts = the adjacent
// interior cell, edges and corners by composition).  The colour passes of
// relax therefore read "virtual ghosts" (own value or 0) instead of memory,
// which equals running bc_scalar before each pass, and a single bc_scalar at
// the end of a block of relax calls leaves the array exactly as the reference.
// All arithmetic keeps the reference's operation order; this file is built
// without FMA contraction so results are bit-identical to a non-contracting
// Fortran build.
#include <algorithm>
#include <cmath>

#include "dsg_internal.cuh"

namespace dsg {
namespace {

// ---- bc_scalar, one launch over the six faces (closed form) -----------------
__global__ void k_bc_scalar(double *__restrict__ s, Dims d) {
  const int face = blockIdx.z;
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  const int q = blockIdx.y * blockDim.y + threadIdx.y;
  int i, j, k;
  if (face < 2) {  // x faces: p -> j, q -> k
    if (p >= d.ny || q >= d.nz) return;
    i = face == 0 ? 1 : d.nx; j = p + 1; k = q + 1;
  } else if (face < 4) {  // y faces: p -> i, q -> k
    if (p >= d.nx || q >= d.nz) return;
    i = p + 1; j = face == 2 ? 1 : d.ny; k = q + 1;
  } else {  // z faces: p -> i, q -> j
    if (p >= d.nx || q >= d.ny) return;
    i = p + 1; j = q + 1; k = face == 4 ? 1 : d.nz;
  }
  if (i == d.nx) { s[d.ix(i, j, k)] = 0.0; return; }
  const int ci = i == 1 ? 2 : i;
  const int cj = j == 1 ? 2 : (j == d.ny ? d.ny - 1 : j);
  const int ck = k == 1 ? 2 : (k == d.nz ? d.nz - 1 : k);
  s[d.ix(i, j, k)] = s[d.ix(ci, cj, ck)];
}

// bc_resid (main.f:4441-4461: plane 1 = plane 2 and plane nx = plane nx-1 over
// all j, k, then the y and z ghosts of interior i = 0) and bc_out
// (main.f:4406-4427: the same x step, then every y ghost, all i, and the z
// ghosts of interior i from the adjacent cell), their ordered steps in one
// launch.  The x step copies old ghosts of planes 2 and nx-1 that the z step
// (bc_resid: and the y step) overwrites; the threads that overwrite them copy
// them first.
template <bool ZERO>
__global__ void k_bc_copy(double *__restrict__ s, Dims d) {
  const int face = blockIdx.z;
  const int p = blockIdx.x * blockDim.x + threadIdx.x, q = blockIdx.y * blockDim.y + threadIdx.y;
  if (face == 0) {  // p -> j, q -> k
    const int j = p + 2, k = q + 2;
    if (j > d.ny - 1 || k > d.nz - 1) return;
    s[d.ix(1, j, k)] = s[d.ix(2, j, k)];
    s[d.ix(d.nx, j, k)] = s[d.ix(d.nx - 1, j, k)];
    return;
  }
  auto put = [&](int i, int j, int k, double x) {
    const size_t n = d.ix(i, j, k);
    if (i == 2) s[n - 1] = s[n];
    if (i == d.nx - 1) s[n + 1] = s[n];
    s[n] = x;
  };
  if (face == 1) {  // p -> i, q -> k
    const int i = p + (ZERO ? 2 : 1), k = q + 2;
    if (i > d.nx - (ZERO ? 1 : 0) || k > d.nz - 1) return;
    if (ZERO) {
      put(i, 1, k, 0.0);
      put(i, d.ny, k, 0.0);
    } else {
      const int ci = i == 1 ? 2 : (i == d.nx ? d.nx - 1 : i);
      s[d.ix(i, 1, k)] = s[d.ix(ci, 2, k)];
      s[d.ix(i, d.ny, k)] = s[d.ix(ci, d.ny - 1, k)];
    }
    return;
  }
  const int i = p + 2, j = q + 1;  // ghost rows included
  if (i > d.nx - 1 || j > d.ny) return;
  const int cj = j == 1 ? 2 : (j == d.ny ? d.ny - 1 : j);
  put(i, j, 1, ZERO ? 0.0 : s[d.ix(i, cj, 2)]);
  put(i, j, d.nz, ZERO ? 0.0 : s[d.ix(i, cj, d.nz - 1)]);
}

// ---- relax: one colour pass (main.f:3973-3992) ----------------------------
// How an update is rounded.
// REF: the reference's operation order, no contraction (17 FP64 operations
// per cell, bit-identical to the oracle).
// REF2: the same bits in 15 operations, where h2 and 1 - omega are plus or
// minus powers of two (2^k cells along x; the reference's omega = 1.5): their
// products are exact, so a fused multiply-add rounds exactly once where the
// separate multiply and add did.
// FMA: the same sum as a fused multiply-add chain and the update written as
// u + omega*(temp - u) (10 operations).
// GB300's FP64 pipe bounds the REF forms, so the operation count sets their
// speed (128^3 pass: 39.1 us with 17, 34.6 with 15): an SM starts one FP64
// instruction per warp scheduler every 64 cycles, whatever its lanes do.
enum Round { REF, REF2, FMA };

// Warps of k_relax_colour in a plane.
__host__ __device__ inline unsigned plane_warps(Dims d) {
  return ((unsigned)(d.nx - 1) / 2 * (unsigned)(d.ny - 2) + 31) / 32;
}

// The update from the sum over the faces, REF and REF2.
template <Round R>
__device__ __forceinline__ double relax_update(double uc, double sum, double ei, double rhs, double h2, double omega) {
  if (R == REF2) return __fma_rn(1.0 - omega, uc, omega * (__fma_rn(-h2, rhs, sum) * ei));
  return omega * ((sum - h2 * rhs) * ei) + (1.0 - omega) * uc;
}

template <Round R>
__device__ __forceinline__ double relax_value(double uc, double xp, double xm, double yp, double ym, double zp,
                                              double zm, double ae, double aw, double bn, double bs, double ct,
                                              double cb, double ei, double rhs, double h2, double omega) {
  if (R == FMA) {
    double t = ae * xp;
    t = __fma_rn(aw, xm, t);
    t = __fma_rn(bn, yp, t);
    t = __fma_rn(bs, ym, t);
    t = __fma_rn(ct, zp, t);
    t = __fma_rn(cb, zm, t);
    t = __fma_rn(-h2, rhs, t) * ei;
    return __fma_rn(omega, t - uc, uc);
  }
  return relax_update<R>(uc, ae * xp + aw * xm + bn * yp + bs * ym + ct * zp + cb * zm, ei, rhs, h2, omega);
}

// Residual of a cell, rhs - (1/h^2) sum a_nb (u_nb - u) (main.f:3912-3925).
template <Round R>
__device__ __forceinline__ double resid_value(double uc, double xp, double xm, double yp, double ym, double zp,
                                              double zm, double ae, double aw, double bn, double bs, double ct,
                                              double cb, double rhs, double h2i) {
  if (R == FMA) {
    double t = ae * (xp - uc);
    t = __fma_rn(aw, xm - uc, t);
    t = __fma_rn(bn, yp - uc, t);
    t = __fma_rn(bs, ym - uc, t);
    t = __fma_rn(ct, zp - uc, t);
    t = __fma_rn(cb, zm - uc, t);
    return __fma_rn(-h2i, t, rhs);
  }
  const double sum = ae * (xp - uc) + aw * (xm - uc) + bn * (yp - uc) + bs * (ym - uc) + ct * (zp - uc) +
                     cb * (zm - uc);
  if (R == REF2) return __fma_rn(-h2i, sum, rhs);
  return -h2i * sum + rhs;
}

// |x| is a power of two in the range where its product with a value of the
// fields stays exact (no overflow or underflow for magnitudes in 2^+-600).
bool power_of_two(double x) {
  int e;
  return std::isfinite(x) && x != 0.0 && std::fabs(std::frexp(x, &e)) == 0.5 && e > -300 && e < 300;
}

// colour 0 updates i+j+k even (first pass), colour 1 odd.  A plane's threads
// count through its rows, half = ceil((nx - 2) / 2) per row, and thread (t, j)
// updates i = i0 + 2t: no lane stays idle at the end of a row, which the FP64
// pipe would charge like any other (96 x 48 x 96: 18.8 us with whole warps per
// row, 15.2 so).  Ghost neighbours are virtual (see file header).
// GHOSTS: the cells at the boundary also write the ghosts they determine (the
// last sweep of a block, in place of a bc_scalar launch).
//
// V: with the short forms for one fluid.  In gas every face has the same
// coefficient k, so a cell's six products k * u are those that its neighbours
// need as well: each pass also stores its own (V > 0), and from the second pass
// of a phase on (V = 2) the warps whose cells lie in gas sum stored products,
// 10 operations instead of 15 (REF 12 instead of 17) and neither coefficients
// nor ei to read.  In liquid, where k is 1, u itself is the product.  The
// products are rounded as before: same bits.  The fused form has no product to
// share, but in either fluid it needs only the plain sum of the neighbours and
// three constants, 8 operations instead of 10 (192^3 pass 67 -> 56 us, 256^3
// 153 -> 128), with fewer roundings.  128^3 pass 34.9 -> 27.1 us, 64^3
// 6.6 -> 5.9.
template <Round R, bool GHOSTS, int V>
__global__ void k_relax_colour(double *__restrict__ u, const double *__restrict__ rhs,
                               const double *__restrict__ a, const double *__restrict__ b,
                               const double *__restrict__ c, const double *__restrict__ ei, Dims d,
                               double h2, double omega, int colour, Products P) {
  const unsigned half = (unsigned)(d.nx - 1) / 2, e = blockIdx.x * blockDim.x + threadIdx.x, row = e / half;
  const int j = (int)row + 2;
  const int k = blockIdx.y + 2;
  if (j > d.ny - 1) return;
  const int i = 2 + ((j + k + colour) & 1) + 2 * (int)(e - row * half);
  if (i > d.nx - 1) return;
  const size_t q = d.ix(i, j, k);
  const size_t sy = d.sy(), sz = d.sz();
  const double uc = u[q];
  const unsigned flag = V == 2 ? P.flags[(e >> 5) + (size_t)plane_warps(d) * (k - 2)] : 0;
  if (V == 2 && R == FMA && flag) {
    const double xp = (i + 1 == d.nx) ? 0.0 : u[q + 1];
    const double xm = (i - 1 == 1) ? uc : u[q - 1];
    const double yp = (j + 1 == d.ny) ? uc : u[q + sy];
    const double ym = (j - 1 == 1) ? uc : u[q - sy];
    const double zp = (k + 1 == d.nz) ? uc : u[q + sz];
    const double zm = (k - 1 == 1) ? uc : u[q - sz];
    const double sum = ((xp + xm) + (yp + ym)) + (zp + zm);
    const double v = __fma_rn(flag == 1 ? P.w : P.w1, sum, __fma_rn(flag == 1 ? P.z : P.z1, rhs[q], P.keep * uc));
    u[q] = v;
    if (GHOSTS) write_ghosts(u, d, i, j, k, v);
    return;
  }
  if (V == 2 && R != FMA && flag) {
    const double *x = flag == 1 ? P.v : u;
    double own = uc;
    if (flag == 1 && (i == 2 || j == 2 || j == d.ny - 1 || k == 2 || k == d.nz - 1)) own = P.k * uc;
    const double xp = (i + 1 == d.nx) ? 0.0 : x[q + 1];
    const double xm = (i - 1 == 1) ? own : x[q - 1];
    const double yp = (j + 1 == d.ny) ? own : x[q + sy];
    const double ym = (j - 1 == 1) ? own : x[q - sy];
    const double zp = (k + 1 == d.nz) ? own : x[q + sz];
    const double zm = (k - 1 == 1) ? own : x[q - sz];
    const double v = relax_update<R>(uc, xp + xm + yp + ym + zp + zm, flag == 1 ? P.e : P.e1, rhs[q], h2, omega);
    u[q] = v;
    P.v[q] = P.k * v;
    if (GHOSTS) write_ghosts(u, d, i, j, k, v);
    return;
  }
  const double xp = (i + 1 == d.nx) ? 0.0 : u[q + 1];
  const double xm = (i - 1 == 1) ? uc : u[q - 1];
  const double yp = (j + 1 == d.ny) ? uc : u[q + sy];
  const double ym = (j - 1 == 1) ? uc : u[q - sy];
  const double zp = (k + 1 == d.nz) ? uc : u[q + sz];
  const double zm = (k - 1 == 1) ? uc : u[q - sz];
  const double v = relax_value<R>(uc, xp, xm, yp, ym, zp, zm, a[q], a[q - 1], b[q], b[q - sy], c[q], c[q - sz], ei[q],
                                  rhs[q], h2, omega);
  u[q] = v;
  if (V && R != FMA) P.v[q] = P.k * v;
  if (GHOSTS) write_ghosts(u, d, i, j, k, v);
}

// Flags of k_relax_colour's warps, for the cells of both colours: whether all
// their faces and ei are gas's (1) or liquid's (2; for shared products only
// where its coefficient is 1).
// One warp per flag.
__global__ void k_bulk_flags(unsigned char *__restrict__ flags, const double *__restrict__ a, const double *__restrict__ b,
                             const double *__restrict__ c, const double *__restrict__ ei, Dims d, Products P) {
  const unsigned half = (unsigned)(d.nx - 1) / 2, pw = plane_warps(d), total = pw * (unsigned)(d.nz - 2);
  const size_t sy = d.sy(), sz = d.sz();
  for (unsigned t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < total; t += gridDim.x * blockDim.x >> 5) {
    const unsigned k = t / pw, e = min(32 * (t - k * pw) + (threadIdx.x & 31), half * (unsigned)(d.ny - 2) - 1), row = e / half;
    bool gas = true, liquid = !P.v || same_bits(P.k1, 1.0);
#pragma unroll
    for (int m = 0; m < 2; m++) {
      const size_t q = d.ix(min(2 + 2 * (int)(e - row * half) + m, d.nx - 1), (int)row + 2, (int)k + 2);
      const double f = a[q], x = ei[q];
      const bool same = same_bits(a[q - 1], f) & same_bits(b[q], f) & same_bits(b[q - sy], f) & same_bits(c[q], f) & same_bits(c[q - sz], f);
      gas &= same & same_bits(f, P.k) & same_bits(x, P.e);
      liquid &= same & same_bits(f, P.k1) & same_bits(x, P.e1);
    }
    gas = __all_sync(0xffffffffu, gas);
    liquid = __all_sync(0xffffffffu, liquid);
    if ((threadIdx.x & 31) == 0) flags[t] = gas ? 1 : liquid ? 2 : 0;
  }
}

// Arithmetic of the cluster kernel on the FP64 levels: the two forms of
// k_relax_colour and k_resid, and rstrct's and interp's transfers.
template <Round R>
struct Cluster64 {
  typedef double T;
  // the first coarsest solve has lengthscale for its spacing, no power of two
  typedef Cluster64<R == REF2 ? REF : R> First;
  static constexpr int kMaxCells = kCluster64Cells;
  template <class... X>
  static __device__ __forceinline__ double relax(X... x) {
    return relax_value<R>(x...);
  }
  template <class... X>
  static __device__ __forceinline__ double resid(X... x) {
    return resid_value<R>(x...);
  }
  static __device__ __forceinline__ double mean8(double r0, double r1, double r2, double r3, double r4, double r5,
                                                 double r6, double r7) {
    return 0.125 * (r0 + r1 + r2 + r3 + r4 + r5 + r6 + r7);
  }
  // u of a coarse node array at fine node (i, j, k)
  static __device__ __forceinline__ double coarse(const double *uc, Dims dc, int i, int j, int k, int) {
    return uc[dc.ix((i >> 1) + 1, (j >> 1) + 1, (k >> 1) + 1)];
  }
  static __device__ __forceinline__ double prolong(const double *buf, int nx, int ny, int, int c0, int x, int y, int k,
                                                   int) {
    return buf[((k >> 1) - c0) * nx * ny + (y >> 1) * nx + (x >> 1)];
  }
};

template <Round R>
__global__ void __launch_bounds__(mgc::kThreads, 1) k_cluster64(const __grid_constant__ mgc::Args<double> G) {
  mgc::cluster_mg<Cluster64<R>>(G);
}

template <Round R>
__global__ void __launch_bounds__(mgg::kThreads, 1) k_grid64(const __grid_constant__ mgg::Args<double> G) {
  mgg::phase<Cluster64<R>, kGrid64Cells, kGrid64Halo, false>(G);
}

// Residual of an interior cell, its neighbours' values from memory.
template <Round R>
__device__ __forceinline__ double cell_resid(const double *__restrict__ u, const double *__restrict__ rhs,
                                             const double *__restrict__ a, const double *__restrict__ b,
                                             const double *__restrict__ c, size_t q, size_t sy, size_t sz,
                                             double h2i) {
  return resid_value<R>(u[q], u[q + 1], u[q - 1], u[q + sy], u[q - sy], u[q + sz], u[q - sz], a[q], a[q - 1], b[q],
                        b[q - sy], c[q], c[q - sz], rhs[q], h2i);
}

// ---- resid (main.f:3912-3925), reads the ghosts from memory ----------------
template <Round R>
__global__ void k_resid(double *__restrict__ res, const double *__restrict__ u,
                        const double *__restrict__ rhs, const double *__restrict__ a,
                        const double *__restrict__ b, const double *__restrict__ c, Dims d,
                        double h2i) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 2;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 2;
  const int k = blockIdx.z + 2;
  if (i > d.nx - 1 || j > d.ny - 1) return;
  const size_t q = d.ix(i, j, k);
  res[q] = cell_resid<R>(u, rhs, a, b, c, q, d.sy(), d.sz(), h2i);
}

// ---- resid and rstrct in one pass (main.f:3718-3726) -----------------------
// Coarse right-hand side = mean of the 8 fine residuals, coarse correction = 0
// (interiors; the sweeps read ghosts virtually).  The residual itself is not
// stored.  A thread forms the four residuals of fine column i in a coarse
// cell's y-z square, and the even lane of a pair adds the pair's eight in
// rstrct's order (128^3: 83 us, one pass where resid, its ghosts, rstrct and
// the zeroing took 79 + 6 + 20 us and a residual array).
template <Round R>
__global__ void k_resid_rstrct(double *__restrict__ rhs_c, double *__restrict__ u_c, const double *__restrict__ u,
                               const double *__restrict__ rhs, const double *__restrict__ a,
                               const double *__restrict__ b, const double *__restrict__ c, Dims dc, Dims df,
                               double h2i) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 2;  // fine column; blockDim.x = 32
  const int jc = blockIdx.y * blockDim.y + threadIdx.y + 2, kc = blockIdx.z + 2;
  if (jc > dc.ny - 1) return;
  const size_t sy = df.sy(), sz = df.sz();
  double r[4] = {0.0, 0.0, 0.0, 0.0};
  if (i <= df.nx - 1) {
#pragma unroll
    for (int m = 0; m < 4; m++) {
      const int j = 2 * jc - 2 + (m & 1), k = 2 * kc - 2 + (m >> 1);
      const size_t q = df.ix(i, j, k);
      const double uc = u[q];
      r[m] = resid_value<R>(uc, i + 1 == df.nx ? 0.0 : u[q + 1], i == 2 ? uc : u[q - 1], j + 1 == df.ny ? uc : u[q + sy],
                            j == 2 ? uc : u[q - sy], k + 1 == df.nz ? uc : u[q + sz], k == 2 ? uc : u[q - sz], a[q],
                            a[q - 1], b[q], b[q - sy], c[q], c[q - sz], rhs[q], h2i);
    }
  }
  double o[4];
#pragma unroll
  for (int m = 0; m < 4; m++) o[m] = __shfl_down_sync(0xffffffffu, r[m], 1);
  if ((i & 1) || i > df.nx - 1) return;
  const size_t qc = dc.ix(i / 2 + 1, jc, kc);
  rhs_c[qc] = 0.125 * (r[0] + o[0] + r[1] + o[1] + r[2] + o[2] + r[3] + o[3]);
  u_c[qc] = 0.0;
}

// ---- rstrct fused with the coarse bc_scalar (main.f:3765-3791) ------------
__global__ void k_rstrct(double *__restrict__ uc, const double *__restrict__ uf, Dims dc, Dims df) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  const int k = blockIdx.z + 1;
  if (i > dc.nx || j > dc.ny) return;
  if (i == dc.nx && (j >= 2 && j <= dc.ny - 1 && k >= 2 && k <= dc.nz - 1)) {
    uc[dc.ix(i, j, k)] = 0.0;
    return;
  }
  if (i == dc.nx) { uc[dc.ix(i, j, k)] = 0.0; return; }
  const int ci = i == 1 ? 2 : i;
  const int cj = j == 1 ? 2 : (j == dc.ny ? dc.ny - 1 : j);
  const int ck = k == 1 ? 2 : (k == dc.nz ? dc.nz - 1 : k);
  const int fi = 2 * ci - 2, fj = 2 * cj - 2, fk = 2 * ck - 2;
  const size_t f = df.ix(fi, fj, fk);
  const size_t sy = df.sy(), sz = df.sz();
  uc[dc.ix(i, j, k)] = 0.125 * (uf[f] + uf[f + 1] + uf[f + sy] + uf[f + 1 + sy] + uf[f + sz] +
                                uf[f + 1 + sz] + uf[f + sy + sz] + uf[f + 1 + sy + sz]);
}

// ---- interp fused with the fine bc_scalar (main.f:3866-3900) --------------
__global__ void k_interp(double *__restrict__ uf, const double *__restrict__ uc, Dims df, Dims dc) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  const int k = blockIdx.z + 1;
  if (i > df.nx || j > df.ny) return;
  double x = 0.0;
  if (i != df.nx) {
    const int ci = i == 1 ? 2 : i;
    const int cj = j == 1 ? 2 : (j == df.ny ? df.ny - 1 : j);
    const int ck = k == 1 ? 2 : (k == df.nz ? df.nz - 1 : k);
    x = uc[dc.ix((ci >> 1) + 1, (cj >> 1) + 1, (ck >> 1) + 1)];
  }
  uf[df.ix(i, j, k)] = x;
}

// ---- addint: res = interp(uc) (+bc_scalar); uf += res everywhere ----------
// (res may be null where no one reads it)
__global__ void k_addint(double *__restrict__ uf, double *__restrict__ res, const double *__restrict__ uc,
                         Dims df, Dims dc) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  const int k = blockIdx.z + 1;
  if (i > df.nx || j > df.ny) return;
  double x = 0.0;
  if (i != df.nx) {
    const int ci = i == 1 ? 2 : i;
    const int cj = j == 1 ? 2 : (j == df.ny ? df.ny - 1 : j);
    const int ck = k == 1 ? 2 : (k == df.nz ? df.nz - 1 : k);
    x = uc[dc.ix((ci >> 1) + 1, (cj >> 1) + 1, (ck >> 1) + 1)];
  }
  const size_t q = df.ix(i, j, k);
  if (res) res[q] = x;
  uf[q] = uf[q] + x;
}

// ---- acfromac (main.f:3793-3844), one thread per coarse cell --------------
__device__ __forceinline__ double ac_a(const double *a2, Dims df, int i, int j, int k) {
  return 0.25 * (a2[df.ix(2 * i - 1, 2 * j - 1, 2 * k - 1)] + a2[df.ix(2 * i - 1, 2 * j - 2, 2 * k - 1)] +
                 a2[df.ix(2 * i - 1, 2 * j - 1, 2 * k - 2)] + a2[df.ix(2 * i - 1, 2 * j - 2, 2 * k - 2)]);
}
__device__ __forceinline__ double ac_b(const double *b2, Dims df, int i, int j, int k) {
  return 0.25 * (b2[df.ix(2 * i - 1, 2 * j - 1, 2 * k - 1)] + b2[df.ix(2 * i - 2, 2 * j - 1, 2 * k - 1)] +
                 b2[df.ix(2 * i - 1, 2 * j - 1, 2 * k - 2)] + b2[df.ix(2 * i - 2, 2 * j - 1, 2 * k - 2)]);
}
__device__ __forceinline__ double ac_c(const double *c2, Dims df, int i, int j, int k) {
  return 0.25 * (c2[df.ix(2 * i - 1, 2 * j - 1, 2 * k - 1)] + c2[df.ix(2 * i - 2, 2 * j - 1, 2 * k - 1)] +
                 c2[df.ix(2 * i - 1, 2 * j - 2, 2 * k - 1)] + c2[df.ix(2 * i - 2, 2 * j - 2, 2 * k - 1)]);
}

__global__ void k_acfromac(double *__restrict__ a, double *__restrict__ b, double *__restrict__ c,
                           double *__restrict__ ei, const double *__restrict__ a2,
                           const double *__restrict__ b2, const double *__restrict__ c2, Dims dc,
                           Dims df) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  const int k = blockIdx.z + 1;
  if (i > dc.nx || j > dc.ny) return;
  const bool ii = i >= 2 && i <= dc.nx - 1, ji = j >= 2 && j <= dc.ny - 1, ki = k >= 2 && k <= dc.nz - 1;
  const size_t q = dc.ix(i, j, k);
  double va = 0.0, vb = 0.0, vc = 0.0;
  if (i <= dc.nx - 1 && ji && ki) { va = ac_a(a2, df, i, j, k); a[q] = va; }
  if (j <= dc.ny - 1 && ii && ki) { vb = ac_b(b2, df, i, j, k); b[q] = vb; }
  if (k <= dc.nz - 1 && ii && ji) { vc = ac_c(c2, df, i, j, k); c[q] = vc; }
  if (ii && ji && ki) {
    const double am = ac_a(a2, df, i - 1, j, k);
    const double bm = ac_b(b2, df, i, j - 1, k);
    const double cm = ac_c(c2, df, i, j, k - 1);
    ei[q] = 1.0 / (va + am + vb + bm + vc + cm);
  }
}

// ---- abcei (main.f:3582-3615) and bc_coef (main.f:4465-4494) --------------
// Face coefficients, ei = 1 / (sum of the six) and, with diag non-null, the sum
// itself (the diagonal of the operator, for the mixed solve's flux-form
// defect), in one pass: a cell forms its lower faces again, with the
// neighbour's operations, instead of reading them back.  Cells of one phase
// with their neighbours take values formed once on the host with the same
// operations.  256^3: 207 us as two kernels, 177 now
// (118 us of memory traffic).
struct Bulk64 {
  double k[2], e[2], d[2];  // face coefficient, ei and sum of gas and of liquid
};
__global__ void __launch_bounds__(kBandThreads) k_abcei(double *__restrict__ a, double *__restrict__ b,
                                                        double *__restrict__ c, double *__restrict__ ei,
                                                        double *__restrict__ diag, const double *__restrict__ cc,
                                                        double r1, double r2, Bulk64 B, Dims d) {
  const size_t sy = d.sy(), sz = d.sz();
  bulk_then_cells<1>(d, [&](int i, int j, int k, int) {
    const size_t q = d.ix(i, j, k);
    const double c0 = cc[q];
    const bool gas = is_zero_bits(c0);
    if (!((gas | is_one_bits(c0)) & same_bits(cc[q + 1], c0) & same_bits(cc[q - 1], c0) & same_bits(cc[q + sy], c0) &
          same_bits(cc[q - sy], c0) & same_bits(cc[q + sz], c0) & same_bits(cc[q - sz], c0)))
      return false;
    a[q] = b[q] = c[q] = gas ? B.k[0] : B.k[1];
    ei[q] = gas ? B.e[0] : B.e[1];
    if (diag) diag[q] = gas ? B.d[0] : B.d[1];
    return true;
  }, [&](int i, int j, int k) {
    const size_t q = d.ix(i, j, k);
    const double c0 = cc[q];
    auto face = [&](double lo, double hi) { return 1.0 / (r1 * (lo + hi) + r2); };
    const double s0 = face(c0, cc[q + 1]), s2 = face(c0, cc[q + sy]), s4 = face(c0, cc[q + sz]);
    // bc_coef's a(1) = a(2)
    const double s1 = i == 2 ? s0 : face(cc[q - 1], c0), s3 = face(cc[q - sy], c0), s5 = face(cc[q - sz], c0);
    a[q] = s0;
    b[q] = s2;
    c[q] = s4;
    const double sum = s0 + s1 + s2 + s3 + s4 + s5;
    ei[q] = 1.0 / sum;
    if (diag) diag[q] = sum;
  });
}

// bc_coef: face 0 = a x-faces (all j,k), 1 = b(i,1,k) (i,k interior),
// 2 = c(i,j,1) (i interior, all j).
__global__ void k_bc_coef(double *__restrict__ a, double *__restrict__ b, double *__restrict__ c,
                          const double *__restrict__ cc, double r1, double r2, Dims d) {
  const int face = blockIdx.z;
  const int p = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int q = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (face == 0) {
    if (p > d.ny || q > d.nz) return;
    a[d.ix(1, p, q)] = a[d.ix(2, p, q)];
    a[d.ix(d.nx, p, q)] = a[d.ix(d.nx - 1, p, q)];
  } else if (face == 1) {
    if (p < 2 || p > d.nx - 1 || q < 2 || q > d.nz - 1) return;
    b[d.ix(p, 1, q)] = 1.0 / (r1 * (cc[d.ix(p, 1, q)] + cc[d.ix(p, 2, q)]) + r2);
  } else {
    if (p < 2 || p > d.nx - 1 || q > d.ny) return;
    c[d.ix(p, q, 1)] = 1.0 / (r1 * (cc[d.ix(p, q, 1)] + cc[d.ix(p, q, 2)]) + r2);
  }
}

// diag = the sum of the six face coefficients of every interior cell.
__global__ void k_diag(double *__restrict__ diag, const double *__restrict__ a, const double *__restrict__ b,
                       const double *__restrict__ c, Dims d) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 2;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 2;
  const int k = blockIdx.z + 2;
  if (i > d.nx - 1 || j > d.ny - 1) return;
  const size_t q = d.ix(i, j, k);
  diag[q] = a[q] + a[q - 1] + b[q] + b[q - d.sy()] + c[q] + c[q - d.sz()];
}

// ---- filterc27 (main.f:5473-5511), default-REAL weights -------------------
template <int P>
__global__ void __launch_bounds__(kBandThreads) k_filterc27(const double *__restrict__ cc, double *__restrict__ cf, Dims d) {
  const double w0 = (double)0.2729f, w1 = (double)0.08185f, w2 = (double)0.0178f, w3 = (double)0.0028f;
  const long sy = (long)d.sy(), sz = (long)d.sz();
#define C(di, dj, dk) cc[(long)q + (long)(di) + (long)(dj) * sy + (long)(dk) * sz]
  const Flat<P> flat(cc, d);
  bulk_then_cells<P>(d, [&](int i, int j, int k, int p) {
    // Uniform 27-point neighbourhood of 0 or 1: the partial sums are exact
    // multiples of the value, so the weighted sum equals the precomputed one.
    const bool gas = is_zero_bits(flat.f[p + 1]);
    if (!((gas | is_one_bits(flat.f[p + 1])) & flat.uniform(p, true))) return false;
    const size_t q = d.ix(i, j, k);
    double x = gas ? 0.0 : w0 * 1.0 + w1 * 6.0 + w2 * 12.0 + w3 * 8.0;
    if (x > 1.0) x = 1.0;
    cf[q] = x;
    return true;
  }, [&](int i, int j, int k) {
    const size_t q = d.ix(i, j, k);
    const double s6 = C(-1, 0, 0) + C(1, 0, 0) + C(0, -1, 0) + C(0, 1, 0) + C(0, 0, 1) + C(0, 0, -1);
    const double s12 = C(-1, -1, 0) + C(-1, 1, 0) + C(1, -1, 0) + C(1, 1, 0) + C(0, 1, 1) + C(0, -1, 1) +
                       C(1, 0, 1) + C(-1, 0, 1) + C(0, 1, -1) + C(0, -1, -1) + C(1, 0, -1) + C(-1, 0, -1);
    const double s8 = C(1, 1, 1) + C(1, 1, -1) + C(1, -1, 1) + C(1, -1, -1) + C(-1, 1, 1) + C(-1, 1, -1) +
                      C(-1, -1, 1) + C(-1, -1, -1);
    double x = w0 * C(0, 0, 0) + w1 * s6 + w2 * s12 + w3 * s8;
    if (x > 1.0) x = 1.0;
    cf[q] = x;
  });
#undef C
}

// ---- deterministic block reductions ----------------------------------------
template <int K>
__device__ __forceinline__ void block_sum_store(double (&v)[K], double *out) {
  __shared__ double sh[K][kRedThreads / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int m = 0; m < K; m++) {
    double x = v[m];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) sh[m][w] = x;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int m = 0; m < K; m++) {
      double x = 0.0;
      for (int q = 0; q < kRedThreads / 32; q++) x += sh[m][q];
      out[(size_t)blockIdx.x * K + m] = x;
    }
  }
}

template <int K>
__device__ __forceinline__ void block_max_store(double (&v)[K], double *out) {
  __shared__ double sh[K][kRedThreads / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int m = 0; m < K; m++) {
    double x = v[m];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x = fmax(x, __shfl_down_sync(0xffffffffu, x, o));
    if (lane == 0) sh[m][w] = x;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int m = 0; m < K; m++) {
      double x = sh[m][0];
      for (int q = 1; q < kRedThreads / 32; q++) x = fmax(x, sh[m][q]);
      out[(size_t)blockIdx.x * K + m] = x;
    }
  }
}

// Second stage: one block folds kRedBlocks partials (fixed order).
template <int K, bool MAX>
__global__ void k_fold(const double *__restrict__ partials, double *__restrict__ out) {
  double v[K];
#pragma unroll
  for (int m = 0; m < K; m++) v[m] = MAX ? -1.0 : 0.0;
  for (int b = threadIdx.x; b < kRedBlocks; b += kRedThreads)
#pragma unroll
    for (int m = 0; m < K; m++) {
      const double x = partials[(size_t)b * K + m];
      v[m] = MAX ? fmax(v[m], x) : v[m] + x;
    }
  __shared__ double sh[K][kRedThreads];
#pragma unroll
  for (int m = 0; m < K; m++) sh[m][threadIdx.x] = v[m];
  __syncthreads();
  for (int s = kRedThreads / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s)
#pragma unroll
      for (int m = 0; m < K; m++)
        sh[m][threadIdx.x] = MAX ? fmax(sh[m][threadIdx.x], sh[m][threadIdx.x + s])
                                 : sh[m][threadIdx.x] + sh[m][threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0)
#pragma unroll
    for (int m = 0; m < K; m++) out[m] = sh[m][0];
}

// Interior cell of flat interior index t (i fastest).
// Interior cell t -> (i, j, k) with 32-bit division (interior counts stay
// below 2^32; 64-bit division is a long instruction sequence).
__device__ __forceinline__ size_t interior_cell(size_t t, Dims d, int &i, int &j, int &k) {
  const unsigned ni = (unsigned)(d.nx - 2), nj = (unsigned)(d.ny - 2), tt = (unsigned)t;
  const unsigned r = tt / ni;
  i = (int)(tt - r * ni) + 2;
  const unsigned kk = r / nj;
  j = (int)(r - kk * nj) + 2;
  k = (int)kk + 2;
  return d.ix(i, j, k);
}

// |x| as an ordered integer: the bit pattern of a non-negative double orders
// like its value, so maxima of |x| run on the integer pipe (a NaN is the
// largest pattern and propagates).
__device__ __forceinline__ long long abs_bits(double x) {
  return __double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFLL;
}

template <bool F>
__global__ void k_relres_partial(double *__restrict__ partials, const double *__restrict__ u,
                                 const double *__restrict__ rhs, const double *__restrict__ a,
                                 const double *__restrict__ b, const double *__restrict__ c, Dims d,
                                 double h2i) {
  const size_t n = (size_t)(d.nx - 2) * (d.ny - 2) * (d.nz - 2);
  const size_t sy = d.sy(), sz = d.sz();
  double v[2] = {0.0, 0.0};
  for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x) {
    int i, j, k;
    const size_t q = interior_cell(t, d, i, j, k);
    const double r = cell_resid<F ? FMA : REF>(u, rhs, a, b, c, q, sy, sz, h2i);
    if (F) {
      v[0] = __fma_rn(r, r, v[0]);
      v[1] = __fma_rn(rhs[q], rhs[q], v[1]);
    } else {
      v[0] += r * r;
      v[1] += rhs[q] * rhs[q];
    }
  }
  block_sum_store<2>(v, partials);
}

__global__ void k_sum_partial(double *__restrict__ partials, const double *__restrict__ f, Dims d) {
  const size_t n = (size_t)(d.nx - 2) * (d.ny - 2) * (d.nz - 2);
  double v[1] = {0.0};
  for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x) {
    int i, j, k;
    v[0] += f[interior_cell(t, d, i, j, k)];
  }
  block_sum_store<1>(v, partials);
}

__global__ void k_absmax3_partial(double *__restrict__ partials, const double *__restrict__ f0,
                                  const double *__restrict__ f1, const double *__restrict__ f2, Dims d) {
  const size_t n = (size_t)(d.nx - 2) * (d.ny - 2) * (d.nz - 2);
  long long m = 0;
  for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x) {
    int i, j, k;
    const size_t q = interior_cell(t, d, i, j, k);
    m = max(m, abs_bits(f0[q]));
    if (f1) m = max(m, abs_bits(f1[q]));
    if (f2) m = max(m, abs_bits(f2[q]));
  }
  double v[1] = {__longlong_as_double(m)};
  block_max_store<1>(v, partials);
}

__global__ void k_divmax_partial(double *__restrict__ partials, const double *__restrict__ u,
                                 const double *__restrict__ v_, const double *__restrict__ w, Dims d,
                                 double hi2) {
  const size_t n = (size_t)(d.nx - 2) * (d.ny - 2) * (d.nz - 2);
  const size_t sy = d.sy(), sz = d.sz();
  long long m = 0;
  for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x) {
    int i, j, k;
    const size_t q = interior_cell(t, d, i, j, k);
    const double dv = (u[q + 1] - u[q] + v_[q + sy] - v_[q] + w[q + sz] - w[q]) * hi2;
    m = max(m, abs_bits(dv));
  }
  double v[1] = {__longlong_as_double(m)};
  block_max_store<1>(v, partials);
}

const dim3 kBlk(32, 4, 1);

dim3 face_grid(Dims d, dim3 blk) {
  int m = d.nx > d.ny ? d.nx : d.ny;
  m = m > d.nz ? m : d.nz;
  return dim3((unsigned)((m + blk.x - 1) / blk.x), (unsigned)((m + blk.y - 1) / blk.y), 6);
}

dim3 full_grid(Dims d, dim3 blk) {
  return dim3((unsigned)((d.nx + blk.x - 1) / blk.x), (unsigned)((d.ny + blk.y - 1) / blk.y), (unsigned)d.nz);
}

}  // namespace

// ---- host launchers ---------------------------------------------------------
cudaError_t bc_scalar(double *s, Dims d, cudaStream_t st) {
  const dim3 blk(32, 8);
  DSG_COUNT k_bc_scalar<<<face_grid(d, blk), blk, 0, st>>>(s, d);
  return cudaGetLastError();
}

static dim3 bc_grid(Dims d) {
  const int p = d.nx > d.ny ? d.nx : d.ny, q = d.ny > d.nz ? d.ny : d.nz;
  return dim3((unsigned)((p + 31) / 32), (unsigned)((q + 7) / 8), 3);
}

cudaError_t bc_resid(double *s, Dims d, cudaStream_t st) {
  DSG_COUNT k_bc_copy<true><<<bc_grid(d), dim3(32, 8), 0, st>>>(s, d);
  return cudaGetLastError();
}

cudaError_t bc_out(double *s, Dims d, cudaStream_t st) {
  DSG_COUNT k_bc_copy<false><<<bc_grid(d), dim3(32, 8), 0, st>>>(s, d);
  return cudaGetLastError();
}

// The form of the sweeps and residuals on spacing h2: the fused multiply-add
// chain, or the reference's rounding in as few operations as h2 and omega allow.
static Round rounding(bool fma, double h2, double omega) {
  return fma ? FMA : (power_of_two(h2) && power_of_two(1.0 - omega) ? REF2 : REF);
}

template <Round R>
static void relax_passes(int n, double *u, double h2, const double *rhs, const double *a, const double *b,
                         const double *c, const double *ei, Dims d, double omega, cudaStream_t st, const Products *P) {
  const dim3 grid((plane_warps(d) + 3) / 4, (unsigned)(d.nz - 2));
  Products S = P ? *P : Products{};
  S.keep = 1.0 - omega;
  S.w = omega * (S.k * S.e);
  S.z = -omega * (h2 * S.e);
  S.w1 = omega * (S.k1 * S.e1);
  S.z1 = -omega * (h2 * S.e1);
  auto pass = [&](auto kernel, int colour) {
    DSG_COUNT kernel<<<grid, 128, 0, st>>>(u, rhs, a, b, c, ei, d, h2, omega, colour, S);
  };
  for (int q = 0; q < n; q++)
    for (int colour = 0; colour < 2; colour++) {
      const bool last = q == n - 1;
      if (!P)
        last ? pass(k_relax_colour<R, true, 0>, colour) : pass(k_relax_colour<R, false, 0>, colour);
      else if (R != FMA && q == 0 && colour == 0)
        last ? pass(k_relax_colour<R, true, 1>, colour) : pass(k_relax_colour<R, false, 1>, colour);
      else
        last ? pass(k_relax_colour<R, true, 2>, colour) : pass(k_relax_colour<R, false, 2>, colour);
    }
}

int cluster64_size() {
  const int n = mgc::cluster_size(k_cluster64<REF>);
  return mgc::cluster_size(k_cluster64<REF2>) < n || mgc::cluster_size(k_cluster64<FMA>) < n ? 0 : n;
}

cudaError_t cluster64(const mgc::Args<double> &args, bool fma, cudaStream_t st) {
  Round r = rounding(fma, args.lv[1].h2, args.omega);
  for (int l = 2; l <= args.top && r == REF2; l++) r = rounding(fma, args.lv[l].h2, args.omega);
  return r == FMA ? mgc::launch(k_cluster64<FMA>, args, st)
                  : (r == REF2 ? mgc::launch(k_cluster64<REF2>, args, st) : mgc::launch(k_cluster64<REF>, args, st));
}

int grid64_blocks() { return mgg::grid_blocks(mgg::kThreads, mgg::kMaxShared, k_grid64<REF>, k_grid64<REF2>, k_grid64<FMA>); }

cudaError_t grid64(const mgg::Args<double> &args, bool fma, cudaStream_t st) {
  switch (rounding(fma, args.h2, args.omega)) {
    case FMA: return mgg::launch(k_grid64<FMA>, mgg::kThreads, args, st);
    case REF2: return mgg::launch(k_grid64<REF2>, mgg::kThreads, args, st);
    default: return mgg::launch(k_grid64<REF>, mgg::kThreads, args, st);
  }
}

cudaError_t relax(double *u, double lengthsize, const double *rhs, const double *a, const double *b,
                  const double *c, const double *ei, Dims d, double omega, cudaStream_t st) {
  return relax_n(1, u, lengthsize, rhs, a, b, c, ei, d, omega, st);
}

cudaError_t relax_n(int n, double *u, double lengthsize, const double *rhs, const double *a,
                    const double *b, const double *c, const double *ei, Dims d, double omega,
                    cudaStream_t st, bool fma, const Products *P) {
  if (n <= 0) return cudaSuccess;
  const double h1 = lengthsize / (d.nx - 2);
  const double h2 = h1 * h1;
  switch (rounding(fma, h2, omega)) {
    case FMA: relax_passes<FMA>(n, u, h2, rhs, a, b, c, ei, d, omega, st, P); break;
    case REF2: relax_passes<REF2>(n, u, h2, rhs, a, b, c, ei, d, omega, st, P); break;
    default: relax_passes<REF>(n, u, h2, rhs, a, b, c, ei, d, omega, st, P);
  }
  return cudaGetLastError();
}

cudaError_t bulk_flags(const Products &P, const double *a, const double *b, const double *c, const double *ei, Dims d,
                       cudaStream_t st) {
  const size_t warps = (size_t)plane_warps(d) * (d.nz - 2);
  DSG_COUNT k_bulk_flags<<<(unsigned)std::min<size_t>((warps + 7) / 8, 152 * 32), 256, 0, st>>>(P.flags, a, b, c, ei, d, P);
  return cudaGetLastError();
}

cudaError_t resid(double lengthsize, double *res, const double *u, const double *rhs, const double *a,
                  const double *b, const double *c, Dims d, cudaStream_t st, bool fma) {
  const double h1 = lengthsize / (d.nx - 2);
  const double h2i = 1.0 / (h1 * h1);
  switch (rounding(fma, h2i, 1.5)) {
    case FMA: DSG_COUNT k_resid<FMA><<<interior_grid(d, kBlk), kBlk, 0, st>>>(res, u, rhs, a, b, c, d, h2i); break;
    case REF2: DSG_COUNT k_resid<REF2><<<interior_grid(d, kBlk), kBlk, 0, st>>>(res, u, rhs, a, b, c, d, h2i); break;
    default: DSG_COUNT k_resid<REF><<<interior_grid(d, kBlk), kBlk, 0, st>>>(res, u, rhs, a, b, c, d, h2i);
  }
  return bc_resid(res, d, st);
}

cudaError_t resid_rstrct(double lengthsize, double *rhs_c, double *u_c, const double *u, const double *rhs,
                         const double *a, const double *b, const double *c, Dims df, cudaStream_t st, bool fma) {
  const double h1 = lengthsize / (df.nx - 2);
  const double h2i = 1.0 / (h1 * h1);
  const Dims dc{df.nx / 2 + 1, df.ny / 2 + 1, df.nz / 2 + 1};
  const dim3 grid((unsigned)((df.nx - 2 + 31) / 32), (unsigned)((dc.ny - 2 + 3) / 4), (unsigned)(dc.nz - 2));
  switch (rounding(fma, h2i, 1.5)) {
    case FMA: DSG_COUNT k_resid_rstrct<FMA><<<grid, kBlk, 0, st>>>(rhs_c, u_c, u, rhs, a, b, c, dc, df, h2i); break;
    case REF2: DSG_COUNT k_resid_rstrct<REF2><<<grid, kBlk, 0, st>>>(rhs_c, u_c, u, rhs, a, b, c, dc, df, h2i); break;
    default: DSG_COUNT k_resid_rstrct<REF><<<grid, kBlk, 0, st>>>(rhs_c, u_c, u, rhs, a, b, c, dc, df, h2i);
  }
  return cudaGetLastError();
}

cudaError_t rstrct(double *uc, const double *uf, Dims dc, cudaStream_t st) {
  const Dims df{2 * dc.nx - 2, 2 * dc.ny - 2, 2 * dc.nz - 2};
  DSG_COUNT k_rstrct<<<full_grid(dc, kBlk), kBlk, 0, st>>>(uc, uf, dc, df);
  return cudaGetLastError();
}

cudaError_t interp(double *uf, const double *uc, Dims df, cudaStream_t st) {
  const Dims dc{df.nx / 2 + 1, df.ny / 2 + 1, df.nz / 2 + 1};
  DSG_COUNT k_interp<<<full_grid(df, kBlk), kBlk, 0, st>>>(uf, uc, df, dc);
  return cudaGetLastError();
}

cudaError_t addint(double *uf, const double *uc, double *res, Dims df, cudaStream_t st) {
  const Dims dc{df.nx / 2 + 1, df.ny / 2 + 1, df.nz / 2 + 1};
  DSG_COUNT k_addint<<<full_grid(df, kBlk), kBlk, 0, st>>>(uf, res, uc, df, dc);
  return cudaGetLastError();
}

cudaError_t acfromac(double *a, double *b, double *c, double *ei, const double *a2, const double *b2,
                     const double *c2, Dims dc, cudaStream_t st) {
  const Dims df{2 * dc.nx - 2, 2 * dc.ny - 2, 2 * dc.nz - 2};
  DSG_COUNT k_acfromac<<<full_grid(dc, kBlk), kBlk, 0, st>>>(a, b, c, ei, a2, b2, c2, dc, df);
  return cudaGetLastError();
}

cudaError_t abcei(double *a, double *b, double *c, double *ei, const double *cc, double r1, double r2,
                  Dims d, cudaStream_t st, double *diag) {
  // bulk constants, same operation order as the kernel
  Bulk64 B;
  for (int q = 0; q < 2; q++) {
    const double k = 1.0 / (r1 * ((double)q + (double)q) + r2), sum = k + k + k + k + k + k;
    B.k[q] = k;
    B.d[q] = sum;
    B.e[q] = 1.0 / sum;
  }
  DSG_COUNT k_abcei<<<band_grid(d, 1), dim3(32, 8), 0, st>>>(a, b, c, ei, diag, cc, r1, r2, B, d);
  const dim3 blk(32, 8);
  DSG_COUNT k_bc_coef<<<face_grid(d, blk), blk, 0, st>>>(a, b, c, cc, r1, r2, d);
  return cudaGetLastError();
}

cudaError_t diag_sum(double *diag, const double *a, const double *b, const double *c, Dims d, cudaStream_t st) {
  DSG_COUNT k_diag<<<interior_grid(d, kBlk), kBlk, 0, st>>>(diag, a, b, c, d);
  return cudaGetLastError();
}

cudaError_t filterc27(const double *cc, double *cf, Dims d, cudaStream_t st) {
  DSG_BAND(k_filterc27, d, st, cc, cf, d);
  return cudaGetLastError();
}

cudaError_t relres_sums(double *out, double *partials, double lengthsize, const double *u,
                        const double *rhs, const double *a, const double *b, const double *c, Dims d,
                        cudaStream_t st, bool fma) {
  const double h1 = lengthsize / (d.nx - 2);
  const double h2i = 1.0 / (h1 * h1);
  if (fma)
    DSG_COUNT k_relres_partial<true><<<kRedBlocks, kRedThreads, 0, st>>>(partials, u, rhs, a, b, c, d, h2i);
  else
    DSG_COUNT k_relres_partial<false><<<kRedBlocks, kRedThreads, 0, st>>>(partials, u, rhs, a, b, c, d, h2i);
  DSG_COUNT k_fold<2, false><<<1, kRedThreads, 0, st>>>(partials, out);
  return cudaGetLastError();
}

cudaError_t sumfield(double *out, double *partials, const double *f, Dims d, cudaStream_t st) {
  DSG_COUNT k_sum_partial<<<kRedBlocks, kRedThreads, 0, st>>>(partials, f, d);
  DSG_COUNT k_fold<1, false><<<1, kRedThreads, 0, st>>>(partials, out);
  return cudaGetLastError();
}

cudaError_t absmax3(double *out, double *partials, const double *f0, const double *f1, const double *f2,
                    Dims d, cudaStream_t st) {
  DSG_COUNT k_absmax3_partial<<<kRedBlocks, kRedThreads, 0, st>>>(partials, f0, f1, f2, d);
  DSG_COUNT k_fold<1, true><<<1, kRedThreads, 0, st>>>(partials, out);
  return cudaGetLastError();
}

cudaError_t divmax(double *out, double *partials, const double *u, const double *v, const double *w,
                   double hi2, Dims d, cudaStream_t st) {
  DSG_COUNT k_divmax_partial<<<kRedBlocks, kRedThreads, 0, st>>>(partials, u, v, w, d, hi2);
  DSG_COUNT k_fold<1, true><<<1, kRedThreads, 0, st>>>(partials, out);
  return cudaGetLastError();
}

cudaError_t fill_zero(double *f, size_t n, cudaStream_t st) {
  return cudaMemsetAsync(f, 0, n * sizeof(double), st);
}

}  // namespace dsg

// ---- array-level C ABI --------------------------------------------------------
static int check_dims(int nx, int ny, int nz) {
  return (nx >= 3 && ny >= 3 && nz >= 3) ? DSG_OK : DSG_E_ARG;
}
static int cuda_rc(cudaError_t e) { return e == cudaSuccess ? DSG_OK : DSG_E_CUDA; }

extern "C" int dsg_relax(double *u, double lengthsize, const double *rhs, const double *a, const double *b,
                         const double *c, const double *ei, int nx, int ny, int nz, double omega,
                         void *stream) {
  if (check_dims(nx, ny, nz) || !u || !rhs || !a || !b || !c || !ei) return DSG_E_ARG;
  return cuda_rc(dsg::relax(u, lengthsize, rhs, a, b, c, ei, dsg::Dims{nx, ny, nz}, omega,
                            (cudaStream_t)stream));
}

extern "C" int dsg_resid(double lengthsize, double *res, const double *u, const double *rhs,
                         const double *a, const double *b, const double *c, int nx, int ny, int nz,
                         void *stream) {
  if (check_dims(nx, ny, nz) || !res || !u || !rhs || !a || !b || !c) return DSG_E_ARG;
  return cuda_rc(dsg::resid(lengthsize, res, u, rhs, a, b, c, dsg::Dims{nx, ny, nz}, (cudaStream_t)stream));
}

extern "C" int dsg_rstrct(double *uc, const double *uf, int ncx, int ncy, int ncz, void *stream) {
  if (check_dims(ncx, ncy, ncz) || !uc || !uf) return DSG_E_ARG;
  return cuda_rc(dsg::rstrct(uc, uf, dsg::Dims{ncx, ncy, ncz}, (cudaStream_t)stream));
}

extern "C" int dsg_interp(double *uf, const double *uc, int nfx, int nfy, int nfz, void *stream) {
  if (check_dims(nfx, nfy, nfz) || !uf || !uc || (nfx & 1) || (nfy & 1) || (nfz & 1)) return DSG_E_ARG;
  return cuda_rc(dsg::interp(uf, uc, dsg::Dims{nfx, nfy, nfz}, (cudaStream_t)stream));
}

extern "C" int dsg_addint(double *uf, const double *uc, double *res, int nfx, int nfy, int nfz, void *stream) {
  if (check_dims(nfx, nfy, nfz) || !uf || !uc || !res || (nfx & 1) || (nfy & 1) || (nfz & 1)) return DSG_E_ARG;
  return cuda_rc(dsg::addint(uf, uc, res, dsg::Dims{nfx, nfy, nfz}, (cudaStream_t)stream));
}

extern "C" int dsg_acfromac(double *a, double *b, double *c, double *ei, const double *a2, const double *b2,
                            const double *c2, int nx, int ny, int nz, void *stream) {
  if (check_dims(nx, ny, nz) || !a || !b || !c || !ei || !a2 || !b2 || !c2) return DSG_E_ARG;
  return cuda_rc(dsg::acfromac(a, b, c, ei, a2, b2, c2, dsg::Dims{nx, ny, nz}, (cudaStream_t)stream));
}

extern "C" int dsg_abcei(double *a, double *b, double *c, double *ei, const double *cc, double r1, double r2,
                         int nx, int ny, int nz, void *stream) {
  if (check_dims(nx, ny, nz) || !a || !b || !c || !ei || !cc) return DSG_E_ARG;
  return cuda_rc(dsg::abcei(a, b, c, ei, cc, r1, r2, dsg::Dims{nx, ny, nz}, (cudaStream_t)stream));
}

extern "C" int dsg_bc_scalar(double *s, int nx, int ny, int nz, void *stream) {
  if (check_dims(nx, ny, nz) || !s) return DSG_E_ARG;
  return cuda_rc(dsg::bc_scalar(s, dsg::Dims{nx, ny, nz}, (cudaStream_t)stream));
}

extern "C" int dsg_bc_resid(double *s, int nx, int ny, int nz, void *stream) {
  if (check_dims(nx, ny, nz) || !s) return DSG_E_ARG;
  return cuda_rc(dsg::bc_resid(s, dsg::Dims{nx, ny, nz}, (cudaStream_t)stream));
}

extern "C" int dsg_bc_out(double *s, int nx, int ny, int nz, void *stream) {
  if (check_dims(nx, ny, nz) || !s) return DSG_E_ARG;
  return cuda_rc(dsg::bc_out(s, dsg::Dims{nx, ny, nz}, (cudaStream_t)stream));
}

extern "C" int dsg_filterc27(const double *cc, double *cf, int nx, int ny, int nz, void *stream) {
  if (check_dims(nx, ny, nz) || !cc || !cf) return DSG_E_ARG;
  return cuda_rc(dsg::filterc27(cc, cf, dsg::Dims{nx, ny, nz}, (cudaStream_t)stream));
}
