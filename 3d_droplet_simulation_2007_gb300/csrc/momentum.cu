// momentum.cu -- the step glue of solvelpres (main.f:3236-3439): viscous stress
// update, explicit predictor with gravity, bc_w (main.f:4143-4220), central
// convection (convective, main.f:3525-3566), bc_v (main.f:4064-4141), the
// divergence right-hand side and the pressure projection.
//
// Laminar runs: mut, turbst and the u2p/uvp... arrays of the reference are zero,
// so the terms they feed add exact zeros and are left out.
#include <cmath>

#include "dsg_internal.cuh"

namespace dsg {
namespace {

// Viscosity factors of the stress update: the cell's r2 + r1 c and the edges'
// r20 + r10 (sum of the four cells around the edge).  Where the seven volume
// fractions a cell reads are all exactly 0 or all exactly 1 (tested on the
// integer pipe), the factors are the precomputed values of the same fused
// multiply-adds (pure[0] for 0, pure[1] for 1: cell, edge), which skips 13 of
// the 31 FP64 operations of a cell on GB300's narrow FP64 pipe with the same
// bits.  The branch is taken per warp.
struct StressPure {
  double cell[2], edge[2];
};

__global__ void k_stress(double *__restrict__ S11, double *__restrict__ S22, double *__restrict__ S33,
                         double *__restrict__ S12, double *__restrict__ S13, double *__restrict__ S23,
                         const double *__restrict__ u, const double *__restrict__ v,
                         const double *__restrict__ w, const double *__restrict__ cc, Dims d, double r1,
                         double r2, double r10, double r20, StressPure pure, int k0) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 2;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 2;
  const int k = blockIdx.z + k0;
  if (i > d.nx - 1 || j > d.ny - 1) return;
  const size_t q = d.ix(i, j, k);
  const size_t sy = d.sy(), sz = d.sz();
  const double c0 = cc[q], c1 = cc[q - 1], c2 = cc[q - sy], c3 = cc[q - 1 - sy], c4 = cc[q - sz],
               c5 = cc[q - 1 - sz], c6 = cc[q - sy - sz];
  const bool one = is_one_bits(c0);
  const bool uniform = (one || is_zero_bits(c0)) && same_bits(c1, c0) && same_bits(c2, c0) && same_bits(c3, c0) &&
                       same_bits(c4, c0) && same_bits(c5, c0) && same_bits(c6, c0);
  double tc, t12, t13, t23;
  if (__all_sync(__activemask(), uniform)) {
    tc = one ? pure.cell[1] : pure.cell[0];
    t12 = t13 = t23 = one ? pure.edge[1] : pure.edge[0];
  } else {
    tc = fma(r1, c0, r2);
    t12 = fma(r10, c0 + c1 + c2 + c3, r20);
    t13 = fma(r10, c0 + c1 + c4 + c5, r20);
    t23 = fma(r10, c0 + c2 + c4 + c6, r20);
  }
  S11[q] = -S11[q] + tc * (u[q + 1] - u[q]);
  S22[q] = -S22[q] + tc * (v[q + sy] - v[q]);
  S33[q] = -S33[q] + tc * (w[q + sz] - w[q]);
  S12[q] = -S12[q] + t12 * (u[q] - u[q - sy] + v[q] - v[q - 1]);
  S13[q] = -S13[q] + t13 * (u[q] - u[q - sz] + w[q] - w[q - 1]);
  S23[q] = -S23[q] + t23 * (v[q] - v[q - sz] + w[q] - w[q - sy]);
}

__global__ void k_predictor(double *__restrict__ w1, double *__restrict__ w2, double *__restrict__ w3,
                            const double *__restrict__ u, const double *__restrict__ v,
                            const double *__restrict__ w, const double *__restrict__ a,
                            const double *__restrict__ b, const double *__restrict__ c,
                            const double *__restrict__ S11, const double *__restrict__ S22,
                            const double *__restrict__ S33, const double *__restrict__ S12,
                            const double *__restrict__ S13, const double *__restrict__ S23, Dims d,
                            double horgrav, double stdgrav, int k0) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 2;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 2;
  const int k = blockIdx.z + k0;
  if (i > d.nx - 1 || j > d.ny - 1) return;
  const size_t q = d.ix(i, j, k);
  const size_t sy = d.sy(), sz = d.sz();
  w1[q] = u[q] + a[q - 1] * (S11[q] - S11[q - 1] + S12[q + sy] - S12[q] + S13[q + sz] - S13[q]) + horgrav;
  w2[q] = v[q] + b[q - sy] * (S12[q + 1] - S12[q] + S22[q] - S22[q - sy] + S23[q + sz] - S23[q]) + stdgrav;
  w3[q] = w[q] + c[q - sz] * (S13[q + 1] - S13[q] + S23[q + sy] - S23[q] + S33[q] - S33[q - sz]);
}

// Explicit convection (main.f's convective): per component three differences of
// products of two-point sums.  The FP64 pipe bounds it, and cell by cell it
// takes 51 instructions per cell, 30 of them sums that its neighbours along x, y
// and z form as well: 1360 us at 256^3.  Here a cell forms nine sums once and
// takes its neighbours': along x by shuffle, along y through shared memory,
// along z from the plane before: 30 instructions.  A block is kConvRows rows of
// 32 cells, one warp each, and marches through `planes` planes; two more warps
// form the sums of the row and the column of cells beyond.  256^3: 963 us,
// 904 at the pipe's rate; 128^3 173 -> 133, 64^3 24.5 -> 22.0.
//
// tauq = 0.25*tauh: the reference's tauh*(0.25*x) equals tauq*x bit for bit
// (scaling by 0.25 is exact, so both round the same product once), one FP64
// multiply per component less.
constexpr int kConvRows = 8, kConvThreads = 32 * (kConvRows + 2);

// p*p - m*m + a*b - c*e + f*g - r*t, rounded as the compiler rounds that expression
__device__ __forceinline__ double flux_balance(double p, double m, double a, double b, double c, double e, double f,
                                               double g, double r, double t) {
  double x = fma(p, p, -(m * m));
  x = fma(a, b, x);
  x = fma(-c, e, x);
  x = fma(f, g, x);
  return fma(-r, t, x);
}

__global__ void __launch_bounds__(kConvThreads) k_convective(double *__restrict__ u, double *__restrict__ v,
                                                             double *__restrict__ w, const double *__restrict__ w1,
                                                             const double *__restrict__ w2,
                                                             const double *__restrict__ w3, Dims d, double tauq,
                                                             int planes) {
  __shared__ double rows[2][5][kConvRows + 1][32], column[2][5][kConvRows];
  const int lane = threadIdx.x & 31, wy = threadIdx.x >> 5;
  const bool beside = wy == kConvRows + 1, below = wy == kConvRows;  // the column's, the row's warp
  int i = 2 + 32 * (int)blockIdx.x + (beside ? 32 : lane);
  int j = 2 + kConvRows * (int)blockIdx.y + (beside ? min(lane, kConvRows - 1) : wy);
  const bool cell = wy < kConvRows && i <= d.nx - 1 && j <= d.ny - 1;
  i = min(i, d.nx);
  j = min(j, d.ny);
  const int k0 = 2 + planes * (int)blockIdx.z, k1 = min(k0 + planes, d.nz);
  const long sy = (long)d.sy(), sz = (long)d.sz();
  long q = (long)d.ix(i, j, k0);
  // sums with the neighbour below: a1x = w1 here + w1 at x - 1, and so on
  double c1 = w1[q], c2 = w2[q], c3 = w3[q];
  double a1z = c1 + w1[q - sz], a2z = c2 + w2[q - sz], a3z = c3 + w3[q - sz], a3x = c3 + w3[q - 1], a3y = c3 + w3[q - sy];
  for (int k = k0, b = 0; k < k1; k++, b ^= 1, q += sz) {
    const double n1 = w1[q + sz], n2 = w2[q + sz], n3 = w3[q + sz];
    const double a1y = c1 + w1[q - sy], a2x = c2 + w2[q - 1];
    double a1x = 0.0, a2y = 0.0, n1z = 0.0, n2z = 0.0, n3z = 0.0, n3x = 0.0, n3y = 0.0;
    if (!below) {
      a1x = c1 + w1[q - 1];
      n1z = n1 + c1;
      n3x = n3 + w3[q + sz - 1];
    }
    if (!beside) {
      a2y = c2 + w2[q - sy];
      n2z = n2 + c2;
      n3y = n3 + w3[q + sz - sy];
      double(&r)[5][kConvRows + 1][32] = rows[b];
      r[0][wy][lane] = a1y;
      r[1][wy][lane] = a2x;
      r[2][wy][lane] = a2y;
      r[3][wy][lane] = a2z;
      r[4][wy][lane] = a3y;
    } else if (lane < kConvRows) {
      double(&r)[5][kConvRows] = column[b];
      r[0][lane] = a1x;
      r[1][lane] = a1y;
      r[2][lane] = a1z;
      r[3][lane] = a2x;
      r[4][lane] = a3x;
    }
    __syncthreads();
    if (wy < kConvRows) {
      n3z = n3 + c3;
      double x[5] = {a1x, a1y, a1z, a2x, a3x};  // of the cell at x + 1
#pragma unroll
      for (int t = 0; t < 5; t++) {
        x[t] = __shfl_down_sync(0xffffffffu, x[t], 1);
        if (lane == 31) x[t] = column[b][t][wy];
      }
      const double y1y = rows[b][0][wy + 1][lane], y2x = rows[b][1][wy + 1][lane], y2y = rows[b][2][wy + 1][lane],
                   y2z = rows[b][3][wy + 1][lane], y3y = rows[b][4][wy + 1][lane];
      if (cell) {
        u[q] = fma(tauq, flux_balance(a1x, x[0], a1y, a2x, y1y, y2x, a1z, a3x, n1z, n3x), c1);
        v[q] = fma(tauq, flux_balance(a2y, y2y, a2x, a1y, x[3], x[1], a2z, a3y, n2z, n3y), c2);
        w[q] = fma(tauq, flux_balance(a3z, n3z, a3x, a1z, x[4], x[2], a3y, a2z, y3y, y2z), c3);
      }
    }
    c1 = n1;
    c2 = n2;
    c3 = n3;
    a1z = n1z;
    a2z = n2z;
    a3z = n3z;
    a3x = n3x;
    a3y = n3y;
  }
}

__global__ void k_copy3_interior(double *__restrict__ u, double *__restrict__ v, double *__restrict__ w,
                                 const double *__restrict__ w1, const double *__restrict__ w2,
                                 const double *__restrict__ w3, Dims d) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 2;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 2;
  const int k = blockIdx.z + 2;
  if (i > d.nx - 1 || j > d.ny - 1) return;
  const size_t q = d.ix(i, j, k);
  u[q] = w1[q];
  v[q] = w2[q];
  w[q] = w3[q];
}

__global__ void k_div(double *__restrict__ out, const double *__restrict__ u, const double *__restrict__ v,
                      const double *__restrict__ w, Dims d, double hi2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 2;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 2;
  const int k = blockIdx.z + 2;
  if (i > d.nx - 1 || j > d.ny - 1) return;
  const size_t q = d.ix(i, j, k);
  out[q] = (u[q + 1] - u[q] + v[q + d.sy()] - v[q] + w[q + d.sz()] - w[q]) * hi2;
}

__global__ void k_project(double *__restrict__ u, double *__restrict__ v, double *__restrict__ w,
                          const double *__restrict__ p, const double *__restrict__ a,
                          const double *__restrict__ b, const double *__restrict__ c, Dims d) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 2;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 2;
  const int k = blockIdx.z + 2;
  if (i > d.nx - 1 || j > d.ny - 1) return;
  const size_t q = d.ix(i, j, k);
  const size_t sy = d.sy(), sz = d.sz();
  const double pq = p[q];
  u[q] = u[q] - (pq - p[q - 1]) * a[q - 1];
  v[q] = v[q] - (pq - p[q - sy]) * b[q - sy];
  w[q] = w[q] - (pq - p[q - sz]) * c[q - sz];
}

// ---- bc_v (main.f:4064-4141) ---------------------------------------------------
//
// The ordered steps of bc_v and bc_w (x planes, y planes, z planes) in one
// launch each.  A y or z ghost is a function of interior cells that no step
// writes or of constants; where the x step copies a value that a later step
// overwrites (plane nx-1's ghosts and zero planes into plane nx), the thread
// that overwrites it copies it first.  Their fourth step, plane 2 from plane 1,
// comes with the outlet sums, because y and z ghosts are formed from plane 2
// before it.
__global__ void k_bcv(double *__restrict__ u, double *__restrict__ v, double *__restrict__ w, Dims d, double xvel2) {
  const int face = blockIdx.z;
  const int p = blockIdx.x * blockDim.x + threadIdx.x, q = blockIdx.y * blockDim.y + threadIdx.y;
  if (face == 0) {  // p -> j, q -> k, all of them for the inflow
    const int j = p + 1, k = q + 1;
    if (j > d.ny || k > d.nz) return;
    const int jj = j == 1 ? 2 : j;
    const double x = (jj * 1.0 - 1.5) / (d.ny * 1.0 - 1.5) - 1.0;
    const double val = xvel2 * (-(x * x) + 1.0);
    u[d.ix(1, j, k)] = j == 1 ? -val : val;
    const bool kin = k >= 2 && k <= d.nz - 1;
    // v: rows 1, 2 and ny and planes 1 and nz of plane nx-1 change below; w:
    // rows 1 and ny and planes 2 and nz
    if (j >= 3 && j <= d.ny - 1 && kin) v[d.ix(d.nx, j, k)] = v[d.ix(d.nx - 1, j, k)];
    if (j >= 2 && j <= d.ny - 1 && (k == 1 || (k >= 3 && k <= d.nz - 1)))
      w[d.ix(d.nx, j, k)] = w[d.ix(d.nx - 1, j, k)];
    if ((j == 1 || j == d.ny) && k == 1) w[d.ix(d.nx, j, k)] = w[d.ix(d.nx - 1, j, k)];
    return;
  }
  const int i = p + 2;
  if (i > d.nx - 1) return;
  const bool last = i == d.nx - 1;
  auto put = [&](double *f, int j, int k, double x) {
    const size_t n = d.ix(i, j, k);
    if (last) f[n + 1] = f[n];
    f[n] = x;
  };
  if (face == 1) {  // q -> k
    const int k = q + 2;
    if (k > d.nz - 1) return;
    u[d.ix(i, 1, k)] = -u[d.ix(i, 2, k)];
    u[d.ix(i, d.ny, k)] = u[d.ix(i, d.ny - 1, k)];
    put(v, 2, k, 0.0);
    put(v, 1, k, 0.0);
    put(v, d.ny, k, 0.0);
    if (k == 2) return;  // w's plane 2 is the z step's
    put(w, 1, k, -w[d.ix(i, 2, k)]);
    put(w, d.ny, k, w[d.ix(i, d.ny - 1, k)]);
    return;
  }
  const int j = q + 1;  // q -> j, ghost rows included
  if (j > d.ny) return;
  for (int s = 0; s < 2; s++) {
    const int k = s ? d.nz : 1, kin = s ? d.nz - 1 : 2;
    u[d.ix(i, j, k)] = j == 1 ? -u[d.ix(i, 2, kin)] : u[d.ix(i, j == d.ny ? d.ny - 1 : j, kin)];
    put(v, j, k, j <= 2 || j == d.ny ? 0.0 : v[d.ix(i, j, kin)]);
  }
  put(w, j, 2, 0.0);
  put(w, j, d.nz, 0.0);
}

// Sums of f0(1,j,k) and f1(nx-1,j,k) over interior j,k (deterministic order),
// and f1's planes 2 (and with `one` 1) = f0's plane 1 there.
__global__ void k_outlet_partial(double *__restrict__ partials, const double *f0, double *f1, bool one, Dims d) {
  const size_t n = (size_t)(d.ny - 2) * (d.nz - 2);
  double s0 = 0.0, s1 = 0.0;
  for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x) {
    const int j = (int)(t % (size_t)(d.ny - 2)) + 2, k = (int)(t / (size_t)(d.ny - 2)) + 2;
    const double in = f0[d.ix(1, j, k)];
    if (one) f1[d.ix(1, j, k)] = in;
    f1[d.ix(2, j, k)] = in;
    s0 += in;
    s1 += f1[d.ix(d.nx - 1, j, k)];
  }
  __shared__ double sh0[256], sh1[256];
  sh0[threadIdx.x] = s0;
  sh1[threadIdx.x] = s1;
  __syncthreads();
  for (int s = 128; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      sh0[threadIdx.x] += sh0[threadIdx.x + s];
      sh1[threadIdx.x] += sh1[threadIdx.x + s];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    partials[2 * blockIdx.x] = sh0[0];
    partials[2 * blockIdx.x + 1] = sh1[0];
  }
}

constexpr int kOutletBlocks = 64;

// Every block folds the partial sums itself, in their order: fetched by all
// threads at once, then added by one thread of two warps each (6.8 us; 9.6 us
// with each value fetched inside the sum).
__global__ void k_outlet_apply(double *__restrict__ x, const double *__restrict__ partials, Dims d) {
  __shared__ double sh[2 * kOutletBlocks], mean[2];
  const int t = threadIdx.y * 32 + threadIdx.x;
  if (t < 2 * kOutletBlocks) sh[t] = partials[t];
  __syncthreads();
  if (threadIdx.x == 0 && threadIdx.y < 2) {
    double s = 0.0;
    for (int b = 0; b < kOutletBlocks; b++) s += sh[2 * b + threadIdx.y];
    mean[threadIdx.y] = s / (d.ny - 2) / (d.nz - 2);
  }
  __syncthreads();
  const double vout = mean[0], vout2 = mean[1];
  const int j = blockIdx.x * blockDim.x + threadIdx.x + 2;
  const int k = blockIdx.y * blockDim.y + threadIdx.y + 2;
  if (j > d.ny - 1 || k > d.nz - 1) return;
  x[d.ix(d.nx, j, k)] = x[d.ix(d.nx - 1, j, k)] + vout - vout2;
}

// ---- bc_w (main.f:4143-4220) ---------------------------------------------------
__global__ void k_bcw(double *__restrict__ w1, double *__restrict__ w2, double *__restrict__ w3,
                      const double *__restrict__ v, const double *__restrict__ w, Dims d) {
  const int face = blockIdx.z;
  const int p = blockIdx.x * blockDim.x + threadIdx.x, q = blockIdx.y * blockDim.y + threadIdx.y;
  if (face == 0) {  // p -> j, q -> k
    const int j = p + 2, k = q + 2;
    if (j > d.ny - 1 || k > d.nz - 1) return;
    const double v1 = v[d.ix(1, j, k)], wv1 = w[d.ix(1, j, k)];
    w2[d.ix(1, j, k)] = v1;
    if (j > 2) w2[d.ix(2, j, k)] = v1;  // row 2 is the y step's
    w2[d.ix(d.nx, j, k)] = v[d.ix(d.nx, j, k)];
    w3[d.ix(1, j, k)] = wv1;
    if (k > 2) w3[d.ix(2, j, k)] = wv1;  // plane 2 is the z step's
    w3[d.ix(d.nx, j, k)] = w[d.ix(d.nx, j, k)];
    return;
  }
  const int i = p + 2;
  if (i > d.nx - 1) return;
  // w2 and w3 of an interior cell after the x step
  auto in2 = [&](int j, int k) { return i == 2 ? v[d.ix(1, j, k)] : w2[d.ix(i, j, k)]; };
  auto in3 = [&](int j, int k) { return i == 2 ? w[d.ix(1, j, k)] : w3[d.ix(i, j, k)]; };
  if (face == 1) {  // q -> k
    const int k = q + 2;
    if (k > d.nz - 1) return;
    w1[d.ix(i, 1, k)] = -w1[d.ix(i, 2, k)];
    w1[d.ix(i, d.ny, k)] = w1[d.ix(i, d.ny - 1, k)];
    w2[d.ix(i, 1, k)] = 0.0;
    w2[d.ix(i, 2, k)] = 0.0;
    w2[d.ix(i, d.ny, k)] = v[d.ix(i, d.ny, k)];
    if (k == 2) return;
    w3[d.ix(i, 1, k)] = -in3(2, k);
    w3[d.ix(i, d.ny, k)] = in3(d.ny - 1, k);
    return;
  }
  const int j = q + 1;  // q -> j, ghost rows included
  if (j > d.ny) return;
  for (int s = 0; s < 2; s++) {
    const int k = s ? d.nz : 1, kin = s ? d.nz - 1 : 2;
    w1[d.ix(i, j, k)] = j == 1 ? -w1[d.ix(i, 2, kin)] : w1[d.ix(i, j == d.ny ? d.ny - 1 : j, kin)];
    w2[d.ix(i, j, k)] = j <= 2 ? 0.0 : (j == d.ny ? v[d.ix(i, d.ny, kin)] : in2(j, kin));
  }
  const double wb = w[d.ix(i, j, 1)];
  w3[d.ix(i, j, 1)] = wb;
  w3[d.ix(i, j, 2)] = wb;
  w3[d.ix(i, j, d.nz)] = w[d.ix(i, j, d.nz)];
}

const dim3 kBlk(32, 4, 1);
const dim3 kFace(32, 8, 1);

inline dim3 fgrid(int p, int q) { return dim3((unsigned)((p + 31) / 32), (unsigned)((q + 7) / 8)); }

inline dim3 fgrid3(Dims d) {
  const int p = d.nx > d.ny ? d.nx : d.ny, q = d.ny > d.nz ? d.ny : d.nz;
  return dim3((unsigned)((p + 31) / 32), (unsigned)((q + 7) / 8), 3);
}

// Outlet flux balance shared by bc_v and bc_w: x(nx,j,k) = x(nx-1,j,k) + vout - vout2
// with vout the mean of u(1,j,k) and vout2 the mean of x(nx-1,j,k).
void outlet(double *x, const double *u, bool one, double *partials, Dims d, cudaStream_t st) {
  DSG_COUNT k_outlet_partial<<<kOutletBlocks, 256, 0, st>>>(partials, u, x, one, d);
  DSG_COUNT k_outlet_apply<<<fgrid(d.ny, d.nz), kFace, 0, st>>>(x, partials, d);
}

}  // namespace

cudaError_t bc_v(double *u, double *v, double *w, double *partials, Dims d, double xvel2, cudaStream_t st) {
  DSG_COUNT k_bcv<<<fgrid3(d), kFace, 0, st>>>(u, v, w, d, xvel2);
  outlet(u, u, false, partials, d, st);
  return cudaGetLastError();
}

cudaError_t bc_w(double *w1, double *w2, double *w3, const double *u, const double *v, const double *w,
                 double *partials, Dims d, cudaStream_t st) {
  DSG_COUNT k_bcw<<<fgrid3(d), kFace, 0, st>>>(w1, w2, w3, v, w, d);
  outlet(w1, u, true, partials, d, st);
  return cudaGetLastError();
}

// Interior planes k0 .. k1-1 (k1 = 0: all interior planes, 2 .. nz-1).
inline dim3 plane_grid(const Dims &d, int k0, int k1) {
  const dim3 g = interior_grid(d, kBlk);
  return dim3(g.x, g.y, (unsigned)((k1 ? k1 : d.nz) - k0));
}

cudaError_t stress(double *const S[6], const double *u, const double *v, const double *w, const double *cc,
                   Dims d, double r1, double r2, double r10, double r20, cudaStream_t st, int k0, int k1) {
  if ((k1 ? k1 : d.nz) <= k0) return cudaSuccess;
  const StressPure pure{{std::fma(r1, 0.0, r2), std::fma(r1, 1.0, r2)},
                        {std::fma(r10, 0.0, r20), std::fma(r10, 4.0, r20)}};
  DSG_COUNT k_stress<<<plane_grid(d, k0, k1), kBlk, 0, st>>>(S[0], S[1], S[2], S[3], S[4], S[5], u, v, w, cc, d, r1,
                                                              r2, r10, r20, pure, k0);
  return cudaGetLastError();
}

cudaError_t predictor(double *w1, double *w2, double *w3, const double *u, const double *v, const double *w,
                      const double *a, const double *b, const double *c, double *const S[6], Dims d,
                      double horgrav, double stdgrav, cudaStream_t st, int k0, int k1) {
  if ((k1 ? k1 : d.nz) <= k0) return cudaSuccess;
  DSG_COUNT k_predictor<<<plane_grid(d, k0, k1), kBlk, 0, st>>>(w1, w2, w3, u, v, w, a, b, c, S[0], S[1], S[2],
                                                                 S[3], S[4], S[5], d, horgrav, stdgrav, k0);
  return cudaGetLastError();
}

cudaError_t convective(double *u, double *v, double *w, const double *w1, const double *w2, const double *w3,
                       Dims d, double tauh, int convectype, cudaStream_t st) {
  if (convectype == 2) {
    // up to 16 planes per block (the first costs five sums more), fewer where
    // the GPU would get less than about four blocks per SM
    const unsigned bx = (d.nx - 2 + 31) / 32, by = (d.ny - 2 + kConvRows - 1) / kConvRows, nz = d.nz - 2;
    int planes = 16;
    while (planes > 2 && bx * by * ((nz + planes - 1) / planes) < 608) planes /= 2;
    DSG_COUNT k_convective<<<dim3(bx, by, (nz + planes - 1) / planes), kConvThreads, 0, st>>>(u, v, w, w1, w2, w3, d,
                                                                                             0.25 * tauh, planes);
  } else
    DSG_COUNT k_copy3_interior<<<interior_grid(d, kBlk), kBlk, 0, st>>>(u, v, w, w1, w2, w3, d);
  return cudaGetLastError();
}

cudaError_t divergence(double *out, const double *u, const double *v, const double *w, Dims d, double hi2,
                       cudaStream_t st) {
  DSG_COUNT k_div<<<interior_grid(d, kBlk), kBlk, 0, st>>>(out, u, v, w, d, hi2);
  return cudaGetLastError();
}

cudaError_t project(double *u, double *v, double *w, const double *p, const double *a, const double *b,
                    const double *c, Dims d, cudaStream_t st) {
  DSG_COUNT k_project<<<interior_grid(d, kBlk), kBlk, 0, st>>>(u, v, w, p, a, b, c, d);
  return cudaGetLastError();
}

}  // namespace dsg
