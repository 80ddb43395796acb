// vof.cu -- PLIC-VOF direction-split advection (VOFmethod/swp, main.f:795-1000),
// the plane/volume relations AL3D/FL3D (main.f:4562-4698), bc_flux
// (main.f:4496-4539), bc_c (main.f:4331-4396) and calcrho (main.f:2177-2190).
//
// One sweep = scan kernel (a bit per cell: not empty; the fluxes of the full
// cells, the list of the interface cells) -> flux kernel of the listed cells
// (left-out, stay, right-out volumes in the three scratch arrays the reference
// uses: z(iei), z(ires), z(irhs) of the finest level) -> update kernel
// (c = vof3(i-1)+vof2(i)+vof1(i+1) clipped to [0,1]) -> bc_c.  A cell whose own
// and two neighbours' bits are clear stays at zero, so the update and the flux
// arrays touch the liquid and its rim only: most of a sweep's traffic is the
// scan's one read of c.
#include "dsg_internal.cuh"

namespace dsg {
namespace {

// The lanes of a warp take different branches of AL3D and FL3D, and a warp
// executes every branch that one of its lanes takes, at 16 cycles of the SM's
// FP64 pipe per instruction.  The branches below therefore only pick operands;
// the divisions, square roots and acos/cos that several of them share stand
// behind the branches and are executed once (same operations per cell).

// AL3D: plane constant alpha of m1 x1 + m2 x2 + m3 x3 = alpha cutting volume cc
// from the unit cube (m1+m2+m3 = 1, 0 <= m1 <= m2 <= m3).  Scardovelli-Zaleski
// analytic inversion with five regimes; here its parts, as flux_cells deals
// them out.
struct Ordered {
  double m1, m2, m3, m12;
};
// Comparisons on the integer pipe, where one of the values is >= 0: then the bit
// patterns order like the values (an FP64 comparison costs as much as an FMA).
__device__ __forceinline__ bool less_bits(double a, double b) {
  return __double_as_longlong(a) < __double_as_longlong(b);
}
__device__ __forceinline__ double min_bits(double a, double b) { return less_bits(b, a) ? b : a; }
__device__ __forceinline__ double max_bits(double a, double b) { return less_bits(a, b) ? b : a; }
// x < 0, x == 0 (either sign), max(0, x), min(0, x); a NaN stays one
__device__ __forceinline__ bool negative(double x) {
  return __double_as_longlong(x) < 0 && (__double_as_longlong(x) << 1) != 0;
}
__device__ __forceinline__ bool zero(double x) { return (__double_as_longlong(x) << 1) == 0; }
__device__ __forceinline__ bool is_nan(double x) {
  return (__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFLL) > 0x7FF0000000000000LL;
}
__device__ __forceinline__ double max0(double x) { return positive_bits(x) || is_nan(x) ? x : 0.0; }
__device__ __forceinline__ double min0(double x) { return negative(x) || is_nan(x) ? x : 0.0; }
__device__ __forceinline__ Ordered ordered(double b1, double b2, double b3) {
  double m1 = min_bits(b1, b2), m3 = max_bits(b1, b2), m2 = b3, tmp;
  if (less_bits(m2, m1)) {
    tmp = m1; m1 = m2; m2 = tmp;
  } else if (less_bits(m3, m2)) {
    tmp = m3; m3 = m2; m2 = tmp;
  }
  return {m1, m2, m3, m1 + m2};
}
__device__ __forceinline__ double al3d_pr(const Ordered &o) { return max_bits(6.0 * o.m1 * o.m2 * o.m3, 1.0e-50); }
// V1 = m1^3 / pr; V2 = V1 + 0.5 (m2 - m1) / m3; V3:
__device__ __forceinline__ double al3d_v3(const Ordered &o) {
  const double m1 = o.m1, m2 = o.m2, m3 = o.m3, m12 = o.m12;
  const bool five = less_bits(m3, m12);  // regimes 3 and 5 up to m3, else 3 and 4 up to m12
  double num = 0.5 * m12, den = m3;
  if (five) {
    num = m3 * m3 * (3.0 * m12 - m3) + m1 * m1 * (m1 - 3.0 * m3) + m2 * m2 * (m2 - 3.0 * m3);
    den = al3d_pr(o);
  }
  return num / den;
}
__device__ __forceinline__ double al3d_cubic(const Ordered &o, double ch, bool below_v3) {
  const double m1 = o.m1, m2 = o.m2, m3 = o.m3, m12 = o.m12;
  double p = 2.0 * m1 * m2, q = 1.5 * m1 * m2 * (m12 - 2.0 * m3 * ch), add = m12;
  if (!below_v3) {
    p = m1 * (m2 + m3) + m2 * m3 - 0.25;
    q = 1.5 * m1 * m2 * m3 * (0.5 - ch);
    add = 0.5;
  }
  const double p12 = sqrt(p);
  double cst = q / (p * p12);
  if (cst > 1.0) cst = 1.0;
  if (cst < -1.0) cst = -1.0;
  const double cs = cos(acos(cst) / 3.0);
  return p12 * (sqrt(3.0 * (1.0 - cs * cs)) - cs) + add;
}

// FL3D: volume of the part of [r0, r0+dr0] x [0,1]^2 below the plane.
__device__ double fl3d(double m1, double m2, double m3, double alpha, double r0, double dr0) {
  double al = alpha - m1 * r0;
  al = al + max0(-m1 * dr0) + max0(-m2) + max0(-m3);
  double tmp = fabs(m1) * dr0 + fabs(m2) + fabs(m3);
  const double n1 = fabs(m1) / tmp, n2 = fabs(m2) / tmp, n3 = fabs(m3) / tmp;
  al = al / tmp;
  al = is_nan(al) ? al : max0(min_bits(1.0, al));
  const double al0 = min_bits(al, 1.0 - al);
  double b1 = min_bits(n1 * dr0, n2), b3 = max_bits(n1 * dr0, n2), b2 = n3;
  if (less_bits(b2, b1)) {
    tmp = b1; b1 = b2; b2 = tmp;
  } else if (less_bits(b3, b2)) {
    tmp = b3; b3 = b2; b2 = tmp;
  }
  const double b12 = b1 + b2;
  const double bm = min_bits(b12, b3);
  const double pr = max_bits(6.0 * b1 * b2 * b3, 1.0e-50);
  double num, den = pr;
  const bool two = !less_bits(al0, b1) && less_bits(al0, b2);  // the regime with a second term, b1^3 / pr
  if (less_bits(al0, b1)) {
    num = al0 * al0 * al0;
  } else if (less_bits(al0, b2)) {
    num = 0.5 * al0 * (al0 - b1);
    den = b2 * b3;
  } else if (less_bits(al0, bm)) {
    num = al0 * al0 * (3.0 * b12 - al0) + b1 * b1 * (b1 - 3.0 * al0) + b2 * b2 * (b2 - 3.0 * al0);
  } else if (same_bits(bm, b12)) {
    num = al0 - 0.5 * bm;
    den = b3;
  } else {
    num = al0 * al0 * (3.0 - 2.0 * al0) + b1 * b1 * (b1 - 3.0 * al0) + b2 * b2 * (b2 - 3.0 * al0) +
          b3 * b3 * (b3 - 3.0 * al0);
  }
  tmp = num / den;
  if (two) tmp = tmp + b1 * b1 * b1 / pr;
  return (less_bits(0.5, al) ? 1.0 - tmp : tmp) * dr0;
}

// Youngs normal from the 27-point stencil, component A (swp, main.f:896-925).
template <int A>
__device__ __forceinline__ double youngs(size_t q, const double *__restrict__ cc, long sy, long sz) {
  const long sa = A == 1 ? 1 : (A == 2 ? sy : sz), sb = A == 1 ? sy : 1, sc = A == 3 ? sy : sz;
  // the sums' order of the reference: the corners' two other axes, ...
#define C(a, b, c) cc[(long)q + (long)(a) * sa + (long)(b) * sb + (long)(c) * sc]
  double mm[2];
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int s = 2 * h - 1;
    mm[h] = C(s, -1, -1) + C(s, -1, 1) + C(s, 1, -1) + C(s, 1, 1) +
            2.0 * (C(s, -1, 0) + C(s, 1, 0) + C(s, 0, -1) + C(s, 0, 1)) + 4.0 * C(s, 0, 0);
  }
#undef C
  return mm[0] - mm[1];
}

// Fluxes of interface cells (0 < c < 1): Youngs normal, AL3D plane constant,
// Lagrangian stretch along D and the FL3D cut volumes (swp, main.f:896-995).
//
// A warp scheduler starts one FP64 instruction every 64 cycles, and a cell is
// some 900 of them in a row: 30 us, whatever the grid.  So a block's four warps
// (one per scheduler) take the same 32 cells and deal out what is independent:
// the components of the normal and their divisions, AL3D's three volumes and
// its regimes, FL3D's calls.  64^3: 30 -> 16.5 us per sweep,
// 128^3 32 -> 20; at 256^3, with many cells per scheduler, 39 and 41.
template <int D>
__device__ __forceinline__ void flux_cells(size_t q, bool in, const double *__restrict__ us,
                                           const double *__restrict__ cc, double *__restrict__ vof1,
                                           double *__restrict__ vof2, double *__restrict__ vof3, Dims d, double tauh) {
  __shared__ double part[9][32];  // normal, its quotients, AL3D's parts
  const int lane = threadIdx.x & 31, role = threadIdx.x >> 5;
  const long sy = (long)d.sy(), sz = (long)d.sz();
  const long sd = D == 1 ? 1 : (D == 2 ? sy : sz);
  const double a1 = us[q] * tauh, a2 = us[q + sd] * tauh, c0 = cc[q];
  if (role == 0) part[0][lane] = youngs<1>(q, cc, sy, sz);
  if (role == 1) part[1][lane] = youngs<2>(q, cc, sy, sz);
  if (role == 2) part[2][lane] = youngs<3>(q, cc, sy, sz);
  __syncthreads();
  double mx = part[0][lane], my = part[1][lane], mz = part[2][lane];
  const bool flat = zero(mx) && zero(my) && zero(mz), store = in && !flat;
  const bool nx = negative(mx), ny = negative(my), nz = negative(mz);
  if (nx) mx = -mx;
  if (ny) my = -my;
  if (nz) mz = -mz;
  if (role < 3) {
    const double mm2 = mx + my + mz + (double)1.e-30f;  // default-REAL literal of main.f:927
    part[3 + role][lane] = (role == 0 ? mx : role == 1 ? my : mz) / mm2;
  } else if (in && flat) {
    // Deviation from swp: a symmetric neighbourhood gives an all-zero Youngs
    // normal, for which FL3D divides 0/0.  Such a cell is advected as a
    // uniformly filled one (donor-cell fluxes scaled by c).
    vof1[q] = c0 * dmax1(-a1, 0.0);
    vof2[q] = c0 * (1.0 - dmax1(a1, 0.0) + dmin1(a2, 0.0));
    vof3[q] = c0 * dmax1(a2, 0.0);
  }
  __syncthreads();
  mx = part[3][lane];
  my = part[4][lane];
  mz = part[5][lane];
  const Ordered o = ordered(mx, my, mz);
  const double ch = min_bits(c0, 1.0 - c0);
  if (nx) mx = -mx;
  if (ny) my = -my;
  if (nz) mz = -mz;
  // The sweep direction's normal component goes first in FL3D.
  double n1, n2, n3;
  if (D == 1) { n1 = mx; n2 = my; n3 = mz; }
  else if (D == 2) { n1 = my; n2 = mz; n3 = mx; }
  else { n1 = mz; n2 = mx; n3 = my; }
  if (role == 0) part[6][lane] = o.m1 * o.m1 * o.m1 / al3d_pr(o);
  if (role == 1) part[7][lane] = 0.5 * (o.m2 - o.m1) / o.m3;
  if (role == 2) part[8][lane] = al3d_v3(o);
  if (role == 3) part[0][lane] = n1 / (1.0 - a1 + a2);
  __syncthreads();
  const double V1 = part[6][lane], V2 = V1 + part[7][lane], V3 = part[8][lane];
  n1 = part[0][lane];
  const bool one = less_bits(ch, V1), two = !one && less_bits(ch, V2), third = less_bits(ch, V3);
  const bool four = !one && !two && !third && !less_bits(o.m3, o.m12);
  if (role == 0 && one) part[1][lane] = pow(al3d_pr(o) * ch, 1.0 / 3.0);
  if (role == 1 && two) part[1][lane] = 0.5 * (o.m1 + sqrt(o.m1 * o.m1 + 8.0 * o.m2 * o.m3 * (ch - V1)));
  if (role == 1 && four) part[1][lane] = o.m3 * ch + 0.5 * o.m12;
  if (role == 2 && !(one || two || four)) part[1][lane] = al3d_cubic(o, ch, third);
  __syncthreads();
  if (role < 3) {
    double alpha = part[1][lane];
    if (less_bits(0.5, c0)) alpha = 1.0 - alpha;
    alpha = alpha + min0(mx) + min0(my) + min0(mz);
    alpha = alpha + n1 * a1;
    // The outflow at either end: in most cells there is one at most, so lanes
    // with an outflow to the left and lanes with one to the right share a call.
    const bool left = negative(a1), right = positive_bits(a2);
    if (role == 0 && store) {
      const double mm1 = max0(a1);
      vof2[q] = fl3d(n1, n2, n3, alpha, mm1, 1.0 - mm1 + min0(a2));
    }
    if (role == 1 && store) {
      double f = 0.0;
      if (left || right) f = fl3d(n1, n2, n3, alpha, left ? a1 : 1.0, left ? -a1 : a2);
      vof1[q] = left ? f : 0.0;
      if (!(left && right)) vof3[q] = left ? 0.0 : f;
    }
    if (role == 2 && store && left && right) vof3[q] = fl3d(n1, n2, n3, alpha, 1.0, a2);
  }
  __syncthreads();
}

// Bits of the cells with c != +0, one word per 32 cells along x: word w of row
// (j, k) at (k - 2) * (ny - 2) + (j - 2) rows of wpr = ceil((nx - 2) / 32).
__host__ __device__ __forceinline__ int words_per_row(Dims d) { return (d.nx - 2 + 31) / 32; }

constexpr int kScanRows = 4;  // rows a warp scans, all loaded before the first is used

// Sweep, pass 1: the bits, the fluxes of full cells (the reference's c == 1
// branch; zero for values that are neither positive nor +0) and the list of
// interface cells (one atomic per warp), so that the PLIC geometry runs on
// full warps instead of one busy lane per warp.  Also bc_flux's zeros beyond the
// upper face along D: vof1 is EI, whose ghosts nothing else in a step writes.
template <int D>
__global__ void k_swp_scan(const double *__restrict__ us, const double *__restrict__ cc, double *__restrict__ vof1,
                           double *__restrict__ vof2, double *__restrict__ vof3, Dims d, double tauh,
                           unsigned *__restrict__ bits, unsigned *__restrict__ list, unsigned *__restrict__ count) {
  const int i = blockIdx.x * 32 + threadIdx.x + 2, k = blockIdx.z + 2;
  const int j0 = (blockIdx.y * blockDim.y + threadIdx.y) * kScanRows + 2;
  const unsigned lane = threadIdx.x;
  double c[kScanRows];
#pragma unroll
  for (int r = 0; r < kScanRows; r++)
    c[r] = i <= d.nx - 1 && j0 + r <= d.ny - 1 ? cc[d.ix(i, j0 + r, k)] : 0.0;
  unsigned mask[kScanRows], total = 0, some = 0;
#pragma unroll
  for (int r = 0; r < kScanRows; r++) {
    const unsigned any = __ballot_sync(0xffffffffu, !is_zero_bits(c[r]));
    mask[r] = __ballot_sync(0xffffffffu, positive_bits(c[r]) && !is_one_bits(c[r]));
    total += __popc(mask[r]);
    some |= any;
    if (lane == 0 && j0 + r <= d.ny - 1)
      bits[((size_t)(k - 2) * (d.ny - 2) + (j0 + r - 2)) * words_per_row(d) + blockIdx.x] = any;
    if (i <= d.nx - 1 && j0 + r <= d.ny - 1 &&
        (D == 1 ? i == d.nx - 1 : (D == 2 ? j0 + r == d.ny - 1 : k == d.nz - 1)))
      vof1[d.ix(i, j0 + r, k) + (D == 1 ? 1 : (D == 2 ? d.sy() : d.sz()))] = 0.0;
  }
  if (!some) return;
  unsigned base = 0;
  if (total) {
    if (lane == 0) base = atomicAdd(count, total);
    base = __shfl_sync(0xffffffffu, base, 0);
  }
#pragma unroll
  for (int r = 0; r < kScanRows; r++) {
    const size_t q = d.ix(i, j0 + r, k);
    const bool iface = mask[r] >> lane & 1u;
    if (iface) list[base + __popc(mask[r] & ((1u << lane) - 1u))] = (unsigned)q;
    base += __popc(mask[r]);
    if (iface || is_zero_bits(c[r])) continue;  // lanes past the grid's end hold zeros
    double f1 = 0.0, f2 = 0.0, f3 = 0.0;
    if (is_one_bits(c[r])) {
      const long sd = D == 1 ? 1 : (D == 2 ? (long)d.sy() : (long)d.sz());
      const double a1 = us[q] * tauh, a2 = us[q + sd] * tauh;
      f1 = dmax1(-a1, 0.0);
      f2 = 1.0 - dmax1(a1, 0.0) + dmin1(a2, 0.0);
      f3 = dmax1(a2, 0.0);
    }
    vof1[q] = f1;
    vof2[q] = f2;
    vof3[q] = f3;
  }
}

// Pass 2: the listed interface cells, 32 per block at a time.
template <int D>
__global__ void k_swp_flux_iface(const unsigned *__restrict__ list, const unsigned *__restrict__ count,
                                 const double *__restrict__ us, const double *__restrict__ cc,
                                 double *__restrict__ vof1, double *__restrict__ vof2, double *__restrict__ vof3,
                                 Dims d, double tauh) {
  const unsigned n = *count, lane = threadIdx.x & 31;
  for (unsigned t = 32 * blockIdx.x; t < n; t += 32 * gridDim.x)
    flux_cells<D>(list[min(t + lane, n - 1)], t + lane < n, us, cc, vof1, vof2, vof3, d, tauh);
}

// Pass 3: c = vof3(-1) + vof2 + vof1(+1) along D clipped to [0,1], a missing
// bit's fluxes being zero, and so those that enter through the domain's faces
// (bc_flux, main.f:4496-4539).  A warp takes wpw words of the bits,
// and its 32 lanes go together through those that have something to do.  The
// list's length is reset for the next sweep.
template <int D>
__global__ void k_swp_update(double *__restrict__ cc, const double *__restrict__ vof1,
                             const double *__restrict__ vof2, const double *__restrict__ vof3,
                             const unsigned *__restrict__ bits, unsigned *__restrict__ count, Dims d, int wpw) {
  const int wpr = words_per_row(d), ny2 = d.ny - 2;
  const long long rows = (long long)ny2 * (d.nz - 2), words = rows * wpr;
  const unsigned lane = threadIdx.x & 31;
  const long long w0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / 32 * wpw, w = w0 + lane;
  if (w == 0) *count = 0u;
  unsigned own = 0, lo = 0, hi = 0;  // bits of a cell, its lower and its upper neighbour
  if ((int)lane < wpw && w < words) {
    own = bits[w];
    const long long row = w / wpr;
    const int x = (int)(w - row * wpr), j = (int)(row % ny2);
    if (D == 1) {
      lo = own << 1 | (x > 0 ? bits[w - 1] >> 31 : 0u);
      hi = own >> 1 | (x + 1 < wpr ? bits[w + 1] << 31 : 0u);
    } else if (D == 2) {
      lo = j > 0 ? bits[w - wpr] : 0u;
      hi = j + 1 < ny2 ? bits[w + wpr] : 0u;
    } else {
      lo = row >= ny2 ? bits[w - (long long)ny2 * wpr] : 0u;
      hi = row + ny2 < rows ? bits[w + (long long)ny2 * wpr] : 0u;
    }
  }
  const size_t sd = D == 1 ? 1 : (D == 2 ? d.sy() : d.sz());
  unsigned busy = __ballot_sync(0xffffffffu, (own | lo | hi) != 0u);
  while (busy) {
    const int b = __ffs(busy) - 1;
    busy &= busy - 1;
    const unsigned o = __shfl_sync(0xffffffffu, own, b), l = __shfl_sync(0xffffffffu, lo, b),
                   h = __shfl_sync(0xffffffffu, hi, b);
    const long long row = (w0 + b) / wpr;
    const int i = (int)(w0 + b - row * wpr) * 32 + (int)lane + 2;
    if (i > d.nx - 1 || !((o | l | h) >> lane & 1u)) continue;
    const size_t q = d.ix(i, (int)(row % ny2) + 2, (int)(row / ny2) + 2);
    const double x = (l >> lane & 1u ? vof3[q - sd] : 0.0) + (o >> lane & 1u ? vof2[q] : 0.0) +
                     (h >> lane & 1u ? vof1[q + sd] : 0.0);
    // dmax1(0, dmin1(1, x)) on the bit patterns (same result for every non-NaN x)
    const double y = __double_as_longlong(x) >= 0x3FF0000000000000LL ? 1.0 : x;
    cc[q] = __double_as_longlong(y) <= 0LL ? 0.0 : y;
  }
}

// The parts of the flux arrays that a sweep neither writes nor reads, for callers
// that see the arrays: all of the interior (the sweep then writes the cells that
// are not empty) and bc_flux's zeros beyond the lower face (main.f:4496-4539).
template <int D>
__global__ void k_zero_fluxes(double *__restrict__ vof1, double *__restrict__ vof2, double *__restrict__ vof3, Dims d) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 2;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 2;
  const int k = blockIdx.z + 2;
  if (i > d.nx - 1 || j > d.ny - 1) return;
  const size_t q = d.ix(i, j, k), sd = D == 1 ? 1 : (D == 2 ? d.sy() : d.sz());
  vof1[q] = vof2[q] = vof3[q] = 0.0;
  if ((D == 1 ? i : (D == 2 ? j : k)) == 2) vof3[q - sd] = 0.0;
}

// bc_c (main.f:4340-4395 without the dead filter block).  Its three ordered
// steps -- x: plane 2 = plane 1, plane nx = plane nx-1; y: ghosts of i in
// 2..nx-1 (the lower one clipped); z: likewise over all j -- in one launch: a
// y or z ghost is a function of cells that no step writes (plane 1 in place of
// plane 2).  The x step copies the old y and z ghosts of plane nx-1 to plane
// nx; the threads that overwrite them do that first.
__global__ void k_bc_c(double *__restrict__ cc, Dims d) {
  const int face = blockIdx.z;
  const int p = blockIdx.x * blockDim.x + threadIdx.x, q = blockIdx.y * blockDim.y + threadIdx.y;
  auto src = [&](int i, int j, int k) { return cc[d.ix(i == 2 ? 1 : i, j, k)]; };
  if (face == 0) {  // p -> j, q -> k
    const int j = p + 2, k = q + 2;
    if (j > d.ny - 1 || k > d.nz - 1) return;
    cc[d.ix(2, j, k)] = cc[d.ix(1, j, k)];
    cc[d.ix(d.nx, j, k)] = cc[d.ix(d.nx - 1, j, k)];
    return;
  }
  const int i = p + 2;
  if (i > d.nx - 1) return;
  const bool last = i == d.nx - 1;
  if (face == 1) {  // q -> k
    const int k = q + 2;
    if (k > d.nz - 1) return;
    if (last) {
      cc[d.ix(d.nx, 1, k)] = cc[d.ix(i, 1, k)];
      cc[d.ix(d.nx, d.ny, k)] = cc[d.ix(i, d.ny, k)];
    }
    double x = src(i, 2, k);
    if (x > 1.0) x = 1.0;
    if (x < 0.0) x = 0.0;
    cc[d.ix(i, 1, k)] = x;
    cc[d.ix(i, d.ny, k)] = src(i, d.ny - 1, k);
    return;
  }
  const int j = q + 1;  // q -> j, ghost rows included
  if (j > d.ny) return;
  for (int s = 0; s < 2; s++) {
    const int k = s ? d.nz : 1, kin = s ? d.nz - 1 : 2;
    if (last) cc[d.ix(d.nx, j, k)] = cc[d.ix(i, j, k)];
    double x;
    if (j == 1) {
      x = src(i, 2, kin);
      if (x > 1.0) x = 1.0;
      if (x < 0.0) x = 0.0;
    } else {
      x = src(i, j == d.ny ? d.ny - 1 : j, kin);
    }
    cc[d.ix(i, j, k)] = x;
  }
}

// calcrho (main.f:2177-2190); for c = 0 and c = 1 the same operations are
// evaluated once on the host (rho_l = rho2 + 1*(rho1-rho2), ...).
__global__ void k_calcrho(double *__restrict__ rhon, double *__restrict__ mun, const double *__restrict__ cc,
                          size_t n, double rho1, double rho2, double mu1, double mu2, double rho_g, double rho_l,
                          double mu_g, double mu_l) {
  for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (size_t)gridDim.x * blockDim.x) {
    const double c = cc[q];
    if (is_zero_bits(c)) {
      rhon[q] = rho_g;
      mun[q] = mu_g;
    } else if (is_one_bits(c)) {
      rhon[q] = rho_l;
      mun[q] = mu_l;
    } else {
      rhon[q] = rho2 + c * (rho1 - rho2);
      mun[q] = mu2 + c * (mu1 - mu2);
    }
  }
}

const dim3 kBlk(32, 4, 1);

template <int D>
void sweep(const double *us, double *cc, double *v1, double *v2, double *v3, Dims d, double tauh, unsigned *list,
           unsigned *count, cudaStream_t st, bool whole) {
  if (whole) DSG_COUNT k_zero_fluxes<D><<<interior_grid(d, kBlk), kBlk, 0, st>>>(v1, v2, v3, d);
  unsigned *bits = list + (size_t)(d.nx - 2) * (d.ny - 2) * (d.nz - 2);
  const int wpr = words_per_row(d), rows = 4 * kScanRows;
  DSG_COUNT k_swp_scan<D><<<dim3((unsigned)wpr, (unsigned)((d.ny - 2 + rows - 1) / rows), (unsigned)(d.nz - 2)), kBlk,
                            0, st>>>(us, cc, v1, v2, v3, d, tauh, bits, list, count);
  // 32 cells and four warps per block: a short list goes to as many SMs as it
  // has sets of 32 cells; a block beyond its end has nothing to do.
  DSG_COUNT k_swp_flux_iface<D><<<kRedBlocks, 128, 0, st>>>(list, count, us, cc, v1, v2, v3, d, tauh);
  const size_t words = (size_t)wpr * (d.ny - 2) * (d.nz - 2);
  // Words per warp: on small grids few, because a warp goes through its busy
  // words one after the other (64^3: 4 us with 4, 12 us with 32); on large ones
  // more, because most warps find nothing to do (256^3: 19 us with 4, 13 with 32).
  const int wpw = words < ((size_t)1 << 17) ? 4 : 16;
  DSG_COUNT k_swp_update<D><<<(unsigned)((words + 4 * wpw - 1) / (4 * wpw)), 128, 0, st>>>(cc, v1, v2, v3, bits, count,
                                                                                          d, wpw);
}

}  // namespace

cudaError_t bc_c(double *cc, Dims d, cudaStream_t st) {
  const int p = d.nx > d.ny ? d.nx : d.ny, q = d.ny > d.nz ? d.ny : d.nz;
  DSG_COUNT k_bc_c<<<dim3((p + 31) / 32, (q + 7) / 8, 3), dim3(32, 8), 0, st>>>(cc, d);
  return cudaGetLastError();
}

cudaError_t swp(const double *us, double *cc, double *vof1, double *vof2, double *vof3, int dir, Dims d,
                double tauh, unsigned *list, unsigned *count, cudaStream_t st, bool whole) {
  if (dir == 1) sweep<1>(us, cc, vof1, vof2, vof3, d, tauh, list, count, st, whole);
  else if (dir == 2) sweep<2>(us, cc, vof1, vof2, vof3, d, tauh, list, count, st, whole);
  else sweep<3>(us, cc, vof1, vof2, vof3, d, tauh, list, count, st, whole);
  return bc_c(cc, d, st);
}

cudaError_t calcrho(double *rhon, double *mun, const double *cc, Dims d, double rho1, double rho2,
                    double mu1, double mu2, cudaStream_t st) {
  const size_t n = d.count();
  const int blocks = (int)((n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096);
  const double z = 0.0, one = 1.0;
  const double rho_g = rho2 + z * (rho1 - rho2), rho_l = rho2 + one * (rho1 - rho2);
  const double mu_g = mu2 + z * (mu1 - mu2), mu_l = mu2 + one * (mu1 - mu2);
  DSG_COUNT k_calcrho<<<blocks, 256, 0, st>>>(rhon, mun, cc, n, rho1, rho2, mu1, mu2, rho_g, rho_l, mu_g, mu_l);
  return cudaGetLastError();
}

}  // namespace dsg
