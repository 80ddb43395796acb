// csf.cu -- CSF surface-tension force (csf, main.f:2363-2481): 27-point filter
// of the volume fraction, face-normal curvature kappa = -div(n), and the face
// forces S11/S22/S33 = sigh * (c~_i - c~_{i-1}) * kappa_i, plus bc_tensor
// (main.f:4222-4296).
#include "dsg_internal.cuh"

namespace dsg {
namespace {

// Curvature and face forces at interior cells: six face-normal magnitudes with
// transverse 4-point means (+1e-50 inside the root), kappa =
// -(d1x-d2x+d1y-d2y+d1z-d2z); S = sigh * (difference of f) * kappa.  The
// curvature is used by its own cell only, so it stays in a register.  Bound by
// memory and, around the interface, the FP64 pipe: 256^3 367 us as two kernels,
// each warp doing its own interface cells, 124 us now
// (79 us of memory traffic); 128^3 61 and 26.
template <int P>
__global__ void __launch_bounds__(kBandThreads) k_csf(double *__restrict__ s11, double *__restrict__ s22,
                                                      double *__restrict__ s33, const double *__restrict__ f, Dims d,
                                                      double sigh) {
  const long sy = (long)d.sy(), sz = (long)d.sz();
  auto force = [&](size_t q, double kq) {
    const double fq = f[q], fx = f[q - 1], fy = f[q - sy], fz = f[q - sz];
    if (same_bits(fx, fq) && same_bits(fy, fq) && same_bits(fz, fq)) {
      // every difference is +0, so each force is (sigh * +0) * kappa, a zero
      // whose sign is sign(sigh) xor sign(kappa) (kappa is finite), formed on
      // the integer pipe
      const double z = __longlong_as_double((__double_as_longlong(sigh) ^ __double_as_longlong(kq)) &
                                            (long long)0x8000000000000000ULL);
      s11[q] = z;
      s22[q] = z;
      s33[q] = z;
      return;
    }
    s11[q] = sigh * (fq - fx) * kq;
    s22[q] = sigh * (fq - fy) * kq;
    s33[q] = sigh * (fq - fz) * kq;
  };
#define F(di, dj, dk) f[(long)q + (long)(di) + (long)(dj) * sy + (long)(dk) * sz]
  const Flat<P> flat(f, d);
  bulk_then_cells<P>(d, [&](int i, int j, int k, int p) {
    // Uniform 19-point neighbourhood (bulk liquid or gas): every difference is
    // +0, every d is 0/sqrt(1e-50) = +0 and kappa = -(+0) = -0 exactly.
    if (!flat.uniform(p, false)) return false;
    const double z = __longlong_as_double((__double_as_longlong(sigh) & (long long)0x8000000000000000ULL) ^
                                          (long long)0x8000000000000000ULL);  // (sigh * +0) * -0
    const size_t q = d.ix(i, j, k);
    s11[q] = s22[q] = s33[q] = z;
    return true;
  }, [&](int i, int j, int k) {
    const size_t q = d.ix(i, j, k);
    // d = difference / |normal| as difference * rsqrt(|normal|^2): one FP64
    // reciprocal square root in place of a square root and a division on
    // GB300's narrow FP64 pipe (results within a few ulps of the quotient)
    double t0, t1, t2;
    t0 = F(1, 0, 0) - F(0, 0, 0);
    t1 = F(0, 1, 0) - F(0, -1, 0) + F(1, 1, 0) - F(1, -1, 0);
    t2 = F(0, 0, 1) - F(0, 0, -1) + F(1, 0, 1) - F(1, 0, -1);
    const double d1x = t0 * rsqrt(t0 * t0 + 0.0625 * (t1 * t1) + 0.0625 * (t2 * t2) + 1.e-50);
    t0 = F(0, 0, 0) - F(-1, 0, 0);
    t1 = F(0, 1, 0) - F(0, -1, 0) + F(-1, 1, 0) - F(-1, -1, 0);
    t2 = F(0, 0, 1) - F(0, 0, -1) + F(-1, 0, 1) - F(-1, 0, -1);
    const double d2x = t0 * rsqrt(t0 * t0 + 0.0625 * (t1 * t1) + 0.0625 * (t2 * t2) + 1.e-50);
    t0 = F(0, 1, 0) - F(0, 0, 0);
    t1 = F(1, 0, 0) - F(-1, 0, 0) + F(1, 1, 0) - F(-1, 1, 0);
    t2 = F(0, 0, 1) - F(0, 0, -1) + F(0, 1, 1) - F(0, 1, -1);
    const double d1y = t0 * rsqrt(t0 * t0 + 0.0625 * (t1 * t1) + 0.0625 * (t2 * t2) + 1.e-50);
    t0 = F(0, 0, 0) - F(0, -1, 0);
    t1 = F(1, 0, 0) - F(-1, 0, 0) + F(1, -1, 0) - F(-1, -1, 0);
    t2 = F(0, 0, 1) - F(0, 0, -1) + F(0, -1, 1) - F(0, -1, -1);
    const double d2y = t0 * rsqrt(t0 * t0 + 0.0625 * (t1 * t1) + 0.0625 * (t2 * t2) + 1.e-50);
    t0 = F(0, 0, 1) - F(0, 0, 0);
    t1 = F(1, 0, 0) - F(-1, 0, 0) + F(1, 0, 1) - F(-1, 0, 1);
    t2 = F(0, 1, 0) - F(0, -1, 0) + F(0, 1, 1) - F(0, -1, 1);
    const double d1z = t0 * rsqrt(t0 * t0 + 0.0625 * (t1 * t1) + 0.0625 * (t2 * t2) + 1.e-50);
    t0 = F(0, 0, 0) - F(0, 0, -1);
    t1 = F(1, 0, 0) - F(-1, 0, 0) + F(1, 0, -1) - F(-1, 0, -1);
    t2 = F(0, 1, 0) - F(0, -1, 0) + F(0, 1, -1) - F(0, -1, -1);
    const double d2z = t0 * rsqrt(t0 * t0 + 0.0625 * (t1 * t1) + 0.0625 * (t2 * t2) + 1.e-50);
    force(q, -(d1x - d2x + d1y - d2y + d1z - d2z));
  });
#undef F
}

// bc_tensor, its three ordered steps in one launch: every cell two steps write
// gets the same constant from both, and S22's ghosts come from interior cells.
// It splits into ranges of planes (the x and y faces of planes kx0 .. kx1-1,
// the z planes 1, 2 and nz where they lie in kz0 .. kz1-1).  ALL = false: the
// constant faces of S12, S13, S23 alone.
template <bool ALL>
__global__ void k_bct(double *__restrict__ s11, double *__restrict__ s22, double *__restrict__ s33,
                      double *__restrict__ s12, double *__restrict__ s13, double *__restrict__ s23, Dims d, int kx0,
                      int kx1, int kz0, int kz1) {
  const int face = blockIdx.z;
  const int p = blockIdx.x * blockDim.x + threadIdx.x, q = blockIdx.y * blockDim.y + threadIdx.y;
  if (face == 0) {  // p -> j, q -> k
    const int j = p + 2, k = q + kx0;
    if (j > d.ny - 1 || k >= kx1) return;
    if (ALL) s11[d.ix(1, j, k)] = 0.0;
    s12[d.ix(d.nx, j, k)] = 0.0;
    s13[d.ix(d.nx, j, k)] = 0.0;
  } else if (face == 1) {  // p -> i, q -> k
    const int i = p + 1, k = q + kx0;
    if (i > d.nx || k >= kx1) return;
    if (ALL) s22[d.ix(i, 1, k)] = s22[d.ix(i, 2, k)];
    s12[d.ix(i, d.ny, k)] = 0.0;
    s23[d.ix(i, d.ny, k)] = 0.0;
  } else {  // p -> i, q -> j
    const int i = p + 1, j = q + 1;
    if (i > d.nx || j > d.ny) return;
    if (ALL && kz0 <= 1 && 1 < kz1) s33[d.ix(i, j, 1)] = 0.0;
    if (kz0 <= 2 && 2 < kz1) s13[d.ix(i, j, 2)] = 0.0;
    if (kz0 <= d.nz && d.nz < kz1) s13[d.ix(i, j, d.nz)] = 0.0;
    if (kz0 <= 2 && 2 < kz1) s23[d.ix(i, j, 2)] = 0.0;
    if (kz0 <= d.nz && d.nz < kz1) s23[d.ix(i, j, d.nz)] = 0.0;
  }
}

template <bool ALL>
void bct(double *const S[6], Dims d, cudaStream_t st, int k0, int k1) {
  const int kx0 = k0 > 2 ? k0 : 2, kx1 = k1 < d.nz ? k1 : d.nz;
  const int p = d.nx > d.ny ? d.nx : d.ny, q = d.ny > kx1 - kx0 ? d.ny : kx1 - kx0;
  DSG_COUNT k_bct<ALL><<<dim3((p + 31) / 32, (q + 7) / 8, 3), dim3(32, 8), 0, st>>>(S[0], S[1], S[2], S[3], S[4], S[5],
                                                                                    d, kx0, kx1, k0, k1);
}


}  // namespace

// x and y faces of the interior planes among k0 .. k1-1, and the z planes in
// that range (k0 = 1, k1 = nz + 1: everything).
cudaError_t bc_tensor_offdiag(double *s12, double *s13, double *s23, Dims d, cudaStream_t st, int k0, int k1) {
  double *const S[6] = {nullptr, nullptr, nullptr, s12, s13, s23};
  bct<false>(S, d, st, k0, k1);
  return cudaGetLastError();
}

cudaError_t bc_tensor(double *const S[6], Dims d, cudaStream_t st, int k0, int k1) {
  bct<true>(S, d, st, k0, k1);  // S = {S11, S22, S33, S12, S13, S23}
  return cudaGetLastError();
}

// csf with the reference's scratch aliasing: w11 = pressure array, w22 = fine
// residual array, w33 = fine rhs array; ccf is the routine's local array.
// scratch = false (inside a whole step, where the pressure phase overwrites
// all three before reading them): the filtered field goes straight to ccf
// and S11..S33 are not copied into w11..w33.
cudaError_t csf(const double *ccc, double *w11, double *w22, double *w33, double *ccf, double *const S[6],
                Dims d, double tau, double sigma, double h, cudaStream_t st, bool scratch) {
  const size_t bytes = d.count() * sizeof(double);
  // copy(ccf,ccc); filterc27(ccf,w22); copy(ccf,w22): filtering ccf == filtering ccc
  cudaError_t e = filterc27(ccc, scratch ? w22 : ccf, d, st);
  if (e != cudaSuccess) return e;
  if (scratch) {
    e = cudaMemcpyAsync(ccf, w22, bytes, cudaMemcpyDeviceToDevice, st);
    if (e != cudaSuccess) return e;
  }
  e = bc_out(ccf, d, st);
  if (e != cudaSuccess) return e;
  if (sigma == 0.0) {
    for (int m = 0; m < 6; m++) {
      e = cudaMemsetAsync(S[m], 0, bytes, st);
      if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
  }
  const double sigh = 0.5 * (tau * tau) * sigma / (h * h * h);
  DSG_BAND(k_csf, d, st, S[0], S[1], S[2], ccf, d, sigh);
  if (scratch) {
    if ((e = cudaMemcpyAsync(w11, S[0], bytes, cudaMemcpyDeviceToDevice, st)) != cudaSuccess) return e;
    if ((e = cudaMemcpyAsync(w22, S[1], bytes, cudaMemcpyDeviceToDevice, st)) != cudaSuccess) return e;
    if ((e = cudaMemcpyAsync(w33, S[2], bytes, cudaMemcpyDeviceToDevice, st)) != cudaSuccess) return e;
  }
  return bc_tensor(S, d, st);
}

}  // namespace dsg
