// mg32_cells.cuh -- per-cell operations and per-block bodies of the FP32
// multigrid and FP64 defect-correction kernels (mg32.cu).
//
// Every kernel of mg32.cu is a thin wrapper that calls its block body here with
// its own blockIdx and gridDim.  The batched kernels of batch.cu call the same
// bodies with the block index a block has inside one ensemble member's grid,
// so a member solved in a batch computes exactly the bits it computes alone.
// Both translation units are compiled with FMA contraction.
#pragma once
#include "dsg_internal.cuh"

namespace dsg {
namespace mg32 {
namespace {  // each including translation unit keeps its own copies

// 32-bit linear index of node (i,j,k) (1-based, ghosts included): grids stay
// below 2^31 nodes, and 32-bit index arithmetic is markedly cheaper than
// 64-bit in these issue-bound sweeps.
__device__ __forceinline__ unsigned ix32(Dims d, int i, int j, int k) {
  return (unsigned)(i - 1) + (unsigned)d.nx * ((unsigned)(j - 1) + (unsigned)d.ny * (unsigned)(k - 1));
}

// Virtual-ghost neighbour reads of bc_scalar semantics on level dims d.
struct Nb {
  float xp, xm, yp, ym, zp, zm;
};

__device__ __forceinline__ Nb neighbours(const float *__restrict__ u, unsigned q, int i, int j, int k, Dims d,
                                         float uc) {
  Nb n;
  const float *uq = u + q;
  const int sy = d.nx, sz = d.nx * d.ny;
  n.xp = (i + 1 == d.nx) ? 0.f : uq[1];
  n.xm = (i - 1 == 1) ? uc : uq[-1];
  n.yp = (j + 1 == d.ny) ? uc : uq[sy];
  n.ym = (j - 1 == 1) ? uc : uq[-sy];
  n.zp = (k + 1 == d.nz) ? uc : uq[sz];
  n.zm = (k - 1 == 1) ? uc : uq[-sz];
  return n;
}

// ---- finest level: colour-split storage --------------------------------------
//
// On the finest level the FP32 correction u and right-hand side are stored
// split by colour: cells with i+j+k even (the first pass of relax) in one
// array, odd in another, each (nx-2)/2 x (ny-2) x (nz-2) over the interior
// only (ghosts are virtual).  In row (j,k) the colour-c cells are
// i = 2 + 2m + p with p = (j+k+c) & 1.  A colour pass then reads the other
// colour, reads and writes its own colour and reads cc for the face
// coefficients, all with full 32-byte sectors: 24 bytes per cell per relax.
// Face coefficients are formed from the FP32 volume fraction as abcei does,
// a = 1/(r1*(c_i+c_{i+1}) + r2), with bc_coef's a(1) = a(2).  (Storing cc
// colour-split as well, so that every load of a pass is a contiguous run, was
// measured slower: 3.88 against 4.25 TB/s at 256^3.)
struct Split {
  int hx, ny2, nz2;  // (nx-2)/2, ny-2, nz-2
  __host__ __device__ __forceinline__ size_t at(int m, int j, int k) const {
    return (size_t)m + (size_t)hx * ((size_t)(j - 2) + (size_t)ny2 * (size_t)(k - 2));
  }
};


__device__ __forceinline__ unsigned at32(Split sp, int m, int j, int k) {
  return (unsigned)m + (unsigned)sp.hx * ((unsigned)(j - 2) + (unsigned)sp.ny2 * (unsigned)(k - 2));
}

// Single-instruction reciprocal (MUFU): the FP32 V-cycle is a preconditioner
// of the FP64 defect correction, so an approximate 1/x is sufficient.
__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Sum over the six faces of coefficient times neighbour minus h2 * rhs, with
// every rounding spelled out: the compiler's own choice of fused operations
// differs between kernels (which product of the first sum it rounds, whether a
// loop-invariant h2 * rhs is formed on its own).
__device__ __forceinline__ float face_sum(float ae, float xp, float aw, float xm, float bn, float yp, float bs, float ym,
                                          float ct, float zp, float cb, float zm, float h2, float rhs) {
  float t = fmaf(ae, xp, aw * xm);
  t = fmaf(bn, yp, t);
  t = fmaf(bs, ym, t);
  t = fmaf(ct, zp, t);
  t = fmaf(cb, zm, t);
  return fmaf(-h2, rhs, t);
}
// Sum over the six faces of coefficient times the difference to the
// neighbour, and the residual that follows from it.
__device__ __forceinline__ float face_diff(float uc, float ae, float xp, float aw, float xm, float bn, float yp,
                                           float bs, float ym, float ct, float zp, float cb, float zm) {
  float t = fmaf(ae, xp - uc, aw * (xm - uc));
  t = fmaf(bn, yp - uc, t);
  t = fmaf(bs, ym - uc, t);
  t = fmaf(ct, zp - uc, t);
  return fmaf(cb, zm - uc, t);
}
// omega * t + (1 - omega) * u
__device__ __forceinline__ float over_relax(float omega, float t, float u) {
  return fmaf(1.f - omega, u, omega * t);
}

__device__ __forceinline__ float face_coef(float x, float y, float r1, float r2) {
  return rcp_approx(r1 * (x + y) + r2);
}

// ---- uniform segments ---------------------------------------------------------
//
// Most of the domain is pure gas or pure liquid.  A segment is 32 split
// indices of one row, both colours (i = 2 + 64 s .. 65 + 64 s): what one warp
// updates.  Where the volume fractions that a segment's cells read (theirs and
// their six neighbours') are all exactly 0 or all exactly 1, its flag is 1 or
// 2, every face coefficient is face_coef of that value twice, and a sweep
// reads neither cc nor forms seven reciprocals per cell: 16 instead of 24
// bytes and a third of the instructions, with the same bits.  The flag is read
// before anything depends on it, so that no load waits for a vote (a vote over
// the seven loaded fractions lost more than the reciprocals cost).  Else the
// flag is 0.  Only the grids that split_vec names use them (b_relax32_split).
constexpr int kVecCells = 200000;
__host__ __device__ __forceinline__ bool split_vec(Split sp) { return (sp.hx & 3) == 0 && (long long)sp.hx * sp.ny2 * sp.nz2 >= kVecCells; }
__host__ __device__ __forceinline__ int segments(Dims d) { return (((d.nx - 2) >> 1) + 31) / 32; }

__device__ __forceinline__ const unsigned char *seg_flag(const unsigned char *flags, Dims d, int j, int k) {
  return flags + ((unsigned)(j - 2) + (unsigned)(d.ny - 2) * (unsigned)(k - 2)) * (unsigned)segments(d);
}

// FP64 -> FP32 volume fraction of all nodes, and a code per segment and row
// (ghost rows included): 1 or 2 if the row's fractions from one cell before
// the segment to one after it (within 2..nx) are all 0 or all 1, else 0.  One
// warp per segment.
__device__ __forceinline__ void b_codes(const uint3 B, const uint3 G, float *__restrict__ dst,
                                        unsigned char *__restrict__ codes, const double *__restrict__ src, Dims d) {
  const unsigned ns = segments(d), total = ns * (unsigned)d.ny * (unsigned)d.nz, lane = threadIdx.x & 31;
  for (unsigned t = (B.x * blockDim.x + threadIdx.x) >> 5; t < total; t += G.x * blockDim.x >> 5) {
    const unsigned row = t / ns, s = t - row * ns;
    const double *in = src + (size_t)row * d.nx - 1;  // in[i]: node i of the row
    float *out = dst + (size_t)row * d.nx - 1;
    const int i0 = 2 + 64 * (int)s, ia = i0 + (int)lane, ib = ia + 32;
    const int before = i0 > 2 ? i0 - 1 : 2, after = i0 + 64 < d.nx ? i0 + 64 : d.nx;
    const float first = (float)in[i0];
    const float a = ia <= d.nx ? (float)in[ia] : first, b = ib <= d.nx ? (float)in[ib] : first;
    const float e = (float)in[lane == 0 ? before : after];
    if (ia <= d.nx) out[ia] = a;
    if (ib <= d.nx) out[ib] = b;
    if (s == 0 && lane == 0) out[1] = (float)in[1];
    if (s == ns - 1)
      for (int i = i0 + 64 + (int)lane; i <= d.nx; i += 32) out[i] = (float)in[i];
    const unsigned f = __float_as_uint(first);
    const bool same = __float_as_uint(a) == f && __float_as_uint(b) == f && __float_as_uint(e) == f;
    const bool all = __all_sync(0xffffffffu, same);
    if (lane == 0) codes[t] = !all ? 0 : (f == 0u ? 1 : (f == 0x3F800000u ? 2 : 0));
  }
}

// The flag of each interior segment: its row's code if the four rows around it
// have the same one.
__device__ __forceinline__ void b_flags(const uint3 B, const uint3 G, unsigned char *__restrict__ flags,
                                        const unsigned char *__restrict__ codes, Dims d) {
  const unsigned ns = segments(d), ny2 = d.ny - 2, total = ns * ny2 * (unsigned)(d.nz - 2);
  for (unsigned t = B.x * blockDim.x + threadIdx.x; t < total; t += G.x * blockDim.x) {
    const unsigned row = t / ns, s = t - row * ns, k = row / ny2, j = row - k * ny2;
    const unsigned sy = ns, sz = ns * (unsigned)d.ny, q = s + sy * (j + 1) + sz * (k + 1);
    const unsigned char c = codes[q];
    flags[t] = (codes[q - sy] == c) & (codes[q + sy] == c) & (codes[q - sz] == c) & (codes[q + sz] == c) ? c : 0;
  }
}

// Value of cell (i,j,k) of a colour-split pair {even, odd}.
__device__ __forceinline__ float split_get(const float *__restrict__ ev, const float *__restrict__ od, Split sp,
                                           int i, int j, int k) {
  const unsigned q = at32(sp, (i - 2) >> 1, j, k);
  return ((i + j + k) & 1) ? od[q] : ev[q];
}

// ---- prolongation of a coarse correction ------------------------------------
//
// Two interpolations: the reference's piecewise-constant injection (interp /
// addint, main.f:3866-3954: a fine cell takes its parent's value) and
// cell-centred trilinear interpolation, where a fine cell takes 3/4 of its
// parent plus 1/4 of the parent's neighbour on the fine cell's side along
// each axis (weights 27/64, 9/64, 3/64, 1/64).  Trilinear reaches the
// tolerance in fewer V-cycles (7 against 9 from a zero start on a 128^3
// splash system, V(4,4)).  Coarse ghosts are read virtually as bc_scalar
// sets them: the own value, and 0 beyond the x = nx face.  Explicit fmaf
// fixes the rounding, so that every kernel that interpolates gives the same
// bits.

// Bilinear y-z combination of the parent row's value (a) and its neighbours'
// along y (b), z (c) and both (e).
__device__ __forceinline__ float tri_yz_value(float a, float b, float c, float e) {
  return fmaf(0.0625f, e, fmaf(0.1875f, c, fmaf(0.1875f, b, 0.5625f * a)));
}

// Bilinear y-z combination at coarse x-index x (parent row pj, pk; neighbours nj, nk).
__device__ __forceinline__ float tri_yz(const float *__restrict__ uc, Dims dc, int x, int pj, int nj, int pk,
                                        int nk) {
  const float a = uc[ix32(dc, x, pj, pk)], b = uc[ix32(dc, x, nj, pk)];
  const float c = uc[ix32(dc, x, pj, nk)], e = uc[ix32(dc, x, nj, nk)];
  return tri_yz_value(a, b, c, e);
}

// Coarse neighbour of parent p on the side of fine index f (odd f: +1, even:
// -1); a Neumann ghost (index 1 or nc) resolves to the parent itself.
__device__ __forceinline__ int tri_nb(int f, int p, int nc) {
  const int n = p + ((f & 1) ? 1 : -1);
  return (n == 1 || n == nc) ? p : n;
}

// x-combination of the parent's and the neighbour's y-z values.
__device__ __forceinline__ float tri_x(float yp, float yn) { return fmaf(0.25f, yn, 0.75f * yp); }

// Trilinear value of the coarse correction uc at fine cell (i,j,k).
__device__ __forceinline__ float trilin32(const float *__restrict__ uc, Dims dc, int i, int j, int k) {
  const int pi = (i >> 1) + 1, pj = (j >> 1) + 1, pk = (k >> 1) + 1;
  const int nj = tri_nb(j, pj, dc.ny), nk = tri_nb(k, pk, dc.nz);
  const float yp = tri_yz(uc, dc, pi, pj, nj, pk, nk);
  const int ni = pi + ((i & 1) ? 1 : -1);
  const float yn = ni == dc.nx ? 0.f : (ni == 1 ? yp : tri_yz(uc, dc, ni, pj, nj, pk, nk));
  return tri_x(yp, yn);
}

// Coarse correction at fine cell (i,j,k): trilinear (TRI) or injection.
template <bool TRI>
__device__ __forceinline__ float coarse_at(const float *__restrict__ uc, Dims dc, int i, int j, int k) {
  return TRI ? trilin32(uc, dc, i, j, k) : uc[ix32(dc, (i >> 1) + 1, (j >> 1) + 1, (k >> 1) + 1)];
}

// One colour-c update (0 = i+j+k even) of the finest-level cell at split
// index (m, j, k).  Offsets are 32-bit (grids stay below 2^31 nodes) and
// taken from one base pointer per array, which cut the pass from 51.3 to
// 47.2 us at 258^3 against 64-bit indexing, with the same bits.  flag: of the
// cell's segment.
__device__ __forceinline__ void relax32_split_cell(float *__restrict__ self, const float *__restrict__ other,
                                                   const float *__restrict__ rhs_self, const float *__restrict__ cc,
                                                   Dims d, Split sp, int c, float h2, float omega, float r1, float r2,
                                                   int m, int j, int k, unsigned flag) {
  const int p = (j + k + c) & 1;
  const int i = 2 + 2 * m + p;
  const int row = sp.hx, plane = sp.hx * sp.ny2;
  const unsigned qs = (unsigned)m + (unsigned)sp.hx * ((unsigned)(j - 2) + (unsigned)sp.ny2 * (unsigned)(k - 2));
  const float *o = other + qs;
  const float uc = self[qs];
  const float xm = (m == 0 && p == 0) ? uc : o[p - 1];
  const float xp = (m == sp.hx - 1 && p == 1) ? 0.f : o[p];
  const float ym = (j == 2) ? uc : o[-row];
  const float yp = (j == d.ny - 1) ? uc : o[row];
  const float zm = (k == 2) ? uc : o[-plane];
  const float zp = (k == d.nz - 1) ? uc : o[plane];
  const float f = rhs_self[qs];
  float ae, aw, bn, bs, ct, cb;
  if (flag) {
    const float c0 = flag == 1 ? 0.f : 1.f;
    ae = aw = bn = bs = ct = cb = face_coef(c0, c0, r1, r2);
  } else {
    const unsigned q = (unsigned)(i - 1) + (unsigned)d.nx * ((unsigned)(j - 1) + (unsigned)d.ny * (unsigned)(k - 1));
    const float *cq = cc + q;
    const int sy = d.nx, sz = d.nx * d.ny;
    const float c0 = cq[0];
    ae = face_coef(c0, cq[1], r1, r2);
    aw = (i == 2) ? ae : face_coef(cq[-1], c0, r1, r2);
    bn = face_coef(c0, cq[sy], r1, r2);
    bs = face_coef(cq[-sy], c0, r1, r2);
    ct = face_coef(c0, cq[sz], r1, r2);
    cb = face_coef(cq[-sz], c0, r1, r2);
  }
  const float ei = rcp_approx(ae + aw + bn + bs + ct + cb);
  self[qs] = over_relax(omega, face_sum(ae, xp, aw, xm, bn, yp, bs, ym, ct, zp, cb, zm, h2, f) * ei, uc);
}

// Operator of the finest-level FP32 correction equation at the colour-c cell of
// split index (m, j, k) (qs its offset): sum_f a_f (z_f - z) over the six faces,
// with the neighbours, virtual ghosts and face coefficients of
// relax32_split_cell.  The residual of relax is rhs - lap / h^2.
__device__ __forceinline__ float lap32_split_cell(const float *__restrict__ self, const float *__restrict__ other,
                                                  const float *__restrict__ cc, Dims d, Split sp, int c, float r1,
                                                  float r2, int m, int j, int k, unsigned qs) {
  const int p = (j + k + c) & 1;
  const int i = 2 + 2 * m + p;
  const int row = sp.hx, plane = sp.hx * sp.ny2;
  const float *o = other + qs;
  const float uc = self[qs];
  const float xm = (m == 0 && p == 0) ? uc : o[p - 1];
  const float xp = (m == sp.hx - 1 && p == 1) ? 0.f : o[p];
  const float ym = (j == 2) ? uc : o[-row];
  const float yp = (j == d.ny - 1) ? uc : o[row];
  const float zm = (k == 2) ? uc : o[-plane];
  const float zp = (k == d.nz - 1) ? uc : o[plane];
  const unsigned q = (unsigned)(i - 1) + (unsigned)d.nx * ((unsigned)(j - 1) + (unsigned)d.ny * (unsigned)(k - 1));
  const float *cq = cc + q;
  const int sy = d.nx, sz = d.nx * d.ny;
  const float c0 = cq[0];
  const float ae = face_coef(c0, cq[1], r1, r2);
  const float aw = (i == 2) ? ae : face_coef(cq[-1], c0, r1, r2);
  const float bn = face_coef(c0, cq[sy], r1, r2);
  const float bs = face_coef(cq[-sy], c0, r1, r2);
  const float ct = face_coef(c0, cq[sz], r1, r2);
  const float cb = face_coef(cq[-sz], c0, r1, r2);
  return ae * (xp - uc) + aw * (xm - uc) + bn * (yp - uc) + bs * (ym - uc) + ct * (zp - uc) + cb * (zm - uc);
}

// One colour pass on the finest level.  Rows of a multiple of four split
// indices: a thread updates four neighbours; a warp whose cells all lie in
// uniform segments reads and writes them as 16-byte vectors, any other warp one
// by one (256^3: 28.4 us per pass, 45.4 with two cells per thread, uniform or
// not: that form issues 110 instructions per cell; 160^3: 7.6 against 12.9).
// Other rows, and grids of fewer than kVecCells cells per colour, which have
// too few threads that way (64^3: 3.3 us with two cells per thread, 3.7 with
// four): split indices m and m + blockDim.x.  split_cells: the split indices
// a block covers along a row.  VEC = split_vec(sp).
//
// The passes go through the planes back and forth (prolongation up, colour 0
// down, colour 1 up, restriction down), so that each begins with what the one
// before left in L2, and the right-hand side, which comes only every second
// pass, is loaded as streaming data that need not stay there: at 256^3, where u
// (67 MB) fits L2 and u and the right-hand side do not, a pass takes 28.4 us in
// one direction, 25.0 back and forth, 22.0 with both (the prolongation 42, 38,
// 33); at 160^3, which fits, it makes no difference.
__host__ __device__ __forceinline__ int split_cells(Split sp, int blk_x) { return (split_vec(sp) ? 4 : 2) * blk_x; }

template <bool VEC>
__device__ __forceinline__ void b_relax32_split(const uint3 B, const uint3 G, float *__restrict__ self, const float *__restrict__ other,
                                const float *__restrict__ rhs_self, const float *__restrict__ cc,
                                const unsigned char *__restrict__ flags, Dims d, Split sp, int c, float h2, float omega,
                                float r1, float r2) {
  const int j = B.y * blockDim.y + threadIdx.y + 2;
  const int k = (int)(c == 0 ? G.z - 1 - B.z : B.z) + 2;
  if (!VEC) {
    const int m = B.x * 2 * blockDim.x + threadIdx.x, m2 = m + (int)blockDim.x;
    if (j > d.ny - 1) return;
    if (m < sp.hx) relax32_split_cell(self, other, rhs_self, cc, d, sp, c, h2, omega, r1, r2, m, j, k, 0);
    if (m2 < sp.hx) relax32_split_cell(self, other, rhs_self, cc, d, sp, c, h2, omega, r1, r2, m2, j, k, 0);
    return;
  }
  const int m = 4 * (int)(B.x * blockDim.x + threadIdx.x);
  const bool in = j <= d.ny - 1 && m < sp.hx;
  const unsigned f = in ? seg_flag(flags, d, j, k)[m >> 5] : 1;  // the four cells lie in one segment
  if (!__all_sync(0xffffffffu, f != 0)) {
    if (in)
      for (int q = 0; q < 4; q++)
        relax32_split_cell(self, other, rhs_self, cc, d, sp, c, h2, omega, r1, r2, m + q, j, k, f);
    return;
  }
  if (!in) return;
  const int p = (j + k + c) & 1;
  const unsigned row = sp.hx, plane = sp.hx * sp.ny2;
  const unsigned q = (unsigned)m + row * (unsigned)(j - 2) + plane * (unsigned)(k - 2);
  auto vec = [](const float *x) { return *reinterpret_cast<const float4 *>(x); };
  const float *o = other + q;
  const float4 u = vec(self + q), x = vec(o), f4 = __ldcs(reinterpret_cast<const float4 *>(rhs_self + q));
  const float4 ym = (j == 2) ? u : vec(o - row), yp = (j == d.ny - 1) ? u : vec(o + row);
  const float4 zm = (k == 2) ? u : vec(o - plane), zp = (k == d.nz - 1) ? u : vec(o + plane);
  // along x: the cell before (p = 0) or after (p = 1) the vector x as well
  const float side = p ? (m + 4 == sp.hx ? 0.f : o[4]) : (m == 0 ? u.x : o[-1]);
  const float4 xm = p ? x : make_float4(side, x.x, x.y, x.z);
  const float4 xp = p ? make_float4(x.y, x.z, x.w, side) : x;
  const float c0 = f == 1 ? 0.f : 1.f;
  const float kf = face_coef(c0, c0, r1, r2);
  const float ei = rcp_approx(kf + kf + kf + kf + kf + kf);
  auto upd = [&](float uc, float e, float w, float n, float s, float t, float b, float f) {
    return over_relax(omega, face_sum(kf, e, kf, w, kf, n, kf, s, kf, t, kf, b, h2, f) * ei, uc);
  };
  *reinterpret_cast<float4 *>(self + q) =
      make_float4(upd(u.x, xp.x, xm.x, yp.x, ym.x, zp.x, zm.x, f4.x), upd(u.y, xp.y, xm.y, yp.y, ym.y, zp.y, zm.y, f4.y),
                  upd(u.z, xp.z, xm.z, yp.z, ym.z, zp.z, zm.z, f4.z), upd(u.w, xp.w, xm.w, yp.w, ym.w, zp.w, zm.w, f4.w));
}

// Mean of the 8 fine residuals of coarse cell (ic, jc, kc), from cc or, where
// its rows lie in one fluid (flag 1 or 2), with that one's coefficient.
__device__ __forceinline__ void resid_restrict32_split_cell(float *__restrict__ rhs_c, float *__restrict__ u_c,
                                                            const float *__restrict__ ue, const float *__restrict__ uo,
                                                            const float *__restrict__ re, const float *__restrict__ ro,
                                                            const float *__restrict__ cc, unsigned flag, Dims df, Split sp,
                                                            Dims dc, float h2i, float r1, float r2, int ic, int jc, int kc) {
  const float cu = flag == 2 ? 1.f : 0.f, ku = face_coef(cu, cu, r1, r2);
  float acc = 0.f;
#pragma unroll
  for (int dk = 0; dk < 2; dk++)
#pragma unroll
    for (int dj = 0; dj < 2; dj++)
#pragma unroll
      for (int di = 0; di < 2; di++) {
        const int i = 2 * ic - 2 + di, j = 2 * jc - 2 + dj, k = 2 * kc - 2 + dk;
        const float uc = split_get(ue, uo, sp, i, j, k);
        const float xp = (i + 1 == df.nx) ? 0.f : split_get(ue, uo, sp, i + 1, j, k);
        const float xm = (i == 2) ? uc : split_get(ue, uo, sp, i - 1, j, k);
        const float yp = (j + 1 == df.ny) ? uc : split_get(ue, uo, sp, i, j + 1, k);
        const float ym = (j == 2) ? uc : split_get(ue, uo, sp, i, j - 1, k);
        const float zp = (k + 1 == df.nz) ? uc : split_get(ue, uo, sp, i, j, k + 1);
        const float zm = (k == 2) ? uc : split_get(ue, uo, sp, i, j, k - 1);
        float ae = ku, aw = ku, bn = ku, bs = ku, ct = ku, cb = ku;
        if (!flag) {
          const float *cq = cc + ix32(df, i, j, k);
          const int sy = df.nx, sz = df.nx * df.ny;
          const float c0 = cq[0];
          ae = face_coef(c0, cq[1], r1, r2);
          aw = (i == 2) ? ae : face_coef(cq[-1], c0, r1, r2);
          bn = face_coef(c0, cq[sy], r1, r2);
          bs = face_coef(cq[-sy], c0, r1, r2);
          ct = face_coef(c0, cq[sz], r1, r2);
          cb = face_coef(cq[-sz], c0, r1, r2);
        }
        acc += fmaf(-h2i, face_diff(uc, ae, xp, aw, xm, bn, yp, bs, ym, ct, zp, cb, zm), split_get(re, ro, sp, i, j, k));
      }
  const unsigned qc = ix32(dc, ic, jc, kc);
  rhs_c[qc] = 0.125f * acc;
  u_c[qc] = 0.f;
}

// Finest-level residual (cc-derived operator, virtual ghosts) restricted to the
// coarse rhs: mean of the 8 fine residuals of each coarse cell.  A thread
// has two coarse cells, and where its rows lie in one fluid it loads the 24 rows
// of u and 8 of the right-hand side that their 16 residuals need as pairs, 40
// loads in place of 128 (256^3: 65 -> 34 us, 160^3 15.5 -> 13); grids below
// kPairCells have too few threads that way (128^3: 8.7 us, 10.1 so).
constexpr int kPairCells = 1500000;  // per colour
__host__ __device__ __forceinline__ bool split_pairs(Split sp) {
  return split_vec(sp) && (long long)sp.hx * sp.ny2 * sp.nz2 >= kPairCells;
}
// V: split_form, 0: no uniform segments, 1: one coarse cell per thread, 2: two.
__host__ __device__ __forceinline__ int split_form(Split sp) { return !split_vec(sp) ? 0 : split_pairs(sp) ? 2 : 1; }
template <int V>
__device__ __forceinline__ void b_resid_restrict32_split(const uint3 B, const uint3 G, float *__restrict__ rhs_c, float *__restrict__ u_c, const float *__restrict__ ue,
                                         const float *__restrict__ uo, const float *__restrict__ re,
                                         const float *__restrict__ ro, const float *__restrict__ cc,
                                         const unsigned char *__restrict__ flags, Dims df, Split sp, Dims dc, float h2i,
                                         float r1, float r2) {
  const int jc = B.y * blockDim.y + threadIdx.y + 2;
  const int kc = (int)(G.z - 1 - B.z) + 2;
  // the warp's coarse cells lie in one segment of each of the four rows
  const int m = (V == 2 ? 2 : 1) * (int)(B.x * blockDim.x + threadIdx.x);
  if (m >= sp.hx || jc > dc.ny - 1) return;
  const int seg = m >> 5, j0 = 2 * jc - 2, k0 = 2 * kc - 2;
  unsigned f00 = 0;
  if (V) {
    f00 = seg_flag(flags, df, j0, k0)[seg];
    const unsigned f10 = seg_flag(flags, df, j0 + 1, k0)[seg], f01 = seg_flag(flags, df, j0, k0 + 1)[seg],
                   f11 = seg_flag(flags, df, j0 + 1, k0 + 1)[seg];
    if (f00 != f10 || f00 != f01 || f00 != f11) f00 = 0;
  }
  if (V < 2 || !f00) {
    for (int t = 0; t < (V == 2 ? 2 : 1); t++)
      resid_restrict32_split_cell(rhs_c, u_c, ue, uo, re, ro, cc, V == 2 ? 0 : f00, df, sp, dc, h2i, r1, r2, m + t + 2, jc, kc);
    return;
  }
  const unsigned row = sp.hx, plane = sp.hx * sp.ny2;
  const unsigned q0 = (unsigned)m + row * (unsigned)(j0 - 2) + plane * (unsigned)(k0 - 2);
  auto vec = [](const float *x) { return *reinterpret_cast<const float2 *>(x); };
  // u of the four rows and of those beside them, even and odd cells
  float2 ev[4][4], od[4][4];
#pragma unroll
  for (int z = 0; z < 4; z++)
#pragma unroll
    for (int y = 0; y < 4; y++) {
      ev[z][y] = od[z][y] = make_float2(0.f, 0.f);
      if (((y == 0 || y == 3) && (z == 0 || z == 3)) || (y == 0 && j0 == 2) || (y == 3 && j0 + 2 == df.ny) ||
          (z == 0 && k0 == 2) || (z == 3 && k0 + 2 == df.nz))
        continue;
      const unsigned q = q0 + row * (unsigned)(y - 1) + plane * (unsigned)(z - 1);
      ev[z][y] = vec(ue + q);
      od[z][y] = vec(uo + q);
    }
  const float cu = f00 == 2 ? 1.f : 0.f, ku = face_coef(cu, cu, r1, r2);
  float acc0 = 0.f, acc1 = 0.f;
#pragma unroll
  for (int dk = 0; dk < 2; dk++)
#pragma unroll
    for (int dj = 0; dj < 2; dj++) {
      const int z = dk + 1, y = dj + 1;
      const bool odd = (dj + dk) & 1;  // colour of i = 2 + 2m, as j0 + k0 is even
      const unsigned q = q0 + row * (unsigned)dj + plane * (unsigned)dk;
      // of a row: cells 2 + 2m, 4 + 2m (first) and 3 + 2m, 5 + 2m; in the rows beside it the colours change places
      auto first = [&](int z, int y) { return ((y + z) & 1) ? od[z][y] : ev[z][y]; };
      auto second = [&](int z, int y) { return ((y + z) & 1) ? ev[z][y] : od[z][y]; };
      const float2 a = first(z, y), b = second(z, y);
      const float before = m == 0 ? a.x : (odd ? ue : uo)[q - 1], after = m + 2 == sp.hx ? 0.f : (odd ? uo : ue)[q + 2];
#pragma unroll
      for (int s = 0; s < 2; s++) {
        auto of = [&](int z, int y) { return s ? second(z, y) : first(z, y); };
        const float2 u = s ? b : a, f = __ldcs(reinterpret_cast<const float2 *>(((s != 0) != odd ? ro : re) + q));
        const float2 xp = s ? make_float2(a.y, after) : b, xm = s ? a : make_float2(before, b.x);
        const float2 yp = dj == 1 && j0 + 2 == df.ny ? u : of(z, y + 1), ym = dj == 0 && j0 == 2 ? u : of(z, y - 1);
        const float2 zp = dk == 1 && k0 + 2 == df.nz ? u : of(z + 1, y), zm = dk == 0 && k0 == 2 ? u : of(z - 1, y);
        acc0 += fmaf(-h2i, face_diff(u.x, ku, xp.x, ku, xm.x, ku, yp.x, ku, ym.x, ku, zp.x, ku, zm.x), f.x);
        acc1 += fmaf(-h2i, face_diff(u.y, ku, xp.y, ku, xm.y, ku, yp.y, ku, ym.y, ku, zp.y, ku, zm.y), f.y);
      }
    }
  const unsigned qc = ix32(dc, m + 2, jc, kc);
  rhs_c[qc] = 0.125f * acc0;
  rhs_c[qc + 1] = 0.125f * acc1;
  u_c[qc] = u_c[qc + 1] = 0.f;
}

// Fine (split) u = or += the interpolated coarse correction.
// One thread per coarse cell (m + 2, jc, kc): in each of its four fine rows the
// even and odd cell of split index m are its children, so both arrays are
// updated with coalesced accesses.  The eight children interpolate from 27
// coarse values, which a thread per row and split index would load as 48
// (160^3: 13.5 -> 10.1 us, 128^3 7.6 -> 6.7; at
// 256^3 memory bounds both).
template <bool TRI>
__device__ __forceinline__ void b_prolong32_split(const uint3 B, const uint3 G, float *__restrict__ ue, float *__restrict__ uo, const float *__restrict__ uc,
                                  Dims df, Split sp, Dims dc, int add) {
  const int m = B.x * blockDim.x + threadIdx.x;
  const int jc = B.y * blockDim.y + threadIdx.y + 2;
  const int kc = B.z + 2;
  if (m >= sp.hx || jc > dc.ny - 1) return;
  const int pi = m + 2;
  float v[3][3][3];  // coarse values at x, y, z -1 .. +1, Neumann ghosts resolved
  if (TRI) {
    const int jn[3] = {jc == 2 ? jc : jc - 1, jc, jc + 1 == dc.ny ? jc : jc + 1};
    const int kn[3] = {kc == 2 ? kc : kc - 1, kc, kc + 1 == dc.nz ? kc : kc + 1};
#pragma unroll
    for (int z = 0; z < 3; z++)
#pragma unroll
      for (int y = 0; y < 3; y++) {
        const float *p = uc + ix32(dc, pi, jn[y], kn[z]);
        v[1][y][z] = p[0];
        v[0][y][z] = p[-1];  // beyond the faces: not used
        v[2][y][z] = p[1];
      }
  } else {
    v[1][1][1] = uc[ix32(dc, pi, jc, kc)];
  }
#pragma unroll
  for (int dk = 0; dk < 2; dk++)
#pragma unroll
    for (int dj = 0; dj < 2; dj++) {
      float v0, v1;  // cells i = 2+2m and i = 3+2m
      if (TRI) {
        auto yz = [&](int x) {
          return tri_yz_value(v[x][1][1], v[x][2 * dj][1], v[x][1][2 * dk], v[x][2 * dj][2 * dk]);
        };
        const float yc = yz(1), yl = pi == 2 ? yc : yz(0), yr = pi + 1 == dc.nx ? 0.f : yz(2);
        v0 = tri_x(yc, yl);
        v1 = tri_x(yc, yr);
      } else {
        v0 = v1 = v[1][1][1];
      }
      const bool odd_first = (dj + dk) & 1;  // cell 2+2m of row (2 jc - 2 + dj, 2 kc - 2 + dk) has odd i+j+k
      const float ve = odd_first ? v1 : v0, vo = odd_first ? v0 : v1;
      const unsigned q = at32(sp, m, 2 * jc - 2 + dj, 2 * kc - 2 + dk);
      ue[q] = add ? ue[q] + ve : ve;
      uo[q] = add ? uo[q] + vo : vo;
    }
}

// 8-cell mean of the split fine rhs into the coarse interior (rstrct).
__device__ __forceinline__ void b_restrict32_split(const uint3 B, const uint3 G, float *__restrict__ uc, const float *__restrict__ re,
                                   const float *__restrict__ ro, Dims dc, Split sp) {
  const int ic = B.x * blockDim.x + threadIdx.x + 2;
  const int jc = B.y * blockDim.y + threadIdx.y + 2;
  const int kc = B.z + 2;
  if (ic > dc.nx - 1 || jc > dc.ny - 1) return;
  float acc = 0.f;
#pragma unroll
  for (int dk = 0; dk < 2; dk++)
#pragma unroll
    for (int dj = 0; dj < 2; dj++)
#pragma unroll
      for (int di = 0; di < 2; di++)
        acc += split_get(re, ro, sp, 2 * ic - 2 + di, 2 * jc - 2 + dj, 2 * kc - 2 + dk);
  uc[dc.ix(ic, jc, kc)] = 0.125f * acc;
}

// FP64 -> split FP32 (the fine rhs of the FMG start).
__device__ __forceinline__ void b_split_from64(const uint3 B, const uint3 G, float *__restrict__ ev, float *__restrict__ od, const double *__restrict__ src,
                               Dims d, Split sp) {
  const int i = B.x * blockDim.x + threadIdx.x + 2;
  const int j = B.y * blockDim.y + threadIdx.y + 2;
  const int k = B.z + 2;
  if (i > d.nx - 1 || j > d.ny - 1) return;
  float *dst = ((i + j + k) & 1) ? od : ev;
  dst[sp.at((i - 2) >> 1, j, k)] = (float)src[d.ix(i, j, k)];
}

// ---- coarse levels: natural layout ------------------------------------------
//
// The per-cell operations are shared by the one-launch-per-pass kernels and by
// the single-block tail kernel below, so both give the same bits.

// Red-black update of a cell with value uc from its neighbours and face
// coefficients (relax, main.f:3956-3997), and its residual.
__device__ __forceinline__ float relax32_value(float uc, const Nb &n, float ae, float aw, float bn, float bs, float ct,
                                               float cb, float ei, float rhs, float h2, float omega) {
  const float s = face_sum(ae, n.xp, aw, n.xm, bn, n.yp, bs, n.ym, ct, n.zp, cb, n.zm, h2, rhs);
  return over_relax(omega, s * ei, uc);
}
__device__ __forceinline__ float resid32_value(float uc, const Nb &n, float ae, float aw, float bn, float bs, float ct,
                                               float cb, float rhs, float h2i) {
  return fmaf(-h2i, face_diff(uc, ae, n.xp, aw, n.xm, bn, n.yp, bs, n.ym, ct, n.zp, cb, n.zm), rhs);
}

// One red-black update of cell (i,j,k).
__device__ __forceinline__ void relax32_cell(float *u, const float *rhs, const float *a, const float *b,
                                             const float *c, const float *ei, Dims d, int i, int j, int k,
                                             float h2, float omega) {
  const unsigned q = ix32(d, i, j, k);
  const unsigned sy = (unsigned)d.nx, sz = (unsigned)d.nx * d.ny;
  const float uc = u[q];
  const Nb n = neighbours(u, q, i, j, k, d, uc);
  u[q] = relax32_value(uc, n, a[q], a[q - 1], b[q], b[q - sy], c[q], c[q - sz], ei[q], rhs[q], h2, omega);
}

// Coarse rhs of coarse cell (ic,jc,kc) = mean of its 8 fine residuals (resid +
// rstrct, main.f:3718-3725); the coarse correction starts at zero (main.f:3726).
__device__ __forceinline__ void resid_restrict32_cell(float *rhs_c, float *u_c, const float *u, const float *rhs,
                                                      const float *a, const float *b, const float *c, Dims df,
                                                      Dims dc, float h2i, int ic, int jc, int kc) {
  const unsigned sy = (unsigned)df.nx, sz = (unsigned)df.nx * df.ny;
  float acc = 0.f;
#pragma unroll
  for (int dk = 0; dk < 2; dk++)
#pragma unroll
    for (int dj = 0; dj < 2; dj++)
#pragma unroll
      for (int di = 0; di < 2; di++) {
        const int i = 2 * ic - 2 + di, j = 2 * jc - 2 + dj, k = 2 * kc - 2 + dk;
        const unsigned q = ix32(df, i, j, k);
        const float uc = u[q];
        const Nb n = neighbours(u, q, i, j, k, df, uc);
        acc += resid32_value(uc, n, a[q], a[q - 1], b[q], b[q - sy], c[q], c[q - sz], rhs[q], h2i);
      }
  const unsigned qc = ix32(dc, ic, jc, kc);
  rhs_c[qc] = 0.125f * acc;
  u_c[qc] = 0.f;
}

__device__ __forceinline__ void b_relax32(const uint3 B, const uint3 G, float *__restrict__ u, const float *__restrict__ rhs, const float *__restrict__ a,
                          const float *__restrict__ b, const float *__restrict__ c, const float *__restrict__ ei,
                          Dims d, float h2, float omega, int colour) {
  const int j = B.y * blockDim.y + threadIdx.y + 2;
  const int k = B.z + 2;
  if (j > d.ny - 1) return;
  const int i = 2 + ((j + k + colour) & 1) + 2 * (int)(B.x * blockDim.x + threadIdx.x);
  if (i > d.nx - 1) return;
  relax32_cell(u, rhs, a, b, c, ei, d, i, j, k, h2, omega);
}

// Coarse rhs = mean of the 8 fine residuals; coarse correction = 0 (interior;
// the FP32 kernels never read ghost values).
__device__ __forceinline__ void b_resid_restrict32(const uint3 B, const uint3 G, float *__restrict__ rhs_c, float *__restrict__ u_c, const float *__restrict__ u,
                                   const float *__restrict__ rhs, const float *__restrict__ a,
                                   const float *__restrict__ b, const float *__restrict__ c, Dims df, Dims dc,
                                   float h2i) {
  const int ic = B.x * blockDim.x + threadIdx.x + 2;
  const int jc = B.y * blockDim.y + threadIdx.y + 2;
  const int kc = B.z + 2;
  if (ic > dc.nx - 1 || jc > dc.ny - 1) return;
  resid_restrict32_cell(rhs_c, u_c, u, rhs, a, b, c, df, dc, h2i, ic, jc, kc);
}

// u = or += the interpolated coarse correction (interp / addint,
// main.f:3866-3954), interior.
template <bool TRI>
__device__ __forceinline__ void b_prolong32(const uint3 B, const uint3 G, float *__restrict__ uf, const float *__restrict__ uc, Dims df, Dims dc, int add) {
  const int i = B.x * blockDim.x + threadIdx.x + 2;
  const int j = B.y * blockDim.y + threadIdx.y + 2;
  const int k = B.z + 2;
  if (i > df.nx - 1 || j > df.ny - 1) return;
  const unsigned q = ix32(df, i, j, k);
  const float v = coarse_at<TRI>(uc, dc, i, j, k);
  uf[q] = add ? uf[q] + v : v;
}

// ---- coarse tail: every level at or below `top` in one thread block ---------
//
// The batched ensemble solve's form of the coarse levels (a standalone solve
// runs them in a cluster, mgcluster.cuh; here each member's block must fit
// beside the other members').  The tail runs the rest of a V-cycle from level `top` down to the coarsest
// grid and back (pre-sweeps, residual restriction, NTOP coarsest sweeps,
// prolongation, post-sweeps: mglin's recursion, main.f:3703-3759) inside one
// block, with a block barrier between passes in place of a launch boundary.
// The level arrays stay in L1/L2.
// Threads 0..NT-1 of the block sweep level L n times; WARP: NT = 32 and the
// passes are separated by warp barriers (levels of a few dozen cells), else
// NT = blockDim.x and block barriers.
template <bool WARP>
__device__ void tail_relax(const TailLevel &L, int n, float omega) {
  const int nt = WARP ? 32 : (int)blockDim.x;
  const Dims d = L.d;
  const int hx = (d.nx - 1) / 2;  // cells of one colour per row, rounded up
  const int ny2 = d.ny - 2;
  const int total = hx * ny2 * (d.nz - 2);
  for (int s = 0; s < n; s++)
    for (int colour = 0; colour < 2; colour++) {
      for (int t = threadIdx.x; t < total; t += nt) {
        const int m = t % hx, r = t / hx;
        const int j = 2 + r % ny2, k = 2 + r / ny2;
        const int i = 2 + ((j + k + colour) & 1) + 2 * m;
        if (i <= d.nx - 1) relax32_cell(L.u, L.rhs, L.a, L.b, L.c, L.ei, d, i, j, k, L.h2, omega);
      }
      if (WARP) __syncwarp(); else __syncthreads();
    }
}

// Residual of level F restricted into level C's rhs, C's correction zeroed.
template <bool WARP>
__device__ void tail_restrict(const TailLevel &F, const TailLevel &C) {
  const int nt = WARP ? 32 : (int)blockDim.x;
  const int cx = C.d.nx - 2, cy = C.d.ny - 2, total = cx * cy * (C.d.nz - 2);
  const float h2i = 1.0f / F.h2;
  for (int t = threadIdx.x; t < total; t += nt) {
    const int ic = 2 + t % cx, r = t / cx;
    resid_restrict32_cell(C.rhs, C.u, F.u, F.rhs, F.a, F.b, F.c, F.d, C.d, h2i, ic, 2 + r % cy, 2 + r / cy);
  }
  if (WARP) __syncwarp(); else __syncthreads();
}

// Level F's correction += injection of level C's.
template <bool WARP>
__device__ void tail_addint(const TailLevel &F, const TailLevel &C, bool tri) {
  const int nt = WARP ? 32 : (int)blockDim.x;
  const int fx = F.d.nx - 2, fy = F.d.ny - 2, total = fx * fy * (F.d.nz - 2);
  for (int t = threadIdx.x; t < total; t += nt) {
    const int i = 2 + t % fx, r = t / fx;
    const int j = 2 + r % fy, k = 2 + r / fy;
    const unsigned q = ix32(F.d, i, j, k);
    const float v = tri ? coarse_at<true>(C.u, C.d, i, j, k) : coarse_at<false>(C.u, C.d, i, j, k);
    F.u[q] = F.u[q] + v;
  }
  if (WARP) __syncwarp(); else __syncthreads();
}

// Levels with at most this many interior cells (6^3 nodes and below) run in
// warp 0 alone, at most two cells per lane and pass.
constexpr int kTailWarpCells = 64;

__device__ void tail_body(const TailArgs &A) {
  // lw: the largest level small enough for one warp (0: none)
  int lw = 0;
  for (int l = 1; l <= A.top; l++) {
    const Dims d = A.lv[l].d;
    if ((d.nx - 2) * (d.ny - 2) * (d.nz - 2) <= kTailWarpCells) lw = l;
  }
  for (int l = A.top; l > lw && l >= 2; l--) {
    tail_relax<false>(A.lv[l], A.lv[l].npre, A.omega);
    tail_restrict<false>(A.lv[l], A.lv[l - 1]);
  }
  if (lw == 0) {
    tail_relax<false>(A.lv[1], A.ntop, A.omega);
  } else if (threadIdx.x < 32) {
    for (int l = lw; l >= 2; l--) {
      tail_relax<true>(A.lv[l], A.lv[l].npre, A.omega);
      tail_restrict<true>(A.lv[l], A.lv[l - 1]);
    }
    tail_relax<true>(A.lv[1], A.ntop, A.omega);
    for (int l = 2; l <= lw; l++) {
      tail_addint<true>(A.lv[l], A.lv[l - 1], A.tri);
      tail_relax<true>(A.lv[l], A.lv[l].npost, A.omega);
    }
  }
  if (lw > 0) __syncthreads();
  for (int l = (lw > 1 ? lw : 1) + 1; l <= A.top; l++) {
    tail_addint<false>(A.lv[l], A.lv[l - 1], A.tri);
    tail_relax<false>(A.lv[l], A.lv[l].npost, A.omega);
  }
}



// 8-cell mean of a fine interior field into the coarse interior (rstrct).
__device__ __forceinline__ void b_restrict32(const uint3 B, const uint3 G, float *__restrict__ uc, const float *__restrict__ uf, Dims dc, Dims df) {
  const int ic = B.x * blockDim.x + threadIdx.x + 2;
  const int jc = B.y * blockDim.y + threadIdx.y + 2;
  const int kc = B.z + 2;
  if (ic > dc.nx - 1 || jc > dc.ny - 1) return;
  const size_t f = df.ix(2 * ic - 2, 2 * jc - 2, 2 * kc - 2);
  const size_t sy = df.sy(), sz = df.sz();
  uc[dc.ix(ic, jc, kc)] = 0.125f * (uf[f] + uf[f + 1] + uf[f + sy] + uf[f + 1 + sy] + uf[f + sz] + uf[f + 1 + sz] +
                                    uf[f + sy + sz] + uf[f + 1 + sy + sz]);
}

__device__ __forceinline__ float acf(const float *a2, Dims df, int i1, int j1, int k1, int i2, int j2, int k2,
                                     int i3, int j3, int k3, int i4, int j4, int k4) {
  return 0.25f * (a2[df.ix(i1, j1, k1)] + a2[df.ix(i2, j2, k2)] + a2[df.ix(i3, j3, k3)] + a2[df.ix(i4, j4, k4)]);
}

// acfromac in FP32 (main.f:3793-3844).
__device__ __forceinline__ void b_acfromac32(const uint3 B, const uint3 G, float *__restrict__ a, float *__restrict__ b, float *__restrict__ c,
                             float *__restrict__ ei, const float *__restrict__ a2, const float *__restrict__ b2,
                             const float *__restrict__ c2, Dims dc, Dims df) {
  const int i = B.x * blockDim.x + threadIdx.x + 1;
  const int j = B.y * blockDim.y + threadIdx.y + 1;
  const int k = B.z + 1;
  if (i > dc.nx || j > dc.ny) return;
  const bool ii = i >= 2 && i <= dc.nx - 1, ji = j >= 2 && j <= dc.ny - 1, ki = k >= 2 && k <= dc.nz - 1;
  const size_t q = dc.ix(i, j, k);
#define AA(i, j, k) acf(a2, df, 2 * (i) - 1, 2 * (j) - 1, 2 * (k) - 1, 2 * (i) - 1, 2 * (j) - 2, 2 * (k) - 1, \
                        2 * (i) - 1, 2 * (j) - 1, 2 * (k) - 2, 2 * (i) - 1, 2 * (j) - 2, 2 * (k) - 2)
#define BB(i, j, k) acf(b2, df, 2 * (i) - 1, 2 * (j) - 1, 2 * (k) - 1, 2 * (i) - 2, 2 * (j) - 1, 2 * (k) - 1, \
                        2 * (i) - 1, 2 * (j) - 1, 2 * (k) - 2, 2 * (i) - 2, 2 * (j) - 1, 2 * (k) - 2)
#define CC(i, j, k) acf(c2, df, 2 * (i) - 1, 2 * (j) - 1, 2 * (k) - 1, 2 * (i) - 2, 2 * (j) - 1, 2 * (k) - 1, \
                        2 * (i) - 1, 2 * (j) - 2, 2 * (k) - 1, 2 * (i) - 2, 2 * (j) - 2, 2 * (k) - 1)
  float va = 0.f, vb = 0.f, vc = 0.f;
  if (i <= dc.nx - 1 && ji && ki) { va = AA(i, j, k); a[q] = va; }
  if (j <= dc.ny - 1 && ii && ki) { vb = BB(i, j, k); b[q] = vb; }
  if (k <= dc.nz - 1 && ii && ji) { vc = CC(i, j, k); c[q] = vc; }
  if (ii && ji && ki) ei[q] = 1.f / (va + AA(i - 1, j, k) + vb + BB(i, j - 1, k) + vc + CC(i, j, k - 1));
#undef AA
#undef BB
#undef CC
}

// ---- FP64 defect-correction kernels ----------------------------------------
// r = rhs - L p in FP64 over the interior (resid's operator, main.f:3912-3925,
// with bc_scalar ghosts read virtually), in flux form: L p = h2i (sum of
// a_f p_f - diag p) with p_f the neighbour (the cell itself behind a Neumann
// face, 0 behind the Dirichlet one) and diag the sum of the six face
// coefficients (stored by abcei), the same operator as sum a_f (p_f - p) in
// 11 instead of 17 FP64 operations per cell.  Writes (float)r as the FP32
// fine rhs and per-block partial sums of r^2 and rhs^2.
__device__ __forceinline__ void b_defect64(const uint3 B, const uint3 G, float *__restrict__ r_ev, float *__restrict__ r_od, Split sp,
                           double *__restrict__ partials, const double *__restrict__ p,
                           const double *__restrict__ rhs, const double *__restrict__ a,
                           const double *__restrict__ b, const double *__restrict__ c,
                           const double *__restrict__ diag, Dims d, double h2i) {
  const size_t n = (size_t)(d.nx - 2) * (d.ny - 2) * (d.nz - 2);
  const size_t sy = d.sy(), sz = d.sz();
  double rr = 0.0, bb = 0.0;
  for (size_t t = (size_t)B.x * blockDim.x + threadIdx.x; t < n; t += (size_t)G.x * blockDim.x) {
    const unsigned ni = (unsigned)(d.nx - 2), nj = (unsigned)(d.ny - 2), tt = (unsigned)t;  // < 2^32 cells
    const unsigned rem = tt / ni, kk = rem / nj;
    const int i = (int)(tt - rem * ni) + 2;
    const int j = (int)(rem - kk * nj) + 2, k = (int)kk + 2;
    const size_t q = d.ix(i, j, k);
    const double uc = p[q];
    const double xp = (i + 1 == d.nx) ? 0.0 : p[q + 1];
    const double xm = (i - 1 == 1) ? uc : p[q - 1];
    const double yp = (j + 1 == d.ny) ? uc : p[q + sy];
    const double ym = (j - 1 == 1) ? uc : p[q - sy];
    const double zp = (k + 1 == d.nz) ? uc : p[q + sz];
    const double zm = (k - 1 == 1) ? uc : p[q - sz];
    const double f = rhs[q];
    double lp = a[q] * xp;
    lp = fma(a[q - 1], xm, lp);
    lp = fma(b[q], yp, lp);
    lp = fma(b[q - sy], ym, lp);
    lp = fma(c[q], zp, lp);
    lp = fma(c[q - sz], zm, lp);
    lp = fma(-diag[q], uc, lp);
    const double r = fma(-h2i, lp, f);
    (((i + j + k) & 1) ? r_od : r_ev)[sp.at((i - 2) >> 1, j, k)] = (float)r;
    rr += r * r;
    bb += f * f;
  }
  __shared__ double s0[kRedThreads], s1[kRedThreads];
  s0[threadIdx.x] = rr;
  s1[threadIdx.x] = bb;
  __syncthreads();
  for (int s = kRedThreads / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      s0[threadIdx.x] += s0[threadIdx.x + s];
      s1[threadIdx.x] += s1[threadIdx.x + s];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    partials[2 * B.x] = s0[0];
    partials[2 * B.x + 1] = s1[0];
  }
}

__device__ __forceinline__ void b_fold2(const uint3 B, const uint3 G, const double *__restrict__ partials, double *__restrict__ out) {
  __shared__ double s0[kRedThreads], s1[kRedThreads];
  double a0 = 0.0, a1 = 0.0;
  for (int b = threadIdx.x; b < kRedBlocks; b += kRedThreads) {
    a0 += partials[2 * b];
    a1 += partials[2 * b + 1];
  }
  s0[threadIdx.x] = a0;
  s1[threadIdx.x] = a1;
  __syncthreads();
  for (int s = kRedThreads / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      s0[threadIdx.x] += s0[threadIdx.x + s];
      s1[threadIdx.x] += s1[threadIdx.x + s];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    out[0] = s0[0];
    out[1] = s1[0];
  }
}

// p += e (FP64 accumulation of the split FP32 correction), interior; `init`
// sets p = e.
__device__ __forceinline__ void b_correct64(const uint3 B, const uint3 G, double *__restrict__ p, const float *__restrict__ ev, const float *__restrict__ od,
                            Dims d, Split sp, int init) {
  const int i = B.x * blockDim.x + threadIdx.x + 2;
  const int j = B.y * blockDim.y + threadIdx.y + 2;
  const int k = B.z + 2;
  if (i > d.nx - 1 || j > d.ny - 1) return;
  const unsigned q = ix32(d, i, j, k);
  const double e = (double)split_get(ev, od, sp, i, j, k);
  p[q] = init ? e : p[q] + e;
}

// Coarse FP32 coefficients (acfromac) straight from the FP64 fine ones.
// FP64 fine coefficients to an FP32 coarse level, kAcfPlanes planes per block.
// Where all 24 fine faces of a coarse cell are the same (bulk gas or liquid),
// their means are that value, exactly, and ei is formed once for a run of such
// cells: the FP64 pipe, on which it ran into the momentum kernels beside it,
// has little left to do (256^3: 177 us, 64 now, what
// its memory traffic takes).
constexpr int kAcfPlanes = 2;
__device__ __forceinline__ void b_acfromac64to32(const uint3 B, const uint3 G, float *__restrict__ a, float *__restrict__ b, float *__restrict__ c,
                                 float *__restrict__ ei, const double *__restrict__ a2,
                                 const double *__restrict__ b2, const double *__restrict__ c2, Dims dc, Dims df) {
  const int i = B.x * blockDim.x + threadIdx.x + 1;
  const int j = B.y * blockDim.y + threadIdx.y + 1;
  if (i > dc.nx || j > dc.ny) return;
#define FA(i, j, k) (0.25 * (a2[df.ix(2 * (i) - 1, 2 * (j) - 1, 2 * (k) - 1)] + a2[df.ix(2 * (i) - 1, 2 * (j) - 2, 2 * (k) - 1)] + \
                             a2[df.ix(2 * (i) - 1, 2 * (j) - 1, 2 * (k) - 2)] + a2[df.ix(2 * (i) - 1, 2 * (j) - 2, 2 * (k) - 2)]))
#define FB(i, j, k) (0.25 * (b2[df.ix(2 * (i) - 1, 2 * (j) - 1, 2 * (k) - 1)] + b2[df.ix(2 * (i) - 2, 2 * (j) - 1, 2 * (k) - 1)] + \
                             b2[df.ix(2 * (i) - 1, 2 * (j) - 1, 2 * (k) - 2)] + b2[df.ix(2 * (i) - 2, 2 * (j) - 1, 2 * (k) - 2)]))
#define FC(i, j, k) (0.25 * (c2[df.ix(2 * (i) - 1, 2 * (j) - 1, 2 * (k) - 1)] + c2[df.ix(2 * (i) - 2, 2 * (j) - 1, 2 * (k) - 1)] + \
                             c2[df.ix(2 * (i) - 1, 2 * (j) - 2, 2 * (k) - 1)] + c2[df.ix(2 * (i) - 2, 2 * (j) - 2, 2 * (k) - 1)]))
  // coefficient and ei of the last cell in a uniform neighbourhood
  double v = 0.0;
  float vf = 0.f, ef = 0.f;
  bool some = false;
  const size_t fy = df.sy(), fz = df.sz();
  for (int k = kAcfPlanes * (int)B.z + 1; k <= kAcfPlanes * (int)(B.z + 1) && k <= dc.nz; k++) {
    const bool ii = i >= 2 && i <= dc.nx - 1, ji = j >= 2 && j <= dc.ny - 1, ki = k >= 2 && k <= dc.nz - 1;
    const size_t q = dc.ix(i, j, k);
    if (ii && ji && ki) {
      // its 24 fine faces; node f is the first of the cell's eight
      const size_t f = df.ix(2 * i - 2, 2 * j - 2, 2 * k - 2);
      const double x = a2[f];
      bool same = true;
#pragma unroll
      for (int m = 0; m < 4; m++) {
        const size_t yz = f + (m & 1 ? fy : 0) + (m & 2 ? fz : 0), xz = f + (m & 1) + (m & 2 ? fz : 0), xy = f + (m & 1) + (m & 2 ? fy : 0);
        same &= same_bits(a2[yz + 1], x) & same_bits(a2[yz - 1], x) & same_bits(b2[xz + fy], x) & same_bits(b2[xz - fy], x) &
                same_bits(c2[xy + fz], x) & same_bits(c2[xy - fz], x);
      }
      if (same) {
        if (!some || !same_bits(x, v)) {
          some = true;
          v = x;
          vf = (float)x;
          ef = (float)(1.0 / (x + x + x + x + x + x));
        }
        a[q] = b[q] = c[q] = vf;
        ei[q] = ef;
        continue;
      }
    }
    double va = 0.0, vb = 0.0, vc = 0.0;
    if (i <= dc.nx - 1 && ji && ki) { va = FA(i, j, k); a[q] = (float)va; }
    if (j <= dc.ny - 1 && ii && ki) { vb = FB(i, j, k); b[q] = (float)vb; }
    if (k <= dc.nz - 1 && ii && ji) { vc = FC(i, j, k); c[q] = (float)vc; }
    if (ii && ji && ki) ei[q] = (float)(1.0 / (va + FA(i - 1, j, k) + vb + FB(i, j - 1, k) + vc + FC(i, j, k - 1)));
  }
#undef FA
#undef FB
#undef FC
}


}  // namespace
}  // namespace mg32
}  // namespace dsg
