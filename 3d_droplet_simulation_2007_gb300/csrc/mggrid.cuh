// mggrid.cuh -- a smoothing phase of one multigrid level in one cooperative
// launch of up to one block per SM, for the levels between the cluster kernel
// (mgcluster.cuh) and the levels that fill the GPU for longer than a launch
// takes.
//
// A phase is up to 16 colour passes of a few microseconds each when launched
// one by one, nearly all of it launch and memory latency.  Here a block owns a
// box of the level (all of x, some rows, some planes) for the whole phase: u
// in shared memory split by colour with one halo row and plane on each side, a
// thread's coefficients and neighbour offsets in registers, as in the cluster
// kernel.  After a pass the boundary cells of that colour go to the four
// neighbours through global memory, each value in one 8-byte word with the
// pass's tag (FP64: two words), so that a reader needs no flag and no fence:
// it polls the word itself.  Words alternate between two buffers; a block
// cannot get two passes ahead of a neighbour, because each pass needs the
// neighbour's previous one.  Tags go on counting from launch to launch in a
// word per block.  The phase before a coarser level restricts its residual at
// the end, the phase after it adds the interpolated correction at the start.
//
// A phase has at least one sweep.  At its start a block reads cells of u and of
// the coarse correction that its neighbours own (of the latter diagonal
// neighbours' as well); at its end it writes its own u and, where it restricts,
// zeroes its own coarse cells.  The exchange alone keeps one block's end behind
// another's start: a neighbour posts its first words after its reads, and what
// it posts in the last pass it posts after the words of the pass before from
// its own neighbours.
//
// A pass takes 0.78 us at 40^3 FP32, 0.86 at 64^3, 1.8 at 80^3 and 1.3 at 32^3
// FP64, launched alone 2.2 to 3.0 us; a phase has 3 to 11 us around its passes.
// A whole step: 1054 us against 1138 (48^3, mixed), 5.03 ms against 6.09 (160^3),
// 872 us against 952 (64^3, FP64).  What bounds a pass is the round trip of the
// exchange through L2 and, at 80^3, the cells' instructions.
//
// Every cell gets the operations of the one-launch-per-pass kernels in their
// order, so the results are bit for bit theirs.
#pragma once
#include "mgcluster.cuh"

namespace dsg {
namespace mgg {

constexpr int kThreads = 256;
constexpr size_t kMaxShared = 200 * 1024;

// How a level is cut: py x pz boxes, rows and planes in units of `unit`.
struct Boxes {
  int nx, ny, nz;  // interior cells
  int py, pz;
  int unit;
  int ry, np;      // rows and planes of the largest box
  int hx;          // ceil(nx / 2)
  int cells;       // cells of a colour a thread owns, at most
  __host__ __device__ int y0(int b) const { return unit * (int)((long long)b * (ny / unit) / py); }
  __host__ __device__ int z0(int b) const { return unit * (int)((long long)b * (nz / unit) / pz); }
  __host__ __device__ int words() const { return 2 * hx * (ry + np); }  // values a block sends per pass, at most
  int halo() const { return (words() + kThreads - 1) / kThreads; }  // halo cells a thread owns, at most
  __host__ __device__ int half() const { return (np + 2) * (ry + 2) * hx; }
  __host__ __device__ int blocks() const { return py * pz; }
};

template <class T>
struct Args {
  Boxes g;
  T *u, *rhs;                   // node arrays (null: colour-split pairs, coefficients from cc)
  const T *a, *b, *c, *ei;
  T *us[2], *rs[2];
  const float *cc;
  float r1, r2;
  T h2, h2i, omega;
  int n;                        // sweeps, at least one
  T *rhs_c, *u_c;               // restriction at the end (null: none)
  const T *prolong;             // coarse correction added at the start (null: none)
  int add, tri;                 // u += (else =) the interpolated correction; trilinear
  int ghosts;                   // write u's ghosts as bc_scalar does
  unsigned long long *mail;     // 2 buffers per block
  unsigned *epoch;              // passes so far, per block
  int staged;                   // ei and rhs in shared memory (form)
  int o_er, o_res;              // element offsets in shared memory
  size_t shared;
  int box;                      // a phase of mgbox.cuh
  const unsigned char *flags;   // per eight cells of a row: uniform (1 gas, 2 liquid)
  T bulk[2], bulk_ei[2];        // face coefficient and ei of gas and liquid
};

// The cut of a level over at most `sms` blocks: the boxes with the least work
// per pass, by their cells and the halo they exchange (a halo cell costs about
// two cells), at most max_cells of them per thread and colour and max_halo halo
// cells per thread.  false: none fits.
inline bool plan(Boxes &g, int nx, int ny, int nz, int sms, size_t size, int max_cells, int max_halo) {
  g.nx = nx;
  g.ny = ny;
  g.nz = nz;
  g.hx = (nx + 1) / 2;
  g.unit = (ny & 1) || (nz & 1) ? 1 : 2;
  g.py = g.pz = 0;
  long long best = -1;
  const int uy = ny / g.unit, uz = nz / g.unit;
  for (int py = 1; py <= uy; py++)
    for (int pz = 1; pz <= uz && py * pz <= sms; pz++) {
      Boxes t = g;
      t.py = py;
      t.pz = pz;
      t.ry = (uy + py - 1) / py * g.unit;
      t.np = (uz + pz - 1) / pz * g.unit;
      const long long own = (long long)t.hx * t.ry * t.np, halo = t.words();
      t.cells = (int)((own + kThreads - 1) / kThreads);
      if (t.cells > max_cells || t.halo() > max_halo) continue;
      if (2 * (long long)t.half() * (long long)size + 64 > 0xFFFF) continue;
      const long long cost = own + 2 * halo;
      if (best < 0 || cost < best) {
        best = cost;
        g = t;
      }
    }
  return best >= 0;
}

// The kernel's form for a cut: cells per thread and colour that it has room for
// (1, 2, 4 or 8), with two, four, four and eight halo cells per thread.  Up to
// four a thread keeps its cells' ei and right-hand side in registers, in the
// last form they are staged in shared memory: long rows can need that form for
// their halo alone.
inline int form(const Boxes &g) {
  const int h = g.halo();
  if (g.cells <= 1 && h <= 2) return 1;
  if (h > 4) return 8;
  return g.cells <= 2 ? 2 : g.cells <= 4 ? 4 : 8;
}

template <class T>
bool layout(Args<T> &G) {
  const Boxes &g = G.g;
  size_t n = 64 / sizeof(T) + 2 * (size_t)g.half();
  n = (n + 3) & ~(size_t)3;
  G.staged = form(g) > 4;
  G.o_er = (int)n;
  if (G.staged) n += 4 * (size_t)g.hx * g.ry * g.np;
  G.o_res = (int)n;
  n += (size_t)g.nx * g.ry * g.np;
  G.shared = n * sizeof(T);
  return G.shared <= kMaxShared;
}

// 8-byte words of the exchange buffers of a level.
template <class T>
size_t mail_words(const Boxes &g) {
  return 2 * (size_t)g.blocks() * g.words() * (sizeof(T) / 4);
}

#ifdef __CUDACC__

extern __shared__ __align__(16) unsigned char grid_smem[];

__device__ __forceinline__ void post(unsigned long long *w, float v, unsigned tag) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(w),
               "l"((unsigned long long)tag << 32 | __float_as_uint(v))
               : "memory");
}
__device__ __forceinline__ void post(unsigned long long *w, double v, unsigned tag) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v), t = (unsigned long long)tag << 32;
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(w), "l"(t | (b & 0xFFFFFFFFull)) : "memory");
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(w + 1), "l"(t | b >> 32) : "memory");
}
__device__ __forceinline__ unsigned long long word(const unsigned long long *w) {
  unsigned long long x;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(x) : "l"(w) : "memory");
  return x;
}
// The value in a word or a pair of words, and whether they carry the tag.
__device__ __forceinline__ bool unpack(const unsigned long long (&x)[1], unsigned tag, float &v) {
  v = __uint_as_float((unsigned)x[0]);
  return (unsigned)(x[0] >> 32) == tag;
}
__device__ __forceinline__ bool unpack(const unsigned long long (&x)[2], unsigned tag, double &v) {
  v = __longlong_as_double((long long)((x[0] & 0xFFFFFFFFull) | x[1] << 32));
  return (unsigned)(x[0] >> 32) == tag && (unsigned)(x[1] >> 32) == tag;
}

using mgc::small_div;

// One phase.  NC: cells per thread and colour; NH: halo cells per thread.
template <class A, int NC, int NH, bool SPLIT>
__device__ void phase(const Args<typename A::T> &G) {
  typedef typename A::T T;
  constexpr int B = NC <= 4 ? NC : NC / 2;
  constexpr bool REGS = NC <= 4;
  constexpr int W = sizeof(T) / 4;  // words per value
  T *const sm = reinterpret_cast<T *>(grid_smem);
  volatile int *const dead = reinterpret_cast<volatile int *>(grid_smem + 32);
  const Boxes &g = G.g;
  const int by = (int)blockIdx.x % g.py, bz = (int)blockIdx.x / g.py;
  const int ya = g.y0(by), ry = g.y0(by + 1) - ya, za = g.z0(bz), np = g.z0(bz + 1) - za;
  const int hx = g.hx, rs = g.ry + 2, half = g.half(), total = hx * ry * np;
  const float ihx = 1.0f / hx, iry = 1.0f / ry;
  const Dims d{g.nx + 2, g.ny + 2, g.nz + 2};
  const int tid = threadIdx.x, cells = hx * g.ry * g.np;
  const T omega = G.omega, h2 = G.h2;
  constexpr int U0 = 64 / (int)sizeof(T);
  // element of (colour, m, row, plane), rows and planes from -1
  auto at = [&](int col, int m, int yl, int kl) { return U0 + col * half + ((kl + 1) * rs + yl + 1) * hx + m; };

  if (tid < 16) reinterpret_cast<unsigned *>(grid_smem)[tid] = 0u;  // the ghost beyond x = nx, the flag
  const unsigned epoch = G.epoch[blockIdx.x];
  // initial u of node (x, y, k) of colour col, 0-based, with the coarse correction
  auto start = [&](int col, int x, int y, int k) {
    T v = T(0);
    if (!G.prolong || G.add)
      v = SPLIT ? G.us[col][(unsigned)(x >> 1) + (unsigned)hx * ((unsigned)y + (unsigned)g.ny * (unsigned)k)]
                : G.u[(unsigned)(x + 1) + (unsigned)d.nx * ((unsigned)(y + 1) + (unsigned)d.ny * (unsigned)(k + 1))];
    if (G.prolong) {
      const T p = A::coarse(G.prolong, Dims{g.nx / 2 + 2, g.ny / 2 + 2, g.nz / 2 + 2}, x + 2, y + 2, k + 2, G.tri);
      v = G.add ? v + p : p;
    }
    return v;
  };
  // this thread's cells: coefficients, neighbour offsets (bytes, two to a
  // word), own offset; all global loads before the first store
  enum : unsigned { CELL = 1u << 16 };
  unsigned w[2][NC][3], own[2][NC];
  T u0[2][NC];
  T cf[2][NC][6], er[2][REGS ? NC : 1][2];
#pragma unroll
  for (int col = 0; col < 2; col++)
#pragma unroll
    for (int q = 0; q < NC; q++) {
      const int e = tid + q * kThreads, row = small_div(e, ihx), m = e - row * hx, kl = small_div(row, iry),
                yl = row - kl * ry, y = ya + yl, k = za + kl, p = (y + k + col) & 1, x = 2 * m + p;
      T f[8] = {};
      unsigned l[3] = {0, 0, 0}, o = 0;
      if (e < total && x < g.nx) {
        const int me = at(col, m, yl, kl), nb = at(1 - col, m, yl, kl);
        auto two = [](int a, int b) { return (unsigned)a * (unsigned)sizeof(T) | (unsigned)b * (unsigned)sizeof(T) << 16; };
        l[0] = two(x + 1 == g.nx ? 0 : nb + p, x == 0 ? me : nb + p - 1);
        l[1] = two(y + 1 == g.ny ? me : nb + hx, y == 0 ? me : nb - hx);
        l[2] = two(k + 1 == g.nz ? me : nb + rs * hx, k == 0 ? me : nb - rs * hx);
        o = (unsigned)me * (unsigned)sizeof(T) | CELL;
        u0[col][q] = start(col, x, y, k);
        if constexpr (SPLIT) {
          A::split_coefs(G, d, x + 2, y + 2, k + 2, f);
          f[7] = G.rs[col][(unsigned)m + (unsigned)hx * ((unsigned)y + (unsigned)g.ny * (unsigned)k)];
        } else {
          const unsigned gx = d.nx, gp = d.nx * d.ny, n = (unsigned)(x + 1) + gx * (y + 1) + gp * (k + 1);
          f[0] = __ldg(G.a + n);
          f[1] = __ldg(G.a + n - 1);
          f[2] = __ldg(G.b + n);
          f[3] = __ldg(G.b + n - gx);
          f[4] = __ldg(G.c + n);
          f[5] = __ldg(G.c + n - gp);
          f[6] = __ldg(G.ei + n);
          f[7] = G.rhs[n];
        }
      }
#pragma unroll
      for (int i = 0; i < 6; i++) cf[col][q][i] = f[i];
      if (REGS) {
        er[col][REGS ? q : 0][0] = f[6];
        er[col][REGS ? q : 0][1] = f[7];
      } else if (e < total) {
        sm[G.o_er + col * cells + e] = f[6];
        sm[G.o_er + (2 + col) * cells + e] = f[7];
      }
#pragma unroll
      for (int i = 0; i < 3; i++) w[col][q][i] = l[i];
      own[col][q] = o;
    }
  // this thread's halo cells: the neighbour's word (buffer 0), the byte offset
  // of colour 0, the word of this block's own cell beside it and its offset
  // from the halo's; bits 31 / 30 of dst: not a cell of colour 0 / 1 (the own
  // cell: of colour 1 / 0)
  const int wz = hx * g.ry, wy = hx * g.np;  // words of a z and a y face
  const unsigned long long *const mail = G.mail;
  const size_t per = (size_t)g.words() * W;  // words of a buffer
  unsigned src[NH], dst[NH], snd[NH];
  int step[NH];
  T h0[NH][2];
  const int fz = hx * ry, fy = hx * np;
#pragma unroll
  for (int q = 0; q < NH; q++) {
    int h = tid + q * kThreads, face = 0;
    src[q] = snd[q] = 0;
    step[q] = 0;
    dst[q] = 3u << 30;
    if (h >= fz) { h -= fz; face = 1; }
    if (face == 1 && h >= fz) { h -= fz; face = 2; }
    if (face == 2 && h >= fy) { h -= fy; face = 3; }
    if (face == 3 && h >= fy) face = 4;
    if (face > 3) continue;
    const int row = small_div(h, ihx), m = h - row * hx;
    const int yl = face < 2 ? row : (face == 2 ? -1 : ry), kl = face < 2 ? (face == 0 ? -1 : np) : row;
    const int y = ya + yl, k = za + kl;
    if (y < 0 || y >= g.ny || k < 0 || k >= g.nz) continue;
    const int nb = (by + (face == 2 ? -1 : face == 3 ? 1 : 0)) + g.py * (bz + (face == 0 ? -1 : face == 1 ? 1 : 0));
    // this block's face and the neighbour's opposite one
    const int mine = face < 2 ? face * wz : 2 * wz + (face - 2) * wy, theirs = face < 2 ? (1 - face) * wz : 2 * wz + (3 - face) * wy;
    src[q] = (unsigned)((size_t)nb * 2 * per + (size_t)(theirs + row * hx + m) * W);
    snd[q] = (unsigned)(mine + row * hx + m) * W;
    step[q] = (face < 2 ? (face == 0 ? rs : -rs) : (face == 2 ? 1 : -1)) * hx * (int)sizeof(T);
    dst[q] = (unsigned)at(0, m, yl, kl) * (unsigned)sizeof(T);
    if (2 * m + 1 >= g.nx) dst[q] |= ((y + k) & 1) ? 1u << 31 : 1u << 30;  // only p = 0 has a cell there
#pragma unroll
    for (int col = 0; col < 2; col++) {
      const int x = 2 * m + ((y + k + col) & 1);
      h0[q][col] = x < g.nx ? start(col, x, y, k) : T(0);
    }
  }
#pragma unroll
  for (int col = 0; col < 2; col++) {
#pragma unroll
    for (int q = 0; q < NC; q++)
      if (own[col][q] & CELL) *reinterpret_cast<T *>(grid_smem + (own[col][q] & 0xFFFCu)) = u0[col][q];
#pragma unroll
    for (int q = 0; q < NH; q++)
      if (dst[q] != 3u << 30) *reinterpret_cast<T *>(grid_smem + (dst[q] & 0xFFFFu) + col * half * (int)sizeof(T)) = h0[q][col];
  }
  unsigned long long *const out = G.mail + (size_t)blockIdx.x * 2 * per;
  __syncthreads();

  auto get = [&](unsigned byte) { return *reinterpret_cast<const T *>(grid_smem + byte); };
  auto load = [&](int col, int q0, T(&v)[B][9]) {
#pragma unroll
    for (int b = 0; b < B; b++) {
      const int q = q0 + b;
      unsigned l[3];
#pragma unroll
      for (int m = 0; m < 3; m++) {
        l[m] = w[col][q][m];
        asm volatile("" : "+r"(l[m]));  // keeps the six offsets from being unpacked ahead of the sweeps
      }
      const int e = tid + q * kThreads;
      v[b][0] = get(own[col][q] & 0xFFFCu);
#pragma unroll
      for (int m = 0; m < 3; m++) {
        v[b][1 + 2 * m] = get(l[m] & 0xFFFCu);
        v[b][2 + 2 * m] = get(l[m] >> 16);
      }
      v[b][7] = REGS ? er[col][REGS ? q : 0][0] : (e < total ? sm[G.o_er + col * cells + e] : T(0));
      v[b][8] = REGS ? er[col][REGS ? q : 0][1] : (e < total ? sm[G.o_er + (2 + col) * cells + e] : T(0));
    }
  };
  unsigned tag = epoch;
  for (int s = 0; s < G.n; s++)
#pragma unroll
    for (int col = 0; col < 2; col++) {
      tag++;
      const size_t buf = (tag & 1u) ? per : 0;
#pragma unroll
      for (int q0 = 0; q0 < NC; q0 += B) {
        T v[B][9];
        load(col, q0, v);
#pragma unroll
        for (int b = 0; b < B; b++) {
          const T(&k)[6] = cf[col][q0 + b];
          const T(&x)[9] = v[b];
          // a warp without a cell would take the FP64 pipe from the others
          if (sizeof(T) == 8 && (tid & ~31) + (q0 + b) * kThreads >= total) continue;
          v[b][0] = A::relax(x[0], x[1], x[2], x[3], x[4], x[5], x[6], k[0], k[1], k[2], k[3], k[4], k[5], x[7], x[8],
                             h2, omega);
        }
#pragma unroll
        for (int b = 0; b < B; b++) {
          const unsigned o = own[col][q0 + b];
          if (o & CELL) *reinterpret_cast<T *>(grid_smem + (o & 0xFFFCu)) = v[b][0];
        }
      }
      __syncthreads();
#pragma unroll
      for (int q = 0; q < NH; q++)
        if (!(dst[q] & (col ? 1u << 31 : 1u << 30)))
          post(out + buf + snd[q], get((dst[q] & 0xFFFFu) + step[q] + col * half * (int)sizeof(T)), tag);
      // the neighbours' cells of this colour, polled for a limited number of
      // tries: if they do not come, the block marks itself dead, waits no more
      // and writes NaN, which the residual norm or the CFL check reports
      unsigned left = 0;
#pragma unroll
      for (int q = 0; q < NH; q++)
        if (!(dst[q] & (col ? 1u << 30 : 1u << 31))) left |= 1u << q;
      for (int tries = 0; left; tries++) {
        unsigned long long x[NH][W];
#pragma unroll
        for (int q = 0; q < NH; q++)
          if (left >> q & 1u)
#pragma unroll
            for (int i = 0; i < W; i++) x[q][i] = word(mail + src[q] + buf + i);
#pragma unroll
        for (int q = 0; q < NH; q++) {
          T v;
          if ((left >> q & 1u) && unpack(x[q], tag, v)) {
            left &= ~(1u << q);
            *reinterpret_cast<T *>(grid_smem + (dst[q] & 0xFFFFu) + col * half * (int)sizeof(T)) = v;
          }
        }
        if ((tries & 255) == 255 && (*dead || tries > (1 << 20))) {
          *dead = 1;
          break;
        }
      }
      __syncthreads();
    }
  if (tid == 0) G.epoch[blockIdx.x] = tag;
  const bool bad = *dead != 0;
  // u back (and its ghosts), the residual for the restriction
#pragma unroll
  for (int col = 0; col < 2; col++)
#pragma unroll
    for (int q0 = 0; q0 < NC; q0 += B) {
      T v[B][9];
      load(col, q0, v);
#pragma unroll
      for (int b = 0; b < B; b++) {
        const T(&k6)[6] = cf[col][q0 + b];
        const T(&x)[9] = v[b];
        if (!(own[col][q0 + b] & CELL)) continue;
        const int e = tid + (q0 + b) * kThreads, row = small_div(e, ihx), m = e - row * hx, kl = small_div(row, iry),
                  yl = row - kl * ry, y = ya + yl, k = za + kl, xi = 2 * m + ((y + k + col) & 1);
        const T val = bad ? T(nan("")) : x[0];
        if (SPLIT) {
          G.us[col][(unsigned)m + (unsigned)hx * ((unsigned)y + (unsigned)g.ny * (unsigned)k)] = val;
        } else {
          G.u[(unsigned)(xi + 1) + (unsigned)d.nx * ((unsigned)(y + 1) + (unsigned)d.ny * (unsigned)(k + 1))] = val;
          if (G.ghosts) write_ghosts(G.u, d, xi + 2, y + 2, k + 2, val);
        }
        if (G.rhs_c)
          sm[G.o_res + row * g.nx + xi] = A::resid(x[0], x[1], x[2], x[3], x[4], x[5], x[6], k6[0], k6[1], k6[2], k6[3],
                                                   k6[4], k6[5], x[8], G.h2i);
      }
    }
  if (!G.rhs_c) return;
  __syncthreads();
  const int cx = g.nx / 2, cy = ry / 2, n = cx * cy * (np / 2);
  const unsigned cgx = cx + 2, cgy = g.ny / 2 + 2;
  const float icx = 1.0f / cx, icy = 1.0f / cy;
  for (int e = tid; e < n; e += kThreads) {
    const int row = small_div(e, icx), x = e - row * cx, k = small_div(row, icy), y = row - k * cy;
    const T *p = sm + G.o_res + (2 * k * ry + 2 * y) * g.nx + 2 * x, *p1 = p + ry * g.nx;
    const T r = A::mean8(p[0], p[1], p[g.nx], p[g.nx + 1], p1[0], p1[1], p1[g.nx], p1[g.nx + 1]);
    const unsigned c = (unsigned)(x + 1) + cgx * ((unsigned)(ya / 2 + y + 1) + cgy * (unsigned)(za / 2 + k + 1));
    G.rhs_c[c] = r;
    G.u_c[c] = T(0);
  }
}

// Blocks (one per SM) that a cooperative launch of these kernels may have on
// the current device, a few SMs left to other streams; 0: none.  Sets the
// kernels' shared-memory attribute on that device.
template <class... K>
int grid_blocks(int threads, size_t shared, K... kernels) {
  int dev = 0, sms = 0, coop = 0;
  bool ok = cudaGetDevice(&dev) == cudaSuccess &&
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
            cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) == cudaSuccess && coop;
  auto one = [&](auto k) {
    int n = 0;
    ok = ok && cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shared) == cudaSuccess &&
         cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, threads, shared) == cudaSuccess && n > 0;
  };
  (one(kernels), ...);
  cudaGetLastError();
  return ok && sms > 8 ? sms - 4 : 0;
}

template <class K, class T>
cudaError_t launch(K kernel, int threads, const Args<T> &args, cudaStream_t st) {
  if (args.n < 1) return cudaErrorInvalidValue;  // nothing would order the blocks' reads and writes
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.gridDim = dim3((unsigned)args.g.blocks());
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = args.shared;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  count_launch();
  return cudaLaunchKernelEx(&cfg, kernel, args);
}

#endif  // __CUDACC__

}  // namespace mgg
}  // namespace dsg
