// mgcluster.cuh -- the coarse levels of a multigrid cycle in one launch of one
// thread-block cluster (mglin's recursion, main.f:3703-3759).
//
// Below about 40^3 cells a colour pass is a few hundred nanoseconds of work
// behind a launch of three microseconds or more, and a V-cycle has 16 to 32
// passes on every level.  Here one cluster of up to 16 blocks runs all of
// them.  A level is cut into slabs of z planes, one slab per block, whose u
// stays in the block's shared memory for the whole launch.  A thread owns
// fixed cells of its block's slab for a whole smoothing phase and keeps their
// coefficients, right-hand side and the shared-memory offsets of their
// neighbours in registers: a ghost neighbour's offset is the cell's own (or a
// zero's), so an update is seven loads, the arithmetic and one store, with no
// index arithmetic or tests.  A cell on a slab's first or last plane also goes
// to the neighbour block's halo plane, as an asynchronous store that counts
// its bytes on an mbarrier there: a pass ends when a block has the bytes of
// its two neighbours, and no barrier over the cluster separates the passes.
// What bounds it: the exchange (about 0.25 us) on the small levels, shared-
// memory and issue rate on 32^3 and 40^3, the FP64 pipe of 16 SMs in FP64.
// FP32 passes take 0.25 us at 16^3, 0.45 at 24^3, 0.51 at 32^3, 0.96 at 40^3,
// a V(8,8) from 32^3 down 65 us; as launches a pass took 2.9 us, and the levels
// of at most 16^3 cells 87 us in one block.  With a cluster barrier at the end
// of every pass instead of the counted stores the same passes took 0.65, 0.78,
// 0.84 and 1.64 us.
// Levels that one block updates faster than a cluster barrier takes run in
// block 0 alone with block barriers.
//
// Every cell gets the operations of the one-launch-per-pass kernels in their
// order (the arithmetic policy A calls the same expressions), so the results
// are bit for bit theirs.
#pragma once
#include <cuda_runtime.h>

namespace dsg {
namespace mgc {

constexpr int kThreads = 256;     // threads of a block (255 registers each)
constexpr int kMaxCluster = 16;   // blocks of a cluster (a non-portable size)
constexpr int kMaxLevels = 8;
constexpr size_t kMaxShared = 220 * 1024;  // bytes of shared memory a block may ask for

template <class T>
struct Level {
  T *u, *rhs;                // node arrays in global memory, one ghost layer
  const T *a, *b, *c, *ei;
  int nx, ny, nz;            // interior cells
  int nd;                    // blocks that own a slab of this level
  short lo[kMaxCluster + 1]; // first plane of each block's slab (nz past the last)
  int np;                    // planes of the largest slab
  int hx, hp, half;          // u's row, plane and colour lengths (u_at)
  float i_hx, i_ny, i_nx, i_p, i_nz;  // reciprocals of hx, ny, nx, nx ny, nz
  T h2, h2i;                 // spacing squared and its reciprocal
  int npre, npost, cycles;   // sweeps of a V-cycle; V-cycles of the full-multigrid start
  // element offsets in a block's shared memory: u; the arrays of the slab's
  // cells, o_s values apart -- the six face coefficients, ei and the
  // right-hand side (below the top level; of the top level ei and the
  // right-hand side alone, or nothing: o_s = 0); the three words of neighbour
  // offsets per cell (below the top level)
  int o_u, o_k, o_s, o_x;
};

template <class T>
struct Args {
  Level<T> lv[kMaxLevels + 1];  // 1..top
  int top, ntop;
  int fmg;     // 0: one V-cycle from `top`, from u = 0; 1: full multigrid from level 1 up to `top`
  int tri;     // trilinear prolongation (else injection)
  T omega;
  T h2_first;  // spacing squared of the first coarsest solve of the full multigrid
  int o_res, o_buf;  // residual of one slab; coarse planes gathered for a prolongation
  int csize;         // blocks of the cluster
  size_t shared;     // bytes of shared memory per block
};

// Byte offsets in the head of a block's shared memory (see args() below).
constexpr int kDead = 24, kBars = 32, kArgs = 64;
template <class T>
constexpr size_t kHeadBytes = (kArgs + sizeof(Args<T>) + 31) / 32 * 32;

__host__ __device__ inline int row_len(int nx) { return (nx + 1) / 2; }

#ifdef __CUDACC__

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

__device__ __forceinline__ int cluster_rank() {
  unsigned r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return (int)r;
}

// The block's dynamic shared memory as an array of T.  Device code names it
// through this function instead of passing pointers around, so that every
// access is a shared-memory instruction and not a generic one.
extern __shared__ __align__(16) unsigned char cluster_smem[];
template <class T>
__device__ __forceinline__ T *smem() {
  return reinterpret_cast<T *>(cluster_smem);
}

// Head of the shared memory: a zero (the ghost beyond x = nx), a flag set when
// a wait ran out, the mbarriers of the halo planes [from block rank - 1, from
// block rank + 1][even, odd pass], and a copy of the arguments (reading them
// in place would go through generic loads).
template <class T>
__device__ __forceinline__ const Args<T> &args() {
  return *reinterpret_cast<const Args<T> *>(cluster_smem + kArgs);
}
// Element `off` of the shared memory of block `rank`, as a cluster address;
// its load and store.
template <class T>
__device__ __forceinline__ unsigned remote(int off, int rank) {
  unsigned out;
  const unsigned a = (unsigned)__cvta_generic_to_shared(smem<T>() + off);
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(a), "r"(rank));
  return out;
}
__device__ __forceinline__ float remote_load(unsigned a, float) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ double remote_load(unsigned a, double) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void remote_store(unsigned a, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void remote_store(unsigned a, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
// The same, counted on the mbarrier `bar` of that block.
__device__ __forceinline__ void remote_store_async(unsigned a, float v, unsigned bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(a),
               "r"(__float_as_uint(v)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void remote_store_async(unsigned a, double v, unsigned bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(a),
               "l"(__double_as_longlong(v)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ unsigned bar_at(int i) {
  return (unsigned)__cvta_generic_to_shared(cluster_smem + kBars + 8 * i);
}
__device__ __forceinline__ unsigned bar_remote(int i, int rank) {
  unsigned out;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(bar_at(i)), "r"(rank));
  return out;
}
__device__ __forceinline__ void bar_expect(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Waits for the phase of `parity`, for a limited number of tries: the
// neighbour's stores cannot fail to arrive, but if they did, the block marks
// itself dead, stops waiting and writes NaN as its result, which the solve's
// residual norm and the step's CFL check report.
__device__ __forceinline__ void bar_wait(unsigned bar, unsigned parity) {
  volatile int *dead = reinterpret_cast<volatile int *>(cluster_smem + kDead);
  for (int tries = 0; tries < (1 << 20); tries++) {
    unsigned done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return;
    if ((tries & 255) == 255 && *dead) return;
  }
  *dead = 1;
}

// e / d for 0 <= e < 2^20 and inv = 1 / d: the quotient (e + 0.5) / d is at
// least 0.5 / d away from an integer, further than its rounding error.
__device__ __forceinline__ int small_div(int e, float inv) { return (int)(((float)e + 0.5f) * inv); }

// First plane of block r's slab of a level (nd slabs of nz planes), its
// planes, and the block whose slab holds plane k.
template <class T>
__device__ __forceinline__ int slab_lo(const Level<T> &L, int r) {
  return L.lo[r];
}
template <class T>
__device__ __forceinline__ int slab_planes(const Level<T> &L, int r) {
  return L.lo[r + 1] - L.lo[r];
}
template <class T>
__device__ __forceinline__ int slab_owner(const Level<T> &L, int k) {
  return small_div((k + 1) * L.nd - 1, L.i_nz);
}

// Ordering point between phases on two levels: block 0 alone works on both,
// or the cluster does.
template <class T>
__device__ __forceinline__ void phase_barrier(const Level<T> &x, const Level<T> &y) {
  if (x.nd == 1 && y.nd == 1)
    __syncthreads();
  else
    cluster_barrier();
}

// u of a level lies in shared memory split by colour (i+j+k even, odd), each
// half (planes + 2 halo planes) x ny rows of hx = ceil(nx/2) values: in row
// (y, k) the cells of colour c are x = 2m + p, p = (y + k + c) & 1.  A colour
// pass then reads and writes contiguous runs; in natural order its stride of
// two made every access a two-way bank conflict.
// Offset of cell (x, y, k) in the u of the block whose slab starts at plane lo.
template <class T>
__device__ __forceinline__ int u_at(const Level<T> &L, int lo, int x, int y, int k) {
  return L.o_u + ((x + y + k) & 1) * L.half + (k - lo + 1) * L.hp + y * L.hx + (x >> 1);
}

// Coordinates of entry e of one colour of a slab: row e / hx of (plane, y),
// x = 2 (e % hx) + p.  False past the end and in the padding of a row.
struct Cell {
  int x, y, kl, p;
};
template <class T>
__device__ __forceinline__ bool cell_at(const Level<T> &L, int lo, int total, int col, int e, Cell &c) {
  const int row = small_div(e, L.i_hx);
  c.kl = small_div(row, L.i_ny);
  c.y = row - c.kl * L.ny;
  c.p = (c.y + lo + c.kl + col) & 1;
  c.x = 2 * (e - row * L.hx) + c.p;
  return e < total && c.x < L.nx;
}
// The neighbours of cell c as byte offsets in shared memory, two to a word:
// {x+1, x-1}, {y+1, y-1}, {z+1, z-1}.  A Neumann ghost is the cell itself, the
// ghost beyond x = nx the zero at offset 0 (bc_scalar's values).  Bit 0 of the
// three words (offsets are multiples of 4): a cell at all, stored in block
// rank - 1's halo, stored in block rank + 1's.  No cell: all zero.
struct Links {
  unsigned w[3];
};
template <class T>
__device__ __forceinline__ Links cell_links(const Level<T> &L, int lo, int np, const Cell &c, int col) {
  const int hx = L.hx, hp = L.hp, half = L.half, k = lo + c.kl;
  const int in = ((c.kl + 1) * L.ny + c.y) * hx + (c.x >> 1);
  const int own = L.o_u + col * half + in, w = L.o_u + (1 - col) * half + in;
  const unsigned z = sizeof(T);
  auto two = [&](int a, int b) { return (unsigned)a * z | (unsigned)b * z << 16; };
  Links r;
  r.w[0] = two(c.x + 1 == L.nx ? 0 : w + c.p, c.x == 0 ? own : w + c.p - 1) | 1u;
  r.w[1] = two(c.y + 1 == L.ny ? own : w + hx, c.y == 0 ? own : w - hx) | (c.kl == 0 && k > 0 ? 1u : 0u);
  r.w[2] = two(k + 1 == L.nz ? own : w + hp, k == 0 ? own : w - hp) | (c.kl == np - 1 && k + 1 < L.nz ? 1u : 0u);
  return r;
}

// The face coefficients, ei and right-hand side of a cell from global memory.
template <class T>
__device__ __forceinline__ void cell_load(const Level<T> &L, int lo, const Cell &c, T (&k)[8]) {
  const unsigned gx = L.nx + 2, gp = gx * (L.ny + 2);
  const unsigned g = (unsigned)(c.x + 1) + gx * (c.y + 1) + gp * (lo + c.kl + 1);
  k[0] = __ldg(L.a + g);
  k[1] = __ldg(L.a + g - 1);
  k[2] = __ldg(L.b + g);
  k[3] = __ldg(L.b + g - gx);
  k[4] = __ldg(L.c + g);
  k[5] = __ldg(L.c + g - gp);
  k[6] = __ldg(L.ei + g);
  k[7] = L.rhs[g];
}

// What the smoothing phases read from shared memory, in the order of cell_at,
// for all levels in one loop (their global loads overlap): coefficients, ei
// and neighbour offsets of the slabs' cells (of the top level ei and the
// right-hand side, where it has arrays); the right-hand sides too for the
// full-multigrid start (a V-cycle's restriction forms them).
template <class T>
__device__ void stage(const Args<T> &G, int rank) {
#pragma unroll 2
  for (int t0 = threadIdx.x;; t0 += kThreads) {
    int l = 1, t = t0, total = 0;
    for (; l <= G.top; l++) {
      total = G.lv[l].o_s ? G.lv[l].hp * slab_planes(G.lv[l], rank) : 0;
      if (t < 2 * total) break;
      t -= 2 * total;
    }
    if (l > G.top) break;
    const Level<T> &L = G.lv[l];
    const int lo = slab_lo(L, rank), np = slab_planes(L, rank), S = L.o_s;
    T *s = smem<T>() + L.o_k;
    unsigned *x = reinterpret_cast<unsigned *>(smem<T>() + L.o_x);
    const int col = t >= total, e = t - col * total, o = col * (S / 2) + e;
    Cell c;
    const bool cell = cell_at(L, lo, total, col, e, c);
    T k[8] = {};
    if (cell) cell_load(L, lo, c, k);
    if (l == G.top) {
      s[o] = k[6];
      s[S + o] = k[7];
    } else {
      Links w = {};
      if (cell) w = cell_links(L, lo, np, c, col);
#pragma unroll
      for (int m = 0; m < 7; m++) s[m * S + o] = k[m];
      if (G.fmg) s[7 * S + o] = k[7];
#pragma unroll
      for (int m = 0; m < 3; m++) x[m * S + o] = w.w[m];
    }
  }
}

// n sweeps of level L, NC cells per thread and colour, then (want_res) the
// residual of the slab at o_res, plane by plane.  A thread loads the
// neighbours of up to five cells before it stores the first: the loads of a
// colour pass never depend on its stores, but the compiler cannot know that.
// Above four cells per thread ei and the right-hand side stay in shared
// memory, for want of registers.
template <class A, int NC>
__device__ __noinline__ void smooth(int level, int rank, int n, typename A::T h2, bool want_res, int pass_lo,
                                    int pass_hi) {
  typedef typename A::T T;
  constexpr int B = NC <= 5 ? NC : NC / 2;
  constexpr bool REGS = NC <= 4;
  static_assert(NC % B == 0, "cells per thread in whole batches");
  T *const sm = smem<T>();
  const Args<T> &G = args<T>();
  const Level<T> &L = G.lv[level];
  const bool top = level == G.top;
  const int S = L.o_s, lo = slab_lo(L, rank), np = slab_planes(L, rank), hp = L.hp, total = hp * np, half = L.half;
  const T omega = G.omega;
  unsigned w[2][NC][3];
  T cf[2][NC][6], er[2][REGS ? NC : 1][2];
#pragma unroll
  for (int col = 0; col < 2; col++)
#pragma unroll
    for (int q = 0; q < NC; q++) {
      const int e = (int)threadIdx.x + q * kThreads, o = col * (S / 2) + e;
      T k[8] = {};
      Links l = {};
      if (top) {
        Cell c;
        if (cell_at(L, lo, total, col, e, c)) {
          l = cell_links(L, lo, np, c, col);
          cell_load(L, lo, c, k);
        }
      } else if (e < total) {
#pragma unroll
        for (int m = 0; m < 8; m++) k[m] = sm[L.o_k + m * S + o];
#pragma unroll
        for (int m = 0; m < 3; m++) l.w[m] = reinterpret_cast<const unsigned *>(sm + L.o_x)[m * S + o];
      }
#pragma unroll
      for (int m = 0; m < 6; m++) cf[col][q][m] = k[m];
      if (REGS) {
        er[col][REGS ? q : 0][0] = k[6];
        er[col][REGS ? q : 0][1] = k[7];
      }
#pragma unroll
      for (int m = 0; m < 3; m++) w[col][q][m] = l.w[m];
    }
  const T *ser = sm + L.o_k + (top ? 0 : 6 * S) + threadIdx.x;  // ei and, S further on, the right-hand side
  // this thread's first cell of colour 0 in its own u, in the upper halo plane
  // of block rank - 1 and in the lower halo plane of block rank + 1
  const bool has_lo = lo > 0, has_hi = lo + np < L.nz;
  const int o0 = L.o_u + hp + (int)threadIdx.x;
  const unsigned to_lo = has_lo ? remote<T>(o0 + slab_planes(L, rank - 1) * hp, rank - 1) : 0;
  const unsigned to_hi = has_hi ? remote<T>(o0, rank + 1) - np * hp * (unsigned)sizeof(T) : 0;
  const unsigned bar_lo = has_lo ? bar_remote(2, rank - 1) : 0, bar_hi = has_hi ? bar_remote(0, rank + 1) : 0;
  const int P = L.nx * L.ny, first = (int)threadIdx.x & ~31;
  // bytes of plane k's cells of colour c
  auto plane_bytes = [&](int k, int c) { return (unsigned)((P + 1 - ((k + c) & 1)) / 2 * (int)sizeof(T)); };
  auto at = [&](unsigned byte) { return *reinterpret_cast<const T *>(cluster_smem + byte); };
  // Own value, neighbours, ei and right-hand side of B cells of one colour.
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
      const bool in = (int)threadIdx.x + q * kThreads < total;
      v[b][0] = in ? sm[o0 + q * kThreads + col * half] : T(0);
#pragma unroll
      for (int m = 0; m < 3; m++) {
        v[b][1 + 2 * m] = at(l[m] & 0xFFFCu);
        v[b][2 + 2 * m] = at(l[m] >> 16);
      }
      v[b][7] = REGS ? er[col][REGS ? q : 0][0] : (in ? ser[col * (S / 2) + q * kThreads] : T(0));
      v[b][8] = REGS ? er[col][REGS ? q : 0][1] : (in ? ser[S + col * (S / 2) + q * kThreads] : T(0));
    }
  };
  for (int s = 0; s < n; s++)
#pragma unroll
    for (int col = 0; col < 2; col++) {
      const int odd_lo = (pass_lo + col) & 1, odd_hi = (pass_hi + col) & 1;
      if (threadIdx.x == 0) {
        if (has_lo) bar_expect(bar_at(odd_lo), plane_bytes(lo - 1, col));
        if (has_hi) bar_expect(bar_at(2 + odd_hi), plane_bytes(lo + np, col));
      }
#pragma unroll
      for (int q0 = 0; q0 < NC; q0 += B) {
        T v[B][9];
        load(col, q0, v);
#pragma unroll
        for (int b = 0; b < B; b++) {
          const T(&k)[6] = cf[col][q0 + b];
          const T(&x)[9] = v[b];
          // an FP64 instruction holds its warp scheduler's FP64 pipe for 64
          // cycles, also for a warp without a cell: skipping those took a pass
          // at 4^3 from 1.5 to 0.8 us, at 16^3 from 2.3 to 1.4
          if (sizeof(T) == 8 && first + (q0 + b) * kThreads >= total) continue;
          v[b][0] = A::relax(x[0], x[1], x[2], x[3], x[4], x[5], x[6], k[0], k[1], k[2], k[3], k[4], k[5], x[7], x[8],
                             h2, omega);
        }
#pragma unroll
        for (int b = 0; b < B; b++) {
          const int o = (q0 + b) * kThreads + col * half;
          const unsigned(&l)[3] = w[col][q0 + b];
          if (l[0] & 1u) sm[o0 + o] = v[b][0];
          if (l[1] & 1u) remote_store_async(to_lo + o * (unsigned)sizeof(T), v[b][0], bar_lo + 8 * odd_lo);
          if (l[2] & 1u) remote_store_async(to_hi + o * (unsigned)sizeof(T), v[b][0], bar_hi + 8 * odd_hi);
        }
      }
      __syncthreads();
      if (has_lo) bar_wait(bar_at(odd_lo), (unsigned)((pass_lo + col) >> 1) & 1u);
      if (has_hi) bar_wait(bar_at(2 + odd_hi), (unsigned)((pass_hi + col) >> 1) & 1u);
      if (col == 1) {
        pass_lo += 2;
        pass_hi += 2;
      }
    }
  if (want_res) {
#pragma unroll
    for (int col = 0; col < 2; col++)
#pragma unroll
      for (int q0 = 0; q0 < NC; q0 += B) {
        T v[B][9];
        load(col, q0, v);
#pragma unroll
        for (int b = 0; b < B; b++) {
          const T(&k)[6] = cf[col][q0 + b];
          const T(&x)[9] = v[b];
          if (sizeof(T) == 8 && first + (q0 + b) * kThreads >= total) continue;
          const T r = A::resid(x[0], x[1], x[2], x[3], x[4], x[5], x[6], k[0], k[1], k[2], k[3], k[4], k[5], x[8],
                               L.h2i);
          Cell c;
          if (cell_at(L, lo, total, col, (int)threadIdx.x + (q0 + b) * kThreads, c))
            sm[G.o_res + (c.kl * L.ny + c.y) * L.nx + c.x] = r;
        }
      }
  }
}

// Passes exchanged so far with block rank - 1 and with block rank + 1 (their
// parity picks the mbarrier and its phase).
struct Passes {
  int lo, hi;
};

template <class A>
__device__ void smooth_level(int l, int rank, int n, typename A::T h2, bool want_res, Passes &p) {
  const Level<typename A::T> &L = args<typename A::T>().lv[l];
  const int np = slab_planes(L, rank);
  if (np == 0) return;
  const int per = (L.hp * L.np + kThreads - 1) / kThreads;
  constexpr int M = A::kMaxCells;
  if (per <= 1) smooth<A, 1>(l, rank, n, h2, want_res, p.lo, p.hi);
  else if (per <= 2) smooth<A, 2>(l, rank, n, h2, want_res, p.lo, p.hi);
  else if (per <= 4) smooth<A, 4>(l, rank, n, h2, want_res, p.lo, p.hi);
  else smooth<A, M>(l, rank, n, h2, want_res, p.lo, p.hi);
  if (n > 0 && L.lo[rank] > 0) p.lo += 2 * n;
  if (n > 0 && L.lo[rank + 1] < L.nz) p.hi += 2 * n;
}

// u of a level = 0, halo planes included.
template <class T>
__device__ __forceinline__ void zero_u(const Level<T> &L) {
  for (int e = threadIdx.x; e < 2 * L.half; e += kThreads) smem<T>()[L.o_u + e] = T(0);
}

// Right-hand side of the coarse level = mean of the 8 fine residuals; its
// correction and halo planes = 0.  The block that owns fine plane 2 kc forms
// coarse plane kc (reading the residual of plane 2 kc + 1 from its
// neighbour's memory where the pair is split) and stores it at kc's owner.
template <class A>
__device__ void restrict_level(const Level<typename A::T> &F, const Level<typename A::T> &C, int rank, int o_res) {
  typedef typename A::T T;
  if (slab_planes(C, rank) > 0) zero_u(C);
  const int lo = slab_lo(F, rank), np = slab_planes(F, rank), P = F.nx * F.ny, Pc = C.nx * C.ny;
  if (np == 0) return;
  const int kc0 = (lo + 1) / 2, kc1 = (lo + np + 1) / 2;  // coarse planes of the slab's even planes
  const float ipc = C.i_p, inx = C.i_nx;
  const int chx = C.hx;
#pragma unroll 2
  for (int e = threadIdx.x; e < (kc1 - kc0) * Pc; e += kThreads) {
    const int kc = kc0 + small_div(e, ipc), r = e - (kc - kc0) * Pc, y = small_div(r, inx), x = r - y * C.nx;
    const int kl = 2 * kc - lo, f = 2 * y * F.nx + 2 * x;
    const T *p0 = smem<T>() + o_res + kl * P + f;
    T v[4];
    if (kl + 1 < np) {
      v[0] = p0[P];
      v[1] = p0[P + 1];
      v[2] = p0[P + F.nx];
      v[3] = p0[P + F.nx + 1];
    } else {
      const unsigned p1 = remote<T>(o_res + f, rank + 1), w = sizeof(T), row = F.nx * (unsigned)sizeof(T);
      v[0] = remote_load(p1, T(0));
      v[1] = remote_load(p1 + w, T(0));
      v[2] = remote_load(p1 + row, T(0));
      v[3] = remote_load(p1 + row + w, T(0));
    }
    const int owner = slab_owner(C, kc), klc = kc - slab_lo(C, owner);
    const int o = ((x + y + kc) & 1) * (C.o_s / 2) + (klc * C.ny + y) * chx + (x >> 1);
    remote_store(remote<T>(C.o_k + 7 * C.o_s + o, owner),
                 A::mean8(p0[0], p0[1], p0[F.nx], p0[F.nx + 1], v[0], v[1], v[2], v[3]));
  }
}

// Level F's u = or += the interpolated u of level C, on the slab and its halo
// planes (which then hold what their owners compute).
template <class A>
__device__ void prolong_level(const Level<typename A::T> &F, const Level<typename A::T> &C, int rank, int o_buf,
                              int add, int tri) {
  typedef typename A::T T;
  T *const sm = smem<T>();
  const int lo = slab_lo(F, rank), np = slab_planes(F, rank), P = F.nx * F.ny, Pc = C.nx * C.ny;
  if (np == 0) return;
  const int k0 = lo > 0 ? lo - 1 : 0, k1 = lo + np < F.nz ? lo + np : F.nz - 1;
  const int c0 = (k0 >> 1) > 0 ? (k0 >> 1) - 1 : 0, c1 = (k1 >> 1) + 1 < C.nz ? (k1 >> 1) + 1 : C.nz - 1;
  const float ipc = C.i_p, icx = C.i_nx;
#pragma unroll 4
  for (int e = threadIdx.x; e < (c1 - c0 + 1) * Pc; e += kThreads) {
    const int kl = small_div(e, ipc), k = c0 + kl, r = e - kl * Pc, y = small_div(r, icx), x = r - y * C.nx;
    const int owner = slab_owner(C, k);
    sm[o_buf + e] = remote_load(remote<T>(u_at(C, slab_lo(C, owner), x, y, k), owner), T(0));
  }
  __syncthreads();
  const float ip = F.i_p, inx = F.i_nx;
#pragma unroll 4
  for (int e = threadIdx.x; e < (k1 - k0 + 1) * P; e += kThreads) {
    const int kl = small_div(e, ip), r = e - kl * P, y = small_div(r, inx), x = r - y * F.nx, k = k0 + kl;
    const T v = A::prolong(sm + o_buf, C.nx, C.ny, C.nz, c0, x, y, k, tri);
    T *u = sm + u_at(F, lo, x, y, k);
    *u = add ? *u + v : v;
  }
}

template <class A>
__device__ void vcycle(int j, int rank, Passes &p) {
  const Args<typename A::T> &G = args<typename A::T>();
  for (int l = j; l >= 2; l--) {
    smooth_level<A>(l, rank, G.lv[l].npre, G.lv[l].h2, true, p);
    phase_barrier(G.lv[l], G.lv[l - 1]);
    restrict_level<A>(G.lv[l], G.lv[l - 1], rank, G.o_res);
    phase_barrier(G.lv[l], G.lv[l - 1]);
  }
  smooth_level<A>(1, rank, G.ntop, G.lv[1].h2, false, p);
  for (int l = 2; l <= j; l++) {
    phase_barrier(G.lv[l], G.lv[l - 1]);
    prolong_level<A>(G.lv[l], G.lv[l - 1], rank, G.o_buf, 1, G.tri);
    phase_barrier(G.lv[l], G.lv[l - 1]);
    smooth_level<A>(l, rank, G.lv[l].npost, G.lv[l].h2, false, p);
  }
}

template <class A>
__device__ void cluster_mg(const Args<typename A::T> &params) {
  typedef typename A::T T;
  static_assert(sizeof(Args<T>) % 4 == 0, "copied as words");
  const int rank = cluster_rank();
  for (int i = threadIdx.x; i < (int)(sizeof(Args<T>) / 4); i += kThreads)
    reinterpret_cast<unsigned *>(cluster_smem + kArgs)[i] = reinterpret_cast<const unsigned *>(&params)[i];
  if (threadIdx.x < kBars / 4) reinterpret_cast<unsigned *>(cluster_smem)[threadIdx.x] = 0u;
  if (threadIdx.x == 0) {
    for (int i = 0; i < 4; i++) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar_at(i)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  const Args<T> &G = args<T>();
  T *const sm = smem<T>();
  Passes p = {0, 0};
  stage(G, rank);
  zero_u(G.lv[G.fmg ? 1 : G.top]);
  cluster_barrier();
  if (G.fmg) {
    smooth_level<typename A::First>(1, rank, G.ntop, G.h2_first, false, p);
    for (int j = 2; j <= G.top; j++) {
      phase_barrier(G.lv[j], G.lv[j - 1]);
      prolong_level<A>(G.lv[j], G.lv[j - 1], rank, G.o_buf, 0, G.tri);
      phase_barrier(G.lv[j], G.lv[j - 1]);
      for (int c = 0; c < G.lv[j].cycles; c++) vcycle<A>(j, rank, p);
    }
  } else {
    vcycle<A>(G.top, rank, p);
  }
  __syncthreads();
  const Level<T> &L = G.lv[G.top];
  const int lo = slab_lo(L, rank), np = slab_planes(L, rank), P = L.nx * L.ny;
  const bool dead = *reinterpret_cast<volatile int *>(cluster_smem + kDead) != 0;
#pragma unroll 4
  for (int e = threadIdx.x; e < np * P; e += kThreads) {
    const int kl = small_div(e, L.i_p), r = e - kl * P, y = small_div(r, L.i_nx), x = r - y * L.nx;
    const T v = sm[u_at(L, lo, x, y, lo + kl)];
    L.u[(unsigned)(x + 1) + (unsigned)(L.nx + 2) * ((unsigned)(y + 1) + (unsigned)(L.ny + 2) * (unsigned)(lo + kl + 1))] =
        dead ? T(nan("")) : v;
  }
  cluster_barrier();  // no block leaves while another may still store into its shared memory
}

#endif  // __CUDACC__

// ---- host side ----------------------------------------------------------------

// Slabs and shared-memory layout of levels 1..top of G (their extents set),
// for clusters of csize blocks.  single: levels of at most this many cells run
// in one block.  Returns false when a block cannot hold them (shared memory,
// cells per thread).
template <class T>
bool layout(Args<T> &G, int top, int csize, int single, int max_cells) {
  size_t n = 0;
  int res = 0, buf = 0;
  auto take = [&](size_t k) {
    const size_t o = n;
    n += (k + 3) & ~(size_t)3;
    return (int)o;
  };
  n = kHeadBytes<T> / sizeof(T);
  for (int l = 1; l <= top; l++) {  // u first: the neighbour offsets are 16 bits
    Level<T> &L = G.lv[l];
    const long long cells = (long long)L.nx * L.ny * L.nz;
    if (cells > (1 << 20)) return false;
    L.nd = 1;
    if (cells > single) {
      const int most = L.nz < csize ? L.nz : csize, planes = (L.nz + most - 1) / most;
      L.nd = (L.nz + planes - 1) / planes;
    }
    for (int r = 0; r <= kMaxCluster; r++) L.lo[r] = (short)(r >= L.nd ? L.nz : r * L.nz / L.nd);
    L.np = (L.nz + L.nd - 1) / L.nd;
    L.hx = row_len(L.nx);
    L.hp = L.hx * L.ny;
    L.half = (L.np + 2) * L.hp;
    L.i_hx = 1.0f / (float)L.hx;
    L.i_ny = 1.0f / (float)L.ny;
    L.i_nx = 1.0f / (float)L.nx;
    L.i_p = 1.0f / (float)(L.nx * L.ny);
    L.i_nz = 1.0f / (float)L.nz;
    L.o_u = take((size_t)2 * L.half);
  }
  if (n * sizeof(T) > 0x10000) return false;
  for (int l = 1; l <= top; l++) {
    Level<T> &L = G.lv[l];
    const int np = L.np, P = L.nx * L.ny;
    const size_t half = (size_t)np * L.hp;  // one colour of a slab
    const size_t per = (half + kThreads - 1) / kThreads;
    if (per > (size_t)max_cells) return false;
    L.o_s = l < top || per > 4 ? (int)(2 * half) : 0;
    L.o_k = take((size_t)(l < top ? 8 : 2) * L.o_s);
    L.o_x = l < top ? take((3 * 2 * half * sizeof(unsigned) + sizeof(T) - 1) / sizeof(T)) : 0;
    if (l >= 2 && np * P > res) res = np * P;
    if (l < top) {
      // planes a slab of the finer level gathers: parents of its planes and
      // halo planes, and one more on either side
      const Level<T> &F = G.lv[l + 1];
      const int planes = F.np / 2 + 4;
      if ((planes < L.nz ? planes : L.nz) * P > buf) buf = (planes < L.nz ? planes : L.nz) * P;
    }
  }
  G.o_res = take(res);
  G.o_buf = take(buf);
  G.top = top;
  G.csize = csize;
  G.shared = n * sizeof(T);
  return G.shared <= kMaxShared;
}

#ifdef __CUDACC__

// Blocks of the largest cluster (16 or 8) of `kernel` the current device
// runs, 0 if none; sets the kernel's attributes on that device.
template <class K>
int cluster_size(K kernel) {
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxShared) != cudaSuccess ||
      cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  for (int c = kMaxCluster; c >= 8; c /= 2) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)c;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)c);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kMaxShared;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess && n > 0) return c;
    cudaGetLastError();
  }
  return 0;
}

template <class K, class T>
cudaError_t launch(K kernel, const Args<T> &args, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)args.csize;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)args.csize);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = args.shared;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  count_launch();
  return cudaLaunchKernelEx(&cfg, kernel, args);
}

#endif  // __CUDACC__

}  // namespace mgc
}  // namespace dsg
