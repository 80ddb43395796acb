// mgbox.cuh -- a smoothing phase of one large FP32 multigrid level in one
// cooperative launch: levels below the finest whose u and right-hand side, but
// not their coefficients, fit the SMs' shared memory (about 86^3 to 130^3
// cells).  Boxes, exchange words and arguments are mggrid.cuh's; what differs
// is the work per block.
//
// Launched pass by pass such a level moves u, right-hand side and coefficients
// through L2 for every colour.  Here u and the right-hand side stay in shared
// memory for the phase, and the cells that lie in one fluid with their
// neighbours -- nearly all of them -- need no coefficients.  A thread updates
// four cells of a row and colour at a time (an item), with 16-byte shared
// loads for the cells, their neighbours and the right-hand side; the other
// items are updated one cell per thread, with coefficients from global memory
// that are under way while the thread updates its uniform items.  The items on
// the box's faces go first: their values are on the way to the neighbours
// while the rest is updated.
//
// At 128^3 cells a phase of 16 passes takes 73 us in one fluid and about 95
// with a droplet's interface, 134 us as 18 launches (a pass 3.0 us against 7.7;
// a 256^3 step 11183 -> 10929 us).  What bounds a pass: shared-memory bandwidth
// (36 wavefronts per 32 items, 0.37 us per 512), the posting of the faces, and
// 0.5 us for the exchange.  The finest level has no such phase: with three
// sweeps its launches are too few to make up for the loads and the interface
// (160^3: 101 us against 60).
//
// Every cell gets the operations of the one-launch-per-pass kernels in their
// order, so the results are bit for bit theirs.
#pragma once
#include "mggrid.cuh"

namespace dsg {
namespace mgg {

constexpr int kBoxThreads = 512;
constexpr int kBoxHalo = 4;                     // halo items a thread fetches per pass
constexpr size_t kBoxShared = 224 * 1024;
constexpr int kBoxHead = 64;                    // bytes before u

// The cut of a level, whole rows of items (nx a multiple of 8), rows and
// planes in pairs, and its shared memory: u (even, odd cells), the item table,
// the right-hand side in u's layout.  false: none fits.
inline bool plan_box(Args<float> &G, int nx, int ny, int nz, int sms) {
  Boxes &g = G.g;
  g.nx = nx;
  g.ny = ny;
  g.nz = nz;
  g.hx = nx / 2;
  g.unit = 2;
  g.py = g.pz = 0;
  if ((nx & 7) || (ny & 1) || (nz & 1)) return false;
  long long best = -1;
  for (int py = 1; py <= ny / 2; py++)
    for (int pz = 1; pz <= nz / 2 && py * pz <= sms; pz++) {
      Boxes t = g;
      t.py = py;
      t.pz = pz;
      t.ry = (ny / 2 + py - 1) / py * 2;
      t.np = (nz / 2 + pz - 1) / pz * 2;
      const long long items = (long long)g.hx / 4 * t.ry * t.np, halo = t.words() / 4;
      const long long shared = kBoxHead + 16 * (long long)t.half() + (8 * items + 15) / 16 * 16;
      if (halo > kBoxHalo * kBoxThreads || shared > (long long)kBoxShared) continue;
      const long long cost = (items + kBoxThreads - 1) / kBoxThreads * kBoxThreads + 2 * halo;
      if (best < 0 || cost < best) {
        best = cost;
        g = t;
        G.shared = (size_t)shared;
      }
    }
  G.box = best >= 0;
  return best >= 0;
}

#ifdef __CUDACC__

// Four values and their tags: two words at w, two `far` words on (a warp's
// items are neighbours, so each store and load covers whole lines).
__device__ __forceinline__ void post4(unsigned long long *w, size_t far, float4 v, unsigned tag) {
  const unsigned long long t = (unsigned long long)tag << 32;
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(w), "l"(t | __float_as_uint(v.x)),
               "l"(t | __float_as_uint(v.y))
               : "memory");
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(w + far), "l"(t | __float_as_uint(v.z)),
               "l"(t | __float_as_uint(v.w))
               : "memory");
}
__device__ __forceinline__ void words2(const unsigned long long *w, unsigned long long &a, unsigned long long &b) {
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(w) : "memory");
}

__device__ __forceinline__ void copy_async(float *shared, const float *global) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(shared)), "l"(global) : "memory");
}

// An item's table entry.  x: its offset (of four values) in u, and above 16
// bits: its colour-0 cells start at x = 1 instead of 0; first and last of its
// row; on the domain's first / last row and plane (where a neighbour is the
// cell itself); liquid (else, if uniform, gas).  y: 1 + its words (of four) to
// the neighbour in z, and above 16 bits in y.
enum : unsigned {
  BOX_P = 1u << 16, BOX_X0 = 1u << 17, BOX_X1 = 1u << 18, BOX_Y0 = 1u << 19, BOX_Y1 = 1u << 20, BOX_Z0 = 1u << 21,
  BOX_Z1 = 1u << 22, BOX_LIQ = 1u << 23
};

template <class A>
__device__ void box_phase(const Args<float> &G) {
  unsigned char *const sm = grid_smem;
  volatile int *const dead = reinterpret_cast<volatile int *>(sm);
  int *const fill = reinterpret_cast<int *>(sm + 16);  // entries in each of the four lists
  const Boxes &g = G.g;
  const int by = (int)blockIdx.x % g.py, bz = (int)blockIdx.x / g.py;
  const int ya = g.y0(by), ry = g.y0(by + 1) - ya, za = g.z0(bz), np = g.z0(bz + 1) - za;
  const int hx = g.hx, h4 = hx / 4, rs = h4, ps = (g.ry + 2) * h4, half4 = g.half() / 4;
  const Dims d{g.nx + 2, g.ny + 2, g.nz + 2}, dc{g.nx / 2 + 2, g.ny / 2 + 2, g.nz / 2 + 2};
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, items = h4 * ry * np;
  const float ih4 = 1.0f / h4, iry = 1.0f / ry, irow = 1.0f / (g.ry + 2);
  const float omega = G.omega, h2 = G.h2;
  float4 *const U = reinterpret_cast<float4 *>(sm + kBoxHead);
  float4 *const R = U + 2 * half4;
  uint2 *const tab = reinterpret_cast<uint2 *>(R + 2 * half4);
  float *const uf = reinterpret_cast<float *>(U), *const rf = reinterpret_cast<float *>(R);
  const int half = 4 * half4;
  auto at4 = [&](int yl, int kl) { return (kl + 1) * ps + (yl + 1) * rs; };  // of a row
  auto node = [&](int x, int y, int k) {
    return (unsigned)(x + 1) + (unsigned)d.nx * ((unsigned)(y + 1) + (unsigned)d.ny * (unsigned)(k + 1));
  };
  const int faces = items - (ry - 2) * (np - 2) * h4;  // items on the box's faces

  if (tid < kBoxHead / 4) reinterpret_cast<int *>(sm)[tid] = 0;
  const unsigned epoch = G.epoch[blockIdx.x];
  __syncthreads();
  // u of the box's rows and of those beside it that the neighbours own, and
  // the right-hand side: a warp a row at a time, all copies under way at once
  const float iry2 = 1.0f / (ry + 2);
  for (int r = warp; r < (ry + 2) * (np + 2); r += kBoxThreads / 32) {
    const int kl = small_div(r, iry2) - 1, yl = r - (kl + 1) * (ry + 2) - 1, y = ya + yl, k = za + kl;
    const bool oy = yl < 0 || yl >= ry, ok = kl < 0 || kl >= np;
    if ((oy && ok) || y < 0 || y >= g.ny || k < 0 || k >= g.nz) continue;
    // x and x + 32 have the same colour
    const int o = 4 * at4(yl, kl) + (lane >> 1) + (((lane + y + k) & 1) ? half : 0);
    const unsigned n = node(lane, y, k);
    for (int x = lane; x < g.nx; x += 32) {
      const int i = o + ((x - lane) >> 1);
      if (!G.prolong || G.add) copy_async(uf + i, G.u + n + (x - lane));
      if (!oy && !ok) copy_async(rf + i, G.rhs + n + (x - lane));
    }
  }
  // the item table: from the front the items on the faces with coefficients of
  // their own, up to `faces` those without, and the same for the other items
  // behind them
  const int wz = g.hx * g.ry, wy = g.hx * g.np;
  for (int e0 = 0; e0 < items; e0 += kBoxThreads) {
    const int e = e0 + tid, row = small_div(e, ih4), m4 = e - row * h4, kl = small_div(row, iry), yl = row - kl * ry;
    const int y = ya + yl, k = za + kl;
    int list = -1;
    uint2 t = make_uint2(0, 0);
    if (e < items) {
      const unsigned code = G.flags[(unsigned)m4 + (unsigned)h4 * ((unsigned)y + (unsigned)g.ny * (unsigned)k)];
      t.x = (unsigned)(at4(yl, kl) + m4) | ((y + k) & 1 ? BOX_P : 0) | (m4 == 0 ? BOX_X0 : 0) | (m4 == h4 - 1 ? BOX_X1 : 0) |
            (y == 0 ? BOX_Y0 : 0) | (y == g.ny - 1 ? BOX_Y1 : 0) | (k == 0 ? BOX_Z0 : 0) | (k == g.nz - 1 ? BOX_Z1 : 0) |
            (code == 2 ? BOX_LIQ : 0);
      const unsigned z = (unsigned)(yl * h4 + m4 + 1), w = (unsigned)(wz / 2 + kl * h4 + m4 + 1);
      if (kl == 0 && k > 0) t.y = z;
      if (kl == np - 1 && k + 1 < g.nz) t.y = z + wz / 4;
      if (yl == 0 && y > 0) t.y |= w << 16;
      if (yl == ry - 1 && y + 1 < g.ny) t.y |= (w + wy / 4) << 16;
      const bool face = yl == 0 || yl == ry - 1 || kl == 0 || kl == np - 1;
      list = (face ? 0 : 2) + (code ? 1 : 0);
    }
#pragma unroll
    for (int l = 0; l < 4; l++) {
      const unsigned m = __ballot_sync(0xffffffffu, list == l);
      if (!m) continue;
      int base = 0;
      if (lane == 0) base = atomicAdd(fill + l, __popc(m));
      base = __shfl_sync(0xffffffffu, base, 0) + __popc(m & ((1u << lane) - 1));
      if (list == l) tab[l == 0 ? base : l == 1 ? faces - 1 - base : l == 2 ? faces + base : items - 1 - base] = t;
    }
  }
  // this thread's halo items: the neighbour's words (buffer 0), the offset in u
  const size_t per = (size_t)g.words(), far = per / 2;
  unsigned src[kBoxHalo];
  int dst[kBoxHalo];
  const int fz = h4 * ry, fy = h4 * np;
#pragma unroll
  for (int q = 0; q < kBoxHalo; q++) {
    int h = tid + q * kBoxThreads, face = 0;
    src[q] = 0;
    dst[q] = -1;
    if (h >= fz) { h -= fz; face = 1; }
    if (face == 1 && h >= fz) { h -= fz; face = 2; }
    if (face == 2 && h >= fy) { h -= fy; face = 3; }
    if (face == 3 && h >= fy) face = 4;
    if (face > 3) continue;
    const int row = small_div(h, ih4), m4 = h - row * h4;
    const int yl = face < 2 ? row : (face == 2 ? -1 : ry), kl = face < 2 ? (face == 0 ? -1 : np) : row;
    const int y = ya + yl, k = za + kl;
    if (y < 0 || y >= g.ny || k < 0 || k >= g.nz) continue;
    const int nb = (by + (face == 2 ? -1 : face == 3 ? 1 : 0)) + g.py * (bz + (face == 0 ? -1 : face == 1 ? 1 : 0));
    const int theirs = face < 2 ? (1 - face) * wz : 2 * wz + (3 - face) * wy;
    src[q] = (unsigned)((size_t)nb * 2 * per + (size_t)(theirs + row * hx + 4 * m4) / 2);
    dst[q] = at4(yl, kl) + m4;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  // the coarse correction: a lane has the two cells of a coarse one, whose
  // neighbours along x the next lanes interpolate; four such units at a time
  if (G.prolong) {
    constexpr int L = 4;
    const int chunks = (hx + 31) / 32, units = (ry + 2) * (np + 2) * chunks;
    const float ich = 1.0f / chunks;
    for (int t0 = warp; t0 < units; t0 += L * kBoxThreads / 32) {
      float c[L], lo[L], hi[L];
      int o[L];  // offset in u, + half for odd rows; -1: none
#pragma unroll
      for (int b = 0; b < L; b++) {
        const int t = t0 + b * kBoxThreads / 32, r = small_div(t, ich), m = 32 * (t - r * chunks) + lane, i = m + 2;
        const int kl = small_div(r, iry2) - 1, yl = r - (kl + 1) * (ry + 2) - 1, y = ya + yl, k = za + kl;
        const bool out = (yl < 0 || yl >= ry) && (kl < 0 || kl >= np);
        o[b] = t < units && !out && y >= 0 && y < g.ny && k >= 0 && k < g.nz && m < hx
                   ? 4 * at4(yl, kl) + m + ((y + k) & 1 ? half : 0)
                   : -1;
        c[b] = lo[b] = hi[b] = 0.f;
        if (o[b] < 0) continue;
        if (G.tri) {
          c[b] = A::coarse_yz(G.prolong, dc, i, y + 2, k + 2);
          if (lane == 0 && i > 2) lo[b] = A::coarse_yz(G.prolong, dc, i - 1, y + 2, k + 2);
          if (lane == 31 && i + 1 < dc.nx) hi[b] = A::coarse_yz(G.prolong, dc, i + 1, y + 2, k + 2);
        } else {
          c[b] = A::coarse(G.prolong, dc, 2 * m + 2, y + 2, k + 2, 0);
        }
      }
#pragma unroll
      for (int b = 0; b < L; b++) {
        const int m = (32 * ((t0 + b * kBoxThreads / 32) % chunks)) + lane;
        const float below = __shfl_up_sync(0xffffffffu, c[b], 1), above = __shfl_down_sync(0xffffffffu, c[b], 1);
        if (o[b] < 0) continue;
        float c0 = c[b], c1 = c[b];
        if (G.tri) {
          c0 = A::coarse_x(c[b], m == 0 ? c[b] : lane == 0 ? lo[b] : below);
          c1 = A::coarse_x(c[b], m == hx - 1 ? 0.f : lane == 31 ? hi[b] : above);
        }
        float &u0 = uf[o[b]], &u1 = uf[o[b] >= half ? o[b] - half : o[b] + half];
        u0 = G.add ? u0 + c0 : c0;
        u1 = G.add ? u1 + c1 : c1;
      }
    }
    __syncthreads();
  }
  const int slow_f = fill[0], fast_f = fill[1], slow_i = fill[2], fast_i = fill[3];

  // own value and neighbours of cell q of an item, colour col
  auto gather = [&](unsigned t, int col, int q, float (&v)[7]) {
    const int o = 4 * (int)(t & 0xFFFFu) + q;
    const float *own = uf + col * half + o;
    const float *b = uf + (1 - col) * half + o;
    const bool p = ((t & BOX_P) != 0) != (col != 0);
    v[0] = *own;
    v[1] = !p ? b[0] : ((t & BOX_X1) && q == 3 ? 0.f : b[1]);
    v[2] = p ? b[0] : ((t & BOX_X0) && q == 0 ? v[0] : b[-1]);
    v[3] = (t & BOX_Y1) ? v[0] : b[4 * rs];
    v[4] = (t & BOX_Y0) ? v[0] : b[-4 * rs];
    v[5] = (t & BOX_Z1) ? v[0] : b[4 * ps];
    v[6] = (t & BOX_Z0) ? v[0] : b[-4 * ps];
  };
  // its face coefficients and ei
  auto coefs = [&](unsigned t, int col, int q, float (&f)[7]) {
    const int o = (int)(t & 0xFFFFu), row = small_div(o, ih4), kk = small_div(row, irow);
    const int x = 8 * (o - row * h4) + 2 * q + (((t & BOX_P) != 0) != (col != 0) ? 1 : 0);
    const unsigned gx = d.nx, gp = d.nx * d.ny, n = node(x, ya + row - kk * (g.ry + 2) - 1, za + kk - 1);
    f[0] = __ldg(G.a + n);
    f[1] = __ldg(G.a + n - 1);
    f[2] = __ldg(G.b + n);
    f[3] = __ldg(G.b + n - gx);
    f[4] = __ldg(G.c + n);
    f[5] = __ldg(G.c + n - gp);
    f[6] = __ldg(G.ei + n);
  };
  unsigned long long *const mine = G.mail + (size_t)blockIdx.x * 2 * per;
  // items [slow0, slow0 + slow) cell by cell, [fast0, fast0 + fast) four cells at a time
  auto update = [&](int col, int slow0, int slow, int fast0, int fast, unsigned long long *out, unsigned tag) {
    constexpr int B = 2;  // cells whose coefficients are under way
    uint2 ts[B];
    float f[B][7];
    auto fetch = [&](int i) {
#pragma unroll
      for (int b = 0; b < B; b++)
        if (i + b * kBoxThreads < 4 * slow) {
          ts[b] = tab[slow0 + ((i + b * kBoxThreads) >> 2)];
          coefs(ts[b].x, col, i & 3, f[b]);
        }
    };
    auto finish = [&](int i) {
#pragma unroll
      for (int b = 0; b < B; b++)
        if (i + b * kBoxThreads < 4 * slow) {
          const int q = i & 3, o = col * half + 4 * (int)(ts[b].x & 0xFFFFu) + q;
          float v[7];
          gather(ts[b].x, col, q, v);
          const float r = A::relax(v[0], v[1], v[2], v[3], v[4], v[5], v[6], f[b][0], f[b][1], f[b][2], f[b][3], f[b][4],
                                   f[b][5], f[b][6], rf[o], h2, omega);
          uf[o] = r;
          const size_t w = (q & 2 ? far : 0) + (q & 1);
          if (ts[b].y & 0xFFFFu) post(out + 2 * (ts[b].y & 0xFFFFu) - 2 + w, r, tag);
          if (ts[b].y >> 16) post(out + 2 * (ts[b].y >> 16) - 2 + w, r, tag);
        }
    };
    fetch(tid);
    for (int i = tid; i < fast; i += kBoxThreads) {
      const uint2 t = tab[fast0 + i];
      float4 *const own = U + col * half4 + (t.x & 0xFFFFu);
      const float4 *const o = U + (1 - col) * half4 + (t.x & 0xFFFFu);
      const bool p = ((t.x & BOX_P) != 0) != (col != 0);
      const float4 u = *own, x = *o, r = R[col * half4 + (t.x & 0xFFFFu)];
      const float4 ym = *((t.x & BOX_Y0) ? own : o - rs), yp = *((t.x & BOX_Y1) ? own : o + rs);
      const float4 zm = *((t.x & BOX_Z0) ? own : o - ps), zp = *((t.x & BOX_Z1) ? own : o + ps);
      const float *const xs = reinterpret_cast<const float *>(o);
      const float side = p ? ((t.x & BOX_X1) ? 0.f : xs[4]) : ((t.x & BOX_X0) ? u.x : xs[-1]);
      const float4 xm = p ? x : make_float4(side, x.x, x.y, x.z);
      const float4 xp = p ? make_float4(x.y, x.z, x.w, side) : x;
      const int l = (t.x & BOX_LIQ) ? 1 : 0;
      const float kf = G.bulk[l], ei = G.bulk_ei[l];
      auto upd = [&](float uc, float e, float w, float n, float s, float a, float z, float rhs) {
        return A::relax(uc, e, w, n, s, a, z, kf, kf, kf, kf, kf, kf, ei, rhs, h2, omega);
      };
      const float4 v =
          make_float4(upd(u.x, xp.x, xm.x, yp.x, ym.x, zp.x, zm.x, r.x), upd(u.y, xp.y, xm.y, yp.y, ym.y, zp.y, zm.y, r.y),
                      upd(u.z, xp.z, xm.z, yp.z, ym.z, zp.z, zm.z, r.z), upd(u.w, xp.w, xm.w, yp.w, ym.w, zp.w, zm.w, r.w));
      *own = v;
      if (t.y & 0xFFFFu) post4(out + 2 * (t.y & 0xFFFFu) - 2, far, v, tag);
      if (t.y >> 16) post4(out + 2 * (t.y >> 16) - 2, far, v, tag);
    }
    finish(tid);
    for (int i = tid + B * kBoxThreads; i < 4 * slow; i += B * kBoxThreads) {
      fetch(i);
      finish(i);
    }
  };
  unsigned tag = epoch;
  for (int s = 0; s < G.n; s++)
    for (int col = 0; col < 2; col++) {
      tag++;
      const size_t buf = (tag & 1u) ? per : 0;
      float4 *const V = U + col * half4;
      update(col, 0, slow_f, faces - fast_f, fast_f, mine + buf, tag);
      update(col, faces, slow_i, items - fast_i, fast_i, mine + buf, tag);
      // the neighbours' values, polled for a limited number of tries: if they
      // do not come, the block marks itself dead, waits no more and writes
      // NaN, which the residual norm or the CFL check reports
      unsigned left = 0;
#pragma unroll
      for (int q = 0; q < kBoxHalo; q++)
        if (dst[q] >= 0) left |= 1u << q;
      for (int tries = 0; left; tries++) {
        unsigned long long x[kBoxHalo][4];
#pragma unroll
        for (int q = 0; q < kBoxHalo; q++)
          if (left >> q & 1u) {
            words2(G.mail + src[q] + buf, x[q][0], x[q][1]);
            words2(G.mail + src[q] + buf + far, x[q][2], x[q][3]);
          }
#pragma unroll
        for (int q = 0; q < kBoxHalo; q++)
          if ((left >> q & 1u) && (unsigned)(x[q][0] >> 32) == tag && (unsigned)(x[q][1] >> 32) == tag &&
              (unsigned)(x[q][2] >> 32) == tag && (unsigned)(x[q][3] >> 32) == tag) {
            left &= ~(1u << q);
            V[dst[q]] = make_float4(__uint_as_float((unsigned)x[q][0]), __uint_as_float((unsigned)x[q][1]),
                                    __uint_as_float((unsigned)x[q][2]), __uint_as_float((unsigned)x[q][3]));
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
  // u back
  for (int r = warp; r < ry * np; r += kBoxThreads / 32) {
    const int kl = small_div(r, iry), yl = r - kl * ry, y = ya + yl, k = za + kl, p0 = (y + k) & 1, o = 4 * at4(yl, kl);
    for (int m = lane; m < hx; m += 32) {
      float *p = G.u + node(2 * m, y, k);
      p[0] = bad ? nanf("") : uf[o + m + (p0 ? half : 0)];
      p[1] = bad ? nanf("") : uf[o + m + (p0 ? 0 : half)];
    }
  }
  if (!G.rhs_c) return;
  // the mean residual of each coarse cell's eight cells, and a zero correction
  const int cx = g.nx / 2, cy = ry / 2, n = cx * cy * (np / 2);
  const float icx = 1.0f / cx, icy = 1.0f / cy;
  for (int e = tid; e < n; e += kBoxThreads) {
    const int row = small_div(e, icx), m = e - row * cx, kc = small_div(row, icy), yc = row - kc * cy;
    float r[8];
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const int yl = 2 * yc + (q >> 1 & 1), kl = 2 * kc + (q >> 2), y = ya + yl, k = za + kl, col = (q + y + k) & 1;
      const int o = at4(yl, kl) + (m >> 2);
      const unsigned code = G.flags[(unsigned)(m >> 2) + (unsigned)h4 * ((unsigned)y + (unsigned)g.ny * (unsigned)k)];
      const unsigned t = (unsigned)o | ((y + k) & 1 ? BOX_P : 0) | (m < 4 ? BOX_X0 : 0) | (m >= hx - 4 ? BOX_X1 : 0) |
                         (y == 0 ? BOX_Y0 : 0) | (y == g.ny - 1 ? BOX_Y1 : 0) | (k == 0 ? BOX_Z0 : 0) | (k == g.nz - 1 ? BOX_Z1 : 0);
      float v[7], f[7];
      gather(t, col, m & 3, v);
      if (code)
        f[0] = f[1] = f[2] = f[3] = f[4] = f[5] = G.bulk[code - 1];
      else
        coefs(t, col, m & 3, f);
      r[q] = A::resid(v[0], v[1], v[2], v[3], v[4], v[5], v[6], f[0], f[1], f[2], f[3], f[4], f[5],
                      rf[col * half + 4 * o + (m & 3)], G.h2i);
    }
    const unsigned c = (unsigned)(m + 1) + (unsigned)dc.nx * ((unsigned)(ya / 2 + yc + 1) + (unsigned)dc.ny * (unsigned)(za / 2 + kc + 1));
    G.rhs_c[c] = A::mean8(r[0], r[1], r[2], r[3], r[4], r[5], r[6], r[7]);
    G.u_c[c] = 0.f;
  }
}

#endif  // __CUDACC__

}  // namespace mgg
}  // namespace dsg
