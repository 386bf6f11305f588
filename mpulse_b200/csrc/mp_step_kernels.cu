// mp_step_kernels.cu - the two half-step kernels of one MPulse time step,
// global-load form (mp_step_tma.cu and mp_step_fused.cu hold two opt-in forms).
//
// e_half: FDTD_PLRCSolver::stepScheme's E side (fdtd_plrc.t:129-146) in one
//   pass: the CPML psi_E recursions (CPMLBorderECurrent::stepScheme,
//   cpml_border.cpp:398-425), the TF/SF J plane (incsource.t:40-73, values from
//   mp_source_kernels.cu), the current sum (fdtd_plrc.t:342-374, never
//   materialised), the PLRC recursion and D -> E update of plrcStepD
//   (fdtd_plrc.cpp:94-261, nonlinear :304-427) or of FDTD_Plain / FDTD_Nonlinear
//   (fdtd_plain.cpp:37-77, fdtd_nl.cpp:38-100), and the periodic boundary as an
//   index wrap (periodic_bound.cpp:10-71).
// b_half: the H side (fdtd_plrc.t:148-167): CPML psi_H
//   (cpml_border.cpp:499-527), TF/SF M plane (incsource.t:112-145) and plrcStepB
//   (fdtd_plrc.cpp:263-293).
//
// Thread mapping: V consecutive cells of a row per thread, the columns of a
// plane dealt to warps as row_cells describes, whatever nx and ny are.  A block
// marches up a chunk of z-planes, so that the z-neighbour of the previous plane
// is carried in registers and every field element is read from HBM once per
// half step (x/y neighbours are re-read through L1).  The medium test, the CPML
// z-faces and the injection plane depend on z only and are uniform per plane.  A
// plane's address is uniform too: each access is that address plus a 32-bit
// column offset fixed through the march.
//
// What bounds them.  The stencil has no contraction, so no tensor cores.  On
// grids that exceed L2 both kernels are bound by HBM, on smaller ones by the
// instructions they issue (before this form 541 per 32 cells in the E half and
// 394 in the B half of a 96^3 grid with CPML on all faces, issue slots 68% and
// 60% busy; now 390 and 170), which is why the faces are found from six
// thresholds, rows from a multiplication, and nothing is tested per cell that is
// fixed per thread or per plane.  On large grids the loads of one plane per
// warp do not cover the latency of HBM: the next plane's lines are prefetched
// into L2 while this plane is computed, which needs no registers.
// Measured per half step, before -> after (B200, us):
//   256 x 256 x 512 PLRC + Kerr FP32   E 758 -> 670   B 276 -> 250
//   192 x 192 x 384 PLRC + Kerr FP64   E 659 -> 549   B 225 -> 197
//   150 x 131 x 210 fdtd-plain FP32    E  37 ->  30   B  48 ->  31
//   101 x 75 x 163 fdtd-nl FP64        E  49 ->  23   B  40 ->  17
//   128 x 128 x 192 + plasma FP32      E 135 ->  98   B  56 ->  37
#include "mp_cell.cuh"
#include "mp_pdl.cuh"
#include "mp_row.cuh"

#include <algorithm>

namespace mpb {

// Resident threads per SM asked of the register allocator.  E half: FP32 with
// one cell per thread 1024 (64 registers; 896: 687 instead of 666 us on 256 x 256 x
// 512 run with one cell), with the plasma plug-ins 896 (106 instead of 114 us on 128 x
// 128 x 192),
// with two cells 768 (80 registers); FP64 640 (96 registers; 768 spill: 96
// instead of 87 us with a design region, 120 x 104 x 136).  B half: FP32 1280 (48
// registers; 1024: 264 instead of 257 us on 256 x 256 x 512), with the faces
// loaded early 768 (80 registers; 1024: 263 instead of 250), FP64 768 (640: 205,
// 1024: 206, 768: 198 us on 192 x 192 x 384).
template <typename T>
__host__ __device__ constexpr int e_threads(int V, bool plasma) {
  return sizeof(T) == 8 ? 640 : V == 2 ? 768 : plasma ? 896 : 1024;
}
template <typename T>
__host__ __device__ constexpr int b_threads(bool early) {
  return sizeof(T) == 8 ? 768 : early ? 768 : 1280;
}

// What a half step's grid needs beside the row mapping.
struct HalfGrid : RowMap {
  int kchunk;           // planes per block
  int ahead;            // prefetch the next plane into L2
  // the CPML layers: cells with MPulse index <= lo[a] or >= hi[a] along axis a
  // lie in a layer
  int lo[3], hi[3];
  int src;              // the injection plane (-1: none)
  // there are x / y layers, and no thread's cells reach into both layers of an axis
  bool apart;
};

// Bits of the x faces (slots 2 high, 3 low) at the V cells of a thread, bits 2c
// and 2c + 1, and of the y faces (slots 0 high, 1 low), bits 2V and 2V + 1.
template <int V>
__device__ __forceinline__ unsigned row_face_mask(const HalfGrid &g, int i0, int j) {
  unsigned m = (j + 1 >= g.hi[1] ? 1u << (2 * V) : 0u) | (j + 1 <= g.lo[1] ? 2u << (2 * V) : 0u);
#pragma unroll
  for (int c = 0; c < V; ++c)
    m |= (i0 + c + 1 >= g.hi[0] ? 1u << (2 * c) : 0u) | (i0 + c + 1 <= g.lo[0] ? 2u << (2 * c) : 0u);
  return m;
}

// One CPML face over the V cells of a thread at plane k: psi <- b psi + c d
// for both components, the new psi stored and added to the two current
// components the face feeds (x faces y and z, y faces z and x, z faces x and
// y).  d0, d1: the differences along the face's axis.  ONE: only cell c0 (x
// faces, whose layers begin and end inside a row).
template <typename T, int V, int F>
__device__ __forceinline__ void face_row(const CpmlFace<T> &L, int nx, int ny, int i0, int j, int k, int c0,
                                         const T (&d0)[V], const T (&d1)[V], T (&cur)[V][3], int *st) {
  constexpr int dim = face_axis(F);
  constexpr int u = (dim + 1) % 3, w = (dim + 2) % 3;
  if (dim == 0) {
    const int li = ((k - L.zlo) * ny + j) * L.ex + (i0 + c0 + 1 - L.lo);
    const T b = ld(L.b + i0 + c0 + 1), c = ld(L.c + i0 + c0 + 1);
    const T p0 = fma_pp(b, ld_c(L.psi0, li, L.n, st), c, d0[c0]);
    const T p1 = fma_pp(b, ld_c(L.psi1, li, L.n, st), c, d1[c0]);
    st_c(L.psi0, li, L.n, st, p0);
    st_c(L.psi1, li, L.n, st, p1);
    cur[c0][u] += p0;
    cur[c0][w] += p1;
  } else {
    const int idx = dim == 1 ? j + 1 : k;
    const unsigned li = dim == 1 ? unsigned(((k - L.zlo) * L.ey + (j + 1 - L.lo)) * nx + i0)
                                 : unsigned(((k - L.lo) * ny + j) * nx + i0);
    const T b = ld(L.b + idx), c = ld(L.c + idx);
    RowV<T, V> p0 = ldp<V>(L.psi0, 0, li, L.n, st), p1 = ldp<V>(L.psi1, 0, li, L.n, st);
#pragma unroll
    for (int q = 0; q < V; ++q) {
      p0.v[q] = fma_pp(b, p0.v[q], c, d0[q]);
      p1.v[q] = fma_pp(b, p1.v[q], c, d1[q]);
      cur[q][u] += p0.v[q];
      cur[q][w] += p1.v[q];
    }
    stp<V>(L.psi0, 0, li, L.n, st, p0);
    stp<V>(L.psi1, 0, li, L.n, st, p1);
  }
}

// All faces containing the cells of a thread, in MPulse's order (slots 0..5):
// the differences along y, x and z of the components the faces take, with the
// sign of the side.
template <typename T, int V>
__device__ __forceinline__ void face_currents(const CpmlFace<T> (&cpml)[6], int nx, int ny, unsigned mask, bool zlow,
                                              bool zhigh, int i0, int j, int k, const T (&dy0)[V], const T (&dy1)[V],
                                              const T (&dx0)[V], const T (&dx1)[V], const T (&dz0)[V],
                                              const T (&dz1)[V], T (&cur)[V][3], int *st) {
  if (mask) {
    if (mask & (1u << (2 * V))) face_row<T, V, 0>(cpml[0], nx, ny, i0, j, k, 0, dy0, dy1, cur, st);
    if (mask & (2u << (2 * V))) face_row<T, V, 1>(cpml[1], nx, ny, i0, j, k, 0, dy0, dy1, cur, st);
#pragma unroll
    for (int c = 0; c < V; ++c) {
      if (mask & (1u << (2 * c))) face_row<T, V, 2>(cpml[2], nx, ny, i0, j, k, c, dx0, dx1, cur, st);
      if (mask & (2u << (2 * c))) face_row<T, V, 3>(cpml[3], nx, ny, i0, j, k, c, dx0, dx1, cur, st);
    }
  }
  if (zhigh) face_row<T, V, 4>(cpml[4], nx, ny, i0, j, k, 0, dz0, dz1, cur, st);
  if (zlow) face_row<T, V, 5>(cpml[5], nx, ny, i0, j, k, 0, dz0, dz1, cur, st);
}

// The same for grids whose layers lie apart (HalfGrid::apart: a thread's cells
// are in at most one face per axis), in two parts: load_faces asks for the psi
// and coefficients of all faces of the plane beside the plane's other loads, so
// that a face costs no memory latency of its own; add_faces then does the rest,
// in the same order.  face_currents waits once per face, and a warp with x-face
// cells does so on every plane.  B half with CPML on all faces (FP32, us): 96^3
// 18.8 -> 14.1, 128 x 128 x 192 44 -> 37, 128 x 128 x 256 54 -> 45, 256 x 256 x 512
// 260 -> 250; E half 128 x 128 x 256 Kerr 107 -> 102, 101 x 131 x 120 with two poles
// 49 -> 43, FP64 120 x 104 x 136 87 -> 82.  Grids
// without x / y layers keep face_currents, which needs fewer registers (160 x 144
// x 250 with z layers, B half 44 us; with the early loads 50), and so do grids
// whose layers meet.
template <typename T, int V>
struct FaceRows {
  RowV<T, V> y0, y1, z0, z1;
  T x0[V], x1[V];
  T by, cy, bz, cz, bx[V], cx[V];
  unsigned ly, lz;
  int lx;
};

template <typename T, int V>
__device__ __forceinline__ void load_faces(const CpmlFace<T> (&cpml)[6], int nx, int ny, unsigned mask, bool zlow,
                                           bool zhigh, int i0, int j, int k, FaceRows<T, V> &f, int *st) {
  constexpr unsigned kX = (1u << (2 * V)) - 1u;
  if (mask) {
    if (mask & ~kX) {
      const CpmlFace<T> &L = cpml[(mask >> (2 * V)) & 1u ? 0 : 1];
      f.ly = unsigned(((k - L.zlo) * L.ey + (j + 1 - L.lo)) * nx + i0);
      f.by = ld(L.b + j + 1);
      f.cy = ld(L.c + j + 1);
      f.y0 = ldp<V>(L.psi0, 0, f.ly, L.n, st);
      f.y1 = ldp<V>(L.psi1, 0, f.ly, L.n, st);
    }
    if (mask & kX) {
      const CpmlFace<T> &L = cpml[mask & (0x55555555u & kX) ? 2 : 3];
      f.lx = ((k - L.zlo) * ny + j) * L.ex + (i0 + 1 - L.lo);
#pragma unroll
      for (int c = 0; c < V; ++c)
        if (mask & (3u << (2 * c))) {
          f.bx[c] = ld(L.b + i0 + c + 1);
          f.cx[c] = ld(L.c + i0 + c + 1);
          f.x0[c] = ld_c(L.psi0, f.lx + c, L.n, st);
          f.x1[c] = ld_c(L.psi1, f.lx + c, L.n, st);
        }
    }
  }
  if (zlow || zhigh) {
    const CpmlFace<T> &L = cpml[zhigh ? 4 : 5];
    f.lz = unsigned(((k - L.lo) * ny + j) * nx + i0);
    f.bz = ld(L.b + k);
    f.cz = ld(L.c + k);
    f.z0 = ldp<V>(L.psi0, 0, f.lz, L.n, st);
    f.z1 = ldp<V>(L.psi1, 0, f.lz, L.n, st);
  }
}

template <typename T, int V>
__device__ __forceinline__ void add_faces(const CpmlFace<T> (&cpml)[6], unsigned mask, bool zlow, bool zhigh,
                                          FaceRows<T, V> &f, const T (&dy0)[V], const T (&dy1)[V], const T (&dx0)[V],
                                          const T (&dx1)[V], const T (&dz0)[V], const T (&dz1)[V], T (&cur)[V][3],
                                          int *st) {
  constexpr unsigned kX = (1u << (2 * V)) - 1u;
  if (mask) {
    if (mask & ~kX) {
      const CpmlFace<T> &L = cpml[(mask >> (2 * V)) & 1u ? 0 : 1];
#pragma unroll
      for (int c = 0; c < V; ++c) {
        f.y0.v[c] = fma_pp(f.by, f.y0.v[c], f.cy, dy0[c]);
        f.y1.v[c] = fma_pp(f.by, f.y1.v[c], f.cy, dy1[c]);
        cur[c][2] += f.y0.v[c];
        cur[c][0] += f.y1.v[c];
      }
      stp<V>(L.psi0, 0, f.ly, L.n, st, f.y0);
      stp<V>(L.psi1, 0, f.ly, L.n, st, f.y1);
    }
    if (mask & kX) {
      const CpmlFace<T> &L = cpml[mask & (0x55555555u & kX) ? 2 : 3];
#pragma unroll
      for (int c = 0; c < V; ++c)
        if (mask & (3u << (2 * c))) {
          const T p0 = fma_pp(f.bx[c], f.x0[c], f.cx[c], dx0[c]);
          const T p1 = fma_pp(f.bx[c], f.x1[c], f.cx[c], dx1[c]);
          st_c(L.psi0, f.lx + c, L.n, st, p0);
          st_c(L.psi1, f.lx + c, L.n, st, p1);
          cur[c][1] += p0;
          cur[c][2] += p1;
        }
    }
  }
  if (zlow || zhigh) {
    const CpmlFace<T> &L = cpml[zhigh ? 4 : 5];
#pragma unroll
    for (int c = 0; c < V; ++c) {
      f.z0.v[c] = fma_pp(f.bz, f.z0.v[c], f.cz, dz0[c]);
      f.z1.v[c] = fma_pp(f.bz, f.z1.v[c], f.cz, dz1[c]);
      cur[c][0] += f.z0.v[c];
      cur[c][1] += f.z1.v[c];
    }
    stp<V>(L.psi0, 0, f.lz, L.n, st, f.z0);
    stp<V>(L.psi1, 0, f.lz, L.n, st, f.z1);
  }
}

// The injection plane's currents of the V cells.
template <typename T, int V, typename P>
__device__ __forceinline__ void source_currents(const P &p, unsigned col, T (&cur)[V][3]) {
  const RowV<T, V> a = ldp<V>(p.src[0].v0, 0, col, p.plane, p.status);
  const RowV<T, V> b = ldp<V>(p.src[0].v1, 0, col, p.plane, p.status);
#pragma unroll
  for (int c = 0; c < V; ++c)
    for (int q = 0; q < p.src_mult; ++q) {
      cur[c][0] += a.v[c];
      cur[c][1] += b.v[c];
    }
}

// Whether the adjoint history of cell (i, j, k) is stored (EParams::hist_box).
template <typename T>
__device__ __forceinline__ bool hist_cell(const EParams<T> &p, int i, int j, int k) {
  if (p.hist_all) return true;
#pragma unroll
  for (int b = 0; b < 2; ++b) {
    const int *h = p.hist_box[b];
    if (i >= h[0] && i <= h[1] && j >= h[2] && j <= h[3] && k >= h[4] && k <= h[5]) return true;
  }
  return false;
}

template <typename T, int V, int MODE, int NP, bool DESIGN, bool PLASMA, bool EARLY>
__global__ void __launch_bounds__(kRowThreads, e_threads<T>(V, PLASMA) / kRowThreads)
    e_half_kernel(const EParams<T> p, const HalfGrid g) {
  typedef typename Vec2<T>::type T2;
  constexpr bool PLRC = MODE == MODE_PLRC_LIN || MODE == MODE_PLRC_NONLIN;
  const int nx = p.nx, ny = p.ny;
  int i0, j;  // 0-based: MPulse i + 1, j + 1
  if (!row_cells<V>(g, blockIdx.x, ny, i0, j)) return;
  const int k0 = p.k_first + blockIdx.y * g.kchunk;
  const int k1 = min(k0 + g.kchunk - 1, p.k_last);
  const long long plane = p.plane;
  const unsigned row = unsigned(j) * unsigned(nx);
  const unsigned col = row + i0;
  const unsigned colxm = row + (i0 == 0 ? nx - 1 : i0 - 1);  // x-1 of the first cell
  const unsigned colym = (j == 0 ? unsigned(plane) : row) - nx + i0;
  const T *Bx = p.B[0], *By = p.B[1], *Bz = p.B[2];
  T *Ex = p.E[0], *Ey = p.E[1], *Ez = p.E[2];
  RowV<T, V> ikx;
#pragma unroll
  for (int c = 0; c < V; ++c) ikx.v[c] = ld(p.ik[0] + i0 + c + 1);
  const T iky = ld(p.ik[1] + j + 1);
  const unsigned fmask = PLRC ? row_face_mask<V>(g, i0, j) : 0u;
  const long long nf = p.n_field;
  int *const st = p.status;
  KerrCount kc;
  pdl_wait();

  const int km = p.zperiodic && k0 == 1 ? p.nz : k0 - 1;
  RowV<T, V> bx_km = ldp<V>(Bx, km * plane, col, nf, st), by_km = ldp<V>(By, km * plane, col, nf, st);
  for (int k = k0; k <= k1; ++k) {
    const long long base = (long long)k * plane;
    // ---- every load of this plane first
    const RowV<T, V> bx = ldp<V>(Bx, base, col, nf, st), by = ldp<V>(By, base, col, nf, st),
                     bz = ldp<V>(Bz, base, col, nf, st);
    const RowV<T, V> bz_ym = ldp<V>(Bz, base, colym, nf, st), bx_ym = ldp<V>(Bx, base, colym, nf, st);
    const RowV<T, 1> bz_xl = ldp<1>(Bz, base, colxm, nf, st), by_xl = ldp<1>(By, base, colxm, nf, st);
    const RowV<T, V> ex = ldp<V>(Ex, base, col, nf, st), ey = ldp<V>(Ey, base, col, nf, st),
                     ez = ldp<V>(Ez, base, col, nf, st);
    const bool med = PLRC && k >= p.mz0 && k <= p.mz1;
    const long long pbase = (long long)(k - p.mz0) * plane;
    RowV<T2, V> q[NP > 0 ? NP : 1][3];
    if (NP > 0 && med) {
#pragma unroll
      for (int n = 0; n < NP; ++n)
#pragma unroll
        for (int c = 0; c < 3; ++c)
          q[n][c] = ldp<V>(reinterpret_cast<const T2 *>(p.psi[n][c]), pbase, col, p.n_psi, st);
    }
    RowV<T, V> rho, j0 = {}, j1 = {}, j2 = {};
    if (PLASMA) {
      rho = ldp<V>(p.rho, base, col, nf, st);
      if (p.pl_current) {
        j0 = ldp<V>(p.pj[0], base, col, nf, st);
        j1 = ldp<V>(p.pj[1], base, col, nf, st);
        j2 = ldp<V>(p.pj[2], base, col, nf, st);
      }
    }
    const T ikz = ld(p.ik[2] + k);
    const bool zlow = PLRC && k <= g.lo[2], zhigh = PLRC && k >= g.hi[2];
    FaceRows<T, V> fr;
    if (PLRC && EARLY) load_faces<T, V>(p.cpml, nx, ny, fmask, zlow, zhigh, i0, j, k, fr, st);
    if (g.ahead && k < k1) {
      const long long ba = base + plane;
      prefetch_l2(Bx + ba + col);
      prefetch_l2(By + ba + col);
      prefetch_l2(Bz + ba + col);
      prefetch_l2(Ex + ba + col);
      prefetch_l2(Ey + ba + col);
      prefetch_l2(Ez + ba + col);
      if (NP > 0 && med && k < p.mz1) {
#pragma unroll
        for (int n = 0; n < NP; ++n)
#pragma unroll
          for (int c = 0; c < 3; ++c)
            prefetch_l2(reinterpret_cast<const T2 *>(p.psi[n][c]) + pbase + plane + col);
      }
    }

    // ---- the differences of B, then the E-side currents in MPulse's order
    T dzy[V], dyz[V], dxz[V], dzx[V], dyx[V], dxy[V];  // d<component><axis>
#pragma unroll
    for (int c = 0; c < V; ++c) {
      dzy[c] = bz.v[c] - bz_ym.v[c];
      dxy[c] = bx.v[c] - bx_ym.v[c];
      dzx[c] = bz.v[c] - (c ? bz.v[c ? c - 1 : 0] : bz_xl.v[0]);
      dyx[c] = by.v[c] - (c ? by.v[c ? c - 1 : 0] : by_xl.v[0]);
      dxz[c] = bx.v[c] - bx_km.v[c];
      dyz[c] = by.v[c] - by_km.v[c];
    }
    T cur[V][3];
#pragma unroll
    for (int c = 0; c < V; ++c) cur[c][0] = cur[c][1] = cur[c][2] = T(0);
    if (PLRC) {
      if (fmask || zlow || zhigh) {
        T nxy[V], nzx[V], nyz[V];
#pragma unroll
        for (int c = 0; c < V; ++c) {
          nxy[c] = -dxy[c];
          nzx[c] = -dzx[c];
          nyz[c] = -dyz[c];
        }
        if (EARLY)
          add_faces<T, V>(p.cpml, fmask, zlow, zhigh, fr, nxy, dzy, nzx, dyx, nyz, dxz, cur, st);
        else
          face_currents<T, V>(p.cpml, nx, ny, fmask, zlow, zhigh, i0, j, k, nxy, dzy, nzx, dyx, nyz, dxz, cur, st);
      }
      if (k == g.src) source_currents<T, V>(p, col, cur);
    }

    // ---- the E update, cell by cell
    RowV<T, V> exn, eyn, ezn;
#pragma unroll
    for (int c = 0; c < V; ++c) {
      CellCoef<T, NP> lc;
      cell_coef<T, NP, DESIGN>(p, i0 + c, j, k, med, lc);
      PlasmaCell<T> pc;
      if (PLASMA) {
        plasma_cell(p, ex.v[c], ey.v[c], ez.v[c], rho.v[c], j0.v[c], j1.v[c], j2.v[c], pc);
        if (med && p.pl_density) plasma_coef(p, pc.sig, lc);
        rho.v[c] = pc.rho;
        j0.v[c] = pc.j[0];
        j1.v[c] = pc.j[1];
        j2.v[c] = pc.j[2];
        // the plasma current, after the other currents
        cur[c][0] += pc.j[0];
        cur[c][1] += pc.j[1];
        cur[c][2] += pc.j[2];
      }
      // curl_kappa B (fdtd_plrc.cpp:207-244)
      const T cbx = fma_pm(dzy[c], iky, dyz[c], ikz);
      const T cby = fma_pm(dxz[c], ikz, dzx[c], ikx.v[c]);
      const T cbz = fma_pm(dyx[c], ikx.v[c], dxy[c], iky);
      T2 qc[NP > 0 ? NP : 1][3];
#pragma unroll
      for (int n = 0; n < NP; ++n)
#pragma unroll
        for (int a = 0; a < 3; ++a) qc[n][a] = q[n][a].v[c];
      e_update<T, MODE, NP, PLASMA>(p, lc, med, ex.v[c], ey.v[c], ez.v[c], cbx, cby, cbz, cur[c][0], cur[c][1],
                                    cur[c][2], qc, exn.v[c], eyn.v[c], ezn.v[c], kc, &pc);
#pragma unroll
      for (int n = 0; n < NP; ++n)
#pragma unroll
        for (int a = 0; a < 3; ++a) q[n][a].v[c] = qc[n][a];
    }
    // ---- stores
    stp<V>(Ex, base, col, nf, st, exn);
    stp<V>(Ey, base, col, nf, st, eyn);
    stp<V>(Ez, base, col, nf, st, ezn);
    if (PLASMA) {
      stp<V>(p.rho, base, col, nf, st, rho);
      if (p.pl_current) {
        stp<V>(p.pj[0], base, col, nf, st, j0);
        stp<V>(p.pj[1], base, col, nf, st, j1);
        stp<V>(p.pj[2], base, col, nf, st, j2);
      }
    }
    if (DESIGN && p.hist[0]) {
#pragma unroll
      for (int c = 0; c < V; ++c)
        if (hist_cell(p, i0 + c, j, k)) {
          st_c(p.hist[0], base + col + c, nf, st, exn.v[c]);
          st_c(p.hist[1], base + col + c, nf, st, eyn.v[c]);
          st_c(p.hist[2], base + col + c, nf, st, ezn.v[c]);
        }
    }
    if (NP > 0 && med) {
#pragma unroll
      for (int n = 0; n < NP; ++n)
#pragma unroll
        for (int c = 0; c < 3; ++c) stp<V>(reinterpret_cast<T2 *>(p.psi[n][c]), pbase, col, p.n_psi, st, q[n][c]);
    }
    bx_km = bx;
    by_km = by;
  }
  pdl_launch_dependents();
  flush_kerr_count<MODE>(p.kerr_count, kc);
}

template <typename T, int V, bool EARLY>
__global__ void __launch_bounds__(kRowThreads, b_threads<T>(EARLY) / kRowThreads)
    b_half_kernel(const BParams<T> p, const HalfGrid g) {
  // the chunks from the top down: the E half wrote the top planes last, and
  // what of them is still in L2 is read from there (2-6% of both halves on grids
  // of up to twice the L2)
  const int nx = p.nx, ny = p.ny;
  int i0, j;
  if (!row_cells<V>(g, blockIdx.x, ny, i0, j)) return;
  const int k0 = p.k_first + (gridDim.y - 1 - blockIdx.y) * g.kchunk;
  const int k1 = min(k0 + g.kchunk - 1, p.k_last);
  const long long plane = p.plane;
  const unsigned row = unsigned(j) * unsigned(nx);
  const unsigned col = row + i0;
  const unsigned colxp = row + (i0 + V == nx ? 0 : i0 + V);  // x+1 of the last cell
  const unsigned colyp = (j == ny - 1 ? 0u : row + nx) + i0;
  const T *Ex = p.E[0], *Ey = p.E[1], *Ez = p.E[2];
  T *Bx = p.B[0], *By = p.B[1], *Bz = p.B[2];
  RowV<T, V> ikx;
#pragma unroll
  for (int c = 0; c < V; ++c) ikx.v[c] = ld(p.ik[0] + i0 + c + 1);
  const T iky = ld(p.ik[1] + j + 1);
  const T iky_bz = ld(p.ik_bz_y + j + 1);
  const unsigned fmask = row_face_mask<V>(g, i0, j);
  const long long nf = p.n_field;
  int *const st = p.status;
  pdl_wait();

  RowV<T, V> ex = ldp<V>(Ex, k0 * plane, col, nf, st), ey = ldp<V>(Ey, k0 * plane, col, nf, st);
  for (int k = k0; k <= k1; ++k) {
    const long long base = (long long)k * plane;
    const long long basep = (p.zperiodic && k == p.nz ? 1 : k + 1) * plane;
    // ---- every load of this plane first
    const RowV<T, V> ex_kp = ldp<V>(Ex, basep, col, nf, st), ey_kp = ldp<V>(Ey, basep, col, nf, st);
    const RowV<T, V> ez = ldp<V>(Ez, base, col, nf, st);
    const RowV<T, V> bx = ldp<V>(Bx, base, col, nf, st), by = ldp<V>(By, base, col, nf, st),
                     bz = ldp<V>(Bz, base, col, nf, st);
    const RowV<T, V> ez_yp = ldp<V>(Ez, base, colyp, nf, st), ex_yp = ldp<V>(Ex, base, colyp, nf, st);
    const RowV<T, 1> ez_xl = ldp<1>(Ez, base, colxp, nf, st), ey_xl = ldp<1>(Ey, base, colxp, nf, st);
    const T ikz = ld(p.ik[2] + k);
    const bool zlow = k <= g.lo[2], zhigh = k >= g.hi[2];
    FaceRows<T, V> fr;
    if (EARLY) load_faces<T, V>(p.cpml, nx, ny, fmask, zlow, zhigh, i0, j, k, fr, st);
    if (g.ahead && k < k1) {
      const long long ba = base + plane;
      prefetch_l2(Bx + ba + col);
      prefetch_l2(By + ba + col);
      prefetch_l2(Bz + ba + col);
      prefetch_l2(Ex + ba + plane + col);
      prefetch_l2(Ey + ba + plane + col);
      prefetch_l2(Ez + ba + col);
    }

    // ---- the differences of E, then the H-side currents in MPulse's order
    T dzy[V], dyz[V], dxz[V], dzx[V], dyx[V], dxy[V];  // d<component><axis>
#pragma unroll
    for (int c = 0; c < V; ++c) {
      dzy[c] = ez_yp.v[c] - ez.v[c];
      dxy[c] = ex_yp.v[c] - ex.v[c];
      dzx[c] = (c + 1 < V ? ez.v[c + 1 < V ? c + 1 : 0] : ez_xl.v[0]) - ez.v[c];
      dyx[c] = (c + 1 < V ? ey.v[c + 1 < V ? c + 1 : 0] : ey_xl.v[0]) - ey.v[c];
      dxz[c] = ex_kp.v[c] - ex.v[c];
      dyz[c] = ey_kp.v[c] - ey.v[c];
    }
    T cur[V][3];
#pragma unroll
    for (int c = 0; c < V; ++c) cur[c][0] = cur[c][1] = cur[c][2] = T(0);
    if (fmask || zlow || zhigh) {
      T nzy[V], nyx[V], nxz[V];
#pragma unroll
      for (int c = 0; c < V; ++c) {
        nzy[c] = -dzy[c];
        nyx[c] = -dyx[c];
        nxz[c] = -dxz[c];
      }
      if (EARLY)
        add_faces<T, V>(p.cpml, fmask, zlow, zhigh, fr, dxy, nzy, dzx, nyx, dyz, nxz, cur, st);
      else
        face_currents<T, V>(p.cpml, nx, ny, fmask, zlow, zhigh, i0, j, k, dxy, nzy, dzx, nyx, dyz, nxz, cur, st);
    }
    if (k == g.src) source_currents<T, V>(p, col, cur);

    // ---- plrcStepB (fdtd_plrc.cpp:263-293)
    RowV<T, V> bxn, byn, bzn;
#pragma unroll
    for (int c = 0; c < V; ++c) {
      bxn.v[c] = add_dt(bx.v[c], p.dt, p.dt_lo, fma_pm(dyz[c], ikz, dzy[c], iky) + cur[c][0]);
      byn.v[c] = add_dt(by.v[c], p.dt, p.dt_lo, fma_pm(dzx[c], ikx.v[c], dxz[c], ikz) + cur[c][1]);
      bzn.v[c] = add_dt(bz.v[c], p.dt, p.dt_lo, fma_pm(dxy[c], iky_bz, dyx[c], ikx.v[c]) + cur[c][2]);
    }
    stp<V>(Bx, base, col, nf, st, bxn);
    stp<V>(By, base, col, nf, st, byn);
    stp<V>(Bz, base, col, nf, st, bzn);
    ex = ex_kp;
    ey = ey_kp;
  }
  pdl_launch_dependents();
}

// ---------------------------------------------------------------------------
// Launchers (called from mp_api.cu)

template <typename P>
static bool xy_faces(const P &p) {
  return p.cpml[0].active || p.cpml[1].active || p.cpml[2].active || p.cpml[3].active;
}

// The grid of a half step: V cells per thread, z-chunks of the planes.
// Planes per block: one where two would leave SMs without four blocks (32^3
// FP64: E 9.1 instead of 10.2 us; 72^3 12.2 instead of 13.1 us a step); else at least
// two, and more while 50 blocks per SM remain, up to max_planes.  Longer chunks save the two carried loads of
// each chunk's first plane but leave fewer warps and a longer tail (256 x 256 x
// 512 FP32 E half, one cell per thread, with 2 / 4 / 8 / 16 / 24 planes 725 / 682 /
// 677 / 700 / 715 us, 128 x 128 x 256 112 / 107 / 112 us with 2 / 4 / 8).  The prefetch
// is for states that do not stay in L2 (126 MB): 256 x 256 x 512 E half, one cell, 748
// -> 677 us, 120 x 104 x 136 FP64 93 -> 89; on a 99 MB state 29.8 -> 31.5.
template <typename P>
static HalfGrid row_grid(const P &p, int V, int max_planes, dim3 *d) {
  HalfGrid r;
  static_cast<RowMap &>(r) = row_map(p.nx, p.ny, V);
  const int axis_high[3] = {2, 0, 4};  // the slot of the high face; the low one follows
  for (int a = 0; a < 3; ++a) {
    const auto &H = p.cpml[axis_high[a]], &L = p.cpml[axis_high[a] + 1];
    r.hi[a] = H.active ? H.lo : 1 << 30;
    r.lo[a] = L.active ? L.hi : -1;
  }
  r.apart = xy_faces(p) && r.hi[0] - r.lo[0] > V && r.hi[1] > r.lo[1] && r.hi[2] > r.lo[2];
  r.src = p.n_src > 0 ? p.src[0].plane : -1;
  const int nk = p.k_last - p.k_first + 1;
  const long long bxy = (r.nvec + 31) / 32, all = bxy * nk;
  r.kchunk = all < 1600 ? 1 : int(std::min<long long>(std::max(2LL, all / (148 * 50)), max_planes));
  r.kchunk = std::max(r.kchunk, (nk + 65534) / 65535);  // blocks in y
  r.ahead = p.state_bytes > (160LL << 20);
  *d = dim3(unsigned(bxy), unsigned((nk + r.kchunk - 1) / r.kchunk), 1);
  return r;
}

// (Both kernels go out with programmatic dependent launch: 32^3 FP64 6.0 -> 3.6
// us per step, 64^3 FP32 9.1 -> 5.8.)
template <typename T>
constexpr int max_planes() {
  return sizeof(T) == 4 ? 8 : 4;
}

template <typename T, int V, int MODE, bool DESIGN, bool PLASMA, bool EARLY>
static cudaError_t launch_e_np(const EParams<T> &p, int np, const HalfGrid &g, dim3 d, cudaStream_t st) {
  constexpr bool PLRC = MODE == MODE_PLRC_LIN || MODE == MODE_PLRC_NONLIN;
  // the most poles launch_e sends here
  constexpr int most = !PLRC ? 0 : V == 1 ? 3 : MODE == MODE_PLRC_NONLIN ? 2 : EARLY ? 1 : 3;
  const dim3 b(kRowThreads, 1, 1);
  if (np > most) return cudaErrorInvalidValue;
  switch (np) {
    case 0: return launch_pdl(e_half_kernel<T, V, MODE, 0, DESIGN, PLASMA, EARLY>, d, b, st, p, g);
    case 1: return launch_pdl(e_half_kernel<T, V, MODE, std::min(1, most), DESIGN, PLASMA, EARLY>, d, b, st, p, g);
    case 2: return launch_pdl(e_half_kernel<T, V, MODE, std::min(2, most), DESIGN, PLASMA, EARLY>, d, b, st, p, g);
    default: return launch_pdl(e_half_kernel<T, V, MODE, most, DESIGN, PLASMA, EARLY>, d, b, st, p, g);
  }
}

template <typename T, int V, int MODE, bool DESIGN, bool PLASMA>
static cudaError_t launch_e_v(const EParams<T> &p, int np, cudaStream_t st) {
  constexpr bool PLRC = MODE == MODE_PLRC_LIN || MODE == MODE_PLRC_NONLIN;
  dim3 d;
  const HalfGrid g = row_grid(p, V, max_planes<T>(), &d);
  constexpr bool EARLY = PLRC && !(MODE == MODE_PLRC_NONLIN && V == 2);
  return EARLY && g.apart ? launch_e_np<T, V, MODE, DESIGN, PLASMA, EARLY>(p, np, g, d, st)
                         : launch_e_np<T, V, MODE, DESIGN, PLASMA, false>(p, np, g, d, st);
}

// Two cells per thread in FP32 where the update is short (150 x 131 x 210
// fdtd-plain 30 instead of 38 us, 160 x 144 x 250 PLRC with one pole 79 instead
// of 81, 128^3 with two poles 46 instead of 49), but not with two poles and x / y
// layers (160 x 144 x 250 124 us with one cell, 141 with two); one with the plasma
// plug-ins (128 x 128 x 192 109 instead of 116), with a design region (96^3 21.6
// instead of 23.0) and in FP64, whose two-cell form spills (192 x 192 x 384 551
// instead of 691 us).
// Kerr: two cells issue 27% fewer instructions (256 x 256 x 320 223 instead of 307 M),
// which counts where the GPU works at its power limit, but lack the registers for the early face loads (827 us
// with them on 256 x 256 x 512) and, with three poles, for the update itself (52
// bytes spilled).  So states above 1 GB take two unless they have three poles, or x /
// y layers in rows of less than 192 cells.  Us a step, one cell -> two, 64 steps / a
// second of steps on end:
//   two poles, x / y layers  256 x 256 x 512 917 -> 919 / 945 -> 934, 384 x 384 x 320
//     1282 -> 1272 / 1318 -> 1294, 256 x 256 x 256 481 -> 484 / 493 -> 492, 192 x 192 x
//     512 536 -> 540 / 569 -> 568, 160 x 160 x 740 546 -> 569 / 571 -> 586, 128 x 128 x
//     1100 521 -> 527 / 527 -> 534
//   two poles, z layers      256 x 256 x 280 477 -> 469 / 496 -> 483, 128 x 128 x 1100
//     454 -> 446 / 461 -> 451
//   three poles              256 x 256 x 400 927 -> 945 / 947 -> 959, 256 x 256 x 220 with
//     z layers 478 -> 499 / 488 -> 504
//   one pole                 256 x 256 x 400 584 -> 574 / 644 -> 622, 192 x 192 x 760 618 ->
//     625 / 703 -> 688, 128 x 128 x 1700 631 -> 659 / 649 -> 670
//   none                     256 x 256 x 640 711 -> 657 / 795 -> 740
// Below, one cell: 128 x 128 x 256 with two poles 147 -> 156 / 137 -> 144, 192 x 192 x
// 256 284 -> 281 / 289 -> 289, 256 x 256 x 128 260 -> 255 / 262 -> 257.
template <typename T, int MODE, bool DESIGN, bool PLASMA>
static cudaError_t launch_e(const EParams<T> &p, int np, cudaStream_t st) {
  constexpr int V = sizeof(T) == 4 && !DESIGN && !PLASMA ? 2 : 1;
  const bool kerr_two = np <= 2 && p.state_bytes > (1LL << 30) && (!xy_faces(p) || p.nx >= 192);
  const bool two =
      p.nx % V == 0 && p.nx > V && (MODE == MODE_PLRC_NONLIN ? kerr_two : !(np >= 2 && xy_faces(p)));
  return two ? launch_e_v<T, V, MODE, DESIGN, PLASMA>(p, np, st) : launch_e_v<T, 1, MODE, DESIGN, PLASMA>(p, np, st);
}

template <typename T>
cudaError_t launch_e_half(const EParams<T> &p, int mode, int np, cudaStream_t st) {
  // design regions and the plasma plug-ins exist only with the PLRC solvers
  // (and not together)
  const bool design = p.design.x0 <= p.design.x1;
  const bool plasma = p.rho != nullptr;
  switch (mode) {
    case MODE_PLAIN: return launch_e<T, MODE_PLAIN, false, false>(p, 0, st);
    case MODE_NL: return launch_e<T, MODE_NL, false, false>(p, 0, st);
    case MODE_PLRC_LIN:
      return design   ? launch_e<T, MODE_PLRC_LIN, true, false>(p, np, st)
             : plasma ? launch_e<T, MODE_PLRC_LIN, false, true>(p, np, st)
                      : launch_e<T, MODE_PLRC_LIN, false, false>(p, np, st);
    default:
      return design   ? launch_e<T, MODE_PLRC_NONLIN, true, false>(p, np, st)
             : plasma ? launch_e<T, MODE_PLRC_NONLIN, false, true>(p, np, st)
                      : launch_e<T, MODE_PLRC_NONLIN, false, false>(p, np, st);
  }
}

template <typename T, int V>
static cudaError_t launch_b_v(const BParams<T> &p, cudaStream_t st) {
  dim3 d;
  const HalfGrid g = row_grid(p, V, max_planes<T>(), &d);
  // early loads in FP32 only (FP64: 120 x 104 x 136 38 us either way, 192 x 192 x
  // 384 220 instead of 200)
  constexpr bool EARLY = sizeof(T) == 4;
  return g.apart ? launch_pdl(b_half_kernel<T, V, EARLY>, d, dim3(kRowThreads, 1, 1), st, p, g)
                 : launch_pdl(b_half_kernel<T, V, false>, d, dim3(kRowThreads, 1, 1), st, p, g);
}

// Two cells per thread in FP32 (256 x 256 x 512: 257 us, one cell 293, four
// 338), one in FP64 (192 x 192 x 384: 198 us, two cells 217).
template <typename T>
cudaError_t launch_b_half(const BParams<T> &p, cudaStream_t st) {
  constexpr int V = sizeof(T) == 4 ? 2 : 1;
  return p.nx % V == 0 && p.nx > V ? launch_b_v<T, V>(p, st) : launch_b_v<T, 1>(p, st);
}

template cudaError_t launch_e_half<float>(const EParams<float> &, int, int, cudaStream_t);
template cudaError_t launch_e_half<double>(const EParams<double> &, int, int, cudaStream_t);
template cudaError_t launch_b_half<float>(const BParams<float> &, cudaStream_t);
template cudaError_t launch_b_half<double>(const BParams<double> &, cudaStream_t);

}  // namespace mpb
