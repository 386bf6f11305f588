// mp_adjoint_kernels.cu - the discrete adjoint of one PLRC step and the
// objective kernels of mp_objective / mp_adjoint.
//
// The forward step (mp_step_kernels.cu) maps the state (E, B, PLRC
// accumulators psi, CPML psi) of step n to that of step n+1:
//   E half  psiE' = b psiE + c d(B);  X = (numer + chi|E|^2) E + dt (curl_E B +
//           J) + Re sum psi~;  E' = X / denom (linear) or the Kerr solve
//           |E'| + A |E'|^3 = |X / denom| along X (nonlinear);
//           psi' = s dxi0 E + Crec psi~, psi~ = s (dchi0 - dxi0) E + psi;
//   B half  psiH' = b psiH + c d(E');  B' = B + dt (curl_H E' + M).
// Its adjoint runs the two halves backwards.  The adjoint of a CPML psi is
// carried as a "total" (its own adjoint after the half plus dt times the
// adjoint of the component it feeds), so that every kernel writes only its
// own cell:
//   adj_e_kernel (E cells, planes 1..nz)  gathers the adjoint of E' from the
//     adjoint of B' through the transposed curl_H and the H-face totals, then
//     undoes the E half locally (linearised Kerr, reverse PLRC recursion),
//     accumulates the design gradients, stores the numerator adjoint G and
//     advances its E-face totals;
//   adj_b_kernel (B cells, planes 0..nz)  gathers the adjoint of B from G
//     through the transposed curl_E and the E-face totals, adds the
//     objective's B term and advances its H-face totals;
//   the design gradients of the step (design cells only), accumulated from
//     G, E before and after the step and the PLRC accumulator adjoints adj_e
//     saved for the design cells, by extra blocks of the adj_b launch, so
//     that adj_e, which every cell runs, carries none of the FP64 gradient
//     arithmetic.
// The kernels of the reverse pass are launched with programmatic dependent
// launch: a kernel's blocks may start while the previous kernel's last blocks
// run, do their set-up, and wait (griddepcontrol.wait) for the previous
// kernel's writes before reading anything it produced.
// The Kerr linearisation and the gradient accumulation are FP64; the rest is
// in the precision of the forward state.  Latency-bound at small grids; one
// thread per (x, y) column and chunk of planes.
#include "mp_cell.cuh"
#include "mp_device.h"
#include "mp_pdl.cuh"
#include "mp_row.cuh"

#include <algorithm>

#include <cuda_runtime.h>

namespace mpb {

// Resident threads per SM asked of the register allocator: adj_e FP32 768 (512 /
// 640 / 896 / 1024: the 96^3 reverse step 1.09 / 1.05 / 1.03 / 1.17 times as long),
// FP64 512 (640: 216 instead of 180 us); adj_b FP32 1024, FP64 640 (512: 176
// instead of 171 us, 120 x 104 x 136).
template <typename T>
__host__ __device__ constexpr int adj_e_threads() {
  return sizeof(T) == 4 ? 768 : 512;
}
template <typename T>
__host__ __device__ constexpr int adj_b_threads() {
  return sizeof(T) == 4 ? 1024 : 640;
}

namespace {

// Position of axis index idx in a face entry (-1: outside its layers; an entry
// that is not active has empty layers).
template <typename T>
__device__ __forceinline__ int face_pos(const AdjFace<T> &F, int idx) {
  if (idx >= F.lo0 && idx <= F.hi0) return idx - F.lo0;
  if (idx >= F.lo1 && idx <= F.hi1) return F.n0 + idx - F.lo1;
  return -1;
}

// The components fed by psi0 / psi1 of a face along D (cpml_border.cpp:357-386):
// x faces (y, z), y faces (z, x), z faces (x, y).
template <int D, typename R>
__device__ __forceinline__ R comp0(const R v[3]) {
  return D == 0 ? v[1] : (D == 1 ? v[2] : v[0]);
}
template <int D, typename R>
__device__ __forceinline__ R comp1(const R v[3]) {
  return D == 0 ? v[2] : (D == 1 ? v[0] : v[1]);
}

// A thread's place in the x (D = 0) or y (D = 1) entry of a face pair: the
// element of plane zlo, or -1 outside the layers.  32-bit: the host keeps every
// face array below 2^31 elements.
template <int D, typename T>
__device__ __forceinline__ int face_at(const AdjFace<T> &F, int i, int j, int nx) {
  const int pos = face_pos(F, D == 0 ? i + 1 : j + 1);
  return pos < 0 ? -1 : (D == 0 ? j * F.ex + pos : pos * nx + i);
}
template <int D, typename T>
__device__ __forceinline__ int face_plane(const AdjFace<T> &F, int k, int nx, int ny) {
  return D == 0 ? (k - F.zlo) * ny * F.ex : (k - F.zlo) * F.ey * nx;
}

// c * total of both components at element li of an entry
template <typename T>
__device__ __forceinline__ void face_w(const AdjFace<T> &F, int li, T c, T &w0, T &w1, int *st) {
  w0 = c * ld_c(F.a0, li, F.n, st);
  w1 = c * ld_c(F.a1, li, F.n, st);
}

// One element of column c of the plane at element `base` (a uniform address
// plus a 32-bit offset, as ldp / stp).
template <typename T>
__device__ __forceinline__ T at(const T *a, long long base, unsigned c, long long n, int *st) {
  return ldp<1>(a, base, c, n, st).v[0];
}
template <typename T>
__device__ __forceinline__ void put(T *a, long long base, unsigned c, long long n, int *st, T v) {
  RowV<T, 1> r;
  r.v[0] = v;
  stp<1>(a, base, c, n, st, r);
}

// The new total of an entry: b * total + dt * what it feeds
template <typename T>
__device__ __forceinline__ void face_step(const AdjFace<T> &F, int li, T b, T t0, T t1, T dt, T f0, T f1, int *st) {
  st_c(F.a0, li, F.n, st, T(b * t0 + dt * f0));
  st_c(F.a1, li, F.n, st, T(b * t1 + dt * f1));
}

}  // namespace

// The z-chunks of the reverse kernels over the row mapping of mp_row.cuh, and
// the planes whose z faces hold something: k <= zlo or k >= zhi.
struct AdjGrid : RowMap {
  int kchunk, zlo, zhi;
  int ahead;  // prefetch the next plane into L2
};

// Arithmetic is in T (the precision of the state); the Kerr linearisation and
// the design gradients are FP64.  One thread per (x, y) column marches up a
// chunk of planes, carrying the z-neighbours in registers; the cells are dealt
// to threads as in the half steps (row_cells).  NL: the Kerr medium (PLRC
// nonlinear); the linear form leaves out the Kerr linearisation, whose terms are
// zero there.
// A thread finds its place in the x and y face entries once, before the march,
// and a plane tests three flags: its columns lie in an x entry, in a y entry, the
// plane in a z entry.  On grids that exceed L2 bound by HBM and its latency (the
// next plane is prefetched into L2), on smaller ones by instruction issue (96^3
// with CPML on all faces: 60% of the issue slots).  Reverse step (adj_e + adj_b),
// before -> after: 96^3 FP32 43.6 -> 39.7 us, 120 x 104 x 136 FP64 Kerr 207 -> 164,
// 160 x 144 x 160 FP32 Kerr 229 -> 182, 256^3 FP32 Kerr 1100 -> 795, 192 x 192 x
// 256 FP64 774 -> 548.
template <typename T, int NP, bool NL>
__global__ void __launch_bounds__(kRowThreads, adj_e_threads<T>() / kRowThreads)
    adj_e_kernel(const AdjParams<T> p, const AdjGrid g) {
  typedef T R;
  typedef typename Vec2<T>::type T2;
  pdl_launch_dependents();
  const int nx = p.nx, ny = p.ny;
  int i, j;
  if (!row_cells<1>(g, blockIdx.x, ny, i, j)) return;
  const int k0 = 1 + blockIdx.y * g.kchunk;
  const int k1 = min(k0 + g.kchunk - 1, p.nz);
  const int im = i == 0 ? nx - 1 : i - 1;
  const int jm = j == 0 ? ny - 1 : j - 1;
  const long long pl = p.plane;
  const unsigned row = unsigned(j) * unsigned(nx);
  const unsigned col = row + i, colxm = row + im, colym = unsigned(jm) * unsigned(nx) + i;
  const R dt = R(p.dt);
  const long long nf = p.n_field;
  int *const st = p.status;
  const R kxi = ld(p.ikH[0] + i + 1), kxm = ld(p.ikH[0] + im + 1);
  const R kyj = ld(p.ikH[1] + j + 1), kym = ld(p.ikH[1] + jm + 1);
  const R bzj = ld(p.ikH_bzy + j + 1), bzm = ld(p.ikH_bzy + jm + 1);
  const T *Bx = p.Bb[0], *By = p.Bb[1], *Bz = p.Bb[2];
  const AdjFace<T> &HX = p.fh[0], &HY = p.fh[1], &HZ = p.fh[2];
  const AdjFace<T> &EX = p.fe[0], &EY = p.fe[1], &EZ = p.fe[2];
  // this column (o) and its x-1 / y-1 neighbour (m) in the face entries
  const int hxo = face_at<0>(HX, i, j, nx), hxm = face_at<0>(HX, im, j, nx), exo = face_at<0>(EX, i, j, nx);
  const int hyo = face_at<1>(HY, i, j, nx), hym = face_at<1>(HY, i, jm, nx), eyo = face_at<1>(EY, i, j, nx);
  const bool fx = (hxo & hxm & exo) != -1, fy = (hyo & hym & eyo) != -1;
  const DesignParams &d = p.design;
  const bool dxy = i >= d.x0 && i <= d.x1 && j >= d.y0 && j <= d.y1;
  const bool oxy = p.add_obj && i >= p.ox0 && i <= p.ox1 && j >= p.oy0 && j <= p.oy1;
  // everything below reads what the previous reverse kernel wrote
  pdl_wait();
  R bx_km = at(Bx, (k0 - 1) * pl, col, nf, st);
  R by_km = at(By, (k0 - 1) * pl, col, nf, st);

  for (int k = k0; k <= k1; ++k) {
    const long long base = (long long)k * pl;
    const bool med = k >= p.mz0 && k <= p.mz1;
    const bool dcell = med && dxy && k >= d.z0 && k <= d.z1;
    // ---- every load of this plane first, so that their latencies overlap
    const R bx = at(Bx, base, col, nf, st), by = at(By, base, col, nf, st), bz = at(Bz, base, col, nf, st);
    const R bx_ym = at(Bx, base, colym, nf, st), by_xm = at(By, base, colxm, nf, st),
            bz_ym = at(Bz, base, colym, nf, st), bz_xm = at(Bz, base, colxm, nf, st);
    const R kzk = ld(p.ikH[2] + k), kzm = ld(p.ikH[2] + k - 1);
    R a[3] = {at(p.Eb[0], base, col, nf, st), at(p.Eb[1], base, col, nf, st), at(p.Eb[2], base, col, nf, st)};
    // E^n enters here only through the Kerr term (its coefficient is zero in
    // a linear medium) and the |E|^2 objective's box: elsewhere it is not read
    R En[3] = {R(0), R(0), R(0)};
    if (NL || (oxy && p.obj_kind == 1 && k >= p.oz0 && k <= p.oz1)) {
#pragma unroll
      for (int c = 0; c < 3; ++c) En[c] = at(p.En[c], base, col, nf, st);
    }
    R En1[3] = {R(0), R(0), R(0)};
    if (NL && med) {
#pragma unroll
      for (int c = 0; c < 3; ++c) En1[c] = at(p.En1[c], base, col, nf, st);
    }
    const long long pbase = (long long)(k - p.mz0) * pl;
    T2 pq[NP > 0 ? NP : 1][3];
    if (NP > 0 && med) {
#pragma unroll
      for (int n = 0; n < NP; ++n)
#pragma unroll
        for (int c = 0; c < 3; ++c)
          pq[n][c] = at(reinterpret_cast<const T2 *>(p.psib[n][c]), pbase, col, p.n_psi, st);
    }
    long long di = 0;
    double e = p.eps, s = 1.0, u = 1.0;
    if (dcell) {
      di = ((long long)(k - d.z0) * d.by + (j - d.y0)) * d.bx + (i - d.x0);
      e = ld_c(d.eps, di, p.n_design, st);
      s = ld_c(d.dscale, di, p.n_design, st);
      u = ld_c(d.chiscale, di, p.n_design, st);
    }
    if (g.ahead && k < k1) {
      const long long bn = base + pl;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        prefetch_l2(p.Bb[c] + bn + col);
        prefetch_l2(p.Eb[c] + bn + col);
        if (NL) prefetch_l2(p.En[c] + bn + col);
        if (NL) prefetch_l2(p.En1[c] + bn + col);
        if (med && k < p.mz1) {
#pragma unroll
          for (int n = 0; n < NP; ++n)
            prefetch_l2(reinterpret_cast<const T2 *>(p.psib[n][c]) + pbase + pl + col);
        }
      }
    }
    // H-face totals (at this column and x-1 / y-1, at this plane and k-1) and
    // E-face totals of this cell
    const bool fz = k <= g.zlo || k >= g.zhi;
    R hx0o = R(0), hx1o = R(0), hx0m = R(0), hx1m = R(0), hy0o = R(0), hy1o = R(0), hy0m = R(0), hy1m = R(0);
    R hz0 = R(0), hz1 = R(0), cw0 = R(0), cw1 = R(0);
    R ex0 = R(0), ex1 = R(0), ey0 = R(0), ey1 = R(0), ez0 = R(0), ez1 = R(0);
    int lex = 0, ley = 0, lez = 0, ezp = -1;
    if (fx) {
      const int sh = face_plane<0>(HX, k, nx, ny);
      if (hxo >= 0) face_w(HX, hxo + sh, ld(HX.c + i + 1), hx0o, hx1o, st);
      if (hxm >= 0) face_w(HX, hxm + sh, ld(HX.c + im + 1), hx0m, hx1m, st);
      lex = exo + face_plane<0>(EX, k, nx, ny);
      if (exo >= 0) face_w(EX, lex, R(1), ex0, ex1, st);
    }
    if (fy) {
      const int sh = face_plane<1>(HY, k, nx, ny);
      if (hyo >= 0) face_w(HY, hyo + sh, ld(HY.c + j + 1), hy0o, hy1o, st);
      if (hym >= 0) face_w(HY, hym + sh, ld(HY.c + jm + 1), hy0m, hy1m, st);
      ley = eyo + face_plane<1>(EY, k, nx, ny);
      if (eyo >= 0) face_w(EY, ley, R(1), ey0, ey1, st);
    }
    if (fz) {
      const int hzp = face_pos(HZ, k), hzm = face_pos(HZ, k - 1);
      if (hzp >= 0) face_w(HZ, hzp * int(pl) + int(col), ld(HZ.c + k), hz0, hz1, st);
      if (hzm >= 0) face_w(HZ, hzm * int(pl) + int(col), ld(HZ.c + k - 1), cw0, cw1, st);
      ezp = face_pos(EZ, k);
      lez = ezp * int(pl) + int(col);
      if (ezp >= 0) face_w(EZ, lez, R(1), ez0, ez1, st);
    }
    R obx = R(0), oby = R(0);
    const bool osz = oxy && p.obj_kind == 2 && k == p.oz0;
    if (osz) {
      obx = ld_c(p.obx, col, pl, st);
      oby = ld_c(p.oby, col, pl, st);
    }

    // ---- adjoint of E' (B half transposed)
    // Bx' = .. + dt ((ey(k+1) - ey) ikz - (ez(j+1) - ez) iky)
    a[1] += dt * (kzm * bx_km - kzk * bx);
    a[2] += dt * (-kym * bx_ym + kyj * bx);
    // By' = .. + dt ((ez(i+1) - ez) ikx - (ex(k+1) - ex) ikz)
    a[2] += dt * (kxm * by_xm - kxi * by);
    a[0] += dt * (-kzm * by_km + kzk * by);
    // Bz' = .. + dt ((ex(j+1) - ex) iky_bz - (ey(i+1) - ey) ikx)
    a[0] += dt * (bzm * bz_ym - bzj * bz);
    a[1] += dt * (-kxm * bz_xm + kxi * bz);
    // H faces: psi0 / psi1 feed (y, z) on x faces, (z, x) on y faces, (x, y) on
    // z faces; their differences of E run forward along the axis
    if (fx) {
      a[2] += hx0m - hx0o;
      a[1] += hx1o - hx1m;
    }
    if (fy) {
      a[0] += hy0m - hy0o;
      a[2] += hy1o - hy1m;
    }
    if (fz) {
      a[1] += cw0 - hz0;
      a[0] += hz1 - cw1;
    }

    // ---- E half, locally
    R gg[3], ne[3];
    if (!med) {
      // background: E' = (eps_bg E + dt (curl + J)) / eps_bg
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        gg[c] = a[c] * p.inv_eps_bg_t;
        ne[c] = p.eps_bg_t * gg[c];
      }
    } else {
      double A = NL ? p.A0 : 0.0;
      R idn = p.inv_denom0_t, numer = p.numer0_t, Rchi = NL ? p.chi_nl_t : R(0);
      if (dcell) {
        const double denom = d.lin ? e + s * (p.sumChi0 - p.sumXi0) : e + s * p.sumChi0 - s * p.sumXi0;
        A = NL ? u * p.chi / denom : 0.0;
        idn = R(1.0 / denom);
        numer = R(e - s * p.sumXi0);
        Rchi = NL ? R(u * p.chi) : R(0);
      }
      R cb[3] = {a[0], a[1], a[2]};
      if (NL) {
        // E' = r c/|c| with r + A r^3 = |c|: dE'/dc = (I - e e^T) / (1 + A r^2)
        // + e e^T / (1 + 3 A r^2), dr/dA = -r^3 / (1 + 3 A r^2), c = E' (1 + A r^2);
        // the reciprocals of the denominators (>= 1) and of r as in the forward
        // Kerr update (FP64, exact to rounding)
        const double r2 = sq3((double)En1[0], (double)En1[1], (double)En1[2]);
        const double al = rcp_pos(1.0 + A * r2), be = rcp_pos(1.0 + 3.0 * A * r2);
        const double ir = r2 > 0 ? rsqrt(r2) : 0.0;
        double eh[3], ea = 0.0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          eh[c] = En1[c] * ir;
          ea += eh[c] * a[c];
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) cb[c] = R(al * (a[c] - eh[c] * ea) + be * eh[c] * ea);
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) gg[c] = cb[c] * idn;
      if (NL) {
        const R E2 = En[0] * En[0] + En[1] * En[1] + En[2] * En[2];
        const R Eg = En[0] * gg[0] + En[1] * gg[1] + En[2] * gg[2];
        const R f = numer + Rchi * E2;
#pragma unroll
        for (int c = 0; c < 3; ++c) ne[c] = f * gg[c] + R(2) * Rchi * En[c] * Eg;
      } else {
#pragma unroll
        for (int c = 0; c < 3; ++c) ne[c] = numer * gg[c];
      }
      // the design cells' accumulator adjoints before the reverse recursion,
      // for adj_grad
      if (dcell) {
#pragma unroll
        for (int n = 0; n < NP; ++n)
#pragma unroll
          for (int c = 0; c < 3; ++c)
            st_c(reinterpret_cast<T2 *>(p.dpsi), (di * NP + n) * 3 + c, p.n_design * NP * 3, st, pq[n][c]);
      }
      // reverse PLRC recursion: psi~bar = conj(Crec) psibar + g
      const R Rs = dcell ? R(s) : R(1);
#pragma unroll
      for (int n = 0; n < NP; ++n) {
        const R Dr = p.pDt[n][0], Di = p.pDt[n][1];
        const R Xr = p.pxit[n][0], Xi = p.pxit[n][1];
        const R Cr = p.pCt[n][0], Ci = p.pCt[n][1];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const R pr = pq[n][c].x, pim = pq[n][c].y;
          const R tr = Cr * pr + Ci * pim + gg[c];
          const R ti = Cr * pim - Ci * pr;
          ne[c] += Rs * (Dr * tr + Di * ti + Xr * pr + Xi * pim);
          pq[n][c].x = tr;
          pq[n][c].y = ti;
        }
      }
    }
    // the objective's E term of the state before the step
    if (oxy && p.obj_kind == 1 && k >= p.oz0 && k <= p.oz1) {
#pragma unroll
      for (int c = 0; c < 3; ++c) ne[c] += p.obj_f_t * En[c];
    }
    if (osz) {
      ne[0] += p.obj_f_t * oby;
      ne[1] -= p.obj_f_t * obx;
    }

    // ---- stores
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      put(p.G[c], base, col, nf, st, gg[c]);
      put(p.Eb[c], base, col, nf, st, ne[c]);
    }
    if (NP > 0 && med) {
#pragma unroll
      for (int n = 0; n < NP; ++n)
#pragma unroll
        for (int c = 0; c < 3; ++c) put(reinterpret_cast<T2 *>(p.psib[n][c]), pbase, col, p.n_psi, st, pq[n][c]);
    }
    // E-face totals of this cell: b * total + dt * G
    if (fx && exo >= 0) face_step(EX, lex, ld(EX.b + i + 1), ex0, ex1, dt, comp0<0>(gg), comp1<0>(gg), st);
    if (fy && eyo >= 0) face_step(EY, ley, ld(EY.b + j + 1), ey0, ey1, dt, comp0<1>(gg), comp1<1>(gg), st);
    if (fz && ezp >= 0) face_step(EZ, lez, ld(EZ.b + k), ez0, ez1, dt, comp0<2>(gg), comp1<2>(gg), st);
    bx_km = bx;
    by_km = by;
  }
}

// The design gradients of one step, one thread per design cell (the design
// box lies inside the medium planes and the interior).  From the E half
// X = (numer + chi |E|^2) E + dt (curl + J) + Re sum psi~ with numer = e - s
// sumXi0, denom = e + s (sumChi0 - sumXi0), psi~ = s (dchi0 - dxi0) E + psi,
// psi' = s dxi0 E + Crec psi~ and (nonlinear) A = u chi / denom, with g the
// adjoint of X / denom that adj_e stored in G:
//   dJ/de += g . (E - c) - Abar A / denom
//   dJ/ds += sum_n,c psibar_nc . (dxi0 + Crec (dchi0 - dxi0)) E_c
//            + g . ((sum_n Re(dchi0 - dxi0) - sumXi0) E - c dD) - Abar A dD / denom
//   dJ/du += g . chi |E|^2 E + Abar chi / denom
// where c = E' (1 + A |E'|^2) is X / denom, dD = sumChi0 - sumXi0 and Abar,
// the adjoint of A through the Kerr solve, is -(e^ . c_bar) r^3 with r = |E'|,
// e^ = E' / r and c_bar = g denom the adjoint of c (the Kerr linearisation of
// adj_e gives e^ . c_bar = be (e^ . a) with be = 1 / (1 + 3 A r^2)).
template <typename T, int NP, bool NL>
__device__ __forceinline__ void adj_grad_cells(const AdjParams<T> &p, int gbx, int gby, int kk) {
  const DesignParams &d = p.design;
  const int ii = gbx * 32 + (threadIdx.x & 31), jj = gby * kRowTile + (threadIdx.x >> 5);
  if (ii >= d.bx || jj >= d.by) return;
  pdl_wait();
  const int i = d.x0 + ii, j = d.y0 + jj, k = d.z0 + kk;
  const long long nf = p.n_field;
  int *const st = p.status;
  const long long di = ((long long)kk * d.by + jj) * d.bx + ii;
  const long long c0 = (long long)k * p.plane + (long long)j * p.nx + i;
  const double e = ld_c(d.eps, di, p.n_design, st), s = ld_c(d.dscale, di, p.n_design, st),
               u = ld_c(d.chiscale, di, p.n_design, st);
  T g[3], En[3], En1[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    g[c] = ld_c(p.G[c], c0, nf, st);
    En[c] = ld_c(p.En[c], c0, nf, st);
    En1[c] = ld_c(p.En1[c], c0, nf, st);
  }
  const double dD = p.sumChi0 - p.sumXi0;
  const double denom = d.lin ? e + s * dD : e + s * p.sumChi0 - s * p.sumXi0;
  const double A = NL ? u * p.chi / denom : 0.0;
  const double r2 = NL ? (double)En1[0] * En1[0] + (double)En1[1] * En1[1] + (double)En1[2] * En1[2] : 0.0;
  double Abar = 0.0;
  if (NL && r2 > 0) {
    const double r = sqrt(r2);
    double ecb = 0.0;
#pragma unroll
    for (int c = 0; c < 3; ++c) ecb += (double)En1[c] / r * ((double)g[c] * denom);
    Abar = -ecb * r * r2;
  }
  double gs = 0.0, SD = 0.0;
#pragma unroll
  for (int n = 0; n < NP; ++n) {
    SD += p.pD[n][0];
    const double CDr = p.pC[n][0] * p.pD[n][0] - p.pC[n][1] * p.pD[n][1];
    const double CDi = p.pC[n][0] * p.pD[n][1] + p.pC[n][1] * p.pD[n][0];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const long long q = ((di * NP + n) * 3 + c) * 2;
      const double pr = ld_c(p.dpsi, q, p.n_design * NP * 6, st), pim = ld_c(p.dpsi, q + 1, p.n_design * NP * 6, st);
      gs += (pr * (p.pxi[n][0] + CDr) + pim * (p.pxi[n][1] + CDi)) * (double)En[c];
    }
  }
  double ge = NL ? -Abar * A / denom : 0.0, gu = 0.0;
  if (NL) gs -= Abar * A * dD / denom;
  const double grow = NL ? 1.0 + A * r2 : 1.0;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double cv = (double)En1[c] * grow;
    ge += (double)g[c] * ((double)En[c] - cv);
    gs += (double)g[c] * ((SD - p.sumXi0) * (double)En[c] - cv * dD);
  }
  if (NL) {
    const T E2 = En[0] * En[0] + En[1] * En[1] + En[2] * En[2];
    gu = Abar * p.chi / denom;
#pragma unroll
    for (int c = 0; c < 3; ++c) gu += (double)g[c] * p.chi * (double)E2 * (double)En[c];
  }
  st_c(p.grad[0], di, p.n_design, st, ld_c(p.grad[0], di, p.n_design, st) + ge);
  st_c(p.grad[1], di, p.n_design, st, ld_c(p.grad[1], di, p.n_design, st) + gs);
  st_c(p.grad[2], di, p.n_design, st, ld_c(p.grad[2], di, p.n_design, st) + gu);
}

template <typename T>
__device__ __forceinline__ void adj_b_cells(const AdjParams<T> &p, const AdjGrid &g, unsigned block, int chunk) {
  typedef T R;
  const int nx = p.nx, ny = p.ny;
  int i, j;
  if (!row_cells<1>(g, block, ny, i, j)) return;
  const int k0 = chunk * g.kchunk;
  const int k1 = min(k0 + g.kchunk - 1, p.nz);
  const int ip = i == nx - 1 ? 0 : i + 1;
  const int jp = j == ny - 1 ? 0 : j + 1;
  const long long pl = p.plane;
  const unsigned row = unsigned(j) * unsigned(nx);
  const unsigned col = row + i, colxp = row + ip, colyp = unsigned(jp) * unsigned(nx) + i;
  const R dt = R(p.dt);
  const long long nf = p.n_field;
  int *const st = p.status;
  const R kxi = ld(p.ikE[0] + i + 1), kxp = ld(p.ikE[0] + ip + 1);
  const R kyj = ld(p.ikE[1] + j + 1), kyp = ld(p.ikE[1] + jp + 1);
  const T *gx = p.G[0], *gy = p.G[1], *gz = p.G[2];
  const AdjFace<T> &HX = p.fh[0], &HY = p.fh[1], &HZ = p.fh[2];
  const AdjFace<T> &EX = p.fe[0], &EY = p.fe[1], &EZ = p.fe[2];
  // this column (o) and its x+1 / y+1 neighbour (p) in the face entries
  const int exo = face_at<0>(EX, i, j, nx), exp_ = face_at<0>(EX, ip, j, nx), hxo = face_at<0>(HX, i, j, nx);
  const int eyo = face_at<1>(EY, i, j, nx), eyp = face_at<1>(EY, i, jp, nx), hyo = face_at<1>(HY, i, j, nx);
  const bool fx = (exo & exp_ & hxo) != -1, fy = (eyo & eyp & hyo) != -1;
  const bool oxy = p.add_obj && p.obj_kind == 2 && i >= p.ox0 && i <= p.ox1 && j >= p.oy0 && j <= p.oy1;
  // everything below reads what adj_e wrote
  pdl_wait();
  // G at plane k, carried from the previous plane's k + 1
  R gx_k = at(gx, k0 * pl, col, nf, st), gy_k = at(gy, k0 * pl, col, nf, st);

  for (int k = k0; k <= k1; ++k) {
    const long long base = (long long)k * pl;
    // ---- every load of this plane first
    const R gx_kp = at(gx, base + pl, col, nf, st), gy_kp = at(gy, base + pl, col, nf, st);
    const R gzk = at(gz, base, col, nf, st);
    const R gx_yp = at(gx, base, colyp, nf, st), gy_xp = at(gy, base, colxp, nf, st),
            gz_xp = at(gz, base, colxp, nf, st), gz_yp = at(gz, base, colyp, nf, st);
    const R kzk = ld(p.ikE[2] + k), kzp = ld(p.ikE[2] + k + 1);
    R b[3] = {at(p.Bb[0], base, col, nf, st), at(p.Bb[1], base, col, nf, st), at(p.Bb[2], base, col, nf, st)};
    if (g.ahead && k < k1) {
      const long long bn = base + pl;
      prefetch_l2(gx + bn + pl + col);
      prefetch_l2(gy + bn + pl + col);
      prefetch_l2(gz + bn + col);
#pragma unroll
      for (int c = 0; c < 3; ++c) prefetch_l2(p.Bb[c] + bn + col);
    }
    // E faces (x / y hold planes 1..nz; z at planes k and k + 1) and the
    // H-face totals of this cell
    const bool fz = k <= g.zlo || k >= g.zhi;
    R ex0o = R(0), ex1o = R(0), ex0p = R(0), ex1p = R(0), ey0o = R(0), ey1o = R(0), ey0p = R(0), ey1p = R(0);
    R zw0 = R(0), zw1 = R(0), ez0p = R(0), ez1p = R(0);
    R hx0 = R(0), hx1 = R(0), hy0 = R(0), hy1 = R(0), hz0 = R(0), hz1 = R(0);
    int lhx = -1, lhy = -1, lhz = 0, hzp = -1;
    if (fx) {
      const int se = face_plane<0>(EX, k, nx, ny);
      if (exo >= 0 && k >= 1) face_w(EX, exo + se, ld(EX.c + i + 1), ex0o, ex1o, st);
      if (exp_ >= 0 && k >= 1) face_w(EX, exp_ + se, ld(EX.c + ip + 1), ex0p, ex1p, st);
      if (hxo >= 0 && k >= HX.zlo) {
        lhx = hxo + face_plane<0>(HX, k, nx, ny);
        face_w(HX, lhx, R(1), hx0, hx1, st);
      }
    }
    if (fy) {
      const int se = face_plane<1>(EY, k, nx, ny);
      if (eyo >= 0 && k >= 1) face_w(EY, eyo + se, ld(EY.c + j + 1), ey0o, ey1o, st);
      if (eyp >= 0 && k >= 1) face_w(EY, eyp + se, ld(EY.c + jp + 1), ey0p, ey1p, st);
      if (hyo >= 0 && k >= HY.zlo) {
        lhy = hyo + face_plane<1>(HY, k, nx, ny);
        face_w(HY, lhy, R(1), hy0, hy1, st);
      }
    }
    if (fz) {
      const int ezo = face_pos(EZ, k), ezq = face_pos(EZ, k + 1);
      if (ezo >= 0) face_w(EZ, ezo * int(pl) + int(col), ld(EZ.c + k), zw0, zw1, st);
      if (ezq >= 0) face_w(EZ, ezq * int(pl) + int(col), ld(EZ.c + k + 1), ez0p, ez1p, st);
      hzp = face_pos(HZ, k);
      lhz = hzp * int(pl) + int(col);
      if (hzp >= 0) face_w(HZ, lhz, R(1), hz0, hz1, st);
    }
    const bool obj = oxy && k == p.oz0;
    R oex = R(0), oey = R(0);
    if (obj) {
      oex = at(p.En[0], base, col, nf, st);
      oey = at(p.En[1], base, col, nf, st);
    }

    // ---- transposed curl_E and E faces
    // cbx = (bz - bz(j-1)) iky - (by - by(k-1)) ikz
    b[2] += dt * (kyj * gx_k - kyp * gx_yp);
    b[1] += dt * (-kzk * gx_k + kzp * gx_kp);
    // cby = (bx - bx(k-1)) ikz - (bz - bz(i-1)) ikx
    b[0] += dt * (kzk * gy_k - kzp * gy_kp);
    b[2] += dt * (-kxi * gy_k + kxp * gy_xp);
    // cbz = (by - by(i-1)) ikx - (bx - bx(j-1)) iky
    b[1] += dt * (kxi * gzk - kxp * gz_xp);
    b[0] += dt * (-kyj * gzk + kyp * gz_yp);
    // E faces: psi0 / psi1 feed (y, z) on x faces, (z, x) on y faces, (x, y) on
    // z faces; their differences of B run backward along the axis
    if (fx) {
      b[2] += -ex0o + ex0p;
      b[1] += ex1o - ex1p;
    }
    if (fy) {
      b[0] += -ey0o + ey0p;
      b[2] += ey1o - ey1p;
    }
    if (fz) {
      b[1] += -zw0 + ez0p;
      b[0] += zw1 - ez1p;
    }
    // the objective's B term of the state before the step (Sz plane)
    if (obj) {
      b[0] -= p.obj_f_t * oey;
      b[1] += p.obj_f_t * oex;
    }

    // ---- stores: B adjoint, H-face totals for the step before (b * total + dt * B adjoint)
#pragma unroll
    for (int c = 0; c < 3; ++c) put(p.Bb[c], base, col, nf, st, b[c]);
    if (fx && lhx >= 0) face_step(HX, lhx, ld(HX.b + i + 1), hx0, hx1, dt, comp0<0>(b), comp1<0>(b), st);
    if (fy && lhy >= 0) face_step(HY, lhy, ld(HY.b + j + 1), hy0, hy1, dt, comp0<1>(b), comp1<1>(b), st);
    if (fz && hzp >= 0) face_step(HZ, lhz, ld(HZ.b + k), hz0, hz1, dt, comp0<2>(b), comp1<2>(b), st);
    gx_k = gx_kp;
    gy_k = gy_kp;
  }
}

// The B half of the reverse step (blocks 0 .. nb-1 of a one-dimensional grid,
// gx blocks a z-chunk) and the design gradients of the step (the blocks after
// them, over the design box in tiles of 32 x kRowTile, one plane each).
template <typename T, int NP, bool NL>
__global__ void __launch_bounds__(kRowThreads, adj_b_threads<T>() / kRowThreads)
    adj_b_kernel(const AdjParams<T> p, const AdjGrid g, const int gx, const int nb) {
  pdl_launch_dependents();
  const int b = blockIdx.x;
  if (b < nb) {
    adj_b_cells<T>(p, g, b % gx, b / gx);
  } else {
    const int q = b - nb;
    const int tx = (p.design.bx + 31) / 32, ty = (p.design.by + kRowTile - 1) / kRowTile;
    adj_grad_cells<T, NP, NL>(p, q % tx, (q / tx) % ty, q / (tx * ty));
  }
}

// Start of the reverse pass (state T): the adjoint of E and B is the
// objective's derivative with respect to that state, the H-face totals dt times
// the adjoint of B, everything else zero (the arrays arrive zeroed).
template <typename T>
__global__ void __launch_bounds__(256) adj_init_kernel(const AdjParams<T> p) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int k = blockIdx.z;  // 0..nz
  if (i >= p.nx || j >= p.ny) return;
  const long long col = (long long)j * p.nx + i, c0 = (long long)k * p.plane + col;
  const long long nf = p.n_field;
  int *const st = p.status;
  double e[3] = {0.0, 0.0, 0.0}, b[3] = {0.0, 0.0, 0.0};
  const bool inxy = i >= p.ox0 && i <= p.ox1 && j >= p.oy0 && j <= p.oy1;
  if (p.obj_kind == 1) {
    if (inxy && k >= p.oz0 && k <= p.oz1)
      for (int c = 0; c < 3; ++c) e[c] = p.obj_f * (double)ld_c(p.En[c], c0, nf, st);
  } else if (inxy && k == p.oz0) {
    e[0] = p.obj_f * (double)ld_c(p.oby, col, p.plane, st);
    e[1] = -p.obj_f * (double)ld_c(p.obx, col, p.plane, st);
    b[0] = -p.obj_f * (double)ld_c(p.En[1], c0, nf, st);
    b[1] = p.obj_f * (double)ld_c(p.En[0], c0, nf, st);
  }
  for (int c = 0; c < 3; ++c) {
    st_c(p.Eb[c], c0, nf, st, T(e[c]));
    st_c(p.Bb[c], c0, nf, st, T(b[c]));
  }
  // H-face totals: dt times the adjoint of B
  const int hxo = face_at<0>(p.fh[0], i, j, p.nx), hyo = face_at<1>(p.fh[1], i, j, p.nx), hzo = face_pos(p.fh[2], k);
  if (hxo >= 0 && k >= p.fh[0].zlo) {
    const int li = hxo + face_plane<0>(p.fh[0], k, p.nx, p.ny);
    st_c(p.fh[0].a0, li, p.fh[0].n, st, T(p.dt * comp0<0>(b)));
    st_c(p.fh[0].a1, li, p.fh[0].n, st, T(p.dt * comp1<0>(b)));
  }
  if (hyo >= 0 && k >= p.fh[1].zlo) {
    const int li = hyo + face_plane<1>(p.fh[1], k, p.nx, p.ny);
    st_c(p.fh[1].a0, li, p.fh[1].n, st, T(p.dt * comp0<1>(b)));
    st_c(p.fh[1].a1, li, p.fh[1].n, st, T(p.dt * comp1<1>(b)));
  }
  if (hzo >= 0) {
    const long long li = (long long)hzo * p.plane + col;
    st_c(p.fh[2].a0, li, p.fh[2].n, st, T(p.dt * comp0<2>(b)));
    st_c(p.fh[2].a1, li, p.fh[2].n, st, T(p.dt * comp1<2>(b)));
  }
}

// One step's objective term as gridDim.x partial sums, out[block], FP64 in a
// fixed order.  `lanes` threads (a power of two) run along a row of the box, so
// a block takes 256 / lanes rows at a time.  Latency-bound at the sizes in use:
// with the one block of 256 threads that it had, the term of a 128 x 128 plane
// cost 37 us a step beside 162 us of half steps, that of an 8^3 box 4.6; with
// four cells per thread 5 and 2.5 (launched early, beside the half steps).
template <typename T>
__global__ void __launch_bounds__(256) objective_term_kernel(const T *Ex, const T *Ey, const T *Ez, const T *Bx,
                                                             const T *By, int nx, long long plane, int kind, int x0,
                                                             int x1, int y0, unsigned by, int z0, unsigned rows,
                                                             int lanes, double f, double *out) {
  __shared__ double red[8];
  pdl_launch_dependents();
  const unsigned per = 256u / unsigned(lanes);
  const int lane = threadIdx.x & (lanes - 1);
  double acc = 0.0;
  pdl_wait();
  for (unsigned r = blockIdx.x * per + threadIdx.x / unsigned(lanes); r < rows; r += gridDim.x * per) {
    const unsigned k = r / by;
    const long long row = (long long)(z0 + int(k)) * plane + (long long)(y0 + int(r - k * by)) * nx;
    for (int i = x0 + lane; i <= x1; i += lanes) {
      const long long c = row + i;
      if (kind == 1) {
        const double ex = Ex[c], ey = Ey[c], ez = Ez[c];
        acc += ex * ex + ey * ey + ez * ez;
      } else {
        acc += (double)Ex[c] * (double)By[c] - (double)Ey[c] * (double)Bx[c];
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) acc += red[w];
    out[blockIdx.x] = f * acc;
  }
}

__global__ void __launch_bounds__(256) sum_terms_kernel(const double *terms, long long n, double *out) {
  __shared__ double red[256];
  double acc = 0.0;
  for (long long q = threadIdx.x; q < n; q += blockDim.x) acc += terms[q];
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int s = 128; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = red[0];
}

// ---------------------------------------------------------------------------
// Launchers

// The grid of a reverse kernel over nk planes (zlo / zhi: set by the caller).
// One plane per block on the smallest grids, up to 8 on large ones (reverse step
// with 2 / 3 / 4 / 8 planes: 96^3 FP32 40 / 40 / 42 / 49 us, 120 x 104 x 136 FP64
// Kerr 165 / 162 / 165 / 184, 256^3 FP32 Kerr 877 / 823 / 804 / 778; 64 x 56 x 70
// with 1 / 2 / 3 21 / 23 / 26).  The next plane is prefetched into L2 where the
// adjoint state does not stay there (256^3 855 -> 778 us, 192 x 192 x 256 FP64
// 602 -> 546; 96^3 40 -> 41).
template <typename T>
static AdjGrid adj_grid(const AdjParams<T> &p, int nk, int *blocks) {
  AdjGrid g;
  static_cast<RowMap &>(g) = row_map(p.nx, p.ny, 1);
  const long long bxy = (g.nvec + 31) / 32, all = bxy * nk;
  *blocks = int(bxy);
  g.kchunk = std::max(int(std::min(8LL, (all + 6499) / 6500)), (nk + 65534) / 65535);
  g.ahead = (long long)sizeof(T) * (9 * p.n_field + 6 * p.np * p.n_psi) > (160LL << 20);
  return g;
}

template <typename T>
cudaError_t launch_adj_e(const AdjParams<T> &p, cudaStream_t st) {
  int gx;
  AdjGrid q = adj_grid(p, p.nz, &gx);
  // planes k with k or k - 1 in an H layer, or k in an E layer
  const AdjFace<T> &H = p.fh[2], &E = p.fe[2];
  q.zlo = std::max(H.active ? H.hi0 + 1 : -1, E.active ? E.hi0 : -1);
  q.zhi = std::min(H.active && H.lo1 <= H.hi1 ? H.lo1 : 1 << 30, E.active && E.lo1 <= E.hi1 ? E.lo1 : 1 << 30);
  const dim3 b(kRowThreads, 1, 1), g(gx, (p.nz + q.kchunk - 1) / q.kchunk);
  const bool nl = p.nonlin != 0;
  switch (p.np) {
    case 0: return nl ? launch_pdl(adj_e_kernel<T, 0, true>, g, b, st, p, q) : launch_pdl(adj_e_kernel<T, 0, false>, g, b, st, p, q);
    case 1: return nl ? launch_pdl(adj_e_kernel<T, 1, true>, g, b, st, p, q) : launch_pdl(adj_e_kernel<T, 1, false>, g, b, st, p, q);
    case 2: return nl ? launch_pdl(adj_e_kernel<T, 2, true>, g, b, st, p, q) : launch_pdl(adj_e_kernel<T, 2, false>, g, b, st, p, q);
    default: return nl ? launch_pdl(adj_e_kernel<T, 3, true>, g, b, st, p, q) : launch_pdl(adj_e_kernel<T, 3, false>, g, b, st, p, q);
  }
}

// adj_b of the step, with the design gradients (when there is a design box) in
// extra blocks of the same launch.
template <typename T>
cudaError_t launch_adj_b(const AdjParams<T> &p, cudaStream_t st) {
  int gx;
  AdjGrid q = adj_grid(p, p.nz + 1, &gx);
  // planes k with k or k + 1 in an E layer, or k in an H layer
  const AdjFace<T> &H = p.fh[2], &E = p.fe[2];
  q.zlo = std::max(H.active ? H.hi0 : -1, E.active ? E.hi0 : -1);
  q.zhi = std::min(H.active && H.lo1 <= H.hi1 ? H.lo1 : 1 << 30, E.active && E.lo1 <= E.hi1 ? E.lo1 - 1 : 1 << 30);
  const int nb = gx * ((p.nz + 1 + q.kchunk - 1) / q.kchunk);
  const DesignParams &d = p.design;
  const int ng = d.x0 <= d.x1 ? ((d.bx + 31) / 32) * ((d.by + kRowTile - 1) / kRowTile) * (d.z1 - d.z0 + 1) : 0;
  const dim3 b(kRowThreads, 1, 1), g(nb + ng, 1, 1);
  const bool nl = p.nonlin != 0;
  switch (p.np) {
    case 0: return nl ? launch_pdl(adj_b_kernel<T, 0, true>, g, b, st, p, q, gx, nb) : launch_pdl(adj_b_kernel<T, 0, false>, g, b, st, p, q, gx, nb);
    case 1: return nl ? launch_pdl(adj_b_kernel<T, 1, true>, g, b, st, p, q, gx, nb) : launch_pdl(adj_b_kernel<T, 1, false>, g, b, st, p, q, gx, nb);
    case 2: return nl ? launch_pdl(adj_b_kernel<T, 2, true>, g, b, st, p, q, gx, nb) : launch_pdl(adj_b_kernel<T, 2, false>, g, b, st, p, q, gx, nb);
    default: return nl ? launch_pdl(adj_b_kernel<T, 3, true>, g, b, st, p, q, gx, nb) : launch_pdl(adj_b_kernel<T, 3, false>, g, b, st, p, q, gx, nb);
  }
}

template <typename T>
cudaError_t launch_adj_init(const AdjParams<T> &p, cudaStream_t st) {
  const dim3 b(32, 8, 1), g((p.nx + 31) / 32, (p.ny + 7) / 8, p.nz + 1);
  adj_init_kernel<T><<<g, b, 0, st>>>(p);
  return cudaGetLastError();
}

// Blocks (partial sums) of a step's term over a box: four cells per thread, at
// most one block per SM.
int objective_blocks(const int box0[6]) {
  const long long cells =
      (long long)(box0[1] - box0[0] + 1) * (box0[3] - box0[2] + 1) * (box0[5] - box0[4] + 1);
  return int(cells > 1024 * 148 ? 148 : (cells + 1023) / 1024);
}

template <typename T>
cudaError_t launch_objective_term(const T *const E[3], const T *const B[3], int nx, long long plane, int kind,
                                  const int box0[6], double f, double *out, cudaStream_t st) {
  const unsigned by = unsigned(box0[3] - box0[2] + 1), rows = by * unsigned(box0[5] - box0[4] + 1);
  int lanes = 1;
  while (lanes < 32 && lanes < box0[1] - box0[0] + 1) lanes *= 2;
  return launch_pdl(objective_term_kernel<T>, dim3(objective_blocks(box0), 1, 1), dim3(256, 1, 1), st, E[0], E[1],
                    E[2], B[0], B[1], nx, plane, kind, box0[0], box0[1], box0[2], by, box0[4], rows, lanes, f, out);
}

cudaError_t launch_sum_terms(const double *terms, long long n, double *out, cudaStream_t st) {
  sum_terms_kernel<<<1, 256, 0, st>>>(terms, n, out);
  return cudaGetLastError();
}

template cudaError_t launch_adj_e<float>(const AdjParams<float> &, cudaStream_t);
template cudaError_t launch_adj_e<double>(const AdjParams<double> &, cudaStream_t);
template cudaError_t launch_adj_b<float>(const AdjParams<float> &, cudaStream_t);
template cudaError_t launch_adj_b<double>(const AdjParams<double> &, cudaStream_t);
template cudaError_t launch_adj_init<float>(const AdjParams<float> &, cudaStream_t);
template cudaError_t launch_adj_init<double>(const AdjParams<double> &, cudaStream_t);
template cudaError_t launch_objective_term<float>(const float *const[3], const float *const[3], int, long long, int,
                                                  const int[6], double, double *, cudaStream_t);
template cudaError_t launch_objective_term<double>(const double *const[3], const double *const[3], int, long long, int,
                                                   const int[6], double, double *, cudaStream_t);

}  // namespace mpb
