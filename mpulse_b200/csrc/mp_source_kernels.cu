// mp_source_kernels.cu - per-step values of the TF/SF injection planes.
//
// For every built injector kind MPulse adds currents on the `down` face only
// (PlaneWaveSource / PlaneGaussSource::needCurrent, sources.cpp:8-11, :179-182;
// ShortPulseInject::needCurrent, shortpulseinject.cpp:28-31).  Per step:
//   E side (IncidentSourceECurrent::stepScheme, incsource.t:40-73): on plane
//     z = d, J_x = H_inc,y(i, j, d-1, t) / dz and J_y = H_inc,x / dz;
//   H side (IncidentSourceHCurrent::stepScheme, incsource.t:112-145): on plane
//     z = d-1, M_x = E_inc,y(i, j, d-1, t) / dz and M_y = E_inc,x / dz,
// with t = Process::time.  One thread per interior (i, j); the step kernels
// read the two planes written here.
#include "mp_device.h"
#include "mp_pulse_math.h"

#include <cuda_runtime.h>

namespace mpb {

// getHField of PlaneWaveSourceEFunc / PlaneGaussSourceEFunc (sources.cpp:107-125,
// :266-284) and getEField of the H functions (sources.cpp:150-173, :308-331).
__device__ void plane_source_field(const SourceEvalParams &q, int i, int j, int l, double out[3]) {
  const double *k = q.k;
  double pos[3];
  if (!q.isH) {
    const double realtime = q.dt * ((double)q.time - 0.5);
    pos[0] = k[0] * i * q.dx + k[1] * (j + 0.5) * q.dy + k[2] * (l + 0.5) * q.dz + q.om * realtime;
    pos[1] = k[0] * (i + 0.5) * q.dx + k[1] * j * q.dy + k[2] * (l + 0.5) * q.dz + q.om * realtime;
    pos[2] = k[0] * (i + 0.5) * q.dx + k[1] * (j + 0.5) * q.dy + k[2] * l * q.dz + q.om * realtime;
  } else {
    const double realtime = q.dt * (double)q.time;
    pos[0] = k[0] * (i + 0.5) * q.dx + k[1] * j * q.dy + k[2] * l * q.dz + q.om * realtime;
    pos[1] = k[0] * i * q.dx + k[1] * (j + 0.5) * q.dy + k[2] * l * q.dz + q.om * realtime;
    pos[2] = k[0] * i * q.dx + k[1] * j * q.dy + k[2] * (l + 0.5) * q.dz + q.om * realtime;
  }
  for (int c = 0; c < 3; ++c) {
    if (q.kind == 1) {  // MP_SOURCE_PLANE_WAVE
      double v = q.amp3[c] * sin(pos[c]) + q.bg[c];
      if (pos[c] < q.ramp) v *= pos[c] / q.ramp;
      out[c] = v;
    } else {            // MP_SOURCE_PLANE_GAUSS
      const double a = (pos[c] - q.offset) / q.width;
      out[c] = q.amp3[c] * exp(-(a * a)) * sin(pos[c]);
    }
  }
}

__device__ __forceinline__ ShortPulse short_pulse_of(const SourceEvalParams &q) {
  ShortPulse sp;
  sp.c = q.lightspeed; sp.ZRl = q.ZRl; sp.phase = q.phase; sp.T = q.length; sp.om0 = q.om0;
  sp.coef = q.w_coef; sp.L = q.w_L;
  sp.eiphi = cd(q.sp_eiphi[0], q.sp_eiphi[1]);
  sp.emip = cd(q.sp_emip[0], q.sp_emip[1]);
  sp.g = q.sp_g;
  return sp;
}

// ShortPulseInjectSourceFunc::getHField / getEField (shortpulseinject.cpp:126-178),
// one component: Ex of getEField, Bx or By of getHField (the others are zero).
enum PulsePart { PULSE_EX, PULSE_BX, PULSE_BY };
template <PulsePart PART>
__device__ __forceinline__ double short_pulse_part(const SourceEvalParams &q, int i, int j, int l) {
  const ShortPulse sp = short_pulse_of(q);
  if (PART == PULSE_EX) {
    const double posxh = (i + 0.5 - q.centre[0]) * q.dx;
    const double posyo = (j - q.centre[1]) * q.dy;
    const double poszo = (l - q.centre[2]) * q.dz - q.zshift;
    const double t = (double)q.time * q.dt - q.tshift;
    return q.amp * short_pulse_e(sp, posxh, posyo, poszo, t).re;
  }
  const double poszh = (l - 0.5 - q.centre[2]) * q.dz - q.zshift;
  const double t = ((double)q.time - 0.5) * q.dt - q.tshift;
  if (PART == PULSE_BX) {
    const double posxo = (i - q.centre[0]) * q.dx;
    const double posyh = (j + 0.5 - q.centre[1]) * q.dy;
    return q.amp * short_pulse_b(sp, posxo, posyh, poszh, t, true).re;
  }
  const double posxh = (i + 0.5 - q.centre[0]) * q.dx;
  const double posyo = (j - q.centre[1]) * q.dy;
  return q.amp * short_pulse_b(sp, posxh, posyo, poszh, t, false).re;
}

// GaussInjectSourceFunc::getHField / getEField (gaussinject.cpp:204-222) on
// the block precomputed by mp_gauss_kernels.cu.
__device__ void gauss_beam_field(const SourceEvalParams &q, int i, int j, double out[3]) {
  out[0] = out[1] = out[2] = 0.0;
  if (!q.g_active) return;
  const long long o = (q.time - q.g_toff) * ((long long)q.nx * q.ny) + (long long)j * q.nx + i;
  out[0] = q.g_scale * q.g_f1[o];
  if (q.isH) out[1] = q.g_scale * q.g_f2[o];
}

// The incident field of every other kind at interior column (i, j) (0-based; MPulse
// i + 1, j + 1).
__device__ void source_field(const SourceEvalParams &q, int i, int j, double f[3]) {
  if (q.kind == 5) gauss_beam_field(q, i, j, f);
  else plane_source_field(q, i + 1, j + 1, q.l, f);
}

// The planes of `nsteps` consecutive steps at once: the values depend only on
// Process::time, so step t0 + q's E-side pair goes to out + (4 q + 0, 1) * plane
// and its H-side pair to out + (4 q + 2, 3) * plane, each pair (J0, J1) = (F[t2],
// F[t1]) / DX with (t1, t2) = (x, y) on z faces.
template <typename T>
__global__ void __launch_bounds__(256) source_batch_kernel(const SourceEvalParams qe, const SourceEvalParams qh,
                                                          long long t0, T *out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= qe.nx || j >= qe.ny) return;
  const int step = blockIdx.z >> 1, side = blockIdx.z & 1;
  SourceEvalParams q = side ? qh : qe;
  q.time = t0 + step;
  double f[3];
  source_field(q, i, j, f);
  const long long plane = (long long)qe.nx * qe.ny;
  const long long col = (long long)j * qe.nx + i;
  T *v0 = out + (4LL * step + 2 * side) * plane;
  v0[col] = T(f[1] / q.DX);
  v0[plane + col] = T(f[0] / q.DX);
}

// The short pulse is centred on the plane, so its fields are even (Ex, By) or odd
// (Bx) in x and in y, exactly, and a quarter of the plane is evaluated.  Along an
// axis of n cells the points on cells (i - (n + 1) / 2) pair as i and n + 1 - i, the
// points half a cell on as i and n - i, with i = n left over: thread t of
// 1 .. n / 2 + 1 takes cell *i and its partner *m (*m = *i: none).
__device__ __forceinline__ bool mirror_pair(int t, int n, bool half, int *i, int *m) {
  *i = t;
  if (!half) {
    *m = n + 1 - t;
    return t <= (n + 1) / 2;
  }
  *m = n - t;
  if (t == n / 2 + 1) *i = *m = n;
  return t <= n / 2 + 1;
}

// One component over its quarter: value / DX to the plane at `out` and, with the
// component's parity, to the partners.
template <PulsePart PART, typename T>
__device__ __forceinline__ void pulse_quarter(const SourceEvalParams &q, int tx, int ty, T *out) {
  constexpr bool kHalfX = PART != PULSE_BX, kHalfY = PART == PULSE_BX;
  int i, im, j, jm;
  if (!mirror_pair(tx, q.nx, kHalfX, &i, &im) || !mirror_pair(ty, q.ny, kHalfY, &j, &jm)) return;
  const double f = short_pulse_part<PART>(q, i, j, q.l) / q.DX;
  const T v = T(f), w = PART == PULSE_BX ? T(-f) : v;
  out[(long long)(jm - 1) * q.nx + im - 1] = v;
  out[(long long)(jm - 1) * q.nx + i - 1] = jm == j ? v : w;
  out[(long long)(j - 1) * q.nx + im - 1] = im == i ? v : w;
  out[(long long)(j - 1) * q.nx + i - 1] = v;
}

// One component of the short pulse for a batch of steps (blockIdx.z), laid out as
// source_batch_kernel does; Ex brings the zero plane beside it.  The closed forms are
// long FP64 expressions (about 200 registers unbounded, one block of 256 threads per
// SM): MPB_SRC_MIN_BLOCKS blocks per SM trade spills for occupancy (the whole plane
// of 256 x 256 with 1 / 2 / 3 / 4 blocks per SM 0.042 / 0.0196 / 0.0183 / 0.0194 ms per
// step).  Whole planes took 17.4 us a step (64-step batches, beside the step kernels
// on another stream), quarters, one kernel per component, 6.5.
#ifndef MPB_SRC_MIN_BLOCKS
#define MPB_SRC_MIN_BLOCKS 3
#endif
template <typename T, PulsePart PART>
__global__ void __launch_bounds__(256, MPB_SRC_MIN_BLOCKS) pulse_batch_kernel(const SourceEvalParams qs, long long t0,
                                                                              T *out) {
  const int tx = blockIdx.x * blockDim.x + threadIdx.x + 1, ty = blockIdx.y * blockDim.y + threadIdx.y + 1;
  const long long plane = (long long)qs.nx * qs.ny;
  T *v = out + 4LL * blockIdx.z * plane;  // By, Bx (E side), Ey = 0, Ex (H side)
  SourceEvalParams q = qs;
  q.time = t0 + blockIdx.z;
  pulse_quarter<PART>(q, tx, ty, v + (PART == PULSE_BY ? 0 : PART == PULSE_BX ? 1 : 3) * plane);
  if (PART == PULSE_EX) {  // four cells of the zero plane per thread
    const int i = 2 * tx - 1, j = 2 * ty - 1;
    for (int dj = 0; dj < 2; ++dj)
      for (int di = 0; di < 2; ++di)
        if (i + di <= q.nx && j + dj <= q.ny) v[2 * plane + (long long)(j + dj - 1) * q.nx + i + di - 1] = T(0);
  }
}

// Kernels of one batch.
int source_batch_launches(const SourceEvalParams &q) { return q.kind == 3 || q.kind == 4 ? 3 : 1; }

template <typename T>
cudaError_t launch_source_batch(const SourceEvalParams &qe, const SourceEvalParams &qh, long long t0, int nsteps,
                                T *out, cudaStream_t st) {
  const dim3 b(32, 8, 1);
  if (qe.kind == 3 || qe.kind == 4) {  // short / focused pulse
    const dim3 g((qe.nx / 2 + 1 + 31) / 32, (qe.ny / 2 + 1 + 7) / 8, nsteps);
    pulse_batch_kernel<T, PULSE_BY><<<g, b, 0, st>>>(qe, t0, out);
    pulse_batch_kernel<T, PULSE_BX><<<g, b, 0, st>>>(qe, t0, out);
    pulse_batch_kernel<T, PULSE_EX><<<g, b, 0, st>>>(qh, t0, out);
    return cudaGetLastError();
  }
  const dim3 g((qe.nx + 31) / 32, (qe.ny + 7) / 8, 2 * nsteps);
  source_batch_kernel<T><<<g, b, 0, st>>>(qe, qh, t0, out);
  return cudaGetLastError();
}

template cudaError_t launch_source_batch<float>(const SourceEvalParams &, const SourceEvalParams &, long long, int,
                                                float *, cudaStream_t);
template cudaError_t launch_source_batch<double>(const SourceEvalParams &, const SourceEvalParams &, long long, int,
                                                 double *, cudaStream_t);

}  // namespace mpb
