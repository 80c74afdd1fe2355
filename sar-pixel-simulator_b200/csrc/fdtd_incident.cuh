// fdtd_incident.cuh -- what the incident run does beside its steps: the hard
// source's cells and the read-out plane (recorded planes, incident phasors),
// for the kernels of fdtd_incident.cu and the resident run.
#pragma once

#include "fdtd_launch.h"

namespace fdtd {

// cells of plane feed_in that the source sets
template <class T>
__device__ __forceinline__ bool inc_source_cell(const State<T>& s, int y, int x) {
  return x < s.nx - 1 && y >= 1 && y < s.ny - 1;
}

template <class T>
__device__ __forceinline__ void inc_acc(T* p, double m, double c, double sn) {
  // float64 sum of the stored value and the float64 term, rounded to T
  p[0] = R<T>::from_double(__dadd_rn((double)p[0], __dmul_rn(m, c)));
  p[1] = R<T>::from_double(__dadd_rn((double)p[1], __dmul_rn(m, sn)));
}

// Read-out plane of step t at (y, x) into the recorded planes (all y, x) and
// the incident phasors of cpu/field_updates.py:465-491 at (y, x) in
// [1, ny_ph) x [1, nx_ph): E averaged with phase exp(-i omega (t - 1/2) dt),
// H with exp(-i omega t dt) (phase table columns 2-3 and 0-1).
template <class T>
__device__ __forceinline__ void inc_record_e(const IncidentRecord<T>& r, const T* ex, const T* ey, int t, int y, int x) {
  const long long W = r.pitch;
  const long long i = (long long)r.read_out * r.plane + (long long)y * W + x;
  const long long o = ((long long)t * r.ny + y) * W + x;
  r.rex[o] = ex[i];
  r.rey[o] = ey[i];
  const int a = y - r.npml, b = x - r.npml;
  if (a < 1 || b < 1 || a >= r.ny_ph || b >= r.nx_ph) return;
  const double* ph = r.phase + 4 * (long long)t;
  using M = R<T>;
  const long long k = 2 * ((long long)a * r.nx_ph + b), n = 2 * (long long)r.ny_ph * r.nx_ph;
  inc_acc(r.ph + k, 0.5 * (double)M::add(ex[i], ex[i - 1]), ph[2], ph[3]);
  inc_acc(r.ph + n + k, 0.5 * (double)M::add(ey[i], ey[i - W]), ph[2], ph[3]);
}
template <class T>
__device__ __forceinline__ void inc_record_h(const IncidentRecord<T>& r, const T* hx, const T* hy, int t, int y, int x) {
  const long long P = r.plane, W = r.pitch;
  const long long i = (long long)r.read_out * P + (long long)y * W + x;
  const long long o = ((long long)t * r.ny + y) * W + x;
  r.rhx[o] = hx[i];
  r.rhy[o] = hy[i];
  const int a = y - r.npml, b = x - r.npml;
  if (a < 1 || b < 1 || a >= r.ny_ph || b >= r.nx_ph) return;
  const double* ph = r.phase + 4 * (long long)t;
  using M = R<T>;
  const long long k = 2 * ((long long)a * r.nx_ph + b), n = 2 * (long long)r.ny_ph * r.nx_ph;
  inc_acc(r.ph + 2 * n + k, 0.25 * (double)M::add(M::add(M::add(hx[i], hx[i - W]), hx[i - P]), hx[i - P - W]), ph[0],
          ph[1]);
  inc_acc(r.ph + 3 * n + k, 0.25 * (double)M::add(M::add(M::add(hy[i], hy[i - 1]), hy[i - P]), hy[i - P - 1]), ph[0],
          ph[1]);
}

}  // namespace fdtd
