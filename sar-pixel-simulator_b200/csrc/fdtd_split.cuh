// fdtd_split.cuh -- the split step's H and E updates of one vector, for the
// split passes (fdtd_split.cu), and the phasor update of one cell, which the
// resident step (fdtd_resident.cu) shares.
#pragma once

#include "fdtd_vec.cuh"

namespace fdtd {

// H pass on one vector: H^{n+1/2} = H^{n-1/2} - Db curl E^n, CPML and
// E-field injection. Reads E and H from the source pointers and writes H
// (and psi_H) to the destination pointers, so it serves both the in-place
// step (source == destination) and the ping-pong shell of the fused step.
// `lane` is the thread's position in a row segment of `width` lanes
// (width * kVec consecutive x cells); every lane of the segment calls this
// (the +x neighbour comes by shuffle), and only lanes with `act` update
// and store their vector.
template <class T>
__device__ __forceinline__ void h_split_vec(const State<T>& s, int t, int z, int y, int x0,
                                            int lane, int width, bool act) {
  const bool vin = x0 < s.pitch && y < s.ny;          // vector inside the row storage
  const long long P = s.plane, W = s.pitch;
  const long long i = (long long)z * P + (long long)y * W + x0;
  const bool plain = interior(s, z, y, x0, t);
  if (act && vin && !plain) h_psi_prefetch(s, z, y, x0);
  EVec<T> e;
  T hx[kVec], hy[kVec], hz[kVec];
  if (vin) {
    ld4(e.ex, s.iex + i); ld4(e.ey, s.iey + i); ld4(e.ez, s.iez + i);
    ld4(hx, s.ihx + i); ld4(hy, s.ihy + i); ld4(hz, s.ihz + i);
  } else {
    zero4(e.ex); zero4(e.ey); zero4(e.ez); zero4(hx); zero4(hy); zero4(hz);
  }
  if (vin && y + 1 < s.ny) { ld4(e.exy, s.iex + i + W); ld4(e.ezy, s.iez + i + W); }
  else { zero4(e.exy); zero4(e.ezy); }
  if (vin && z + 1 < s.nz) { ld4(e.exz, s.iex + i + P); ld4(e.eyz, s.iey + i + P); }
  else { zero4(e.exz); zero4(e.eyz); }
  // x+1 neighbour of the last cell: first cell of the next lane's vector
  e.eyn = __shfl_down_sync(0xffffffffu, e.ey[0], 1, width);
  e.ezn = __shfl_down_sync(0xffffffffu, e.ez[0], 1, width);
  if (lane == width - 1) {
    const bool ok = vin && x0 + kVec < s.nx;
    e.eyn = ok ? ldc(s.iey + (i + kVec)) : T(0);
    e.ezn = ok ? ldc(s.iez + (i + kVec)) : T(0);
  }
  if (!(act && vin)) return;
  if (plain) h_vec_interior(s, e, hx, hy, hz);
  else h_vec(s, e, z, y, x0, t, true, hx, hy, hz);
  st4(s.ohx + i, hx); st4(s.ohy + i, hy); st4(s.ohz + i, hz);
}

// E pass on one vector: E^{n+1} = Ca E^n + Cb curl H^{n+1/2}, CPML and
// H-field injection. Reads H^{n+1/2} and E^n from the source pointers and
// writes E (and psi_E) to the destination pointers.
template <class T>
__device__ __forceinline__ void e_split_vec(const State<T>& s, int t, int z, int y, int x0,
                                            int lane, int width, bool act) {
  const bool vin = x0 < s.pitch && y < s.ny;
  const long long P = s.plane, W = s.pitch;
  const long long i = (long long)z * P + (long long)y * W + x0;
  const bool plain = interior(s, z, y, x0, t);
  if (act && vin && !plain) e_psi_prefetch(s, z, y, x0);
  HVec<T> h;
  T ex[kVec], ey[kVec], ez[kVec], ca[kVec], cb[kVec];
  if (vin) {
    ld4(h.hx, s.ihx + i); ld4(h.hy, s.ihy + i); ld4(h.hz, s.ihz + i);
    ld4(ex, s.iex + i); ld4(ey, s.iey + i); ld4(ez, s.iez + i);
    ld4(ca, s.ca + i); ld4(cb, s.cb + i);
  } else {
    zero4(h.hx); zero4(h.hy); zero4(h.hz); zero4(ex); zero4(ey); zero4(ez); zero4(ca); zero4(cb);
  }
  if (vin && y >= 1) { ld4(h.hxy, s.ihx + i - W); ld4(h.hzy, s.ihz + i - W); }
  else { zero4(h.hxy); zero4(h.hzy); }
  if (vin && z >= 1) { ld4(h.hxz, s.ihx + i - P); ld4(h.hyz, s.ihy + i - P); }
  else { zero4(h.hxz); zero4(h.hyz); }
  // x-1 neighbour of the first cell: last cell of the previous lane's vector
  h.hyp = __shfl_up_sync(0xffffffffu, h.hy[kVec - 1], 1, width);
  h.hzp = __shfl_up_sync(0xffffffffu, h.hz[kVec - 1], 1, width);
  if (lane == 0) {
    const bool ok = vin && x0 >= 1;
    h.hyp = ok ? ldc(s.ihy + (i - 1)) : T(0);
    h.hzp = ok ? ldc(s.ihz + (i - 1)) : T(0);
  }
  if (!(act && vin)) return;
  if (plain) e_vec_interior(h, ca, cb, ex, ey, ez);
  else e_vec(s, h, ca, cb, z, y, x0, t, true, ex, ey, ez);
  st4(s.oex + i, ex); st4(s.oey + i, ey); st4(s.oez + i, ez);
}

// ---------------------------------------------------------------------------
// phasors (cpu/field_updates.py:373-461, gpu/field_updates.py:680-906)
// ---------------------------------------------------------------------------
template <class T>
__device__ __forceinline__ void ph_acc(const State<T>& s, int plane, long long k,
                                       double m, double c, double sn) {
  using M = R<T>;
  T* p = s.ph + s.ph_off[plane] + 2 * k;
  if (!s.kahan) {
    // float64 sum of the stored value and the float64 term, rounded to T
    stc(p, M::from_double(__dadd_rn((double)ldc(p), __dmul_rn(m, c))));
    stc(p + 1, M::from_double(__dadd_rn((double)ldc(p + 1), __dmul_rn(m, sn))));
  } else {
    T* pc = s.phc + s.ph_off[plane] + 2 * k;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const T term = M::from_double(__dmul_rn(m, j ? sn : c));
      const T yv = M::sub(term, ldc(pc + j));
      const T pj = ldc(p + j);
      const T tv = M::add(pj, yv);
      stc(pc + j, M::sub(M::sub(tv, pj), yv));
      stc(p + j, tv);
    }
  }
}

template <class T>
__device__ __forceinline__ double mean2(T a, T b) {
  return 0.5 * (double)R<T>::add(a, b);
}
template <class T>
__device__ __forceinline__ double mean4(T a, T b, T c, T d) {
  using M = R<T>;
  return 0.25 * (double)M::add(M::add(M::add(a, b), c), d);
}

// one complex phasor value (re, im) as a single 8-byte (float) or 16-byte
// (double) access: planes start at even element offsets of an aligned base
template <class T>
__device__ __forceinline__ void ld2(T (&d)[2], const T* p) {
  if (!FDTD_CHECK_PTR(p, 2 * (int)sizeof(T))) {   // bounds-checked build only
    d[0] = d[1] = T(0);
    return;
  }
  if constexpr (sizeof(T) == 4) {
    const float2 v = *reinterpret_cast<const float2*>(p);
    d[0] = v.x; d[1] = v.y;
  } else {
    const double2 v = *reinterpret_cast<const double2*>(p);
    d[0] = v.x; d[1] = v.y;
  }
}

template <class T>
__device__ __forceinline__ void st2(T* p, T re, T im) {
  if (!FDTD_CHECK_PTR(p, 2 * (int)sizeof(T))) return;   // bounds-checked build only
  if constexpr (sizeof(T) == 4) *reinterpret_cast<float2*>(p) = make_float2(re, im);
  else *reinterpret_cast<double2*>(p) = make_double2(re, im);
}

// The four components of one phasor cell: base plane `base`, field means
// m[0..3] (E, E, H, H). Every load (the four stored values) is issued before
// any store, so the cell costs one memory round trip rather than four.
template <class T>
__device__ __forceinline__ void ph_acc4(const State<T>& s, int base, long long k, const double (&m)[4],
                                        double cE, double sE, double cH, double sH) {
  using M = R<T>;
  if (s.kahan) {
#pragma unroll
    for (int j = 0; j < 4; ++j) ph_acc(s, base + j, k, m[j], j < 2 ? cE : cH, j < 2 ? sE : sH);
    return;
  }
  T v[4][2];
#pragma unroll
  for (int j = 0; j < 4; ++j) ld2(v[j], s.ph + s.ph_off[base + j] + 2 * k);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const double c = j < 2 ? cE : cH, sn = j < 2 ? sE : sH;
    // float64 sum of the stored value and the float64 term, rounded to T
    st2(s.ph + s.ph_off[base + j] + 2 * k, M::from_double(__dadd_rn((double)v[j][0], __dmul_rn(m[j], c))),
        M::from_double(__dadd_rn((double)v[j][1], __dmul_rn(m[j], sn))));
  }
}

// The six fields a phasor plane averages.
template <class T>
struct PhFields {
  const T* ex; const T* ey; const T* ez;
  const T* hx; const T* hy; const T* hz;
};

// The field means (E, E, H, H) of one phasor cell of plane group g (0 d, 1 u:
// z planes, components ex, ey, hx, hy; 2 l, 3 r: x planes, ey, ez, hy, hz;
// 4 f, 5 b: y planes, ex, ez, hx, hz) from those components at index i, with
// the strides P of z and W of y.
template <class T>
__device__ __forceinline__ void phasor_means(int g, const T* e0, const T* e1, const T* h0, const T* h1, long long i,
                                             long long P, long long W, double (&mv)[4]) {
  if (g < 2) {
    mv[0] = mean2(ldc(e0 + i), ldc(e0 + i - 1));
    mv[1] = mean2(ldc(e1 + i), ldc(e1 + i - W));
    mv[2] = mean4(ldc(h0 + i), ldc(h0 + i - W), ldc(h0 + i - P), ldc(h0 + i - P - W));
    mv[3] = mean4(ldc(h1 + i), ldc(h1 + i - 1), ldc(h1 + i - P), ldc(h1 + i - P - 1));
  } else if (g < 4) {
    mv[0] = mean2(ldc(e0 + i), ldc(e0 + i - W));
    mv[1] = mean2(ldc(e1 + i), ldc(e1 + i - P));
    mv[2] = mean4(ldc(h0 + i), ldc(h0 + i - 1), ldc(h0 + i - P), ldc(h0 + i - P - 1));
    mv[3] = mean4(ldc(h1 + i), ldc(h1 + i - 1), ldc(h1 + i - W), ldc(h1 + i - W - 1));
  } else {
    mv[0] = mean2(ldc(e0 + i), ldc(e0 + i - 1));
    mv[1] = mean2(ldc(e1 + i), ldc(e1 + i - P));
    mv[2] = mean4(ldc(h0 + i), ldc(h0 + i - W), ldc(h0 + i - P), ldc(h0 + i - P - W));
    mv[3] = mean4(ldc(h1 + i), ldc(h1 + i - W), ldc(h1 + i - 1), ldc(h1 + i - W - 1));
  }
}

// The same of cell (a, b) of the group's plane, from whole fields.
template <class T>
__device__ __forceinline__ void phasor_means(const State<T>& s, const PhFields<T>& f, int g, int a, int b,
                                             double (&mv)[4]) {
  const int m = s.npml;
  const long long P = s.plane, W = s.pitch;
  if (g < 2) {
    const int pz = g == 0 ? m + 1 : s.nz - m - 1;
    phasor_means(g, f.ex, f.ey, f.hx, f.hy, pz * P + (long long)(m + a) * W + (m + b), P, W, mv);
  } else if (g < 4) {
    const int px = g == 2 ? m + 1 : s.nx - m - 1;
    phasor_means(g, f.ey, f.ez, f.hy, f.hz, (long long)(m + a) * P + (long long)(m + b) * W + px, P, W, mv);
  } else {
    const int py = g == 4 ? m + 1 : s.ny - m - 1;
    phasor_means(g, f.ex, f.ez, f.hx, f.hz, (long long)(m + a) * P + (long long)py * W + (m + b), P, W, mv);
  }
}

// One phasor cell of plane group g; idx runs over the group's plane. False
// when idx is past the plane or on its first row or column, which no
// phasor accumulates.
template <class T>
__device__ __forceinline__ bool phasor_at(const State<T>& s, int g, int idx, int& a, int& b) {
  int d0, d1;
  if (g < 2) { d0 = s.ny_ph; d1 = s.nx_ph; }
  else if (g < 4) { d0 = s.nz_ph; d1 = s.ny_ph; }
  else { d0 = s.nz_ph; d1 = s.nx_ph; }
  if (idx >= d0 * d1) return false;
  a = idx / d1;
  b = idx - a * d1;
  return a != 0 && b != 0;
}

// The field loads of all four components come first, then the update.
template <class T>
__device__ __forceinline__ void phasor_cell(const State<T>& s, const PhFields<T>& f, int g, int idx, int t) {
  int a, b;
  if (!phasor_at(s, g, idx, a, b)) return;
  const double* ph = s.phase + 4 * (long long)t;
  const double cE = ph[0], sE = ph[1], cH = ph[2], sH = ph[3];
  double mv[4];
  phasor_means(s, f, g, a, b, mv);
  ph_acc4(s, 4 * g, idx, mv, cE, sE, cH, sH);
}
template <class T>
__device__ __forceinline__ void phasor_cell(const State<T>& s, int g, int idx, int t) {
  phasor_cell(s, PhFields<T>{s.oex, s.oey, s.oez, s.ohx, s.ohy, s.ohz}, g, idx, t);
}

}  // namespace fdtd
