// fdtd_adjoint.cu -- the transposed (adjoint) FDTD step.
//
// The forward step is linear in the fields and the CPML auxiliaries:
//   H' = H - Db curl_E(E) + CPML_H(psi_H'),   psi_H' = bh psi_H + (ch/dx) dE
//   E' = Ca E + Cb curl_H(H') + Cb dx CPML_E(psi_E'),  psi_E' = be psi_E + (ce/dx) dH'
// and the phasors are running sums of plane averages. Reverse-mode
// differentiation of one step is therefore the transposed step run
// backwards in time: the adjoint fields (lambda) of the step's outputs give
// the adjoint fields of its inputs and the step's contribution to
// dJ/dCa = sum_n lambda_E^{n+1} . E^n and dJ/dCb = sum_n lambda_E^{n+1} .
// (curl_H(H^{n+1/2}) + dx psi_E^{n+1}). The transposed curls are the
// backward-difference (for H -> E) and forward-difference (for E -> H)
// stencils of the forward step, with the forward step's index ranges moved
// onto the neighbour that owned the term.
//
// Every kernel is written in gather form (each thread writes only its own
// cell). The reverse sweep of step n is, in order:
//   a. lambda_E on the upper phasor plane += dJ/dE^{n+1}
//   b. lambda_H += (E update and E CPML)^T lambda_E
//   c. gradients; psi_E adjoint; lambda_E = Ca lambda_E
//   d. lambda_H on the two planes += dJ/dH^{n+1/2}
//   e. lambda_E += (H update and H CPML)^T lambda_H
//   f. psi_H adjoint
// b reads lambda_E and the E auxiliaries' adjoint of neighbours before c
// overwrites them; e reads lambda_H and the H auxiliaries' adjoint of
// neighbours before f overwrites them. Two kernels per step do all six:
// k_adj_k1 = f of step n + 1, b, d; k_adj_k2 = c, e, a of step n - 1; only
// the first backward step needs a on its own (k_adj_phasor_e).
#include "fdtd_launch.h"
#include "fdtd_vec.cuh"

namespace fdtd {

namespace {

// index ranges of the forward main updates (cpu/field_updates.py:18-63,
// 198-240)
template <class T>
__device__ __forceinline__ bool re_x(const State<T>& s, int z, int y, int x) {
  return z >= 1 && z < s.nz - 1 && y >= 1 && y < s.ny - 1 && x >= 0 && x < s.nx - 1;
}
template <class T>
__device__ __forceinline__ bool re_y(const State<T>& s, int z, int y, int x) {
  return z >= 1 && z < s.nz - 1 && y >= 0 && y < s.ny - 1 && x >= 1 && x < s.nx - 1;
}
template <class T>
__device__ __forceinline__ bool re_z(const State<T>& s, int z, int y, int x) {
  return z >= 0 && z < s.nz - 1 && y >= 1 && y < s.ny - 1 && x >= 1 && x < s.nx - 1;
}
template <class T>
__device__ __forceinline__ bool rh_x(const State<T>& s, int z, int y, int x) {
  return z >= 0 && z < s.nz - 1 && y >= 0 && y < s.ny - 1 && x >= 1 && x < s.nx - 1;
}
template <class T>
__device__ __forceinline__ bool rh_y(const State<T>& s, int z, int y, int x) {
  return z >= 0 && z < s.nz - 1 && y >= 1 && y < s.ny - 1 && x >= 0 && x < s.nx - 1;
}
template <class T>
__device__ __forceinline__ bool rh_z(const State<T>& s, int z, int y, int x) {
  return z >= 1 && z < s.nz - 1 && y >= 0 && y < s.ny - 1 && x >= 0 && x < s.nx - 1;
}
template <class T>
__device__ __forceinline__ bool box(const State<T>& s, int z, int y, int x) {
  return z >= 0 && y >= 0 && x >= 0 && z < s.nz - 1 && y < s.ny - 1 && x < s.nx - 1;
}

// CPML face membership of a cell: side (0 low, 1 high) and profile index q,
// or false. E faces: 1 <= i < m low, i >= n - m high; H faces: i < m - 1
// low, i >= n - m high (cpu/field_updates.py:66-366); both inside the box.
__device__ __forceinline__ bool e_face(int i, int n, int m, int& side, int& q) {
  if (i >= 1 && i < m) { side = 0; q = i; return true; }
  if (i >= n - m) { side = 1; q = i - (n - m); return true; }
  return false;
}
__device__ __forceinline__ bool h_face(int i, int n, int m, int& side, int& q) {
  if (i >= 0 && i < m - 1) { side = 0; q = i; return true; }
  if (i >= n - m) { side = 1; q = i - (n - m); return true; }
  return false;
}

template <class T>
__device__ __forceinline__ long long idx(const State<T>& s, int z, int y, int x) {
  return ((long long)z * s.ny + y) * s.pitch + x;
}

// psi element of each face layout (z: (m, ny, pitch), x: (nz, ny, m),
// y: (nz, m, pitch))
template <class T>
__device__ __forceinline__ long long kz(const State<T>& s, int q, int y, int x) {
  return ((long long)q * s.ny + y) * s.pitch + x;
}
template <class T>
__device__ __forceinline__ long long kx(const State<T>& s, int z, int y, int side, int q) {
  return xpsi_index(s, z, y, side, side ? q + (s.nx - s.npml) : q);
}
template <class T>
__device__ __forceinline__ long long ky(const State<T>& s, int z, int q, int x) {
  return ((long long)z * s.npml + q) * s.pitch + x;
}

}  // namespace

// ---- 1 / 4: phasor sources -------------------------------------------------
// p(a, b) += avg(F)(a, b) (c + i s) for a in [1, ny_ph), b in [1, nx_ph),
// F sampled around (m + a, m + b) on plane nz - m - 1 (cpu/field_updates.py:
// 373-461, the upper plane). dJ/dF = g_re c + g_im s spread back over the
// averaged samples.
template <class T>
__device__ __forceinline__ double ph_g(const Adj<T>& a, int comp, int ia, int ib, int nyp, int nxp,
                                       double c, double sn) {
  if (ia < 1 || ib < 1 || ia >= nyp || ib >= nxp) return 0.0;
  const long long k = ((long long)comp * nyp + ia) * nxp + ib;
  return a.g_re[k] * c + a.g_im[k] * sn;
}

// phasor E source of step t at cell (z, y, x): (d ex, d ey)
template <class T>
__device__ __forceinline__ void phasor_e_src(const State<T>& s, const Adj<T>& a, int t, int z, int y,
                                             int x, T& dex, T& dey) {
  dex = T(0);
  dey = T(0);
  const int m = s.npml;
  if (z != s.nz - m - 1) return;
  const double* ph = s.phase + 4 * (long long)t;
  const double c = ph[0], sn = ph[1];
  const int ia = y - m, ib = x - m;
  const double gx = ph_g(a, 0, ia, ib, s.ny_ph, s.nx_ph, c, sn) + ph_g(a, 0, ia, ib + 1, s.ny_ph, s.nx_ph, c, sn);
  const double gy = ph_g(a, 1, ia, ib, s.ny_ph, s.nx_ph, c, sn) + ph_g(a, 1, ia + 1, ib, s.ny_ph, s.nx_ph, c, sn);
  dex = (T)(0.5 * gx);
  dey = (T)(0.5 * gy);
}

// phasor H source of step t at cell (z, y, x): (d hx, d hy), planes pz - 1, pz
template <class T>
__device__ __forceinline__ void phasor_h_src(const State<T>& s, const Adj<T>& a, int t, int z, int y,
                                             int x, T& dhx, T& dhy) {
  dhx = T(0);
  dhy = T(0);
  const int m = s.npml, pz = s.nz - m - 1;
  if (z != pz && z != pz - 1) return;
  const double* ph = s.phase + 4 * (long long)t;
  const double c = ph[2], sn = ph[3];
  const int ia = y - m, ib = x - m;
  const double gx = ph_g(a, 2, ia, ib, s.ny_ph, s.nx_ph, c, sn) + ph_g(a, 2, ia + 1, ib, s.ny_ph, s.nx_ph, c, sn);
  const double gy = ph_g(a, 3, ia, ib, s.ny_ph, s.nx_ph, c, sn) + ph_g(a, 3, ia, ib + 1, s.ny_ph, s.nx_ph, c, sn);
  dhx = (T)(0.25 * gx);
  dhy = (T)(0.25 * gy);
}

// standalone E source of the first backward step (the later ones are added
// by k_adj_k2 of the step after them)
template <class T>
__global__ void k_adj_phasor_e(const __grid_constant__ State<T> s, Adj<T> a, int t) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= s.nx || y >= s.ny) return;
  const int z = s.nz - s.npml - 1;
  T dex, dey;
  phasor_e_src(s, a, t, z, y, x, dex, dey);
  const long long i = idx(s, z, y, x);
  if (re_x(s, z, y, x)) a.lex[i] += dex;
  if (re_y(s, z, y, x)) a.ley[i] += dey;
}

// ---- vector form ------------------------------------------------------------
// A thread owns two consecutive x cells of one row (x0 even; the pitch is a
// multiple of 32 elements, so the two are one aligned vector in every (..,
// pitch)-strided array). z- and y-face auxiliaries have coefficients uniform
// over the vector; x-face auxiliaries ((z, y, npml) layout) run per cell.
//
// Two cells, not the forward step's four: the kernels are bound by latency
// (IPC 1 at 96 and 128 registers with four cells, 16 to 20 warps per SM),
// and two cells take half the registers, 64 and 72. The backward half per
// step with four and two cells, us: 55 x 133 x 133 cells float 82 and 72,
// 81 x 231 x 229 381 and 308, 39 x 61 x 57 29 and 26, 55 x 133 x 133 double
// 201 and 149 (one cell, 55 x 133 x 133 float: 75). Blocks per SM: 8 and 7
// for float (2 to 3 us better than 10 and 8; no minimum: 8 us worse), 7 and
// 6 for double (5 and 4: 156, none: 163).
constexpr int kAdj = 2;

template <class T>
struct alignas(kAdj * sizeof(T)) AdjVec {
  T v[kAdj];
};

template <class T>
__device__ __forceinline__ void zero_adj(T (&d)[kAdj]) {
#pragma unroll
  for (int j = 0; j < kAdj; ++j) d[j] = T(0);
}

template <class T>
__device__ __forceinline__ void ld_adj(T (&d)[kAdj], const T* p) {
  if (!FDTD_CHECK_PTR(p, (int)sizeof(T) * kAdj)) {   // bounds-checked build only
    zero_adj(d);
    return;
  }
  const AdjVec<T> q = *reinterpret_cast<const AdjVec<T>*>(p);
#pragma unroll
  for (int j = 0; j < kAdj; ++j) d[j] = q.v[j];
}

template <class T>
__device__ __forceinline__ void st_adj(T* p, const T (&d)[kAdj]) {
  if (!FDTD_CHECK_PTR(p, (int)sizeof(T) * kAdj)) return;   // bounds-checked build only
  AdjVec<T> q;
#pragma unroll
  for (int j = 0; j < kAdj; ++j) q.v[j] = d[j];
  *reinterpret_cast<AdjVec<T>*>(p) = q;
}

// main-update ranges of the E components of the vector's cells
template <class T>
__device__ __forceinline__ void e_ranges(const State<T>& s, int z, int y, int x0, bool (&rx)[kAdj],
                                         bool (&ry)[kAdj], bool (&rz)[kAdj]) {
  const bool zi = z >= 1 && z < s.nz - 1, yi = y >= 1 && y < s.ny - 1;
  const bool zb = z >= 0 && z < s.nz - 1, yb = y >= 0 && y < s.ny - 1;
#pragma unroll
  for (int j = 0; j < kAdj; ++j) {
    const int x = x0 + j;
    const bool xb = x < s.nx - 1, xi = x >= 1 && x < s.nx - 1;
    rx[j] = zi && yi && xb;
    ry[j] = zi && yb && xi;
    rz[j] = zb && yi && xi;
  }
}

// and of the H components
template <class T>
__device__ __forceinline__ void h_ranges(const State<T>& s, int z, int y, int x0, bool (&rx)[kAdj],
                                         bool (&ry)[kAdj], bool (&rz)[kAdj]) {
  const bool zi = z >= 1 && z < s.nz - 1, yi = y >= 1 && y < s.ny - 1;
  const bool zb = z >= 0 && z < s.nz - 1, yb = y >= 0 && y < s.ny - 1;
#pragma unroll
  for (int j = 0; j < kAdj; ++j) {
    const int x = x0 + j;
    const bool xb = x < s.nx - 1, xi = x >= 1 && x < s.nx - 1;
    rx[j] = zb && yb && xi;
    ry[j] = zb && yi && xb;
    rz[j] = zi && yb && xb;
  }
}

// F = Cb lambda_E of one component where `r` holds
template <class T>
__device__ __forceinline__ void masked_prod(T (&f)[kAdj], const T (&cb)[kAdj], const T (&l)[kAdj],
                                            const bool (&r)[kAdj]) {
#pragma unroll
  for (int j = 0; j < kAdj; ++j) f[j] = r[j] ? cb[j] * l[j] : T(0);
}

// E-face auxiliaries of plane zz (z faces) or row yy (y faces): c/dx times
// their total adjoint lambda_psi + sign Cb dx lambda_E, zero off the faces
// and outside the box. With F = Cb lambda_E of the two components involved.
// z faces: t0 Exz (F = fx, sign -), t1 Eyz (fy, +).
template <class T>
__device__ __forceinline__ void e_zface(const State<T>& s, const Adj<T>& a, int zz, int y, int x0,
                                        const T (&fx)[kAdj], const T (&fy)[kAdj], T (&t0)[kAdj],
                                        T (&t1)[kAdj]) {
  zero_adj(t0);
  zero_adj(t1);
  int side, q;
  if (zz >= s.nz - 1 || y >= s.ny - 1 || !e_face(zz, s.nz, s.npml, side, q)) return;
  const long long k = kz(s, q, y, x0);
  const T c = s.prof[side ? CE_U : CE_D][q] * s.rdx;
  T p0[kAdj], p1[kAdj];
  ld_adj(p0, a.lps.z[side][0] + k);
  ld_adj(p1, a.lps.z[side][1] + k);
#pragma unroll
  for (int j = 0; j < kAdj; ++j) {
    if (x0 + j >= s.nx - 1) continue;
    t0[j] = c * (p0[j] - s.dx * fx[j]);
    t1[j] = c * (p1[j] + s.dx * fy[j]);
  }
}

// y faces: t0 Exy (F = fx, sign +), t1 Ezy (fz, -).
template <class T>
__device__ __forceinline__ void e_yface(const State<T>& s, const Adj<T>& a, int z, int yy, int x0,
                                        const T (&fx)[kAdj], const T (&fz)[kAdj], T (&t0)[kAdj],
                                        T (&t1)[kAdj]) {
  zero_adj(t0);
  zero_adj(t1);
  int side, q;
  if (z >= s.nz - 1 || yy >= s.ny - 1 || !e_face(yy, s.ny, s.npml, side, q)) return;
  const long long k = ky(s, z, q, x0);
  const T c = s.prof[side ? CE_U : CE_D][q] * s.rdx;
  T p0[kAdj], p1[kAdj];
  ld_adj(p0, a.lps.y[side][0] + k);
  ld_adj(p1, a.lps.y[side][1] + k);
#pragma unroll
  for (int j = 0; j < kAdj; ++j) {
    if (x0 + j >= s.nx - 1) continue;
    t0[j] = c * (p0[j] + s.dx * fx[j]);
    t1[j] = c * (p1[j] - s.dx * fz[j]);
  }
}

// H-face auxiliaries: c/dx times lambda_psi + sign dtm0 lambda_H.
// z faces: t2 Hxz (lhx, +), t3 Hyz (lhy, -).
template <class T>
__device__ __forceinline__ void h_zface(const State<T>& s, const Adj<T>& a, int zz, int y, int x0,
                                        const T (&lx)[kAdj], const T (&ly)[kAdj], T (&t2)[kAdj],
                                        T (&t3)[kAdj]) {
  zero_adj(t2);
  zero_adj(t3);
  int side, q;
  if (zz < 0 || zz >= s.nz - 1 || y >= s.ny - 1 || !h_face(zz, s.nz, s.npml, side, q)) return;
  const long long k = kz(s, q, y, x0);
  const T c = s.prof[side ? CH_U : CH_D][q] * s.rdx;
  T p2[kAdj], p3[kAdj];
  ld_adj(p2, a.lps.z[side][2] + k);
  ld_adj(p3, a.lps.z[side][3] + k);
#pragma unroll
  for (int j = 0; j < kAdj; ++j) {
    if (x0 + j >= s.nx - 1) continue;
    t2[j] = c * (p2[j] + s.dtm0 * lx[j]);
    t3[j] = c * (p3[j] - s.dtm0 * ly[j]);
  }
}

// y faces: t2 Hxy (lhx, -), t3 Hzy (lhz, +).
template <class T>
__device__ __forceinline__ void h_yface(const State<T>& s, const Adj<T>& a, int z, int yy, int x0,
                                        const T (&lx)[kAdj], const T (&lz)[kAdj], T (&t2)[kAdj],
                                        T (&t3)[kAdj]) {
  zero_adj(t2);
  zero_adj(t3);
  int side, q;
  if (yy < 0 || z >= s.nz - 1 || yy >= s.ny - 1 || !h_face(yy, s.ny, s.npml, side, q)) return;
  const long long k = ky(s, z, q, x0);
  const T c = s.prof[side ? CH_U : CH_D][q] * s.rdx;
  T p2[kAdj], p3[kAdj];
  ld_adj(p2, a.lps.y[side][2] + k);
  ld_adj(p3, a.lps.y[side][3] + k);
#pragma unroll
  for (int j = 0; j < kAdj; ++j) {
    if (x0 + j >= s.nx - 1) continue;
    t2[j] = c * (p2[j] - s.dtm0 * lx[j]);
    t3[j] = c * (p3[j] + s.dtm0 * lz[j]);
  }
}

// H auxiliaries' adjoint (f) of the vector, from its lambda_H:
// lambda_psi = bh (lambda_psi + sign dtm0 lambda_H) on every H face.
template <class T>
__device__ __forceinline__ void h_own_vec(const State<T>& s, const Adj<T>& a, int z, int y, int x0,
                                          const T (&lhx)[kAdj], const T (&lhy)[kAdj],
                                          const T (&lhz)[kAdj]) {
  const int nx = s.nx, ny = s.ny, nz = s.nz, m = s.npml;
  if (z >= nz - 1 || y >= ny - 1) return;
  int side, q;
  if (h_face(z, nz, m, side, q)) {
    const long long k = kz(s, q, y, x0);
    const T b = s.prof[side ? BH_U : BH_D][q];
    T p2[kAdj], p3[kAdj];
    ld_adj(p2, a.lps.z[side][2] + k);
    ld_adj(p3, a.lps.z[side][3] + k);
#pragma unroll
    for (int j = 0; j < kAdj; ++j) {
      if (x0 + j >= nx - 1) continue;
      p3[j] = b * (p3[j] - s.dtm0 * lhy[j]);
      p2[j] = b * (p2[j] + s.dtm0 * lhx[j]);
    }
    st_adj(a.lps.z[side][2] + k, p2);
    st_adj(a.lps.z[side][3] + k, p3);
  }
  if (x0 < m - 1 || x0 + kAdj - 1 >= nx - m) {
#pragma unroll
    for (int j = 0; j < kAdj; ++j) {
      const int x = x0 + j;
      if (x >= nx - 1 || !h_face(x, nx, m, side, q)) continue;
      const long long k = kx(s, z, y, side, q);
      const T b = s.prof[side ? BH_U : BH_D][q];
      T* p3 = a.lps.x[side][3];
      T* p2 = a.lps.x[side][2];
      p3[k] = b * (p3[k] - s.dtm0 * lhz[j]);
      p2[k] = b * (p2[k] + s.dtm0 * lhy[j]);
    }
  }
  if (h_face(y, ny, m, side, q)) {
    const long long k = ky(s, z, q, x0);
    const T b = s.prof[side ? BH_U : BH_D][q];
    T p2[kAdj], p3[kAdj];
    ld_adj(p2, a.lps.y[side][2] + k);
    ld_adj(p3, a.lps.y[side][3] + k);
#pragma unroll
    for (int j = 0; j < kAdj; ++j) {
      if (x0 + j >= nx - 1) continue;
      p2[j] = b * (p2[j] - s.dtm0 * lhx[j]);
      p3[j] = b * (p3[j] + s.dtm0 * lhz[j]);
    }
    st_adj(a.lps.y[side][2] + k, p2);
    st_adj(a.lps.y[side][3] + k, p3);
  }
}

// (b) lambda_H increments of the vector: the transposed curl of
// F = Cb lambda_E (backward differences of F: the forward E update of the
// cell and of its +x, +y, +z neighbours reads H of this cell) and the E-face
// auxiliaries of the cell and of those neighbours. `fast`: the vector and
// every neighbour it reads lie away from every CPML face and domain edge.
template <class T, bool kFast>
__device__ __forceinline__ void e_to_h_vec(const State<T>& s, const Adj<T>& a, int z, int y, int x0,
                                           T (&dhx)[kAdj], T (&dhy)[kAdj], T (&dhz)[kAdj]) {
  const int nx = s.nx, ny = s.ny, nz = s.nz, m = s.npml;
  const long long P = s.plane, W = s.pitch, i = idx(s, z, y, x0);
  T cb[kAdj], l0[kAdj], l1[kAdj], l2[kAdj];
  T fx[kAdj], fy[kAdj], fz[kAdj];       // cell
  ld_adj(cb, s.cb + i);
  ld_adj(l0, a.lex + i);
  ld_adj(l1, a.ley + i);
  ld_adj(l2, a.lez + i);
  if constexpr (kFast) {
    // The neighbours' products go into the differences unrounded, but for
    // the x neighbour inside an aligned group of four cells, whose product
    // is rounded as that cell's own: written out, so that the rounding of a
    // cell depends on neither kAdj nor the compiler's contraction.
    using M = R<T>;
    T yz[kAdj], zy[kAdj], zx[kAdj], xz[kAdj], xy[kAdj], yx[kAdj];
#pragma unroll
    for (int j = 0; j < kAdj; ++j) {
      fx[j] = M::mul(cb[j], l0[j]);
      fy[j] = M::mul(cb[j], l1[j]);
      fz[j] = M::mul(cb[j], l2[j]);
    }
    ld_adj(cb, s.cb + i + P);
    ld_adj(l0, a.lex + i + P);
    ld_adj(l1, a.ley + i + P);
#pragma unroll
    for (int j = 0; j < kAdj; ++j) {
      xz[j] = M::fma(-cb[j], l0[j], fx[j]);
      yz[j] = M::fma(-cb[j], l1[j], fy[j]);
    }
    ld_adj(cb, s.cb + i + W);
    ld_adj(l0, a.lex + i + W);
    ld_adj(l2, a.lez + i + W);
#pragma unroll
    for (int j = 0; j < kAdj; ++j) {
      xy[j] = M::fma(-cb[j], l0[j], fx[j]);
      zy[j] = M::fma(-cb[j], l2[j], fz[j]);
    }
    const T cbn = s.cb[i + kAdj], yn = a.ley[i + kAdj], zn = a.lez[i + kAdj];
    const bool group = ((x0 + kAdj) & 3) == 0;   // x0 + kAdj starts the next group
#pragma unroll
    for (int j = 0; j < kAdj; ++j) {
      if (j + 1 < kAdj) {
        yx[j] = M::sub(fy[j], fy[j + 1 < kAdj ? j + 1 : j]);
        zx[j] = M::sub(fz[j], fz[j + 1 < kAdj ? j + 1 : j]);
      } else {
        yx[j] = group ? M::fma(-cbn, yn, fy[j]) : M::sub(fy[j], M::mul(cbn, yn));
        zx[j] = group ? M::fma(-cbn, zn, fz[j]) : M::sub(fz[j], M::mul(cbn, zn));
      }
    }
#pragma unroll
    for (int j = 0; j < kAdj; ++j) {
      dhx[j] = M::sub(yz[j], zy[j]);
      dhy[j] = M::sub(zx[j], xz[j]);
      dhz[j] = M::sub(xy[j], yx[j]);
    }
  } else {
    T fxz[kAdj], fyz[kAdj];             // z + 1
    T fxy[kAdj], fzy[kAdj];             // y + 1
    T fyn = T(0), fzn = T(0);           // x0 + kAdj
    bool rx[kAdj], ry[kAdj], rz[kAdj];
    e_ranges(s, z, y, x0, rx, ry, rz);
    masked_prod(fx, cb, l0, rx);
    masked_prod(fy, cb, l1, ry);
    masked_prod(fz, cb, l2, rz);
    zero_adj(fxz);
    zero_adj(fyz);
    if (z + 1 < nz - 1) {
      e_ranges(s, z + 1, y, x0, rx, ry, rz);
      ld_adj(cb, s.cb + i + P);
      ld_adj(l0, a.lex + i + P);
      ld_adj(l1, a.ley + i + P);
      masked_prod(fxz, cb, l0, rx);
      masked_prod(fyz, cb, l1, ry);
    }
    zero_adj(fxy);
    zero_adj(fzy);
    if (y + 1 < ny - 1) {
      e_ranges(s, z, y + 1, x0, rx, ry, rz);
      ld_adj(cb, s.cb + i + W);
      ld_adj(l0, a.lex + i + W);
      ld_adj(l2, a.lez + i + W);
      masked_prod(fxy, cb, l0, rx);
      masked_prod(fzy, cb, l2, rz);
    }
    if (x0 + kAdj < nx - 1) {   // the cell x0 + kAdj is inside the x ranges
      const T cbn = s.cb[i + kAdj];
      if (z >= 1 && z < nz - 1 && y < ny - 1) fyn = cbn * a.ley[i + kAdj];
      if (z < nz - 1 && y >= 1 && y < ny - 1) fzn = cbn * a.lez[i + kAdj];
    }
#pragma unroll
    for (int j = 0; j < kAdj; ++j) {
      const T fy_x = j + 1 < kAdj ? fy[j + 1 < kAdj ? j + 1 : j] : fyn;
      const T fz_x = j + 1 < kAdj ? fz[j + 1 < kAdj ? j + 1 : j] : fzn;
      dhx[j] = (fy[j] - fyz[j]) - (fz[j] - fzy[j]);
      dhy[j] = (fz[j] - fz_x) - (fx[j] - fxz[j]);
      dhz[j] = (fx[j] - fxy[j]) - (fy[j] - fy_x);
    }
    T t0[kAdj], t1[kAdj], u0[kAdj], u1[kAdj];
    // z faces of the cell and of z + 1: Eyz reads hx(c) - hx(c - z), Exz hy
    e_zface(s, a, z, y, x0, fx, fy, t0, t1);
    e_zface(s, a, z + 1, y, x0, fxz, fyz, u0, u1);
#pragma unroll
    for (int j = 0; j < kAdj; ++j) {
      dhx[j] += t1[j] - u1[j];
      dhy[j] += t0[j] - u0[j];
    }
    // y faces of the cell and of y + 1: Exy reads hz(c) - hz(c - y), Ezy hx
    e_yface(s, a, z, y, x0, fx, fz, t0, t1);
    e_yface(s, a, z, y + 1, x0, fxy, fzy, u0, u1);
#pragma unroll
    for (int j = 0; j < kAdj; ++j) {
      dhz[j] += t0[j] - u0[j];
      dhx[j] += t1[j] - u1[j];
    }
    // x faces of x0 .. x0 + kAdj: Ezx reads hy(c) - hy(c - x), Eyx hz
    if (x0 < m || x0 + kAdj >= nx - m) {
      T xt0[kAdj + 1], xt1[kAdj + 1];
#pragma unroll
      for (int p = 0; p <= kAdj; ++p) {
        const int xx = x0 + p;
        const T fyv = p < kAdj ? fy[p < kAdj ? p : 0] : fyn;
        const T fzv = p < kAdj ? fz[p < kAdj ? p : 0] : fzn;
        xt0[p] = T(0);
        xt1[p] = T(0);
        int side, q;
        if (z < nz - 1 && y < ny - 1 && xx < nx - 1 && e_face(xx, nx, m, side, q)) {
          const long long k = kx(s, z, y, side, q);
          const T c = s.prof[side ? CE_U : CE_D][q] * s.rdx;
          xt0[p] = c * (a.lps.x[side][0][k] - s.dx * fyv);
          xt1[p] = c * (a.lps.x[side][1][k] + s.dx * fzv);
        }
      }
#pragma unroll
      for (int j = 0; j < kAdj; ++j) {
        dhy[j] += xt1[j] - xt1[j + 1];
        dhz[j] += xt0[j] - xt0[j + 1];
      }
    }
  }
}

// (c) gradients and the E auxiliaries' adjoint of the vector; returns
// Ca lambda_E (zero outside the update ranges). s.iex.. hold E^n, s.ihx..
// H^{n+1/2}, s.ps the auxiliaries after the step.
template <class T, bool kFast>
__device__ __forceinline__ void e_own_vec(const State<T>& s, const Adj<T>& a, int z, int y, int x0,
                                          T (&ox)[kAdj], T (&oy)[kAdj], T (&oz)[kAdj]) {
  const int nx = s.nx, ny = s.ny, nz = s.nz, m = s.npml;
  const long long P = s.plane, W = s.pitch, i = idx(s, z, y, x0);
  T lx[kAdj], ly[kAdj], lz[kAdj], ca[kAdj], cb[kAdj];
  ld_adj(lx, a.lex + i);
  ld_adj(ly, a.ley + i);
  ld_adj(lz, a.lez + i);
  ld_adj(ca, s.ca + i);
  ld_adj(cb, s.cb + i);
  bool rx[kAdj], ry[kAdj], rz[kAdj];
  if constexpr (kFast) {
#pragma unroll
    for (int j = 0; j < kAdj; ++j) rx[j] = ry[j] = rz[j] = true;
  } else {
    e_ranges(s, z, y, x0, rx, ry, rz);
  }
  const bool grad = z < a.nz_grad;   // gradients only over the requested planes
  double gca[kAdj], gcb[kAdj];
  if (grad) {
    T e[kAdj], h0[kAdj], h1[kAdj], h2[kAdj], hn0[kAdj], hn1[kAdj];
    ld_adj(e, s.iex + i);
#pragma unroll
    for (int j = 0; j < kAdj; ++j) gca[j] = rx[j] ? (double)lx[j] * (double)e[j] : 0.0;
    ld_adj(e, s.iey + i);
#pragma unroll
    for (int j = 0; j < kAdj; ++j) gca[j] += ry[j] ? (double)ly[j] * (double)e[j] : 0.0;
    ld_adj(e, s.iez + i);
#pragma unroll
    for (int j = 0; j < kAdj; ++j) gca[j] += rz[j] ? (double)lz[j] * (double)e[j] : 0.0;
    ld_adj(h0, s.ihx + i);
    ld_adj(h1, s.ihy + i);
    ld_adj(h2, s.ihz + i);
    // ex: (hz - hz(y-1)) - (hy - hy(z-1))
    if (kFast || (z >= 1 && y >= 1)) {
      ld_adj(hn0, s.ihz + i - W);
      ld_adj(hn1, s.ihy + i - P);
    } else {
      zero_adj(hn0);
      zero_adj(hn1);
    }
#pragma unroll
    for (int j = 0; j < kAdj; ++j)
      gcb[j] = rx[j] ? (double)lx[j] * (double)((h2[j] - hn0[j]) - (h1[j] - hn1[j])) : 0.0;
    // ey: (hx - hx(z-1)) - (hz - hz(x-1))
    const T hzp = (kFast || (x0 >= 1 && z >= 1)) ? s.ihz[i - 1] : T(0);
    if (kFast || z >= 1) ld_adj(hn0, s.ihx + i - P); else zero_adj(hn0);
#pragma unroll
    for (int j = 0; j < kAdj; ++j) {
      const T hz_x = j > 0 ? h2[j > 0 ? j - 1 : 0] : hzp;
      gcb[j] += ry[j] ? (double)ly[j] * (double)((h0[j] - hn0[j]) - (h2[j] - hz_x)) : 0.0;
    }
    // ez: (hy - hy(x-1)) - (hx - hx(y-1))
    const T hyp = (kFast || (x0 >= 1 && y >= 1)) ? s.ihy[i - 1] : T(0);
    if (kFast || y >= 1) ld_adj(hn0, s.ihx + i - W); else zero_adj(hn0);
#pragma unroll
    for (int j = 0; j < kAdj; ++j) {
      const T hy_x = j > 0 ? h1[j > 0 ? j - 1 : 0] : hyp;
      gcb[j] += rz[j] ? (double)lz[j] * (double)((h1[j] - hy_x) - (h0[j] - hn0[j])) : 0.0;
    }
  }
  if constexpr (!kFast) {
    if (z < nz - 1 && y < ny - 1) {
      const T dx = s.dx;
      int side, q;
      if (e_face(z, nz, m, side, q)) {
        const long long k = kz(s, q, y, x0);
        const T b = s.prof[side ? BE_U : BE_D][q];
        T p0[kAdj], p1[kAdj], s0[kAdj], s1[kAdj];
        ld_adj(p0, a.lps.z[side][0] + k);
        ld_adj(p1, a.lps.z[side][1] + k);
        if (grad) {
          ld_adj(s0, s.ps.z[side][0] + k);
          ld_adj(s1, s.ps.z[side][1] + k);
        }
#pragma unroll
        for (int j = 0; j < kAdj; ++j) {
          if (x0 + j >= nx - 1) continue;
          if (grad) gcb[j] += (double)dx * ((double)s1[j] * ly[j] - (double)s0[j] * lx[j]);
          p1[j] = b * (p1[j] + cb[j] * dx * ly[j]);
          p0[j] = b * (p0[j] - cb[j] * dx * lx[j]);
        }
        st_adj(a.lps.z[side][0] + k, p0);
        st_adj(a.lps.z[side][1] + k, p1);
      }
      if (x0 < m || x0 + kAdj - 1 >= nx - m) {
#pragma unroll
        for (int j = 0; j < kAdj; ++j) {
          const int x = x0 + j;
          if (x >= nx - 1 || !e_face(x, nx, m, side, q)) continue;
          const long long k = kx(s, z, y, side, q);
          const T b = s.prof[side ? BE_U : BE_D][q];
          T* p1 = a.lps.x[side][1];
          T* p0 = a.lps.x[side][0];
          if (grad)
            gcb[j] += (double)dx * ((double)s.ps.x[side][1][k] * lz[j] - (double)s.ps.x[side][0][k] * ly[j]);
          p1[k] = b * (p1[k] + cb[j] * dx * lz[j]);
          p0[k] = b * (p0[k] - cb[j] * dx * ly[j]);
        }
      }
      if (e_face(y, ny, m, side, q)) {
        const long long k = ky(s, z, q, x0);
        const T b = s.prof[side ? BE_U : BE_D][q];
        T p0[kAdj], p1[kAdj], s0[kAdj], s1[kAdj];
        ld_adj(p0, a.lps.y[side][0] + k);
        ld_adj(p1, a.lps.y[side][1] + k);
        if (grad) {
          ld_adj(s0, s.ps.y[side][0] + k);
          ld_adj(s1, s.ps.y[side][1] + k);
        }
#pragma unroll
        for (int j = 0; j < kAdj; ++j) {
          if (x0 + j >= nx - 1) continue;
          if (grad) gcb[j] += (double)dx * ((double)s0[j] * lx[j] - (double)s1[j] * lz[j]);
          p0[j] = b * (p0[j] + cb[j] * dx * lx[j]);
          p1[j] = b * (p1[j] - cb[j] * dx * lz[j]);
        }
        st_adj(a.lps.y[side][0] + k, p0);
        st_adj(a.lps.y[side][1] + k, p1);
      }
    }
  }
  if (grad) {
    double g[kAdj];
    ld_adj(g, a.gca + i);
#pragma unroll
    for (int j = 0; j < kAdj; ++j) g[j] += gca[j];
    st_adj(a.gca + i, g);
    ld_adj(g, a.gcb + i);
#pragma unroll
    for (int j = 0; j < kAdj; ++j) g[j] += gcb[j];
    st_adj(a.gcb + i, g);
  }
  // A component outside its main-update range is updated in the forward
  // step only by CPML corrections and injection terms that read other such
  // components (the edge sub-systems, e.g. ey, ez, hx on x = 0), or not at
  // all. With an incident beam that vanishes on those edges (as the
  // reference's does) it stays exactly zero, so no parameter reaches J
  // through it, and nothing in range reads it back in the transposed step.
  // Its exact adjoint, fed by the interior's, grows exponentially like the
  // forward sub-system would if driven; it is held at zero instead (here
  // and in k_adj_k1), which leaves every gradient unchanged and keeps the
  // sweep finite. Every reader below relies on that: adjoint fields are
  // exactly zero outside their update ranges.
#pragma unroll
  for (int j = 0; j < kAdj; ++j) {
    ox[j] = rx[j] ? ca[j] * lx[j] : T(0);
    oy[j] = ry[j] ? ca[j] * ly[j] : T(0);
    oz[j] = rz[j] ? ca[j] * lz[j] : T(0);
  }
}

// (e) lambda_E increments of the vector: the transposed curl of
// G = Db lambda_H (forward differences: the forward H update of the cell
// and of its -x, -y, -z neighbours reads E of this cell) and the H-face
// auxiliaries of the cell and of those neighbours.
template <class T, bool kFast>
__device__ __forceinline__ void h_to_e_vec(const State<T>& s, const Adj<T>& a, int z, int y, int x0,
                                           T (&dex)[kAdj], T (&dey)[kAdj], T (&dez)[kAdj]) {
  const int nx = s.nx, ny = s.ny, nz = s.nz, m = s.npml;
  const long long P = s.plane, W = s.pitch, i = idx(s, z, y, x0);
  T hx[kAdj], hy[kAdj], hz[kAdj];       // lambda_H of the cell
  T hxz[kAdj], hyz[kAdj];               // z - 1
  T hxy[kAdj], hzy[kAdj];               // y - 1
  ld_adj(hx, a.lhx + i);
  ld_adj(hy, a.lhy + i);
  ld_adj(hz, a.lhz + i);
  if (kFast || z >= 1) {
    ld_adj(hxz, a.lhx + i - P);
    ld_adj(hyz, a.lhy + i - P);
  } else {
    zero_adj(hxz);
    zero_adj(hyz);
  }
  if (kFast || y >= 1) {
    ld_adj(hxy, a.lhx + i - W);
    ld_adj(hzy, a.lhz + i - W);
  } else {
    zero_adj(hxy);
    zero_adj(hzy);
  }
  T hyp = T(0), hzp = T(0);             // x0 - 1
  if (kFast || x0 >= 1) {
    hyp = a.lhy[i - 1];
    hzp = a.lhz[i - 1];
  }
  const T db = s.db;
#pragma unroll
  for (int j = 0; j < kAdj; ++j) {
    const T hy_x = j > 0 ? hy[j > 0 ? j - 1 : 0] : hyp;
    const T hz_x = j > 0 ? hz[j > 0 ? j - 1 : 0] : hzp;
    dex[j] = db * ((hy[j] - hyz[j]) - (hz[j] - hzy[j]));
    dey[j] = db * ((hz[j] - hz_x) - (hx[j] - hxz[j]));
    dez[j] = db * ((hx[j] - hxy[j]) - (hy[j] - hy_x));
  }
  if constexpr (!kFast) {
    T t2[kAdj], t3[kAdj], u2[kAdj], u3[kAdj];
    // z faces of z - 1 and of the cell: Hyz reads ex(c + z) - ex(c), Hxz ey
    h_zface(s, a, z - 1, y, x0, hxz, hyz, t2, t3);
    h_zface(s, a, z, y, x0, hx, hy, u2, u3);
#pragma unroll
    for (int j = 0; j < kAdj; ++j) {
      dex[j] += t3[j] - u3[j];
      dey[j] += t2[j] - u2[j];
    }
    // y faces of y - 1 and of the cell: Hxy reads ez(c + y) - ez(c), Hzy ex
    h_yface(s, a, z, y - 1, x0, hxy, hzy, t2, t3);
    h_yface(s, a, z, y, x0, hx, hz, u2, u3);
#pragma unroll
    for (int j = 0; j < kAdj; ++j) {
      dez[j] += t2[j] - u2[j];
      dex[j] += t3[j] - u3[j];
    }
    // x faces of x0 - 1 .. x0 + kAdj - 1: Hzx reads ey(c + x) - ey(c), Hyx ez
    if (x0 < m || x0 + kAdj - 1 >= nx - m) {
      T xt2[kAdj + 1], xt3[kAdj + 1];
#pragma unroll
      for (int p = 0; p <= kAdj; ++p) {
        const int xx = x0 - 1 + p;
        const T lyv = p > 0 ? hy[p > 0 ? p - 1 : 0] : hyp;
        const T lzv = p > 0 ? hz[p > 0 ? p - 1 : 0] : hzp;
        xt2[p] = T(0);
        xt3[p] = T(0);
        int side, q;
        if (xx >= 0 && z < nz - 1 && y < ny - 1 && xx < nx - 1 && h_face(xx, nx, m, side, q)) {
          const long long k = kx(s, z, y, side, q);
          const T c = s.prof[side ? CH_U : CH_D][q] * s.rdx;
          xt2[p] = c * (a.lps.x[side][2][k] + s.dtm0 * lyv);
          xt3[p] = c * (a.lps.x[side][3][k] - s.dtm0 * lzv);
        }
      }
#pragma unroll
      for (int j = 0; j < kAdj; ++j) {
        dey[j] += xt3[j] - xt3[j + 1];
        dez[j] += xt2[j] - xt2[j + 1];
      }
    }
  }
}

// ---- the two kernels of one backward step ------------------------------------
// Blocks of (lanes, 128 / lanes) threads, each thread kAdj x cells; grid
// (x tiles, y tiles, nz).
template <class T>
__device__ __forceinline__ bool vec_cell(const State<T>& s, int& z, int& y, int& x0) {
  x0 = kAdj * (blockIdx.x * blockDim.x + threadIdx.x);
  y = blockIdx.y * blockDim.y + threadIdx.y;
  z = blockIdx.z;
  return x0 < s.nx && y < s.ny;
}

// K1 (step n): the H auxiliaries' adjoint of step n + 1 (skipped for the
// first backward step), then lambda_H += (E step)^T lambda_E + the H phasor
// source of step n.
template <class T>
__global__ void __launch_bounds__(128, sizeof(T) == 4 ? 8 : 7)
    k_adj_k1(const __grid_constant__ State<T> s, Adj<T> a, int t, int first) {
  int z, y, x0;
  if (!vec_cell(s, z, y, x0)) return;
  const int m = s.npml;
  const long long i = idx(s, z, y, x0);
  T lhx[kAdj], lhy[kAdj], lhz[kAdj], dhx[kAdj], dhy[kAdj], dhz[kAdj];
  ld_adj(lhx, a.lhx + i);
  ld_adj(lhy, a.lhy + i);
  ld_adj(lhz, a.lhz + i);
  const int xg = x0 & ~3;
  if (z >= m && z < s.nz - m - 1 && y >= m && y < s.ny - m - 1 && xg >= m && xg + 4 < s.nx - m) {
    // no H face at the vector, no E face or domain edge at it or its +x,
    // +y, +z neighbours. The line is drawn for the aligned four cells: the
    // general form rounds every product, the fast one does not, so the line
    // decides a cell's last bit, which kAdj must not.
    e_to_h_vec<T, true>(s, a, z, y, x0, dhx, dhy, dhz);
  } else {
    if (!first) h_own_vec(s, a, z, y, x0, lhx, lhy, lhz);
    e_to_h_vec<T, false>(s, a, z, y, x0, dhx, dhy, dhz);
  }
  const int pz = s.nz - m - 1;
  if (z == pz || z == pz - 1) {
#pragma unroll
    for (int j = 0; j < kAdj; ++j) {
      T phx, phy;
      phasor_h_src(s, a, t, z, y, x0 + j, phx, phy);
      dhx[j] += phx;
      dhy[j] += phy;
    }
  }
  bool rx[kAdj], ry[kAdj], rz[kAdj];
  h_ranges(s, z, y, x0, rx, ry, rz);
#pragma unroll
  for (int j = 0; j < kAdj; ++j) {
    lhx[j] = rx[j] ? lhx[j] + dhx[j] : T(0);
    lhy[j] = ry[j] ? lhy[j] + dhy[j] : T(0);
    lhz[j] = rz[j] ? lhz[j] + dhz[j] : T(0);
  }
  st_adj(a.lhx + i, lhx);
  st_adj(a.lhy + i, lhy);
  st_adj(a.lhz + i, lhz);
}

// K2 (step n): gradients and the E auxiliaries' adjoint, then
// lambda_E = Ca lambda_E + (H step)^T lambda_H + the E phasor source of
// step n - 1 (t_prev < 0: none).
template <class T>
__global__ void __launch_bounds__(128, sizeof(T) == 4 ? 7 : 6)
    k_adj_k2(const __grid_constant__ State<T> s, Adj<T> a, int t_prev) {
  int z, y, x0;
  if (!vec_cell(s, z, y, x0)) return;
  const int m = s.npml;
  const long long i = idx(s, z, y, x0);
  T ex[kAdj], ey[kAdj], ez[kAdj], dex[kAdj], dey[kAdj], dez[kAdj];
  const int xg = x0 & ~3;
  if (z >= m && z < s.nz - m && y >= m && y < s.ny - m && xg >= m && xg + 3 < s.nx - m) {
    // no E or H face at the vector, no H face or domain edge at its -x, -y,
    // -z neighbours; by four cells, as in k_adj_k1
    e_own_vec<T, true>(s, a, z, y, x0, ex, ey, ez);
    h_to_e_vec<T, true>(s, a, z, y, x0, dex, dey, dez);
  } else {
    e_own_vec<T, false>(s, a, z, y, x0, ex, ey, ez);
    h_to_e_vec<T, false>(s, a, z, y, x0, dex, dey, dez);
  }
  if (t_prev >= 0 && z == s.nz - m - 1) {
#pragma unroll
    for (int j = 0; j < kAdj; ++j) {
      T pex, pey;
      phasor_e_src(s, a, t_prev, z, y, x0 + j, pex, pey);
      dex[j] += pex;
      dey[j] += pey;
    }
  }
  bool rx[kAdj], ry[kAdj], rz[kAdj];
  e_ranges(s, z, y, x0, rx, ry, rz);
#pragma unroll
  for (int j = 0; j < kAdj; ++j) {
    ex[j] = rx[j] ? ex[j] + dex[j] : T(0);
    ey[j] = ry[j] ? ey[j] + dey[j] : T(0);
    ez[j] = rz[j] ? ez[j] + dez[j] : T(0);
  }
  st_adj(a.lex + i, ex);
  st_adj(a.ley + i, ey);
  st_adj(a.lez + i, ez);
}

// lanes per row: the width (8, 16 or 32 threads of kAdj cells) that pads the
// row least, the wider on a tie
inline int adj_lanes(int nx) {
  int best = 32, pad = 1 << 30;
  for (int w : {32, 16, 8}) {
    const int cells = kAdj * w, p = ((nx + cells - 1) / cells) * cells - nx;
    if (p < pad) {
      pad = p;
      best = w;
    }
  }
  return best;
}

// 32 x 4 cells per block: little x padding on grids a few hundred cells wide
template <class T>
void launch_adjoint_first(const State<T>& s, const Adj<T>& a, int t, cudaStream_t st) {
  k_adj_phasor_e<T><<<dim3((s.nx + 31) / 32, (s.ny + 3) / 4, 1), dim3(32, 4, 1), 0, st>>>(s, a, t);
}

template <class T>
void launch_adjoint_step(const State<T>& s, const Adj<T>& a, int t, bool first, cudaStream_t st) {
  const int w = adj_lanes(s.nx), rows = 128 / w;
  const dim3 grd((s.nx + kAdj * w - 1) / (kAdj * w), (s.ny + rows - 1) / rows, s.nz), blk(w, rows, 1);
  k_adj_k1<T><<<grd, blk, 0, st>>>(s, a, t, first ? 1 : 0);
  k_adj_k2<T><<<grd, blk, 0, st>>>(s, a, t - 1);
}

template void launch_adjoint_first<float>(const State<float>&, const Adj<float>&, int, cudaStream_t);
template void launch_adjoint_first<double>(const State<double>&, const Adj<double>&, int, cudaStream_t);
template void launch_adjoint_step<float>(const State<float>&, const Adj<float>&, int, bool, cudaStream_t);
template void launch_adjoint_step<double>(const State<double>&, const Adj<double>&, int, bool,
                                          cudaStream_t);

// dJ/deps_r and dJ/dsigma of the material block's cells from dJ/dCa, dJ/dCb
// (pitched): the closed form of compute_material_arrays (Ca = (1 - x) / (1 + x),
// Cb = (dt / (eps_r eps0 dx)) / (1 + x), x = sigma dt / (2 eps_r eps0);
// materials/materials.py:45-63), operation for operation as
// adjoint.ca_cb_partials evaluates it in float64. eps, sig, ge, gs: (rows,
// nx) packed. HBM-bound, one pass over 48 bytes a cell. On the host the
// combination took 20 ms of a 109 ms gradient (584 thousand cells).
__global__ void __launch_bounds__(256) k_grad_eps_sigma(int nx, long long rows, int pitch, double dt, double dx,
                                                        const double* __restrict__ gca,
                                                        const double* __restrict__ gcb,
                                                        const double* __restrict__ eps,
                                                        const double* __restrict__ sig, double* __restrict__ ge,
                                                        double* __restrict__ gs) {
  using M = R<double>;
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= nx) return;
  for (long long r = blockIdx.y; r < rows; r += gridDim.y) {
    const long long k = r * nx + x, i = r * pitch + x;
    const double e = eps[k], a = gca[i], b = gcb[i];
    const double perm = M::mul(e, 8.8541878128e-12);
    const double den = M::mul(2.0, perm);
    const double xl = M::div(M::mul(sig[k], dt), den);
    const double x_de = M::div(-xl, e), x_ds = M::div(dt, den);
    const double p = M::add(1.0, xl), p2 = M::mul(p, p);
    const double ca_x = M::div(-2.0, p2);
    const double cb0 = M::div(dt, M::mul(perm, dx));
    const double ca_e = M::mul(ca_x, x_de), ca_s = M::mul(ca_x, x_ds);
    const double cb_e = M::sub(M::div(M::div(-cb0, e), p), M::mul(M::div(cb0, p2), x_de));
    const double cb_s = M::mul(M::div(-cb0, p2), x_ds);
    ge[k] = M::add(M::mul(a, ca_e), M::mul(b, cb_e));
    gs[k] = M::add(M::mul(a, ca_s), M::mul(b, cb_s));
  }
}

void launch_grad_eps_sigma(int nx, long long rows, int pitch, double dt, double dx, const double* gca,
                           const double* gcb, const double* eps, const double* sig, double* ge, double* gs,
                           cudaStream_t st) {
  const dim3 grd((nx + 255) / 256, (unsigned)(rows < 65535 ? rows : 65535), 1);
  k_grad_eps_sigma<<<grd, 256, 0, st>>>(nx, rows, pitch, dt, dx, gca, gcb, eps, sig, ge, gs);
}

}  // namespace fdtd
