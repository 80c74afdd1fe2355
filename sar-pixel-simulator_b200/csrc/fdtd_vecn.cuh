// fdtd_vecn.cuh -- H and E updates of a vector of V cells with the CPML terms
// of all faces, shared by the pair step (fdtd_pair.cu) and the resident step
// (fdtd_resident.cu).
//
// The same values as h_vec / e_vec (fdtd_vec.cuh), which the split passes
// use, with a vector's position (faces, ranges, x-face coefficients) worked
// out beforehand, the CPML auxiliaries handed in and out, floats computed in
// pairs (f32x2), and no branch in the CPML terms. A kind C names the boundary
// terms that can occur (C::kX, C::kY, C::kZ); the others cost nothing.
// Element indices are 32-bit (one instruction per address): 14 or more
// arrays of a grid's volume share the device's 180 GB, so no array has 2^32
// elements.
#pragma once

#include "fdtd_vec.cuh"

namespace fdtd {

// V elements as one access.
template <class T, int V>
struct alignas(sizeof(T) * V) PairVec {
  T v[V];
};
template <class T, int V>
__device__ __forceinline__ void lds(T (&d)[V], const T* p) {
  const PairVec<T, V> a = *reinterpret_cast<const PairVec<T, V>*>(p);
#pragma unroll
  for (int j = 0; j < V; ++j) d[j] = a.v[j];
}
template <class T, int V>
__device__ __forceinline__ void sts(T* p, const T (&d)[V]) {
  PairVec<T, V> a;
#pragma unroll
  for (int j = 0; j < V; ++j) a.v[j] = d[j];
  *reinterpret_cast<PairVec<T, V>*>(p) = a;
}
// Global forms of the same, checked in the bounds-checked build.
template <class T, int V>
__device__ __forceinline__ void ldg(T (&d)[V], const T* p) {
  if (!FDTD_CHECK_PTR(p, (int)sizeof(T) * V)) {
#pragma unroll
    for (int j = 0; j < V; ++j) d[j] = T(0);
    return;
  }
  lds(d, p);
}
template <class T, int V>
__device__ __forceinline__ void stg(T* p, const T (&d)[V]) {
  if (!FDTD_CHECK_PTR(p, (int)sizeof(T) * V)) return;
  sts(p, d);
}

// d = a op b for the cells of a vector; floats go in pairs (f32x2), whose
// halves round like the scalar operations (round to nearest, no contraction).
#define FDTD_PAIR_OP2(NAME, PTX, SCALAR)                                                     \
  template <class T, int V>                                                                  \
  __device__ __forceinline__ void NAME(T (&d)[V], const T (&a)[V], const T (&b)[V]) {        \
    if constexpr (sizeof(T) == 4 && V % 2 == 0) {                                            \
      _Pragma("unroll") for (int j = 0; j < V; j += 2)                                       \
          asm("{\n .reg .b64 x, y;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n " PTX     \
              " x, x, y;\n mov.b64 {%0, %1}, x;\n}\n"                                        \
              : "=f"(d[j]), "=f"(d[j + 1])                                                   \
              : "f"(a[j]), "f"(a[j + 1]), "f"(b[j]), "f"(b[j + 1]));                         \
    } else {                                                                                 \
      _Pragma("unroll") for (int j = 0; j < V; ++j) d[j] = R<T>::SCALAR(a[j], b[j]);         \
    }                                                                                        \
  }
FDTD_PAIR_OP2(vadd, "add.rn.f32x2", add)
FDTD_PAIR_OP2(vsub, "sub.rn.f32x2", sub)
#undef FDTD_PAIR_OP2
template <class T, int V>
__device__ __forceinline__ void vfma(T (&d)[V], const T (&a)[V], const T (&b)[V], const T (&c)[V]) {
  if constexpr (sizeof(T) == 4 && V % 2 == 0) {
#pragma unroll
    for (int j = 0; j < V; j += 2)
      asm("{\n .reg .b64 x, y, z;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n mov.b64 z, {%6, %7};\n"
          " fma.rn.f32x2 x, x, y, z;\n mov.b64 {%0, %1}, x;\n}\n"
          : "=f"(d[j]), "=f"(d[j + 1])
          : "f"(a[j]), "f"(a[j + 1]), "f"(b[j]), "f"(b[j + 1]), "f"(c[j]), "f"(c[j + 1]));
  } else {
#pragma unroll
    for (int j = 0; j < V; ++j) d[j] = R<T>::fma(a[j], b[j], c[j]);
  }
}
// The product, for floats as a fused multiply-add of mz = -0, which leaves
// every product as it is. mz must be a value the compiler cannot know: it
// merges a plain f32x2 product (or one plus a constant -0) into a following
// f32x2 addition, which would then round once instead of twice.
template <class T, int V>
__device__ __forceinline__ void vmul(T (&d)[V], const T (&a)[V], const T (&b)[V], T mz) {
  if constexpr (sizeof(T) == 4 && V % 2 == 0) {
    T c[V];
#pragma unroll
    for (int j = 0; j < V; ++j) c[j] = mz;
    vfma(d, a, b, c);
  } else {
#pragma unroll
    for (int j = 0; j < V; ++j) d[j] = R<T>::mul(a[j], b[j]);
  }
}
template <class T, int V>
__device__ __forceinline__ void vset(T (&d)[V], T a) {
#pragma unroll
  for (int j = 0; j < V; ++j) d[j] = a;
}

// Two CPML auxiliaries of a face: p0 = b p0 + (c d0) / dx, p1 likewise.
template <class T, int V>
__device__ __forceinline__ void psi_pair(const State<T>& s, T mz, const T (&b)[V], const T (&c)[V],
                                         const T (&d0)[V], const T (&d1)[V], T (&p0)[V], T (&p1)[V]) {
  T q0[V], q1[V];
  vmul(q0, c, d0, mz);
  vmul(q1, c, d1, mz);
#pragma unroll
  for (int j = 0; j < V; ++j) {
    q0[j] = div_off_boundary(q0[j], s.dx, s.rdx64);
    q1[j] = div_off_boundary(q1[j], s.dx, s.rdx64);
  }
  vmul(p0, b, p0, mz);
  vmul(p1, b, p1, mz);
  vadd(p0, p0, q0);
  vadd(p1, p1, q1);
}

// The vector a thread computes on a tile, and what of the boundary it meets
// there, fixed over the march.
template <class T, int V>
struct PairPos {
  int y, x0;
  unsigned kx;          // y * pitch + x0 (0 outside the storage)
  bool vin;             // inside the row storage
  bool yplain, plain;   // it meets no y face or edge; nor an x one
  bool yb, y1;          // y < ny - 1, y >= 1
  bool xb[V], x1[V];    // x < nx - 1, x >= 1
  bool xh, xe;          // some cell in an x face, for H and for E
  bool xhc[V], xec[V];  // which
  T xbh[V], xch[V], xbe[V], xce[V];   // the x face's coefficients
  bool yh, ye;          // in a y face, for H and for E
  int yq;               // its plane there (either face's)
  int xs, ys;           // the faces' sides
  T mz;                 // -0 (vmul)
};

// H update of one vector on plane z at step t (its new value in hx, hy, hz):
// the curl update (Taflove 3.30), the CPML terms of the z, x and y faces,
// the E-field injection, in h_vec's order of operations (fdtd_vec.cuh).
// ex, ey, ez: E(z); exz, eyz: E(z+1); exy, ezy: E(y+1); eyn, ezn: the next
// lane's first cell. ph: psi_H of the faces, in and out: Hyz, Hxz (z face),
// Hzx, Hyx (x face), Hxy, Hzy (y face).
template <class C, class T, int V>
__device__ __forceinline__ void pair_h(const State<T>& s, const PairPos<T, V>& p, int z, int t, const T (&ex)[V],
                                       const T (&ey)[V], const T (&ez)[V], const T (&exz)[V], const T (&eyz)[V],
                                       const T (&exy)[V], const T (&ezy)[V], T eyn, T ezn, T (&hx)[V], T (&hy)[V],
                                       T (&hz)[V], T (&ph)[6][V]) {
  using M = R<T>;
  const int m = s.npml;
  const bool zb = !C::kZ || z < s.nz - 1, zyb = zb && (!C::kY || p.yb);
  T dex_z[V], dey_z[V], dez_x[V], dey_x[V], dez_y[V], dex_y[V], db[V], dtm0[V], n[V];
  vset(db, s.db);
  vset(dtm0, s.dtm0);
  vsub(dey_z, eyz, ey);
  vsub(dez_y, ezy, ez);
  vsub(dex_z, exz, ex);
  vsub(dex_y, exy, ex);
#pragma unroll
  for (int j = 0; j < V; ++j) {
    dez_x[j] = M::sub(j + 1 < V ? ez[j + 1 < V ? j + 1 : j] : ezn, ez[j]);
    dey_x[j] = M::sub(j + 1 < V ? ey[j + 1 < V ? j + 1 : j] : eyn, ey[j]);
  }
  // a component's new value where the cell lies in its range
  auto put = [&](T (&h)[V], bool in, const bool* xr) {
    if (!C::kX && !in) return;   // uniform over a row
#pragma unroll
    for (int j = 0; j < V; ++j)
      h[j] = !C::kX || (in && p.xb[j] && (!xr || xr[j])) ? n[j] : h[j];
  };
  vsub(n, dez_y, dey_z);
  vmul(n, db, n, p.mz);
  vsub(n, hx, n);
  put(hx, zyb, p.x1);
  vsub(n, dex_z, dez_x);
  vmul(n, db, n, p.mz);
  vsub(n, hy, n);
  put(hy, zyb && (!C::kY || p.y1), nullptr);
  vsub(n, dey_x, dex_y);
  vmul(n, db, n, p.mz);
  vsub(n, hz, n);
  put(hz, zyb && (!C::kZ || z >= 1), nullptr);
  if (C::kZ && zyb && (z < m - 1 || z >= s.nz - m)) {
    const int side = z < m - 1 ? 0 : 1, q = side ? z - (s.nz - m) : z;
    T b[V], c[V];
    vset(b, s.prof[side ? BH_U : BH_D][q]);
    vset(c, s.prof[side ? CH_U : CH_D][q]);
    psi_pair(s, p.mz, b, c, dex_z, dey_z, ph[0], ph[1]);
    vmul(n, dtm0, ph[0], p.mz);
    vsub(n, hy, n);
    put(hy, true, nullptr);
    vmul(n, dtm0, ph[1], p.mz);
    vadd(n, hx, n);
    put(hx, true, nullptr);
  }
  if (C::kX && zyb && p.xh) {
    psi_pair(s, p.mz, p.xbh, p.xch, dey_x, dez_x, ph[2], ph[3]);
    vmul(n, dtm0, ph[2], p.mz);
    vsub(n, hz, n);
    put(hz, true, p.xhc);
    vmul(n, dtm0, ph[3], p.mz);
    vadd(n, hy, n);
    put(hy, true, p.xhc);
  }
  if (C::kY && zyb && p.yh) {
    T b[V], c[V];
    vset(b, s.prof[p.ys ? BH_U : BH_D][p.yq]);
    vset(c, s.prof[p.ys ? CH_U : CH_D][p.yq]);
    psi_pair(s, p.mz, b, c, dez_y, dex_y, ph[4], ph[5]);
    vmul(n, dtm0, ph[4], p.mz);
    vsub(n, hx, n);
    put(hx, true, nullptr);
    vmul(n, dtm0, ph[5], p.mz);
    vadd(n, hz, n);
    put(hz, true, nullptr);
  }
  if (z == s.tfsf_z && t < s.nt_inc && p.vin) {   // cpu/main_sim.py:147-150
    T iey[V], iex[V];
    const long long k = (long long)t * s.plane + p.kx;
    ldg(iey, s.inc_ey + k);
    ldg(iex, s.inc_ex + k);
#pragma unroll
    for (int j = 0; j < V; ++j) {
      if (C::kX && p.x0 + j >= s.nx) continue;
      hx[j] = M::add(hx[j], M::mul(s.db, iey[j]));
      hy[j] = M::sub(hy[j], M::mul(s.db, iex[j]));
    }
  }
}

// E update of one vector on plane z at step t (Taflove 3.29, the faces, the
// H-field injection), in e_vec's order. hxz, hyz: H(z-1); hxy, hzy: H(y-1);
// hyp, hzp: the previous lane's last cell. pe: psi_E of the faces, in and
// out: Eyz, Exz (z face), Ezx, Eyx (x face), Exy, Ezy (y face).
template <class C, class T, int V>
__device__ __forceinline__ void pair_e(const State<T>& s, const PairPos<T, V>& p, int z, int t, const T (&hx)[V],
                                       const T (&hy)[V], const T (&hz)[V], const T (&hxz)[V], const T (&hyz)[V],
                                       const T (&hxy)[V], const T (&hzy)[V], T hyp, T hzp, const T (&ca)[V],
                                       const T (&cb)[V], T (&ex)[V], T (&ey)[V], T (&ez)[V], T (&pe)[6][V]) {
  using M = R<T>;
  const int m = s.npml;
  const bool zb = !C::kZ || z < s.nz - 1, zyb = zb && (!C::kY || p.yb);
  const bool z1 = !C::kZ || z >= 1, y1 = !C::kY || p.y1;
  T dhz_y[V], dhy_z[V], dhx_z[V], dhz_x[V], dhx_y[V], dhy_x[V], cbdx[V], n[V], w[V];
  vsub(dhz_y, hz, hzy);
  vsub(dhy_z, hy, hyz);
  vsub(dhx_z, hx, hxz);
  vsub(dhx_y, hx, hxy);
#pragma unroll
  for (int j = 0; j < V; ++j) {
    dhz_x[j] = M::sub(hz[j], j > 0 ? hz[j > 0 ? j - 1 : 0] : hzp);
    dhy_x[j] = M::sub(hy[j], j > 0 ? hy[j > 0 ? j - 1 : 0] : hyp);
  }
  auto put = [&](T (&e)[V], bool in, const bool* xr) {
    if (!C::kX && !in) return;
#pragma unroll
    for (int j = 0; j < V; ++j)
      e[j] = !C::kX || (in && p.xb[j] && (!xr || xr[j])) ? n[j] : e[j];
  };
  vsub(n, dhz_y, dhy_z);
  vmul(n, cb, n, p.mz);
  vmul(w, ex, ca, p.mz);
  vadd(n, w, n);
  put(ex, zyb && z1 && y1, nullptr);
  vsub(n, dhx_z, dhz_x);
  vmul(n, cb, n, p.mz);
  vmul(w, ey, ca, p.mz);
  vadd(n, w, n);
  put(ey, zyb && z1, p.x1);
  vsub(n, dhy_x, dhx_y);
  vmul(n, cb, n, p.mz);
  vmul(w, ez, ca, p.mz);
  vadd(n, w, n);
  put(ez, zyb && y1, p.x1);
  if (C::kX || C::kY || C::kZ) {
    vset(w, s.dx);
    vmul(cbdx, cb, w, p.mz);
  }
  if (C::kZ && zyb && ((z >= 1 && z < m) || z >= s.nz - m)) {
    const int side = z < m ? 0 : 1, q = side ? z - (s.nz - m) : z;
    T b[V], c[V];
    vset(b, s.prof[side ? BE_U : BE_D][q]);
    vset(c, s.prof[side ? CE_U : CE_D][q]);
    psi_pair(s, p.mz, b, c, dhx_z, dhy_z, pe[0], pe[1]);
    vmul(n, cbdx, pe[0], p.mz);
    vadd(n, ey, n);
    put(ey, true, nullptr);
    vmul(n, cbdx, pe[1], p.mz);
    vsub(n, ex, n);
    put(ex, true, nullptr);
  }
  if (C::kX && zyb && p.xe) {
    psi_pair(s, p.mz, p.xbe, p.xce, dhy_x, dhz_x, pe[2], pe[3]);
    vmul(n, cbdx, pe[2], p.mz);
    vadd(n, ez, n);
    put(ez, true, p.xec);
    vmul(n, cbdx, pe[3], p.mz);
    vsub(n, ey, n);
    put(ey, true, p.xec);
  }
  if (C::kY && zyb && p.ye) {
    T b[V], c[V];
    vset(b, s.prof[p.ys ? BE_U : BE_D][p.yq]);
    vset(c, s.prof[p.ys ? CE_U : CE_D][p.yq]);
    psi_pair(s, p.mz, b, c, dhz_y, dhx_y, pe[4], pe[5]);
    vmul(n, cbdx, pe[4], p.mz);
    vadd(n, ex, n);
    put(ex, true, nullptr);
    vmul(n, cbdx, pe[5], p.mz);
    vsub(n, ez, n);
    put(ez, true, nullptr);
  }
  if (z == s.tfsf_z && t < s.nt_inc && p.vin) {   // cpu/main_sim.py:158-161
    T ihx[V], ihy[V];
    const long long k = (long long)t * s.plane + p.kx;
    ldg(ihx, s.inc_hx + k);
    ldg(ihy, s.inc_hy + k);
#pragma unroll
    for (int j = 0; j < V; ++j) {
      if (C::kX && p.x0 + j >= s.nx) continue;
      ey[j] = M::add(ey[j], M::mul(s.dte0dx, ihx[j]));
      ex[j] = M::sub(ex[j], M::mul(s.dte0dx, ihy[j]));
    }
  }
}

// What of the boundary the vector at (y, x0) meets.
template <class C, class T, int V>
__device__ __forceinline__ void pair_pos(const State<T>& s, PairPos<T, V>& p) {
  const int m = s.npml;
  p.vin = p.x0 >= 0 && p.x0 < s.pitch && p.y >= 0 && p.y < s.ny;
  p.kx = p.vin ? (unsigned)(p.y * s.pitch + p.x0) : 0u;
  p.yb = p.y < s.ny - 1;
  p.y1 = p.y >= 1;
  p.ys = p.y >= s.ny - m ? 1 : 0;
  p.yq = p.ys ? p.y - (s.ny - m) : p.y;
  p.yh = p.vin && (p.ys || p.y < m - 1);
  p.ye = p.vin && (p.ys || (p.y >= 1 && p.y < m));
  p.yq = p.yh || p.ye ? p.yq : 0;
  p.yplain = !C::kY || (p.y >= m && p.y < s.ny - m);
  p.plain = p.yplain && (!C::kX || (p.x0 >= m && p.x0 + V <= s.nx - m));
  p.xs = p.x0 + V - 1 >= s.nx - m ? 1 : 0;   // no vector reaches both faces (nx >= 2 npml + 3)
  p.xh = p.xe = false;
#pragma unroll
  for (int j = 0; j < V; ++j) {
    const int x = p.x0 + j;
    p.xb[j] = x < s.nx - 1;
    p.x1[j] = x >= 1;
    p.xhc[j] = p.xec[j] = false;
    p.xbh[j] = p.xch[j] = p.xbe[j] = p.xce[j] = T(0);
    if (C::kX && p.vin && p.xb[j]) {
      const int q = p.xs ? x - (s.nx - m) : x;
      p.xhc[j] = p.xs ? q >= 0 : q < m - 1;
      p.xec[j] = p.xs ? q >= 0 : (q >= 1 && q < m);
      if (p.xhc[j]) {
        p.xbh[j] = s.prof[p.xs ? BH_U : BH_D][q];
        p.xch[j] = s.prof[p.xs ? CH_U : CH_D][q];
        p.xh = true;
      }
      if (p.xec[j]) {
        p.xbe[j] = s.prof[p.xs ? BE_U : BE_D][q];
        p.xce[j] = s.prof[p.xs ? CE_U : CE_D][q];
        p.xe = true;
      }
    }
  }
}

// The CPML auxiliaries of the vector on plane z: each face's pairs of psi_H
// and psi_E moved by op(register vector, address in the source set, address
// in the destination set), exactly where the updates use them. An x-face
// pair is moved whole: cells outside the face keep their (unread) slot.
// kF: bit 0 psi_H, bit 1 psi_E.
template <class C, int kF = 3, class T, int V, class Op>
__device__ __forceinline__ void pair_psi(const State<T>& s, const PairPos<T, V>& p, int z, T (&ph)[6][V],
                                         T (&pe)[6][V], Op op) {
  const int m = s.npml;
  if (!p.vin || !((!C::kZ || z < s.nz - 1) && (!C::kY || p.yb))) return;
  if (C::kZ) {
    if ((kF & 1) && (z < m - 1 || z >= s.nz - m)) {
      const int side = z < m - 1 ? 0 : 1;
      const unsigned k = (unsigned)(side ? z - (s.nz - m) : z) * (unsigned)s.plane + p.kx;
      op(ph[0], s.ps.z[side][3] + k, s.pd.z[side][3] + k);
      op(ph[1], s.ps.z[side][2] + k, s.pd.z[side][2] + k);
    }
    if ((kF & 2) && ((z >= 1 && z < m) || z >= s.nz - m)) {
      const int side = z < m ? 0 : 1;
      const unsigned k = (unsigned)(side ? z - (s.nz - m) : z) * (unsigned)s.plane + p.kx;
      op(pe[0], s.ps.z[side][1] + k, s.pd.z[side][1] + k);
      op(pe[1], s.ps.z[side][0] + k, s.pd.z[side][0] + k);
    }
  }
  if (C::kX && (p.xh || p.xe)) {
    const unsigned k = ((unsigned)(z * s.ny + p.y)) * (unsigned)s.xw + (unsigned)(p.x0 - (p.xs ? s.xo1 : 0));
    if ((kF & 1) && p.xh) {
      op(ph[2], s.ps.x[p.xs][3] + k, s.pd.x[p.xs][3] + k);
      op(ph[3], s.ps.x[p.xs][2] + k, s.pd.x[p.xs][2] + k);
    }
    if ((kF & 2) && p.xe) {
      op(pe[2], s.ps.x[p.xs][1] + k, s.pd.x[p.xs][1] + k);
      op(pe[3], s.ps.x[p.xs][0] + k, s.pd.x[p.xs][0] + k);
    }
  }
  if (C::kY && (p.yh || p.ye)) {
    const unsigned k = (unsigned)((z * m + p.yq) * s.pitch + p.x0);
    if ((kF & 1) && p.yh) {
      op(ph[4], s.ps.y[p.ys][2] + k, s.pd.y[p.ys][2] + k);
      op(ph[5], s.ps.y[p.ys][3] + k, s.pd.y[p.ys][3] + k);
    }
    if ((kF & 2) && p.ye) {
      op(pe[4], s.ps.y[p.ys][0] + k, s.pd.y[p.ys][0] + k);
      op(pe[5], s.ps.y[p.ys][1] + k, s.pd.y[p.ys][1] + k);
    }
  }
}

}  // namespace fdtd
