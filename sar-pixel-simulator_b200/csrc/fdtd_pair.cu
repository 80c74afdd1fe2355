// fdtd_pair.cu -- two time steps in one pass over the grid (the pair step).
//
// A single fused step reads and writes every field once per step: 56 B per
// FP32 cell-update, which the interior march of fdtd_fused.cu runs at 95 %
// of the copy bandwidth. The pair step advances n -> n + 2 while each field
// crosses HBM once: a z-march that computes H^{n+1/2}, E^{n+1}, H^{n+3/2},
// E^{n+2} of a tile before it leaves the SM, source set -> destination set.
//
// k_pair. A block is TR warps; a tile row is L threads, each holding one
// vector of 16 bytes (4 floats or 2 doubles), so a tile has 32 TR / L rows.
// It marches up in z; at plane z it computes
//   1. H1(z) = H^{n+1/2}(z) from E(z), E(z+1), H(z);
//   2. E1(z) = E^{n+1}(z) from H1(z), H1(z-1);
//   3. H2(z-1) = H^{n+3/2}(z-1) from E1(z-1), E1(z), H1(z-1);
//   4. E2(z-1) = E^{n+2}(z-1) from H2(z-1), H2(z-2), and stores H2, E2.
// Planes of E (one row more than the tile), H, Ca, Cb arrive by TMA, E
// three planes deep and the rest two, so that two planes are in flight while
// one is computed; H1, E1, H2 pass between rows through shared memory (two
// barriers per plane) and between lanes by shuffle. A tile recomputes two
// rows below, one above, and a vector at either end (unless the domain ends
// there); a chunk of planes [z0, z1) starts two planes below and reads one
// plane above.
//
// The grid is cut into four kinds of regions, each with the boundary terms
// it can meet and no others:
//   plain   the box two cells inside every CPML face; the injection plane is
//           uniform over a plane and stays in it (32 x 16 thread tiles)
//   z faces the same x-y box, bottom and top planes: z-face CPML terms,
//           uniform over a plane (32 x 12)
//   y ends  the rows at either y end, same x range: y and z faces (16 x 14)
//   x ends  the columns at either x end, all y, all z: every face. Tiles of
//           128-byte rows by 32 rows: the rows of an x face are short, and a
//           wide tile would march mostly plain cells with the general update.
//           (At the low end 64-byte rows by 64 would do; that tile, a launch
//           of its own, made the step slower: 198 us against 184 there.)
//           (Tiles turned so that a warp is one column of vectors, where an x
//           face is uniform over a warp, ran fewer instructions, but the face
//           warps kept the others waiting at the barriers: 183 us against
//           148 at 101 x 381 x 381.)
// The z-face, x-face and y-face CPML auxiliaries of the two steps stay in
// registers between them (read from the source set, written to the
// destination set once).
//
// Phasors read both steps' fields: the marches write the fields between the
// steps of the planes that phasors read (PairMid).
//
// Why this shape: a march is HBM-bound as long as a plane of 1560 output
// cells (32 x 16 threads: 30 x 4 x 13) is computed in less than the ~2 us
// that its 87 KB take at an SM's share of the bandwidth; 16 rows keep 76 %
// of the computed cells, 8 rows would keep 59 % and read 1.3x as much from
// L2.
//
// Measured (float, us per step, single steps and pairs, phasors included):
// 203 x 761 x 761 cells 1485 and 930; 101 x 381 x 381 243 and 179 to 193 (by
// where the fields lie); double, 101 x 381 x 381 650 and 320. At 203 x 761 x 761 the plain march takes 973 us
// per pair (6.0 TB/s; 5.9 GB, of which 10 % is halo), the z faces 302, the
// x ends 463, the y ends 123; those three are bound by instructions and
// latency (IPC 1.3 to 1.5 at one block of 12 to 16 warps per SM), not by HBM.
#include <algorithm>
#include <cstring>

#include <cuda.h>

#include "fdtd_launch.h"
#include "fdtd_vecn.cuh"

namespace fdtd {

namespace {

constexpr unsigned long long kWaitNs = 2000000000ull;   // one mbarrier wait gives up after this long

// A tile of L threads per row and TR warps, elements T, V cells per thread,
// with the CPML faces it can meet (none: a plain tile). Shared memory: E ring
// (3 planes of 3 components of kRows + 1 rows), ring of H, Ca, Cb (2 planes
// of 5 components of kRows rows), exchange rows x and z of H1, E1 (two
// buffers), H2; the five mbarriers.
template <class T_, int V_, int L_, int TR_, bool kX_, bool kY_, bool kZ_>
struct PairTile {
  using T = T_;
  static constexpr int V = V_, L = L_, TR = TR_;
  static constexpr bool kX = kX_, kY = kY_, kZ = kZ_, kEdge = kX || kY || kZ;
  static constexpr int kCells = L * V;   // cells of a row
  static constexpr int kRows = 32 * TR / L;
  static constexpr int kRowBytes = kCells * (int)sizeof(T);
  static constexpr int kEComp = (kRows + 1) * kRowBytes, kHComp = kRows * kRowBytes;
  static constexpr int kEBytes = 3 * kEComp, kHBytes = 5 * kHComp;   // a plane of each ring
  static constexpr int kHRing = 3 * kEBytes, kXchAt = kHRing + 2 * kHBytes;
  static constexpr int kXch = 2 * kHComp;
  static constexpr int kBars = kXchAt + 4 * kXch;
  static constexpr int kBytes = kBars + 64;
  // recomputed cells at either x end: two, rounded up to the 16 bytes a copy starts on
  static constexpr int kHalo = 16 / (int)sizeof(T);
  static constexpr int kOutX = kCells - 2 * kHalo, kOutY = kRows - 3;
};

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
// Waits for the phase `parity`; false when the time limit ran out.
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity) {
  if (mbar_try(bar, parity)) return true;
  const unsigned long long end = now_ns() + kWaitNs;
  do {
    if (mbar_try(bar, parity)) return true;
  } while (now_ns() < end);
  return false;
}
__device__ __forceinline__ void tma_plane(unsigned dst, const CUtensorMap* map, unsigned bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
          dst),
      "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z)
      : "memory");
}

// What a thread carries from one plane of the march to the next: E1, H1,
// Ca, Cb and the psi (after the first step) of its plane, and H2 of the
// plane below it.
template <class T, int V>
struct PairCarry {
  T ex[V], ey[V], ez[V], hx[V], hy[V], hz[V], ca[V], cb[V], h2x[V], h2y[V];
  T ph[6][V], pe[6][V];
};

// The kinds of tile a warp computes as on a plane where it meets no boundary,
// or only an x face.
template <class C>
using PairPlain = PairTile<typename C::T, C::V, C::L, C::TR, false, false, false>;
template <class C>
using PairOnlyX = PairTile<typename C::T, C::V, C::L, C::TR, C::kX, false, false>;

template <class C>
__global__ void __launch_bounds__(32 * C::TR, 1)
k_pair(const __grid_constant__ State<typename C::T> s, const __grid_constant__ PairMaps maps,
       const __grid_constant__ PairRegions rg, PairMid<typename C::T> mid, const int* __restrict__ tp, int toff,
       int* err) {
  using T = typename C::T;
  constexpr int V = C::V, NR = C::kRows, kSz = (int)sizeof(T);
  constexpr unsigned kAll = 0xffffffffu;
  extern __shared__ __align__(1024) unsigned char smem[];
  const unsigned base = smem_u32(smem);
  const unsigned bars = base + C::kBars;   // E slots 0..2, then HC slots 0..1
  const int lane = threadIdx.x % C::L, r = threadIdx.x / C::L;

  int bid = blockIdx.x;
  const PairRegion& b = rg.r[rg.n > 1 && bid >= rg.r[1].first ? 1 : 0];
  bid -= b.first;
  const int bx = bid % b.gx;
  bid /= b.gx;
  const int by = bid % b.gy, c = bid / b.gy;
  const int z0 = b.z0 + c * b.zchunk, z1 = min(b.z1, z0 + b.zchunk);
  const int nz = s.nz, m = s.npml;
  const int zs = max(z0 - 2, 0);
  const int zl = min(z1, nz - 1);        // last plane of H1, E1
  const int ze = min(zl + 1, nz - 1);    // last plane of E read
  const int xt = b.xt + bx * b.sx, yt = b.yt + by * b.sy;   // the tile's first cell and row
  const int xo = b.x0 + bx * b.sx, yo = b.y0 + by * b.sy;   // its first own ones
  PairPos<T, V> p;
  p.x0 = xt + lane * V;
  p.y = yt + r;
  p.mz = (T)rg.minus0;
  pair_pos<C>(s, p);
  p.yplain = __all_sync(kAll, p.yplain);   // of the warp's vectors
  p.plain = __all_sync(kAll, p.plain);
  const bool own = p.vin && p.x0 >= xo && p.x0 < min(b.x1, xo + b.sx) && p.y >= yo && p.y < min(b.y1, yo + b.sy);
  // where the vector lies in the mid planes (-1: not)
  auto mid_slot = [&](int v, int n) { return v == m ? 0 : v == m + 1 ? 1 : v == n - m - 2 ? 2 : v == n - m - 1 ? 3 : -1; };
  const int mid_y = C::kY && own ? mid_slot(p.y, s.ny) : -1;
  bool mid_x = false;
  if (C::kX && own)
    for (int j = 0; j < V; ++j) mid_x = mid_x || mid_slot(p.x0 + j, s.nx) >= 0;
  const unsigned P = (unsigned)s.plane;
  const int t = *tp + toff;

  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < 5; ++k) mbar_init(bars + 8 * k);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();

  auto issue_e = [&](int z) {
    const int slot = (z - zs) % 3;
    const unsigned bar = bars + 8 * slot, dst = base + slot * C::kEBytes;
    mbar_expect(bar, C::kEBytes);
#pragma unroll
    for (int k = 0; k < 3; ++k) tma_plane(dst + k * C::kEComp, &maps.m[k], bar, xt, yt, z);
  };
  auto issue_hc = [&](int z) {
    const int slot = (z - zs) & 1;
    const unsigned bar = bars + 24 + 8 * slot, dst = base + C::kHRing + slot * C::kHBytes;
    mbar_expect(bar, C::kHBytes);
#pragma unroll
    for (int k = 0; k < 5; ++k) tma_plane(dst + k * C::kHComp, &maps.m[3 + k], bar, xt, yt, z);
  };
  if (threadIdx.x == 0) {
    issue_e(zs);
    issue_hc(zs);
    if (zs + 1 <= ze) issue_e(zs + 1);
    if (zs + 1 <= zl) issue_hc(zs + 1);
    if (zs + 2 <= ze) issue_e(zs + 2);
  }

  // this thread's place in a tile plane, and those of the rows below and
  // above (rows at the tile's edge read a stand-in: they compute nothing
  // that counts), in elements
  const int at = r * C::kCells + lane * V;
  const int dn = r > 0 ? at - C::kCells : at, up = r < NR - 1 ? at + C::kCells : at;
  constexpr int kHalf = C::kHComp / kSz;   // the second row set of an exchange buffer
  auto xch = [&](int k) { return reinterpret_cast<T*>(smem + C::kXchAt + k * C::kXch); };
  // H of the row below (x, z) and the previous lane's last cell (y, z)
  auto h_in = [&](const T* w, const T (&hy)[V], const T (&hz)[V], T (&hxy)[V], T (&hzy)[V], T& hyp, T& hzp) {
    lds(hxy, w + dn);
    lds(hzy, w + kHalf + dn);
    hyp = __shfl_up_sync(kAll, hy[V - 1], 1, C::L);
    hzp = __shfl_up_sync(kAll, hz[V - 1], 1, C::L);
  };
  auto out = [&](T* w, const T (&a)[V], const T (&b)[V]) {
    sts(w + at, a);
    sts(w + kHalf + at, b);
  };

  // the vector's cells in the phasors' x columns
  auto x_columns = [&](int z, T* const (&to)[4], const T (&a0)[V], const T (&a1)[V], const T (&a2)[V],
                       const T (&a3)[V]) {
#pragma unroll
    for (int j = 0; j < V; ++j) {
      const int k = mid_slot(p.x0 + j, s.nx);
      if (k < 0) continue;
      const unsigned i = (unsigned)((z * s.ny + p.y) * 4 + k);
      stc(to[0] + i, a0[j]); stc(to[1] + i, a1[j]); stc(to[2] + i, a2[j]); stc(to[3] + i, a3[j]);
    }
  };

  PairCarry<T, V> A, B;
  vset(A.ex, T(0)); vset(A.ey, T(0)); vset(A.ez, T(0));
  vset(A.hx, T(0)); vset(A.hy, T(0)); vset(A.hz, T(0));
  vset(A.ca, T(0)); vset(A.cb, T(0)); vset(A.h2x, T(0)); vset(A.h2y, T(0));
#pragma unroll
  for (int q = 0; q < 6; ++q) { vset(A.ph[q], T(0)); vset(A.pe[q], T(0)); }
  B = A;
  // good: every copy so far arrived within the time limit. After the first
  // that did not, at plane `lost` (thread 0), nothing is waited for and no more
  // start.
  int lost = zs;
  bool good = mbar_wait(bars, 0);   // E(zs)
  int es = 0;                       // E ring slot of plane z
  unsigned ep = 1;                  // bit k: parity of E slot k's next wait

  // plane z; d: what it leaves, g: what plane z - 1 left (its fields end as
  // H2, E2)
  auto plane = [&](int z, PairCarry<T, V>& d, PairCarry<T, V>& g) __attribute__((always_inline)) {
    const int k = z - zs;
    const int en = es == 2 ? 0 : es + 1;
    const bool first = !C::kZ || z < nz;   // z == nz only ends the topmost chunk
    // warps that meet no boundary on the plane take the plain update
    const bool zp1 = z >= m && z < nz - m, zp2 = z - 1 >= m && z - 1 < nz - m;
    const bool easy1 = C::kEdge && p.plain && zp1, easy2 = C::kEdge && p.plain && zp2;
    const bool xonly1 = C::kX && p.yplain && zp1, xonly2 = C::kX && p.yplain && zp2;
    if (C::kEdge && first && !easy1) {
      auto load = [](T (&v)[V], const T* from, T*) { ldg(v, from); };
      if (xonly1) pair_psi<PairOnlyX<C>>(s, p, z, d.ph, d.pe, load);
      else pair_psi<C>(s, p, z, d.ph, d.pe, load);
    }
    if (first) {
      if (z + 1 <= ze) {
        good = good && mbar_wait(bars + 8 * en, (ep >> en) & 1u);
        ep ^= 1u << en;
      }
      good = good && mbar_wait(bars + 24 + 8 * (k & 1), (k >> 1) & 1);
      const T* const E0 = reinterpret_cast<const T*>(smem + es * C::kEBytes) + at;
      const T* const E1 = reinterpret_cast<const T*>(smem + en * C::kEBytes) + at;
      const T* const HC = reinterpret_cast<const T*>(smem + C::kHRing + (k & 1) * C::kHBytes) + at;
      constexpr int kEc = C::kEComp / kSz, kHc = C::kHComp / kSz;
      T exz[V], eyz[V], exy[V], ezy[V];
      lds(d.ex, E0);
      lds(d.ey, E0 + kEc);
      lds(d.ez, E0 + 2 * kEc);
      lds(exy, E0 + C::kCells);
      lds(ezy, E0 + 2 * kEc + C::kCells);
      lds(exz, E1);
      lds(eyz, E1 + kEc);
      lds(d.hx, HC);
      lds(d.hy, HC + kHc);
      lds(d.hz, HC + 2 * kHc);
      lds(d.ca, HC + 3 * kHc);
      lds(d.cb, HC + 4 * kHc);
      const T eyn = __shfl_down_sync(kAll, d.ey[0], 1, C::L);
      const T ezn = __shfl_down_sync(kAll, d.ez[0], 1, C::L);
      if (easy1) pair_h<PairPlain<C>>(s, p, z, t, d.ex, d.ey, d.ez, exz, eyz, exy, ezy, eyn, ezn, d.hx, d.hy, d.hz, d.ph);
      else if (xonly1) pair_h<PairOnlyX<C>>(s, p, z, t, d.ex, d.ey, d.ez, exz, eyz, exy, ezy, eyn, ezn, d.hx, d.hy, d.hz, d.ph);
      else pair_h<C>(s, p, z, t, d.ex, d.ey, d.ez, exz, eyz, exy, ezy, eyn, ezn, d.hx, d.hy, d.hz, d.ph);
      out(xch(0), d.hx, d.hz);
    }
    __syncthreads();
    // every thread has read plane z of the rings: their slots take new planes
    if (threadIdx.x == 0 && good) {
      lost = z + 1;
      if (z + 3 <= ze) issue_e(z + 3);
      if (z + 2 <= zl) issue_hc(z + 2);
    }
    if (first) {
      T hxy[V], hzy[V], hyp, hzp;
      h_in(xch(0), d.hy, d.hz, hxy, hzy, hyp, hzp);
      if (easy1)
        pair_e<PairPlain<C>>(s, p, z, t, d.hx, d.hy, d.hz, g.hx, g.hy, hxy, hzy, hyp, hzp, d.ca, d.cb, d.ex, d.ey, d.ez,
                             d.pe);
      else if (xonly1) pair_e<PairOnlyX<C>>(s, p, z, t, d.hx, d.hy, d.hz, g.hx, g.hy, hxy, hzy, hyp, hzp, d.ca, d.cb, d.ex, d.ey, d.ez, d.pe);
      else pair_e<C>(s, p, z, t, d.hx, d.hy, d.hz, g.hx, g.hy, hxy, hzy, hyp, hzp, d.ca, d.cb, d.ex, d.ey, d.ez, d.pe);
      out(xch(1 + (k & 1)), d.ex, d.ez);
      if (own && z >= z0 && z < z1) {
        const int mz = mid_slot(z, nz);
        if (mz >= 0) {
          const unsigned i = (unsigned)mz * P + p.kx;
          stg(mid.z[0] + i, d.ex); stg(mid.z[1] + i, d.ey); stg(mid.z[2] + i, d.hx); stg(mid.z[3] + i, d.hy);
        }
        if (C::kY && mid_y >= 0) {
          const unsigned i = (unsigned)((z * 4 + mid_y) * s.pitch + p.x0);
          stg(mid.y[0] + i, d.ex); stg(mid.y[1] + i, d.ez); stg(mid.y[2] + i, d.hx); stg(mid.y[3] + i, d.hz);
        }
        if (C::kX && mid_x) x_columns(z, mid.x[0], d.ey, d.ez, d.hy, d.hz);
      }
    }
    // ---- second step, plane z - 1
    const bool second = k >= 1;
    T h2z[V];
    if (second) {
      T exy[V], ezy[V];
      const T* const w = xch(1 + ((k - 1) & 1));
      lds(exy, w + up);
      lds(ezy, w + kHalf + up);
      const T eyn = __shfl_down_sync(kAll, g.ey[0], 1, C::L);
      const T ezn = __shfl_down_sync(kAll, g.ez[0], 1, C::L);
#pragma unroll
      for (int j = 0; j < V; ++j) { d.h2x[j] = g.hx[j]; d.h2y[j] = g.hy[j]; h2z[j] = g.hz[j]; }
      if (easy2)
        pair_h<PairPlain<C>>(s, p, z - 1, t + 1, g.ex, g.ey, g.ez, d.ex, d.ey, exy, ezy, eyn, ezn, d.h2x, d.h2y, h2z,
                             g.ph);
      else if (xonly2) pair_h<PairOnlyX<C>>(s, p, z - 1, t + 1, g.ex, g.ey, g.ez, d.ex, d.ey, exy, ezy, eyn, ezn, d.h2x, d.h2y, h2z, g.ph);
      else pair_h<C>(s, p, z - 1, t + 1, g.ex, g.ey, g.ez, d.ex, d.ey, exy, ezy, eyn, ezn, d.h2x, d.h2y, h2z, g.ph);
      out(xch(3), d.h2x, h2z);
    }
    __syncthreads();
    if (second) {
      T hxy[V], hzy[V], hyp, hzp;
      h_in(xch(3), d.h2y, h2z, hxy, hzy, hyp, hzp);
      if (easy2)
        pair_e<PairPlain<C>>(s, p, z - 1, t + 1, d.h2x, d.h2y, h2z, g.h2x, g.h2y, hxy, hzy, hyp, hzp, g.ca, g.cb, g.ex,
                             g.ey, g.ez, g.pe);
      else if (xonly2) pair_e<PairOnlyX<C>>(s, p, z - 1, t + 1, d.h2x, d.h2y, h2z, g.h2x, g.h2y, hxy, hzy, hyp, hzp, g.ca, g.cb, g.ex, g.ey,
                     g.ez, g.pe);
      else pair_e<C>(s, p, z - 1, t + 1, d.h2x, d.h2y, h2z, g.h2x, g.h2y, hxy, hzy, hyp, hzp, g.ca, g.cb, g.ex, g.ey,
                     g.ez, g.pe);
      if (own && z - 1 >= z0) {
        const unsigned i = (unsigned)(z - 1) * P + p.kx;
        stg(s.ohx + i, d.h2x); stg(s.ohy + i, d.h2y); stg(s.ohz + i, h2z);
        stg(s.oex + i, g.ex); stg(s.oey + i, g.ey); stg(s.oez + i, g.ez);
        if (C::kX && mid_x) x_columns(z - 1, mid.x[1], g.ey, g.ez, d.h2y, h2z);
        if (C::kEdge && !easy2) {
          auto store = [](T (&v)[V], const T*, T* to) { stg(to, v); };
          if (xonly2) pair_psi<PairOnlyX<C>>(s, p, z - 1, g.ph, g.pe, store);
          else pair_psi<C>(s, p, z - 1, g.ph, g.pe, store);
        }
      }
    }
    es = en;
  };
  // two planes per turn, so that what a plane leaves is never moved
  for (int z = zs; z <= z1; z += 2) {
    plane(z, A, B);
    if (z < z1) plane(z + 1, B, A);
  }
  if (!good) {
    *err = 1;
    // the copies in flight still land in this block's memory: a bounded wait
    // for the last that were started
    if (threadIdx.x == 0) {
      for (int z = lost; z <= min(lost + 2, ze); ++z) mbar_wait(bars + 8 * ((z - zs) % 3), ((z - zs) / 3) & 1);
      for (int z = lost; z <= min(lost + 1, zl); ++z) mbar_wait(bars + 24 + 8 * ((z - zs) & 1), ((z - zs) >> 1) & 1);
    }
  }
}

// The four tile kinds (registers per thread are bounded by 65536 / threads).
template <class T> constexpr int kWide = 16 / (int)sizeof(T);
template <class T> using PlainTile = PairTile<T, kWide<T>, 32, 16, false, false, false>;
template <class T> using ZTile = PairTile<T, kWide<T>, 32, 12, false, false, true>;
template <class T> using YTile = PairTile<T, kWide<T> / 2, 32, 14, false, true, true>;
template <class T> using XTile = PairTile<T, kWide<T> / 2, 16, 16, true, true, true>;
constexpr int kPairSlots = 148;   // blocks in flight

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                              const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn encode_fn() {
  void* p = nullptr;
  cudaDriverEntryPointQueryResult found;
  if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &found) != cudaSuccess ||
      found != cudaDriverEntryPointSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  return reinterpret_cast<EncodeFn>(p);
}

// A map of one (nz, ny, pitch) array for tiles of `cells` x box_rows of one
// plane; parts outside the array read as zeros.
template <class T>
bool encode(CUtensorMap* map, const void* p, const State<T>& s, int cells, int box_rows) {
  static const EncodeFn fn = encode_fn();
  if (!fn) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)s.pitch, (cuuint64_t)s.ny, (cuuint64_t)s.nz};
  const cuuint64_t strides[2] = {(cuuint64_t)s.pitch * sizeof(T), (cuuint64_t)s.plane * sizeof(T)};
  const cuuint32_t box[3] = {(cuuint32_t)cells, (cuuint32_t)box_rows, 1};
  const cuuint32_t one[3] = {1, 1, 1};
  return fn(map, sizeof(T) == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3,
            const_cast<void*>(p), dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <class C>
bool tile_maps(const State<typename C::T>& s, PairMaps* out) {
  const void* f[8] = {s.iex, s.iey, s.iez, s.ihx, s.ihy, s.ihz, s.ca, s.cb};
  for (int k = 0; k < 8; ++k)
    if (!encode(&out->m[k], f[k], s, C::kCells, C::kRows + (k < 3 ? 1 : 0))) return false;
  return true;
}

template <class C>
bool pair_launch(const State<typename C::T>& s, const PairMaps& maps, const PairRegions& rg,
                 const PairMid<typename C::T>& mid, const int* tdev, int toff, int* err, cudaStream_t st) {
  if (rg.blocks == 0) return true;
  if (cudaFuncSetAttribute(k_pair<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kBytes) != cudaSuccess)
    return false;
  k_pair<C><<<rg.blocks, 32 * C::TR, C::kBytes, st>>>(s, maps, rg, mid, tdev, toff, err);
  return true;
}

// Adds the region x [x0, x1), y [y0, y1), z [z0, z1) in x tiles of sx and y
// tiles of sy cells whose first tile starts at (xt, yt).
void add_region(PairRegions& rg, int x0, int x1, int xt, int sx, int y0, int y1, int yt, int sy, int z0, int z1) {
  if (x0 >= x1 || y0 >= y1 || z0 >= z1) return;
  PairRegion& b = rg.r[rg.n++];
  b.x0 = x0; b.x1 = x1; b.xt = xt; b.sx = sx;
  b.y0 = y0; b.y1 = y1; b.yt = yt; b.sy = sy;
  b.z0 = z0; b.z1 = z1;
  b.gx = (x1 - x0 + sx - 1) / sx;
  b.gy = (y1 - y0 + sy - 1) / sy;
}

// z chunks of the regions of one launch: the count with the fewest planes
// marched by the SM that marches most, one block per SM at a time (a chunk
// recomputes two planes, reads a third ahead, and about one more goes to
// filling its pipeline); then the regions' first blocks.
void cut_regions(PairRegions& rg, bool cut) {
  rg.minus0 = -0.0f;
  long long tiles = 0;
  int planes = 0;
  for (int k = 0; k < rg.n; ++k) {
    tiles += (long long)rg.r[k].gx * rg.r[k].gy;
    planes = std::max(planes, rg.r[k].z1 - rg.r[k].z0);
  }
  int zchunk = planes;
  double best = -1;
  for (int n = 1; cut && n <= std::max(1, planes / 4); ++n) {
    const int zc = (planes + n - 1) / n;
    if ((planes + zc - 1) / zc != n) continue;
    const double cost = (double)((tiles * n + kPairSlots - 1) / kPairSlots) * (zc + 4);
    if (best < 0 || cost < best) {
      best = cost;
      zchunk = zc;
    }
  }
  for (int k = 0; k < rg.n; ++k) {
    PairRegion& b = rg.r[k];
    b.zchunk = zchunk;
    b.first = rg.blocks;
    rg.blocks += b.gx * b.gy * ((b.z1 - b.z0 + zchunk - 1) / zchunk);
  }
}

template <class T>
PairPlan plan_for(int nx, int ny, int nz, int npml) {
  PairPlan p;
  memset(&p, 0, sizeof(p));
  const int m = npml;
  using Pl = PlainTile<T>;
  using Xt = XTile<T>;
  using Yt = YTile<T>;
  // the box at least two cells inside the x and y faces. The x ends take as
  // many columns as their one tile of 128-byte rows computes (two cells at
  // the inner side are recomputed; at the high end, copies start on 16
  // bytes), in 32-byte sectors where that leaves room
  const int h = Pl::kHalo, ya = m + 2, yb = ny - m - 2;
  const int sector = 32 / (int)sizeof(T), x_low = Xt::kCells - 2, x_high = Xt::kCells - h;
  int xa = x_low / sector * sector, xb = (nx - x_high + sector - 1) / sector * sector;
  if (xa < m + 2) xa = (m + 2 + h - 1) / h * h;
  if (xb > nx - m - 2) xb = (nx - m - 2) / h * h;
  if (xa > x_low || nx - xb > x_high || ya + 2 > Yt::kRows) return p;
  const int zi0 = m + 2, zi1 = nz - m - 1;
  if (xb - xa < 32 || yb - ya < 8 || zi1 - zi0 < 1) return p;
  add_region(p.plain, xa, xb, xa - h, Pl::kOutX, ya, yb, ya - 2, Pl::kOutY, zi0, zi1);
  add_region(p.zface, xa, xb, xa - h, Pl::kOutX, ya, yb, ya - 2, ZTile<T>::kOutY, 0, zi0);
  add_region(p.zface, xa, xb, xa - h, Pl::kOutX, ya, yb, ya - 2, ZTile<T>::kOutY, zi1, nz);
  add_region(p.yend, xa, xb, xa - h, Yt::kOutX, 0, ya, 0, ya, 0, nz);
  add_region(p.yend, xa, xb, xa - h, Yt::kOutX, yb, ny, yb - 2, ny - yb, 0, nz);
  add_region(p.xend, 0, xa, 0, xa, 0, ny, -2, Xt::kOutY, 0, nz);
  add_region(p.xend, xb, nx, xb - h, nx - xb, 0, ny, -2, Xt::kOutY, 0, nz);
  cut_regions(p.plain, true);
  cut_regions(p.zface, false);
  cut_regions(p.yend, true);
  cut_regions(p.xend, true);
  // us per step, from the planes that the blocks of each kind march (four
  // more per chunk): least squares over 352 float grids of 3 to 60 M cells
  // and 160 or more columns, 5 % rms
  auto planes = [](const PairRegions& rg) {
    double n = 0;
    for (int k = 0; k < rg.n; ++k) {
      const PairRegion& b = rg.r[k];
      const int z = b.z1 - b.z0;
      n += (double)b.gx * b.gy * (z + 4 * ((z + b.zchunk - 1) / b.zchunk));
    }
    return n / kPairSlots;
  };
  p.us = 16.3 + 0.8 * planes(p.plain) + 1.5 * planes(p.zface) + 1.8 * planes(p.yend) + 2.75 * planes(p.xend);
  p.ok = 1;
  return p;
}

}  // namespace

PairPlan make_pair_plan(int nx, int ny, int nz, int npml, int elem_bytes) {
  return elem_bytes == 4 ? plan_for<float>(nx, ny, nz, npml) : plan_for<double>(nx, ny, nz, npml);
}

template <class T>
bool make_pair_maps(const State<T>& s, PairMapSet* out) {
  return tile_maps<PlainTile<T>>(s, &out->plain) && tile_maps<ZTile<T>>(s, &out->zface) &&
         tile_maps<YTile<T>>(s, &out->yend) && tile_maps<XTile<T>>(s, &out->xend);
}

template <class T>
bool launch_pair(PairKind kind, const State<T>& s, const PairPlan& p, const PairMapSet& maps, const PairMid<T>& mid,
                 const int* tdev, int toff, int* err, cudaStream_t st) {
  switch (kind) {
    case kPairPlain: return pair_launch<PlainTile<T>>(s, maps.plain, p.plain, mid, tdev, toff, err, st);
    case kPairZ: return pair_launch<ZTile<T>>(s, maps.zface, p.zface, mid, tdev, toff, err, st);
    case kPairY: return pair_launch<YTile<T>>(s, maps.yend, p.yend, mid, tdev, toff, err, st);
    case kPairX: return pair_launch<XTile<T>>(s, maps.xend, p.xend, mid, tdev, toff, err, st);
  }
  return false;
}

#define FDTD_PAIR_INSTANCES(T)                                                                                    \
  template bool make_pair_maps<T>(const State<T>&, PairMapSet*);                                                  \
  template bool launch_pair<T>(PairKind, const State<T>&, const PairPlan&, const PairMapSet&, const PairMid<T>&, \
                               const int*, int, int*, cudaStream_t);
FDTD_PAIR_INSTANCES(float)
FDTD_PAIR_INSTANCES(double)

}  // namespace fdtd
