// fdtd_resident.cu -- many steps of a small grid in one launch.
//
// A grid whose fields fit in L2 is bound by latency, not by bytes: a split
// step is three launches of a few microseconds each, and issuing them costs
// the host more than they run. Here one cooperative launch (a block per SM)
// runs the split step's passes over the whole grid for many steps, with a
// grid-wide barrier between them instead of a launch:
//   phase 1: the H pass of step n, and the phasors of step n - 1;
//   phase 2: the E pass of step n.
// E and the CPML auxiliaries are updated in place; H alternates between two
// sets, so that the phasors of the finished step can read its H beside the
// H pass that follows. The last of an odd number of steps updates H in place
// (after its predecessor's phasors), so that a launch ends on the set it began
// with. A launch is of about two milliseconds (resident_launch_steps,
// fdtd_capi.cu), because it holds every SM and stops every other stream; one
// launch for the whole run is 0.3 % to 0.8 % faster (31 x 39 x 39 cells 6.85
// and 6.87 ms per 720 steps, 55 x 133 x 133 34.4 and 34.6 per 1200, 47 x 87 x 107
// double 17.20 and 17.34 per 600), launches of four not measurably.
// The updates are those of fdtd_vecn.cuh, equal bit for bit to the split
// passes'; the phasor cell is the split step's (fdtd_split.cuh).
//
// The barrier waits with a time limit, after which every block leaves and
// the launch is reported as failed.
// Measured (us per step; single steps, launched one by one, and so): float,
// 31 x 39 x 39 cells 22.6 and 8.8; 55 x 133 x 133 49 and 28; double,
// 47 x 87 x 107 62 and 27. A phase is latency: at the smallest size about
// 2 us of barrier and 2 us of one vector's loads and update; at 55 x 133 x 133
// five rounds of them per block (IPC 1.1).
// An incident run of 100 x 133 x 133 cells, its source and read-out included:
// 67 and 49.
#include <algorithm>
#include <cstring>

#include "fdtd_incident.cuh"
#include "fdtd_launch.h"
#include "fdtd_split.cuh"
#include "fdtd_vecn.cuh"

namespace fdtd {

namespace {

// Kinds of boundary terms (fdtd_vecn.cuh): everything, and nothing.
struct ResAll {
  static constexpr bool kX = true, kY = true, kZ = true;
};
struct ResPlain {
  static constexpr bool kX = false, kY = false, kZ = false;
};

// a block per SM: 128 registers per thread, 168 for 16-byte vectors
template <class T, int V> constexpr int kResThreads = V * (int)sizeof(T) == 16 ? 384 : 512;
constexpr long long kResOneCell = 160000;

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// All blocks of the launch have arrived `turn` times. sync[0] counts
// arrivals, sync[1] is set when a wait ran out of its limit_ns (cleared by a
// reset of the handle). False: give up.
__device__ __forceinline__ bool grid_barrier(unsigned* sync, unsigned turn, unsigned long long limit_ns) {
  __shared__ int go;
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned want = turn * gridDim.x;
    __threadfence();
    atomicAdd(sync, 1u);
    unsigned n;
    unsigned long long end = 0;
    int ok = 1;
    for (;;) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(n) : "l"(sync) : "memory");
      if (n >= want) break;
      const unsigned long long now = global_ns();
      if (!end) end = now + limit_ns;
      if (now > end || *(volatile unsigned*)(sync + 1)) {
        atomicExch(sync + 1, 1u);
        ok = 0;
        break;
      }
    }
    __threadfence();
    go = ok;
  }
  __syncthreads();
  return go != 0;
}

// n / d for n < 2^31, by a product (d's magic pair, made on the host).
__device__ __forceinline__ int div_by(int n, DivMagic d) {
  return d.mul ? (int)(__umulhi((unsigned)n, d.mul) >> d.shift) : n;
}

// A warp's unit on a plane: 16 cells (64 bytes of a float row) by 2 V rows,
// narrow so that few units meet an x face; a thread holds V of its cells.
constexpr int kResCells = 16;
template <int V> constexpr int kResWidth = kResCells / V;
template <int V> constexpr int kResRows = 32 / kResWidth<V>;

// One launch: `nsteps` steps from *tp + toff; a.st has H in place in the
// current set, a.other the other set's H. A block takes a contiguous run of
// units in (z, y, x) order (neighbouring rows then meet in its L1).
// kBeam: an incident run's steps (a.beam): E of the read-out plane is recorded
// beside the H pass and H beside the E pass, where neither changes, and the
// E pass puts the next step's source on its plane.
template <class T, int V, bool kBeam>
__global__ void __launch_bounds__(kResThreads<T, V>, 1)
k_resident(const __grid_constant__ ResidentArgs<T> a, const int* __restrict__ tp, int toff, int nsteps, int ph_g0,
           int ph_ng, unsigned* sync, int* err) {
  const State<T>& s = a.st;
  const int u0 = (int)(a.units * blockIdx.x / gridDim.x), u1 = (int)(a.units * (blockIdx.x + 1) / gridDim.x);
  const int warps = blockDim.x / 32, warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int ph_units = ph_ng * a.ph_units;
  const int t0 = *tp + toff;
  const unsigned P = (unsigned)s.plane, W = (unsigned)s.pitch;
  const int nz = s.nz, ny = s.ny, m = s.npml;
  auto load = [](T (&v)[V], const T* from, T*) { ldg(v, from); };
  auto store = [](T (&v)[V], const T*, T* to) { stg(to, v); };

  // the phasors of step t, whose H is in h
  auto phasors = [&](T* const (&h)[3], int t) {
    for (int u = warp * gridDim.x + blockIdx.x; u < ph_units; u += warps * gridDim.x) {
      const int g = u / a.ph_units;
      phasor_cell(s, PhFields<T>{s.iex, s.iey, s.iez, h[0], h[1], h[2]}, ph_g0 + g, (u - g * a.ph_units) * 32 + lane, t);
    }
  };
  // f(y, x) for the read-out plane's cells
  auto read_out = [&](auto&& f) {
    const int per_row = (s.nx + 31) / 32;
    for (int u = warp * gridDim.x + blockIdx.x; u < ny * per_row; u += warps * gridDim.x) {
      const int y = u / per_row, x = (u - y * per_row) * 32 + lane;
      if (x < s.nx) f(y, x);
    }
  };
  // pass(z, p, i, easy) for the block's vectors: i the element index; easy:
  // no vector of the warp meets a face or edge
  const int lane_x = (lane % kResWidth<V>) * V, lane_y = lane / kResWidth<V>;
  auto sweep = [&](auto&& pass) {
    for (int u = u0 + warp; u < u1; u += warps) {
      const int r = div_by(u, a.per_row), z = div_by(r, a.per_plane);
      PairPos<T, V> p;
      p.x0 = (u - r * a.gx) * kResCells + lane_x;
      p.y = (r - z * a.gy) * kResRows<V> + lane_y;
      p.mz = (T)a.minus0;
      const bool act = p.x0 < s.nx && p.y < ny;
      const bool easy = __all_sync(0xffffffffu, !act || (z >= m && z < nz - m && p.y >= m && p.y < ny - m &&
                                                         p.x0 >= m && p.x0 + V <= s.nx - m));
      if (!act) continue;
      if (easy) {
        p.vin = true;
        p.kx = (unsigned)p.y * W + (unsigned)p.x0;
      } else {
        pair_pos<ResAll>(s, p);
      }
      pass(z, p, (unsigned)z * P + p.kx, easy);
    }
  };
  unsigned turn = 0;
  for (int n = 0; n < nsteps; ++n) {
    // H: set n & 1 (0: the current one) -> the other; in place at the end of
    // an odd run
    const bool in_place = (nsteps & 1) && n == nsteps - 1, odd = n & 1;
    T* const cur[3] = {s.ohx, s.ohy, s.ohz};
    T* const hs[3] = {odd ? a.other[0] : cur[0], odd ? a.other[1] : cur[1], odd ? a.other[2] : cur[2]};
    const bool dst_cur = odd || in_place;
    T* const hd[3] = {dst_cur ? cur[0] : a.other[0], dst_cur ? cur[1] : a.other[1], dst_cur ? cur[2] : a.other[2]};
    const int t = t0 + n;
    if (n > 0) phasors(hs, t - 1);
    if constexpr (kBeam)
      read_out([&](int y, int x) { inc_record_e<T>(a.beam.rec, s.iex, s.iey, t, y, x); });
    if (in_place && n > 0 && !grid_barrier(sync, ++turn, a.wait_ns)) break;
    sweep([&](int z, const PairPos<T, V>& p, unsigned i, bool easy) {
      T ph[6][V], pe[6][V];
      if (!easy) pair_psi<ResAll, 1>(s, p, z, ph, pe, load);
      T ex[V], ey[V], ez[V], exz[V], eyz[V], exy[V], ezy[V], hx[V], hy[V], hz[V];
      // neighbours outside the grid stand in by the cell itself: no update
      // that counts reads them
      const unsigned iz = z + 1 < nz ? i + P : i, iy = p.y + 1 < ny ? i + W : i, ix = p.x0 + V < s.pitch ? i + V : i;
      ldg(ex, s.iex + i); ldg(ey, s.iey + i); ldg(ez, s.iez + i);
      ldg(exz, s.iex + iz); ldg(eyz, s.iey + iz);
      ldg(exy, s.iex + iy); ldg(ezy, s.iez + iy);
      const T eyn = ldc(s.iey + ix), ezn = ldc(s.iez + ix);
      ldg(hx, (const T*)hs[0] + i); ldg(hy, (const T*)hs[1] + i); ldg(hz, (const T*)hs[2] + i);
      if (easy) pair_h<ResPlain>(s, p, z, t, ex, ey, ez, exz, eyz, exy, ezy, eyn, ezn, hx, hy, hz, ph);
      else pair_h<ResAll>(s, p, z, t, ex, ey, ez, exz, eyz, exy, ezy, eyn, ezn, hx, hy, hz, ph);
      stg(hd[0] + i, hx); stg(hd[1] + i, hy); stg(hd[2] + i, hz);
      if (!easy) pair_psi<ResAll, 1>(s, p, z, ph, pe, store);
    });
    if (!grid_barrier(sync, ++turn, a.wait_ns)) break;
    if constexpr (kBeam)
      read_out([&](int y, int x) { inc_record_h<T>(a.beam.rec, hd[0], hd[1], t, y, x); });
    sweep([&](int z, const PairPos<T, V>& p, unsigned i, bool easy) {
      T ph[6][V], pe[6][V];
      if (!easy) pair_psi<ResAll, 2>(s, p, z, ph, pe, load);
      T hx[V], hy[V], hz[V], hxz[V], hyz[V], hxy[V], hzy[V], ex[V], ey[V], ez[V], ca[V], cb[V];
      const unsigned iz = z > 0 ? i - P : i, iy = p.y > 0 ? i - W : i, ix = p.x0 > 0 ? i - 1 : i;
      ldg(hx, (const T*)hd[0] + i); ldg(hy, (const T*)hd[1] + i); ldg(hz, (const T*)hd[2] + i);
      ldg(hxz, (const T*)hd[0] + iz); ldg(hyz, (const T*)hd[1] + iz);
      ldg(hxy, (const T*)hd[0] + iy); ldg(hzy, (const T*)hd[2] + iy);
      const T hyp = ldc((const T*)hd[1] + ix), hzp = ldc((const T*)hd[2] + ix);
      ldg(ex, s.iex + i); ldg(ey, s.iey + i); ldg(ez, s.iez + i);
      ldg(ca, s.ca + i); ldg(cb, s.cb + i);
      if (easy) pair_e<ResPlain>(s, p, z, t, hx, hy, hz, hxz, hyz, hxy, hzy, hyp, hzp, ca, cb, ex, ey, ez, pe);
      else pair_e<ResAll>(s, p, z, t, hx, hy, hz, hxz, hyz, hxy, hzy, hyp, hzp, ca, cb, ex, ey, ez, pe);
      if constexpr (kBeam) {
        if (z == a.beam.feed_in && t + 1 < a.beam.nt_source) {
          const long long src = ((long long)(t + 1) * ny + p.y) * s.pitch + p.x0;
#pragma unroll
          for (int j = 0; j < V; ++j)
            if (inc_source_cell(s, p.y, p.x0 + j)) {
              ex[j] = a.beam.ex[src + j];
              ey[j] = a.beam.ey[src + j];
            }
        }
      }
      stg(s.oex + i, ex); stg(s.oey + i, ey); stg(s.oez + i, ez);
      if (!easy) pair_psi<ResAll, 2>(s, p, z, ph, pe, store);
    });
    if (!grid_barrier(sync, ++turn, a.wait_ns)) break;
    if (n == nsteps - 1) phasors(cur, t);
  }
  if (threadIdx.x == 0 && *(volatile unsigned*)(sync + 1)) *err = 1;
}

// Blocks of a launch (one per SM), 0 when the device cannot run it.
template <class T, int V, bool kBeam>
int resident_blocks() {
  int dev = 0, sms = 0, coop = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_resident<T, V, kBeam>, kResThreads<T, V>,
                                                    0) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return per_sm >= 1 ? sms : 0;
}

// Magic pair for n / d, n < 2^31: floor(n mul / 2^(32 + shift)); d = 1 has
// none and takes mul = 0.
DivMagic div_magic(unsigned d) {
  DivMagic r{0, 0};
  if (d <= 1) return r;
  unsigned shift = 0;
  while ((1u << shift) < d && shift < 31) ++shift;   // 2^shift >= d
  // n < 2^31: mul = ceil(2^(31 + shift) / d) fits 32 bits and is exact
  r.mul = (unsigned)(((1ULL << (31 + shift)) + d - 1) / d);
  r.shift = shift - 1;
  return r;
}

template <class T, int V, bool kBeam>
bool resident_launch(ResidentArgs<T>& a, const int* tdev, int toff, int nsteps, int ph_g0, int ph_ng, unsigned* sync,
                     int* err, cudaStream_t st) {
  const int blocks = resident_blocks<T, V, kBeam>();
  if (!blocks) return false;
  const State<T>& s = a.st;
  a.gx = (s.nx + kResCells - 1) / kResCells;
  a.gy = (s.ny + kResRows<V> - 1) / kResRows<V>;
  a.units = (long long)s.nz * a.gy * a.gx;
  a.per_row = div_magic((unsigned)a.gx);
  a.per_plane = div_magic((unsigned)a.gy);
  void* args[] = {&a, &tdev, &toff, &nsteps, &ph_g0, &ph_ng, &sync, &err};
  // sync[1] stays: after a wait that ran out the launches that follow leave at
  // their first barrier
  return cudaMemsetAsync(sync, 0, sizeof(unsigned), st) == cudaSuccess &&
         cudaLaunchCooperativeKernel((const void*)k_resident<T, V, kBeam>, dim3(blocks), dim3(kResThreads<T, V>), args, 0,
                                     st) == cudaSuccess;
}

}  // namespace

namespace {

template <class T, bool kBeam>
bool resident(ResidentArgs<T>& a, const State<T>& s, T* const other_h[3], const int* tdev, int toff, int nsteps,
              int ph_g0, int ph_ng, unsigned* sync, int* err, cudaStream_t st) {
  a.st = s;
  for (int k = 0; k < 3; ++k) a.other[k] = other_h[k];
  a.minus0 = -0.0f;
  const int n = std::max(std::max(s.ny_ph * s.nx_ph, s.nz_ph * s.ny_ph), s.nz_ph * s.nx_ph);
  a.ph_units = (n + 31) / 32;
  // one cell per thread while every cell has about a thread: a phase is then
  // one short chain (31 x 39 x 39: 8.8 us per step, 13.0 with four; 47 x 87 x 107 in
  // double: 29 with one cell, 27 with two).
  const long long cells = (long long)s.nz * s.ny * s.nx;
  if (cells <= kResOneCell)
    return resident_launch<T, 1, kBeam>(a, tdev, toff, nsteps, ph_g0, ph_ng, sync, err, st);
  return resident_launch<T, 16 / (int)sizeof(T), kBeam>(a, tdev, toff, nsteps, ph_g0, ph_ng, sync, err, st);
}

}  // namespace

template <class T>
bool launch_resident(const State<T>& s, T* const other_h[3], const int* tdev, int toff, int nsteps, int ph_g0,
                     int ph_ng, unsigned* sync, int* err, unsigned long long wait_ns, cudaStream_t st) {
  ResidentArgs<T> a;
  memset(&a, 0, sizeof(a));
  a.wait_ns = wait_ns;
  return resident<T, false>(a, s, other_h, tdev, toff, nsteps, ph_g0, ph_ng, sync, err, st);
}

template <class T>
bool launch_resident_beam(const State<T>& s, T* const other_h[3], const IncidentBeam<T>& beam, const int* tdev,
                          int toff, int nsteps, unsigned* sync, int* err, unsigned long long wait_ns,
                          cudaStream_t st) {
  ResidentArgs<T> a;
  memset(&a, 0, sizeof(a));
  a.beam = beam;
  a.wait_ns = wait_ns;
  return resident<T, true>(a, s, other_h, tdev, toff, nsteps, 0, 0, sync, err, st);
}

#define FDTD_RESIDENT_INSTANCES(T)                                                                                \
  template bool launch_resident_beam<T>(const State<T>&, T* const[3], const IncidentBeam<T>&, const int*, int,    \
                                        int, unsigned*, int*, unsigned long long, cudaStream_t);                  \
  template bool launch_resident<T>(const State<T>&, T* const[3], const int*, int, int, int, int, unsigned*, int*, \
                                   unsigned long long, cudaStream_t);
FDTD_RESIDENT_INSTANCES(float)
FDTD_RESIDENT_INSTANCES(double)

}  // namespace fdtd
