// fdtd_split.cu -- the split step (H pass, E pass), the phasor pass, the
// step-counter advance and the eps/sigma -> Ca/Cb kernel.
//
// The split step updates the fields in place: the H pass reads E and writes
// H, the E pass reads H and writes E, so no cell is read after another
// thread wrote it within a pass. It moves 80 B per FP32 cell-update
// (H pass 36 B, E pass 44 B) against the 56 B minimum of a fused pass.
// Each thread updates four consecutive x cells with vector loads and
// stores; interior vectors take the plain curl update, the rest (CPML
// faces, domain edges, the injection plane) h_vec / e_vec. The same passes,
// restricted to a list of boxes and run source -> destination, update the
// shell of the fused step (fdtd_fused.cu).
#include <cstring>

#include <algorithm>

#include "fdtd_launch.h"
#include "fdtd_split.cuh"

namespace fdtd {

__global__ void k_advance(int* t, int n) { *t += n; }

// The passes over a list of boxes (the whole grid for the split step, the
// shell of the fused step), bl.planes planes of one box tile per 128-thread block. A box tile is `width` lanes
// (width * kVec x cells) by 128 / width rows.
__device__ __forceinline__ const ShellBox& find_box(const ShellBoxes& bl, int bid) {
  int k = 0;
  while (k + 1 < bl.n && bid >= bl.b[k + 1].first) ++k;
  return bl.b[k];
}

// Resident blocks per SM the split passes ask for (float: register cap 72;
// the passes are latency-bound, but at 64 registers the division's double
// products spill: a 32-member batch takes 1.40 ms per step with 8 blocks,
// 1.31 with 7)
template <class T>
constexpr int split_min_blocks() { return sizeof(T) == 4 ? 7 : 1; }

template <class T, bool kH>
__global__ void __launch_bounds__(128, split_min_blocks<T>()) k_shell(State<T> s, const int* __restrict__ tp, int toff,
                                               ShellBoxes bl) {
  const int bid = blockIdx.x;
  const ShellBox& b = find_box(bl, bid);
  int local = bid - b.first;
  const int bx = local % b.gx;
  local /= b.gx;
  const int by = local % b.gy;
  const int za = b.z0 + (local / b.gy) * bl.planes;
  const int zb = min(b.z1, za + bl.planes);
  const int lane = threadIdx.x % b.width, row = threadIdx.x / b.width;
  const int x0 = b.x0 + (bx * b.width + lane) * kVec;
  const int y = b.y0 + by * (128 / b.width) + row;
  const bool act = x0 < b.x1 && y < b.y1;
  const int t = *tp + toff;
  for (int z = za; z < zb; ++z) {   // block-uniform trip count (shuffles inside)
    if (kH) h_split_vec(s, t, z, y, x0, lane, b.width, act);
    else e_split_vec(s, t, z, y, x0, lane, b.width, act);
  }
}

// One thread per phasor cell; g0 + blockIdx.y selects the plane group.
template <class T>
__global__ void __launch_bounds__(256) k_phasors(State<T> s, const int* __restrict__ tp, int toff, int g0) {
  phasor_cell(s, g0 + (int)blockIdx.y, (int)(blockIdx.x * blockDim.x + threadIdx.x), *tp + toff);
}

// The phasors of two steps (the pair step): of the fields between them at
// step t, then of the destination set at t + 1. The stored values are read
// and written once for both; each addition is rounded to T as in ph_acc4.
// At 203 x 761 x 761 the pass takes 50 us per pair (two single passes 117; 96
// while the x planes were read from the fields, eight columns per sector).
template <class T>
__global__ void __launch_bounds__(256) k_phasors_pair(State<T> s, PairMid<T> mid, const int* __restrict__ tp,
                                                      int toff, int g0) {
  using M = R<T>;
  const int g = g0 + (int)blockIdx.y, idx = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  const int t = *tp + toff;
  int a, b;
  if (!phasor_at(s, g, idx, a, b)) return;
  double m0[4], m1[4], ph[8];
  {
    // cell (a, b) in the mid planes; the x planes of both steps are there
    const int m = s.npml;
    const long long P = s.plane, W = s.pitch;
    if (g < 2) {
      phasor_means(g, mid.z[0], mid.z[1], mid.z[2], mid.z[3], (g == 0 ? 1 : 3) * P + (m + a) * W + (m + b), P, W, m0);
    } else if (g < 4) {
      const long long i = ((long long)(m + a) * s.ny + (m + b)) * 4 + (g == 2 ? 1 : 3);
      phasor_means(g, mid.x[0][0], mid.x[0][1], mid.x[0][2], mid.x[0][3], i, 4LL * s.ny, 4, m0);
      phasor_means(g, mid.x[1][0], mid.x[1][1], mid.x[1][2], mid.x[1][3], i, 4LL * s.ny, 4, m1);
    } else {
      phasor_means(g, mid.y[0], mid.y[1], mid.y[2], mid.y[3], ((long long)(m + a) * 4 + (g == 4 ? 1 : 3)) * W + (m + b),
                   4 * W, W, m0);
    }
  }
  if (g < 2 || g >= 4)
    phasor_means(s, PhFields<T>{s.oex, s.oey, s.oez, s.ohx, s.ohy, s.ohz}, g, a, b, m1);
#pragma unroll
  for (int j = 0; j < 8; ++j) ph[j] = s.phase[4 * (long long)t + j];
  if (s.kahan) {
    ph_acc4(s, 4 * g, idx, m0, ph[0], ph[1], ph[2], ph[3]);
    ph_acc4(s, 4 * g, idx, m1, ph[4], ph[5], ph[6], ph[7]);
    return;
  }
  T v[4][2];
#pragma unroll
  for (int j = 0; j < 4; ++j) ld2(v[j], s.ph + s.ph_off[4 * g + j] + 2 * (long long)idx);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int e = j < 2 ? 0 : 2;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      v[j][q] = M::from_double(__dadd_rn((double)v[j][q], __dmul_rn(m0[j], ph[e + q])));
      v[j][q] = M::from_double(__dadd_rn((double)v[j][q], __dmul_rn(m1[j], ph[4 + e + q])));
    }
    st2(s.ph + s.ph_off[4 * g + j] + 2 * (long long)idx, v[j][0], v[j][1]);
  }
}

// ---------------------------------------------------------------------------
// batched step: the split passes and the phasor pass of many simulations in
// one launch each. Block b belongs to the model m with
// start[m] <= b < start[m + 1]; the model's State lives in device memory.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int find_model(const int* __restrict__ start, int n, int bid) {
  int lo = 0, hi = n - 1;   // last m with start[m] <= bid
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (start[mid] <= bid) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

template <class T, bool kH>
__global__ void __launch_bounds__(128, split_min_blocks<T>()) k_batch_split(const BatchModel<T>* __restrict__ bm,
                                                     const int* __restrict__ start, int n, int toff) {
  const int bid = blockIdx.x;
  const int mi = find_model(start, n, bid);
  const BatchModel<T>& b = bm[mi];
  // the member's State, staged once per block in shared memory: the update
  // reads its scalars, pointers and profiles many times per thread
  static_assert(sizeof(State<T>) % 8 == 0, "State is copied in 8-byte words");
  __shared__ unsigned long long st_words[sizeof(State<T>) / 8];
  {
    const unsigned long long* src = reinterpret_cast<const unsigned long long*>(&b.s);
    for (int k = threadIdx.x; k < (int)(sizeof(State<T>) / 8); k += blockDim.x) st_words[k] = src[k];
  }
  __syncthreads();
  const State<T>& s = *reinterpret_cast<const State<T>*>(st_words);
  int local = bid - start[mi];
  const int bx = local % b.gx;
  local /= b.gx;
  const int by = local % b.gy;
  const int za = (local / b.gy) * kBatchShellPlanes;   // kBatchShellPlanes planes per block
  const int zb = min(s.nz, za + kBatchShellPlanes);
  const int lane = threadIdx.x % b.width, row = threadIdx.x / b.width;
  const int x0 = (bx * b.width + lane) * kVec;
  const int y = by * (128 / b.width) + row;
  const int t = *b.tdev + toff;
  for (int z = za; z < zb; ++z) {   // block-uniform trip count (shuffles inside)
    if (kH) h_split_vec(s, t, z, y, x0, lane, b.width, true);
    else e_split_vec(s, t, z, y, x0, lane, b.width, true);
  }
}

// The shell boxes of every member (BatchShellBox): block b belongs to the
// last box whose first block is <= b and sweeps kBatchShellPlanes planes of
// one box tile (the staged State serves them all). The member's State is
// staged in shared memory; the E pass reads H from the destination set.
template <class T, bool kH>
__global__ void __launch_bounds__(128, split_min_blocks<T>())
k_batch_shell(const BatchModel<T>* __restrict__ bm, const BatchShellBox* __restrict__ boxes, int nboxes, int toff) {
  const int bid = blockIdx.x;
  int lo = 0, hi = nboxes - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (boxes[mid].b.first <= bid) lo = mid;
    else hi = mid - 1;
  }
  const int member = boxes[lo].member;
  const ShellBox b = boxes[lo].b;
  static_assert(sizeof(State<T>) % 8 == 0, "State is copied in 8-byte words");
  __shared__ unsigned long long st_words[sizeof(State<T>) / 8];
  {
    const unsigned long long* src = reinterpret_cast<const unsigned long long*>(&bm[member].s);
    for (int k = threadIdx.x; k < (int)(sizeof(State<T>) / 8); k += blockDim.x) st_words[k] = src[k];
  }
  __syncthreads();
  State<T>& s = *reinterpret_cast<State<T>*>(st_words);
  if (!kH) {
    if (threadIdx.x == 0) { s.ihx = s.ohx; s.ihy = s.ohy; s.ihz = s.ohz; }
    __syncthreads();
  }
  int local = bid - b.first;
  const int bx = local % b.gx;
  local /= b.gx;
  const int by = local % b.gy;
  const int za = b.z0 + (local / b.gy) * kBatchShellPlanes;
  const int zb = min(b.z1, za + kBatchShellPlanes);
  const int lane = threadIdx.x % b.width, row = threadIdx.x / b.width;
  const int x0 = b.x0 + (bx * b.width + lane) * kVec;
  const int y = b.y0 + by * (128 / b.width) + row;
  const bool act = x0 < b.x1 && y < b.y1;
  const int t = *bm[member].tdev + toff;
  for (int z = za; z < zb; ++z) {   // block-uniform trip count (shuffles inside)
    if (kH) h_split_vec(s, t, z, y, x0, lane, b.width, act);
    else e_split_vec(s, t, z, y, x0, lane, b.width, act);
  }
}

template <class T>
__global__ void __launch_bounds__(256) k_batch_phasors(const BatchModel<T>* __restrict__ bm,
                                                       const int* __restrict__ start, int n,
                                                       int toff, int* __restrict__ reset) {
  const int bid = blockIdx.x;
  // the tile counter of the step's tile-queue kernel, which has finished
  // (stream order), starts the next step at zero
  if (reset && bid == 0 && threadIdx.x == 0) *reset = 0;
  const int mi = find_model(start, n, bid);
  const BatchModel<T>& b = bm[mi];
  const int local = bid - start[mi];
  const int per_group = (b.ph_n + 255) / 256;
  const int g = local / per_group;
  const int idx = (local - g * per_group) * 256 + threadIdx.x;
  phasor_cell(b.s, g, idx, *b.tdev + toff);
}

template <class T>
__global__ void k_batch_advance(const BatchModel<T>* __restrict__ bm, int n, int steps) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) *bm[i].tdev += steps;
}

// ---------------------------------------------------------------------------
// Ca, Cb from eps_r, sigma (materials/materials.py:23-68). The reference
// evaluates every operation in the array dtype: eps0, dt and dx are first
// rounded to it (numpy scalar promotion), then
//   perm = eps_r * eps0; x = (sigma * dt) / (2 * perm)
//   Ca = (1 - x) / (1 + x);  Cb = (dt / (perm * dx)) / (1 + x)
// Cells at z >= nz_mat are vacuum (eps_r = 1, sigma = 0).
// ---------------------------------------------------------------------------
template <class T>
__global__ void k_eps_sigma(int nx, int ny, int nz, int nz_mat, int pitch,
                            const T* __restrict__ eps, const T* __restrict__ sig,
                            T eps0, T dt, T dx, T* __restrict__ ca, T* __restrict__ cb) {
  using M = R<T>;
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y;
  const int z = blockIdx.z;
  if (x >= nx) return;
  T e = T(1), sg = T(0);
  if (z < nz_mat) {
    const long long j = ((long long)z * ny + y) * nx + x;
    e = eps[j];
    sg = sig[j];
  }
  const T perm = M::mul(e, eps0);
  const T xx = M::div(M::mul(sg, dt), M::mul(T(2), perm));
  const T den = M::add(T(1), xx);
  const long long i = ((long long)z * ny + y) * pitch + x;
  ca[i] = M::div(M::sub(T(1), xx), den);
  cb[i] = M::div(M::div(dt, M::mul(perm, dx)), den);
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
void add_shell_box(ShellBoxes& bl, int x0, int x1, int y0, int y1, int z0, int z1) {
  if (x0 >= x1 || y0 >= y1 || z0 >= z1) return;
  if (bl.n >= kMaxShellBoxes) {
    ++bl.dropped;
    return;
  }
  ShellBox& b = bl.b[bl.n++];
  b.x0 = x0; b.x1 = x1; b.y0 = y0; b.y1 = y1; b.z0 = z0; b.z1 = z1;
  // row width with the least x padding (ties: the wider rows)
  long long best = -1;
  for (int w : {32, 16, 8, 4}) {
    const long long gx = (x1 - x0 + 4 * w - 1) / (4 * w), gy = (y1 - y0 + 128 / w - 1) / (128 / w);
    const long long padded = gx * 4 * w * gy * (128 / w);
    if (best < 0 || padded < best) { best = padded; b.width = w; }
  }
  b.gx = (x1 - x0 + b.width * kVec - 1) / (b.width * kVec);
  b.gy = (y1 - y0 + 128 / b.width - 1) / (128 / b.width);
  b.first = bl.total_blocks;
  bl.total_blocks += b.gx * b.gy * (z1 - z0);
}

template <class T>
void launch_split_step(const State<T>& s, const int* tdev, int toff, cudaStream_t st) {
  ShellBoxes whole;
  memset(&whole, 0, sizeof(whole));
  add_shell_box(whole, 0, s.nx, 0, s.ny, 0, s.nz);
  launch_shell_pass<T>(s, tdev, toff, whole, true, st);
  launch_shell_pass<T>(s, tdev, toff, whole, false, st);
}

template <class T>
void launch_phasors(const State<T>& s, const int* tdev, int toff, cudaStream_t st, int g0, int ng) {
  if (ng <= 0) return;
  int n = s.ny_ph * s.nx_ph;
  n = max(n, s.nz_ph * s.ny_ph);
  n = max(n, s.nz_ph * s.nx_ph);
  const dim3 grd((n + 255) / 256, ng, 1);
  k_phasors<T><<<grd, 256, 0, st>>>(s, tdev, toff, g0);
}

template <class T>
void launch_phasors_pair(const State<T>& s, const PairMid<T>& mid, const int* tdev, int toff, cudaStream_t st,
                         int g0, int ng) {
  if (ng <= 0) return;
  const int n = max(max(s.ny_ph * s.nx_ph, s.nz_ph * s.ny_ph), s.nz_ph * s.nx_ph);
  const dim3 grd((n + 255) / 256, ng, 1);
  k_phasors_pair<T><<<grd, 256, 0, st>>>(s, mid, tdev, toff, g0);
}

template <class T>
void launch_batch_step(const BatchModel<T>* bm, const int* start, int n, int blocks,
                       const int* start_ph, int blocks_ph, int toff, cudaStream_t st) {
  k_batch_split<T, true><<<blocks, 128, 0, st>>>(bm, start, n, toff);
  k_batch_split<T, false><<<blocks, 128, 0, st>>>(bm, start, n, toff);
  k_batch_phasors<T><<<blocks_ph, 256, 0, st>>>(bm, start_ph, n, toff, nullptr);
}

template <class T>
void launch_batch_phasors(const BatchModel<T>* bm, const int* start_ph, int n, int blocks_ph, int toff,
                          int* reset, cudaStream_t st) {
  k_batch_phasors<T><<<blocks_ph, 256, 0, st>>>(bm, start_ph, n, toff, reset);
}

template <class T>
void launch_batch_shell(const BatchModel<T>* bm, const BatchShellBox* boxes, int nboxes, int blocks, bool h_pass,
                        int toff, cudaStream_t st) {
  if (nboxes <= 0 || blocks <= 0) return;
  if (h_pass) k_batch_shell<T, true><<<blocks, 128, 0, st>>>(bm, boxes, nboxes, toff);
  else k_batch_shell<T, false><<<blocks, 128, 0, st>>>(bm, boxes, nboxes, toff);
}

template <class T>
void launch_batch_advance(const BatchModel<T>* bm, int n, int steps, cudaStream_t st) {
  k_batch_advance<T><<<(n + 127) / 128, 128, 0, st>>>(bm, n, steps);
}

template <class T>
void launch_shell_pass(const State<T>& s, const int* tdev, int toff, const ShellBoxes& bl,
                       bool h_pass, cudaStream_t st) {
  if (bl.n == 0 || bl.total_blocks == 0) return;
  // Several planes per block amortise the block's set-up, but only where
  // one plane per block gives many waves of blocks: 148 SMs hold about
  // 1036 of these blocks at once (7 each). add_shell_box numbered the
  // blocks one plane each; renumber for the choice.
  constexpr int kResident = 148 * 7;
  ShellBoxes p = bl;
  p.planes = bl.total_blocks >= 16 * kResident ? 4 : bl.total_blocks >= 8 * kResident ? 2 : 1;
  p.total_blocks = 0;
  for (int k = 0; k < p.n; ++k) {
    ShellBox& b = p.b[k];
    b.first = p.total_blocks;
    p.total_blocks += b.gx * b.gy * ((b.z1 - b.z0 + p.planes - 1) / p.planes);
  }
  if (h_pass) k_shell<T, true><<<p.total_blocks, 128, 0, st>>>(s, tdev, toff, p);
  else k_shell<T, false><<<p.total_blocks, 128, 0, st>>>(s, tdev, toff, p);
}

void launch_advance(int* tdev, int n, cudaStream_t st) {
  k_advance<<<1, 1, 0, st>>>(tdev, n);
}

// ---------------------------------------------------------------------------
// non-finite check: flags[0] = 1 and flags[1] = step when any of the six
// fields holds a NaN or an infinity (cells, padding included: the padding
// is never written and stays zero). The first detection wins.
// ---------------------------------------------------------------------------
template <class T>
__global__ void __launch_bounds__(256) k_check_finite(FieldPtrs<T> f, long long vol, int step,
                                                      int* __restrict__ flags) {
  if (*(volatile int*)flags) return;
  bool bad = false;
  for (int c = 0; c < 6; ++c) {
    const T* p = f.p[c];
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < vol;
         i += (long long)gridDim.x * blockDim.x)
      bad |= !isfinite(p[i]);
  }
  if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) {
    if (atomicCAS(flags, 0, 1) == 0) flags[1] = step;
  }
}

template <class T>
void launch_check_finite(const FieldPtrs<T>& f, long long vol, int step, int* flags, cudaStream_t st) {
  k_check_finite<T><<<8 * 148, 256, 0, st>>>(f, vol, step, flags);
}

template void launch_check_finite<float>(const FieldPtrs<float>&, long long, int, int*, cudaStream_t);
template void launch_check_finite<double>(const FieldPtrs<double>&, long long, int, int*, cudaStream_t);

// Packed rows (nx elements each) into pitched rows.
template <class T>
__global__ void __launch_bounds__(256) k_repitch(T* __restrict__ dst, const T* __restrict__ src, int nx,
                                                 long long rows, int pitch) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= nx) return;
  for (long long r = blockIdx.y; r < rows; r += gridDim.y) dst[r * pitch + x] = src[r * nx + x];
}

template <class T>
void launch_repitch(T* dst, const T* src, int nx, long long rows, int pitch, cudaStream_t st) {
  const dim3 grd((nx + 255) / 256, (unsigned)std::min<long long>(rows, 65535), 1);
  k_repitch<T><<<grd, 256, 0, st>>>(dst, src, nx, rows, pitch);
}

// Pitched rows into packed ones, for read-backs: a pitched device-to-host
// copy of short rows moves one row at a time (133-cell rows into pageable
// memory: 17 ms for 34 MB).
template <class T>
__global__ void __launch_bounds__(256) k_unpitch(T* __restrict__ dst, const T* __restrict__ src, int nx,
                                                 long long rows, int pitch) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= nx) return;
  for (long long r = blockIdx.y; r < rows; r += gridDim.y) dst[r * nx + x] = src[r * pitch + x];
}

template <class T>
void launch_unpitch(T* dst, const T* src, int nx, long long rows, int pitch, cudaStream_t st) {
  const dim3 grd((nx + 255) / 256, (unsigned)std::min<long long>(rows, 65535), 1);
  k_unpitch<T><<<grd, 256, 0, st>>>(dst, src, nx, rows, pitch);
}

template void launch_unpitch<float>(float*, const float*, int, long long, int, cudaStream_t);
template void launch_unpitch<double>(double*, const double*, int, long long, int, cudaStream_t);
template void launch_repitch<float>(float*, const float*, int, long long, int, cudaStream_t);
template void launch_repitch<double>(double*, const double*, int, long long, int, cudaStream_t);

template <class T>
void launch_eps_sigma(int nx, int ny, int nz, int nz_mat, int pitch, const T* eps,
                      const T* sig, T eps0, T dt, T dx, T* ca, T* cb, cudaStream_t st) {
  const dim3 grd((nx + 127) / 128, ny, nz);
  k_eps_sigma<T><<<grd, 128, 0, st>>>(nx, ny, nz, nz_mat, pitch, eps, sig, eps0, dt, dx, ca, cb);
}

template void launch_split_step<float>(const State<float>&, const int*, int, cudaStream_t);
template void launch_split_step<double>(const State<double>&, const int*, int, cudaStream_t);
template void launch_shell_pass<float>(const State<float>&, const int*, int, const ShellBoxes&,
                                       bool, cudaStream_t);
template void launch_shell_pass<double>(const State<double>&, const int*, int, const ShellBoxes&,
                                        bool, cudaStream_t);
template void launch_batch_step<float>(const BatchModel<float>*, const int*, int, int, const int*,
                                       int, int, cudaStream_t);
template void launch_batch_step<double>(const BatchModel<double>*, const int*, int, int,
                                        const int*, int, int, cudaStream_t);
template void launch_batch_phasors<float>(const BatchModel<float>*, const int*, int, int, int, int*,
                                          cudaStream_t);
template void launch_batch_phasors<double>(const BatchModel<double>*, const int*, int, int, int, int*,
                                           cudaStream_t);
template void launch_batch_shell<float>(const BatchModel<float>*, const BatchShellBox*, int, int, bool, int,
                                       cudaStream_t);
template void launch_batch_shell<double>(const BatchModel<double>*, const BatchShellBox*, int, int, bool, int,
                                        cudaStream_t);
template void launch_batch_advance<float>(const BatchModel<float>*, int, int, cudaStream_t);
template void launch_batch_advance<double>(const BatchModel<double>*, int, int, cudaStream_t);
template void launch_phasors<float>(const State<float>&, const int*, int, cudaStream_t, int, int);
template void launch_phasors<double>(const State<double>&, const int*, int, cudaStream_t, int, int);
template void launch_phasors_pair<float>(const State<float>&, const PairMid<float>&, const int*, int, cudaStream_t,
                                         int, int);
template void launch_phasors_pair<double>(const State<double>&, const PairMid<double>&, const int*, int,
                                          cudaStream_t, int, int);
template void launch_eps_sigma<float>(int, int, int, int, int, const float*, const float*, float,
                                      float, float, float*, float*, cudaStream_t);
template void launch_eps_sigma<double>(int, int, int, int, int, const double*, const double*,
                                       double, double, double, double*, double*, cudaStream_t);

}  // namespace fdtd
