// near2far.cu -- near-to-far transform of the top phasor plane.
//
// Restates FarFieldTransform (fdtdsarsim/near2far.py:28-156) on the device:
// surface currents J = (-Hy, Hx) and M = (Ey, -Ex) on the plane z = z_val
// are integrated against exp(j k r_hat . r') with composite Simpson weights
// (scipy.integrate.simpson on an odd sample count, x first then y), giving
// the N and L potentials, then E/H theta/phi at radius r. All arithmetic is
// float64, as in the reference (complex128, near2far.py:66-68).
//
// The exponential is a product of a factor in x and one in y, so a direction
// needs nx + ny sines and cosines instead of nx ny, and the integral of the
// four planes over x, for all directions, is one complex matrix product
//   R[a, (y, c)] = sum_x A[a, x] P_c[y, x]
// (A the weighted x factors, P_c the planes as given), which k_n2f_rows runs
// in 64 x 64 tiles on the FP64 pipes; k_n2f_finish sums R over y against the
// y factors. 161 directions of a 741 x 741 plane of
// complex64: kernels 1953 us with one block and nx ny sines per direction, 244
// us so (FP64 pipes; the error against 80-bit sums is the same, 1.1e-15);
// the whole call 18.8 ms before, 2.5 ms now (the rest is the 18 MB upload).
#include <cuda_runtime.h>

#include "fdtd_launch.h"

namespace fdtd {

namespace {

constexpr int kN2fThreads = 256;

__device__ __forceinline__ double simpson_w(int i, int n) {
  if (i == 0 || i == n - 1) return 1.0;
  return (i & 1) ? 4.0 : 2.0;
}

// Directions of one pass: a = ip * ntheta + it for it in [0, ntheta).
struct N2fAngles {
  const double* thetas;   // radians
  const double* phis;
  int ntheta, first, count;
  __device__ __forceinline__ double theta(int a) const { return thetas[(first + a) % ntheta]; }
  __device__ __forceinline__ double phi(int a) const { return phis[(first + a) / ntheta]; }
};

// hi + lo: a product or sum carried to twice double precision (the error of
// one operation, by FMA or Knuth's two-sum).
struct Twofold {
  double hi, lo;
};
__device__ __forceinline__ Twofold times(Twofold a, double b) {
  const double p = __dmul_rn(a.hi, b);
  return {p, __fma_rn(a.lo, b, __fma_rn(a.hi, b, -p))};
}
__device__ __forceinline__ Twofold plus(Twofold a, Twofold b) {
  const double s = __dadd_rn(a.hi, b.hi), t = __dsub_rn(s, a.hi);
  const double e = __dadd_rn(__dsub_rn(a.hi, __dsub_rn(s, t)), __dsub_rn(b.hi, t));
  return {s, __dadd_rn(e, __dadd_rn(a.lo, b.lo))};
}

// The weighted factors of every direction: fx (count, nx), fy (count, ny);
// the plane's height goes with y. A column's phase error would enter every
// row of the integral, so the phases (up to some hundred radians) are
// carried beyond double, as the sum over cells with their own roundings
// would average them.
__global__ void __launch_bounds__(kN2fThreads) k_n2f_factors(N2fAngles an, int nx, int ny, double dx, double z_val,
                                                             double k, double2* __restrict__ fx,
                                                             double2* __restrict__ fy) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, a = blockIdx.y;
  if (i >= nx + ny) return;
  const double st = sin(an.theta(a)), ct = cos(an.theta(a)), ph = an.phi(a);
  // x_loc = np.arange(-(nx-1)//2, (nx-1)//2 + 1) * dx  (near2far.py:58-60)
  const Twofold kst = times(times(Twofold{k, 0.0}, dx), st);
  Twofold arg;
  double w, s, c;
  if (i < nx) {
    arg = times(times(kst, cos(ph)), (double)(i - nx / 2));
    w = simpson_w(i, nx);
  } else {
    arg = plus(times(times(kst, sin(ph)), (double)(i - nx - ny / 2)), times(times(Twofold{k, 0.0}, z_val), ct));
    w = simpson_w(i - nx, ny);
  }
  sincos(arg.hi, &s, &c);
  const double re = c - arg.lo * s, im = s + arg.lo * c;
  (i < nx ? fx[(size_t)a * nx + i] : fy[(size_t)a * ny + (i - nx)]) = make_double2(w * re, w * im);
}

constexpr int kN2fTile = 64, kN2fK = 16;   // 4 x 4 complex sums per thread of 256

// R[a][y * 4 + c] = sum_x fx[a][x] P_c[y][x] for a tile of 64 directions by
// 64 columns; planes: P_0 .. P_3, (ny, nx) each, one after another. Where
// there are few tiles of long rows, part z of `parts` sums every cell of its
// share of the rows, into its own R.
template <class C, bool kParts>
__global__ void __launch_bounds__(kN2fThreads)
k_n2f_rows(const C* __restrict__ planes, const double2* __restrict__ fx, int count, int nx, int ny, int part_cells,
           double2* __restrict__ out) {
  __shared__ double2 sa[kN2fK][kN2fTile + 1], sp[kN2fK][kN2fTile + 1];
  const int a0 = blockIdx.x * kN2fTile, j0 = blockIdx.y * kN2fTile, cols = 4 * ny;
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  double2 acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = make_double2(0.0, 0.0);
  const int x_end = kParts ? min(nx, (int)(blockIdx.z + 1) * part_cells) : nx;
  if (kParts) out += (size_t)blockIdx.z * count * cols;
  for (int x0 = kParts ? blockIdx.z * part_cells : 0; x0 < x_end; x0 += kN2fK) {
    // 16 threads read 16 consecutive x of a direction or plane row
    const int x = x0 + tx;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int a = a0 + ty + 16 * i, j = j0 + ty + 16 * i;
      sa[tx][ty + 16 * i] = x < x_end && a < count ? fx[(size_t)a * nx + x] : make_double2(0.0, 0.0);
      double2 v = make_double2(0.0, 0.0);
      if (x < x_end && j < cols) {
        const C q = planes[((size_t)(j & 3) * ny + (j >> 2)) * nx + x];
        v = make_double2((double)q.x, (double)q.y);
      }
      sp[tx][ty + 16 * i] = v;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kN2fK; ++k) {
      double2 u[4], v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        u[i] = sa[k][ty + 16 * i];
        v[i] = sp[k][tx + 16 * i];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[i][j].x += u[i].x * v[j].x - u[i].y * v[j].y;
          acc[i][j].y += u[i].x * v[j].y + u[i].y * v[j].x;
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int a = a0 + ty + 16 * i, col = j0 + tx + 16 * j;
      if (a < count && col < cols) out[(size_t)a * cols + col] = acc[i][j];
    }
}

// One block per direction: the sums of R over y against fy (and over its
// parts), then the potentials and the far field.
template <bool kParts>
__global__ void __launch_bounds__(kN2fThreads)
k_n2f_finish(N2fAngles an, const double2* __restrict__ rows, int parts, const double2* __restrict__ fy, int ny,
             double dx, double k, double r, long long plane, double2* __restrict__ out) {
  const int a = blockIdx.x;
  // sums of ex, ey, hx, hy (re, im)
  double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int y = threadIdx.x; y < ny; y += blockDim.x) {
    const double2 f = fy[(size_t)a * ny + y];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      double2 v = rows[((size_t)a * ny + y) * 4 + c];
      for (int p = 1; kParts && p < parts; ++p) {
        const double2 w = rows[(((size_t)p * an.count + a) * ny + y) * 4 + c];
        v = make_double2(v.x + w.x, v.y + w.y);
      }
      acc[2 * c] += f.x * v.x - f.y * v.y;
      acc[2 * c + 1] += f.x * v.y + f.y * v.x;
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j)
    for (int o = 16; o > 0; o >>= 1) acc[j] += __shfl_down_sync(0xffffffffu, acc[j], o);
  __shared__ double red[kN2fThreads / 32][8];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  if (lane == 0)
    for (int j = 0; j < 8; ++j) red[warp][j] = acc[j];
  __syncthreads();
  if (threadIdx.x != 0) return;
  double s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  const double h = dx / 3.0;  // Simpson factor per axis
  for (int j = 0; j < 8; ++j) {
    for (int w = 0; w < kN2fThreads / 32; ++w) s[j] += red[w][j];
    s[j] *= h * h;
  }
  const double th = an.theta(a), ph = an.phi(a);
  const double ct = cos(th), sp = sin(ph), cp = cos(ph);
  // Taflove 8.33a/b, 8.34a/b with J = (-Hy, Hx), M = (Ey, -Ex)
  const double2 ex = make_double2(s[0], s[1]), ey = make_double2(s[2], s[3]);
  const double2 hx = make_double2(s[4], s[5]), hy = make_double2(s[6], s[7]);
  const double2 Nt = make_double2(ct * (hx.x * sp - hy.x * cp), ct * (hx.y * sp - hy.y * cp));
  const double2 Np = make_double2(hy.x * sp + hx.x * cp, hy.y * sp + hx.y * cp);
  const double2 Lt = make_double2(ct * (ey.x * cp - ex.x * sp), ct * (ey.y * cp - ex.y * sp));
  const double2 Lp = make_double2(-ey.x * sp - ex.x * cp, -ey.y * sp - ex.y * cp);
  const double eta0 = 376.730313668;
  // ff_weight = 1j k exp(-1j k r) / (4 pi r)   (near2far.py:71-72)
  const double c = k / (4.0 * M_PI * r);
  double sr, cr;
  sincos(k * r, &sr, &cr);
  const double2 ffw = make_double2(c * sr, c * cr);  // 1j*c*(cos - j sin)
  auto cm = [](double2 u, double2 v) { return make_double2(u.x * v.x - u.y * v.y, u.x * v.y + u.y * v.x); };
  const long long o = an.first + a;
  out[0 * plane + o] = cm(ffw, make_double2(-Lp.x - eta0 * Nt.x, -Lp.y - eta0 * Nt.y));
  out[1 * plane + o] = cm(ffw, make_double2(Lt.x - eta0 * Np.x, Lt.y - eta0 * Np.y));
  out[2 * plane + o] = cm(ffw, make_double2(Np.x - Lt.x / eta0, Np.y - Lt.y / eta0));
  out[3 * plane + o] = cm(ffw, make_double2(-Nt.x - Lp.x / eta0, -Nt.y - Lp.y / eta0));
}

}  // namespace

namespace {

// Parts of the rows' sums: one, unless a plane of rows of 512 cells or more
// leaves 16 tiles or fewer, whose sums would run one after another on as many
// SMs (4 directions of 3 x 20001 cells: 6.3 ms in one part, 1.0 in 148). By the
// call's directions, not the pass's: a sum does not depend on how much memory
// there is.
int row_parts(int nx, int ny, long long angles) {
  const long long tiles = ((angles + kN2fTile - 1) / kN2fTile) * ((4LL * ny + kN2fTile - 1) / kN2fTile);
  return nx >= 512 && tiles <= 16 ? (int)(148 / tiles < nx / 64 ? 148 / tiles : nx / 64) : 1;
}

size_t direction_bytes(int nx, int ny, int parts) {
  return ((size_t)nx + (size_t)ny * (1 + 4 * (size_t)parts)) * sizeof(double2);
}

}  // namespace

// A pass of 1024 directions, or as many as 32 MB hold where planes are small
// (a pass is three launches; 16384 directions of 19 x 19 cells: 1.3 ms in
// passes of 1024, 1.0 so).
int near2far_pass(int nx, int ny, long long angles) {
  const long long most = (32LL << 20) / (long long)direction_bytes(nx, ny, 1);
  const long long n = most < 1024 ? 1024 : most > 65535 ? 65535 : most;
  return (int)(angles < n ? angles : n);
}

size_t near2far_scratch(int nx, int ny, long long angles, int pass) {
  return (size_t)pass * direction_bytes(nx, ny, row_parts(nx, ny, angles));
}

int near2far_run(const void* planes, bool single, int nx, int ny, double dx, double z_val, double k,
                 const double* thetas, int ntheta, const double* phis, int nphi, double r, void* scratch, int pass,
                 double* out, cudaStream_t st) {
  const long long total = (long long)nphi * ntheta;
  for (long long first = 0; first < total; first += pass) {
    const int n = (int)(total - first < pass ? total - first : pass);
    const N2fAngles an{thetas, phis, ntheta, (int)first, n};
    double2* const fx = static_cast<double2*>(scratch);
    double2* const fy = fx + (size_t)n * nx;
    double2* const rows = fy + (size_t)n * ny;
    k_n2f_factors<<<dim3((nx + ny + kN2fThreads - 1) / kN2fThreads, n), kN2fThreads, 0, st>>>(an, nx, ny, dx, z_val, k,
                                                                                              fx, fy);
    const int parts = row_parts(nx, ny, total), cells = ((nx + parts - 1) / parts + kN2fK - 1) / kN2fK * kN2fK;
    const dim3 grd((n + kN2fTile - 1) / kN2fTile, (4 * ny + kN2fTile - 1) / kN2fTile, parts);
    double2* const o = reinterpret_cast<double2*>(out);
    const bool split = parts > 1;
    if (single) {
      const float2* const p = static_cast<const float2*>(planes);
      (split ? k_n2f_rows<float2, true> : k_n2f_rows<float2, false>)<<<grd, kN2fThreads, 0, st>>>(p, fx, n, nx, ny,
                                                                                               cells, rows);
    } else {
      const double2* const p = static_cast<const double2*>(planes);
      (split ? k_n2f_rows<double2, true> : k_n2f_rows<double2, false>)<<<grd, kN2fThreads, 0, st>>>(p, fx, n, nx, ny,
                                                                                                 cells, rows);
    }
    (split ? k_n2f_finish<true> : k_n2f_finish<false>)<<<n, kN2fThreads, 0, st>>>(an, rows, parts, fy, ny, dx, k, r,
                                                                                 total, o);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

}  // namespace fdtd

// ---------------------------------------------------------------------------
// Allocation-free variant of fdtd_near2far.
//
// Some callers cannot allocate device memory at the moment they need a far
// field: code running under a memory manager that owns every byte of the
// device (a caching pool or a reserved arena), callers that must not grow
// the footprint of a running job, or contexts where device allocation is
// forbidden or would synchronize the device. fdtd_near2far_noalloc does the
// same work as fdtd_near2far but stages its inputs, angles and results in
// one statically sized device array, kN2fScratchBytes, which every GPU that
// loads this library holds until the process exits. The caller still passes
// host inputs and a host output buffer; nothing is allocated per call.
// ---------------------------------------------------------------------------
#include <cstdio>
#include <mutex>

#include "fdtd_b200.h"

namespace fdtd {

namespace {

// Largest plane (nx_ph * ny_ph cells, complex128 inputs; twice as many for
// complex64) and angle set the static scratch can hold.
constexpr long long kN2fMaxCells = 600000;       // covers a 761 x 761 grid's 741 x 741 plane
constexpr int kN2fMaxTheta = 4096;
constexpr int kN2fMaxPhi = 64;
constexpr int kN2fMaxAngles = 8192;              // nphi * ntheta
constexpr size_t kN2fPlaneBytes = (size_t)4 * kN2fMaxCells * 16;
constexpr size_t kN2fAngleBytes = (size_t)(kN2fMaxTheta + kN2fMaxPhi) * 8;
constexpr size_t kN2fOutBytes = (size_t)kN2fMaxAngles * 4 * 16;
constexpr size_t kN2fScratchBytes = kN2fPlaneBytes + kN2fAngleBytes + kN2fOutBytes;

// Layout: [4 input planes as given][thetas (deg)][phis (deg)][output]
static __device__ __align__(256) unsigned char g_n2f_scratch[kN2fScratchBytes];

std::mutex g_n2f_mutex;
void* g_n2f_addr[64] = {};   // device address of g_n2f_scratch, per device

// One block per direction with a sine and cosine per cell (fdtd_near2far's
// matrix product needs scratch beyond the static array), reading the u-plane
// phasors as given (complex64 or complex128), forming J = (-Hy, Hx), M = (Ey, -Ex) on the fly
// and converting the angles from degrees on the device.
template <class C>
__global__ void __launch_bounds__(kN2fThreads)
k_near2far_raw(unsigned char* __restrict__ scratch, long long plane_bytes, int nx, int ny,
               double dx, double z_val, double k, int ntheta, int nphi, double r) {
  const C* ex_u = reinterpret_cast<const C*>(scratch);
  const long long n = (long long)nx * ny;
  const C* ey_u = ex_u + n;
  const C* hx_u = ey_u + n;
  const C* hy_u = hx_u + n;
  const double* thetas = reinterpret_cast<const double*>(scratch + plane_bytes);
  const double* phis = thetas + ntheta;
  double2* out = reinterpret_cast<double2*>(scratch + plane_bytes + kN2fAngleBytes);
  const int it = blockIdx.x, ip = blockIdx.y;
  const double th = thetas[it] * (M_PI / 180.0), ph = phis[ip] * (M_PI / 180.0);
  const double st = sin(th), ct = cos(th), sp = sin(ph), cp = cos(ph);
  const int hx = nx / 2, hy = ny / 2;
  double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int idx = threadIdx.x; idx < n; idx += blockDim.x) {
    const int y = idx / nx, x = idx - y * nx;
    const double xl = (double)(x - hx) * dx;
    const double yl = (double)(y - hy) * dx;
    const double arg = k * (((xl * st) * cp + (yl * st) * sp) + z_val * ct);
    double es, ec;
    sincos(arg, &es, &ec);
    const double w = simpson_w(x, nx) * simpson_w(y, ny);
    const double2 Jx = make_double2(-(double)hy_u[idx].x, -(double)hy_u[idx].y);
    const double2 Jy = make_double2((double)hx_u[idx].x, (double)hx_u[idx].y);
    const double2 Mx = make_double2((double)ey_u[idx].x, (double)ey_u[idx].y);
    const double2 My = make_double2(-(double)ex_u[idx].x, -(double)ex_u[idx].y);
    const double ntr = Jx.x * ct * cp + Jy.x * ct * sp, nti = Jx.y * ct * cp + Jy.y * ct * sp;
    const double npr = -Jx.x * sp + Jy.x * cp, npi = -Jx.y * sp + Jy.y * cp;
    const double ltr = Mx.x * ct * cp + My.x * ct * sp, lti = Mx.y * ct * cp + My.y * ct * sp;
    const double lpr = -Mx.x * sp + My.x * cp, lpi = -Mx.y * sp + My.y * cp;
    acc[0] += w * (ntr * ec - nti * es); acc[1] += w * (ntr * es + nti * ec);
    acc[2] += w * (npr * ec - npi * es); acc[3] += w * (npr * es + npi * ec);
    acc[4] += w * (ltr * ec - lti * es); acc[5] += w * (ltr * es + lti * ec);
    acc[6] += w * (lpr * ec - lpi * es); acc[7] += w * (lpr * es + lpi * ec);
  }
#pragma unroll
  for (int j = 0; j < 8; ++j)
    for (int o = 16; o > 0; o >>= 1) acc[j] += __shfl_down_sync(0xffffffffu, acc[j], o);
  __shared__ double red[kN2fThreads / 32][8];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  if (lane == 0)
    for (int j = 0; j < 8; ++j) red[warp][j] = acc[j];
  __syncthreads();
  if (threadIdx.x == 0) {
    double s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int w = 0; w < kN2fThreads / 32; ++w)
      for (int j = 0; j < 8; ++j) s[j] += red[w][j];
    const double h = dx / 3.0;
    for (int j = 0; j < 8; ++j) s[j] *= h * h;
    const double eta0 = 376.730313668;
    const double c = k / (4.0 * M_PI * r);
    double sr, cr;
    sincos(k * r, &sr, &cr);
    const double2 ffw = make_double2(c * sr, c * cr);
    const double2 Nt = make_double2(s[0], s[1]), Np = make_double2(s[2], s[3]);
    const double2 Lt = make_double2(s[4], s[5]), Lp = make_double2(s[6], s[7]);
    auto cm = [](double2 a, double2 b) {
      return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
    };
    const long long plane = (long long)nphi * ntheta;
    const long long o = (long long)ip * ntheta + it;
    out[0 * plane + o] = cm(ffw, make_double2(-Lp.x - eta0 * Nt.x, -Lp.y - eta0 * Nt.y));
    out[1 * plane + o] = cm(ffw, make_double2(Lt.x - eta0 * Np.x, Lt.y - eta0 * Np.y));
    out[2 * plane + o] = cm(ffw, make_double2(Np.x - Lt.x / eta0, Np.y - Lt.y / eta0));
    out[3 * plane + o] = cm(ffw, make_double2(-Nt.x - Lp.x / eta0, -Nt.y - Lp.y / eta0));
  }
}

int n2f_fail(int code, const char* msg) { return report_error(code, msg); }

}  // namespace

}  // namespace fdtd

extern "C" int fdtd_near2far_noalloc(const void* ex_u, const void* ey_u, const void* hx_u,
                                     const void* hy_u, int in_dtype, int nx_ph, int ny_ph,
                                     int nz_ph, double dx, double r, const double* thetas_deg,
                                     int ntheta, const double* phis_deg, int nphi, double freq,
                                     int device, double* out) {
  using namespace fdtd;
  char msg[256];
  if (!ex_u || !ey_u || !hx_u || !hy_u || !thetas_deg || !phis_deg || !out)
    return n2f_fail(FDTD_ERR_INVALID, "null argument");
  if (in_dtype != FDTD_F32 && in_dtype != FDTD_F64)
    return n2f_fail(FDTD_ERR_INVALID, "in_dtype must be FDTD_F32 or FDTD_F64");
  if (nx_ph < 3 || ny_ph < 3 || nx_ph % 2 == 0 || ny_ph % 2 == 0)
    return n2f_fail(FDTD_ERR_INVALID, "Simpson integration needs odd sample counts >= 3");
  if (ntheta < 1 || nphi < 1 || nz_ph < 1) return n2f_fail(FDTD_ERR_INVALID, "empty angle or plane set");
  if (!(freq > 0) || !(dx > 0) || !(r > 0)) return n2f_fail(FDTD_ERR_INVALID, "freq, dx, r must be positive");
  const long long cells = (long long)nx_ph * ny_ph;
  const size_t csz = in_dtype == FDTD_F32 ? 8 : 16;
  const size_t plane_bytes = (size_t)cells * csz;
  if (4 * plane_bytes > kN2fPlaneBytes) {
    snprintf(msg, sizeof(msg),
             "plane of %lld cells exceeds the static scratch (at most %lld cells in complex128, "
             "%lld in complex64); use fdtd_near2far", cells, kN2fMaxCells, 2 * kN2fMaxCells);
    return n2f_fail(FDTD_ERR_INVALID, msg);
  }
  if (ntheta > kN2fMaxTheta || nphi > kN2fMaxPhi || (long long)ntheta * nphi > kN2fMaxAngles) {
    snprintf(msg, sizeof(msg), "angle set %d x %d exceeds the static scratch (theta <= %d, "
             "phi <= %d, product <= %d)", nphi, ntheta, kN2fMaxTheta, kN2fMaxPhi, kN2fMaxAngles);
    return n2f_fail(FDTD_ERR_INVALID, msg);
  }
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    return n2f_fail(FDTD_ERR_CUDA, "no CUDA device available");
  }
  if (device < 0 || device >= ndev || device >= 64) return n2f_fail(FDTD_ERR_INVALID, "device out of range");
  std::lock_guard<std::mutex> lock(g_n2f_mutex);
  DeviceGuard device_guard;   // the caller's current device is restored on return
  cudaError_t e = cudaSetDevice(device);
  if (e != cudaSuccess) return n2f_fail(FDTD_ERR_CUDA, cudaGetErrorString(e));
  // set-up, once per device, with that device current: the address of the
  // static scratch on this device (the host-side symbol is not that address)
  if (!g_n2f_addr[device]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_n2f_scratch);
    if (e != cudaSuccess || !p) {
      snprintf(msg, sizeof(msg), "cudaGetSymbolAddress of the near2far scratch: %s",
               cudaGetErrorString(e));
      return n2f_fail(FDTD_ERR_CUDA, msg);
    }
    g_n2f_addr[device] = p;
  }
  unsigned char* base = static_cast<unsigned char*>(g_n2f_addr[device]);
  // every byte the kernel reads is written below and every output it
  // returns is written by the kernel, so no clearing is needed
  const void* planes[4] = {ex_u, ey_u, hx_u, hy_u};
  for (int c = 0; c < 4; ++c) {
    e = cudaMemcpy(base + c * plane_bytes, planes[c], plane_bytes, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return n2f_fail(FDTD_ERR_CUDA, cudaGetErrorString(e));
  }
  unsigned char* ang = base + 4 * plane_bytes;
  if ((e = cudaMemcpy(ang, thetas_deg, (size_t)ntheta * 8, cudaMemcpyHostToDevice)) != cudaSuccess ||
      (e = cudaMemcpy(ang + (size_t)ntheta * 8, phis_deg, (size_t)nphi * 8, cudaMemcpyHostToDevice)) !=
          cudaSuccess)
    return n2f_fail(FDTD_ERR_CUDA, cudaGetErrorString(e));
  const double lam = 299792458.0 / freq;
  const double k = 2.0 * M_PI / lam;
  const double z_val = (double)((nz_ph - 1) / 2) * dx;
  const dim3 grd(ntheta, nphi, 1);
  // the kernel finds the angles at 4 * plane_bytes and the output
  // kN2fAngleBytes after them
  if (in_dtype == FDTD_F32)
    k_near2far_raw<float2><<<grd, kN2fThreads>>>(base, (long long)(4 * plane_bytes), nx_ph, ny_ph,
                                                 dx, z_val, k, ntheta, nphi, r);
  else
    k_near2far_raw<double2><<<grd, kN2fThreads>>>(base, (long long)(4 * plane_bytes), nx_ph, ny_ph,
                                                  dx, z_val, k, ntheta, nphi, r);
  if ((e = cudaGetLastError()) != cudaSuccess) return n2f_fail(FDTD_ERR_CUDA, cudaGetErrorString(e));
  e = cudaMemcpy(out, ang + kN2fAngleBytes, (size_t)4 * ntheta * nphi * 16, cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return n2f_fail(FDTD_ERR_CUDA, cudaGetErrorString(e));
  return FDTD_OK;
}
