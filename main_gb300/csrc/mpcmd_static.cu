// mpcmd_collide_static: the SRD collision of a caller-owned particle set with
// no device allocation at all.
//
// Who needs it: callers that cannot call cudaMalloc.  A Fortran or C host that
// embeds this library inside a larger code whose memory manager owns every
// byte of device memory (a pool sized at start-up, or a framework allocator)
// may not allocate behind that manager's back; and a caller in a tight
// stepping loop cannot afford cudaMalloc/cudaFree, which synchronise the
// device.  The context API (mpcmd_create) allocates its whole state up front,
// so those callers use this entry point instead: they pass device arrays they
// already own, and the only scratch memory is the file-scope array below.
//
// Scratch: g_collide_scratch, a static __device__ array of
// MPCMD_STATIC_MAX_CELLS x 12 doubles (48 MiB).  Every GPU that loads this
// library holds it until the process exits.  Every call on a device shares it
// and it keeps the last call's contents, so each call clears the part it uses
// before accumulating; calls that overlap on the GPU (different streams or
// host threads, same device) race on it and must be serialised by the caller.
//
// Set-up: the first call on each device (with that device current) resolves
// the array's device address with cudaGetSymbolAddress, which also loads this
// module on the device.  Make that first call before any stream capture.  A
// call on a stream that is not capturing resolves the address again (a host
// lookup, no allocation), so after cudaDeviceReset the next uncaptured call
// picks up the reloaded module's array; a captured call uses the address of
// the last uncaptured one.
//
// The arithmetic is the FP64 collision stage of the engine (k_accumulate_main,
// k_cells and k_rotate_main in mpcmd_kernels.cuh; mpc_rotation_mod.f95:102-228
// and RMPC_SelkovDimer.f90:15-120 in the reference) in four kernels: clear,
// accumulate, cells (the map of every cell, in place of its sums) and
// rotate.  GB300 issues FP64 at 1/64 of the FP32 rate (two lanes per SM and
// cycle), so the FP64 instructions per particle set the time, not the 72
// bytes a particle it moves: the axis (Philox, a sine and a cosine, a square
// root) is drawn once per cell instead of once per particle, the shifted cell
// comes from 32.32 fixed-point integers, and the rotation about the centre of
// mass is v_cm + M (v - v_cm), twelve FP64 instructions a particle (as the affine
// map M v + (v_cm - M v_cm) nine, but then a particle alone in its cell, or at rest
// in it, would not keep its velocity bit for bit).  5.1 million
// unsorted particles in 80^3 cells: 342 us against 1615 with the axis drawn
// and the rotation evaluated per particle (450 with 22 FP64 instructions a
// particle from the centre of mass and the axis); the atomics take 126 us,
// the cells 75 (102 with three divisions and unfused products), the rotation 126.
#include <algorithm>
#include <cmath>
#include <mutex>

#include "mpcmd.h"
#include "mpcmd_kernels.cuh"   // rotate_v and the device helpers

using namespace mpcmd;

namespace {

constexpr int64_t kMaxCells = MPCMD_STATIC_MAX_CELLS;
constexpr int kMaxDevices = 64;
constexpr int kThreads = 256;
// Largest set whose particles each form their cell's map: a map takes some 200
// FP64 instructions, 2 us for 8,192 particles on 152 SMs, about what the cells
// kernel's launch costs (calls back to back: 8,192 particles 14.5 us against 15.3
// with the cells kernel, 20,000 17.4 against 15.2).
constexpr int64_t kOwnMap = 8192;

// per shifted cell, 12 doubles (three whole sectors): first the count (an
// unsigned int) and the sums of vx, vy, vz, then the map v -> m + M (v - m) as
// rows M[q][0..2], m[q]
constexpr int kRec = 12;
static __device__ __align__(256) double g_collide_scratch[kRec * kMaxCells];

std::mutex g_setup_mu;
double* g_scratch_ptr[kMaxDevices] = {};

// Cell and in-cell offset of one absolute coordinate, as the engine's upload
// conversion computes them (k_upload_pos).
__device__ __forceinline__ void to_cell(double x, int L, bool wrap, int& c, double& o) {
  double f = floor(x);
  c = (int)f;
  o = x - f;
  if (o >= 1.0) { o -= 1.0; c += 1; }
  if (wrap) {
    c = wrap_cell(c, L);
  } else {
    if (c >= L) { c = L - 1; o = 1.0; }
    if (c < 0) { c = 0; o = 0.0; }
  }
}

__device__ __forceinline__ uint32_t static_key(const KParams<double>& kp, double x, double y, double z,
                                               double sx, double sy, double sz) {
  int cx, cy, cz;
  double ox, oy, oz;
  to_cell(x, kp.lx, true, cx, ox);
  to_cell(y, kp.ly, true, cy, oy);
  to_cell(z, kp.lz, kp.geometry == MPCMD_GEOM_PERIODIC, cz, oz);
  return shifted_key(kp, pack_cell(cx, cy, cz), ox, oy, oz, sx, sy, sz);
}

__global__ void k_static_clear(double* acc, int64_t ncell) {
  let_next_start();
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < ncell; c += stride) {
    double2* a = reinterpret_cast<double2*>(acc + kRec * (size_t)c);
    a[0] = a[1] = make_double2(0.0, 0.0);
  }
}

// The grid shift in FP64 and as floor(s * 2^32).
struct Shift {
  double s[3];
  int64_t f[3];
};

// One axis of the shifted cell in 32.32 fixed point: false when the FP64
// arithmetic has to decide (a coordinate outside [0, L), or a shifted
// coordinate so close below a face that an FP64 sum could round onto it; the
// truncations of x and s leave the sum less than two units low).
__device__ __forceinline__ bool fixed_cell(double x, int L, int64_t s, int& c) {
  const long long b = __double_as_longlong(x);
  const int e = (int)(b >> 52) - 1023;   // negative for the sign bit too
  if (b < 0 || e > 9) return false;      // negative, 1024 or more, not a number
  const int sh = 20 - e;                 // mantissa 2^52 at weight 2^e -> 2^32 at weight 1
  const uint64_t m = ((uint64_t)b & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
  const uint64_t fx = m >> (sh < 63 ? sh : 63);
  if ((int)(fx >> 32) >= L) return false;
  const int64_t q = (int64_t)fx + s;
  c = (int)(q >> 32);
  return (uint32_t)q <= 0xFFFFFFFCu;
}

// static_key through the integer pipes, with the FP64 form where
// fixed_cell cannot decide.
__device__ __forceinline__ uint32_t fast_key(const KParams<double>& kp, double x, double y, double z, const Shift& s) {
  int fx, fy, fz;
  if (fixed_cell(x, kp.lx, s.f[0], fx) && fixed_cell(y, kp.ly, s.f[1], fy) && fixed_cell(z, kp.lz, s.f[2], fz)) {
    fx += fx < 0 ? kp.lx : (fx >= kp.lx ? -kp.lx : 0);
    fy += fy < 0 ? kp.ly : (fy >= kp.ly ? -kp.ly : 0);
    if (kp.geometry == MPCMD_GEOM_PERIODIC) fz += fz < 0 ? kp.lz : (fz >= kp.lz ? -kp.lz : 0);
    else if (s.s[2] < 0.0) fz += 1;   // floor(z + s + 1)
    return (uint32_t)fx + (uint32_t)kp.lx * ((uint32_t)fy + (uint32_t)kp.ly * (uint32_t)fz);
  }
  return static_key(kp, x, y, z, s.s[0], s.s[1], s.s[2]);
}

__global__ void __launch_bounds__(kThreads) k_static_accumulate(KParams<double> kp, const double* x, const double* y,
                                                                const double* z, const double* vx, const double* vy,
                                                                const double* vz, int64_t n, Shift s, double* acc) {
  after_previous();
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += stride) {
    uint32_t key = fast_key(kp, x[i], y[i], z[i], s);
    if ((int64_t)key >= kp.ncell_shift) continue;   // defensive: keys are in range by construction
    double* a = acc + kRec * (size_t)key;
    atomicAdd(reinterpret_cast<unsigned int*>(a), 1u);
    atomicAdd(a + 1, vx[i]);
    atomicAdd(a + 2, vy[i]);
    atomicAdd(a + 3, vz[i]);
  }
}

// The collision of a cell as a map v -> m + M (v - m): m the centre of mass'
// velocity, M the rotation by the angle about the random axis (k_cells; both forms
// of rotate_v, the projection form turns the other way).  a0, a1: the cell's count
// and velocity sums.  False for an empty cell (no particle reads it).
struct Map {
  double M[3][3], m[3];
};
// One component of the map for d = v - m: m itself where d is zero.
__device__ __forceinline__ double turned(double M0, double M1, double M2, double m, const double (&d)[3]) {
  return fma(M0, d[0], fma(M1, d[1], fma(M2, d[2], m)));
}
// sum / n for a count n with rn = 1 / n rounded to nearest, rounded as the
// division (div_const); an infinite or undefined sum stays what it is.
__device__ __forceinline__ double mean_of(double sum, double n, double rn) {
  const double q = div_const(sum, n, rn);
  return (__double2hiint(q) & 0x7FF00000) != 0x7FF00000 ? q : sum * rn;
}
__device__ __forceinline__ bool cell_map(const KParams<double>& kp, uint32_t cell, uint32_t step, double2 a0, double2 a1,
                                         Map& w) {
  const double pi = 3.141592653589793;
  const double c = kp.cosrot, c1 = 1.0 - c, sn = kp.rotation_sense > 0 ? kp.sinrot : -kp.sinrot;
  const unsigned int cnt = (unsigned int)__double2loint(a0.x);
  if (cnt == 0u) return false;
  const double n = (double)cnt;
  const double rn = 1.0 / n;
  w.m[0] = mean_of(a0.y, n, rn); w.m[1] = mean_of(a1.x, n, rn); w.m[2] = mean_of(a1.y, n, rn);
  double u1, u2, sp, cp;
  contract_pair(kp.seed, TAG_AXIS, cell, 0, step, u1, u2);
  sincos(2.0 * pi * u1, &sp, &cp);
  const double theta = fma(2.0, u2, -1.0), r = sqrt(1.0 - theta * theta);
  const double u[3] = {r * cp, r * sp, theta};
  const double su[3] = {sn * u[0], sn * u[1], sn * u[2]};
  const double k0 = c1 * u[0], k1 = c1 * u[1], k2 = c1 * u[2];
  w.M[0][0] = fma(k0, u[0], c); w.M[0][1] = fma(k0, u[1], -su[2]); w.M[0][2] = fma(k0, u[2], su[1]);
  w.M[1][0] = fma(k0, u[1], su[2]); w.M[1][1] = fma(k1, u[1], c); w.M[1][2] = fma(k1, u[2], -su[0]);
  w.M[2][0] = fma(k0, u[2], -su[1]); w.M[2][1] = fma(k1, u[2], su[0]); w.M[2][2] = fma(k2, u[2], c);
  return true;
}

__global__ void __launch_bounds__(kThreads) k_static_cells(KParams<double> kp, uint32_t step, double* acc) {
  after_previous();
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < kp.ncell_shift; i += stride) {
    double2* a = reinterpret_cast<double2*>(acc + kRec * (size_t)i);
    Map w;
    if (!cell_map(kp, (uint32_t)i, step, a[0], a[1], w)) continue;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      a[2 * q] = make_double2(w.M[q][0], w.M[q][1]);
      a[2 * q + 1] = make_double2(w.M[q][2], w.m[q]);
    }
  }
}

// OWN_MAP: every particle forms its cell's map from the sums itself (the sets
// of at most kOwnMap particles, which no cells kernel precedes).
template <bool OWN_MAP>
__global__ void __launch_bounds__(kThreads) k_static_rotate(KParams<double> kp, const double* x, const double* y,
                                                            const double* z, double* vx, double* vy, double* vz,
                                                            int64_t n, Shift s, uint32_t step, const double* acc) {
  wait_for_previous();   // (what follows is the caller's)
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += stride) {
    uint32_t key = fast_key(kp, x[i], y[i], z[i], s);
    if ((int64_t)key >= kp.ncell_shift) continue;
    const double2* a = reinterpret_cast<const double2*>(acc + kRec * (size_t)key);
    const double v0 = vx[i], v1 = vy[i], v2 = vz[i];
    double w[3];
    if constexpr (OWN_MAP) {
      Map c;
      if (!cell_map(kp, key, step, a[0], a[1], c)) continue;
      const double d[3] = {v0 - c.m[0], v1 - c.m[1], v2 - c.m[2]};
#pragma unroll
      for (int q = 0; q < 3; ++q) w[q] = turned(c.M[q][0], c.M[q][1], c.M[q][2], c.m[q], d);
    } else {
      double2 r[6];
#pragma unroll
      for (int q = 0; q < 6; ++q) r[q] = a[q];
      const double d[3] = {v0 - r[1].y, v1 - r[3].y, v2 - r[5].y};
#pragma unroll
      for (int q = 0; q < 3; ++q) w[q] = turned(r[2 * q].x, r[2 * q].y, r[2 * q + 1].x, r[2 * q + 1].y, d);
    }
    vx[i] = w[0]; vy[i] = w[1]; vz[i] = w[2];
  }
}

}  // namespace

extern "C" int mpcmd_collide_static(const double* x, const double* y, const double* z, double* vx,
                                    double* vy, double* vz, int64_t n, int32_t lx, int32_t ly,
                                    int32_t lz, int32_t geometry, double rot_angle,
                                    int32_t rotation_sense, uint64_t seed, int64_t step,
                                    void* stream) {
  // An error the calling thread left pending is its own: report it without
  // launching and leave it in place for the caller's cudaGetLastError.
  if (cudaPeekAtLastError() != cudaSuccess) return MPCMD_ERR_CUDA;
  if (n < 0 || lx <= 0 || ly <= 0 || lz <= 0 || lx > 1024 || ly > 1024 || lz > 1024) return MPCMD_ERR_CONFIG;
  if (geometry != MPCMD_GEOM_WALLS && geometry != MPCMD_GEOM_PERIODIC) return MPCMD_ERR_CONFIG;
  if (rotation_sense != 1 && rotation_sense != -1) return MPCMD_ERR_CONFIG;
  const int64_t ncs = (int64_t)lx * ly * (geometry == MPCMD_GEOM_WALLS ? (int64_t)lz + 1 : (int64_t)lz);
  if (ncs > kMaxCells) return MPCMD_ERR_CONFIG;   // beyond the static scratch array
  if (n > 0 && (!x || !y || !z || !vx || !vy || !vz)) return MPCMD_ERR_CONFIG;

  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return MPCMD_ERR_CUDA;
  if (dev < 0 || dev >= kMaxDevices) return MPCMD_ERR_CONFIG;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &cap) != cudaSuccess) return MPCMD_ERR_CUDA;
  double* acc = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_setup_mu);
    if (!g_scratch_ptr[dev] || cap == cudaStreamCaptureStatusNone) {
      void* p = nullptr;
      if (cudaGetSymbolAddress(&p, g_collide_scratch) != cudaSuccess || !p) return MPCMD_ERR_CUDA;
      g_scratch_ptr[dev] = static_cast<double*>(p);
    }
    acc = g_scratch_ptr[dev];
  }
  if (n == 0) return MPCMD_OK;

  KParams<double> kp{};
  kp.lx = lx; kp.ly = ly; kp.lz = lz;
  kp.geometry = geometry;
  kp.rotation_sense = rotation_sense;
  kp.ncell_shift = ncs;
  kp.seed = seed;
  kp.cosrot = std::cos(rot_angle);
  kp.sinrot = std::sin(rot_angle);
  // grid shift: the contract stream (SHIFT, 0, extra, step) as the engine draws it
  double u0, u1, u2, u3;
  contract_pair(seed, TAG_SHIFT, 0, 0, (uint32_t)step, u0, u1);
  contract_pair(seed, TAG_SHIFT, 0, 1, (uint32_t)step, u2, u3);
  Shift s{{u0 - 0.5, u1 - 0.5, u2 - 0.5}, {}};
  for (int q = 0; q < 3; ++q) s.f[q] = (int64_t)std::floor(s.s[q] * 4294967296.0);

  int nsm = 0;
  if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return MPCMD_ERR_CUDA;
  const int64_t want = (n + kThreads - 1) / kThreads;
  const int grid = (int)std::min<int64_t>(want, (int64_t)nsm * 8);
  const int tgrid = (int)std::min<int64_t>((ncs + kThreads - 1) / kThreads, (int64_t)nsm * 8);
  k_static_clear<<<tgrid, kThreads, 0, st>>>(acc, ncs);
  // Up to three blocks an SM each kernel starts while the one before it ends (calls
  // back to back: 1,536 to 8,192 particles 14.5 us instead of 18.6, 80,000 20.5
  // instead of 24.7, the 116,736 at the edge 19.3 instead of 24.8).  Towards eight
  // blocks an SM, a whole wave, the early blocks crowd the first SMs that fall
  // free, where they share the FP64 pipe (200,000 particles, 5 blocks: 26.9 instead
  // of 29.1 us; 270,000, 7 blocks: 34.7 instead of 32.4).
  const bool early = grid <= 3 * nsm;
  auto next = [&](auto kernel, int blocks, auto... args) {
    if (early) launch_next(kernel, blocks, kThreads, st, args...);
    else kernel<<<blocks, kThreads, 0, st>>>(args...);
  };
  next(k_static_accumulate, grid, kp, x, y, z, vx, vy, vz, n, s, acc);
  if (n <= kOwnMap) {
    next(k_static_rotate<true>, grid, kp, x, y, z, vx, vy, vz, n, s, (uint32_t)step, acc);
  } else {
    next(k_static_cells, tgrid, kp, (uint32_t)step, acc);
    next(k_static_rotate<false>, grid, kp, x, y, z, vx, vy, vz, n, s, (uint32_t)step, acc);
  }
  if (cudaPeekAtLastError() != cudaSuccess) return MPCMD_ERR_CUDA;
  return MPCMD_OK;
}
