// cup2d_adv_diff_noalloc: the advDiff operator on caller-owned device
// buffers, for callers that cannot allocate device memory.
//
// The regular entry points allocate their reduction scratch once per
// context with cudaMalloc.  Some hosts cannot do that: applications that
// hand all of the GPU's memory to their own pool or caching allocator (a raw
// cudaMalloc then fails, or carves memory the pool believes it owns), and
// latency-critical loops that must not call cudaMalloc/cudaFree because those
// calls synchronise the device and take far longer than the stencil itself.
// This entry point therefore keeps its scratch -- the partial sums of the
// boundary outflow -- in one fixed file-scope device array that is part of
// the loaded library.
//
// Contract
//  - scratch: g_advdiff_scratch below, CUP2D_NOALLOC_MAX_BLOCKS partial sums
//    plus a few slots, about 128 KB; every GPU that loads the library holds
//    it until the process exits;
//  - grids with more than CUP2D_NOALLOC_MAX_BLOCKS blocks are rejected with
//    CUP2D_ETOOLARGE before anything is launched;
//  - the first call on a device looks up the array's device address with
//    cudaGetSymbolAddress (with that device current) and caches it; make the
//    first call on each device before any stream capture begins;
//  - all calls share the one array: calls whose executions overlap on the GPU
//    (other streams, other host threads) race on it and give wrong results
//    (nothing in it outlives a call: each call writes the sums it reads);
//  - no cudaMalloc, cudaFree or allocating library routine is called.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <mutex>
#include "launch.hpp"

namespace cup2d {
namespace {

constexpr int kMaxDevices = 64;
constexpr int kScratchHead = 32;

static __device__ __align__(256) double g_advdiff_scratch[kScratchHead + CUP2D_NOALLOC_MAX_BLOCKS];

std::mutex g_mutex;
double* g_scratch_ptr[kMaxDevices] = {nullptr};

constexpr int kMaxParts = 148;     // partial sums of k_outflow_noalloc, at most one per SM of a B200
// Grids of up to this many boundary cells take one launch: every CTA on the
// boundary then sums the whole outflow itself.  B200, device time of a call
// with one launch and with two: 2.1 and 3.6 us at 128 cells (32 x 32), 3.7
// and 4.1 at 768 (256 x 128), 6.6 and 4.1 at 1536 (512 x 256); the second
// launch costs the host about 2 us more.
constexpr int kFusedBoundary = 1024;

// A call's sizes, lab velocity, coefficients and inflow fades of the four
// edges (advDiff.cpp:14-34, 51-58), formed on the host: six double divisions
// in every thread had been two fifths of the update's FP64 instructions.
struct Args {
  int nx, ny;
  double uinfx, uinfy, afac, dfac, fadeW, fadeE, fadeS, fadeN;
};

Args make_args(int bpdx, int bpdy, double h, double nu, double dt, double uinfx, double uinfy) {
  const double norUinf = std::max(std::max(std::fabs(uinfx), std::fabs(uinfy)), EPSd);
  const double rW = std::max(uinfx, 0.0) / norUinf, rS = std::max(uinfy, 0.0) / norUinf;
  const double rE = std::min(uinfx, 0.0) / norUinf, rN = std::min(uinfy, 0.0) / norUinf;
  return {BS * bpdx, BS * bpdy, uinfx, uinfy, -0.5 * dt / h, (nu / h) * (dt / h),
          1 - rW * rW / 100, 1 - rE * rE / 100, 1 - rS * rS / 100, 1 - rN * rN / 100};
}

// one component f of a cell of velocity (uc, vc) from its four neighbours
// (advDiff.cpp:60-87, its expression order)
__device__ __forceinline__ double advance_cell(const Args& a, double uc, double vc, double fc,
                                               double w, double e, double s, double n) {
  const double adv = (uc + a.uinfx) * (e - w) + (vc + a.uinfy) * (n - s);
  const double dif = e + n + w + s - 4 * fc;
  return fc + (a.afac * adv + a.dfac * dif);
}

// This thread's part (cells first, first + stride, ...) of the boundary
// outflow sum of advDiff.cpp:93-102: the new u of the west and east columns
// and the new v of the south and north rows, straight from the old field.
__device__ __forceinline__ double outflow_part(const Args& a, const double* __restrict__ u,
                                               const double* __restrict__ v, int first, int stride) {
  const int nx = a.nx, ny = a.ny, n = 2 * (nx + ny);
  double sum = 0;
#pragma unroll 4
  for (int i = first; i < n; i += stride) {
    const bool x = i < 2 * ny;                        // a west or east cell
    const int j = x ? i : i - 2 * ny;
    const bool far = j >= (x ? ny : nx);              // east or north
    const int q = far ? j - (x ? ny : nx) : j;
    const int gx = x ? (far ? nx - 1 : 0) : q, gy = x ? q : (far ? ny - 1 : 0);
    const size_t c = (size_t)gy * nx + gx;
    const double* f = x ? u : v;
    const double uc = u[c], vc = v[c], fc = x ? uc : vc;
    const double w = gx > 0 ? f[c - 1] : fc * a.fadeW, e = gx < nx - 1 ? f[c + 1] : fc * a.fadeE;
    const double s = gy > 0 ? f[c - nx] : fc * a.fadeS, t = gy < ny - 1 ? f[c + nx] : fc * a.fadeN;
    const double val = advance_cell(a, uc, vc, fc, w, e, s, t);
    sum += far ? val : -val;
  }
  return sum;
}

// The outflow sum of a grid with a long boundary, one partial per CTA.
__global__ void __launch_bounds__(256)
k_outflow_noalloc(Args a, const double* __restrict__ u, const double* __restrict__ v, double* scratch)
{
  __shared__ double red[32];
  pdl_begin();
  pdl_launch_dependents();
  double s[1] = {outflow_part(a, u, v, blockIdx.x * 256 + threadIdx.x, gridDim.x * 256)};
  block_sum<1>(s, red);
  if (threadIdx.x == 0) scratch[kScratchHead + blockIdx.x] = s[0];
}

// a pair of consecutive doubles, in one 16-byte access where every plane is
// aligned for it
template <bool VEC> __device__ __forceinline__ double2 load2(const double* p) {
  if (VEC) return *reinterpret_cast<const double2*>(p);
  return make_double2(p[0], p[1]);
}
// STREAM: written as the first lines to leave the L2
template <bool VEC, bool STREAM> __device__ __forceinline__ void store2(double* p, double2 x) {
  if (VEC) {
    if (STREAM) __stcs(reinterpret_cast<double2*>(p), x);
    else *reinterpret_cast<double2*>(p) = x;
  } else {
    p[0] = x.x;
    p[1] = x.y;
  }
}

// The update (advDiff.cpp:14-87) with the mean outflow taken from the
// boundary cells as they are written (advDiff.cpp:105-115).  A warp owns 64
// columns of RY rows, two columns a lane: x neighbours come from the
// adjacent lanes, y neighbours from the lane's own rows, so a cell is read
// about once (the halo rows hit the L1: the CTA's eight warps are stacked).
// FUSED: each CTA on the boundary forms the whole outflow sum itself; else
// it adds the nparts partials of k_outflow_noalloc.
// Bound by HBM on a large grid (32 B a cell): at 4096 x 2048 the two launches
// take 47 us, 5.7 TB/s, and 88 us at 4096 x 4096 (126 and 236 us before, one
// cell a lane with the six divisions of the coefficients in every thread, a
// cleared ticket and a pass over the boundary after it).  Two rows a warp at
// four CTAs an SM: with four rows 50.6 us (three CTAs), with one 53, with
// eight 51; streaming stores took 50 to 47.  A small grid is bound by
// latency: one row a warp, 256 x 128 in 3.7 us (12.2 before).
template <int RY, bool VEC, bool FUSED>
__global__ void __launch_bounds__(256, FUSED ? 2 : 4)
k_advdiff_noalloc(Args a, const double* __restrict__ u, const double* __restrict__ v,
                  double* __restrict__ un, double* __restrict__ vn, const double* scratch, int nparts)
{
  static_assert(32 % RY == 0, "a warp's rows lie within the grid: ny is a multiple of 32");
  __shared__ double red[32];
  __shared__ double sCorr;
  pdl_begin();
  const int nx = a.nx, ny = a.ny;
  const int lane = threadIdx.x, x0 = blockIdx.x * 64 + 2 * lane;
  const int yCta = blockIdx.y * 8 * RY, y0 = yCta + threadIdx.y * RY;
  const bool act = x0 < nx && y0 < ny;                // nx, ny are multiples of 32
  // every load of the thread's rows is in flight before the first use
  double2 fu[RY + 2], fv[RY + 2];
  double eu[RY], ev[RY];                              // lane 0: column x0 - 1; lane 31: column x0 + 2
#pragma unroll
  for (int r = 0; r < RY + 2; r++) {
    const int gy = y0 + r - 1;
    fu[r] = fv[r] = make_double2(0, 0);
    if (act && gy >= 0 && gy < ny) {
      fu[r] = load2<VEC>(u + (size_t)gy * nx + x0);
      fv[r] = load2<VEC>(v + (size_t)gy * nx + x0);
    }
  }
  const int xe = lane == 0 ? x0 - 1 : x0 + 2;
  const bool edge = act && ((lane == 0 && x0 > 0) || (lane == 31 && x0 + 2 < nx));
#pragma unroll
  for (int r = 0; r < RY; r++) {
    eu[r] = ev[r] = 0;
    if (edge) { eu[r] = u[(size_t)(y0 + r) * nx + xe]; ev[r] = v[(size_t)(y0 + r) * nx + xe]; }
  }
  double corr = 0;
  const bool boundary = blockIdx.x == 0 || blockIdx.x == gridDim.x - 1 || blockIdx.y == 0 ||
                        blockIdx.y == gridDim.y - 1;
  if (boundary) {
    double t[1];
    if (FUSED) {
      t[0] = outflow_part(a, u, v, lin_tid(), 256);
      block_sum<1>(t, red);
    } else {
      if (threadIdx.y == 0) warp_sum_rows<1>(scratch + kScratchHead, nparts, 1, t);
    }
    if (lin_tid() == 0) sCorr = t[0] / (2 * ny + 2 * nx);              // advDiff.cpp:105
    __syncthreads();
    corr = sCorr;
  }
#pragma unroll
  for (int r = 0; r < RY; r++) {
    const int gy = y0 + r;
    const double2 uc = fu[r + 1], vc = fv[r + 1];
    double uw = __shfl_up_sync(0xffffffffu, uc.y, 1), vw = __shfl_up_sync(0xffffffffu, vc.y, 1);
    double ue = __shfl_down_sync(0xffffffffu, uc.x, 1), ve = __shfl_down_sync(0xffffffffu, vc.x, 1);
    if (lane == 0) { uw = x0 > 0 ? eu[r] : uc.x * a.fadeW; vw = x0 > 0 ? ev[r] : vc.x * a.fadeW; }
    if (x0 + 2 >= nx) { ue = uc.y * a.fadeE; ve = vc.y * a.fadeE; }
    else if (lane == 31) { ue = eu[r]; ve = ev[r]; }
    double2 us = fu[r], vs = fv[r], ut = fu[r + 2], vt = fv[r + 2];
    if (gy == 0) { us = make_double2(uc.x * a.fadeS, uc.y * a.fadeS); vs = make_double2(vc.x * a.fadeS, vc.y * a.fadeS); }
    if (gy == ny - 1) { ut = make_double2(uc.x * a.fadeN, uc.y * a.fadeN); vt = make_double2(vc.x * a.fadeN, vc.y * a.fadeN); }
    double2 nu, nv;
    nu.x = advance_cell(a, uc.x, vc.x, uc.x, uw, uc.y, us.x, ut.x);
    nu.y = advance_cell(a, uc.y, vc.y, uc.y, uc.x, ue, us.y, ut.y);
    nv.x = advance_cell(a, uc.x, vc.x, vc.x, vw, vc.y, vs.x, vt.x);
    nv.y = advance_cell(a, uc.y, vc.y, vc.y, vc.x, ve, vs.y, vt.y);
    if (boundary) {
      if (x0 == 0) nu.x += corr;
      if (x0 + 2 == nx) nu.y -= corr;
      if (gy == 0) { nv.x += corr; nv.y += corr; }
      if (gy == ny - 1) { nv.x -= corr; nv.y -= corr; }
    }
    if (act) {
      store2<VEC, !FUSED>(un + (size_t)gy * nx + x0, nu);
      store2<VEC, !FUSED>(vn + (size_t)gy * nx + x0, nv);
    }
  }
}

template <int RY, bool FUSED>
cudaError_t launch_update(const Args& a, bool vec, const double* u, const double* v, double* un, double* vn,
                          const double* scratch, int nparts, cudaStream_t s) {
  const dim3 grid((a.nx + 63) / 64, (a.ny + 8 * RY - 1) / (8 * RY)), block(32, 8);
  return vec ? launch_k(k_advdiff_noalloc<RY, true, FUSED>, grid, block, 0, s, a, u, v, un, vn, scratch, nparts)
             : launch_k(k_advdiff_noalloc<RY, false, FUSED>, grid, block, 0, s, a, u, v, un, vn, scratch, nparts);
}

// Device address of the scratch array on the current device, looked up once.
int scratch_address(double** out) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return CUP2D_ECUDA;
  if (dev < 0 || dev >= kMaxDevices) return CUP2D_EINVAL;
  std::lock_guard<std::mutex> lock(g_mutex);
  if (!g_scratch_ptr[dev]) {
    double* p = nullptr;
    if (cudaGetSymbolAddress((void**)&p, g_advdiff_scratch) != cudaSuccess || !p) return CUP2D_ECUDA;
    g_scratch_ptr[dev] = p;
  }
  *out = g_scratch_ptr[dev];
  return CUP2D_OK;
}

} // namespace
} // namespace cup2d

extern "C" int cup2d_adv_diff_noalloc(const double* u, const double* v, double* u_out, double* v_out,
                                      int bpdx, int bpdy, double h, double nu, double dt,
                                      double uinfx, double uinfy, void* stream)
{
  using namespace cup2d;
  if (!u || !v || !u_out || !v_out || bpdx <= 0 || bpdy <= 0 || !(h > 0) || !(dt >= 0))
    return CUP2D_EINVAL;
  if ((long long)bpdx * bpdy > CUP2D_NOALLOC_MAX_BLOCKS) return CUP2D_ETOOLARGE;
  if (u_out == u || v_out == v || u_out == v || v_out == u) return CUP2D_EINVAL;
  double* scratch = nullptr;
  int rc = scratch_address(&scratch);
  if (rc != CUP2D_OK) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const Args a = make_args(bpdx, bpdy, h, nu, dt, uinfx, uinfy);
  const bool vec = ((reinterpret_cast<uintptr_t>(u) | reinterpret_cast<uintptr_t>(v) |
                     reinterpret_cast<uintptr_t>(u_out) | reinterpret_cast<uintptr_t>(v_out)) & 15) == 0;
  const int nbnd = 2 * (a.nx + a.ny);
  cudaError_t e;
  if (nbnd <= kFusedBoundary) {
    e = launch_update<1, true>(a, vec, u, v, u_out, v_out, scratch, 0, s);
  } else {
    const int nparts = std::min((nbnd + 255) / 256, kMaxParts);
    e = launch_k(k_outflow_noalloc, nparts, 256, 0, s, a, u, v, scratch);
    if (e == cudaSuccess) e = launch_update<2, false>(a, vec, u, v, u_out, v_out, scratch, nparts, s);
  }
  return e == cudaSuccess && cudaGetLastError() == cudaSuccess ? CUP2D_OK : CUP2D_ECUDA;
}
