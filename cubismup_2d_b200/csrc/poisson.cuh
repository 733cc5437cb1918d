// Helpers of the Poisson transforms, FP64 (poisson.cu) and FP32
// (poisson32.cu): complex arithmetic, padded shared-memory indices,
// asynchronous copies, the right-hand side's edge fade.
#pragma once
#include "context.hpp"

namespace cup2d {

struct FadeArgs {
  int enabled;
  Scalars* sc;           // receives fadeCorr (from the first CTA)
  GridDesc g;
  double* writeback;     // rhs buffer receives the faded values (cub2rhs writes tmp)
  const double* partials;   // fade sums of the strip blocks, three each
  int nstrip;
  int bandX, bandY;         // cells of the fade band from each edge, (int)(fadeLen / h) + 2 (host-formed)
  int ready;                // sc->fadeCorr was formed by k_fade_corr
};

namespace {

// complex values: double2 (the FP64 solve) or float2 (the FP32 solve of
// CUP2D_PREC_FP32)
template <class C> struct CT;
template <> struct CT<double2> { using R = double; };
template <> struct CT<float2> { using R = float; };
template <class C> __device__ __forceinline__ C mk(typename CT<C>::R a, typename CT<C>::R b);
template <> __device__ __forceinline__ double2 mk<double2>(double a, double b) { return make_double2(a, b); }
template <> __device__ __forceinline__ float2 mk<float2>(float a, float b) { return make_float2(a, b); }
template <class C> __device__ __forceinline__ C cmul(C a, C b) {
  return mk<C>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
template <class C> __device__ __forceinline__ C cadd(C a, C b) { return mk<C>(a.x + b.x, a.y + b.y); }
template <class C> __device__ __forceinline__ C csub(C a, C b) { return mk<C>(a.x - b.x, a.y - b.y); }
template <class C> __device__ __forceinline__ C conjg(C a) { return mk<C>(a.x, -a.y); }

__device__ __forceinline__ int pad(int i) { return i + (i >> 4); }

// asynchronous global -> shared copies (sm_80+ cp.async), so that every
// load of a CTA's rows or columns is in flight at once
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n"
               :: "r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n"
               :: "r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" :: "n"(N) : "memory");
}

// multiply by -i (forward) or +i (inverse)
template <bool INV, class C> __device__ __forceinline__ C mul_mi(C a) {
  return INV ? mk<C>(-a.y, a.x) : mk<C>(a.y, -a.x);
}

// pad(j + u T + m Q) given pj = pad(j): a multiple C of 16 added to an index
// adds C + C/16 to its padded position, an immediate offset
template <int T, int Q>
__device__ __forceinline__ int pad_at(int pj, int j, int u, int m) {
  if constexpr (T % 16 == 0 && Q % 16 == 0) return pj + u * (T + T / 16) + m * (Q + Q / 16);
  else return pad(j + u * T + m * Q);
}
// pad(o + q NS) given po = pad(o), for an output o of a pass over sub-transforms
// of size NS: with NS = 1, o is a multiple of R (a divisor of 16) and q < R
// stays inside o's group of 16
template <int NS>
__device__ __forceinline__ int pad_out(int po, int o, int q) {
  if constexpr (NS % 16 == 0) return po + q * (NS + NS / 16);
  else if constexpr (NS == 1) return po + q;
  else return pad(o + q * NS);
}

// fadeCorr for this CTA, formed by warp 0 (blockDim.x >= 32) into *s;
// visible to the CTA after its next barrier
__device__ __forceinline__ void fade_corr_cta(const FadeArgs& fa, double* s) {
  if (fa.ready) {
    if (threadIdx.x == 0) *s = fa.sc->fadeCorr;
  } else if (threadIdx.x < 32) {
    const double corr = fade_corr(fa.partials, fa.nstrip);
    if (threadIdx.x == 0) {
      *s = corr;
      if (blockIdx.x == 0) fa.sc->fadeCorr = corr;
    }
  }
}

// PoissonSolver::cub2rhs (PoissonSolver.cpp:101-125): the fade argument's
// part of a row and of a column, and the faded value of a cell
__device__ __forceinline__ double fade_row(const GridDesc& g, int gy) {
  const double py = gy_pos(g, gy);
  return fmax(g.invFadeY * fmax(0.0, g.fadeLenY - g.ext[1] + py), g.invFadeY * fmax(0.0, g.fadeLenY - py));
}
__device__ __forceinline__ double fade_col(const GridDesc& g, int gx) {
  const double px = gx_pos(g, gx);
  return fmax(g.invFadeX * fmax(0.0, g.fadeLenX - g.ext[0] + px), g.invFadeX * fmax(0.0, g.fadeLenX - px));
}
__device__ __forceinline__ double fade_cell(double row, double col, double b, double corr) {
  const double fadeArg = fmin(fmax(row, col), 1.0);
  const double f2 = fadeArg * fadeArg;
  const double fadeRHS = b * f2;
  const double fadeCorrection = corr * (corr > 0 ? fmax(fadeRHS, 0.0) : -fmin(fadeRHS, 0.0));
  return __dadd_rn(__dmul_rn(b, 1 - f2), fadeCorrection);   // never contracted into an FMA
}

#define CUP2D_FFT_LENGTHS(X) X(16) X(32) X(64) X(128) X(256) X(512) X(1024) X(2048) X(4096)

} // namespace

// poisson32.cu: the FP32 passes of the free-space and periodic solves
bool poisson32_setup();                              // shared-memory limits of its kernels
// device tables of the row (column) passes of length L, from tw rounded to FP32
float2* make_tables32(int L, bool cols, const std::vector<float2>& tw, cudaStream_t st);
bool rows_r2c32(int L, cudaStream_t st, const double* in, int inStride, int nrows, int ncolsIn, float2* out,
                int outRows, const float2* tab, const float2* tw, int twLen, FadeArgs fa, bool halfIn);
bool cols32(int L, cudaStream_t st, float2* data, int rows, int ncols, int nrowsIn, int nrowsOut,
            const float* ghat, int mode, const float2* tab, double norm, int MXp, int MYp);
bool rows_c2r32(int L, cudaStream_t st, const float2* in, int inRows, int nrows, double* out, int outStride,
                int ncolsOut, const float2* tab, const float2* tw, int twLen, bool halfOut);

} // namespace cup2d
