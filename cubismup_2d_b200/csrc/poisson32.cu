// FP32 Poisson transforms (CUP2D_PREC_FP32): the free-space and periodic
// passes of poisson.cu on float2 spectra, the fade and its write-back in FP64
// (so the RHS written back is the one of the FP64 path), rows converted to
// FP32 as they enter shared memory, the pressure written back in FP64.
// The transforms keep their own radix passes: their twiddles are products of
// table values in one fixed order, so FP32 results do not move with the FP64
// passes.
#include <algorithm>
#include <vector>
#include "poisson.cuh"

namespace cup2d {
namespace {

// The half spectrum lies in groups of eight columns, 64 bytes a row, as the
// FP64 one does in groups of four (spec_at in poisson.cu): a column pass then
// touches 16 lines for 32 rows instead of 32, and the kernel G^ lies by columns,
// read where it is applied.  B200, forward rows, columns, inverse rows in us,
// after (before) this, the tables laid out once, the first and last row passes
// straight from and to global memory and Col32: 4096 x 2048 68, 112, 57 (81, 180,
// 65); 2048 x 1024 25, 33, 19 (28, 70, 22); 1024 x 512 13.4, 14.0, 11.2 (14.4, 17.2,
// 12.0).  The same arithmetic in the same order: the same bits.
constexpr int SPEC32_LOG = 3;
__device__ __forceinline__ size_t spec32_at(int rows, int r, int k) {
  return (((size_t)(k >> SPEC32_LOG) * rows + r) << SPEC32_LOG) | (k & ((1 << SPEC32_LOG) - 1));
}

// Per transform length L: padded stride SL of one sequence (one spare
// element per 16, plus 4 so that consecutive sequences start in different
// halves of the shared-memory banks), the room TW of the staged tables, the
// rows per CTA B and the threads per CTA NT of the row passes
// (L/E per sequence: every thread owns E = 16 or 8 elements of a pass).
// ---- per-pass twiddle tables ---------------------------------------------
// The passes of fft_inplace<L, ..., E> (fft_passes): sub-transform sizes
// NS = 1, E, E^2, ... with radix E while NS E <= L, then one pass of radix
// L/NS.  The pass over sub-transforms of size NS scales input m of the
// butterfly with k = j mod NS by W^(m k), W = exp(-2 pi i/(R NS)).  For each
// pass with NS > 1 the tables hold W^(p k), k < NS, for the powers p = 1, 2,
// 4, 8 below R (one table of NS entries each): the butterflies of a warp
// read consecutive entries (no shared-memory bank conflicts, where indexing
// one table by m k made every lane of a warp hit the same banks), and the
// other powers are products of at most three table values.
constexpr int tw_npow(int R) { return R >= 16 ? 4 : (R >= 8 ? 3 : (R >= 4 ? 2 : (R >= 2 ? 1 : 0))); }
// offset of the tables of the pass over sub-transforms of size NS
template <int L, int E> constexpr int tw_off(int NS) {
  int off = 0, ns = 1;
  while (ns < L && ns < NS) {
    const int r = ns * E <= L ? E : L / ns;
    if (ns > 1) off += tw_npow(r) * ns;
    ns *= r;
  }
  return off;
}
template <int L, int E> constexpr int tw_size() { return tw_off<L, E>(L); }
// entries staged per CTA: enough for the element counts E = 8 and 16
template <int L> constexpr int tw_max() {
  const int a = tw_size<L, 8>(), b = tw_size<L, 16>();
  return a > b ? (a > 0 ? a : 1) : (b > 0 ? b : 1);
}

template <int L, int E = 16> struct Len {
  static constexpr int SL = L + L / 16 + 4;
  static constexpr int TW = tw_max<L>();
  static constexpr int B = 2048 / L < 1 ? 1 : (2048 / L > 8 ? 8 : 2048 / L);
  static constexpr int NT0 = B * L / E;
  static constexpr int NT = NT0 < 64 ? 64 : (NT0 > 512 ? 512 : NT0);
  static constexpr int MINB = 65536 / (NT * 64);    // 64 registers a thread
};
// elements per thread
constexpr int E_ROWS32 = 8;
constexpr int E_C2R32 = 8;
constexpr int E_COLS32 = 16;
// Columns per CTA of the column pass (of one group, so that a CTA reads runs
// of 16 or 32 bytes): 4096 x 2048, in us, with 1, 2 and 4 columns 130 (80
// registers), 115, 112; 2048-point columns with 1, 2, 4 columns 40, 32, 35.
// Registers a thread: from 2048 points on 64, so that 32 warps an SM hide the
// exchanges that the pass waits for: 2048 x 2048 periodic 26.6 us (28.8 with 128),
// 4096 x 2048 periodic 41.5 (43.5), free space 112 (112, and 137 with 128 and one
// column).  Shorter passes do not fill the chip with warps either way, and the
// 64 registers spill: 64 points (64 x 32) 8.3 us with 64 registers and 8.05 with
// 128; 128 points 8.55, 8.55; 256 8.4, 8.4 and 12.8, 12.7; 512 10.4, 10.4 and 12.5,
// 12.5; 1024 14.0, 14.0 and 14.2, 14.3.
template <int L> struct Col32 {
  static constexpr int CB = L >= 4096 ? 4 : (L >= 1024 ? 2 : Len<L>::B);
  static constexpr int NT0 = CB * L / E_COLS32, NT = NT0 < 64 ? 64 : NT0;
  static constexpr int REGS = L >= 2048 ? 64 : 128;
  static constexpr int MINB = 65536 / (NT * REGS);
};

// Stages the per-pass tables of fft_inplace<L, ..., E>, laid out once for all
// CTAs (make_tables32).  Gathered by every CTA from the table of all
// exp(-2 pi i j / twLen), a stride apart, the 14 KB of a 4096-point row had
// taken as much L2 traffic as the row.
template <int L, int E, class C>
__device__ __forceinline__ void load_twiddles(C* tws, const C* __restrict__ tab) {
  for (int t = threadIdx.x; t < tw_size<L, E>(); t += blockDim.x) tws[t] = tab[t];
}
// the tables on the host, from tw[j] = exp(-2 pi i j / twLen) (twLen a
// multiple of 2 L): entry p NS + k of a pass of radix R holds W^(k 2^p) =
// tw[(k 2^p) twLen / (R NS)]
template <int L, int E> void fill_tables32(const std::vector<float2>& tw, std::vector<float2>& out) {
  out.assign(std::max(1, tw_size<L, E>()), make_float2(0, 0));
  for (int ns = 1; ns < L;) {
    const int r = ns * E <= L ? E : L / ns;
    if (ns > 1)
      for (int p = 0; p < tw_npow(r); p++)
        for (int k = 0; k < ns; k++)
          out[tw_off<L, E>(ns) + p * ns + k] = tw[(size_t)(k << p) * (tw.size() / (size_t)(r * ns))];
    ns *= r;
  }
}

// Scales xb[m], 0 < m < R, of the butterfly k of the pass over
// sub-transforms of size NS by W^(m k) (conjugated for the inverse).
template <int L, int E, int R, int NS, bool INV, class C>
__device__ __forceinline__ void apply_twiddles(C* xb, const C* tws, int k) {
  const C* t = tws + tw_off<L, E>(NS) + k;
  auto ld = [&](int pi) { C w = t[pi * NS]; if (INV) w.y = -w.y; return w; };
  const C w1 = ld(0);
  xb[1] = cmul(xb[1], w1);
  if constexpr (R > 2) {
    const C w2 = ld(1), w3 = cmul(w1, w2);
    xb[2] = cmul(xb[2], w2);
    xb[3] = cmul(xb[3], w3);
    if constexpr (R > 4) {
      const C w4 = ld(2);
      xb[4] = cmul(xb[4], w4);
      xb[5] = cmul(xb[5], cmul(w1, w4));
      xb[6] = cmul(xb[6], cmul(w2, w4));
      xb[7] = cmul(xb[7], cmul(w3, w4));
      if constexpr (R > 8) {
        const C w8 = ld(3), w12 = cmul(w4, w8);
        xb[8] = cmul(xb[8], w8);
        xb[9] = cmul(xb[9], cmul(w1, w8));
        xb[10] = cmul(xb[10], cmul(w2, w8));
        xb[11] = cmul(xb[11], cmul(w3, w8));
        xb[12] = cmul(xb[12], w12);
        xb[13] = cmul(xb[13], cmul(w1, w12));
        xb[14] = cmul(xb[14], cmul(w2, w12));
        xb[15] = cmul(xb[15], cmul(w3, w12));
      }
    }
  }
}

// ---- small DFTs in registers (forward exp(-2 pi i mq/R), inverse exp(+)) --
template <bool INV, class C>
__device__ __forceinline__ void dft4(C& x0, C& x1, C& x2, C& x3) {
  const C t0 = cadd(x0, x2), t1 = csub(x0, x2), t2 = cadd(x1, x3), t3 = mul_mi<INV>(csub(x1, x3));
  x0 = cadd(t0, t2); x2 = csub(t0, t2);
  x1 = cadd(t1, t3); x3 = csub(t1, t3);
}
constexpr double C8 = 0.92387953251128675613;   // cos(pi/8)
constexpr double S8 = 0.38268343236508977173;   // sin(pi/8)
constexpr double R2 = 0.70710678118654752440;   // sqrt(2)/2
// W16^e for e in [0, 16): the first quadrant from (1, C8, R2, S8), the rest
// by exact quarter turns
template <bool INV, class C>
__device__ __forceinline__ C w16(int e) {
  using R = typename CT<C>::R;
  const int q = e >> 2, r = e & 3;
  const R cr = (R)(r == 0 ? 1.0 : (r == 1 ? C8 : (r == 2 ? R2 : S8)));
  const R sr = (R)(r == 0 ? 0.0 : (r == 1 ? S8 : (r == 2 ? R2 : C8)));
  C v = mk<C>(cr, -sr);
  for (int k = 0; k < q; k++) v = mk<C>(v.y, -v.x);
  if (INV) v.y = -v.y;
  return v;
}
// DFT of R values in x[0..R); the result for output q is in x[out_reg<R>(q)]
template <int R> __device__ __forceinline__ constexpr int out_reg(int q) {
  return R == 16 ? 4 * (q & 3) + (q >> 2) : q;
}
template <bool INV, class C> __device__ __forceinline__ void dft8(C* x) {
  // m = m1 + 2 m2: DFT4 over m2, twiddle W8^(m1 q2), DFT2 over m1
  dft4<INV>(x[0], x[2], x[4], x[6]);
  dft4<INV>(x[1], x[3], x[5], x[7]);
  C y[8];
#pragma unroll
  for (int q2 = 0; q2 < 4; q2++) {
    const C z0 = x[2 * q2], z1 = cmul(x[2 * q2 + 1], w16<INV, C>(2 * q2));
    y[q2] = cadd(z0, z1); y[q2 + 4] = csub(z0, z1);
  }
#pragma unroll
  for (int q = 0; q < 8; q++) x[q] = y[q];
}
template <bool INV, class C> __device__ __forceinline__ void dft16(C* x) {
  // m = m1 + 4 m2: DFT4 over m2 (result z[m1][q2] in x[m1 + 4 q2]),
  // twiddle W16^(m1 q2), DFT4 over m1 (output q2 + 4 q1 in x[4 q2 + q1])
#pragma unroll
  for (int m1 = 0; m1 < 4; m1++) dft4<INV>(x[m1], x[m1 + 4], x[m1 + 8], x[m1 + 12]);
#pragma unroll
  for (int m1 = 1; m1 < 4; m1++)
#pragma unroll
    for (int q2 = 1; q2 < 4; q2++) x[m1 + 4 * q2] = cmul(x[m1 + 4 * q2], w16<INV, C>(m1 * q2));
#pragma unroll
  for (int q2 = 0; q2 < 4; q2++) dft4<INV>(x[4 * q2], x[4 * q2 + 1], x[4 * q2 + 2], x[4 * q2 + 3]);
}
template <int R, bool INV, class C> __device__ __forceinline__ void dft(C* x) {
  if constexpr (R == 2) { const C t = x[0]; x[0] = cadd(t, x[1]); x[1] = csub(t, x[1]); }
  else if constexpr (R == 4) dft4<INV>(x[0], x[1], x[2], x[3]);
  else if constexpr (R == 8) dft8<INV>(x);
  else dft16<INV>(x);
}

// One in-place Stockham pass of radix R over sub-transforms of size NS on
// nseq sequences A + q*SL: butterfly j (k = j mod NS) reads x_m =
// a[j + m L/R], scales by w^(m k L/(R NS)), takes the DFT_R and writes
// output q at (j - k) R + k + q NS.  Thread t of a sequence owns the 16/R
// butterflies t + u L/16.  Loads go to registers before the barrier,
// stores after it, so one buffer suffices.
template <int L, int R, int NS, bool INV, bool HIN, bool HOUT, int E, class C>
__device__ __forceinline__ void fft_pass(C* A, int nseq, const C* tws)
{
  constexpr int SL = Len<L>::SL, T = L / E, NB = E / R, Q = L / R;
  // first pass of an input whose upper half is zero: inputs m >= R/2 sit at
  // indices >= L/2 (then NB == 1); last pass of which only the lower half of
  // the output is kept: outputs q >= R/2 land at indices >= L/2
  constexpr bool ZIN = HIN && NS == 1, HALFO = HOUT && NS * R == L;
  const int tid = threadIdx.x;
  const bool act = tid < nseq * T;
  const int sq = act ? tid / T : 0, j = tid - sq * T;
  C* a = A + sq * SL;
  C x[E];
  if (act) {
    const int pj = pad(j);
#pragma unroll
    for (int u = 0; u < NB; u++)
#pragma unroll
      for (int m = 0; m < R; m++)
        x[u * R + m] = (ZIN && m >= R / 2) ? mk<C>(0, 0)
                                           : a[pad_at<T, Q>(pj, j, u, m)];
  }
  __syncthreads();
  if (act) {
#pragma unroll
    for (int u = 0; u < NB; u++) {
      C* xb = x + u * R;
      const int jb = j + u * T, k = jb & (NS - 1);
      if (NS > 1 && k) apply_twiddles<L, E, R, NS, INV>(xb, tws, k);
      dft<R, INV>(xb);
      const int o = (jb - k) * R + k, po = pad(o);
#pragma unroll
      for (int q = 0; q < (HALFO ? R / 2 : R); q++) a[pad_out<NS>(po, o, q)] = xb[out_reg<R>(q)];
    }
  }
  __syncthreads();
}

template <int L, int NS, bool INV, bool HIN, bool HOUT, int E, class C>
__device__ __forceinline__ void fft_passes(C* A, int nseq, const C* tws) {
  if constexpr (NS * E <= L) {
    fft_pass<L, E, NS, INV, HIN, HOUT, E>(A, nseq, tws);
    fft_passes<L, NS * E, INV, HIN, HOUT, E>(A, nseq, tws);
  } else if constexpr (NS < L) {
    fft_pass<L, L / NS, NS, INV, HIN, HOUT, E>(A, nseq, tws);
  }
}

// In-place Stockham autosort FFT of nseq sequences of length L (A + q*SL,
// padded indexing; a power of two >= 16): radix-16 passes and one radix
// 2/4/8 pass for the remaining factor.  Forward exp(-2 pi i jk/L), inverse
// exp(+...), unnormalised.  Needs blockDim.x >= nseq * L/E.  HIN: the
// upper half of the input is zero and never read; HOUT: only the lower half
// of the output is written.
template <int L, bool INV, bool HIN = false, bool HOUT = false, int E = 16, class C>
__device__ void fft_inplace(C* A, int nseq, const C* tws)
{
  fft_passes<L, 1, INV, HIN, HOUT, E>(A, nseq, tws);
}

// sub-transform size NS of the last pass of fft_inplace<L, ..., E>
template <int L, int E> constexpr int last_ns() {
  int ns = 1;
  while (ns * E <= L) ns *= E;
  return ns == L ? ns / E : ns;
}
// the passes of fft_passes<L, NS, ...> whose sub-transform size is below NSEND
template <int L, int NS, int NSEND, bool INV, bool HIN, int E, class C>
__device__ __forceinline__ void fft_passes_below(C* A, int nseq, const C* tws) {
  if constexpr (NS < NSEND) {
    constexpr int R = NS * E <= L ? E : L / NS;
    fft_pass<L, R, NS, INV, HIN, false, E>(A, nseq, tws);
    fft_passes_below<L, NS * R, NSEND, INV, HIN, E>(A, nseq, tws);
  }
}

// Spectral convolution of nseq sequences in place: fft_inplace<L, false,
// HIN>, X[r] = mul(sequence, r, X[r]), fft_inplace<L, true, false, HOUT>.  The
// last forward pass, the multiplier and the first inverse pass run in
// registers: butterfly jb = j + u L/E of the last forward pass (radix R,
// NS = L/R, no stride: k = jb) produces X[jb + q NS] = X[j + (u + (E/R) q)
// L/E], which is input m = u + (E/R) q of thread j's radix-E first inverse
// butterfly (NS = 1).  With L <= E (one pass each way) the three steps run
// one after the other.
template <int L, bool HIN, bool HOUT, int E, class C, class Mul>
__device__ __forceinline__ void fft_convolve(C* A, int nseq, const C* tws, Mul mul)
{
  constexpr int SL = Len<L>::SL, T = L / E, NS = last_ns<L, E>(), R = L / NS, NB = E / R;
  if constexpr (L <= E) {
    fft_inplace<L, false, HIN, false, E>(A, nseq, tws);
    for (int idx = threadIdx.x; idx < nseq * L; idx += blockDim.x) {
      const int sq = idx / L, r = idx - sq * L;
      A[sq * SL + pad(r)] = mul(sq, r, A[sq * SL + pad(r)]);
    }
    __syncthreads();
    fft_inplace<L, true, false, HOUT, E>(A, nseq, tws);
    return;
  }
  fft_passes_below<L, 1, NS, false, HIN, E>(A, nseq, tws);
  const int tid = threadIdx.x;
  const bool act = tid < nseq * T;
  const int sq = act ? tid / T : 0, j = tid - sq * T;
  C* a = A + sq * SL;
  C x[E];
  if (act) {
    const int pj = pad(j);
#pragma unroll
    for (int u = 0; u < NB; u++)
#pragma unroll
      for (int m = 0; m < R; m++) x[u * R + m] = a[pad_at<T, NS>(pj, j, u, m)];
  }
  __syncthreads();
  if (act) {
    C y[E];
#pragma unroll
    for (int u = 0; u < NB; u++) {
      C* xb = x + u * R;
      const int jb = j + u * T;
      if (jb) apply_twiddles<L, E, R, NS, false>(xb, tws, jb);
      dft<R, false>(xb);
#pragma unroll
      for (int q = 0; q < R; q++) y[u + NB * q] = mul(sq, jb + q * NS, xb[out_reg<R>(q)]);
    }
    dft<E, true>(y);
#pragma unroll
    for (int q = 0; q < E; q++) a[pad_out<1>(pad(j * E), j * E, q)] = y[out_reg<E>(q)];
  }
  __syncthreads();
  fft_passes<L, E, true, false, HOUT, E>(A, nseq, tws);
}

// Real FFT of length 2L from the complex FFT Z of length L of its value
// pairs, even/odd split: X[k] = Fe[k] + W^k Fo[k], W = exp(-i pi / L),
// k in [0, L]; written to row row0 + r of out.  Thread t takes k = t + q NT
// of every row; its twiddles are read first, all in flight at once (read
// inside the loop, every iteration waited for its own).
template <int L, int ER, class C>
__device__ __forceinline__ void r2c_split(const C* A, int nb, int row0, C* __restrict__ out,
                                          int outRows, const C* __restrict__ tw, int twLen)
{
  using R = typename CT<C>::R;
  constexpr int SL = Len<L, ER>::SL, NT = Len<L, ER>::NT, KPT = (L + 1 + NT - 1) / NT;
  constexpr int KB = KPT < 8 ? KPT : 8;                 // twiddles in flight per batch
  const int twStep = twLen / (2 * L);
#pragma unroll
  for (int q0 = 0; q0 < KPT; q0 += KB) {
    C w[KB];
#pragma unroll
    for (int q = 0; q < KB; q++) {
      const int k = threadIdx.x + (q0 + q) * NT;
      w[q] = q0 + q < KPT && k <= L ? tw[k * twStep] : mk<C>(0, 0);
    }
#pragma unroll
    for (int q = 0; q < KB; q++) {
      const int k = threadIdx.x + (q0 + q) * NT;
      if (q0 + q >= KPT || k > L) break;                // k grows with q
      for (int r = 0; r < nb; r++) {
        const C Zk = A[r * SL + pad(k == L ? 0 : k)];
        const C Zc = conjg(A[r * SL + pad(k == 0 ? 0 : L - k)]);
        const C Fe = mk<C>(R(0.5) * (Zk.x + Zc.x), R(0.5) * (Zk.y + Zc.y));
        const C d = csub(Zk, Zc);
        const C Fo = mk<C>(R(0.5) * d.y, R(-0.5) * d.x);  // (Zk - Zc) / (2i)
        out[spec32_at(outRows, row0 + r, k)] = cadd(Fe, cmul(w[q], Fo));
      }
    }
  }
}

template <int L, bool HIN>
__global__ void __launch_bounds__(Len<L, E_ROWS32>::NT, Len<L, E_ROWS32>::MINB)
k_rows_r2c32(const double* __restrict__ in, int inStride, int nrows, int ncolsIn,
             float2* __restrict__ out, int outRows, const float2* __restrict__ tab, const float2* __restrict__ tw,
             int twLen, FadeArgs fa)
{
  pdl_begin();
  CUP2D_TRACE_SCOPE(TR_R2C);
  constexpr int SL = Len<L, E_ROWS32>::SL, RB = Len<L, E_ROWS32>::B;
  constexpr int E = E_ROWS32, Q = L / E, N = HIN ? E / 2 : E;
  extern __shared__ float2 sm32[];
  float2* A = sm32;
  float2* tws = sm32 + RB * SL;
  const int row0 = blockIdx.x * RB;
  const int nb = min(RB, nrows - row0);
  // this thread's inputs of the first pass, all loads in flight
  const int sq = threadIdx.x / Q, j = threadIdx.x % Q, row = row0 + sq;
  const bool act = sq < nb;
  double2 v[N];
#pragma unroll
  for (int m = 0; m < N; m++) {
    const int n = j + m * Q;
    v[m] = make_double2(0, 0);
    if (act) {
      if (2 * n + 1 < ncolsIn) v[m] = *reinterpret_cast<const double2*>(in + (size_t)row * inStride + 2 * n);
      else if (2 * n < ncolsIn) v[m].x = in[(size_t)row * inStride + 2 * n];
    }
  }
  __shared__ double sCorr;
  if (fa.enabled) fade_corr_cta(fa, &sCorr);
  load_twiddles<L, E>(tws, tab);
  __syncthreads();
  if (act) {
    // fade band as in k_rows_r2c (cub2rhs, PoissonSolver.cpp:61-141; no band,
    // and no cell looked at, with the fade off)
    const bool rowBand = fa.enabled && (row < fa.bandY || row >= fa.g.ny - fa.bandY);
    const int bandLo = !fa.enabled ? 0 : rowBand ? fa.g.nx : fa.bandX;
    const int bandHi = fa.enabled ? fa.g.nx - fa.bandX : ncolsIn;
    const double rowFade = fade_row(fa.g, row);
    float2 x[E];
#pragma unroll
    for (int m = 0; m < E; m++) x[m] = make_float2(0, 0);    // HIN: the zero upper half
#pragma unroll
    for (int m = 0; m < N; m++) {
      const int n = j + m * Q;
      if ((2 * n < bandLo || 2 * n + 1 >= bandHi) && 2 * n + 1 < ncolsIn) {
        double* y = &v[m].x;
        for (int q = 0; q < 2; q++) {
          const int col = 2 * n + q;
          if (col < bandLo || col >= bandHi) {
            y[q] = fade_cell(rowFade, fade_col(fa.g, col), y[q], sCorr);
            fa.writeback[(size_t)row * inStride + col] = y[q];
          }
        }
      }
      x[m] = make_float2((float)v[m].x, (float)v[m].y);
    }
    dft<E, false>(x);
    float2* a = A + sq * SL;
    const int o = j * E, po = pad(o);
#pragma unroll
    for (int q = 0; q < E; q++) a[pad_out<1>(po, o, q)] = x[out_reg<E>(q)];
  }
  __syncthreads();
  fft_passes<L, E, false, false, false, E>(A, nb, tws);
  r2c_split<L, E_ROWS32>(A, nb, row0, out, outRows, tw, twLen);
}

// mode 0: forward, x G^, inverse, keep nrowsOut rows; mode 2: the periodic
// multiplier -1/|k|^2 / (MX MY) (formed in FP64, applied in FP32)
template <int L, bool FS>
__global__ void __launch_bounds__(Col32<L>::NT, Col32<L>::MINB)
k_cols32(float2* __restrict__ data, int rows, int ncols, int nrowsIn, int nrowsOut,
         const float* __restrict__ ghat, int mode, const float2* __restrict__ tab, double norm, int MXp, int MYp)
{
  pdl_begin();
  CUP2D_TRACE_SCOPE(TR_COLS);
  constexpr int SL = Len<L>::SL, CB = Col32<L>::CB, NT = Col32<L>::NT, GR = L / 2 + 1;
  extern __shared__ float2 sm32[];
  float2* A = sm32;
  float2* tws = sm32 + CB * SL;
  const int c0 = blockIdx.x * CB;
  const int nb = min(CB, ncols - c0);
  for (int idx = threadIdx.x; idx < CB * nrowsIn; idx += NT) {
    const int r = idx / CB, j = idx & (CB - 1);
    if (j < nb) cp_async8(A + j * SL + pad(r), data + spec32_at(rows, r, c0 + j));
  }
  cp_async_commit();
  // rows beyond the input are zero; the free-space solve never reads its
  // upper half
  for (int idx = threadIdx.x; idx < CB * ((FS ? L / 2 : L) - nrowsIn); idx += NT) {
    const int r = nrowsIn + idx / CB, j = idx & (CB - 1);
    A[j * SL + pad(r)] = make_float2(0, 0);
  }
  load_twiddles<L, E_COLS32>(tws, tab);
  cp_async_wait<0>();
  __syncthreads();
  if (mode == 0) {
    fft_convolve<L, FS, FS, E_COLS32>(A, nb, tws, [&](int j, int r, float2 z) {
      const int ky = r <= L / 2 ? r : L - r;
      const float f = __ldg(ghat + (size_t)(c0 + j) * GR + ky);
      return make_float2(z.x * f, z.y * f);
    });
  } else {
    fft_convolve<L, FS, FS, E_COLS32>(A, nb, tws, [&](int j, int r, float2 z) {
      // FFTW_periodic::_solve_spectral (FFTW_periodic.h:77-92)
      const int i = c0 + j;
      if (i == 0 && r == 0) return make_float2(0, 0);
      const int kx = i <= MXp / 2 ? i : MXp - i, ky = r <= MYp / 2 ? r : MYp - r;
      const double waveFactX = 2 * M_PI / MXp, waveFactY = 2 * M_PI / MYp;
      const double rkx = kx * waveFactX, rky = ky * waveFactY;
      const float f = (float)(-1 / (rkx * rkx + rky * rky) * norm);
      return make_float2(z.x * f, z.y * f);
    });
  }
  for (int idx = threadIdx.x; idx < CB * nrowsOut; idx += NT) {
    const int r = idx / CB, j = idx & (CB - 1);
    if (j < nb) data[spec32_at(rows, r, c0 + j)] = A[j * SL + pad(r)];
  }
}

// inverse real FFT of length 2L from X[0..L] (float2); writes the first
// ncolsOut values in FP64
template <int L, bool HOUT>
__global__ void __launch_bounds__(Len<L, E_C2R32>::NT, Len<L, E_C2R32>::MINB)
k_rows_c2r32(const float2* __restrict__ in, int inRows, int nrows, double* __restrict__ out, int outStride,
             int ncolsOut, const float2* __restrict__ tab, const float2* __restrict__ tw, int twLen)
{
  pdl_begin();
  CUP2D_TRACE_SCOPE(TR_C2R);
  constexpr int SL = Len<L, E_C2R32>::SL, RB = Len<L, E_C2R32>::B, NT = Len<L, E_C2R32>::NT, H = L / 2;
  extern __shared__ float2 sm32[];
  float2* A = sm32;
  float2* tws = sm32 + RB * SL;
  const int row0 = blockIdx.x * RB;
  const int nb = min(RB, nrows - row0);
  const int twStep = twLen / (2 * L);
  for (int idx = threadIdx.x; idx < RB * (L + 1); idx += NT) {
    const int r = idx / (L + 1), k = idx - r * (L + 1);
    if (r < nb) cp_async8(A + r * SL + pad(k), in + spec32_at(inRows, row0 + r, k));
  }
  cp_async_commit();
  load_twiddles<L, E_C2R32>(tws, tab);
  // the split's W^-k of the pairs (k, L - k) this thread forms, read while
  // the rows land (as in k_rows_c2r)
  constexpr int KPT = (H + NT - 1) / NT;
  float2 wk[KPT][2];
#pragma unroll
  for (int q = 0; q < KPT; q++) {
    const int k = threadIdx.x + q * NT;
    if (k < H) {
      wk[q][0] = conjg(tw[k * twStep]);
      wk[q][1] = conjg(tw[(k == 0 ? H : L - k) * twStep]);
    }
  }
  cp_async_wait<0>();
  __syncthreads();
#pragma unroll
  for (int q = 0; q < KPT; q++) {
    const int k = threadIdx.x + q * NT;
    if (k >= H) continue;
    const int kk[2] = {k, k == 0 ? H : L - k};
    for (int r = 0; r < nb; r++) {
      float2* a = A + r * SL;
      float2 Xa = a[pad(k)], Xb = a[pad(k == 0 ? L : L - k)];
      if (k == 0) { Xa.y = 0; Xb.y = 0; }
      float2 res[2];
#pragma unroll
      for (int e = 0; e < 2; e++) {
        float2 Xk, XL;
        if (e == 0) { Xk = Xa; XL = Xb; }
        else if (k == 0) { Xk = a[pad(H)]; XL = Xk; }
        else { Xk = Xb; XL = Xa; }
        const float2 Xc = conjg(XL);
        const float2 sv = cadd(Xk, Xc), d = csub(Xk, Xc);
        const float2 t = cmul(wk[q][e], d);
        res[e] = make_float2(sv.x - t.y, sv.y + t.x);
      }
      a[pad(kk[0])] = res[0];
      a[pad(kk[1])] = res[1];
    }
  }
  __syncthreads();
  // the inverse FFT; its last pass writes the value pairs of the row
  constexpr int E = E_C2R32, NS = last_ns<L, E>(), R = L / NS, T = L / E, NB = E / R, Q = L / R;
  fft_passes_below<L, 1, NS, true, false, E>(A, nb, tws);
  const int sq = threadIdx.x / T, j = threadIdx.x % T;
  if (sq >= nb) return;
  const float2* a = A + sq * SL;
  double* o = out + (size_t)(row0 + sq) * outStride;
  float2 x[E];
  const int pj = pad(j);
#pragma unroll
  for (int u = 0; u < NB; u++)
#pragma unroll
    for (int m = 0; m < R; m++) x[u * R + m] = a[pad_at<T, Q>(pj, j, u, m)];
#pragma unroll
  for (int u = 0; u < NB; u++) {
    float2* xb = x + u * R;
    const int k = j + u * T;
    if (k) apply_twiddles<L, E, R, NS, true>(xb, tws, k);
    dft<R, true>(xb);
#pragma unroll
    for (int q = 0; q < (HOUT ? R / 2 : R); q++) {
      const int n = k + q * NS;
      const float2 v = xb[out_reg<R>(q)];
      if (2 * n + 1 < ncolsOut) *reinterpret_cast<double2*>(o + 2 * n) = make_double2(v.x, v.y);
      else if (2 * n < ncolsOut) o[2 * n] = v.x;
    }
  }
}

template <int L> inline size_t smem_for32(int nseq = Len<L>::B) {
  return sizeof(float2) * ((size_t)nseq * Len<L>::SL + Len<L>::TW);
}

} // namespace

bool poisson32_setup() {
  bool ok = true;
  auto allow = [&](const void* f) { ok &= allow_max_dynamic_smem(f) == cudaSuccess; };
#define X(L) allow((const void*)k_rows_r2c32<L, false>); allow((const void*)k_rows_r2c32<L, true>); \
             allow((const void*)k_rows_c2r32<L, false>); allow((const void*)k_rows_c2r32<L, true>); \
             allow((const void*)k_cols32<L, false>); allow((const void*)k_cols32<L, true>);
  CUP2D_FFT_LENGTHS(X)
#undef X
  return ok;
}

float2* make_tables32(int L, bool cols, const std::vector<float2>& tw, cudaStream_t st) {
  static_assert(E_ROWS32 == E_C2R32, "one table serves both row passes");
  std::vector<float2> t;
  switch (L) {
#define X(LL) case LL: if (cols) fill_tables32<LL, E_COLS32>(tw, t); else fill_tables32<LL, E_ROWS32>(tw, t); break;
    CUP2D_FFT_LENGTHS(X)
#undef X
  }
  float2* d = nullptr;
  if (t.empty() || device_malloc(&d, sizeof(float2) * t.size()) != cudaSuccess) return nullptr;
  h2d_sync(d, t.data(), sizeof(float2) * t.size(), st);
  return d;
}

bool rows_r2c32(int L, cudaStream_t st, const double* in, int inStride, int nrows, int ncolsIn,
                float2* out, int outRows, const float2* tab, const float2* tw, int twLen, FadeArgs fa, bool halfIn) {
  switch (L) {
#define X(LL) case LL: \
    if (halfIn) launch_k(k_rows_r2c32<LL, true>, (nrows + Len<LL>::B - 1) / Len<LL>::B, Len<LL, E_ROWS32>::NT, \
        smem_for32<LL>(), st, in, inStride, nrows, ncolsIn, out, outRows, tab, tw, twLen, fa); \
    else launch_k(k_rows_r2c32<LL, false>, (nrows + Len<LL>::B - 1) / Len<LL>::B, Len<LL, E_ROWS32>::NT, \
        smem_for32<LL>(), st, in, inStride, nrows, ncolsIn, out, outRows, tab, tw, twLen, fa); \
    return true;
    CUP2D_FFT_LENGTHS(X)
#undef X
  }
  return false;
}

bool cols32(int L, cudaStream_t st, float2* data, int rows, int ncols, int nrowsIn, int nrowsOut,
            const float* ghat, int mode, const float2* tab, double norm, int MXp, int MYp) {
  switch (L) {
#define X(LL) case LL: \
    if (mode == 0) launch_k(k_cols32<LL, true>, (ncols + Col32<LL>::CB - 1) / Col32<LL>::CB, Col32<LL>::NT, \
        smem_for32<LL>(Col32<LL>::CB), st, data, rows, ncols, nrowsIn, nrowsOut, \
        ghat, mode, tab, norm, MXp, MYp); \
    else launch_k(k_cols32<LL, false>, (ncols + Col32<LL>::CB - 1) / Col32<LL>::CB, Col32<LL>::NT, \
        smem_for32<LL>(Col32<LL>::CB), st, data, rows, ncols, nrowsIn, nrowsOut, \
        ghat, mode, tab, norm, MXp, MYp); \
    return true;
    CUP2D_FFT_LENGTHS(X)
#undef X
  }
  return false;
}

bool rows_c2r32(int L, cudaStream_t st, const float2* in, int inRows, int nrows, double* out, int outStride,
                int ncolsOut, const float2* tab, const float2* tw, int twLen, bool halfOut) {
  switch (L) {
#define X(LL) case LL: \
    if (halfOut) launch_k(k_rows_c2r32<LL, true>, (nrows + Len<LL>::B - 1) / Len<LL>::B, Len<LL, E_C2R32>::NT, \
        smem_for32<LL>(), st, in, inRows, nrows, out, outStride, ncolsOut, tab, tw, twLen); \
    else launch_k(k_rows_c2r32<LL, false>, (nrows + Len<LL>::B - 1) / Len<LL>::B, Len<LL, E_C2R32>::NT, \
        smem_for32<LL>(), st, in, inRows, nrows, out, outStride, ncolsOut, tab, tw, twLen); \
    return true;
    CUP2D_FFT_LENGTHS(X)
#undef X
  }
  return false;
}

} // namespace cup2d

#ifdef CUP2D_TRACE
namespace cup2d { void trace_bind_poisson32(unsigned long long* p) { trace_bind_this_unit(p); } }
#endif
