// Eigenvalue-only path for small Hermitian matrices (order <= 32): Householder reduction to a real
// symmetric tridiagonal T, then Sturm counts on T.
//
// Used where only band energies or energy-window band ranges are needed: the window test of
// src/filter.jl:19,40-72 (first = searchsortedfirst(e, wmin) = #(e < wmin) + 1, last =
// searchsortedlast(e, wmax) = #(e <= wmax)) and eigvals_batched (ext/ElectronPhononCUDAExt.jl:80-98,
// src/wannier_to_bloch_batched.jl:30-46). A window needs two Sturm counts instead of a full
// eigensolve; eigenvalues come from bisection on T.
//
// N lanes per matrix (N = 8, 16 or 32); lane i holds row i of the (zero-padded) N x N matrix in registers. Step k
// (k = 0 .. n-2) reflects x = A[k+1:N, k] onto a multiple of e_1 with the Hermitian unitary
// P = I - beta u u^H, u = x + e^{i theta} ||x|| e_1 (theta = arg x_1), beta = 1 / (||x|| (||x|| + |x_1|)),
// and updates the trailing block as A <- A - u w^H - w u^H with p = beta A u,
// K = (beta / 2) u^H p (real), w = p - K u. The tridiagonal keeps d_k = A[k][k] and the squared
// off-diagonal e_k^2 = ||x||^2 (the phase of the off-diagonal does not change the eigenvalues).
// Rows and columns beyond the true order n are zero and stay decoupled; counts run over the first
// n entries only.
//
// Sturm count (number of eigenvalues below sigma): q_0 = d_0 - sigma,
// q_i = d_i - sigma - e_{i-1}^2 / q_{i-1}, count the negative q_i; |q| < pivmin is replaced by
// -pivmin (the LAPACK dstebz convention).
#include <algorithm>

#include "epb_common.cuh"

namespace epb {

constexpr int TRI_WARPS = 4;  // warps per block
// Blocks per SM to leave registers for: FP64 rows of 32 fit 168 registers, smaller ones 128.
#define TRI_MINB(T, N) (sizeof(T) == 8 ? ((N) == 32 ? 3 : 4) : 4)

struct TriArgs {
  const float* Hp;     // Hermitian-packed FP32 input (n^2 floats per matrix: Re i<=j, then Im i<j)
  const double2* A;    // or c128 column-major input (upper triangle read)
  int n;
  int64_t batch;
  // window mode
  int nsh;             // 2 (exact) or 4 (guarded: wmin -/+ delta, wmax -/+ delta)
  double sh[4];        // shifts; counts are #(lambda < sh)
  int32_t* bmin;       // first in-window band (1-based) or 0
  int32_t* bmax;       // last in-window band or 0
  int32_t* flag;       // guarded mode: 1 if an eigenvalue may lie within delta of a window edge
  // eigenvalue mode
  double* E;           // (n, batch) ascending
  // tridiagonal mode: d and e^2 per matrix (32 doubles each)
  double* Dt;
  double* E2t;
};

// N rows per matrix, one per lane: 32 / N matrices per warp.
template <typename T, int N>
struct TriSmem {
  typename cplx<T>::type u[N];  // reflector u
  typename cplx<T>::type w[N];  // w = p - K u
  T d[N];       // tridiagonal
  T e2[N];
  float stage[sizeof(T) == 4 ? N * N : 1];  // packed FP32 input staging
};

// Sum over the N lanes of a matrix.
template <int N, typename T>
__device__ __forceinline__ T group_sum(T v) {
#pragma unroll
  for (int o = N / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// v = x if j == k, as a predicated move: a chain of C selects over a register array becomes an indexed load from
// local memory.
__device__ __forceinline__ void tri_pick(double& v, double x, int j, int k) {
  asm("{\n\t.reg .pred p;\n\tsetp.eq.s32 p, %2, %3;\n\t@p mov.f64 %0, %1;\n\t}" : "+d"(v) : "d"(x), "r"(j), "r"(k));
}
__device__ __forceinline__ void tri_pick(float& v, float x, int j, int k) {
  asm("{\n\t.reg .pred p;\n\tsetp.eq.s32 p, %2, %3;\n\t@p mov.f32 %0, %1;\n\t}" : "+f"(v) : "f"(x), "r"(j), "r"(k));
}

// Square root of x2 and its reciprocal (1 for zero). FP64 takes one reciprocal square root, good to an ulp, for a square
// root and a division; the FP32 one is good to two only, so FP32 takes the square root and divides.
__device__ __forceinline__ double tri_root(double x2, double& inv) {
  inv = rsqrt(x2 == 0.0 ? 1.0 : x2);
  return x2 * inv;
}
__device__ __forceinline__ float tri_root(float x2, float& inv) {
  const float x = sqrtf(x2);
  inv = 1.f / (x2 == 0.f ? 1.f : x);
  return x;
}

__device__ __forceinline__ double sturm_div(double a, double b) { return a / b; }
// FP32 counts are only used with guard intervals far wider than the 2-ulp fast division error.
__device__ __forceinline__ float sturm_div(float a, float b) { return __fdividef(a, b); }

template <typename T>
__device__ __forceinline__ int sturm_count(const T* d, const T* e2, int n, T sigma, T pivmin) {
  int c = 0;
  T q = d[0] - sigma;
  if (fabs(q) < pivmin) q = -pivmin;
  c += q < T(0);
  for (int i = 1; i < n; ++i) {
    q = (d[i] - sigma) - sturm_div(e2[i - 1], q);
    if (fabs(q) < pivmin) q = -pivmin;
    c += q < T(0);
  }
  return c;
}

// Steps k = J0 .. min(J0 + 8, N - 1) - 1 of the reduction (see the file header). The step loop is not
// unrolled (a fully unrolled 31-step reduction overflows the instruction cache); the inner loops run
// over the compile-time range j = J0 .. N - 1 with the columns j <= k masked, and column k + 1 is
// picked from registers by an 8-way select. xn2 enters as ||A[k+1:, k]||^2 of the first step and leaves as that of the
// step after the last: the next column follows from u and w before the block update, so the sum over its lanes
// runs between the update's FMAs instead of at the head of the next step.
template <typename T, int N, int J0>
__device__ __forceinline__ void householder_phase(T (&ar)[N], T (&ai)[N], TriSmem<T, N>& s, int lane, int n, T& dk,
                                                  T& ek2, T& xn2, T& xr, T& xi) {
  constexpr int KEND = (J0 + 8 < N - 1) ? J0 + 8 : N - 1;
#pragma unroll 1
  for (int k = J0; k < KEND && k < n; ++k) {  // the columns of the padding are zero
    // (xr, xi): column k, row `lane`; column k + 1 is picked for its early update
    T nr = 0, ni = 0;
#pragma unroll
    for (int j = J0 + 1; j < J0 + 9 && j < N; ++j) {
      tri_pick(nr, ar[j], j, k + 1);
      tri_pick(ni, ai[j], j, k + 1);
    }
    if (lane == k) {
      dk = xr;
      ek2 = xn2;
    }
    if (k == N - 2 || k == n - 1) break;  // last off-diagonal, or last row of the matrix: no reflection left to apply
    const T x1r = __shfl_sync(0xffffffffu, xr, k + 1, N), x1i = __shfl_sync(0xffffffffu, xi, k + 1, N);
    const T a2 = x1r * x1r + x1i * x1i;
    T rx, ra;
    const T xn = tri_root(xn2, rx), a1 = tri_root(a2, ra);
    // a column that is already reduced takes beta = 0: nothing changes. In FP64 so does one so short that 1 / xn2 would
    // leave the range of a double.
    const T beta = xn2 <= (sizeof(T) == 8 ? T(1e-290) : T(0)) ? T(0) : T(1) / fma(xn, a1, xn2);
    T ur = T(0), ui = T(0);
    if (lane > k + 1) {
      ur = xr;
      ui = xi;
    } else if (lane == k + 1) {
      // u_1 = e^{i theta} (|x_1| + ||x||)
      const T f = fma(xn, ra, T(1));
      ur = a2 == T(0) ? xn : x1r * f;
      ui = a2 == T(0) ? T(0) : x1i * f;
    }
    s.u[lane] = mk2(ur, ui);  // zero for lanes <= k
    __syncwarp();
    // p_i = beta sum_{j>k} A[i][j] u_j (u_j = 0 for j <= k; four partial sums per part)
    T pr0 = 0, pi0 = 0, pr1 = 0, pi1 = 0, pr2 = 0, pi2 = 0, pr3 = 0, pi3 = 0;
#pragma unroll
    for (int j = J0 + 1; j < N; ++j) {
      const auto v = s.u[j];
      if ((j & 1) == 0) {
        pr0 = fma(ar[j], v.x, pr0);
        pr2 = fma(-ai[j], v.y, pr2);
        pi0 = fma(ar[j], v.y, pi0);
        pi2 = fma(ai[j], v.x, pi2);
      } else {
        pr1 = fma(ar[j], v.x, pr1);
        pr3 = fma(-ai[j], v.y, pr3);
        pi1 = fma(ar[j], v.y, pi1);
        pi3 = fma(ai[j], v.x, pi3);
      }
    }
    T pr = ((pr0 + pr1) + (pr2 + pr3)) * beta, pi = ((pi0 + pi1) + (pi2 + pi3)) * beta;
    if (lane <= k) {
      pr = T(0);
      pi = T(0);
    }
    // K = (beta / 2) Re(u^H p)
    const T kk = T(0.5) * beta * group_sum<N>(fma(ur, pr, ui * pi));
    const T wr = fma(-kk, ur, pr), wi = fma(-kk, ui, pi);
    s.w[lane] = mk2(wr, wi);
    __syncwarp();
    // column k + 1 after the update, its squared length below the diagonal summed in the gaps of the update
    {
      const auto uj = s.u[k + 1], wj = s.w[k + 1];
      nr -= fma(wi, uj.y, fma(wr, uj.x, fma(ui, wj.y, ur * wj.x)));
      ni -= fma(-wr, uj.y, fma(wi, uj.x, fma(-ur, wj.y, ui * wj.x)));
    }
    xr = nr;  // the next step's column
    xi = ni;
    xn2 = lane > k + 1 ? fma(nr, nr, ni * ni) : T(0);
    constexpr int LEN = N - J0 - 1, PARTS = N == 32 ? 5 : N == 16 ? 4 : 3;
    T other = 0;
#pragma unroll
    for (int j = J0 + 1; j < N; ++j) {
#pragma unroll
      for (int p = 0; p < PARTS; ++p)
        if (j - J0 - 1 == p * LEN / PARTS) {  // compile-time: one butterfly step ahead of each part of the update
          xn2 += other;
          other = __shfl_xor_sync(0xffffffffu, xn2, N >> (p + 1));
        }
      if (j > k) {
        const auto uj = s.u[j], wj = s.w[j];
        // A[i][j] -= u_i conj(w_j) + w_i conj(u_j); u_i = w_i = 0 for rows i <= k. The four products are summed first:
        // one rounding at the size of A (four FMAs onto A: eigenvalues of order 8 off by 0.43 eps of the norm in rms
        // instead of 0.35, of order 24 by 0.172 instead of 0.163).
        ar[j] -= fma(wi, uj.y, fma(wr, uj.x, fma(ui, wj.y, ur * wj.x)));
        ai[j] -= fma(-wr, uj.y, fma(wi, uj.x, fma(-ur, wj.y, ui * wj.x)));
      }
    }
    xn2 += other;
    __syncwarp();
  }
}

// Reduce the matrix held row-wise in (ar, ai) to tridiagonal form; writes d, e2 to shared memory.
template <typename T, int N>
__device__ __forceinline__ void householder_tridiag(T (&ar)[N], T (&ai)[N], TriSmem<T, N>& s, int lane, int n) {
  static_assert(N == 8 || N == 16 || N == 32, "the reduction is laid out in phases of eight steps");
  T dk = 0, ek2 = 0, xn2 = group_sum<N>(lane > 0 ? ar[0] * ar[0] + ai[0] * ai[0] : T(0));
  T xr = ar[0], xi = ai[0];
  householder_phase<T, N, 0>(ar, ai, s, lane, n, dk, ek2, xn2, xr, xi);
  if constexpr (N > 8) householder_phase<T, N, 8>(ar, ai, s, lane, n, dk, ek2, xn2, xr, xi);
  if constexpr (N > 16) {
    householder_phase<T, N, 16>(ar, ai, s, lane, n, dk, ek2, xn2, xr, xi);
    householder_phase<T, N, 24>(ar, ai, s, lane, n, dk, ek2, xn2, xr, xi);
  }
  if (lane == N - 1) dk = ar[N - 1];
  s.d[lane] = dk;
  s.e2[lane] = ek2;
  __syncwarp();
}

// Load row `lane` of matrix b (upper triangle as stored, Hermitian completion, zero padding).
template <typename T, int N>
__device__ __forceinline__ void load_rows(const TriArgs& a, int64_t b, int lane, bool live, T (&ar)[N], T (&ai)[N],
                                          TriSmem<T, N>& s) {
  const int n = live ? a.n : 0;
  if (a.Hp) {
    const float* src = a.Hp + b * (int64_t)n * n;
    if (sizeof(T) == 4)  // the FP32 reductions read their packed rows through shared memory
      for (int e = lane; e < n * n; e += N) s.stage[e] = src[e];
    __syncwarp();
    const float* st = sizeof(T) == 4 ? s.stage : src;
    const int nre = n * (n + 1) / 2;
#pragma unroll
    for (int j = 0; j < N; ++j) {
      T re = 0, im = 0;
      if (lane < n && j < n) {
        if (lane <= j) {
          re = st[j * (j + 1) / 2 + lane];
          im = lane < j ? st[nre + j * (j - 1) / 2 + lane] : 0.f;
        } else {
          re = st[lane * (lane + 1) / 2 + j];
          im = -st[nre + lane * (lane - 1) / 2 + j];
        }
      }
      ar[j] = re;
      ai[j] = im;
    }
    __syncwarp();
  } else {
    const double2* src = a.A + b * (int64_t)n * n;
#pragma unroll
    for (int j = 0; j < N; ++j) {
      T re = 0, im = 0;
      if (lane < n && j < n) {
        if (lane <= j) {
          const double2 v = src[lane + (int64_t)j * n];
          re = (T)v.x;
          im = lane < j ? (T)v.y : T(0);
        } else {
          const double2 v = src[j + (int64_t)lane * n];
          re = (T)v.x;
          im = (T)-v.y;
        }
      }
      ar[j] = re;
      ai[j] = im;
    }
  }
}

// Number of sign changes of the Sturm sequence p_i = (d_i - sigma) p_{i-1} - e_{i-1}^2 p_{i-2} of a tridiagonal
// scaled to norm <= 1, i.e. of eigenvalues below sigma. No division on the chain: 53 bisection steps of order 8 take a
// fifth of the quotients' time. Every e^2 is zero or at least STURM_E2 (the caller sees to it).
// A zero p_i takes the sign opposite to its predecessor's; the next one is -e_i^2 p_{i-1} with that sign, so one change
// is counted. Where e_i^2 is zero nothing of the block above reaches p_{i+1}, and after a zero p_i the recurrence would
// stay at zero for good: the row starts a block of its own, p_{i+1} = d_{i+1} - sigma after a one.
// |p_i| <= 3^i. The larger of two neighbours falls by at most STURM_E2 / 2 a step, so lifting both every fourth step
// keeps them out of the underflow range.
constexpr double STURM_E2 = 0x1p-120;
__device__ __forceinline__ int sturm_signs(const double* d, const double* e2, int n, double sigma) {
  double p1 = 1.0, p = d[0] - sigma;
  bool neg = !(p > 0.0);
  int c = neg;
  for (int i = 1; i < n; ++i) {
    const double b = e2[i - 1];
    const bool first = b == 0.0;
    const double q = first ? 1.0 : p;
    const double t = fma(d[i] - sigma, q, -(b * p1));
    neg = neg && !first;
    p1 = q;
    p = t;
    const bool ng = t < 0.0 || (t == 0.0 && !neg);
    c += ng != neg;
    neg = ng;
    if ((i & 3) == 0 && fmax(fabs(p), fabs(p1)) < 0x1p-300) {
      p *= 0x1p600;
      p1 *= 0x1p600;
    }
  }
  return c;
}

// MODE 0: window band ranges from Sturm counts at the shifts; MODE 1: all eigenvalues; MODE 2: the
// tridiagonal itself (d, e^2) for a later per-band bisection. N lanes per matrix. What bounds the FP64 reduction:
// three warps per scheduler (a row of 32 takes 168 registers), each step a chain of two lane sums, two reciprocal
// square roots and a division around 14 FP64 operations per column, and its broadcast reads of u and w. Window counts of
// 98292 matrices of order 32: 5.5 -> 4.4 ms (two blocks per SM, without the few spills, a sixth more).
template <typename T, int N, int MODE>
__global__ void __launch_bounds__(32 * TRI_WARPS, TRI_MINB(T, N)) tridiag_kernel(TriArgs a) {
  constexpr int G = 32 / N;  // matrices per warp
  __shared__ TriSmem<T, N> smem[TRI_WARPS * G];
  const int warp = threadIdx.x >> 5, g = (threadIdx.x & 31) / N, lane = threadIdx.x & (N - 1);
  TriSmem<T, N>& s = smem[warp * G + g];
  const int n = a.n;
  const int64_t w0 = (int64_t)blockIdx.x * TRI_WARPS + warp, nwarps = (int64_t)gridDim.x * TRI_WARPS;
  for (int64_t base = w0 * G; base < a.batch; base += nwarps * G) {
    const int64_t b = base + g;
    const bool live = b < a.batch;
    T ar[N], ai[N];
    load_rows<T, N>(a, b, lane, live, ar, ai, s);
    householder_tridiag<T, N>(ar, ai, s, lane, n);
    if (MODE == 2) {
      if (live) {
        a.Dt[b * 32 + lane] = (double)s.d[lane];
        a.E2t[b * 32 + lane] = (double)s.e2[lane];
      }
      __syncwarp();
      continue;
    }
    if (MODE == 0) {
      // pivmin: smallest safe pivot scaled by the largest off-diagonal (dstebz)
      T emax = 0;
      for (int i = 0; i < n; ++i) emax = fmax(emax, s.e2[i]);
      const T tiny = sizeof(T) == 8 ? T(2.2250738585072014e-308) : T(1.17549435e-38);
      const T pivmin = tiny * fmax(T(1), emax);
      int c = 0;
      const double shv = lane == 0 ? a.sh[0] : lane == 1 ? a.sh[1] : lane == 2 ? a.sh[2] : a.sh[3];
      if (lane < a.nsh) c = sturm_count<T>(s.d, s.e2, n, (T)shv, pivmin);
      const int c0 = __shfl_sync(0xffffffffu, c, 0, N), c1 = __shfl_sync(0xffffffffu, c, 1, N);
      const int c2 = __shfl_sync(0xffffffffu, c, 2, N), c3 = __shfl_sync(0xffffffffu, c, 3, N);
      if (lane == 0 && live) {
        // exact: c0 = #(e < wmin), c1 = #(e <= wmax) (shift 1 is the successor of wmax).
        // guarded: c0/c1 bracket wmin and c2/c3 bracket wmax.
        const int below = c0, upto = a.nsh == 2 ? c1 : c3;
        const int first = below + 1, last = upto;
        const bool keep = last >= first;
        a.bmin[b] = keep ? first : 0;
        a.bmax[b] = keep ? last : 0;
        if (a.flag) a.flag[b] = a.nsh == 4 && ((c0 != c1) || (c2 != c3));
      }
    } else if constexpr (MODE == 1 && sizeof(T) == 8) {
      // Gershgorin interval of T, scaled to [-1, 1], then bisection for eigenvalue `lane` (the (lane+1)-th smallest)
      const double eo = lane < n - 1 ? sqrt(s.e2[lane]) : 0.0;
      const double ep = __shfl_up_sync(0xffffffffu, eo, 1, N);
      const double rad = eo + (lane > 0 ? ep : 0.0);
      double span = lane < n ? fabs(s.d[lane]) + rad : 0.0;
#pragma unroll
      for (int o = N / 2; o > 0; o >>= 1) span = fmax(span, __shfl_xor_sync(0xffffffffu, span, o));
      // An infinity or NaN of the matrix is one in its column's length, hence in T (fmax above drops NaN): no energies.
      const unsigned odd = __ballot_sync(0xffffffffu, lane < n && !(isfinite(s.d[lane]) && isfinite(s.e2[lane])));
      const bool bad = (odd >> (N * g) & (0xffffffffu >> (32 - N))) != 0 || !isfinite(span);
      int ex = 0;
      if (span > 0.0 && !bad) frexp(span, &ex);
      ex = max(ex, -500);  // below, squares underflow anyway, and sc would overflow
      const double sc = ldexp(1.0, -ex);
      __syncwarp();
      s.d[lane] *= sc;
      const double es = s.e2[lane] * sc * sc;
      s.e2[lane] = es < STURM_E2 ? 0.0 : es;  // |e| < 2^-60 of the norm: below a hundredth of its last bit
      __syncwarp();
      const double eps = 2.220446049250313e-16;
      // padding rows do not widen the interval
      double lo = lane < n ? s.d[lane] - rad * sc : 1.0, hi = lane < n ? s.d[lane] + rad * sc : -1.0;
#pragma unroll
      for (int o = N / 2; o > 0; o >>= 1) {
        lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
      }
      if (span > 0.0) {  // the zero matrix keeps [0, 0]
      lo -= 4 * eps;
        hi += 4 * eps;
      }
      if (lane < n && live) {
        for (int it = bad ? 200 : 0; it < 200; ++it) {
          const double mid = 0.5 * (lo + hi);
          if (!(hi - lo > 2 * eps * fmax(fabs(lo), fabs(hi))) || mid <= lo || mid >= hi) break;
          if (sturm_signs(s.d, s.e2, n, mid) > lane)
            hi = mid;
          else
            lo = mid;
        }
        a.E[b * (int64_t)n + lane] = bad ? nan("") : ldexp(0.5 * (lo + hi), ex);
      }
    }
    __syncwarp();
  }
}

// One eigenvalue (0-based index `band`) per stored tridiagonal, one thread per matrix: bisection
// on the Gershgorin interval with Sturm counts, as in MODE 1.
__global__ void tridiag_band_kernel(const double* __restrict__ Dt, const double* __restrict__ E2t, int n, int64_t batch,
                                    int band, double* __restrict__ out) {
  for (int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; b < batch; b += (int64_t)gridDim.x * blockDim.x) {
    double d[32], e2[32];
    double emax = 0, lo = 0, hi = 0;
    for (int i = 0; i < n; ++i) {
      d[i] = Dt[b * 32 + i];
      e2[i] = E2t[b * 32 + i];
    }
    for (int i = 0; i < n; ++i) {
      emax = fmax(emax, e2[i]);
      const double r = (i > 0 ? sqrt(e2[i - 1]) : 0.0) + (i < n - 1 ? sqrt(e2[i]) : 0.0);
      lo = i == 0 ? d[i] - r : fmin(lo, d[i] - r);
      hi = i == 0 ? d[i] + r : fmax(hi, d[i] + r);
    }
    const double pivmin = 2.2250738585072014e-308 * fmax(1.0, emax), eps = 2.220446049250313e-16;
    const double span = fmax(fabs(lo), fabs(hi));
    lo -= 2 * eps * span + 2 * pivmin;
    hi += 2 * eps * span + 2 * pivmin;
    for (int it = 0; it < 200; ++it) {
      const double mid = 0.5 * (lo + hi);
      if (!(hi - lo > 2 * eps * fmax(fabs(lo), fabs(hi)) + pivmin) || mid <= lo || mid >= hi) break;
      if (sturm_count<double>(d, e2, n, mid, pivmin) > band)
        hi = mid;
      else
        lo = mid;
    }
    out[b] = 0.5 * (lo + hi);
  }
}

template <typename T, int N, int MODE>
static int launch_order(epb_ctx* ctx, const TriArgs& a) {
  auto kern = tridiag_kernel<T, N, MODE>;
  int per_sm = 0;
  EPB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * TRI_WARPS, 0));
  if (per_sm < 1) per_sm = 1;
  int64_t blocks = std::min<int64_t>(cdiv(a.batch, TRI_WARPS * (32 / N)), (int64_t)per_sm * ctx->sm_count * 4);
  if (blocks < 1) blocks = 1;
  prof_begin(ctx, EPB_PROF_TRIDIAG);
  kern<<<(unsigned)blocks, 32 * TRI_WARPS, 0, ctx->stream>>>(a);
  prof_end(ctx);
  EPB_LAUNCH_CHECK();
  return EPB_OK;
}

template <typename T, int MODE>
static int launch_tridiag(epb_ctx* ctx, const TriArgs& a) {
  if (a.n <= 8) return launch_order<T, 8, MODE>(ctx, a);
  if (a.n <= 16) return launch_order<T, 16, MODE>(ctx, a);
  return launch_order<T, 32, MODE>(ctx, a);
}

// Window band ranges of a batch of order-n Hermitian matrices (packed FP32 `Hp` or c128 `A`).
// delta == 0: exact counts at wmin and the successor of wmax (FP64 solve). delta > 0: FP32 solve
// with guard shifts wmin -/+ delta and wmax -/+ delta; `flag` marks the matrices whose counts
// differ across a guard interval (an eigenvalue may lie within delta of an edge).
int tridiag_window(epb_ctx* ctx, const float* Hp, const double2* A, int n, int64_t batch, double wmin, double wmax,
                   double delta, int32_t* bmin, int32_t* bmax, int32_t* flag) {
  if (batch == 0) return EPB_OK;
  EPB_CHECK_ARG(n >= 1 && n <= 32, "window counts: order %d outside 1..32", n);
  TriArgs a{};
  a.Hp = Hp;
  a.A = A;
  a.n = n;
  a.batch = batch;
  a.bmin = bmin;
  a.bmax = bmax;
  a.flag = flag;
  if (delta > 0) {
    EPB_CHECK_ARG(flag, "window counts: guarded mode needs a flag array");
    a.nsh = 4;
    a.sh[0] = wmin - delta;
    a.sh[1] = wmin + delta;
    a.sh[2] = wmax - delta;
    a.sh[3] = wmax + delta;
    return launch_tridiag<float, 0>(ctx, a);
  }
  a.nsh = 2;
  a.sh[0] = wmin;
  a.sh[1] = nextafter(wmax, INFINITY);
  return launch_tridiag<double, 0>(ctx, a);
}

// Energy of band `band` (0-based) of each matrix: FP64 reduction stored to Dt/E2t (batch x 32
// doubles each, caller workspace), then one bisection per matrix.
int tridiag_band(epb_ctx* ctx, const float* Hp, const double2* A, int n, int64_t batch, int band, double* Dt,
                 double* E2t, double* out) {
  if (batch == 0) return EPB_OK;
  EPB_CHECK_ARG(n >= 1 && n <= 32 && band >= 0 && band < n, "band energy: order %d / band %d", n, band);
  TriArgs a{};
  a.Hp = Hp;
  a.A = A;
  a.n = n;
  a.batch = batch;
  a.Dt = Dt;
  a.E2t = E2t;
  EPB_TRY((launch_tridiag<double, 2>(ctx, a)));
  const int64_t blocks = std::min<int64_t>(cdiv(batch, 128), (int64_t)ctx->sm_count * 16);
  prof_begin(ctx, EPB_PROF_TRIDIAG);
  tridiag_band_kernel<<<(unsigned)std::max<int64_t>(blocks, 1), 128, 0, ctx->stream>>>(Dt, E2t, n, batch, band, out);
  prof_end(ctx);
  EPB_LAUNCH_CHECK();
  return EPB_OK;
}

// Ascending eigenvalues (FP64 reduction and bisection) of a batch of order-n Hermitian matrices.
int tridiag_eigvals(epb_ctx* ctx, const float* Hp, const double2* A, int n, int64_t batch, double* E) {
  if (batch == 0) return EPB_OK;
  EPB_CHECK_ARG(n >= 1 && n <= 32, "tridiagonal eigenvalues: order %d outside 1..32", n);
  TriArgs a{};
  a.Hp = Hp;
  a.A = A;
  a.n = n;
  a.batch = batch;
  a.E = E;
  return launch_tridiag<double, 1>(ctx, a);
}

}  // namespace epb
