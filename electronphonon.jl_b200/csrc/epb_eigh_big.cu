// Batched Hermitian eigensolver for orders 65 .. 96: FP32 two-sided Jacobi in shared memory, then
// FP64 Rayleigh-Ritz refinement with exact FP64 treatment of near-degenerate clusters.
//
// Replaces eigen_batched / eigvals_batched (ext/ElectronPhononCUDAExt.jl:80-115; CPU reference
// src/wannier_to_bloch_batched.jl:30-65, LAPACK ZHEEV) for the orders whose FP64 Jacobi state
// (A and V, 2 n^2 complex doubles) does not fit in shared memory.
//
// One CTA (512 threads) per matrix, persistent, matrices taken from a device work counter so that
// uneven orders balance. Per matrix:
//  1. A (Hermitian completion of the upper triangle) in FP32 in shared memory, cyclic two-sided
//     Jacobi with round-robin pairs (jacobi_block) accumulating V in FP32.
//  2. FP64 refinement, `refine` iterations, each on the CTA's global scratch (L2-resident):
//       G = V^H V,  V <- V (3/2 I - 1/2 G)               (Loewdin re-orthonormalisation)
//       S = V^H (H V), lambda_i = Re S_ii, tau = max(100 max_{i != j} |S_ij|, 1e-6 max |lambda|)
//       clusters: runs of the sorted lambda with consecutive gaps < tau
//       M_ij = S_ij / (lambda_j - lambda_i) between clusters (first-order Rayleigh-Ritz),
//       Q_c = the FP64 Jacobi eigenvectors of the cluster block S_cc (re-orthogonalisation of the
//             cluster inside its invariant subspace; clusters of up to 32 members)
//       V <- V (I + X) blockdiag(Q_c), X the first-order coefficients (zero inside clusters)
//  3. A last Loewdin step and S; eigenvalues = Re S_ii (Rayleigh quotients) ascending, eigenvectors
//     written over the input in ascending order.
// The FP32 solve leaves |S_ij| ~ 1e-7 ||H||; each refinement squares the relative error, so two
// iterations reach FP64 accuracy. EPB_PREC_FP64 runs three.
#include <algorithm>

#include "epb_jacobi.cuh"

namespace epb {

constexpr int BIG_NMAX = 96;

struct BigArgs {
  double2* A;
  const int64_t* a_off;
  const int32_t* nvec;
  int n_uniform;
  int64_t batch;
  double* E;
  const int64_t* e_off;
  int want_v;
  int max_sweeps;
  int refine;
  int n_lo;                        // orders <= n_lo belong to other kernels (skipped silently)
  int n_hi;                        // > 0: orders above n_hi belong to other kernels (skipped silently)
  int* nonconv;
  int* badsize;
  unsigned long long* counter;     // work counter (zeroed before launch)
  double2* scratch;                // 3 NMAX^2 per CTA
};

// Complex FP64 n x n GEMM, C = op(A) B, on the FP64 tensor cores (mma.m8n8k4): operands in global memory
// (L2-resident scratch or the input), staged through shared memory in panels of 8 k, the next panel read into
// registers during this one's DMMAs. OPA: 0 = A, 1 = A^H, 2 = Hermitian completion of the upper triangle of A
// (diagonal imaginary part dropped). The refinement is 19 such products per FP64 solve; as scalar FMAs on 32 x 32
// tiles each complex FMA read one and a half operands from shared memory, which bound them: 125 matrices of order 96
// 4.15 -> 3.17 ms with the products at the FP64 pipe's rate.
// Warp grid and 8 x 8 tiles per warp: rows cover NMAX, columns go in passes of WN * NTW tiles.
template <int NMAX> struct BigTile;
template <> struct BigTile<32> { static constexpr int WM = 2, WN = 2, MTW = 2, NTW = 2; };
template <> struct BigTile<48> { static constexpr int WM = 4, WN = 2, MTW = 2, NTW = 3; };
template <> struct BigTile<64> { static constexpr int WM = 4, WN = 2, MTW = 2, NTW = 4; };
template <> struct BigTile<80> { static constexpr int WM = 4, WN = 2, MTW = 3, NTW = 3; };
template <> struct BigTile<96> { static constexpr int WM = 4, WN = 4, MTW = 3, NTW = 3; };
constexpr int BIG_KP = 8;  // k per panel

__device__ __forceinline__ void big_mma(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

template <int OPA, int NMAX, int NT>
__device__ void big_gemm(int n, const double2* __restrict__ A, int lda, const double2* __restrict__ B, int ldb,
                         double2* __restrict__ C, int ldc, double2* st) {
  using T = BigTile<NMAX>;
  static_assert(T::WM * T::WN * 32 == NT && T::WM * T::MTW * 8 >= NMAX && T::WN * T::NTW * 8 <= NMAX, "warp grid");
  constexpr int LD = NMAX + 4, PANEL = BIG_KP * LD;  // rows of a k slice padded: 64-bit fragment reads hit every bank
  constexpr int CP = T::WN * T::NTW * 8;              // columns per pass
  constexpr int EA = (NMAX * BIG_KP + NT - 1) / NT, EB = (CP * BIG_KP + NT - 1) / NT;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, lg = lane >> 2, lk = lane & 3, part = lk & 1;
  const int wm = warp % T::WM, wn = warp / T::WM;
  const int sgn = part ? (int)0x80000000 : 0;
  const int tiles = (n + 7) >> 3;
  for (int j0 = 0; j0 < n; j0 += CP) {
    double2 ra[EA], rb[EB];
    auto fetch = [&](int k0) {
#pragma unroll
      for (int e = 0; e < EA; ++e) {
        const int x = tid + e * NT;
        // lanes along the contiguous axis: i for A, k for A^H
        const int i = OPA == 1 ? x / BIG_KP : x % NMAX, k = k0 + (OPA == 1 ? x % BIG_KP : x / NMAX);
        double2 v = make_double2(0.0, 0.0);
        if (x < NMAX * BIG_KP && i < n && k < n) {
          if (OPA == 0) {
            v = A[i + (int64_t)k * lda];
          } else if (OPA == 1) {
            v = A[k + (int64_t)i * lda];
            v.y = -v.y;
          } else if (i <= k) {
            v = A[i + (int64_t)k * lda];
            if (i == k) v.y = 0.0;
          } else {
            v = A[k + (int64_t)i * lda];
            v.y = -v.y;
          }
        }
        ra[e] = v;
      }
#pragma unroll
      for (int e = 0; e < EB; ++e) {
        const int x = tid + e * NT, k = k0 + x % BIG_KP, j = j0 + x / BIG_KP;
        rb[e] = x < CP * BIG_KP && k < n && j < n ? B[k + (int64_t)j * ldb] : make_double2(0.0, 0.0);
      }
    };
    auto stage = [&](int buf) {
      double2* As = st + buf * 2 * PANEL;
      double2* Bs = As + PANEL;
#pragma unroll
      for (int e = 0; e < EA; ++e) {
        const int x = tid + e * NT;
        if (x < NMAX * BIG_KP) As[(OPA == 1 ? x % BIG_KP : x / NMAX) * LD + (OPA == 1 ? x / BIG_KP : x % NMAX)] = ra[e];
      }
#pragma unroll
      for (int e = 0; e < EB; ++e) {
        const int x = tid + e * NT;
        if (x < CP * BIG_KP) Bs[(x % BIG_KP) * LD + x / BIG_KP] = rb[e];
      }
    };
    double cr[T::MTW][T::NTW][2], ci[T::MTW][T::NTW][2];
#pragma unroll
    for (int i = 0; i < T::MTW; ++i)
#pragma unroll
      for (int j = 0; j < T::NTW; ++j) cr[i][j][0] = cr[i][j][1] = ci[i][j][0] = ci[i][j][1] = 0.0;
    fetch(0);
    __syncthreads();  // the last reads of the shared memory under the panels are done
    stage(0);
    __syncthreads();
    for (int k0 = 0, buf = 0; k0 < n; k0 += BIG_KP, buf ^= 1) {
      if (k0 + BIG_KP < n) fetch(k0 + BIG_KP);
      const double2* As = st + buf * 2 * PANEL;
      const double2* Bs = As + PANEL;
#pragma unroll
      for (int ks = 0; ks < BIG_KP / 2; ++ks) {
        // the real K axis of a DMMA runs over (re, im) of two complex k
        const double* ap = reinterpret_cast<const double*>(As + (ks * 2 + (lk >> 1)) * LD + wm * T::MTW * 8 + lg);
        const double* bp = reinterpret_cast<const double*>(Bs + (ks * 2 + (lk >> 1)) * LD + wn * T::NTW * 8 + lg);
        double av[T::MTW];
#pragma unroll
        for (int i = 0; i < T::MTW; ++i) av[i] = ap[i * 16 + part];
#pragma unroll
        for (int j = 0; j < T::NTW; ++j) {
          if (j0 / 8 + wn * T::NTW + j >= tiles) break;
          const double br = bp[j * 16 + part], bi = bp[j * 16 + (part ^ 1)];
          const double bre = __hiloint2double(__double2hiint(br) ^ sgn, __double2loint(br));  // (re, -im)
#pragma unroll
          for (int i = 0; i < T::MTW; ++i)
            if (wm * T::MTW + i < tiles) {
              big_mma(cr[i][j], av[i], bre);
              big_mma(ci[i][j], av[i], bi);
            }
        }
      }
      if (k0 + BIG_KP < n) {
        stage(buf ^ 1);
        __syncthreads();
      }
    }
#pragma unroll
    for (int i = 0; i < T::MTW; ++i)
#pragma unroll
      for (int j = 0; j < T::NTW; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int row = (wm * T::MTW + i) * 8 + lg, col = j0 + (wn * T::NTW + j) * 8 + 2 * lk + h;
          if (row < n && col < n) C[row + (int64_t)col * ldc] = make_double2(cr[i][j][h], ci[i][j][h]);
        }
  }
  __syncthreads();
}

template <int NT>
__device__ __forceinline__ double block_max(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double m = 0.0;
  for (int w = 0; w < NT / 32; ++w) m = fmax(m, red[w]);
  __syncthreads();
  return m;
}

// The solve of jacobi_team<float> for a whole block, bit for bit, in one pass over A per round: a thread owns the
// 2 x 2 blocks (pair i of rows, pairs j of columns) of its i and applies the column and then the row rotation to four
// elements in registers, where two passes read and wrote all of A twice with a barrier between. V lags by a round, so
// that its update (throughput of shared memory) and the next parameters (one long chain) overlap. Odd n: the absent
// index n is a row and column of A's array whose pair never rotates; what it holds meets no other row or column.
// What bounds it now: issue slots (128 FP32 operations per 2 x 2 block, half of all) and the chain of divisions and
// square roots before each round. FP64 solves, refinement included: 125 matrices of order 68 2.35 -> 1.83 ms, of order
// 80 2.89 -> 2.56, of order 96 3.17 -> 2.89.
struct JacParam {
  float c, s;
  float2 e;
};
template <int NT>
__device__ int jacobi_block(float2* A, int lda, float2* V, int n, JacParam* prm, short4* pq, int nprm, int* flag,
                            float thr, int max_sweeps) {
  const int tid = threadIdx.x;
  const int m = (n + 1) & ~1, npair = m / 2, ng = NT / npair;
  const int i = tid % npair, g0 = tid < ng * npair ? tid / npair : npair;  // spare threads: no column pairs
  // (p, q) of a row rotated by its pair of columns (eq = conj e, ep = e), or of a column by its pair of rows
  // (exchanged). Written out so that every form rounds as jacobi_team's does: which of two products is rounded before
  // the other is added is the compiler's choice there.
  auto rot = [](bool rows, const JacParam& P, float2 eq, float2 ep, float2& p, float2& q) {
    auto xy = [](float a, float b, float c, float d) { return __fmaf_rn(a, b, __fmul_rn(c, d)); };  // a b + (c d)
    const float2 sp = make_float2(xy(eq.x, q.x, -eq.y, q.y), rows ? xy(eq.y, q.x, eq.x, q.y) : xy(eq.x, q.y, eq.y, q.x));
    const float2 sq = make_float2(xy(ep.x, p.x, -ep.y, p.y), rows ? xy(ep.x, p.y, ep.y, p.x) : xy(ep.y, p.x, ep.x, p.y));
    const float2 np = make_float2(xy(P.c, p.x, -P.s, sp.x), xy(P.c, p.y, -P.s, sp.y));
    q = make_float2(xy(P.c, q.x, P.s, sq.x), xy(P.s, sq.y, P.c, q.y));
    p = np;
  };
  // V: with one block per SM the two warps that form the next parameters leave it to the others
  constexpr int VT0 = NT >= 512 ? 64 : 0;
  const int vng = (NT - VT0) / npair, iv = max(tid - VT0, 0) % npair, gv = (tid - VT0) / npair;
  const bool vwork = tid >= VT0 && gv < min(vng, npair);
  const int i2 = min(iv + npair, n - 1);
  const bool two = iv + npair < n;
  auto update_v = [&](int buf) {
    if (!vwork) return;
    const short4* xs = pq + buf * nprm;
    const JacParam* Ps = prm + buf * nprm;
    short4 x = xs[gv];
    JacParam P = Ps[gv];
#pragma unroll 1
    for (int j = gv; j < npair; j += vng) {
      const int jn = min(j + vng, npair - 1);
      const short4 xn = xs[jn];
      const JacParam Pn = Ps[jn];
      if (x.z) {
        const int vp = x.x * n, vq = x.y * n;
        const float2 ec = make_float2(P.e.x, -P.e.y);
        float2 p0 = V[vp + iv], q0 = V[vq + iv], p1 = V[vp + i2], q1 = V[vq + i2];
        rot(false, P, ec, P.e, p0, q0);
        rot(false, P, ec, P.e, p1, q1);
        V[vp + iv] = p0;
        V[vq + iv] = q0;
        if (two) {
          V[vp + i2] = p1;
          V[vq + i2] = q1;
        }
      }
      x = xn;
      P = Pn;
    }
  };
  int sweep = 0, cur = 0;
  bool lag = false;
  for (; sweep < max_sweeps; ++sweep) {
    if (tid == 0) *flag = 0;
    __syncthreads();
    for (int r = 0; r < m - 1; ++r, cur ^= 1) {
      if (tid < npair) {
        int pa = tid ? r + tid : m - 1, pb = tid ? r - tid : r;
        if (tid && pa >= m - 1) pa -= m - 1;
        if (pb < 0) pb += m - 1;
        const int p = min(pa, pb), q = max(pa, pb);
        bool rot = false;
        if (q < n) {
          const float2 b = A[p + q * lda];
          const float ab = sqrtf(__fmaf_rn(b.x, b.x, __fmul_rn(b.y, b.y)));
          if (ab > thr) {
            const float a = A[p + p * lda].x, d = A[q + q * lda].x;
            const float tau = (d - a) / (2.f * ab);
            float t;
            if (fabs(tau) > 1e15f)
              t = 0.5f / tau;
            else
              t = (tau >= 0.f ? 1.f : -1.f) / (fabs(tau) + sqrt(1.f + tau * tau));
            const float c = 1.f / sqrt(1.f + t * t);
            prm[cur * nprm + tid] = JacParam{c, t * c, make_float2(b.x / ab, b.y / ab)};
            *flag = 1;
            rot = true;
          }
        }
        pq[cur * nprm + tid] = make_short4((short)p, (short)q, rot, 0);
      }
      if (lag) update_v(cur ^ 1);
      lag = true;
      __syncthreads();
      if (g0 < npair) {
        const short4* xs = pq + cur * nprm;
        const JacParam* Ps = prm + cur * nprm;
        const short4 xi = xs[i];
        const JacParam Pi = Ps[i];
        const float2 eci = make_float2(Pi.e.x, -Pi.e.y);
        short4 x = xs[g0];
        JacParam P = Ps[g0];
#pragma unroll 1
        for (int j = g0; j < npair; j += ng) {
          const int jn = min(j + ng, npair - 1);
          const short4 xn = xs[jn];
          const JacParam Pn = Ps[jn];
          if (xi.z || x.z) {
            const int app = x.x * lda + xi.x, aqp = x.x * lda + xi.y, apq = x.y * lda + xi.x, aqq = x.y * lda + xi.y;
            float2 pp = A[app], qp = A[aqp], pq_ = A[apq], qq = A[aqq];
            if (x.z) {
              const float2 ec = make_float2(P.e.x, -P.e.y);
              rot(false, P, ec, P.e, pp, pq_);
              rot(false, P, ec, P.e, qp, qq);
            }
            if (xi.z) {
              rot(true, Pi, Pi.e, eci, pp, qp);
              rot(true, Pi, Pi.e, eci, pq_, qq);
            }
            A[app] = pp;
            A[aqp] = qp;
            A[apq] = pq_;
            A[aqq] = qq;
          }
          x = xn;
          P = Pn;
        }
      }
      __syncthreads();
    }
    const int any = *flag;
    __syncthreads();
    if (!any) break;
  }
  if (lag) update_v(cur ^ 1);
  __syncthreads();
  return sweep;
}

// Shared memory: FP32 Jacobi state (A32 NMAX x (NMAX+1), V32 NMAX x NMAX, rotation parameters),
// reused by the refinement for GEMM tiles and the cluster solve.
template <int NMAX>
struct BigSmem {
  static constexpr int A32 = NMAX * (NMAX + 1) * 8;
  static constexpr int V32 = NMAX * NMAX * 8;
  static constexpr int PRM = (NMAX / 2 + 1) * 64;
  static constexpr int JAC = A32 + V32 + PRM + 64;
  static constexpr int TILES = 4 * BIG_KP * (NMAX + 4) * 16;
  static constexpr int CLU = 32 * 33 * 16 + 32 * 32 * 16 + 17 * 64 + 64;
  static constexpr int REF = TILES > CLU ? TILES : CLU;
  static constexpr int TOTAL = (JAC > REF ? JAC : REF) + 4 * NMAX * 8 + 64 * 8;
};

template <int NMAX, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) eigh_big_kernel(BigArgs a) {
  using SM = BigSmem<NMAX>;
  extern __shared__ __align__(16) unsigned char sm[];
  // per-matrix vectors after the union region
  constexpr int U = SM::TOTAL - 4 * NMAX * 8 - 64 * 8;
  double* lam = reinterpret_cast<double*>(sm + U);           // NMAX
  int* rank = reinterpret_cast<int*>(lam + NMAX);         // NMAX
  int* perm = rank + NMAX;                                // NMAX
  int* cid = perm + NMAX;                                 // NMAX
  int* csize = cid + NMAX;                                // NMAX (cluster sizes by first sorted index)
  double* red = reinterpret_cast<double*>(sm + SM::TOTAL - 64 * 8);  // reductions, flags
  __shared__ long long s_b;
  __shared__ int s_flag;
  double2* slab = a.scratch + (int64_t)blockIdx.x * 3 * NMAX * NMAX;
  double2* V = slab;
  double2* W = slab + NMAX * NMAX;
  double2* G = slab + 2 * NMAX * NMAX;
  const int tid = threadIdx.x;

  for (;;) {
    if (tid == 0) s_b = (long long)atomicAdd(a.counter, 1ull);
    __syncthreads();
    const int64_t b = s_b;
    __syncthreads();
    if (b >= a.batch) break;
    const int n = a.nvec ? a.nvec[b] : a.n_uniform;
    if (n <= a.n_lo || (a.n_hi > 0 && n > a.n_hi)) continue;
    if (n > NMAX) {
      if (tid == 0 && a.n_lo == 0) atomicAdd(a.badsize, 1);  // varlen batches count bad orders on the host
      continue;
    }
    const int64_t aoff = a.a_off ? a.a_off[b] : b * (int64_t)n * n;
    const int64_t eoff = a.e_off ? a.e_off[b] : b * (int64_t)n;
    double2* H = a.A + aoff;

    // ---- 1. FP32 Jacobi ----
    float2* A32 = reinterpret_cast<float2*>(sm);
    float2* V32 = reinterpret_cast<float2*>(sm + SM::A32);
    int* flag = reinterpret_cast<int*>(sm + SM::A32 + SM::V32 + SM::PRM);
    const int lda = n + 1;
    double fro2 = 0.0;
    for (int e = tid; e < n * n; e += NT) {
      const int i = e % n, j = e / n;
      double2 v;
      if (i <= j) {
        v = H[i + (int64_t)j * n];
        if (i == j) v.y = 0.0;
      } else {
        const double2 u = H[j + (int64_t)i * n];
        v = make_double2(u.x, -u.y);
      }
      A32[i + j * lda] = make_float2((float)v.x, (float)v.y);
      V32[i + j * n] = make_float2(i == j ? 1.f : 0.f, 0.f);
      fro2 += v.x * v.x + v.y * v.y;
    }
    for (int o = 16; o > 0; o >>= 1) fro2 += __shfl_xor_sync(0xffffffffu, fro2, o);
    __syncthreads();
    if ((tid & 31) == 0) red[tid >> 5] = fro2;
    __syncthreads();
    double fro = 0.0;
    for (int w = 0; w < NT / 32; ++w) fro += red[w];
    fro = sqrt(fro);
    __syncthreads();
    // stop at 8 eps32 x the RMS eigenvalue: below that, FP32 rounding of (near-)degenerate pairs would
    // re-trigger 45-degree rotations forever; the FP64 refinement supplies the remaining accuracy
    JacParam* prm = reinterpret_cast<JacParam*>(sm + SM::A32 + SM::V32);
    const int sw = jacobi_block<NT>(A32, lda, V32, n, prm, reinterpret_cast<short4*>(prm + NMAX), NMAX / 2, flag,
                                    8.f * 1.1920929e-07f * (float)(fro / sqrt((double)n)), a.max_sweeps);
    if (sw >= a.max_sweeps && tid == 0) atomicAdd(a.nonconv, 1);
    for (int e = tid; e < n * n; e += NT) {
      const float2 v = V32[e];
      V[e] = make_double2(v.x, v.y);
    }
    __syncthreads();

    // ---- 2./3. FP64 refinement ----

    double2* st = reinterpret_cast<double2*>(sm);  // GEMM panels
    for (int it = 0; it <= a.refine; ++it) {
      // Loewdin: G = V^H V; W = V (3/2 I - 1/2 G); swap
      big_gemm<1, NMAX, NT>(n, V, n, V, n, G, n, st);
      for (int e = tid; e < n * n; e += NT) {
        const int i = e % n, j = e / n;
        double2 g = G[e];
        G[e] = make_double2((i == j ? 1.5 : 0.0) - 0.5 * g.x, -0.5 * g.y);
      }
      __syncthreads();
      big_gemm<0, NMAX, NT>(n, V, n, G, n, W, n, st);
      {
        double2* t = V;
        V = W;
        W = t;
      }
      // S = V^H (H V)
      big_gemm<2, NMAX, NT>(n, H, n, V, n, W, n, st);
      big_gemm<1, NMAX, NT>(n, V, n, W, n, G, n, st);
      double off = 0.0, dmax = 0.0;
      for (int e = tid; e < n * n; e += NT) {
        const int i = e % n, j = e / n;
        const double2 s = G[e];
        if (i == j) {
          lam[i] = s.x;
          dmax = fmax(dmax, fabs(s.x));
        } else {
          off = fmax(off, sqrt(s.x * s.x + s.y * s.y));
        }
      }
      __syncthreads();
      off = block_max<NT>(off, red);
      dmax = block_max<NT>(dmax, red);
      // ascending order (ties by index)
      for (int i = tid; i < n; i += NT) {
        int r = 0;
        for (int j = 0; j < n; ++j) r += (lam[j] < lam[i]) || (lam[j] == lam[i] && j < i);
        rank[i] = r;
        perm[r] = i;
      }
      __syncthreads();
      if (it == a.refine) break;  // final pass: Loewdin + Rayleigh quotients only
      // clusters: consecutive sorted gaps below tau
      // Below a relative gap of 1e-6 the first-order update is never used: the FP64 noise of S
      // (~n eps ||H||) would otherwise rotate near-degenerate vectors by noise / gap.
      const double tau = fmax(100.0 * off, 1e-6 * fmax(dmax, fro / n));
      if (tid == 0) {
        int c = 0, start = 0;
        s_flag = 0;
        cid[perm[0]] = 0;
        for (int r = 1; r < n; ++r) {
          if (lam[perm[r]] - lam[perm[r - 1]] >= tau) {
            csize[start] = r - start;
            if (r - start > 32) s_flag = 1;
            start = r;
            ++c;
          }
          cid[perm[r]] = c;
        }
        csize[start] = n - start;
        if (n - start > 32) s_flag = 1;
      }
      __syncthreads();
      if (s_flag && tid == 0) atomicAdd(a.nonconv, 1);  // oversize cluster: first-order only within it
      // M (in W): first-order Rayleigh-Ritz between clusters, identity inside clusters for now
      for (int e = tid; e < n * n; e += NT) {
        const int i = e % n, j = e / n;
        double2 m = make_double2(i == j ? 1.0 : 0.0, 0.0);
        if (i != j && cid[i] != cid[j]) {
          const double2 s = G[e];
          const double d = lam[j] - lam[i];
          m = make_double2(s.x / d, s.y / d);
        }
        W[e] = m;
      }
      __syncthreads();
      // clusters of 2..32 members: FP64 Jacobi of the block S_cc by warp 0, Q_c into M
      if (tid < 32) {
        double2* Ac = reinterpret_cast<double2*>(sm);       // 32 x 33
        double2* Qc = Ac + 32 * 33;                           // 32 x 32
        void* prmc = Qc + 32 * 32;
        int* flc = reinterpret_cast<int*>(reinterpret_cast<unsigned char*>(prmc) + 17 * 64);
        for (int r0 = 0; r0 < n;) {
          const int k = csize[r0];  // r0 is always the first sorted index of a cluster
          if (k >= 2 && k <= 32) {
            for (int e = tid; e < k * k; e += 32) {
              const int p = e % k, q = e / k;
              Ac[p + q * 33] = G[perm[r0 + p] + (int64_t)perm[r0 + q] * n];
              Qc[p + q * k] = make_double2(p == q ? 1.0 : 0.0, 0.0);
            }
            __syncwarp();
            jacobi_team<double, 32>(Ac, 33, Qc, k, k, true, reinterpret_cast<RotParam<double>*>(prmc), flc,
                                    2.220446049250313e-16 * fmax(dmax, 1e-300), 30);
            // M[:, c] <- M[:, c] Q_c: the cluster columns of (I + X) rotated into the cluster's eigenbasis
            for (int i = tid; i < n; i += 32) {
              double2 row[32];
              for (int p = 0; p < k; ++p) row[p] = W[i + (int64_t)perm[r0 + p] * n];
              for (int q = 0; q < k; ++q) {
                double2 acc = make_double2(0.0, 0.0);
                for (int p = 0; p < k; ++p) cfma(acc, row[p], Qc[p + q * k]);
                W[i + (int64_t)perm[r0 + q] * n] = acc;
              }
            }
            __syncwarp();
          }
          r0 += k;
        }
      }
      __syncthreads();
      // V <- V M
      big_gemm<0, NMAX, NT>(n, V, n, W, n, G, n, st);
      {
        double2* t = V;
        V = G;
        G = t;
      }
    }
    // outputs: eigenvalues ascending, eigenvectors over the input (column rank[i] = V[:, i])
    if (a.E)
      for (int i = tid; i < n; i += NT) a.E[eoff + rank[i]] = lam[i];
    if (a.want_v)
      for (int e = tid; e < n * n; e += NT) {
        const int row = e % n, col = e / n;
        H[row + (int64_t)rank[col] * n] = V[e];
      }
    __syncthreads();
    // restore the slab order for the next matrix
    V = slab;
    W = slab + NMAX * NMAX;
    G = slab + 2 * NMAX * NMAX;
  }
}

}  // namespace epb

namespace epb {

// One instance of the persistent solver over a (uniform or varlen) batch: orders in (n_lo, NMAX] are solved,
// the others left to the other kernels. The L2 scratch slab (3 NMAX^2 complex doubles per CTA) shares the
// workspace slot of every instance; its size is that of the largest instance, so that the slot is not
// reallocated between the launches of one varlen batch (which may be captured in a graph).
template <int NMAX, int NT, int MINB>
static int launch_big(epb_ctx* ctx, BigArgs a, int64_t batch) {
  using SM = BigSmem<NMAX>;
  static bool attr = false;
  if (!attr) {
    EPB_CUDA(cudaFuncSetAttribute(eigh_big_kernel<NMAX, NT, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  SM::TOTAL));
    attr = true;
  }
  const int64_t grid = std::min<int64_t>((int64_t)ctx->sm_count * MINB, batch);
  // largest slab of the instances below: <96, 512, 1>, <80, 256, 2>, <64, 256, 2>, <48, 256, 2>, <32, 128, 4>
  const size_t per_sm = std::max<size_t>({(size_t)3 * 96 * 96, (size_t)3 * 80 * 80 * 2, (size_t)3 * 64 * 64 * 2,
                                          (size_t)3 * 48 * 48 * 2, (size_t)3 * 32 * 32 * 4});
  const size_t slab_max = per_sm * sizeof(double2) * (size_t)ctx->sm_count;
  const size_t slab = (size_t)3 * NMAX * NMAX * sizeof(double2) * (size_t)grid;
  void* ws = nullptr;
  EPB_TRY(scratch_begin(ctx));
  EPB_TRY(ws_get(ctx, EPB_WS_EIGH_BIG, (slab > slab_max ? slab : slab_max) + 256, &ws));
  a.scratch = (double2*)((uint8_t*)ws + 256);
  a.counter = (unsigned long long*)ws;
  EPB_CUDA(cudaMemsetAsync(a.counter, 0, sizeof(unsigned long long), ctx->stream));
  prof_begin(ctx, EPB_PROF_EIGH);
  eigh_big_kernel<NMAX, NT, MINB><<<(unsigned)grid, NT, SM::TOTAL, ctx->stream>>>(a);
  prof_end(ctx);
  EPB_LAUNCH_CHECK();
  return scratch_end(ctx);
}

// Launch the order-65..96 solver over a (uniform or varlen) batch; matrices of order <= n_lo are
// left to the other kernels. Status words as in the other eigensolvers.
int eigh_big_launch(epb_ctx* ctx, double2* A, const int64_t* a_off, const int32_t* nvec, int n_uniform, int64_t batch,
                    double* E, const int64_t* e_off, bool want_v, int n_lo, int prec, int* nonconv, int* badsize) {
  if (batch == 0) return EPB_OK;
  BigArgs a{};
  a.A = A;
  a.a_off = a_off;
  a.nvec = nvec;
  a.n_uniform = n_uniform;
  a.batch = batch;
  a.E = E;
  a.e_off = e_off;
  a.want_v = want_v ? 1 : 0;
  a.max_sweeps = 20;
  a.refine = prec == EPB_PREC_FP64 ? 3 : 2;
  a.n_lo = n_lo;
  a.nonconv = nonconv;
  a.badsize = badsize;
  // orders up to 80 on a two-CTA-per-SM instance (106 KB of shared memory each), 81..96 on one 512-thread
  // CTA per SM; a uniform batch takes the one instance that covers its order
  if (nvec == nullptr) {
    if (n_uniform <= 80) return launch_big<80, 256, 2>(ctx, a, batch);
    return launch_big<BIG_NMAX, 512, 1>(ctx, a, batch);
  }
  const int st = launch_big<80, 256, 2>(ctx, a, batch);
  if (st != EPB_OK) return st;
  a.n_lo = std::max(n_lo, 80);
  return launch_big<BIG_NMAX, 512, 1>(ctx, a, batch);
}

// The same solver for the mixed-precision classes below 65 (c128 in and out): orders (n_lo, n_hi] with
// n_hi = 32, 48 or 64 on instances sized for them -- 18, 40 and 69 KB of shared memory, four 128-thread,
// two 256-thread and two 256-thread CTAs per SM. (The shared-memory FP64 Rayleigh-Ritz solver of
// epb_eigh.cu keeps H, V and S in FP64 in shared memory: 51 KB per matrix at order 32, 111 KB at 48,
// 200 KB at 64, i.e. 4, 2 and 1 matrices per SM.)
int eigh_mid_launch(epb_ctx* ctx, double2* A, const int64_t* a_off, const int32_t* nvec, int n_uniform, int64_t batch,
                    double* E, const int64_t* e_off, bool want_v, int n_lo, int n_hi, int* nonconv, int* badsize) {
  if (batch == 0) return EPB_OK;
  BigArgs a{};
  a.A = A;
  a.a_off = a_off;
  a.nvec = nvec;
  a.n_uniform = n_uniform;
  a.batch = batch;
  a.E = E;
  a.e_off = e_off;
  a.want_v = want_v ? 1 : 0;
  a.max_sweeps = 20;
  a.refine = 2;
  a.n_lo = n_lo;
  a.nonconv = nonconv;
  a.badsize = badsize;
  if (n_hi <= 32) return launch_big<32, 128, 4>(ctx, a, batch);
  if (n_hi <= 48) return launch_big<48, 256, 2>(ctx, a, batch);
  return launch_big<64, 256, 2>(ctx, a, batch);
}

// Any instance of the solver for the orders (n_lo, n_hi] of a (uniform or varlen) batch: inst = 32, 48, 64,
// 80 or 96 picks the instance (the largest order it holds), refine the FP64 refinement iterations (2 mixed, 3
// FP64). Used by the varlen size classes and their autotuner.
int eigh_l2_launch(epb_ctx* ctx, double2* A, const int64_t* a_off, const int32_t* nvec, int n_uniform, int64_t batch,
                   double* E, const int64_t* e_off, bool want_v, int n_lo, int n_hi, int inst, int refine,
                   int* nonconv, int* badsize) {
  if (batch == 0) return EPB_OK;
  BigArgs a{};
  a.A = A;
  a.a_off = a_off;
  a.nvec = nvec;
  a.n_uniform = n_uniform;
  a.batch = batch;
  a.E = E;
  a.e_off = e_off;
  a.want_v = want_v ? 1 : 0;
  a.max_sweeps = 20;
  a.refine = refine;
  a.n_lo = n_lo;
  a.n_hi = n_hi;
  a.nonconv = nonconv;
  a.badsize = badsize;
  switch (inst) {
    case 32: return launch_big<32, 128, 4>(ctx, a, batch);
    case 48: return launch_big<48, 256, 2>(ctx, a, batch);
    case 64: return launch_big<64, 256, 2>(ctx, a, batch);
    case 80: return launch_big<80, 256, 2>(ctx, a, batch);
    default: return launch_big<BIG_NMAX, 512, 1>(ctx, a, batch);
  }
}

}  // namespace epb
