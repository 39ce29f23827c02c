// FP64 complex GEMM on the FP64 tensor cores (mma.sync.m8n8k4.f64), the engine of every FP64 contraction of
// the path:
//
//   out[i, j] = sum_r op_r[i, r] * exp(2 pi i R_r . x_j)   (src/wannier/batched_fourier_core.jl:117-139)
//   C = A B                                                 (kR -> kq, src/wannier_to_bloch_batched.jl:245-273)
//
// The reference materialises the phase matrix (fourier_phase!, batched_fourier_core.jl:24-30) and calls ZGEMM.
// Here the phase never touches HBM: each CTA builds, for its BN points, the 1-D tables exp(2 pi i m x_{d,j})
// for m in [lo_d, hi_d] of each axis once, and forms every phase element of a K stage as the product of three
// table entries while staging it into shared memory.
//
// What bounds it: the FP64 pipe (a register-only DMMA loop measures 37.1 TFLOP/s on B200, the same as DFMA),
// and for few points the read of op_r. DMMA against the CUDA-core form: one m8n8k4 takes 256 FMAs from one
// 8-byte register per operand and thread, so operand reads from shared memory fall by 4x and one warp per
// scheduler keeps the pipe busy. The real K axis of an instruction runs over (re, im) of two complex k:
//   Re C += [a_re, a_im] . [b_re, -b_im],   Im C += [a_re, a_im] . [b_im, b_re],
// one A fragment for both. The instruction adds its four products one after the other with one rounding each
// (checked against fma chains on the device), so every output is the same chain of FMAs over k as the scalar
// loop `acc.x += a.x b.x; acc.x -= a.y b.y`, bit for bit: the mixed-precision pass, which rounds u_k and u_ph
// into 16-bit splits, sees the same inputs as it always did. Rows of a K slice are padded by four elements, so
// that the 16 lanes (four rows, two complex k) of a 64-bit shared-memory phase touch every bank once.
//
// Tiles: BM x BN complex outputs per CTA, K stages brought in by cp.async (ST deep). BN follows the number of
// points: a list of 16 points padded to 64 columns did four times its work. Measured against the CUDA-core kernel
// this replaced (64 x 64 tiles, operands through registers): 384000 rows x 729 R x 16 points 10.9 -> 1.29 ms
// (28 TFLOP/s), 10368 x 343 x 37 0.247 -> 0.06 ms, 1024 x 1331 x 98292 76 -> 35 ms (30 TFLOP/s), kR -> kq
// 3072 x 125 x 8192 1.99 -> 0.9 ms. With WK > 1 the warps split each stage's K slices between them and add
// their sums in a fixed order at the end, for outputs too small to fill the chip.
#include <algorithm>
#include <atomic>

#include "epb_f64gemm.cuh"

namespace epb {

__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool live) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}
// sign flip by a mask on the integer pipe (the FP64 pipe is the bound)
__device__ __forceinline__ double flip(double x, int mask) {
  return __hiloint2double(__double2hiint(x) ^ mask, __double2loint(x));
}

// Row r of the packed upper triangle -> i + j n.
__device__ __forceinline__ int64_t tri_row(int64_t r, int n) {
  int j = (int)((sqrtf(8.f * (float)r + 1.f) - 1.f) * 0.5f);
  while ((int64_t)(j + 1) * (j + 2) / 2 <= r) ++j;
  while ((int64_t)j * (j + 1) / 2 > r) --j;
  return (r - (int64_t)j * (j + 1) / 2) + (int64_t)j * n;
}

template <int BM_, int BN_, int WM_, int WN_, int WK_, int BK_, int ST_, int MINB_>
struct GemmTile {
  static constexpr int BM = BM_, BN = BN_, WM = WM_, WN = WN_, WK = WK_, BK = BK_, ST = ST_;
  static constexpr int MINB = MINB_;
  static constexpr int THREADS = 32 * WM * WN * WK;
  static constexpr int LDA = BM + 4, LDB = BN + 4;
  static constexpr int STAGE = BK * (LDA + LDB);  // double2 elements
  static constexpr int MT = BM / WM / 8, NT = BN / WN / 8;
  static constexpr int RED = (WK - 1) * BM * BN;  // cross-warp sums, over the stages after the K loop
  static size_t smem(bool phase, int64_t K, int L) {
    const size_t stages = sizeof(double2) * (size_t)std::max(ST * STAGE, RED);
    return stages + (phase ? sizeof(double2) * (size_t)L * BN + 4 * (size_t)((K + 3) / 4 * 4) : 0);
  }
};

// One BM x BN tile of the product, rows from m0, columns from n0.
template <class T, int MODE>
__device__ __forceinline__ void gemm_tile(const F64GemmArgs& a, int64_t m0, int64_t n0) {
  constexpr bool PHASE = MODE == B_TABLE;
  constexpr int BM = T::BM, BN = T::BN, BK = T::BK, ST = T::ST, NTH = T::THREADS;
  constexpr int LDA = T::LDA, LDB = T::LDB, MT = T::MT, NT = T::NT, WK = T::WK;
  static_assert(BK % (4 * WK) == 0 && (NTH % BM == 0 || BM % NTH == 0), "tile shape");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* st = reinterpret_cast<double2*>(smem_raw);
  double2* tab = st + (ST * T::STAGE > T::RED ? ST * T::STAGE : T::RED);  // [L0 + L1 + L2][BN]
  const int Lt = a.L0 + a.L1 + a.L2;
  uint32_t* ridx = reinterpret_cast<uint32_t*>(tab + (PHASE ? Lt * BN : 0));

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wm = warp % T::WM, wn = (warp / T::WM) % T::WN, wk = warp / (T::WM * T::WN);
  const int lg = lane >> 2, lk = lane & 3, part = lk & 1;
  const int sgn = part ? (int)0x80000000 : 0;
  const int K = (int)a.K;

  if (PHASE) {
    for (int e = tid; e < Lt * BN; e += NTH) {
      const int j = e % BN, m = e / BN;
      const int d = m < a.L0 ? 0 : m < a.L0 + a.L1 ? 1 : 2;
      const int R = d == 0 ? a.lo0 + m : d == 1 ? a.lo1 + m - a.L0 : a.lo2 + m - a.L0 - a.L1;
      const int64_t col = n0 + j;
      tab[e] = col < a.N ? cis2pi((double)R * a.xk[3 * col + d]) : make_double2(0.0, 0.0);
    }
    for (int e = tid; e < K; e += NTH) {
      const int4 r = a.rv[e];
      ridx[e] = (uint32_t)(r.x - a.lo0) | (uint32_t)(r.y - a.lo1 + a.L0) << 8 |
                (uint32_t)(r.z - a.lo2 + a.L0 + a.L1) << 16;
    }
    __syncthreads();
  }

  // A rows of this thread: fixed over the K loop
  constexpr int RPT = BM > NTH ? BM / NTH : 1;   // rows per thread and K slice
  constexpr int KSTEP = NTH > BM ? NTH / BM : 1;  // K slices loaded per pass over the threads
  const double2* arow[RPT];
  bool alive[RPT];
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const int64_t r = m0 + (tid % BM) + i * NTH;
    alive[i] = r < a.M;
    arow[i] = a.A + (alive[i] ? (a.tri_n ? tri_row(r, a.tri_n) : r) : 0);
  }
  const int ak0 = NTH > BM ? tid / BM : 0;

  auto load = [&](int kt) {
    double2* As = st + (kt % ST) * T::STAGE;
    double2* Bs = As + BK * LDA;
    const int k0 = kt * BK;
#pragma unroll
    for (int kk = 0; kk < BK; kk += KSTEP) {
      const int k = k0 + kk + ak0;
      if (KSTEP > 1 && BK % KSTEP && kk + ak0 >= BK) break;
#pragma unroll
      for (int i = 0; i < RPT; ++i) {
        const bool live = alive[i] && k < K;
        cp_async16(As + (kk + ak0) * LDA + (tid % BM) + i * NTH, arow[i] + (live ? (int64_t)k * a.lda : 0), live);
      }
    }
    if (PHASE) {
#pragma unroll
      for (int e0 = 0; e0 < BK * BN; e0 += NTH) {
        const int e = e0 + tid;
        if ((BK * BN) % NTH && e >= BK * BN) break;
        const int jj = e % BN, kk = e / BN, k = k0 + kk;
        double2 v = make_double2(0.0, 0.0);
        if (k < K) {
          const uint32_t r = ridx[k];
          v = cmul(cmul(tab[(r & 255) * BN + jj], tab[(r >> 8 & 255) * BN + jj]), tab[(r >> 16) * BN + jj]);
        }
        Bs[kk * LDB + jj] = v;
      }
    } else if (MODE == B_DIRECT) {
      for (int e = tid; e < BK * BN; e += NTH) {
        const int jj = e % BN, kk = e / BN, k = k0 + kk;
        const int64_t col = n0 + jj;
        double2 v = make_double2(0.0, 0.0);
        if (k < K && col < a.N) {
          const int4 r = a.rv[k];
          const double* x = a.xk + 3 * col;
          v = cis2pi(rdotx(r.x, r.y, r.z, x[0], x[1], x[2]));
        }
        Bs[kk * LDB + jj] = v;
      }
    } else {
#pragma unroll
      for (int e0 = 0; e0 < BK * BN; e0 += NTH) {
        const int e = e0 + tid;
        if ((BK * BN) % NTH && e >= BK * BN) break;
        const int kk = e % BK, jj = e / BK, k = k0 + kk;
        const int64_t col = n0 + jj;
        const bool live = k < K && col < a.N;
        cp_async16(Bs + kk * LDB + jj, a.B + (live ? k + col * a.ldb : 0), live);
      }
    }
  };

  double cr[MT][NT][2], ci[MT][NT][2];
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j) cr[i][j][0] = cr[i][j][1] = ci[i][j][0] = ci[i][j][1] = 0.0;

  const int KT = (K + BK - 1) / BK;
#pragma unroll
  for (int s = 0; s < ST - 1; ++s) {
    if (s < KT) load(s);
    cp_commit();
  }
  for (int kt = 0; kt < KT; ++kt) {
    cp_wait<ST - 2>();
    __syncthreads();  // stage kt is in, and every warp is done with stage kt - 1
    if (kt + ST - 1 < KT) load(kt + ST - 1);
    cp_commit();
    const double2* As = st + (kt % ST) * T::STAGE;
    const double2* Bs = As + BK * LDA;
#pragma unroll
    for (int ks = 0; ks < BK / 2 / WK; ++ks) {
      const int kc = (ks * WK + wk) * 2 + (lk >> 1);  // complex k of this lane; part: its real or imaginary half
      const double* ap = reinterpret_cast<const double*>(As + kc * LDA + wm * (BM / T::WM) + lg);
      const double* bp = reinterpret_cast<const double*>(Bs + kc * LDB + wn * (BN / T::WN) + lg);
      double av[MT], bre[NT], bim[NT];
#pragma unroll
      for (int i = 0; i < MT; ++i) av[i] = ap[i * 16 + part];
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        bre[j] = flip(bp[j * 16 + part], sgn);  // (re, -im)
        bim[j] = bp[j * 16 + (part ^ 1)];       // (im, re)
      }
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int i = 0; i < MT; ++i) {
          dmma(cr[i][j], av[i], bre[j]);
          dmma(ci[i][j], av[i], bim[j]);
        }
    }
  }

  if (WK > 1) {
    cp_wait<0>();
    __syncthreads();
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int row = wm * (BM / T::WM) + i * 8 + lg, col = wn * (BN / T::WN) + j * 8 + 2 * lk + h;
          if (wk) st[((wk - 1) * BN + col) * BM + row] = make_double2(cr[i][j][h], ci[i][j][h]);
        }
    __syncthreads();
    if (wk) return;
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int row = wm * (BM / T::WM) + i * 8 + lg, col = wn * (BN / T::WN) + j * 8 + 2 * lk + h;
#pragma unroll
          for (int w = 1; w < WK; ++w) {
            const double2 v = st[((w - 1) * BN + col) * BM + row];
            cr[i][j][h] += v.x;
            ci[i][j][h] += v.y;
          }
        }
  }
#pragma unroll
  for (int i = 0; i < MT; ++i) {
    int64_t row = m0 + wm * (BM / T::WM) + i * 8 + lg;
    if (row >= a.M) continue;
    if (a.tri_n) row = tri_row(row, a.tri_n);
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int64_t col = n0 + wn * (BN / T::WN) + j * 8 + 2 * lk + h;
        if (col < a.N) a.C[row + col * a.ldc] = make_double2(cr[i][j][h], ci[i][j][h]);
      }
  }
}

template <class T, int MODE>
__global__ void __launch_bounds__(T::THREADS, T::MINB) f64_gemm_kernel(F64GemmArgs a) {
  gemm_tile<T, MODE>(a, (int64_t)blockIdx.x * T::BM, (int64_t)blockIdx.y * T::BN);
}

// The whole product in one wave, if words say that the digit form could not hold it (epb_f64oz.cu).
template <class T, int MODE>
__global__ void __launch_bounds__(T::THREADS, T::MINB) f64_gemm_guarded_kernel(F64GemmArgs a, const int* words) {
  if (words[0] == 0 && words[1] == 0) return;
  const int64_t mt = (a.M + T::BM - 1) / T::BM, nt = (a.N + T::BN - 1) / T::BN;
  for (int64_t t = blockIdx.x; t < mt * nt; t += gridDim.x) {
    gemm_tile<T, MODE>(a, t % mt * T::BM, t / mt * T::BN);
    __syncthreads();
  }
}

template <class T, int MODE>
static int launch_tile(epb_ctx* ctx, const F64GemmArgs& a) {
  const size_t smem = T::smem(MODE == B_TABLE, a.K, a.L0 + a.L1 + a.L2);
  static std::atomic<uint64_t> allowed{0};  // devices on which the kernel may use more than 48 KB
  const uint64_t bit = uint64_t(1) << (ctx->device & 63);
  if (!(allowed.load() & bit)) {
    EPB_CUDA(cudaFuncSetAttribute(f64_gemm_kernel<T, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    allowed.fetch_or(bit);
  }
  // row tiles along x, column tiles along y in runs of at most 65535
  const int64_t mt = cdiv(a.M, T::BM), nt = cdiv(a.N, T::BN);
  for (int64_t t0 = 0; t0 < nt; t0 += 65535) {
    F64GemmArgs b = a;
    const int64_t c0 = t0 * T::BN;
    b.N = a.N - c0;
    if (MODE == B_MATRIX)
      b.B = a.B + c0 * a.ldb;
    else
      b.xk = a.xk + 3 * c0;
    b.C = a.C + c0 * a.ldc;
    const dim3 grid((unsigned)mt, (unsigned)std::min<int64_t>(65535, nt - t0));
    f64_gemm_kernel<T, MODE><<<grid, T::THREADS, smem, ctx->stream>>>(b);
    EPB_LAUNCH_CHECK();
  }
  return EPB_OK;
}

// Which tile. The cost of a choice is the number of waves of CTAs times a tile's padded work, plus a fixed
// share per tile for its tables, pipeline fill and epilogue: the padding of a narrow column list and a last
// wave that is nearly empty both show up in it. `serial` leaves out the tiles that split K between warps.
template <int MODE>
static int gemm_dispatch(epb_ctx* ctx, const F64GemmArgs& a) {
  struct Shape { int bm, bn, wk; };
  static const Shape shapes[] = {{64, 64, 1}, {64, 48, 1}, {64, 40, 1}, {64, 32, 1}, {64, 24, 1}, {64, 16, 1},
                                 {64, 8, 1},  {32, 32, 2}, {32, 16, 2}, {32, 8, 4}};
  int best = 0;
  double cost = 1e300;
  for (int i = 0; i < (int)(sizeof(shapes) / sizeof(shapes[0])); ++i) {
    if (a.serial && shapes[i].wk > 1) continue;
    const double bm = shapes[i].bm, bn = shapes[i].bn;
    const double waves = (double)cdiv(cdiv(a.M, shapes[i].bm) * cdiv(a.N, shapes[i].bn), ctx->sm_count);
    const double c = waves * ((bm * bn + 128.0) * (double)std::max<int64_t>(a.K, 8) + 16.0 * bm * bn + 40.0 * bn * (a.L0 + a.L1 + a.L2));
    if (c < cost * 0.999) cost = c, best = i;
  }
  switch (best) {
    case 0: return launch_tile<GemmTile<64, 64, 2, 4, 1, 8, 4, 2>, MODE>(ctx, a);
    case 1: return launch_tile<GemmTile<64, 48, 4, 2, 1, 8, 4, 2>, MODE>(ctx, a);
    case 2: return launch_tile<GemmTile<64, 40, 4, 1, 1, 8, 4, 3>, MODE>(ctx, a);
    case 3: return launch_tile<GemmTile<64, 32, 4, 1, 1, 8, 4, 3>, MODE>(ctx, a);
    case 4: return launch_tile<GemmTile<64, 24, 4, 1, 1, 8, 4, 3>, MODE>(ctx, a);
    case 5: return launch_tile<GemmTile<64, 16, 4, 1, 1, 8, 4, 4>, MODE>(ctx, a);
    case 6: return launch_tile<GemmTile<64, 8, 4, 1, 1, 8, 4, 4>, MODE>(ctx, a);
    case 7: return launch_tile<GemmTile<32, 32, 2, 1, 2, 8, 4, 3>, MODE>(ctx, a);
    case 8: return launch_tile<GemmTile<32, 16, 2, 1, 2, 8, 4, 3>, MODE>(ctx, a);
    default: return launch_tile<GemmTile<32, 8, 2, 1, 4, 16, 3, 2>, MODE>(ctx, a);
  }
}

template <int MODE>
static int launch_guarded(epb_ctx* ctx, const F64GemmArgs& a, const int* words) {
  using T = GemmTile<64, 64, 2, 4, 1, 8, 4, 2>;
  static std::atomic<uint64_t> allowed{0};
  const uint64_t bit = uint64_t(1) << (ctx->device & 63);
  if (!(allowed.load() & bit)) {
    EPB_CUDA(cudaFuncSetAttribute(f64_gemm_guarded_kernel<T, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    allowed.fetch_or(bit);
  }
  const size_t smem = T::smem(MODE == B_TABLE, a.K, a.L0 + a.L1 + a.L2);
  f64_gemm_guarded_kernel<T, MODE><<<(unsigned)(2 * ctx->sm_count), T::THREADS, smem, ctx->stream>>>(a, words);
  EPB_LAUNCH_CHECK();
  return EPB_OK;
}

int f64_gemm_guarded(epb_ctx* ctx, const F64GemmArgs& a, int mode, const int* words) {
  if (mode == B_MATRIX) return launch_guarded<B_MATRIX>(ctx, a, words);
  if (mode == B_TABLE) return launch_guarded<B_TABLE>(ctx, a, words);
  return launch_guarded<B_DIRECT>(ctx, a, words);
}

// The digit form where it pays and has its scratch, else the FP64 tensor cores.
static int f64_gemm(epb_ctx* ctx, const F64GemmArgs& a, int mode) {
  if (oz_pays(ctx, a)) {
    const int st = oz_gemm(ctx, a, mode);
    if (st != EPB_ERR_UNSUPPORTED) return st;
  }
  if (mode == B_MATRIX) return gemm_dispatch<B_MATRIX>(ctx, a);
  if (mode == B_TABLE) return gemm_dispatch<B_TABLE>(ctx, a);
  return gemm_dispatch<B_DIRECT>(ctx, a);
}

// C (M x N) = A (M x K) B (K x N), column-major.
int zgemm_nn(epb_ctx* ctx, const double2* A, int64_t lda, const double2* B, int64_t ldb, double2* C, int64_t ldc,
             int64_t M, int64_t N, int64_t K) {
  if (M == 0 || N == 0) return EPB_OK;
  EPB_CHECK_ARG(K <= 0x7fffff00 && cdiv(M, 32) <= 0x7fffffff, "zgemm: M=%lld, K=%lld too large", (long long)M,
                (long long)K);
  F64GemmArgs a = {};
  a.A = A;
  a.lda = lda;
  a.B = B;
  a.ldb = ldb;
  a.C = C;
  a.ldc = ldc;
  a.M = M;
  a.N = N;
  a.K = K;
  prof_begin(ctx, EPB_PROF_ZGEMM);
  const int st = f64_gemm(ctx, a, B_MATRIX);
  prof_end(ctx);
  return st;
}

// out (M x N) = op (M x nr) * phase (nr x N). tri_n > 0: M = tri_n^2, and only the rows i <= j of each matrix are
// formed (the others are left as they were).
static int fourier_rows(epb_ctx* ctx, const double2* op, int64_t ld, int64_t M, const epb_rset* rs, const double* xk,
                        int64_t N, double2* out, int64_t ldo, int tri_n, bool serial) {
  if (M == 0 || N == 0) return EPB_OK;
  F64GemmArgs a = {};
  a.A = op;
  a.lda = ld;
  a.M = tri_n ? (int64_t)tri_n * (tri_n + 1) / 2 : M;
  a.tri_n = tri_n;
  a.K = rs->nr;
  a.N = N;
  a.rv = rs->dev;
  a.xk = xk;
  a.C = out;
  a.ldc = ldo;
  a.serial = serial;
  a.lo0 = rs->lo[0];
  a.lo1 = rs->lo[1];
  a.lo2 = rs->lo[2];
  a.L0 = rs->hi[0] - rs->lo[0] + 1;
  a.L1 = rs->hi[1] - rs->lo[1] + 1;
  a.L2 = rs->hi[2] - rs->lo[2] + 1;
  EPB_CHECK_ARG(a.K <= 0x7fffff00 && cdiv(a.M, 32) <= 0x7fffffff, "fourier: ndata=%lld, nr=%lld too large",
                (long long)M, (long long)a.K);
  const bool table = a.L0 <= GT_MAX && a.L1 <= GT_MAX && a.L2 <= GT_MAX && a.K <= GK_MAX;
  prof_begin(ctx, EPB_PROF_FOURIER_F64);
  const int st = f64_gemm(ctx, a, table ? B_TABLE : B_DIRECT);
  prof_end(ctx);
  return st;
}

int fourier_f64(epb_ctx* ctx, const double2* op, int64_t ld, int64_t M, const epb_rset* rs, const double* xk, int64_t N,
                double2* out, int64_t ldo) {
  return fourier_rows(ctx, op, ld, M, rs, xk, N, out, ldo, 0, false);
}

// H(x) = sum_R H(R) exp(2 pi i R.x) for n x n matrices on their way to an eigensolver, which reads the upper
// triangles only: the strict lower triangles (and, in the digit form, the zero imaginary parts of the diagonal)
// are left as they were. serial: every output one chain of FMAs over R, for the states that the mixed modes round
// to 16 bits. Half the work of the full square: H of 15625 points at 16 bands, 729 R 0.43 -> 0.21 ms.
int fourier_f64_upper(epb_ctx* ctx, const double2* op, int64_t ld, int64_t n, const epb_rset* rs, const double* xk,
                      int64_t N, double2* out, bool serial) {
  return fourier_rows(ctx, op, ld, n * n, rs, xk, N, out, n * n, (int)n, serial);
}

}  // namespace epb
