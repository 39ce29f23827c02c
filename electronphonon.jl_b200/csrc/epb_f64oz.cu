// FP64 complex GEMM on the integer tensor cores (tcgen05 kind::i8): error-free splitting into 8-bit digits.
//
// B200's FP64 pipe gives 37 TFLOP/s, its int8 tensor pipe two orders more operations. A real operand is scaled
// per row (A) or column (B) by a power of two to a 55-bit integer and written in seven balanced base-256 digits,
//   x 2^e = sum_i d_i 256^(6-i),   d_i in [-128, 127],
// each an int8 operand plane. C = sum_{i+j <= 6} 2^(8 (12-i-j)) D_i E_j: 28 int8 GEMMs whose int32 accumulators
// are exact (7 K' 2^14 < 2^31), one accumulator per i + j. The seven sums are joined in 64-bit integers and one FP64 FMA.
// What is lost, per real product and in units of the row's largest |a| times the column's largest |b|: the pairs left
// out, six products of digits of weight 2^40 against 2^108 at least, so up to 2^-51.4 and 2^-54.3 in rms; and the
// operands' own rounding, 2^-55 each. That is on the scale of the rounding of an FP64 FMA onto a sum of that size, and
// unlike it does not grow with the partial sums. Gaussian rows decaying as exp(-|R| / 1.5), error against extended
// precision, normwise, on the device: 125 R 2.8e-16 against 5.3e-16 for the FMA chain, 343 R 4.2e-16 / 8.7e-16, 729 R
// 5.8e-16 / 1.27e-15.
//
// Measured against the FP64 tensor cores at 85 % of their peak, packing included: 3072 x 125 x 8192 0.88 -> 0.34 ms
// (cuBLAS ZGEMM 0.78), x 729 1.36 ms (108 TFLOP/s of FP64 work); upper triangles of 32-band H at 98292 points, 1331 R
// 18 -> 5.1 ms.
//
// A complex product is a real one over K' = 2 K with (re, im) interleaved:
//   rows 2i / 2i+1 of A: (a_re, -a_im) / (a_im, a_re),   column j of B: (b_re, b_im).
// For Hermitian matrices only the upper triangle is formed: n^2 real rows per point instead of 2 n^2.
//
// Operand planes sit in global memory in the shared-memory image the MMA reads: per (128-row tile, 32-wide K' chunk)
// the seven planes of 32-byte rows, SWIZZLE_32B, one after the other, so that a pipeline stage is plain bulk copies.
//
// GEMM kernel, persistent, one CTA per SM, 128 x 128 tiles in two passes over K': first the digit sums 4, 5 and 6 (18
// products), then 0 to 3 (10 products, planes 0-3 only), each pass's int32 accumulators 128 columns of TMEM apiece.
//   warp 0      copies: three 64 KB stages, all planes of a chunk or, in the second pass, planes 0-3 of two
//   warp 1      MMAs, plane by plane of A, which stays in the tensor core's collector buffer for all its products
//   warps 4-19  read each accumulator out as it is done, fold it into one FP64 value per output, scale and store
// What bounds it: shared memory and the tensor core alike. An MMA of 128 x 128 x 32 is 64 clocks of arithmetic; its two
// 4 KB operands would take as long to read at 128 bytes a clock, and the 90 KB that a chunk's copies write come on top,
// hence the collector. In 128 x 64 tiles (all seven sums at once) an MMA took 48 clocks for half the work, and the
// issuing thread's own instructions and waits 60. The accumulators of consecutive passes rotate through four TMEM
// buffers, so that MMAs start in a free one while the others are read out.
//
// Anything the digits cannot hold (an infinity or NaN in an operand, a column of a matrix B that is far from flat, see
// oz_pack_b_kernel) raises a device word, and so does a wait that ran out; the FP64 tensor-core kernel then does the
// product (f64_gemm_guarded), so results are those of that kernel. Without enough scratch the caller uses it in the
// first place.
#include <algorithm>
#include <atomic>
#include <climits>
#include <cmath>
#include <math_constants.h>

#include "epb_f64gemm.cuh"
#include "epb_umma.cuh"

namespace epb {

using namespace umma;

constexpr int OZ_PL = 7;                       // digits
constexpr int OZ_KC = 32;                      // K' per stage
constexpr int OZ_M = 128, OZ_N = 128;          // tile
constexpr int OZ_PLANE = OZ_M * OZ_KC;         // bytes of a plane of a tile and chunk
constexpr int OZ_AB = OZ_PL * OZ_PLANE;        // and of all planes, either operand
constexpr int OZ_BB = OZ_AB;
constexpr int OZ_HI = 4;                       // planes of the second pass (digit sums 0-3)
constexpr int OZ_HALF = 2 * OZ_HI * OZ_PLANE;  // half a pipeline stage: up to four planes of A, then of B
constexpr int OZ_STAGE = 2 * OZ_HALF;          // planes 0-3 and 4-6 of a chunk, or planes 0-3 of two chunks
constexpr int OZ_STAGES = 3;
constexpr int OZ_SMEM = OZ_STAGES * OZ_STAGE + 1024 + 256;
constexpr int OZ_BUF = 4;                      // accumulator buffers of OZ_N TMEM columns
constexpr int OZ_EPI0 = 4, OZ_EPIW = 16;       // epilogue warps
constexpr int OZ_THREADS = 32 * (OZ_EPI0 + OZ_EPIW);
constexpr int64_t OZ_RUN = 512 << 20;          // bytes of A's planes at a time (B: half)
constexpr int64_t OZ_K_MAX = 4000;             // 7 * 2 K 2^14 < 2^31

// Largest e with |x| 2^e within seven balanced digits (127.498 * 256^6) for |x| <= m.
__device__ __forceinline__ int oz_shift(double m) {
  if (!(m > 0.0)) return 0;
  int ex;
  const double f = frexp(m, &ex);  // m = f 2^ex, f in [0.5, 1)
  return (f <= 0.996 ? 55 : 54) - ex;
}
// 2^e as two factors, each a normal number for every exponent of a double.
__device__ __forceinline__ double2 oz_scale(int e) { return make_double2(ldexp(1.0, e / 2), ldexp(1.0, e - e / 2)); }
// The seven digits of x 2^e: byte b of the result, as a signed byte, is the digit of 256^b.
__device__ __forceinline__ unsigned long long oz_bytes(long long v) {
  return (unsigned long long)(v + 0x0080808080808080LL) ^ 0x0080808080808080ULL;
}

// Byte offset of 16-byte half h of row r in a plane of 32-byte rows, SWIZZLE_32B.
__device__ __forceinline__ int oz_sw(int r, int h) { return r * 32 + ((h ^ (r >> 2 & 1)) << 4); }

// Write the 16 K' digits of half h of row r: PLANE bytes between planes, most significant digit first. Two lanes with
// the halves of a row, rows in order over a warp, fill whole sectors.
template <int PLANE>
__device__ __forceinline__ void oz_store(uint8_t* tile, int r, int h, const unsigned long long (&v)[16]) {
#pragma unroll
  for (int p = 0; p < OZ_PL; ++p) {
    const int byte = 6 - p, sel = byte & 3;
    uint32_t w[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      uint32_t x[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) x[e] = byte < 4 ? (uint32_t)v[q * 4 + e] : (uint32_t)(v[q * 4 + e] >> 32);
      w[q] = __byte_perm(__byte_perm(x[0], x[1], sel | (sel + 4) << 4), __byte_perm(x[2], x[3], sel | (sel + 4) << 4), 0x5410);
    }
    *reinterpret_cast<uint4*>(tile + p * PLANE + oz_sw(r, h)) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// ---- operand A ---------------------------------------------------------------------------------
// Complex row e of A: its column offset in the operator, and its first real row (the imaginary row follows, except
// on the diagonal of a Hermitian matrix, where there is none).
struct OzRow {
  int64_t off, row;
  bool im;
};
__device__ __forceinline__ OzRow oz_row(int64_t e, int tri_n) {
  if (!tri_n) return {e, 2 * e, true};
  int j = (int)((sqrtf(8.f * (float)e + 1.f) - 1.f) * 0.5f);
  while ((int64_t)(j + 1) * (j + 2) / 2 <= e) ++j;
  while ((int64_t)j * (j + 1) / 2 > e) --j;
  const int i = (int)(e - (int64_t)j * (j + 1) / 2);
  return {i + (int64_t)j * tri_n, (int64_t)j * j + 2 * i, i < j};  // columns of (re, im) pairs, the last one real
}

// Shift of every complex row (largest of |re|, |im| over k); 8 rows x 32 k lanes per block.
__global__ void __launch_bounds__(256) oz_row_shift_kernel(const double2* __restrict__ a, int64_t ld, int64_t M, int64_t K,
                                                           int tri_n, int* __restrict__ shift, int* __restrict__ words) {
  __shared__ double red[32][9];
  const int r = threadIdx.x & 7, kl = threadIdx.x >> 3;
  const int64_t e = (int64_t)blockIdx.x * 8 + r;
  double m = 0.0;
  bool bad = false;
  if (e < M) {
    const double2* p = a + oz_row(e, tri_n).off;
#pragma unroll 4
    for (int64_t k = kl; k < K; k += 32) {
      const double2 v = p[k * ld];
      bad |= !(isfinite(v.x) && isfinite(v.y));
      m = fmax(m, fmax(fabs(v.x), fabs(v.y)));
    }
  }
  red[kl][r] = m;
  if (bad) words[0] = 1;
  __syncthreads();
  for (int o = 16; o > 0; o >>= 1) {
    if (kl < o) red[kl][r] = fmax(red[kl][r], red[kl + o][r]);
    __syncthreads();
  }
  if (kl == 0 && e < M) shift[e] = oz_shift(red[0][r]);
}

// One thread: 8 complex k of one complex row -> half a 32-wide chunk of its two real rows.
__global__ void __launch_bounds__(128) oz_pack_a_kernel(const double2* __restrict__ a, int64_t ld, int64_t M, int64_t K,
                                                        int64_t KC, int tri_n, const int* __restrict__ shift,
                                                        uint8_t* __restrict__ out) {
  const int64_t e = (int64_t)blockIdx.x * 64 + (threadIdx.x >> 1);
  if (e >= M) return;
  const int h = threadIdx.x & 1;
  const int64_t c = blockIdx.y;
  const OzRow row = oz_row(e, tri_n);
  const double2 sc = oz_scale(shift[e]);
  long long re[8], im[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int64_t k = c * 16 + h * 8 + i;
    const double2 v = k < K ? a[row.off + k * ld] : make_double2(0.0, 0.0);
    re[i] = __double2ll_rn(v.x * sc.x * sc.y);
    im[i] = __double2ll_rn(v.y * sc.x * sc.y);
  }
  unsigned long long v[16];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    v[2 * i] = oz_bytes(re[i]);
    v[2 * i + 1] = oz_bytes(-im[i]);
  }
  oz_store<OZ_PLANE>(out + ((row.row >> 7) * KC + c) * OZ_AB, (int)(row.row & 127), h, v);
  if (!row.im) return;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    v[2 * i] = oz_bytes(im[i]);
    v[2 * i + 1] = oz_bytes(re[i]);
  }
  const int64_t r1 = row.row + 1;
  oz_store<OZ_PLANE>(out + ((r1 >> 7) * KC + c) * OZ_AB, (int)(r1 & 127), h, v);
}

// ---- operand B ---------------------------------------------------------------------------------
// A phase is scaled by 2^54: |cos|, |sin| <= 1.

// Phases of 128 points (one column tile) from per-axis tables, or evaluated directly when the R list is too wide.
template <bool TABLE>
__global__ void __launch_bounds__(256) oz_pack_phase_kernel(const int4* __restrict__ rv, int64_t K, const double* __restrict__ xk,
                                                            int64_t N, int64_t KC, int lo0, int lo1, int lo2, int L0, int L1,
                                                            int L2, uint8_t* __restrict__ out, int* __restrict__ words) {
  extern __shared__ __align__(16) unsigned char oz_sm[];
  double2* tab = reinterpret_cast<double2*>(oz_sm);  // [L0 + L1 + L2][128]
  const int h = threadIdx.x & 1, j = threadIdx.x >> 1;  // half of a chunk, point
  const int64_t col = (int64_t)blockIdx.x * OZ_N + j;
  if (TABLE) {
    const int Lt = L0 + L1 + L2;
    for (int e = threadIdx.x; e < Lt * OZ_N; e += blockDim.x) {
      const int m = e / OZ_N, d = m < L0 ? 0 : m < L0 + L1 ? 1 : 2;
      const int R = d == 0 ? lo0 + m : d == 1 ? lo1 + m - L0 : lo2 + m - L0 - L1;
      const int64_t cc = (int64_t)blockIdx.x * OZ_N + e % OZ_N;
      tab[e] = cc < N ? cis2pi((double)R * xk[3 * cc + d]) : make_double2(0.0, 0.0);
    }
    __syncthreads();
  }
  const double s = 18014398509481984.0;  // 2^54
  bool bad = false;
  double2 p12 = make_double2(1.0, 0.0);  // the factors of R2 and R3, which change least often along an R list
  int y = INT_MIN, z = INT_MIN;
  for (int64_t c = blockIdx.y; c < KC; c += gridDim.y) {
    unsigned long long v[16];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int64_t k = c * 16 + h * 8 + i;
      double2 p = make_double2(0.0, 0.0);
      if (k < K && col < N) {
        const int4 r = rv[k];
        if (TABLE) {
          if (r.y != y || r.z != z) {
            y = r.y;
            z = r.z;
            p12 = cmul(tab[(y - lo1 + L0) * OZ_N + j], tab[(z - lo2 + L0 + L1) * OZ_N + j]);
          }
          p = cmul(tab[(r.x - lo0) * OZ_N + j], p12);
        } else {
          p = cis2pi(rdotx(r.x, r.y, r.z, xk[3 * col], xk[3 * col + 1], xk[3 * col + 2]));
        }
        bad |= !(isfinite(p.x) && isfinite(p.y));
      }
      v[2 * i] = oz_bytes(__double2ll_rn(p.x * s));
      v[2 * i + 1] = oz_bytes(__double2ll_rn(p.y * s));
    }
    oz_store<OZ_PLANE>(out + ((int64_t)blockIdx.x * KC + c) * OZ_BB, j, h, v);
  }
  if (bad) words[0] = 1;
}

// Columns of a K x N matrix: one warp per column finds its shift and packs it. Digits hold every entry to the same
// absolute step, so a column must be as flat as a phase, every entry at least half the largest: then
// sum |a_k| |b_k| >= max |a| max |b| / 2 whatever the row, and an error on the scale of the maxima is one on the scale of
// the terms. A graded column against a graded row could have its largest products where neither is large; it raises the
// word, as an infinity does.
__global__ void __launch_bounds__(128) oz_pack_b_kernel(const double2* __restrict__ b, int64_t ldb, int64_t K, int64_t N,
                                                        int64_t KC, double2* __restrict__ unscale, uint8_t* __restrict__ out,
                                                        int* __restrict__ words) {
  const int lane = threadIdx.x & 31;
  const int64_t col = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (col >= N) return;
  const double2* p = b + col * ldb;
  double m = 0.0, least = CUDART_INF;
  bool bad = false;
  for (int64_t k = lane; k < K; k += 32) {
    const double2 v = p[k];
    bad |= !(isfinite(v.x) && isfinite(v.y));
    const double big = fmax(fabs(v.x), fabs(v.y));
    m = fmax(m, big);
    least = fmin(least, big);
  }
  for (int o = 16; o > 0; o >>= 1) {
    m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    least = fmin(least, __shfl_xor_sync(0xffffffffu, least, o));
  }
  if (bad || least < 0.5 * m) words[0] = 1;
  const int e = oz_shift(m);
  const double2 sc = oz_scale(e);
  if (lane == 0) unscale[col] = oz_scale(-e);
  for (int64_t c2 = lane; c2 < 2 * KC; c2 += 32) {
    unsigned long long v[16];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int64_t k = c2 * 8 + i;
      const double2 z = k < K ? p[k] : make_double2(0.0, 0.0);
      v[2 * i] = oz_bytes(__double2ll_rn(z.x * sc.x * sc.y));
      v[2 * i + 1] = oz_bytes(__double2ll_rn(z.y * sc.x * sc.y));
    }
    oz_store<OZ_PLANE>(out + ((col / OZ_N) * KC + (c2 >> 1)) * OZ_BB, (int)(col % OZ_N), (int)(c2 & 1), v);
  }
}

// ---- GEMM --------------------------------------------------------------------------------------
struct OzGemmArgs {
  const uint8_t* A;
  const uint8_t* B;
  int KC;
  int64_t m_tiles, n_tiles;
  int64_t rows, cols;     // real rows, columns
  const int* a_shift;     // per complex row
  const double2* b_scale; // per column, 2^-shift as two factors, or null: a phase
  double* C;              // complex matrix as doubles
  int64_t ldc2;           // doubles between columns
  int tri_n;
  const int* outside;     // an operand is outside the digits: nothing to do
  int* err;
  long long timeout;
};

// K-major operand, 32-byte rows, SWIZZLE_32B, 8-row atoms 256 bytes apart.
__device__ __forceinline__ uint64_t smem_desc_sw32(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(256 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)6 << 61;
  return d;
}
// kind::i8: D s32 (2), A and B s8 (1), both K-major.
constexpr uint32_t OZ_IDESC =
    (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(OZ_N >> 3) << 17) | ((uint32_t)(OZ_M >> 4) << 24);

// x as a double, by the bits of 2^52 + 2^31 (the conversion instruction runs at a quarter of this).
__device__ __forceinline__ double oz_double(uint32_t x) {
  return __hiloint2double(0x43300000, (int)(x ^ 0x80000000u)) - 4503601774854144.0;
}

__global__ void __launch_bounds__(OZ_THREADS, 1) oz_gemm_kernel(OzGemmArgs a) {
  if (*a.outside) return;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + (((raw + 1023u) & ~1023u) - raw);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + OZ_STAGES * OZ_STAGE);
  uint64_t* empty = full + OZ_STAGES;
  uint64_t* tfull = empty + OZ_STAGES;
  uint64_t* bempty = tfull + 1;
  uint64_t* done = bempty + OZ_BUF;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* err = a.err;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < OZ_STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(tfull, 1);
    for (int b = 0; b < OZ_BUF; ++b) mbar_init(&bempty[b], 32 * OZ_EPIW);
    mbar_init(done, 1);
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const int64_t total = a.m_tiles * a.n_tiles;
  const int units = a.KC + (a.KC + 1) / 2;  // stages per tile: first pass one per chunk, second pass one per two

  if (warp == 0 && lane == 0) {
    // ---- copies ----
    int s = 0;
    uint32_t ph = 0, inflight = 0, inflight_ph = 0;
    bool ok = true;
    for (int64_t t = blockIdx.x; t < total && ok; t += gridDim.x) {
      const uint8_t* A = a.A + (t % a.m_tiles) * a.KC * (int64_t)OZ_AB;
      const uint8_t* B = a.B + (t / a.m_tiles) * a.KC * (int64_t)OZ_BB;
      for (int x = 0; x < units; ++x) {
        if (!mbar_wait(&empty[s], ph ^ 1u, err, a.timeout)) {
          ok = false;
          break;
        }
        uint8_t* st = smem + s * OZ_STAGE;
        constexpr uint32_t HB = OZ_HI * OZ_PLANE, LB = (OZ_PL - OZ_HI) * OZ_PLANE;
        if (x < a.KC) {
          const uint8_t *ax = A + (int64_t)x * OZ_AB, *bx = B + (int64_t)x * OZ_BB;
          mbar_arrive_expect_tx(&full[s], 2 * (HB + LB));
          bulk_g2s(st, ax, HB, &full[s]);
          bulk_g2s(st + HB, bx, HB, &full[s]);
          bulk_g2s(st + OZ_HALF, ax + HB, LB, &full[s]);
          bulk_g2s(st + OZ_HALF + HB, bx + HB, LB, &full[s]);
        } else {
          const int kc = 2 * (x - a.KC), two = kc + 1 < a.KC;
          const uint8_t *ax = A + (int64_t)kc * OZ_AB, *bx = B + (int64_t)kc * OZ_BB;
          mbar_arrive_expect_tx(&full[s], (two ? 4 : 2) * HB);
          bulk_g2s(st, ax, HB, &full[s]);
          bulk_g2s(st + HB, bx, HB, &full[s]);
          if (two) {
            bulk_g2s(st + OZ_HALF, ax + OZ_AB, HB, &full[s]);
            bulk_g2s(st + OZ_HALF + HB, bx + OZ_BB, HB, &full[s]);
          }
        }
        inflight |= 1u << s;
        inflight_ph = (inflight_ph & ~(1u << s)) | (ph << s);
        if (++s == OZ_STAGES) {
          s = 0;
          ph ^= 1u;
        }
      }
    }
    for (int q = 0; q < OZ_STAGES; ++q)  // copies that may still be landing (bounded)
      if (inflight & (1u << q)) {
        const long long t0 = clock64();
        while (!mbar_try_wait(&full[q], (inflight_ph >> q) & 1u) && clock64() - t0 < a.timeout) {
        }
      }
  } else if (warp == 1 && elect_one()) {
    // ---- MMAs. Accumulators in the order they are read out: digit sums 4, 5, 6, then 3, 2, 1, 0; the g-th of the
    // CTA sits in buffer g % 4 and starts once the one four before it has been read out. ----
    int s = 0;
    uint32_t ph = 0, acc = 0;
    bool ok = true;
    const uint64_t base = smem_desc_sw32(smem_u32(smem));
    // operand planes of a chunk: below 4 at d0, the others at d1
    auto a_at = [](uint64_t d0, uint64_t d1, int i) { return (i < OZ_HI ? d0 : d1) + (uint64_t)((i & 3) * OZ_PLANE >> 4); };
    auto b_at = [](uint64_t d0, uint64_t d1, int j) {
      return (j < OZ_HI ? d0 : d1) + (uint64_t)((OZ_HI + (j & 3)) * OZ_PLANE >> 4);
    };
    auto at = [&](uint32_t g) { return tmem + (g & (OZ_BUF - 1)) * OZ_N; };
    // first chunk of a pass, one digit sum after the other: its buffer must have been read out
    auto start = [&](int d, uint32_t g, uint64_t d0, uint64_t d1) {
      ok = ok && mbar_wait(&bempty[g & (OZ_BUF - 1)], (g / OZ_BUF & 1u) ^ 1u, err, a.timeout);
      if (!ok) return;
      tc_fence_after();
#pragma unroll
      for (int i = 0; i < OZ_PL; ++i) {
        if (i > d) break;
        mma_i8<A_DISCARD>(at(g), a_at(d0, d1, i), b_at(d0, d1, d - i), OZ_IDESC, i > 0);
      }
    };
    // later chunks, plane by plane of A, which stays in the collector buffer: digit sums 4, 5, 6 / 3, 2, 1, 0
    auto first_pass = [&](uint32_t g, uint64_t d0, uint64_t d1) {
#pragma unroll
      for (int i = 0; i < OZ_PL; ++i) {
        const int j0 = i < 4 ? 4 - i : 0, j1 = 6 - i;
#pragma unroll
        for (int j = 0; j < OZ_PL; ++j) {
          if (j < j0 || j > j1) continue;
          const uint32_t d = at(g + i + j - 4);
          if (j0 == j1)
            mma_i8<A_DISCARD>(d, a_at(d0, d1, i), b_at(d0, d1, j), OZ_IDESC, 1u);
          else if (j == j0)
            mma_i8<A_KEEP>(d, a_at(d0, d1, i), b_at(d0, d1, j), OZ_IDESC, 1u);
          else if (j < j1)
            mma_i8<A_USE>(d, a_at(d0, d1, i), b_at(d0, d1, j), OZ_IDESC, 1u);
          else
            mma_i8<A_LAST>(d, a_at(d0, d1, i), b_at(d0, d1, j), OZ_IDESC, 1u);
        }
      }
    };
    auto second_pass = [&](uint32_t g, uint64_t d0) {
#pragma unroll
      for (int i = 0; i < OZ_HI; ++i) {
#pragma unroll
        for (int j = 0; j < OZ_HI; ++j) {
          if (j > 3 - i) continue;
          const uint32_t d = at(g + 3 - i - j);
          if (i == 3)
            mma_i8<A_DISCARD>(d, a_at(d0, d0, i), b_at(d0, d0, j), OZ_IDESC, 1u);
          else if (j == 0)
            mma_i8<A_KEEP>(d, a_at(d0, d0, i), b_at(d0, d0, j), OZ_IDESC, 1u);
          else if (j < 3 - i)
            mma_i8<A_USE>(d, a_at(d0, d0, i), b_at(d0, d0, j), OZ_IDESC, 1u);
          else
            mma_i8<A_LAST>(d, a_at(d0, d0, i), b_at(d0, d0, j), OZ_IDESC, 1u);
        }
      }
    };
    for (int64_t t = blockIdx.x; t < total && ok; t += gridDim.x, acc += OZ_PL) {
      for (int x = 0; x < units && ok; ++x) {
        if (!mbar_wait(&full[s], ph, err, a.timeout)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint64_t d0 = base + (uint64_t)(s * OZ_STAGE >> 4), d1 = d0 + (uint64_t)(OZ_HALF >> 4);
        if (x == 0) {
#pragma unroll
          for (int d = 4; d < 7; ++d) start(d, acc + d - 4, d0, d1);
        } else if (x < a.KC) {
          first_pass(acc, d0, d1);
        } else {
          if (x == a.KC) {
#pragma unroll
            for (int d = 3; d >= 0; --d) start(d, acc + 6 - d, d0, d0);
          } else {
            second_pass(acc + 3, d0);
          }
          if (ok && 2 * (x - a.KC) + 1 < a.KC) second_pass(acc + 3, d1);
        }
        mma_commit(&empty[s]);
        if (x == a.KC - 1 || x == units - 1) mma_commit(tfull);  // a pass is complete
        if (++s == OZ_STAGES) {
          s = 0;
          ph ^= 1u;
        }
      }
    }
    mma_commit(done);  // every MMA issued retires before TMEM is released
    const long long t0 = clock64();
    while (!mbar_try_wait(done, 0) && clock64() - t0 < a.timeout) {
    }
  } else if (warp >= OZ_EPI0) {
    // ---- read-out: four warps per TMEM lane quarter, 32 columns each ----
    const int quarter = warp & 3, part = (warp - OZ_EPI0) >> 2;
    uint32_t acc = 0;
    for (int64_t t = blockIdx.x; t < total; t += gridDim.x, acc += OZ_PL) {
      const uint32_t tb = tmem + ((uint32_t)(quarter * 32) << 16) + part * 32;
      // Digit sums 4, 5, 6, 3, 2 join exactly in 64-bit integers (below 2^61, in units of 2^48), one wide multiply-add
      // each, so that a buffer goes back to the MMAs soon; that integer rounds once to FP64 and the last two sums add
      // to it by FMA.
      long long v[32];
      auto take = [&](uint32_t g, auto&& use) {
        const uint32_t buf = g & (OZ_BUF - 1);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t x[16];
          tmem_ld16_nowait(tb + buf * OZ_N + h * 16, x);
          tmem_wait_ld(x);
          if (h == 1) {
            tc_fence_before();
            mbar_arrive(&bempty[buf]);
          }
#pragma unroll
          for (int i = 0; i < 16; ++i) use(v[h * 16 + i], x[i]);
        }
      };
      auto join = [](long long m) { return [m](long long& o, uint32_t x) { o += (long long)(int)x * m; }; };
      auto add = [](double w) {
        return [w](long long& o, uint32_t x) { o = __double_as_longlong(fma(oz_double(x), w, __longlong_as_double(o))); };
      };
      if (!__all_sync(0xffffffffu, mbar_wait(tfull, 0, err, a.timeout))) break;  // the TMEM loads are .sync.aligned
      tc_fence_after();
      take(acc, [](long long& o, uint32_t x) { o = (long long)(int)x * (1 << 16); });
      take(acc + 1, join(1 << 8));
      take(acc + 2, join(1));
      if (!__all_sync(0xffffffffu, mbar_wait(tfull, 1, err, a.timeout))) break;
      tc_fence_after();
      take(acc + 3, join(1LL << 24));
      take(acc + 4, [](long long& o, uint32_t x) {
        o += (long long)((unsigned long long)x << 32);
        // high word signed, low word unsigned, each by the bits of a power of two
        const double lo = __hiloint2double(0x43300000, (int)(uint32_t)o) - 4503599627370496.0;
        o = __double_as_longlong(fma(oz_double((uint32_t)(o >> 32)), 4294967296.0, lo));
      });
      take(acc + 5, add(0x1p40));
      take(acc + 6, add(0x1p48));

      const int64_t r = (t % a.m_tiles) * OZ_M + quarter * 32 + lane;
      const int64_t c0 = (t / a.m_tiles) * OZ_N + part * 32;
      if (r >= a.rows) continue;
      int64_t off = r, e = r >> 1;
      if (a.tri_n) {
        int j = (int)sqrtf((float)r);
        while ((int64_t)(j + 1) * (j + 1) <= r) ++j;
        while ((int64_t)j * j > r) --j;
        const int u = (int)(r - (int64_t)j * j);  // 2 i + part
        off = 2 * ((u >> 1) + (int64_t)j * a.tri_n) + (u & 1);
        e = (int64_t)j * (j + 1) / 2 + (u >> 1);
      }
      double2 sa = oz_scale(48 - a.a_shift[e]);
      if (!a.b_scale) sa = make_double2(sa.x * 0x1p-27, sa.y * 0x1p-27);  // phases: scaled by 2^54
      double* C = a.C + off + c0 * a.ldc2;
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        if (c0 + i >= a.cols) break;
        double w = __longlong_as_double(v[i]) * sa.x;
        if (a.b_scale) {
          const double2 sb = a.b_scale[c0 + i];
          w = w * sb.x * sa.y * sb.y;
        } else {
          w *= sa.y;
        }
        C[i * a.ldc2] = w;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_dealloc(tmem, 512);
}

// ---- host --------------------------------------------------------------------------------------
// Whether the digits pay: SM clocks of both kernels. The FP64 pipe gives 64 FMAs a clock (85 % of them in the
// DMMA kernel); a 32-wide chunk of a tile takes the MMA issuer about OZ_CHUNK clocks, reading a tile out
// OZ_EPI, and the packing kernels their launches plus their traffic.
constexpr double OZ_CHUNK = 2500, OZ_EPI = 6000, OZ_LAUNCH = 60000, OZ_BYTES = 2500;
bool oz_pays(epb_ctx* ctx, const F64GemmArgs& a) {
  if (a.serial || a.K > OZ_K_MAX || a.K < 16) return false;
  const double rows = a.tri_n ? (double)a.tri_n * a.tri_n : 2.0 * (double)a.M, crows = (double)a.M;
  const double kc = (double)cdiv(2 * a.K, OZ_KC);
  const double dm = std::ceil(crows / 64) * 64 * (double)cdiv(a.N, 8) * 8 * (double)a.K * 4.0 / (ctx->sm_count * 64.0 * 0.85);
  const double tiles = std::ceil(rows / OZ_M) * (double)cdiv(a.N, OZ_N);
  const double oz = std::ceil(tiles / ctx->sm_count) * (kc * OZ_CHUNK + OZ_EPI) + OZ_LAUNCH +
                    (crows * a.K * 16 + rows * kc * 224 + (double)a.N * kc * 224) / OZ_BYTES;
  return oz < 0.9 * dm;
}

// Planes of the n columns from c0 (a whole number of tiles from the first).
static int oz_pack_b(epb_ctx* ctx, const F64GemmArgs& a, int mode, int64_t c0, int64_t n, int64_t KC, double2* scale,
                     uint8_t* out, int* words) {
  if (mode == B_MATRIX) {
    oz_pack_b_kernel<<<(unsigned)cdiv(n, 4), 128, 0, ctx->stream>>>(a.B + c0 * a.ldb, a.ldb, a.K, n, KC, scale, out, words);
  } else {
    const int64_t tiles = cdiv(n, OZ_N);
    const dim3 grid((unsigned)tiles, (unsigned)std::max<int64_t>(1, std::min<int64_t>(KC, 6 * ctx->sm_count / tiles)));
    if (mode == B_TABLE)
      oz_pack_phase_kernel<true><<<grid, 256, sizeof(double2) * OZ_N * (a.L0 + a.L1 + a.L2), ctx->stream>>>(
          a.rv, a.K, a.xk + 3 * c0, n, KC, a.lo0, a.lo1, a.lo2, a.L0, a.L1, a.L2, out, words);
    else
      oz_pack_phase_kernel<false><<<grid, 256, 0, ctx->stream>>>(a.rv, a.K, a.xk + 3 * c0, n, KC, 0, 0, 0, 0, 0, 0, out, words);
  }
  EPB_LAUNCH_CHECK();
  return EPB_OK;
}

// C = A B by digits, or EPB_ERR_UNSUPPORTED when there is no scratch for them. A is packed in runs of at most OZ_RUN
// bytes, B of half that: all planes of a g(Re, Rp) of 384000 rows and 729 R would take 8 GB of a workspace that lives as
// long as the context, where runs of whole waves of tiles take 0.5 GB (96 k of it, rotation to 4 bands included: 5.57 ms
// in one run, 5.90 ms in 21; in runs of 256 MB that are no whole waves 6.88). The B runs of several A runs are packed again
// for each, which is under a hundredth of the run's MMAs. The rows of a triangle do not split by tiles; there all of A is
// packed at once, up to two runs.
int oz_gemm(epb_ctx* ctx, const F64GemmArgs& a, int mode) {
  const int64_t rows = a.tri_n ? (int64_t)a.tri_n * a.tri_n : 2 * a.M;
  const int64_t all_mt = cdiv(rows, OZ_M), all_nt = cdiv(a.N, OZ_N), KC = cdiv(2 * a.K, OZ_KC);
  const int64_t cap = std::max<int64_t>(1, OZ_RUN / (KC * OZ_AB));
  if (a.tri_n && all_mt > 2 * cap) return EPB_ERR_UNSUPPORTED;
  int64_t mt = a.tri_n ? all_mt : std::min(all_mt, cap), nt = std::min(all_nt, std::max<int64_t>(1, cap / 2));
  // runs of whole waves of tiles
  const int64_t sm = ctx->sm_count;
  if (mt < all_mt && nt * mt > sm) mt = std::max<int64_t>(1, nt * mt / sm * sm / nt);
  if (nt < all_nt && nt * mt > sm) nt = std::max<int64_t>(1, nt * mt / sm * sm / mt);
  const size_t ab = (size_t)(mt * KC * OZ_AB), bb = (size_t)(nt * KC * OZ_BB);
  const int64_t mc = a.tri_n ? a.M : mt * (OZ_M / 2);  // complex rows per run
  const size_t sa = ((size_t)mc * 4 + 255) / 256 * 256, sb = ((size_t)(nt * OZ_N) * 16 + 255) / 256 * 256;
  void* ws = nullptr;
  EPB_TRY(scratch_begin(ctx));
  EPB_TRY(ws_try(ctx, EPB_WS_FOURIER, ab + bb + sa + sb, &ws));
  uint8_t* ap = (uint8_t*)ws;
  uint8_t* bp = ap + ab;
  int* ash = (int*)(bp + bb);
  double2* bsc = (double2*)((char*)ash + sa);
  int* words = ctx->dstat + EPB_DSTAT_OZ;  // [0] an operand is outside the digits, [1] a wait ran out
  EPB_CUDA(cudaMemsetAsync(words, 0, 2 * sizeof(int), ctx->stream));
  static std::atomic<uint64_t> allowed{0};
  const uint64_t bit = uint64_t(1) << (ctx->device & 63);
  if (!(allowed.load() & bit)) {
    EPB_CUDA(cudaFuncSetAttribute(oz_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, OZ_SMEM));
    EPB_CUDA(cudaFuncSetAttribute(oz_pack_phase_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024));
    allowed.fetch_or(bit);
  }
  for (int64_t r0 = 0; r0 < a.M; r0 += mc) {
    const int64_t m = std::min(mc, a.M - r0), mrows = a.tri_n ? rows : 2 * m;
    const double2* A = a.A + r0;
    oz_row_shift_kernel<<<(unsigned)cdiv(m, 8), 256, 0, ctx->stream>>>(A, a.lda, m, a.K, a.tri_n, ash, words);
    EPB_LAUNCH_CHECK();
    oz_pack_a_kernel<<<dim3((unsigned)cdiv(m, 64), (unsigned)KC), 128, 0, ctx->stream>>>(A, a.lda, m, a.K, KC, a.tri_n, ash, ap);
    EPB_LAUNCH_CHECK();
    for (int64_t t0 = 0; t0 < all_nt; t0 += nt) {
      const int64_t c0 = t0 * OZ_N, n = std::min(nt * OZ_N, a.N - c0), tiles = cdiv(n, OZ_N);
      if (r0 == 0 || nt < all_nt) EPB_TRY(oz_pack_b(ctx, a, mode, c0, n, KC, bsc, bp, words));
      OzGemmArgs g;
      g.A = ap;
      g.B = bp;
      g.KC = (int)KC;
      g.m_tiles = cdiv(mrows, OZ_M);
      g.n_tiles = tiles;
      g.rows = mrows;
      g.cols = n;
      g.a_shift = ash;
      g.b_scale = mode == B_MATRIX ? bsc : nullptr;
      g.C = (double*)(a.C + r0 + c0 * a.ldc);
      g.ldc2 = 2 * a.ldc;
      g.tri_n = a.tri_n;
      g.outside = words;
      g.err = words + 1;
      g.timeout = 4000000000LL;  // ~2 s
      oz_gemm_kernel<<<(unsigned)std::min<int64_t>(ctx->sm_count, g.m_tiles * tiles), OZ_THREADS, OZ_SMEM, ctx->stream>>>(g);
      EPB_LAUNCH_CHECK();
    }
  }
  EPB_TRY(f64_gemm_guarded(ctx, a, mode, words));
  return scratch_end(ctx);
}

}  // namespace epb
