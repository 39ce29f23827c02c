// FP64 gauge rotations of the vertex and the |g|^2 fold on the FP64 tensor cores:
//   ep[m, n, nu, q] = sum_{iw, jm} conj(ukq[iw, m, q]) g[iw, n, jm, q] uph[jm, nu, q],
//   g2 = |ep|^2 / (2 omega)   (ext/ElectronPhononCUDAExt.jl:146-201, src/wannier_to_bloch_batched.jl:442-455).
//
// One warp owns an 8 (m) x 8 (n) tile of one q for all modes and keeps it in registers from g to |g|^2:
//   stage 1, DMMA m8n8k4: T[m, n, jm] = sum_iw conj(ukq) g. A = ukq (rows m, k = iw), B = g (k = iw, columns n),
//     both read from global memory as the 16-byte complex values their fragments want (a warp load of g covers
//     8 columns in 64-byte pieces); real and imaginary halves make four DMMAs.
//   stage 2, FP64 FMAs: the accumulator fragment leaves T[m, n, *] of two n in one lane, so the sum over jm is
//     a small matrix-vector product per lane, without padding nm to a tile (12 modes would be 16). u_ph of the
//     warp's q sits in shared memory and is read as a broadcast.
// No block-wide barrier: warps are independent. What bounds it: the FP64 pipe (16 bands, 12 modes: 344 k FMAs per
// q), with the read of g (49 KB per q) behind it. Before, one CTA per q staged g and T in shared memory and read
// two operands for every complex FMA: 2.01 ms for 16 bands, 12 modes, 8192 q; this way 0.36 ms, and 0.27 with the
// operands staged (the FMAs alone would take 0.16). The FP64 pass ran two strided-batched ZGEMMs and a fold, 0.73 ms
// per k, now 0.29. The next mode's g is fetched during this one's DMMAs (without that 0.39 / 0.50 ms).
#include <algorithm>
#include <atomic>
#include <cmath>

#include "epb_common.cuh"

namespace epb {

struct Rot64Args {
  int64_t ldg, nq;
  const double2* ukq;   // (nw, nbkq, nq)
  const double2* uph;   // (nm, nm, nq)
  const double* omega;  // (nm, nq)
  double2* ep;          // (nbkq, nbk, nm, nq) or null
  double* g2;           // the same, or null
  double* g2sum;        // (nm): sum over m, n, q of g2 added to it, or null
  int64_t stride;       // with g2sum: g2 holds the blocks of q % stride == 0 only
  int nw, nbk, nm, nbkq;
};

constexpr int R64_WARPS = 4;

__device__ __forceinline__ double2 r64_ld(const double2* p) { return *p; }
__device__ __forceinline__ double2 r64_ld(const float2* p) {
  const float2 v = *p;
  return make_double2(v.x, v.y);
}
__device__ __forceinline__ void r64_mma(double (&c)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// KS = ceil(nw / 4) steps of four iw; NM >= nm modes in registers. SUM: the FP64 pass's fold.
template <typename G, int KS, int NM, bool SUM>
__global__ void __launch_bounds__(32 * R64_WARPS) eph_rot64_kernel(const G* __restrict__ g, Rot64Args a) {
  __shared__ double2 ups[R64_WARPS][NM * NM];
  __shared__ double iws[R64_WARPS][NM];
  __shared__ double part[SUM ? R64_WARPS : 1][NM][32];  // each lane's own sums
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, lg = lane >> 2, lk = lane & 3;
  const int nw = a.nw, nm = a.nm;
  const int mt = (a.nbkq + 7) >> 3, nt = (a.nbk + 7) >> 3;
  const int64_t items = a.nq * mt * nt;
  const int64_t mn = (int64_t)a.nbkq * a.nbk;
  if (SUM)
    for (int i = 0; i < nm; ++i) part[warp][i][lane] = 0.0;

  for (int64_t it = (int64_t)blockIdx.x * R64_WARPS + warp; it < items; it += (int64_t)gridDim.x * R64_WARPS) {
    const int64_t q = it / (mt * nt);
    const int t = (int)(it - q * (mt * nt));
    const int m = (t % mt) * 8 + lg, n0 = (t / mt) * 8;
    __syncwarp();  // the previous item's reads of ups are done
    for (int e = lane; e < nm * nm; e += 32) ups[warp][e] = a.uph[q * nm * nm + e];
    if (a.omega && lane < nm) iws[warp][lane] = 1.0 / (2.0 * a.omega[q * nm + lane]);
    // A fragments: ukq[iw = 4 s + lk, m]
    double2 u[KS];
    const double2* uq = a.ukq + (q * a.nbkq + m) * nw;
#pragma unroll
    for (int s = 0; s < KS; ++s)
      u[s] = m < a.nbkq && 4 * s + lk < nw ? uq[4 * s + lk] : make_double2(0.0, 0.0);
    // T of this lane: rows m, columns n0 + 2 lk + h
    double tr[NM][2], ti[NM][2];
    const int nb = n0 + lg;  // the column whose g this lane loads
    const G* gq = g + q * a.ldg + (int64_t)nb * nw + lk;
    const int64_t jstep = (int64_t)a.nbk * nw;
    double2 b[2][KS];  // this mode's g and the next one's
    auto fetch = [&](int jm) {
#pragma unroll
      for (int s = 0; s < KS; ++s)
        b[jm & 1][s] = nb < a.nbk && 4 * s + lk < nw ? r64_ld(gq + jm * jstep + 4 * s) : make_double2(0.0, 0.0);
    };
    fetch(0);
#pragma unroll
    for (int jm = 0; jm < NM; ++jm) {
      tr[jm][0] = tr[jm][1] = ti[jm][0] = ti[jm][1] = 0.0;
      if (jm < nm) {
        if (jm + 1 < NM && jm + 1 < nm) fetch(jm + 1);
#pragma unroll
        for (int s = 0; s < KS; ++s) {
          r64_mma(tr[jm], u[s].x, b[jm & 1][s].x);
          r64_mma(ti[jm], u[s].x, b[jm & 1][s].y);
          r64_mma(tr[jm], u[s].y, b[jm & 1][s].y);
          r64_mma(ti[jm], -u[s].y, b[jm & 1][s].x);
        }
      }
    }
    __syncwarp();
    const bool samp = SUM && a.g2 && q % a.stride == 0;
    const int64_t qo = SUM ? q / a.stride : q;
#pragma unroll 1
    for (int nu = 0; nu < nm; ++nu) {
      double er[2] = {0.0, 0.0}, ei[2] = {0.0, 0.0};
      const double2* up = ups[warp] + nu * nm;
#pragma unroll
      for (int jm = 0; jm < NM; ++jm) {
        if (jm < nm) {
          const double2 w = up[jm];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            er[h] = fma(tr[jm][h], w.x, er[h]);
            ei[h] = fma(tr[jm][h], w.y, ei[h]);
            er[h] = fma(-ti[jm][h], w.y, er[h]);
            ei[h] = fma(ti[jm][h], w.x, ei[h]);
          }
        }
      }
      double s2 = 0.0;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int n = n0 + 2 * lk + h;
        if (m >= a.nbkq || n >= a.nbk) continue;
        const int64_t o = m + (int64_t)a.nbkq * n + mn * (nu + (int64_t)nm * qo);
        if (!SUM && a.ep) a.ep[o] = make_double2(er[h], ei[h]);
        if (SUM || a.g2) {
          const double v = (er[h] * er[h] + ei[h] * ei[h]) * iws[warp][nu];
          if (SUM ? samp : true) a.g2[o] = v;
          s2 += v;
        }
      }
      if (SUM) part[warp][nu][lane] += s2;
    }
  }
  if (SUM) {
    __syncthreads();
    for (int i = warp; i < nm; i += R64_WARPS) {
      double v = 0.0;
      for (int w = 0; w < R64_WARPS; ++w) v += part[w][i][lane];
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) atomicAdd(a.g2sum + i, v);
    }
  }
}

// The same with a q's operands staged in shared memory, for q of four tiles and more: the block copies the next q's g,
// ukq, uph and omega by cp.async while its warps compute this one's tiles, modes and outputs three at a time. Fragments
// read straight from global memory, one mode ahead, waited for it (40 % of all stalls were on loads: the 160 registers
// that T takes leave twelve warps per SM to hide them), and chains of dependent operations for their own latency.
// 16 bands, 12 modes, 8192 q 0.36 -> 0.27 ms; 13 bands, 3 modes 68 -> 58 us; the FP64 pass 0.36 -> 0.29 ms per k. With
// fewer tiles (several q per stage, so that all warps have one) it was slower than the kernel above: 8 bands, 6 modes
// 35 against 33 us, 4 bands, 3 modes 25 against 14.5. Two stages, two blocks per SM: that sets the largest q.
template <typename G>
struct R64Stage {  // element offsets of a q's parts in a stage, in 16-byte units
  int g, u, p, w, total;
  __host__ __device__ R64Stage(int nw, int nbk, int nm, int nbkq) {
    g = 0;
    u = (int)(((size_t)nw * nbk * nm * sizeof(G) + 15) / 16);
    p = u + nw * nbkq;
    w = p + nm * nm;
    total = w + (nm + 1) / 2;
  }
};
constexpr int R64_STAGE_MAX = 55 * 1024 + 512;

__device__ __forceinline__ void r64_cp16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void r64_cp8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}

template <typename G, int KS, int NM, bool SUM>
__global__ void __launch_bounds__(32 * R64_WARPS, NM > 9 ? 2 : NM > 3 ? 3 : 4) eph_rot64_staged_kernel(const G* __restrict__ g, Rot64Args a) {
  constexpr int X = 3;  // outputs at a time
  extern __shared__ __align__(16) unsigned char r64_sm[];
  __shared__ double part[SUM ? R64_WARPS : 1][NM];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, lg = lane >> 2, lk = lane & 3;
  const int nw = a.nw, nm = a.nm, mt = (a.nbkq + 7) >> 3, nt = (a.nbk + 7) >> 3, tiles = mt * nt;
  const R64Stage<G> L(nw, a.nbk, nm, a.nbkq);
  double2* st = reinterpret_cast<double2*>(r64_sm);
  const int64_t mn = (int64_t)a.nbkq * a.nbk;
  const int ng = nw * a.nbk * nm, nu_ = nw * a.nbkq, np = nm * nm;
  if (SUM && tid < R64_WARPS * NM) (&part[0][0])[tid] = 0.0;
  auto copy = [&](int64_t q, int buf) {
    if (q < a.nq) {
      double2* d = st + buf * L.total;
      G* dg = reinterpret_cast<G*>(d);
      const G* sg = g + q * a.ldg;
      for (int e = tid; e < ng; e += 32 * R64_WARPS)
        if (sizeof(G) == 16)
          r64_cp16(dg + e, sg + e);
        else
          r64_cp8(dg + e, sg + e);
      for (int e = tid; e < nu_; e += 32 * R64_WARPS) r64_cp16(d + L.u + e, a.ukq + q * nu_ + e);
      for (int e = tid; e < np; e += 32 * R64_WARPS) r64_cp16(d + L.p + e, a.uph + q * np + e);
      if (a.omega && tid < nm) r64_cp8(reinterpret_cast<double*>(d + L.w) + tid, a.omega + q * nm + tid);
    }
    asm volatile("cp.async.commit_group;");
  };
  copy(blockIdx.x, 0);
  int buf = 0;
  for (int64_t q = blockIdx.x; q < a.nq; q += gridDim.x, buf ^= 1) {
    copy(q + gridDim.x, buf ^ 1);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    const double2* d = st + buf * L.total;
    const double iw = a.omega && lane < nm ? 1.0 / (2.0 * reinterpret_cast<const double*>(d + L.w)[lane]) : 0.0;
    for (int t = warp; t < tiles; t += R64_WARPS) {
      const int m = (t % mt) * 8 + lg, n0 = (t / mt) * 8, nb = n0 + lg;
      double2 u[KS];  // ukq[iw = 4 s + lk, m]
#pragma unroll
      for (int s = 0; s < KS; ++s)
        u[s] = m < a.nbkq && 4 * s + lk < nw ? d[L.u + m * nw + 4 * s + lk] : make_double2(0.0, 0.0);
      double tr[NM][2], ti[NM][2];  // T of this lane: rows m, columns n0 + 2 lk + h
      const G* gq = reinterpret_cast<const G*>(d) + nb * nw + lk;
      const int jstep = a.nbk * nw;
// three modes at a time, and three outputs at a time below (modes come in threes): one chain of dependent operations
// after the other is slower than the pipe
#pragma unroll
      for (int j0 = 0; j0 < NM; j0 += 3) {
#pragma unroll
        for (int j = j0; j < j0 + 3; ++j) tr[j][0] = tr[j][1] = ti[j][0] = ti[j][1] = 0.0;
        if (j0 < nm) {
#pragma unroll
          for (int s = 0; s < KS; ++s) {
            double2 v[3];
#pragma unroll
            for (int j = 0; j < 3; ++j)
              v[j] = nb < a.nbk && 4 * s + lk < nw && j0 + j < nm ? r64_ld(gq + (j0 + j) * jstep + 4 * s)
                                                                  : make_double2(0.0, 0.0);
#pragma unroll
            for (int j = 0; j < 3; ++j) r64_mma(tr[j0 + j], u[s].x, v[j].x);
#pragma unroll
            for (int j = 0; j < 3; ++j) r64_mma(ti[j0 + j], u[s].x, v[j].y);
#pragma unroll
            for (int j = 0; j < 3; ++j) r64_mma(tr[j0 + j], u[s].y, v[j].y);
#pragma unroll
            for (int j = 0; j < 3; ++j) r64_mma(ti[j0 + j], -u[s].y, v[j].x);
          }
        }
      }
      const bool samp = SUM && a.g2 && q % a.stride == 0;
      const int64_t qo = SUM ? q / a.stride : q;
#pragma unroll 1
      for (int nu = 0; nu < nm; nu += X) {
        double er[X][2] = {}, ei[X][2] = {};  // [output][column]
        const double2* up = d + L.p + nu * nm;
        int off[X];
#pragma unroll
        for (int x = 0; x < X; ++x) off[x] = nu + x < nm ? x * nm : 0;
#pragma unroll
        for (int jm = 0; jm < NM; ++jm) {
          if (jm < nm) {
            double2 w[X];
#pragma unroll
            for (int x = 0; x < X; ++x) w[x] = up[off[x] + jm];
#pragma unroll
            for (int x = 0; x < X; ++x)
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                er[x][h] = fma(tr[jm][h], w[x].x, er[x][h]);
                ei[x][h] = fma(tr[jm][h], w[x].y, ei[x][h]);
              }
#pragma unroll
            for (int x = 0; x < X; ++x)
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                er[x][h] = fma(-ti[jm][h], w[x].y, er[x][h]);
                ei[x][h] = fma(ti[jm][h], w[x].x, ei[x][h]);
              }
          }
        }
        double s2[X] = {};
#pragma unroll
        for (int x = 0; x < X; ++x) {
          const double wn = __shfl_sync(0xffffffffu, iw, (nu + x) & 31);
          if (nu + x >= nm) continue;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int n = n0 + 2 * lk + h;
            if (m >= a.nbkq || n >= a.nbk) continue;
            const int64_t o = m + (int64_t)a.nbkq * n + mn * (nu + x + (int64_t)nm * qo);
            if (!SUM && a.ep) a.ep[o] = make_double2(er[x][h], ei[x][h]);
            if (SUM || a.g2) {
              const double v = (er[x][h] * er[x][h] + ei[x][h] * ei[x][h]) * wn;
              if (SUM ? samp : true) a.g2[o] = v;
              s2[x] += v;
            }
          }
        }
        if (SUM) {  // eight lanes end up with the sum of one output each
          const bool hi = lane & 16, odd = lane & 8;
          double v0 = (hi ? s2[2] : s2[0]) + __shfl_xor_sync(0xffffffffu, hi ? s2[0] : s2[2], 16);
          double v1 = (hi ? 0.0 : s2[1]) + __shfl_xor_sync(0xffffffffu, hi ? s2[1] : 0.0, 16);
          double v = (odd ? v1 : v0) + __shfl_xor_sync(0xffffffffu, odd ? v0 : v1, 8);
          for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
          const int nx = nu + 2 * (lane >> 4) + ((lane >> 3) & 1);
          if ((lane & 7) == 0 && lane < 24 && nx < nm) part[warp][nx] += v;
        }
      }
    }
    __syncthreads();  // the next copy overwrites this stage
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (SUM) {
    __syncthreads();
    if (tid < nm) {
      double v = 0.0;
      for (int w = 0; w < R64_WARPS; ++w) v += part[w][tid];
      atomicAdd(a.g2sum + tid, v);
    }
  }
}

template <typename G, int KS, int NM, bool SUM>
static int r64_launch(epb_ctx* ctx, const G* g, const Rot64Args& a) {
  const int tiles = ((a.nbkq + 7) / 8) * ((a.nbk + 7) / 8);
  const size_t stage = (size_t)R64Stage<G>(a.nw, a.nbk, a.nm, a.nbkq).total * 16;
  if (tiles >= R64_WARPS && stage <= R64_STAGE_MAX) {
    static std::atomic<uint64_t> allowed{0};
    const uint64_t bit = uint64_t(1) << (ctx->device & 63);
    auto kern = eph_rot64_staged_kernel<G, KS, NM, SUM>;
    if (!(allowed.load() & bit)) {
      EPB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * R64_STAGE_MAX));
      allowed.fetch_or(bit);
    }
    int per_sm = 1;
    EPB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * R64_WARPS, 2 * stage));
    per_sm = std::max(per_sm, 1);
    const int64_t blocks = std::min<int64_t>(a.nq, (int64_t)ctx->sm_count * per_sm);
    prof_begin(ctx, EPB_PROF_ROT);
    kern<<<(unsigned)blocks, 32 * R64_WARPS, 2 * stage, ctx->stream>>>(g, a);
    prof_end(ctx);
    EPB_LAUNCH_CHECK();
    return EPB_OK;
  }
  static std::atomic<int> per_sm{0};
  int ps = per_sm.load();
  if (!ps) {
    EPB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ps, eph_rot64_kernel<G, KS, NM, SUM>, 32 * R64_WARPS, 0));
    if (ps < 1) ps = 1;
    per_sm.store(ps);
  }
  const int64_t items = a.nq * ((a.nbkq + 7) / 8) * ((a.nbk + 7) / 8);
  const int64_t blocks = std::min<int64_t>(cdiv(items, R64_WARPS), (int64_t)ctx->sm_count * ps);
  prof_begin(ctx, EPB_PROF_ROT);
  eph_rot64_kernel<G, KS, NM, SUM><<<(unsigned)blocks, 32 * R64_WARPS, 0, ctx->stream>>>(g, a);
  prof_end(ctx);
  EPB_LAUNCH_CHECK();
  return EPB_OK;
}

template <typename G, int KS, bool SUM>
static int r64_modes(epb_ctx* ctx, const G* g, const Rot64Args& a) {
  if (a.nm <= 3) return r64_launch<G, KS, 3, SUM>(ctx, g, a);
  if (a.nm <= 6) return r64_launch<G, KS, 6, SUM>(ctx, g, a);
  if (a.nm <= 9) return r64_launch<G, KS, 9, SUM>(ctx, g, a);
  if (a.nm <= 12) return r64_launch<G, KS, 12, SUM>(ctx, g, a);
  return r64_launch<G, KS, 15, SUM>(ctx, g, a);
}

template <typename G, bool SUM>
static int r64_orders(epb_ctx* ctx, const G* g, const Rot64Args& a) {
  if (a.nw <= 4) return r64_modes<G, 1, SUM>(ctx, g, a);
  if (a.nw <= 8) return r64_modes<G, 2, SUM>(ctx, g, a);
  if (a.nw <= 12) return r64_modes<G, 3, SUM>(ctx, g, a);
  if (a.nw <= 16) return r64_modes<G, 4, SUM>(ctx, g, a);
  return r64_modes<G, 8, SUM>(ctx, g, a);
}

// Whether the register kernel covers a shape: all T of a lane (4 nm doubles) and its part of u_kq stay in
// registers up to 15 modes and 32 bands. Beyond, the shared-memory kernel (or the library GEMMs of the pass).
bool rot64_covers(int nw, int nm) { return nw <= 32 && nm <= 15; }
// Whether it is also the faster one: a band slice of a few bands leaves most of an 8 x 8 tile empty, a short q list leaves
// most warps without an item, and one warp does all modes of an item in a chain; the shared-memory kernel works on live
// outputs only, a block per q. Microseconds of the three kernels (launch, rounds of blocks or warps that do not fit the
// chip at once, chains within a round, work per SM), fitted to 900 random shapes of 1 to 32 bands, 1 to 15 modes and 30
// to 9000 q that were timed both ways: 21 % off in rms for shared memory, 11 % for the others. A tenth in favour of shared
// memory leaves the fewest shapes slower than it (on 900 other shapes 17 by more than 5 %). Where the line lies (bands k+q
// x k, of bands, modes, q: shared memory / registers, us): 5 x 3 of 17, 9, 4000 22.6 / 54.4; 8 x 8 of 8, 15, 100
// 12.3 / 18.5; 6 x 6 of 6, 15, 4000 51 / 72; 16 x 2 of 16, 12, 8192 240 / 183; 16 x 16 of 16, 12, 8192 2010 / 273.
bool rot64_pays(epb_ctx* ctx, int nw, int nbk, int nbkq, int nm, int64_t nq) {
  const double sm = ctx->sm_count, q = (double)nq;
  const int tiles = ((nbkq + 7) / 8) * ((nbk + 7) / 8), slot = (nm - 1) / 3;  // which of the mode counts 3, 6, .. 15
  const double ks = nw <= 16 ? (nw + 3) / 4 : 8, mk = nm * ks, m2 = nm * nm;
  // shared memory: blocks per SM by threads and memory; elements of T per thread
  const int64_t nt = (int64_t)nbkq * nbk * nm, ng = (int64_t)nw * nbk * nm;
  const double fit = std::floor(227.0 * 1024 / (16.0 * (ng + nt + (int64_t)nw * nbkq + nm * nm) + 1024));
  const double blocks = std::min(8.0, std::max(1.0, fit)), ro = std::ceil(q / (sm * blocks)), et = std::ceil(nt / 256.0);
  const double shared = 7.86 + ro * (0.0495 + et * (0.0604 * nw + 0.0048 * nm)) + 0.000141 * q / sm * nt * (nw + nm);
  double reg;
  const size_t stage = (size_t)R64Stage<double2>(nw, nbk, nm, nbkq).total * 16;
  if (tiles >= R64_WARPS && stage <= R64_STAGE_MAX) {
    const double per = std::min(nm > 9 ? 2.0 : nm > 3 ? 3.0 : 4.0, std::floor(227.0 * 1024 / (2.0 * stage + 2048)));
    const double rs = std::ceil(q / (sm * per)), e = (tiles + R64_WARPS - 1) / R64_WARPS;
    reg = 6.35 + rs * (0.527 + e * (0.0214 * mk + 0.0171 * m2)) + q / sm * (tiles * (0.00767 * mk + 0.00235 * m2) + 6.32e-6 * stage);
  } else {
    static const int per_lo[] = {6, 4, 4, 3, 2}, per_hi[] = {3, 3, 2, 2, 2};  // blocks per SM by registers
    const double rd = std::ceil(q * tiles / (sm * R64_WARPS * (nw > 16 ? per_hi : per_lo)[slot]));
    reg = 6.44 + rd * (0.447 + 0.0319 * mk + 0.0362 * m2) + q / sm * tiles * (0.00935 * mk + 0.00185 * m2);
  }
  return reg <= 0.9 * shared;
}

int eph_rot64(epb_ctx* ctx, const double2* g, int64_t ldg, int nw, int nbk, int nm, int64_t nq, const double2* ukq,
              int nbkq, const double2* uph, const double* omega, double2* ep, double* g2) {
  return r64_orders<double2, false>(ctx, g, Rot64Args{ldg, nq, ukq, uph, omega, ep, g2, nullptr, 1, nw, nbk, nm, nbkq});
}
int eph_rot64(epb_ctx* ctx, const float2* g, int64_t ldg, int nw, int nbk, int nm, int64_t nq, const double2* ukq,
              int nbkq, const double2* uph, const double* omega, double2* ep, double* g2) {
  return r64_orders<float2, false>(ctx, g, Rot64Args{ldg, nq, ukq, uph, omega, ep, g2, nullptr, 1, nw, nbk, nm, nbkq});
}
// The FP64 pass's fold of one k: adds sum_{m, n, q} g2 to g2sum[nu], writes the blocks of q % stride == 0.
int eph_rot64_sum(epb_ctx* ctx, const double2* g, int nw, int nm, int64_t nq, const double2* ukq, const double2* uph,
                  const double* omega, double* g2sum, double* sample, int64_t stride) {
  return r64_orders<double2, true>(ctx, g, Rot64Args{(int64_t)nw * nw * nm, nq, ukq, uph, omega, nullptr, sample, g2sum,
                                                     stride < 1 ? 1 : stride, nw, nw, nm, nw});
}

}  // namespace epb
