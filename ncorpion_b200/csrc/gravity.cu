// Brute-force O(N^2) gravity with the central-mass term: the device
// replacement of vector_field's brute-force branch (src/physics.c:120-202,
// 264-266).
//
// Three arithmetic modes share the same driver:
//
// EXACT  pair terms computed by whole CTAs, a few targets each, and added in
//        ascending slot order by a warp of their own.  Every operation is the
//        reference's, in the reference's order and rounding (explicit _rn
//        intrinsics, no FMA contraction), so accelerations are bit-identical to
//        vector_field:
//          a_i = central_i ; for j ascending, j != i:
//          a_i += ((G*m_j) * (x_j - x_i)) / (D*D*D),   (the three quotients by
//          D^3 correctly rounded from one correctly rounded reciprocal)
//          D = sqrt(((dx*dx + dy*dy) + dz*dz) + (s*(R_i+R_j))^2)
//        (the reference subtracts ((G*m_j)*(x_i-x_j))/D^3 for j < i, which is
//        the same IEEE value).  CM_acc is summed sequentially in slot order.
// FP64   bodies ordered along a Morton curve, 128-body tiles, one FP64 rsqrt per
//        pair.  The whole field takes every unordered pair once (pairsym.cuh); a
//        part of it (one of several GPUs) sums its target blocks by themselves,
//        (target block, source chunk) work units.  Partial sums reduced in a
//        fixed order (deterministic).
// MIXED  same tiling; pair terms in FP32 on coordinates relative to a tile's
//        centre (one MUFU rsqrt per pair), short FP32 sums accumulated in FP64;
//        tile pairs whose bounding boxes are closer than near_theta x the larger
//        box diagonal (1.45 times as far in the sums over unordered pairs; always
//        including the target's own tile) are summed in FP64.
//        The central-mass term and G are applied in FP64.
#include <algorithm>
#include "common.cuh"
#include "bulk.cuh"
#include "pairsym.cuh"

namespace ncg {

namespace {

constexpr int T = 128;        // bodies per tile
constexpr int MXB = 64;       // threads per block, tiled kernels (2 targets each)

// ---------------------------------------------------------------- packing --

__global__ void k_pack_exact(BodyView bv, const int *__restrict__ cidx, const int *__restrict__ n_dev, double G,
                             D4 *__restrict__ src, double *__restrict__ srcR)
{
      int p = blockIdx.x * blockDim.x + threadIdx.x;
      if (p >= *n_dev) return;  // (the grid covers every slot)
      long s = (long)cidx[p] * bv.stride;
      D4 d;
      d.x = bv.x[s];
      d.y = bv.y[s];
      d.z = bv.z[s];
      d.w = __dmul_rn(G, bv.m[s]);  // G*mp, evaluated first in G*mp*DX/D3
      src[p] = d;
      srcR[p] = bv.R[s];
}

// ------------------------------------------------------------ exact kernel --

// The central body: in device memory, or by value.
struct CmArg {
      const double *dev;
      double x, y, z, m;
};

// The central mass's acceleration of a body (with J2, src/physics.c:123-160) and
// CM_acc's terms from it: c[0..2] the central ones, c[3..5] J2's share.
__device__ __forceinline__ void central_terms(const D4 &me, double cmx, double cmy, double cmz, double M,
                                              double mu, const J2Arg &j2, double mk, double (&a)[3],
                                              double (&c)[6])
{
      // src/physics.c:123-139: DX = X - XX, rk = sqrt(DX*DX + DY*DY + DZ*DZ)
      const double DX = __dsub_rn(me.x, cmx), DY = __dsub_rn(me.y, cmy), DZ = __dsub_rn(me.z, cmz);
      const double rk = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(DX, DX), __dmul_rn(DY, DY)), __dmul_rn(DZ, DZ)));
      const double r3 = __dmul_rn(__dmul_rn(rk, rk), rk);
      const double y3 = __drcp_rn(r3);  // the six quotients by r3 share RN(1/r3)
      a[0] = div_by_recip(__dmul_rn(-mu, DX), r3, y3);
      a[1] = div_by_recip(__dmul_rn(-mu, DY), r3, y3);
      a[2] = div_by_recip(__dmul_rn(-mu, DZ), r3, y3);
      c[0] = div_by_recip(__dmul_rn(me.w, DX), r3, y3);
      c[1] = div_by_recip(__dmul_rn(me.w, DY), r3, y3);
      c[2] = div_by_recip(__dmul_rn(me.w, DZ), r3, y3);
      c[3] = c[4] = c[5] = 0.;
      if (j2.on) d_j2(j2, M, mu, DX, DY, DZ, rk, r3, mk, a[0], a[1], a[2], c + 3);  // src/physics.c:149-160
}

// div_by_recip for x != 0.
__device__ __forceinline__ double div_by_recip_nz(double x, double b, double y)
{
      double q = __dmul_rn(x, y);
      double r = __fma_rn(-q, b, x);
      q = __fma_rn(r, y, q);
      r = __fma_rn(-q, b, x);
      return __fma_rn(r, y, q);
}

// Whether x may be a zero: its high word is (on the integer pipe; true as well for
// the smallest subnormals, which either division handles).
__device__ __forceinline__ bool maybe_zero(double x)
{
      return (__double2hiint(x) & 0x7fffffff) == 0;
}

// Named barriers: `threads` threads in all arrive at or wait on barrier id.
__device__ __forceinline__ void bar_sync(int id, int threads)
{
      asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int threads)
{
      asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// The exact field of XT targets a CTA.  What has an order is the additions: a
// target's terms in ascending source order, 8 cycles each.  So XP / 32 warps compute
// the pair terms, XS sources a round, into one of two buffers in shared memory, and
// one more warp adds the round before: a lane per target and component, one
// dependent addition a source.  Block 0 (with a central mass) makes CM_acc's three
// sequential sums the same way, its warps computing the bodies' terms.
// Bound by the additions' latency below ~2,000 bodies (and by the FP64 pipe they
// share with the terms: about 1,100 cycles a round with one CTA an SM), by the FP64
// pipe and issue above (49 FP64 instructions a pair of 102: pipe and issue slots 60 %
// busy).  One thread a target, computing and adding its own terms, had 128 targets a
// CTA: 4.44 ms at 20,011 bodies (157 CTAs, one an SM; now 1.85) and 20.9 ms at 65,536
// (19.2); computing and adding a round in turn 35 us at 1,000 (16.4), 65 at 2,000
// (34.8) and 412 at 8,192 (334), with CM_acc's sums in a kernel of their own behind.
constexpr int XT = 8;            // targets a CTA
constexpr int XS = 64;           // sources a round
constexpr int XROW = XS * XT + 8;  // a component's terms of a round (the pad keeps the adders off each other's banks)
constexpr int XCM = 256;         // bodies a round of block 0
constexpr int XV = 8;            // terms an adding lane loads ahead

template <bool SOFT, int XP, int OCC>
__global__ void __launch_bounds__(XP + 32, OCC) k_grav_exact(const D4 *__restrict__ src, const double *__restrict__ srcR,
                                                       const int *__restrict__ cidx, const int *__restrict__ n_dev,
                                                       CmArg cm, double G, double sp, int central, J2Arg j2,
                                                       BodyView bv, int part, int nparts,
                                                       double *__restrict__ ax, double *__restrict__ ay,
                                                       double *__restrict__ az, double *__restrict__ cm_acc)
{
      constexpr int FULL = 1, EMPTY = 3;  // barriers FULL + buffer, EMPTY + buffer
      constexpr int XTH = XP + 32;        // the threads that compute and the adding warp
      constexpr int SL = XP / XT, NS = XS / SL;  // source lanes a target, sources a thread
      __shared__ double tm[2][3 * XROW];
      const int tid = threadIdx.x, n = *n_dev;
      const double cmx = cm.dev ? cm.dev[0] : cm.x, cmy = cm.dev ? cm.dev[1] : cm.y, cmz = cm.dev ? cm.dev[2] : cm.z;
      const double M = cm.dev ? cm.dev[6] : cm.m, mu = G * M;
      const bool adder = tid >= XP;
      const int lane = tid & 31;
      if (central && blockIdx.x == 0) {
            const int f = j2.on ? 2 : 1, rounds = (n + XCM - 1) / XCM;
            double acc = 0.;
            for (int k = 0; k < rounds; k++) {
                  double *t = tm[k & 1];
                  if (!adder) {
                        const int p = k * XCM + tid;
                        double a[3], c[6] = {0., 0., 0., 0., 0., 0.};
                        if (tid < XCM && p < n)
                              central_terms(src[p], cmx, cmy, cmz, M, mu, j2,
                                            j2.on ? bv.m[(long)cidx[p] * bv.stride] : 0., a, c);
                        if (k >= 2) bar_sync(EMPTY + (k & 1), XTH);
                        for (int d = 0; d < 3 && tid < XCM; d++) {
                              t[d * f * XCM + f * tid] = c[d];
                              if (j2.on) t[d * f * XCM + f * tid + 1] = c[3 + d];
                        }
                        bar_arrive(FULL + (k & 1), XTH);
                  } else {
                        bar_sync(FULL + (k & 1), XTH);
                        if (lane < 3) {
                              const int m = f * min(XCM, n - k * XCM);
                              const volatile double *u = t + lane * f * XCM;
                              double v[XV], w[XV];
#pragma unroll
                              for (int e = 0; e < XV; e++) v[e] = u[e];
                              int q = 0;
                              for (; q + XV <= m; q += XV) {
#pragma unroll
                                    for (int e = 0; e < XV; e++) w[e] = u[min(q + XV, f * XCM - XV) + e];
#pragma unroll
                                    for (int e = 0; e < XV; e++) {
                                          acc = __dadd_rn(acc, v[e]);
                                          v[e] = w[e];
                                    }
                              }
                              for (; q < m; q++) acc = __dadd_rn(acc, u[q]);
                        }
                        __syncwarp();
                        if (k + 2 < rounds) bar_arrive(EMPTY + (k & 1), XTH);
                  }
            }
            if (adder && lane < 3) cm_acc[lane] = acc;
            return;
      }
      const int pbase = (blockIdx.x - (central ? 1 : 0)) * XT;
      if (pbase >= n) return;
      // the part's slice of the existing bodies; the others get -0.0, the identity
      // of the sum that combines the parts
      const int p_lo = (int)((long)n * part / nparts), p_hi = (int)((long)n * (part + 1) / nparts);
      if (pbase + XT <= p_lo || pbase >= p_hi) {
            if (tid < XT && pbase + tid < n) {
                  const int slot = cidx[pbase + tid];
                  ax[slot] = -0.0; ay[slot] = -0.0; az[slot] = -0.0;
            }
            return;
      }
      const int rounds = (n + XS - 1) / XS;
      if (!adder) {
            const int tt = tid % XT, sl = tid / XT;  // target; sources sl, sl + XP / XT of a round
            const int pt = pbase + tt;
            const D4 me = src[pt < n ? pt : 0];
            const double Ri = SOFT ? srcR[pt < n ? pt : 0] : 0.;
            const int kself = pbase / XS;  // the round of the targets themselves
            D4 s[NS];
            double sR[NS];
            auto fetch = [&](int k) {
#pragma unroll
                  for (int u = 0; u < NS; u++) {
                        const int j = min(k * XS + sl + SL * u, n - 1);
                        s[u] = src[j];
                        sR[u] = SOFT ? srcR[j] : 0.;
                  }
            };
            if (NS == 1) fetch(0);
            for (int k = 0; k < rounds; k++) {
                  double t[NS][3];
                  if (NS > 1) fetch(k);
#pragma unroll
                  for (int u = 0; u < NS; u++) {
                        const double dx = __dsub_rn(s[u].x, me.x);
                        const double dy = __dsub_rn(s[u].y, me.y);
                        const double dz = __dsub_rn(s[u].z, me.z);
                        double r2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
                        if (SOFT) {
                              const double sf = __dmul_rn(sp, __dadd_rn(Ri, sR[u]));
                              r2 = __dadd_rn(r2, __dmul_rn(sf, sf));
                        }
                        const double D = __dsqrt_rn(r2);
                        const double D3 = __dmul_rn(__dmul_rn(D, D), D);
                        const double y = __drcp_rn(D3);  // the three quotients by D3 share RN(1/D3)
                        const double gx = __dmul_rn(s[u].w, dx), gy = __dmul_rn(s[u].w, dy), gz = __dmul_rn(s[u].w, dz);
                        if (maybe_zero(gx) || maybe_zero(gy) || maybe_zero(gz)) {
                              t[u][0] = div_by_recip(gx, D3, y);
                              t[u][1] = div_by_recip(gy, D3, y);
                              t[u][2] = div_by_recip(gz, D3, y);
                        } else {
                              t[u][0] = div_by_recip_nz(gx, D3, y);
                              t[u][1] = div_by_recip_nz(gy, D3, y);
                              t[u][2] = div_by_recip_nz(gz, D3, y);
                        }
                  }
                  if (k == kself || k == rounds - 1) {  // -0.0 leaves every sum as it is
#pragma unroll
                        for (int u = 0; u < NS; u++) {
                              const int j = k * XS + sl + SL * u;
                              if (j >= n || j == pt) t[u][0] = t[u][1] = t[u][2] = -0.0;
                        }
                  }
                  if (NS == 1 && k + 1 < rounds) fetch(k + 1);  // (few CTAs an SM: the load's latency shows)
                  const int b = k & 1;
                  if (k >= 2) bar_sync(EMPTY + b, XTH);
#pragma unroll
                  for (int u = 0; u < NS; u++)
#pragma unroll
                        for (int d = 0; d < 3; d++) tm[b][d * XROW + (sl + SL * u) * XT + tt] = t[u][d];
                  bar_arrive(FULL + b, XTH);
            }
            return;
      }
      const int d = min(lane / XT, 2), ps = pbase + lane % XT;
      const bool live = lane < 3 * XT && ps < n;
      double acc = 0.;
      if (central && live) {
            double a[3], c[6];
            central_terms(src[ps], cmx, cmy, cmz, M, mu, j2, j2.on ? bv.m[(long)cidx[ps] * bv.stride] : 0., a, c);
            acc = d == 0 ? a[0] : d == 1 ? a[1] : a[2];
      }
      for (int k = 0; k < rounds; k++) {
            const int b = k & 1;
            bar_sync(FULL + b, XTH);
            const volatile double *u = tm[b] + d * XROW + lane % XT;
            double v[XV], w[XV];  // XV loads in flight while XV terms are added
#pragma unroll
            for (int e = 0; e < XV; e++) v[e] = u[e * XT];
#pragma unroll
            for (int q = 0; q < XS; q += XV) {
                  if (q + XV < XS)
#pragma unroll
                        for (int e = 0; e < XV; e++) w[e] = u[(q + XV + e) * XT];
#pragma unroll
                  for (int e = 0; e < XV; e++) {
                        acc = __dadd_rn(acc, v[e]);
                        v[e] = w[e];
                  }
            }
            if (k + 2 < rounds) bar_arrive(EMPTY + b, XTH);
      }
      if (live) {
            const int slot = cidx[ps];
            double *out = d == 0 ? ax : d == 1 ? ay : az;
            out[slot] = ps >= p_lo && ps < p_hi ? acc : -0.0;
      }
}

// Up to PREP_N slots in one CTA: the compaction of the existing ones, their packed
// copies (k_pack_exact) and `fill` in the empty slots' rows, instead of five
// launches of about 2 us each.
constexpr int PREP_U = 8, PREP_N = 1024 * PREP_U;

__global__ void __launch_bounds__(1024) k_prep_exact(BodyView bv, int nslots, double G, double fill,
                                                     int *__restrict__ cidx, int *__restrict__ n_dev,
                                                     D4 *__restrict__ src, double *__restrict__ srcR,
                                                     double *__restrict__ ax, double *__restrict__ ay,
                                                     double *__restrict__ az)
{
      __shared__ int cnt[PREP_U * 32];
      const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
      bool in[PREP_U];
      unsigned below[PREP_U];
#pragma unroll
      for (int u = 0; u < PREP_U; u++) {
            const int i = u * 1024 + tid;
            in[u] = i < nslots && bv.ex[i] != 0;
            const unsigned m = __ballot_sync(0xffffffffu, in[u]);
            below[u] = __popc(m & ((1u << lane) - 1u));
            if (lane == 0) cnt[u * 32 + w] = __popc(m);
            if (i < nslots && !in[u]) {
                  ax[i] = fill;
                  ay[i] = fill;
                  az[i] = fill;
            }
      }
      __syncthreads();
      if (w == 0) {  // exclusive prefix of the 256 warp counts, eight a lane
            int c[PREP_U], s = 0;
#pragma unroll
            for (int u = 0; u < PREP_U; u++) {
                  c[u] = cnt[lane * PREP_U + u];
                  s += c[u];
            }
            int incl = s;
            for (int o = 1; o < 32; o <<= 1) {
                  const int v = __shfl_up_sync(0xffffffffu, incl, o);
                  if (lane >= o) incl += v;
            }
            int run = incl - s;
#pragma unroll
            for (int u = 0; u < PREP_U; u++) {
                  cnt[lane * PREP_U + u] = run;
                  run += c[u];
            }
            if (lane == 31) *n_dev = incl;
      }
      __syncthreads();
#pragma unroll
      for (int u = 0; u < PREP_U; u++) {
            const int i = u * 1024 + tid;
            if (!in[u]) continue;
            const int p = cnt[u * 32 + w] + (int)below[u];
            const long s = (long)i * bv.stride;
            cidx[p] = i;
            src[p] = D4{bv.x[s], bv.y[s], bv.z[s], __dmul_rn(G, bv.m[s])};
            srcR[p] = bv.R[s];
      }
}

// CM_acc += G*mk*DX/r3 in slot order (src/physics.c:137-139): sequential FP64
// sums of the 3 arrays cterm[c*N .. c*N + n), in index order, from init[c] (0
// without init), one CTA (one warp) per component, so the result matches the
// reference bit for bit.  out may alias init.
__global__ void __launch_bounds__(32) k_seq_sum3(const double *__restrict__ cterm, int N,
                                                 const int *__restrict__ n_dev, const double *init, double *out)
{
      const int n = n_dev ? *n_dev : N;
      __shared__ __align__(16) double stage[CHN];
      const int w = blockIdx.x;
      const double s = warp_chain_sum(cterm + (size_t)w * N, n, init ? init[w] : 0., stage);
      if (threadIdx.x == 0) out[w] = s;
}

// ------------------------------------------------------------ tiled modes --

constexpr int RB = 256;

// bounding box (lo xyz, hi xyz) and radius range (min, max) of the existing bodies
__global__ void k_bbox_part(BodyView bv, const int *__restrict__ cidx, const int *__restrict__ n_dev,
                            double *__restrict__ part)
{
      __shared__ double sh[8][RB];
      const int n = *n_dev;
      double lo[4] = {1e300, 1e300, 1e300, 1e300}, hi[4] = {-1e300, -1e300, -1e300, -1e300};
      for (int p = blockIdx.x * RB + threadIdx.x; p < n; p += gridDim.x * RB) {
            long s = (long)cidx[p] * bv.stride;
            double v[4] = {bv.x[s], bv.y[s], bv.z[s], bv.R[s]};
            for (int d = 0; d < 4; d++) {
                  lo[d] = fmin(lo[d], v[d]);
                  hi[d] = fmax(hi[d], v[d]);
            }
      }
      for (int d = 0; d < 3; d++) {
            sh[d][threadIdx.x] = lo[d];
            sh[3 + d][threadIdx.x] = hi[d];
      }
      sh[6][threadIdx.x] = lo[3];
      sh[7][threadIdx.x] = hi[3];
      __syncthreads();
      for (int o = RB / 2; o > 0; o >>= 1) {
            if (threadIdx.x < o)
                  for (int d = 0; d < 8; d++) {
                        const bool mx = d == 3 || d == 4 || d == 5 || d == 7;
                        double a = sh[d][threadIdx.x], b = sh[d][threadIdx.x + o];
                        sh[d][threadIdx.x] = mx ? fmax(a, b) : fmin(a, b);
                  }
            __syncthreads();
      }
      if (threadIdx.x < 8) part[blockIdx.x * 8 + threadIdx.x] = sh[threadIdx.x][0];
}

// Folds the (at most 256) block partials: lo xyz, hi xyz, R min, R max in part[0..7],
// the count of existing bodies in part[8]; the last three in page-locked host memory too.
__global__ void __launch_bounds__(256) k_bbox_final(double *__restrict__ part, int nparts,
                                                    const int *__restrict__ n_dev, double *__restrict__ answer)
{
      __shared__ double sh[8][256];
      const int t = threadIdx.x;
      for (int d = 0; d < 8; d++) {
            const bool mx = d == 3 || d == 4 || d == 5 || d == 7;
            sh[d][t] = t < nparts ? part[t * 8 + d] : (mx ? -1e300 : 1e300);
      }
      __syncthreads();
      for (int o = 128; o > 0; o >>= 1) {
            if (t < o)
                  for (int d = 0; d < 8; d++) {
                        const bool mx = d == 3 || d == 4 || d == 5 || d == 7;
                        const double a = sh[d][t], b = sh[d][t + o];
                        sh[d][t] = mx ? fmax(a, b) : fmin(a, b);
                  }
            __syncthreads();
      }
      if (t < 8) part[t] = sh[t][0];
      if (t == 8) part[8] = (double)*n_dev;
      if (t >= 6 && t < 9) answer[t - 6] = t == 8 ? (double)*n_dev : sh[t][0];
}

__device__ __forceinline__ uint32_t spread3(uint32_t v)
{
      v &= 0x3ffu;
      v = (v | (v << 16)) & 0x030000ffu;
      v = (v | (v << 8)) & 0x0300f00fu;
      v = (v | (v << 4)) & 0x030c30c3u;
      v = (v | (v << 2)) & 0x09249249u;
      return v;
}

__device__ __forceinline__ uint32_t morton_key(double x, double y, double z, const double *box)
{
      const double v[3] = {x, y, z};
      uint32_t q[3];
      // one scale for all axes (the largest extent): cells stay cubic, so a
      // thin disk gives compact tiles instead of slabs
      const double ext = fmax(fmax(box[3] - box[0], box[4] - box[1]), box[5] - box[2]);
      for (int d = 0; d < 3; d++) {
            double f = ext > 0. ? (v[d] - box[d]) / ext : 0.;
            int iq = (int)(f * 1023.999);
            q[d] = (uint32_t)min(max(iq, 0), 1023);
      }
      return spread3(q[0]) | (spread3(q[1]) << 1) | (spread3(q[2]) << 2);
}

// (n: the existing bodies, from device memory; entries n .. nub - 1 get the
// largest key, so that they sort after every body)
__global__ void k_morton(BodyView bv, const int *__restrict__ cidx, const int *__restrict__ n_dev, int nub,
                         const double *__restrict__ box, uint32_t *__restrict__ keys, int *__restrict__ vals)
{
      int p = blockIdx.x * blockDim.x + threadIdx.x;
      if (p >= nub) return;
      if (p >= *n_dev) {
            keys[p] = 0xffffffffu;
            vals[p] = -1;
            return;
      }
      int slot = cidx[p];
      long s = (long)slot * bv.stride;
      keys[p] = morton_key(bv.x[s], bv.y[s], bv.z[s], box);
      vals[p] = slot;
}

// Up to 1024 U slots in one CTA: the compaction of the existing ones, `fill` in the
// empty slots' rows, the bounding box, radius range and count (box[0..8], the last three
// in `answer` too, page-locked host memory) and, with KEYS, the Morton keys, instead of
// seven launches (with CM_acc added up by the final pass: a 1,000-body call 124 -> 102 us,
// a 12,345-body one 234 -> 209).  The host waits for the answer only, while the sort and
// the tile preparation run: with the rank sort 93 -> 54 us at 1,000 bodies.  Beyond
// 4,096 slots k_morton makes the keys, on all SMs (12,345: 31 us with them here, 23 and
// 2.5 without).
template <int U, bool KEYS>
__global__ void __launch_bounds__(1024) k_prep_tiled(BodyView bv, int nslots, double fill, int *__restrict__ cidx,
                                                     int *__restrict__ n_dev, double *__restrict__ box,
                                                     double *__restrict__ answer, uint32_t *__restrict__ keys, int *__restrict__ vals,
                                                     double *__restrict__ ax, double *__restrict__ ay,
                                                     double *__restrict__ az)
{
      __shared__ int cnt[U * 32];
      __shared__ double sh[8][32];
      __shared__ double bx[8];
      __shared__ int n_s;
      const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
      unsigned in = 0u;
      unsigned char below[U];
      double v[8] = {1e300, 1e300, 1e300, -1e300, -1e300, -1e300, 1e300, -1e300};  // lo xyz, hi xyz, R min, R max
#pragma unroll
      for (int u = 0; u < U; u++) {
            const int i = u * 1024 + tid;
            const bool e = i < nslots && bv.ex[i] != 0;
            const unsigned m = __ballot_sync(0xffffffffu, e);
            below[u] = (unsigned char)__popc(m & ((1u << lane) - 1u));
            if (lane == 0) cnt[u * 32 + w] = __popc(m);
            if (e) in |= 1u << u;
      }
      // the fields V slots at a time, their loads in flight together
      constexpr int V = KEYS ? 2 : 4;  // (the keys take registers)
#pragma unroll
      for (int u0 = 0; u0 < U; u0 += V) {
            double b[V][4];
#pragma unroll
            for (int u = 0; u < V; u++)
                  if ((in >> (u0 + u)) & 1u) {
                        const long s = (long)((u0 + u) * 1024 + tid) * bv.stride;
                        b[u][0] = bv.x[s];
                        b[u][1] = bv.y[s];
                        b[u][2] = bv.z[s];
                        b[u][3] = bv.R[s];
                  }
#pragma unroll
            for (int u = 0; u < V; u++)
                  if ((in >> (u0 + u)) & 1u) {
                        for (int d = 0; d < 3; d++) {
                              v[d] = fmin(v[d], b[u][d]);
                              v[3 + d] = fmax(v[3 + d], b[u][d]);
                        }
                        v[6] = fmin(v[6], b[u][3]);
                        v[7] = fmax(v[7], b[u][3]);
                  }
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
            const int i = u * 1024 + tid;
            if (i < nslots && !((in >> u) & 1u)) {
                  ax[i] = fill;
                  ay[i] = fill;
                  az[i] = fill;
            }
      }
      auto fold = [&](int d, double a, double b) { return d < 3 || d == 6 ? fmin(a, b) : fmax(a, b); };
#pragma unroll
      for (int d = 0; d < 8; d++) {
            for (int o = 16; o > 0; o >>= 1) v[d] = fold(d, v[d], __shfl_xor_sync(0xffffffffu, v[d], o));
            if (lane == 0) sh[d][w] = v[d];
      }
      __syncthreads();
      if (w < 8) {
            double a = sh[w][lane];
            for (int o = 16; o > 0; o >>= 1) a = fold(w, a, __shfl_xor_sync(0xffffffffu, a, o));
            if (lane == 0) {
                  bx[w] = a;
                  box[w] = a;
                  if (w >= 6) answer[w - 6] = a;
            }
      } else if (w == 8) {  // exclusive prefix of the 32 U warp counts, U a lane
            int s = 0;
            for (int u = 0; u < U; u++) s += cnt[lane * U + u];
            int incl = s;
            for (int o = 1; o < 32; o <<= 1) {
                  const int x = __shfl_up_sync(0xffffffffu, incl, o);
                  if (lane >= o) incl += x;
            }
            int run = incl - s;
            for (int u = 0; u < U; u++) {
                  const int c = cnt[lane * U + u];
                  cnt[lane * U + u] = run;
                  run += c;
            }
            if (lane == 31) {
                  n_s = incl;
                  *n_dev = incl;
                  box[8] = (double)incl;
                  answer[2] = (double)incl;
            }
      }
      __syncthreads();
#pragma unroll
      for (int u = 0; u < U; u++) {
            const int i = u * 1024 + tid;
            if (!((in >> u) & 1u)) continue;
            const int p = cnt[u * 32 + w] + below[u];
            cidx[p] = i;
            if constexpr (KEYS) {
                  const long s = (long)i * bv.stride;
                  keys[p] = morton_key(bv.x[s], bv.y[s], bv.z[s], bx);
                  vals[p] = i;
            }
      }
      if constexpr (KEYS)
            for (int p = n_s + tid; p < nslots; p += 1024) {  // sorted after every body
                  keys[p] = 0xffffffffu;
                  vals[p] = -1;
            }
}

// FP32 tile-relative sources, one SoA block per tile of T bodies:
// x[T] y[T] z[T] m[T] (coordinates minus the tile's box centre).  Padding
// sources sit at 1e18 with zero mass, so their pair terms are exactly zero.
//
// One warp per tile, in one launch: the tile's bodies gathered in sorted order
// as FP64 sources (x, y, z, m) and softening * R (zero padding), the centre and
// half extents of its box, and with `mixed` the FP32 tile-relative copy.
__global__ void k_tile_prep(BodyView bv, const int *__restrict__ slots, const int *__restrict__ n_dev, int ntiles,
                            double sp, int mixed, D4 *__restrict__ s64, double *__restrict__ sR,
                            double *__restrict__ box, float *__restrict__ s32, float *__restrict__ sR32,
                            unsigned *__restrict__ count)
{
      const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
      if (warp >= ntiles) return;
      if (warp == 0 && lane == 0) *count = 0u;  // the final pass's arrivals
      const int n = *n_dev, base = warp * T;
      D4 d[T / 32];
      double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
#pragma unroll
      for (int u = 0; u < T / 32; u++) {
            const int q = base + lane + 32 * u;
            if (q < n) {
                  const long s = (long)slots[q] * bv.stride;
                  d[u] = D4{bv.x[s], bv.y[s], bv.z[s], bv.m[s]};
                  const double r = sp * bv.R[s];
                  s64[q] = d[u];
                  sR[q] = r;
                  if (mixed) sR32[q] = (float)r;
                  lo[0] = fmin(lo[0], d[u].x); hi[0] = fmax(hi[0], d[u].x);
                  lo[1] = fmin(lo[1], d[u].y); hi[1] = fmax(hi[1], d[u].y);
                  lo[2] = fmin(lo[2], d[u].z); hi[2] = fmax(hi[2], d[u].z);
            } else {
                  d[u] = D4{0., 0., 0., 0.};
                  s64[q] = d[u];
                  sR[q] = 0.;
                  if (mixed) sR32[q] = 0.f;
            }
      }
      for (int o = 16; o > 0; o >>= 1)
            for (int k = 0; k < 3; k++) {
                  lo[k] = fmin(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
                  hi[k] = fmax(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
            }
      const double c[3] = {0.5 * (lo[0] + hi[0]), 0.5 * (lo[1] + hi[1]), 0.5 * (lo[2] + hi[2])};
      if (lane < 3) {
            box[warp * 6 + lane] = c[lane];
            box[warp * 6 + 3 + lane] = 0.5 * (hi[lane] - lo[lane]);
      }
      if (!mixed) return;
      float *tile = s32 + (size_t)warp * 4 * T;
#pragma unroll
      for (int u = 0; u < T / 32; u++) {
            const int j = lane + 32 * u;
            if (base + j < n) {
                  tile[j] = (float)(d[u].x - c[0]);
                  tile[T + j] = (float)(d[u].y - c[1]);
                  tile[2 * T + j] = (float)(d[u].z - c[2]);
                  tile[3 * T + j] = (float)d[u].w;
            } else {
                  tile[j] = 1e18f;
                  tile[T + j] = 1e18f;
                  tile[2 * T + j] = 1e18f;
                  tile[3 * T + j] = 0.f;
            }
      }
}

// FP64 pair sum of one tile against this thread's two targets.
template <int SOFT>
__device__ __forceinline__ void fp64_tile(const D4 *__restrict__ tl, const double *__restrict__ tr, int cnt,
                                          int self0, int self1, const D4 &m0, const D4 &m1, double r0, double r1,
                                          double eps2, double (&a0)[3], double (&a1)[3])
{
      for (int j = 0; j < cnt; ++j) {
            const D4 s = tl[j];
            const double sj = SOFT == 2 ? tr[j] : 0.;
            {
                  double dx = s.x - m0.x, dy = s.y - m0.y, dz = s.z - m0.z;
                  double r2 = SOFT == 1 ? eps2 : 0.;
                  if (SOFT == 2) {
                        double e = r0 + sj;
                        r2 = e * e;
                  }
                  r2 = fma(dx, dx, fma(dy, dy, fma(dz, dz, r2)));
                  double ri = rsqrt(r2);
                  double w = (j == self0) ? 0. : s.w * ri * ri * ri;
                  a0[0] = fma(w, dx, a0[0]);
                  a0[1] = fma(w, dy, a0[1]);
                  a0[2] = fma(w, dz, a0[2]);
            }
            {
                  double dx = s.x - m1.x, dy = s.y - m1.y, dz = s.z - m1.z;
                  double r2 = SOFT == 1 ? eps2 : 0.;
                  if (SOFT == 2) {
                        double e = r1 + sj;
                        r2 = e * e;
                  }
                  r2 = fma(dx, dx, fma(dy, dy, fma(dz, dz, r2)));
                  double ri = rsqrt(r2);
                  double w = (j == self1) ? 0. : s.w * ri * ri * ri;
                  a1[0] = fma(w, dx, a1[0]);
                  a1[1] = fma(w, dy, a1[1]);
                  a1[2] = fma(w, dz, a1[2]);
            }
      }
}

// A run's packed FP32 partial sums into the FP64 accumulator: both halves
// converted exactly and added in FP64 (the FP64 pipe is otherwise idle in the
// far tiles, so the fold costs the FP32 pipe nothing).
__device__ __forceinline__ void fold_f64(double &a, f2 v)
{
      float lo, hi;
      f2_unpack(v, lo, hi);
      a += (double)lo + (double)hi;
}

// One source pair against one target: adds m_j dx / (r^2 + eps^2)^(3/2) of
// both sources into the packed partial sums P (SM 0: no softening; 1: uniform
// eps^2 in E; 2: eps = R_target + R_source, with RT/RS the radii).
template <int SM>
__device__ __forceinline__ void pair_term(f2 XS, f2 YS, f2 ZS, f2 MS, f2 RS, f2 XT, f2 YT, f2 ZT, f2 RT, f2 E,
                                          f2 &Px, f2 &Py, f2 &Pz)
{
      const f2 dx = f2_sub(XS, XT), dy = f2_sub(YS, YT), dz = f2_sub(ZS, ZT);
      f2 q;
      if (SM == 0) {
            q = f2_mul(dx, dx);
      } else if (SM == 1) {
            q = f2_fma(dx, dx, E);
      } else {
            const f2 e = f2_add(RS, RT);
            q = f2_fma(dx, dx, f2_mul(e, e));
      }
      q = f2_fma(dy, dy, q);
      q = f2_fma(dz, dz, q);
      const f2 i = f2_rsqrt(q);
      const f2 w = f2_mul(f2_mul(MS, i), f2_mul(i, i));
      Px = f2_fma(w, dx, Px);
      Py = f2_fma(w, dy, Py);
      Pz = f2_fma(w, dz, Pz);
}

// FP32 pair sums of one far tile (SoA x[T] y[T] z[T] m[T], radii tr[T]) for two
// targets at tile-relative positions (x0..z0), (x1..z1).  Each 128-bit shared
// load brings four sources of one component, processed as two f32x2 pairs.
// Runs of 64 sources are summed in FP32 (32 per half of each packed pair) and
// folded into the FP64 accumulators.  (Measured at N = 65,536: runs of 32 ->
// 64 -> 128 sources give 2.02 / 1.94 / 1.96 ms and max mutual errors 5.0e-7 /
// 5.9e-7 / 9.5e-7.)
template <int SM>
__device__ __forceinline__ void far_tile(const float *__restrict__ tl, const float *__restrict__ tr, float x0,
                                         float y0, float z0, float x1, float y1, float z1, float r0f, float r1f,
                                         float eps2f, double (&a0)[3], double (&a1)[3])
{
      const f2 X0 = f2_pack(x0, x0), Y0 = f2_pack(y0, y0), Z0 = f2_pack(z0, z0);
      const f2 X1 = f2_pack(x1, x1), Y1 = f2_pack(y1, y1), Z1 = f2_pack(z1, z1);
      const f2 R0 = f2_pack(r0f, r0f), R1 = f2_pack(r1f, r1f), E = f2_pack(eps2f, eps2f);
      const ulonglong2 *xs = (const ulonglong2 *)tl, *ys = (const ulonglong2 *)(tl + T);
      const ulonglong2 *zs = (const ulonglong2 *)(tl + 2 * T), *ms = (const ulonglong2 *)(tl + 3 * T);
      const ulonglong2 *rs = (const ulonglong2 *)tr;
      for (int jb = 0; jb < T / 4; jb += 16) {
            f2 p0x = 0ull, p0y = 0ull, p0z = 0ull, p1x = 0ull, p1y = 0ull, p1z = 0ull;
#pragma unroll
            for (int jj = 0; jj < 16; ++jj) {
                  const int j = jb + jj;
                  const ulonglong2 X = xs[j], Y = ys[j], Z = zs[j], M = ms[j];
                  ulonglong2 R = make_ulonglong2(0ull, 0ull);
                  if (SM == 2) R = rs[j];
                  pair_term<SM>(X.x, Y.x, Z.x, M.x, R.x, X0, Y0, Z0, R0, E, p0x, p0y, p0z);
                  pair_term<SM>(X.x, Y.x, Z.x, M.x, R.x, X1, Y1, Z1, R1, E, p1x, p1y, p1z);
                  pair_term<SM>(X.y, Y.y, Z.y, M.y, R.y, X0, Y0, Z0, R0, E, p0x, p0y, p0z);
                  pair_term<SM>(X.y, Y.y, Z.y, M.y, R.y, X1, Y1, Z1, R1, E, p1x, p1y, p1z);
            }
            fold_f64(a0[0], p0x); fold_f64(a0[1], p0y); fold_f64(a0[2], p0z);
            fold_f64(a1[0], p1x); fold_f64(a1[1], p1y); fold_f64(a1[2], p1z);
      }
}

// One CTA = one (target block of T sorted bodies, chunk of source tiles).
// MODE 0: mixed (FP32 far tiles + FP64 near tiles); MODE 1: all tiles FP64.
// SOFT 0: no softening; 1: uniform epsilon^2 (all radii equal); 2: general.
// At most 80 registers, 12 CTAs per SM: the mixed instances measured 1.5-2 %
// faster than at 96 registers and 10 CTAs per SM (the general-softening one
// spills 16 bytes and still gains), the FP64 ones 0.5 % slower than at 64.
template <int MODE, int SOFT>
__global__ void __launch_bounds__(MXB, 12) k_grav_tiled(const D4 *__restrict__ s64, const double *__restrict__ sR64,
                                                    const float *__restrict__ s32, const float *__restrict__ sR32,
                                                    const double *__restrict__ box, int n, int ntiles, int tpc,
                                                    double theta, double eps2, double *__restrict__ partial,
                                                    long npad, unsigned *__restrict__ err,
                                                    const double *__restrict__ rrange, double sp, int ib_lo)
{
      __shared__ alignas(16) float f4[2][4 * T];
      __shared__ alignas(16) float fr[2][T];
      __shared__ D4 d4[MODE == 1 ? 2 : 1][T];
      __shared__ alignas(16) double dr[MODE == 1 ? 2 : 1][T];
      __shared__ uint64_t bar[2];

      const int tid = threadIdx.x;
      const int ib = blockIdx.y + ib_lo;  // target block (the part's blocks start at ib_lo)
      const int t0 = blockIdx.x * tpc;
      const int t1 = min(ntiles, t0 + tpc);
      const int q0 = ib * T + tid, q1 = q0 + MXB;
      const bool v0 = q0 < n, v1 = q1 < n;
      const D4 m0 = s64[v0 ? q0 : 0], m1 = s64[v1 ? q1 : 0];
      const double r0 = sR64[v0 ? q0 : 0], r1 = sR64[v1 ? q1 : 0];
      const float r0f = (float)r0, r1f = (float)r1;
      const double *bi = box + ib * 6;
      // all radii equal: eps = 2 softening R for every pair (the loads of R skip)
      // (SOFT 1: the host found all radii equal and passes eps^2 = (2 sp R)^2)
      const bool uni = SOFT == 2 && rrange[0] == rrange[1];
      const double eu = 2.0 * sp * rrange[0];
      const float eps2u = SOFT == 1 ? (float)eps2 : (float)(eu * eu);

      double a0[3] = {0., 0., 0.}, a1[3] = {0., 0., 0.};

      if (tid == 0) {
            mbar_init(&bar[0], 1);
            mbar_init(&bar[1], 1);
            mbar_fence_init();
      }
      __syncthreads();
      const unsigned bytes = MODE == 1 ? T * (sizeof(D4) + (SOFT == 2 ? sizeof(double) : 0))
                                       : T * (4 * sizeof(float) + (SOFT == 2 ? sizeof(float) : 0));
      auto issue = [&](int t, int b) {
            mbar_arrive_expect(&bar[b], bytes);
            if (MODE == 1) {
                  bulk_g2s(d4[b], s64 + (size_t)t * T, T * sizeof(D4), &bar[b]);
                  if (SOFT == 2) bulk_g2s(dr[b], sR64 + (size_t)t * T, T * sizeof(double), &bar[b]);
            } else {
                  bulk_g2s(f4[b], s32 + (size_t)t * 4 * T, 4 * T * sizeof(float), &bar[b]);
                  if (SOFT == 2) bulk_g2s(fr[b], sR32 + (size_t)t * T, T * sizeof(float), &bar[b]);
            }
      };
      if (tid == 0 && t0 < t1) issue(t0, 0);

      for (int t = t0; t < t1; ++t) {
            const int k = t - t0, b = k & 1;
            if (tid == 0 && t + 1 < t1) {
                  fence_proxy_async_smem();
                  issue(t + 1, b ^ 1);
            }
            bool ok = mbar_wait_bounded(&bar[b], (k >> 1) & 1);
            if (__syncthreads_or(!ok)) {
                  if (tid == 0) {
                        atomicOr(err, ERR_TIMEOUT);
                        mbar_wait_bounded(&bar[b], (k >> 1) & 1);
                        if (t + 1 < t1) mbar_wait_bounded(&bar[b ^ 1], ((k + 1) >> 1) & 1);
                  }
                  return;
            }
            const int jbase = t * T;
            const int cnt = min(T, n - jbase);
            const int self0 = (t == ib) ? tid : -1;
            const int self1 = (t == ib) ? tid + MXB : -1;
            if (MODE == 1) {
                  fp64_tile<SOFT>(d4[b], dr[b], cnt, self0, self1, m0, m1, r0, r1, eps2, a0, a1);
            } else {
                  const double *bj = box + t * 6;
                  const bool near = (t == ib) || tiles_near(bi, bj, theta);
                  if (near) {
                        // FP64 path: stage this tile's FP64 sources (plain loads)
                        for (int j = tid; j < T; j += MXB) {
                              d4[0][j] = s64[jbase + j];
                              dr[0][j] = sR64[jbase + j];
                        }
                        __syncthreads();
                        fp64_tile<SOFT>(d4[0], dr[0], cnt, self0, self1, m0, m1, r0, r1, eps2, a0, a1);
                  } else {
                        // FP32 path, coordinates relative to the source tile's centre
                        const float x0 = (float)(m0.x - bj[0]), y0 = (float)(m0.y - bj[1]), z0 = (float)(m0.z - bj[2]);
                        const float x1 = (float)(m1.x - bj[0]), y1 = (float)(m1.y - bj[1]), z1 = (float)(m1.z - bj[2]);
                        const float *tl = f4[b];
                        const float *tr = fr[b];
                        if (SOFT == 0) far_tile<0>(tl, tr, x0, y0, z0, x1, y1, z1, r0f, r1f, 0.f, a0, a1);
                        else if (SOFT == 1 || uni) far_tile<1>(tl, tr, x0, y0, z0, x1, y1, z1, r0f, r1f, eps2u, a0, a1);
                        else far_tile<2>(tl, tr, x0, y0, z0, x1, y1, z1, r0f, r1f, 0.f, a0, a1);
                  }
            }
            __syncthreads();
      }
      const size_t base = (size_t)blockIdx.x * 3 * npad;
      if (v0) {
            partial[base + q0] = a0[0];
            partial[base + npad + q0] = a0[1];
            partial[base + 2 * npad + q0] = a0[2];
      }
      if (v1) {
            partial[base + q1] = a1[0];
            partial[base + npad + q1] = a1[1];
            partial[base + 2 * npad + q1] = a1[2];
      }
}

// Sum the chunk partials in chunk order, multiply by G, add the FP64 central
// term and scatter back to slot order; per-body CM_acc terms for the reduction.
// c: the body's CM_acc terms.
__device__ __forceinline__ void grav_finish(int q, bool own, const double (&m)[3], const D4 *__restrict__ s64,
                                            const int *__restrict__ slots, double cmx, double cmy, double cmz,
                                            double M, double G, int central, const J2Arg &j2,
                                            double *__restrict__ ax, double *__restrict__ ay, double *__restrict__ az,
                                            double (&c)[3])
{
      D4 s = s64[q];
      double a[3] = {G * m[0], G * m[1], G * m[2]};
      if (central) {
            double DX = s.x - cmx, DY = s.y - cmy, DZ = s.z - cmz;
            double rk = sqrt(DX * DX + DY * DY + DZ * DZ);
            double r3 = rk * rk * rk;
            const double mu = G * M;
            a[0] += -mu * DX / r3;
            a[1] += -mu * DY / r3;
            a[2] += -mu * DZ / r3;
            double gm = G * s.w;
            double cj[3] = {0., 0., 0.};
            if (j2.on) d_j2(j2, M, mu, DX, DY, DZ, rk, r3, s.w, a[0], a[1], a[2], cj);
            c[0] = gm * DX / r3 + cj[0];
            c[1] = gm * DY / r3 + cj[1];
            c[2] = gm * DZ / r3 + cj[2];
      }
      int slot = slots[q];
      ax[slot] = own ? a[0] : -0.0;
      ay[slot] = own ? a[1] : -0.0;
      az[slot] = own ? a[2] : -0.0;
}

__global__ void k_grav_final(const double *__restrict__ partial, int nchunks, long npad, const D4 *__restrict__ s64,
                             const int *__restrict__ slots, int n, double cmx, double cmy, double cmz, double M,
                             double G, int central, J2Arg j2, int q_lo, int q_hi, double *__restrict__ ax,
                             double *__restrict__ ay, double *__restrict__ az, double *__restrict__ cterm)
{
      int q = blockIdx.x * blockDim.x + threadIdx.x;
      if (q >= n) return;
      const bool own = q >= q_lo && q < q_hi;  // this part's targets (sorted order)
      double m[3] = {0., 0., 0.};
      if (own) {
#pragma unroll 8  // the chunks' loads in flight together (sums still in chunk order)
            for (int c = 0; c < nchunks; c++)
                  for (int d = 0; d < 3; d++) m[d] += partial[(size_t)c * 3 * npad + d * npad + q];
      }
      double c[3];
      grav_finish(q, own, m, s64, slots, cmx, cmy, cmz, M, G, central, j2, ax, ay, az, c);
      if (central)
            for (int d = 0; d < 3; d++) cterm[(size_t)d * n + q] = c[d];
}

// The same from the rows of k_pair_sym and, when not null, the sums of the
// earlier offsets in base; the last block to finish adds up CM_acc (zero without a
// central mass), red: 3 doubles a block, count: zero before and after.
__global__ void __launch_bounds__(GS) k_pair_final(PairRun pr, const D4 *__restrict__ s64,
                                                    const int *__restrict__ slots, int n, double cmx, double cmy,
                                                    double cmz, double M, double G, int central, J2Arg j2,
                                                    double *__restrict__ ax, double *__restrict__ ay,
                                                    double *__restrict__ az, double *__restrict__ red,
                                                    unsigned *__restrict__ count, double *__restrict__ cm_acc)
{
      __shared__ double sh[3][8][32];
      __shared__ double tot[3];
      const long q = (long)blockIdx.x * 32 + (threadIdx.x & 31);
      double v[3];
      pair_rows_sum<3>(pr.part, pr.npad, pr.nb, (int)(q / pr.bsize), pr.k0, pr.nk, q, q < n, sh, v);
      double c[3] = {0., 0., 0.};
      if (threadIdx.x < 32 && q < n) {
            if (pr.base)
                  for (int d = 0; d < 3; d++) v[d] = pr.base[d * pr.npad + q] + v[d];
            grav_finish((int)q, true, v, s64, slots, cmx, cmy, cmz, M, G, central, j2, ax, ay, az, c);
      }
      if (!central) {
            if (blockIdx.x == 0 && threadIdx.x < 3) cm_acc[threadIdx.x] = 0.;
            return;
      }
      if (grid_sum3(c[0], c[1], c[2], red, count, tot) && threadIdx.x < 3) cm_acc[threadIdx.x] = tot[threadIdx.x];
}

// Deterministic two-level sum of 3 component arrays of length n.
__global__ void k_sum3_part(const double *__restrict__ v, int N, const int *__restrict__ n_dev,
                            double *__restrict__ part)
{
      const int n = n_dev ? *n_dev : N;
      __shared__ double sh[3][RB];
      double s[3] = {0., 0., 0.};
      for (int i = blockIdx.x * RB + threadIdx.x; i < n; i += gridDim.x * RB)
            for (int d = 0; d < 3; d++) s[d] += v[(size_t)d * N + i];
      for (int d = 0; d < 3; d++) sh[d][threadIdx.x] = s[d];
      __syncthreads();
      for (int o = RB / 2; o > 0; o >>= 1) {
            if (threadIdx.x < o)
                  for (int d = 0; d < 3; d++) sh[d][threadIdx.x] += sh[d][threadIdx.x + o];
            __syncthreads();
      }
      if (threadIdx.x < 3) part[blockIdx.x * 3 + threadIdx.x] = sh[threadIdx.x][0];
}

// One warp per component, a fixed-shape (deterministic) fold of the partials,
// plus init[d] when given (out may alias init).
__global__ void k_sum3_final(const double *__restrict__ part, int nparts, const double *init, double *out)
{
      const int d = threadIdx.x >> 5, lane = threadIdx.x & 31;
      if (d >= 3) return;
      double s = 0.;
      for (int b = lane; b < nparts; b += 32) s += part[b * 3 + d];
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) out[d] = init ? init[d] + s : s;
}

__global__ void k_fill3(double *__restrict__ ax, double *__restrict__ ay, double *__restrict__ az, int n, double v)
{
      int i = blockIdx.x * blockDim.x + threadIdx.x;
      if (i < n) {
            ax[i] = v;
            ay[i] = v;
            az[i] = v;
      }
}

__global__ void k_set3(double *__restrict__ out, double a, double b, double c)
{
      out[0] = a;
      out[1] = b;
      out[2] = c;
}

}  // namespace

int par_sum3(const double *terms, int N, const int *n_dev, const double *init, double *out, cudaStream_t st)
{
      Ctx &c = ctx();
      const int np = min(128, max(1, (N + RB - 1) / RB));
      k_sum3_part<<<np, RB, 0, st>>>(terms, N, n_dev, c.red + 2048);
      NCG_LAUNCHED();
      k_sum3_final<<<1, 96, 0, st>>>(c.red + 2048, np, init, out);
      NCG_LAUNCHED();
      return NCGPU_OK;
}

int seq_sum3(const double *terms, int N, const int *n_dev, const double *init, double *out, cudaStream_t st)
{
      k_seq_sum3<<<3, 32, 0, st>>>(terms, N, n_dev, init, out);
      NCG_LAUNCHED();
      return NCGPU_OK;
}

namespace {

// The exact field of the existing bodies of slots 0 .. nslots - 1 into ax, ay, az
// (`fill` in the empty slots' rows) and cm_acc, on the scratch it is given.  started
// (may be null): recorded before the field kernel.
int exact_field(const BodyView &bv, int nslots, const CmArg &cm, double G, double sp, int central, const J2Arg &j2,
                int part, int nparts, double fill, int *cidx, D4 *src, double *srcR, int *blockcnt, int *n_dev,
                double *ax, double *ay, double *az, double *cm_acc, cudaStream_t st, cudaEvent_t started)
{
      if (nslots == 0 || !central) {
            k_set3<<<1, 1, 0, st>>>(cm_acc, 0., 0., 0.);
            NCG_LAUNCHED();
            if (nslots == 0) return NCGPU_OK;
      }
      if (nslots <= PREP_N) {
            k_prep_exact<<<1, 1024, 0, st>>>(bv, nslots, G, fill, cidx, n_dev, src, srcR, ax, ay, az);
            NCG_LAUNCHED();
      } else {
            k_fill3<<<(nslots + 255) / 256, 256, 0, st>>>(ax, ay, az, nslots, fill);
            NCG_LAUNCHED();
            NCG_TRY(compact_flags_dev(bv.ex, nslots, blockcnt, n_dev, cidx, st));
            k_pack_exact<<<(nslots + 255) / 256, 256, 0, st>>>(bv, cidx, n_dev, G, src, srcR);
            NCG_LAUNCHED();
      }
      if (started) NCG_CK(cudaEventRecord(started, st));
      const int nb = (nslots + XT - 1) / XT + (central ? 1 : 0);
#define NCG_EXACT(XP_, OCC_)                                                                                          \
      do {                                                                                                           \
            if (sp != 0.)                                                                                            \
                  k_grav_exact<true, XP_, OCC_><<<nb, XP_ + 32, 0, st>>>(src, srcR, cidx, n_dev, cm, G, sp, central, \
                                                                         j2, bv, part, nparts, ax, ay, az, cm_acc);  \
            else                                                                                                     \
                  k_grav_exact<false, XP_, OCC_><<<nb, XP_ + 32, 0, st>>>(src, srcR, cidx, n_dev, cm, G, sp, central,\
                                                                          j2, bv, part, nparts, ax, ay, az, cm_acc); \
      } while (0)
      // (512 threads a CTA while there are fewer than two CTAs an SM: 16.4 against 20.5 us
      // at 1,000 bodies, both 34.8 at 2,000, 113 against 102 at 4,001)
      if (nslots <= 2048) NCG_EXACT(512, 2);
      else NCG_EXACT(256, 4);
#undef NCG_EXACT
      NCG_LAUNCHED();
      return NCGPU_OK;
}

// Slots up to which the Morton order is a rank sort (n^2 compares in one launch), beyond
// it a radix sort (eight launches).  Whole mixed calls, rank / radix, us: 49 / 69 at 250
// bodies, 55 / 79 at 1,000, 73 / 99 at 4,096, 117 / 143 at 8,192, 175 / 188 at 12,345,
// 241 / 238 at 16,384, 394 / 356 at 24,000.
constexpr int RANK_MAX = 14336;

// CM_acc of the tiled modes: the two-level sum of its terms, or zero.
int finish_cm(int central, int n, double *d_cm_acc, cudaStream_t st)
{
      Ctx &c = ctx();
      if (central) return par_sum3(c.cmterm, n, nullptr, nullptr, d_cm_acc, st);
      k_set3<<<1, 1, 0, st>>>(d_cm_acc, 0., 0., 0.);
      NCG_LAUNCHED();
      return NCGPU_OK;
}

}  // namespace

int gravity_eval(const BodyView &bv, int largest_id, const double *cmh, const J2Arg &j2, double *d_acc, long bs,
                 double *d_cm_acc, int mode, cudaStream_t st, int part, int nparts, const double *cm_dev)
{
      Ctx &c = ctx();
      const ncgpu_params &P = c.P;
      if (largest_id + 1 > c.n_max) return NCGPU_E_ARG;
      if (nparts < 1 || part < 0 || part >= nparts) return NCGPU_E_ARG;
      const int nslots = largest_id + 1;
      double *ax = d_acc, *ay = d_acc + bs, *az = d_acc + 2 * bs;
      // empty slots: +0.0 from part 0, -0.0 (the identity of the parts' sum) from the others
      const double fill = part == 0 ? 0. : -0.;
      const bool tiled = mode == NCGPU_GRAVITY_FP64 || mode == NCGPU_GRAVITY_MIXED;
      const int central = P.par_central_mass_bool;
      if (!tiled) {
            // (nothing comes back to the host: the kernels read the count of existing
            // bodies from device memory)
            if (mode != NCGPU_GRAVITY_EXACT && nslots > EXACT_SMALL_N) {  // an unknown mode: refused with any body
                  int n = 0;
                  NCG_TRY(compact_existing(bv.ex, largest_id, &n, st));
                  if (n > 0) return NCGPU_E_ARG;
            }
            NCG_TRY(exact_field(bv, nslots, CmArg{cm_dev, cmh[0], cmh[1], cmh[2], cmh[6]}, P.par_G,
                                P.par_softening_parameter, central, j2, part, nparts, fill, c.cidx, (D4 *)c.src64,
                                c.srcR, c.cnt, c.n_dev, ax, ay, az, d_cm_acc, st, c.kev0));
            if (nslots == 0) return NCGPU_OK;  // (no field kernel: the last one's time stays)
            NCG_CK(cudaEventRecord(c.kev1, st));
            c.kev_valid = 1;
            return NCGPU_OK;
      }
      int n = 0;
      double rr[2] = {0., 0.};  // radius range of the existing bodies
      if (nslots > 0) {
            // compaction, bounding box, Morton order and the tile data sized for
            // every slot, the count of existing bodies read in the kernels; the
            // count and the radius range come back to the host (for the pair
            // kernel's grid and instance) while the GPU sorts and packs
            const int ntub = (nslots + T - 1) / T;
            volatile double *answer = c.pinned + 8 * (size_t)c.n_max + 96;  // (behind the output text's answers)
            double *ans = const_cast<double *>(answer);
            int *vals = nslots <= RANK_MAX ? c.vals2 : c.vals;  // (the rank sort is not in place)
            if (nslots <= 4096) {
                  k_prep_tiled<4, true><<<1, 1024, 0, st>>>(bv, nslots, fill, c.cidx, c.n_dev, c.red, ans, c.keys, vals, ax,
                                                            ay, az);
                  NCG_LAUNCHED();
            } else if (nslots <= 16384) {
                  k_prep_tiled<16, false><<<1, 1024, 0, st>>>(bv, nslots, fill, c.cidx, c.n_dev, c.red, ans, nullptr, nullptr,
                                                              ax, ay, az);
                  NCG_LAUNCHED();
            } else {
                  k_fill3<<<(nslots + 255) / 256, 256, 0, st>>>(ax, ay, az, nslots, fill);
                  NCG_LAUNCHED();
                  NCG_TRY(compact_existing_dev(bv.ex, largest_id, st));
                  const int nbb = min(256, (nslots + RB - 1) / RB);
                  k_bbox_part<<<nbb, RB, 0, st>>>(bv, c.cidx, c.n_dev, c.red);
                  NCG_LAUNCHED();
                  k_bbox_final<<<1, 256, 0, st>>>(c.red, nbb, c.n_dev, ans);
                  NCG_LAUNCHED();
            }
            NCG_CK(cudaEventRecord(c.prep_done, st));
            if (nslots > 4096) {
                  k_morton<<<(nslots + 255) / 256, 256, 0, st>>>(bv, c.cidx, c.n_dev, nslots, c.red, c.keys, vals);
                  NCG_LAUNCHED();
            }
            if (nslots <= RANK_MAX) NCG_TRY(rank_sort(c.keys, vals, nslots, c.vals, st));
            else NCG_TRY(radix_sort_pairs(c.keys, c.vals, nslots, 30, st));
            k_tile_prep<<<(ntub * 32 + 255) / 256, 256, 0, st>>>(bv, c.vals, c.n_dev, ntub, P.par_softening_parameter,
                                                                 mode == NCGPU_GRAVITY_MIXED, (D4 *)c.src64, c.srcR,
                                                                 c.tilebox, (float *)c.src32, c.srcR32,
                                                                 (unsigned *)(c.n_dev + 1));
            NCG_LAUNCHED();
            NCG_CK(cudaEventSynchronize(c.prep_done));
            rr[0] = answer[0];
            rr[1] = answer[1];
            n = (int)answer[2];
      }
      const double G = P.par_G;
      if (n == 0) {
            k_set3<<<1, 1, 0, st>>>(d_cm_acc, 0., 0., 0.);
            NCG_LAUNCHED();
            return NCGPU_OK;
      }
      const int ntiles = (n + T - 1) / T;
      const int npad = ntiles * T;
      const double sp = P.par_softening_parameter;
      const bool soft = sp != 0.;
      // (the Morton order and the tile data were made above, before the count came back)
      D4 *s64 = (D4 *)c.src64;
      double eps2 = 0.;
      int soft_kind = soft ? 2 : 0;
      if (soft) {
            // the largest softening length; with all radii equal (the bounding-box pass
            // found R_min == R_max) it is every pair's: the uniform-epsilon instance, with
            // fewer registers
            const double eu = 2.0 * sp * std::max(std::abs(rr[0]), std::abs(rr[1]));
            eps2 = eu * eu;
            if (rr[0] == rr[1]) soft_kind = 1;
      }
      const double theta = P.par_near_theta > 0. ? P.par_near_theta : 0.15;
      if (nparts == 1) {
            // the whole field: every pair once
            PairData pd{s64, c.srcR, (const float *)c.src32, c.srcR32, c.tilebox, n, ntiles, 0, nullptr, nullptr};
            PairPlan pl = pair_plan<0>(n);
            int got;
            while ((got = ensure_partial(pl.doubles)) != NCGPU_OK && pair_halve<0>(pl)) {}
            NCG_TRY(got);
            PairRun pr;
            NCG_CK(cudaEventRecord(c.kev0, st));
            NCG_TRY(pair_sums<0>(pd, pl, mode == NCGPU_GRAVITY_MIXED ? 0 : 1, soft_kind, theta, eps2, c.partial, pr, st));
            NCG_CK(cudaEventRecord(c.kev1, st));
            c.kev_valid = 1;
            k_pair_final<<<(n + 31) / 32, GS, 0, st>>>(pr, s64, c.vals, n, cmh[0], cmh[1], cmh[2], cmh[6], G, central,
                                                       j2, ax, ay, az, c.cmterm, (unsigned *)(c.n_dev + 1), d_cm_acc);
            NCG_LAUNCHED();
            return NCGPU_OK;
      }
      // softening: general (eps = sp (R_i + R_j)) unless sp == 0; the kernel
      // takes its uniform-eps^2 path itself when all radii are equal
      const int sm = soft ? 2 : 0;
      // work decomposition: (target block, source chunk) CTAs, about
      // grav_slots_mult per resident CTA slot, so that the last wave is short
      // next to the whole launch (CTAs with near tiles run longer)
      int occ = 1;
      if (mode == NCGPU_GRAVITY_MIXED)
            NCG_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, sm ? k_grav_tiled<0, 2> : k_grav_tiled<0, 0>, MXB, 0));
      else
            NCG_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, sm ? k_grav_tiled<1, 2> : k_grav_tiled<1, 0>, MXB, 0));
      // this part's target blocks
      const int ib_lo = (int)((long)ntiles * part / nparts), ib_hi = (int)((long)ntiles * (part + 1) / nparts);
      const int nblk = ib_hi - ib_lo;
      const long want = (long)max(occ, 1) * c.sm_count * c.grav_slots_mult;
      long nch = (want + max(nblk, 1) - 1) / max(nblk, 1);
      if (nch < 1) nch = 1;
      if (nch > ntiles) nch = ntiles;
      int nchunks = (int)nch;
      const int tpc = (ntiles + nchunks - 1) / nchunks;
      nchunks = (ntiles + tpc - 1) / tpc;
      NCG_TRY(ensure_partial((size_t)nchunks * 3 * npad));
      dim3 grid(nchunks, nblk);
      const float *s32 = (const float *)c.src32;
      NCG_CK(cudaEventRecord(c.kev0, st));
#define NCG_TILED(MODE_, SOFT_)                                                                              \
      k_grav_tiled<MODE_, SOFT_><<<grid, MXB, 0, st>>>(s64, c.srcR, s32, c.srcR32, c.tilebox, n, ntiles, tpc, \
                                                      theta, eps2, c.partial, npad, c.err, c.red + 6, sp, ib_lo)
      if (nblk > 0) {  // (a part without target blocks has only the central terms below)
            if (mode == NCGPU_GRAVITY_MIXED) {
                  if (soft_kind == 0) NCG_TILED(0, 0); else if (soft_kind == 1) NCG_TILED(0, 1); else NCG_TILED(0, 2);
            } else {
                  if (soft_kind == 0) NCG_TILED(1, 0); else if (soft_kind == 1) NCG_TILED(1, 1); else NCG_TILED(1, 2);
            }
            NCG_LAUNCHED();
      }
#undef NCG_TILED
      NCG_CK(cudaEventRecord(c.kev1, st));
      c.kev_valid = 1;
      k_grav_final<<<(n + 255) / 256, 256, 0, st>>>(c.partial, nchunks, npad, s64, c.vals, n, cmh[0], cmh[1], cmh[2],
                                                    cmh[6], G, central, j2, ib_lo * T, min(n, ib_hi * T), ax, ay, az,
                                                    c.cmterm);
      NCG_LAUNCHED();
      return finish_cm(central, n, d_cm_acc, st);
}

}  // namespace ncg

namespace ncg {

// The EXACT gravity of gravity_eval on caller-provided scratch, without the
// library context: cidx (n), src (n double4), srcR (n), blockcnt/n_dev for the
// compaction.  Writes ax, ay, az (slots 0..largest_id, zero for empty slots) and
// d_cm_acc.
int gravity_exact_into(const BodyView &bv, int largest_id, const double *cmh, double G, double sp, int central,
                       const J2Arg &j2, int *cidx, double *src, double *srcR, int *blockcnt, int *n_dev, double *ax,
                       double *ay, double *az, double *d_cm_acc, cudaStream_t st)
{
      return exact_field(bv, largest_id + 1, CmArg{nullptr, cmh[0], cmh[1], cmh[2], cmh[6]}, G, sp, central, j2, 0, 1, 0., cidx, (D4 *)src, srcR, blockcnt, n_dev,
                         ax, ay, az, d_cm_acc, st, nullptr);
}

}  // namespace ncg
