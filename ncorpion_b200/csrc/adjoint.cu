// Differentiable gravity + leapfrog: forward integration and its hand-written
// adjoint (reverse mode), no collisions.  There is no reference counterpart for
// the adjoint; the forward is the brute-force driver of the reference
// (src/rk4.c:873-936 with collision_bool = 0): half drift, then n x (kick with
// vector_field, drift), then the half back-drift of the final output, with the
// central mass integrated as a body (kick with CM_acc, drift).
//
// For body k and source j, r = x_j - x_k, D^2 = |r|^2 + eps_kj^2
// (eps_kj = softening_parameter * (R_k + R_j)), a_k = sum_j G m_j r / D^3.
// Tidal tensor T_kj = I/D^3 - 3 r r^T / D^5 (symmetric in k, j).
// Vector-Jacobian products with adjoint velocities lambda (bodies) and Lambda
// (central mass), central-mass offsets s_k = x_k - X, J_k = I/|s|^3 - 3 s s^T/|s|^5:
//   (da/dx)^T lambda |_k  = sum_j G T_kj (m_k lambda_j - m_j lambda_k)
//                           + G J_k (m_k Lambda - M lambda_k)
//   (da/dX)^T ...          = sum_k G J_k (M lambda_k - m_k Lambda)
//   (da/dm)^T ...     |_k  = -sum_j G (lambda_j . r) / D^3 + G Lambda . s_k / |s_k|^3
// The force and its VJP are pairsym.cuh's sums over unordered pairs (FP64, one
// rsqrt per pair); the JVP is summed body by body, tiled through shared memory
// with (target block, source chunk) work units reduced in a fixed order.  In the
// MIXED gravity mode the bodies are taken in the Morton order of their initial
// positions (a permutation at the call's boundary), every
// evaluation computes the 128-body tiles' boxes, and only the tile pairs whose
// boxes are near (1.45 near_theta x the larger diagonal, near_theta x it in the JVP,
// and each tile with itself) are summed in FP64; the others in FP32 on coordinates relative to a tile's
// centre, short FP32 sums folded into FP64 -- the force kernel's scheme applied
// to the force, its VJP and its JVP.
//
// A kick and drift is three launches (tile data, pair sums, final pass with the
// kick, the drift and the central body's), a step of the reverse sweep three
// more.  N = 16,384, mixed: a force's pair sums take 128 us and a VJP's 268 (208
// and 396 when each body's were made by themselves, bound by the FP32 pipe and the
// near tiles' FP64), a forward call and a forward + adjoint call of 32 steps
// 24.7 ms (42.3 with those, with six to nine launches a step and strided copies of the
// caller's arrays).  N = 5,003, FP64: 30 us and 57 (50 and 86), 24 steps 5.50 ms (9.47).
#include <algorithm>
#include <vector>
#include "common.cuh"
#include "pairsym.cuh"

namespace ncg {

namespace {

constexpr int AT = PT;  // bodies per tile / threads per block of the JVP's pair sums

struct Src {
      const double *x, *y, *z, *m, *sR, *lx, *ly, *lz;  // lx.. : adjoints (VJP) or position tangents (JVP)
      const double *dm;                                 // mass tangents (JVP)
};

// The JVP's pair sums, d a_k = sum_j G [dm_j r + m_j T_kj (dx_j - dx_k)] / ...,
// of target block blockIdx.y against source chunk blockIdx.x, in FP64.
template <bool SOFT>
__global__ void __launch_bounds__(AT) k_pairs_jvp(Src s, int n, int tpc, double *__restrict__ part, long stride)
{
      __shared__ double sx[AT], sy[AT], sz[AT], sm[AT], sr[AT], slx[AT], sly[AT], slz[AT], sdm[AT];
      const int k = blockIdx.y * AT + threadIdx.x;
      const bool act = k < n;
      const int kk = act ? k : 0;
      const double xk = s.x[kk], yk = s.y[kk], zk = s.z[kk], rk = SOFT ? s.sR[kk] : 0.;
      const double lxk = s.lx[kk], lyk = s.ly[kk], lzk = s.lz[kk];
      double o0 = 0., o1 = 0., o2 = 0.;
      const int ntiles = (n + AT - 1) / AT;
      const int t0 = blockIdx.x * tpc, t1 = min(ntiles, t0 + tpc);
      for (int t = t0; t < t1; ++t) {
            const int j = t * AT + threadIdx.x;
            __syncthreads();
            if (j < n) {
                  sx[threadIdx.x] = s.x[j]; sy[threadIdx.x] = s.y[j]; sz[threadIdx.x] = s.z[j];
                  sm[threadIdx.x] = s.m[j];
                  if (SOFT) sr[threadIdx.x] = s.sR[j];
                  slx[threadIdx.x] = s.lx[j]; sly[threadIdx.x] = s.ly[j]; slz[threadIdx.x] = s.lz[j];
                  sdm[threadIdx.x] = s.dm[j];
            }
            __syncthreads();
            const int cnt = min(AT, n - t * AT);
            for (int q = 0; q < cnt; ++q) {
                  if (t * AT + q == k) continue;
                  const double rx = sx[q] - xk, ry = sy[q] - yk, rz = sz[q] - zk;
                  double d2 = 0.;
                  if (SOFT) { const double e = rk + sr[q]; d2 = e * e; }
                  d2 = fma(rx, rx, fma(ry, ry, fma(rz, rz, d2)));
                  const double ri = rsqrt(d2);
                  const double i3 = ri * ri * ri;
                  const double i5 = i3 * ri * ri;
                  const double dx = slx[q] - lxk, dy = sly[q] - lyk, dz = slz[q] - lzk;
                  const double rd = rx * dx + ry * dy + rz * dz;
                  const double mj = sm[q], c = 3.0 * rd * i5 * mj, g = sdm[q] * i3;
                  o0 += g * rx + mj * i3 * dx - rx * c;
                  o1 += g * ry + mj * i3 * dy - ry * c;
                  o2 += g * rz + mj * i3 * dz - rz * c;
            }
      }
      if (act) {
            double *p = part + (size_t)blockIdx.x * 3 * stride;
            p[k] = o0; p[stride + k] = o1; p[2 * stride + k] = o2;
      }
}

// One warp per tile: centre and half extents of its bodies' box.
__global__ void k_adj_tilebox(const double *__restrict__ pos, int n, int ntiles, double *__restrict__ box)
{
      const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
      if (warp >= ntiles) return;
      const int base = warp * AT, cnt = min(AT, n - base);
      double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
      for (int j = lane; j < cnt; j += 32)
            for (int d = 0; d < 3; d++) {
                  const double v = pos[(size_t)d * n + base + j];
                  lo[d] = fmin(lo[d], v);
                  hi[d] = fmax(hi[d], v);
            }
      for (int o = 16; o > 0; o >>= 1)
            for (int d = 0; d < 3; d++) {
                  lo[d] = fmin(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
                  hi[d] = fmax(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
            }
      if (lane < 3) {
            box[warp * 6 + lane] = 0.5 * (lo[lane] + hi[lane]);
            box[warp * 6 + 3 + lane] = 0.5 * (hi[lane] - lo[lane]);
      }
}

// k_pairs_jvp in the MIXED mode: FP64 for near tile pairs (the same pair terms),
// FP32 relative to the source tile's centre for the others.
template <bool SOFT>
__global__ void __launch_bounds__(AT) k_pairs_jvp_mx(Src s, int n, int tpc, const double *__restrict__ box,
                                                     double theta, double *__restrict__ part, long stride)
{
      __shared__ double sx[AT], sy[AT], sz[AT], sm[AT], sr[AT], slx[AT], sly[AT], slz[AT], sdm[AT];
      __shared__ float fx[AT], fy[AT], fz[AT], fm[AT], fr[AT], flx[AT], fly[AT], flz[AT], fdm[AT];
      const int ib = blockIdx.y;
      const int k = ib * AT + threadIdx.x;
      const bool act = k < n;
      const int kk = act ? k : 0;
      const double xk = s.x[kk], yk = s.y[kk], zk = s.z[kk], rk = SOFT ? s.sR[kk] : 0.;
      const double lxk = s.lx[kk], lyk = s.ly[kk], lzk = s.lz[kk];
      const float rkf = (float)rk, lxkf = (float)lxk, lykf = (float)lyk, lzkf = (float)lzk;
      double o0 = 0., o1 = 0., o2 = 0.;
      const int ntiles = (n + AT - 1) / AT;
      const int t0 = blockIdx.x * tpc, t1 = min(ntiles, t0 + tpc);
      const double *bi = box + 6 * ib;
      for (int t = t0; t < t1; ++t) {
            const int j = t * AT + threadIdx.x;
            const double *bj = box + 6 * t;
            const bool near = t == ib || tiles_near(bi, bj, theta);
            __syncthreads();
            if (j < n) {
                  if (near) {
                        sx[threadIdx.x] = s.x[j]; sy[threadIdx.x] = s.y[j]; sz[threadIdx.x] = s.z[j];
                        sm[threadIdx.x] = s.m[j];
                        if (SOFT) sr[threadIdx.x] = s.sR[j];
                        slx[threadIdx.x] = s.lx[j]; sly[threadIdx.x] = s.ly[j]; slz[threadIdx.x] = s.lz[j];
                        sdm[threadIdx.x] = s.dm[j];
                  } else {
                        fx[threadIdx.x] = (float)(s.x[j] - bj[0]);
                        fy[threadIdx.x] = (float)(s.y[j] - bj[1]);
                        fz[threadIdx.x] = (float)(s.z[j] - bj[2]);
                        fm[threadIdx.x] = (float)s.m[j];
                        if (SOFT) fr[threadIdx.x] = (float)s.sR[j];
                        flx[threadIdx.x] = (float)s.lx[j]; fly[threadIdx.x] = (float)s.ly[j];
                        flz[threadIdx.x] = (float)s.lz[j];
                        fdm[threadIdx.x] = (float)s.dm[j];
                  }
            }
            __syncthreads();
            const int cnt = min(AT, n - t * AT);
            if (near) {
                  for (int q = 0; q < cnt; ++q) {
                        if (t * AT + q == k) continue;
                        const double rx = sx[q] - xk, ry = sy[q] - yk, rz = sz[q] - zk;
                        double d2 = 0.;
                        if (SOFT) { const double e = rk + sr[q]; d2 = e * e; }
                        d2 = fma(rx, rx, fma(ry, ry, fma(rz, rz, d2)));
                        const double ri = rsqrt(d2);
                        const double i3 = ri * ri * ri;
                        const double i5 = i3 * ri * ri;
                        const double dx = slx[q] - lxk, dy = sly[q] - lyk, dz = slz[q] - lzk;
                        const double rd = rx * dx + ry * dy + rz * dz;
                        const double mj = sm[q], c = 3.0 * rd * i5 * mj, g = sdm[q] * i3;
                        o0 += g * rx + mj * i3 * dx - rx * c;
                        o1 += g * ry + mj * i3 * dy - ry * c;
                        o2 += g * rz + mj * i3 * dz - rz * c;
                  }
            } else {
                  const float xr = (float)(xk - bj[0]), yr = (float)(yk - bj[1]), zr = (float)(zk - bj[2]);
                  for (int q0 = 0; q0 < cnt; q0 += 64) {  // FP32 runs of 64 sources
                        float p0 = 0.f, p1 = 0.f, p2 = 0.f;
                        const int qe = min(cnt, q0 + 64);
                        for (int q = q0; q < qe; ++q) {
                              const float rx = fx[q] - xr, ry = fy[q] - yr, rz = fz[q] - zr;
                              float d2 = 0.f;
                              if (SOFT) { const float e = rkf + fr[q]; d2 = e * e; }
                              d2 = fmaf(rx, rx, fmaf(ry, ry, fmaf(rz, rz, d2)));
                              const float ri = rsqrtf(d2);
                              const float i3 = ri * ri * ri, i5 = i3 * ri * ri;
                              const float dx = flx[q] - lxkf, dy = fly[q] - lykf, dz = flz[q] - lzkf;
                              const float rd = rx * dx + ry * dy + rz * dz;
                              const float mj = fm[q], c = 3.f * rd * i5 * mj, g = fdm[q] * i3;
                              p0 += g * rx + mj * i3 * dx - rx * c;
                              p1 += g * ry + mj * i3 * dy - ry * c;
                              p2 += g * rz + mj * i3 * dz - rz * c;
                        }
                        o0 += (double)p0; o1 += (double)p1; o2 += (double)p2;
                  }
            }
      }
      if (act) {
            double *p = part + (size_t)blockIdx.x * 3 * stride;
            p[k] = o0; p[stride + k] = o1; p[2 * stride + k] = o2;
      }
}

// The pair sums' tile data of positions pos (3 blocks of n), one warp per tile:
// FP64 records and, with `mixed`, the tile's box and its FP32 copy.  pos_out
// (may be null): a copy of pos and, behind it, of the central body's position.
// lv (may be null): the reverse sweep's adjoint velocities, first advanced by the
// adjoint of the drift, lv += dt lx (and LV += dt LX), then copied to l32.
__global__ void k_lf_tiles(const double *__restrict__ pos, const double *__restrict__ m, int n, int ntiles, int mixed,
                           D4 *__restrict__ s64, float *__restrict__ s32, double *__restrict__ box,
                           double *__restrict__ pos_out, const double *__restrict__ cm, double dt,
                           const double *__restrict__ lx, double *__restrict__ lv, float *__restrict__ l32,
                           const double *__restrict__ LX, double *__restrict__ LV)
{
      const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
      if (warp >= ntiles) return;
      if (warp == 0 && lane < 3) {
            if (pos_out) pos_out[3 * (size_t)n + lane] = cm[lane];
            if (lv) LV[lane] += dt * LX[lane];
      }
      const int base = warp * PT;
      D4 b[PU];
      double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
#pragma unroll
      for (int u = 0; u < PU; u++) {
            const int k = base + lane + 32 * u;
            if (k < n) {
                  b[u] = D4{pos[k], pos[(size_t)n + k], pos[2 * (size_t)n + k], m[k]};
                  s64[k] = b[u];
                  if (pos_out) {
                        pos_out[k] = b[u].x;
                        pos_out[(size_t)n + k] = b[u].y;
                        pos_out[2 * (size_t)n + k] = b[u].z;
                  }
                  lo[0] = fmin(lo[0], b[u].x); hi[0] = fmax(hi[0], b[u].x);
                  lo[1] = fmin(lo[1], b[u].y); hi[1] = fmax(hi[1], b[u].y);
                  lo[2] = fmin(lo[2], b[u].z); hi[2] = fmax(hi[2], b[u].z);
            }
            if (lv)
                  for (int d = 0; d < 3; d++) {
                        double v = 0.;
                        if (k < n) {
                              const size_t q = (size_t)d * n + k;
                              v = lv[q] + dt * lx[q];
                              lv[q] = v;
                        }
                        if (mixed) l32[((size_t)warp * 3 + d) * PT + lane + 32 * u] = (float)v;
                  }
      }
      if (!mixed) return;
      for (int o = 16; o > 0; o >>= 1)
            for (int d = 0; d < 3; d++) {
                  lo[d] = fmin(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
                  hi[d] = fmax(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
            }
      const double c[3] = {0.5 * (lo[0] + hi[0]), 0.5 * (lo[1] + hi[1]), 0.5 * (lo[2] + hi[2])};
      if (lane < 3) {
            box[warp * 6 + lane] = c[lane];
            box[warp * 6 + 3 + lane] = 0.5 * (hi[lane] - lo[lane]);
      }
      float *tile = s32 + (size_t)warp * 4 * PT;
#pragma unroll
      for (int u = 0; u < PU; u++) {
            const int j = lane + 32 * u;
            const bool in = base + j < n;
            tile[j] = in ? (float)(b[u].x - c[0]) : 1e18f;
            tile[PT + j] = in ? (float)(b[u].y - c[1]) : 1e18f;
            tile[2 * PT + j] = in ? (float)(b[u].z - c[2]) : 1e18f;
            tile[3 * PT + j] = in ? (float)b[u].w : 0.f;
      }
}

}  // namespace

namespace {
constexpr int SB = 256;  // threads of the fold kernels and of the two-level sums

// The block's sums of three per-body terms (zero past n): part[3 b + d] for
// block b; k_sum3f then adds the blocks' sums in block order (deterministic).
__device__ __forceinline__ void block_sum3(double v0, double v1, double v2, double *__restrict__ part)
{
      __shared__ double sh[3][SB];
      sh[0][threadIdx.x] = v0;
      sh[1][threadIdx.x] = v1;
      sh[2][threadIdx.x] = v2;
      __syncthreads();
      for (int o = SB / 2; o > 0; o >>= 1) {
            if (threadIdx.x < o)
                  for (int d = 0; d < 3; d++) sh[d][threadIdx.x] += sh[d][threadIdx.x + o];
            __syncthreads();
      }
      if (threadIdx.x < 3) part[blockIdx.x * 3 + threadIdx.x] = sh[threadIdx.x][0];
}


// The force's final pass, 32 bodies a block: a = G * (the pair sums) + central
// term, then the kick v += dt a and the drift x += dt v; the last block kicks and
// drifts the central body with the sum of its terms.
__global__ void __launch_bounds__(SB) k_lf_force(PairRun pr, int n, double *__restrict__ X, double *__restrict__ V,
                                                 const double *__restrict__ m, double *__restrict__ cm, double G,
                                                 double M, int central, double dt, double *__restrict__ red,
                                                 unsigned *__restrict__ count)
{
      __shared__ double sh[3][8][32];
      __shared__ double tot[3];
      const long k = (long)blockIdx.x * 32 + (threadIdx.x & 31);
      double a[3], c[3] = {0., 0., 0.};
      pair_rows_sum<3>(pr.part, pr.npad, pr.nb, (int)(k / pr.bsize), pr.k0, pr.nk, k, k < n, sh, a);
      if (threadIdx.x < 32 && k < n) {
            double x[3];
            for (int d = 0; d < 3; d++) {
                  if (pr.base) a[d] = pr.base[d * pr.npad + k] + a[d];
                  a[d] *= G;
                  x[d] = X[(size_t)d * n + k];
            }
            if (central) {
                  double s[3] = {x[0] - cm[0], x[1] - cm[1], x[2] - cm[2]};
                  double r2 = s[0] * s[0] + s[1] * s[1] + s[2] * s[2];
                  double ri = rsqrt(r2), i3 = ri * ri * ri;
                  const double g = G * m[k] * i3;
                  for (int d = 0; d < 3; d++) {
                        a[d] -= G * M * s[d] * i3;
                        c[d] = g * s[d];
                  }
            }
            for (int d = 0; d < 3; d++) {
                  const size_t q = (size_t)d * n + k;
                  const double v = V[q] + dt * a[d];
                  V[q] = v;
                  X[q] = x[d] + dt * v;
            }
      }
      if (!central) return;
      if (grid_sum3(c[0], c[1], c[2], red, count, tot) && threadIdx.x < 3) {
            const double v = cm[3 + threadIdx.x] + dt * tot[threadIdx.x];
            cm[3 + threadIdx.x] = v;
            cm[threadIdx.x] += dt * v;
      }
}

// The VJP's final pass: lx += dt (its position part), gm += dt (its mass part);
// the last block advances the central body's LX.
__global__ void __launch_bounds__(SB) k_lf_vjp(PairRun pr, int n, const double *__restrict__ pos,
                                               const double *__restrict__ m, const double *__restrict__ lv,
                                               const double *__restrict__ cm, const double *__restrict__ Lam, double G,
                                               double M, int central, double dt, double *__restrict__ lx,
                                               double *__restrict__ gm, double *__restrict__ LX,
                                               double *__restrict__ red, unsigned *__restrict__ count)
{
      __shared__ double sh[4][8][32];
      __shared__ double tot[3];
      const long k = (long)blockIdx.x * 32 + (threadIdx.x & 31);
      double o[4], xt[3] = {0., 0., 0.};
      pair_rows_sum<4>(pr.part, pr.npad, pr.nb, (int)(k / pr.bsize), pr.k0, pr.nk, k, k < n, sh, o);
      if (threadIdx.x < 32 && k < n) {
            for (int d = 0; d < 4; d++) {
                  if (pr.base) o[d] = pr.base[d * pr.npad + k] + o[d];
                  o[d] *= G;
            }
            if (central) {
                  double sv[3], lam[3];
                  for (int d = 0; d < 3; d++) {
                        sv[d] = pos[(size_t)d * n + k] - cm[d];
                        lam[d] = lv[(size_t)d * n + k];
                  }
                  double r2 = sv[0] * sv[0] + sv[1] * sv[1] + sv[2] * sv[2];
                  double ri = rsqrt(r2), i3 = ri * ri * ri, i5 = i3 * ri * ri;
                  const double mk = m[k];
                  // w = m_k Lambda - M lambda_k ;  J w = w/|s|^3 - 3 s (s.w)/|s|^5
                  double w[3], sw = 0.;
                  for (int d = 0; d < 3; d++) { w[d] = mk * Lam[d] - M * lam[d]; sw += sv[d] * w[d]; }
                  for (int d = 0; d < 3; d++) {
                        const double Jw = w[d] * i3 - 3.0 * sv[d] * sw * i5;
                        o[d] += G * Jw;
                        xt[d] = -G * Jw;  // G J (M lambda - m Lambda)
                  }
                  o[3] += G * (Lam[0] * sv[0] + Lam[1] * sv[1] + Lam[2] * sv[2]) * i3;
            }
            for (int d = 0; d < 3; d++) lx[(size_t)d * n + k] += dt * o[d];
            gm[k] += dt * o[3];
      }
      if (!central) return;
      if (grid_sum3(xt[0], xt[1], xt[2], red, count, tot) && threadIdx.x < 3) LX[threadIdx.x] += dt * tot[threadIdx.x];
}

// JVP: d a = G * sum of chunk partials - G M J_k (dx_k - dX); per-body terms
// of d A_cm = sum_k G [dm_k s_k/|s|^3 + m_k J_k (dx_k - dX)].
__global__ void __launch_bounds__(SB) k_jvp_final(const double *__restrict__ part, int nch, long stride, Src s,
                                                  int n, const double *__restrict__ cm,
                                                  const double *__restrict__ dX, double G, double M, int central,
                                                  double *dax, double *day, double *daz, double *__restrict__ red)
{
      const int k = blockIdx.x * blockDim.x + threadIdx.x;
      double ct[3] = {0., 0., 0.};
      if (k < n) {
      double o[3] = {0., 0., 0.};
#pragma unroll 8  // the chunks' loads in flight together (sums still in chunk order)
      for (int c = 0; c < nch; c++)
            for (int d = 0; d < 3; d++) o[d] += part[(size_t)c * 3 * stride + d * stride + k];
      for (int d = 0; d < 3; d++) o[d] *= G;
      if (central) {
            double sv[3] = {s.x[k] - cm[0], s.y[k] - cm[1], s.z[k] - cm[2]};
            double r2 = sv[0] * sv[0] + sv[1] * sv[1] + sv[2] * sv[2];
            double ri = rsqrt(r2), i3 = ri * ri * ri, i5 = i3 * ri * ri;
            double u[3] = {s.lx[k] - dX[0], s.ly[k] - dX[1], s.lz[k] - dX[2]};
            double su = sv[0] * u[0] + sv[1] * u[1] + sv[2] * u[2];
            double Ju[3];
            for (int d = 0; d < 3; d++) Ju[d] = u[d] * i3 - 3.0 * sv[d] * su * i5;
            const double mk = s.m[k], dmk = s.dm[k];
            for (int d = 0; d < 3; d++) {
                  o[d] -= G * M * Ju[d];
                  ct[d] = G * (dmk * sv[d] * i3 + mk * Ju[d]);
            }
      }
      dax[k] = o[0]; day[k] = o[1]; daz[k] = o[2];
      }
      if (central) block_sum3(ct[0], ct[1], ct[2], red);  // the terms of d A_cm
}

// out[d] = the sum of the blocks' partial sums part[3 b + d] (block_sum3), in
// block order (d < 3)
__global__ void k_sum3f(const double *__restrict__ part, int np, double *__restrict__ out)
{
      int d = threadIdx.x;
      if (d >= 3) return;
      double s = 0.;
      for (int b = 0; b < np; b++) s += part[3 * b + d];
      out[d] = s;
}

// y += a * x over 3 SoA blocks of n (and 3 CM components when cmy != nullptr)
__global__ void k_axpy3(double a, const double *__restrict__ x, double *__restrict__ y, int n, long stride,
                        const double *__restrict__ cmx, double *cmy)
{
      int k = blockIdx.x * blockDim.x + threadIdx.x;
      if (k < n)
            for (int d = 0; d < 3; d++) y[d * stride + k] += a * x[d * stride + k];
      if (k < 3 && cmy) cmy[k] += a * cmx[k];
}

}  // namespace

namespace {

struct LF {
      int n, ntiles, tpc, nch;
      int soft;                    // 0: none, 1: uniform (eps2), 2: general
      bool central;
      double G, M, eps2;
      double *X, *V, *m, *sR, *cm, *out, *part, *red;
      double *lx, *lv, *LX, *LV, *gm;
      double *ckpt, *seg;
      double *tx, *tv, *tm, *tX, *da, *dA;  // tangents (JVP)
      double *jpart;               // the JVP's chunk partials
      D4 *s64;
      float *s32, *sR32, *l32;
      unsigned *count;
      PairPlan pf, pv;             // the force's and the VJP's pair sums
      int C, ncp;
      bool mixed;                  // MIXED gravity mode
      double theta, *box;
      double *stage;               // the caller's arrays, 3 n
      const int *perm;             // the caller's body at each position (null: the same)
      cudaStream_t st;
};

// the pair sums of OP over positions pos; VJP: after lv += dt lx.  pos_out: see k_lf_tiles.
template <int OP>
int lf_pairs(LF &L, const double *pos, const double *cmpos, double *pos_out, double dt, PairRun &run)
{
      const int n = L.n;
      k_lf_tiles<<<(L.ntiles * 32 + 127) / 128, 128, 0, L.st>>>(pos, L.m, n, L.ntiles, L.mixed, L.s64, L.s32, L.box,
                                                                pos_out, cmpos, dt, L.lx, OP == 1 ? L.lv : nullptr,
                                                                L.l32, L.LX, L.LV);
      NCG_LAUNCHED();
      PairData pd{L.s64, L.sR, L.s32, L.sR32, L.box, n, L.ntiles, 0, L.lv, L.l32};
      return pair_sums<OP>(pd, OP == 0 ? L.pf : L.pv, L.mixed ? 0 : 1, L.soft, L.theta, L.eps2, L.part, run, L.st);
}

// kick (v += dt a, CM too) then drift (x += dt v, CM too); pos_out (may be null):
// the positions that the kick sees
int lf_step(LF &L, double dt, double *pos_out = nullptr)
{
      PairRun run;
      NCG_TRY(lf_pairs<0>(L, L.X, L.cm, pos_out, dt, run));
      k_lf_force<<<(L.n + 31) / 32, SB, 0, L.st>>>(run, L.n, L.X, L.V, L.m, L.cm, L.G, L.M, L.central, dt, L.red,
                                                   L.count);
      NCG_LAUNCHED();
      return NCGPU_OK;
}

// The adjoint of one kick and drift: lv += dt lx, then lx and gm by the kick's VJP.
int lf_vjp(LF &L, const double *pos, const double *cmpos, double dt)
{
      PairRun run;
      NCG_TRY(lf_pairs<1>(L, pos, cmpos, nullptr, dt, run));
      k_lf_vjp<<<(L.n + 31) / 32, SB, 0, L.st>>>(run, L.n, pos, L.m, L.lv, cmpos, L.LV, L.G, L.M, L.central, dt, L.lx,
                                                 L.gm, L.LX, L.red, L.count);
      NCG_LAUNCHED();
      return NCGPU_OK;
}

// One kick + drift of the state and of its tangents.
int lf_step_jvp(LF &L, double dt)
{
      const int n = L.n, nb = (n + 255) / 256;
      Src s{L.X, L.X + n, L.X + 2 * n, L.m, L.sR, L.tx, L.tx + n, L.tx + 2 * n, L.tm};
      dim3 grid(L.nch, L.ntiles);
      if (L.mixed) {
            k_adj_tilebox<<<(L.ntiles * 32 + 255) / 256, 256, 0, L.st>>>(L.X, n, L.ntiles, L.box);
            NCG_LAUNCHED();
            if (L.soft) k_pairs_jvp_mx<true><<<grid, AT, 0, L.st>>>(s, n, L.tpc, L.box, L.theta, L.jpart, n);
            else k_pairs_jvp_mx<false><<<grid, AT, 0, L.st>>>(s, n, L.tpc, L.box, L.theta, L.jpart, n);
      } else {
            if (L.soft) k_pairs_jvp<true><<<grid, AT, 0, L.st>>>(s, n, L.tpc, L.jpart, n);
            else k_pairs_jvp<false><<<grid, AT, 0, L.st>>>(s, n, L.tpc, L.jpart, n);
      }
      NCG_LAUNCHED();
      const int nbs = (n + SB - 1) / SB;
      k_jvp_final<<<nbs, SB, 0, L.st>>>(L.jpart, L.nch, n, s, n, L.cm, L.tX, L.G, L.M, L.central, L.da, L.da + n,
                                        L.da + 2 * n, L.red);
      NCG_LAUNCHED();
      if (L.central) {
            k_sum3f<<<1, 32, 0, L.st>>>(L.red, nbs, L.dA);
            NCG_LAUNCHED();
      }
      NCG_TRY(lf_step(L, dt));
      k_axpy3<<<nb, 256, 0, L.st>>>(dt, L.da, L.tv, n, n, L.dA, L.central ? L.tX + 3 : nullptr);
      NCG_LAUNCHED();
      k_axpy3<<<nb, 256, 0, L.st>>>(dt, L.tv, L.tx, n, n, L.tX + 3, L.central ? L.tX : nullptr);
      NCG_LAUNCHED();
      return NCGPU_OK;
}

// The caller's arrays cross in one contiguous copy each and are put in the pair
// sums' order (perm: the body at each position; null: the caller's order) and into
// three blocks of n on the device.  (Three strided copies of 8-byte rows an array,
// and the permutation on the host, took 1.0-1.3 ms a call at 16,384 bodies before
// any step.)
__global__ void k_gather_rows(const double *__restrict__ in, const int *__restrict__ perm, int n, int width,
                              double *__restrict__ out)
{
      const int k = blockIdx.x * blockDim.x + threadIdx.x;
      if (k >= n) return;
      const size_t b = perm ? perm[k] : k;
      for (int d = 0; d < width; d++) out[(size_t)d * n + k] = in[width * b + d];
}

__global__ void k_scatter_rows(const double *__restrict__ in, const int *__restrict__ perm, int n, int width,
                               double *__restrict__ out)
{
      const int k = blockIdx.x * blockDim.x + threadIdx.x;
      if (k >= n) return;
      const size_t b = perm ? perm[k] : k;
      for (int d = 0; d < width; d++) out[width * b + d] = in[(size_t)d * n + k];
}

// src (host, n rows of `width` doubles) into dst (device, `width` blocks of n)
int rows_in(LF &L, double *dst, const double *src, int width)
{
      NCG_CK(cudaMemcpyAsync(L.stage, src, sizeof(double) * width * (size_t)L.n, cudaMemcpyHostToDevice, L.st));
      k_gather_rows<<<(L.n + 255) / 256, 256, 0, L.st>>>(L.stage, L.perm, L.n, width, dst);
      NCG_LAUNCHED();
      return NCGPU_OK;
}

int rows_out(LF &L, double *dst, const double *src, int width)
{
      k_scatter_rows<<<(L.n + 255) / 256, 256, 0, L.st>>>(src, L.perm, L.n, width, L.stage);
      NCG_LAUNCHED();
      NCG_CK(cudaMemcpyAsync(dst, L.stage, sizeof(double) * width * (size_t)L.n, cudaMemcpyDeviceToHost, L.st));
      return NCGPU_OK;
}

// sR = sp * R, element by element (in place when sR == R), and its FP32 copy with
// zero padding up to npad
__global__ void k_scale_R(const double *R, double sp, double *sR, int n, float *__restrict__ sR32, int npad)
{
      int k = blockIdx.x * blockDim.x + threadIdx.x;
      if (k >= npad) return;
      const double r = k < n ? sp * R[k] : 0.;
      if (k < n) sR[k] = r;
      sR32[k] = (float)r;
}

__global__ void k_xf(const double *__restrict__ X, const double *__restrict__ V, double h, double *__restrict__ out,
                     int n)
{
      int k = blockIdx.x * blockDim.x + threadIdx.x;
      if (k < n)
            for (int d = 0; d < 3; d++) out[(size_t)d * n + k] = X[(size_t)d * n + k] - h * V[(size_t)d * n + k];
}

// perm (host, may be null): the caller's body at each position of the sums' order.
int lf_core(const struct ncgpu_leapfrog_args *a, int mode, bool mixed, const int *perm)
{
      const bool vjp = mode == 1, jvp = mode == 2;
      Ctx &c = ctx();
      const int n = a->n;
      if (n <= 0 || !a->x0 || !a->v0 || !a->m || !a->R || !a->cm || a->nsteps < 0) return NCGPU_E_ARG;
      if (c.P.par_J2_bool) return NCGPU_E_UNSUPPORTED;  // the J2 term has no derivative kernels
      if (vjp && (!a->adj_x_final || !a->grad_x0 || !a->grad_v0 || !a->grad_m)) return NCGPU_E_ARG;
      if (jvp && (!a->tan_x0 || !a->tan_v0 || !a->tan_m || !a->tan_x_final)) return NCGPU_E_ARG;
      LF L{};
      L.n = n;
      L.st = c.s;
      L.G = c.P.par_G;
      L.M = a->cm[6];
      L.central = c.P.par_central_mass_bool != 0;
      const double sp = c.P.par_softening_parameter;
      L.soft = 0;
      L.eps2 = 0.;
      if (sp != 0.) {  // (all radii equal: one softening length)
            const auto mm = std::minmax_element(a->R, a->R + n);
            L.soft = *mm.first == *mm.second ? 1 : 2;
            const double eu = 2.0 * sp * std::max(std::abs(*mm.first), std::abs(*mm.second));  // the largest
            L.eps2 = eu * eu;
      }
      L.ntiles = (n + AT - 1) / AT;
      L.nch = 0;
      if (jvp) {
            if (mixed) {
                  // (target tile, source chunk) work units: about 8 per resident CTA
                  // slot, so that the last wave is short
                  int occ = 1;
                  NCG_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_pairs_jvp_mx<true>, AT, 0));
                  const long want = 8L * std::max(occ, 1) * c.sm_count;
                  L.nch = (int)std::max(1L, std::min((long)L.ntiles, (want + L.ntiles - 1) / L.ntiles));
            } else {
                  L.nch = std::max(1, std::min(L.ntiles, (2048 + L.ntiles - 1) / L.ntiles));
            }
            L.tpc = (L.ntiles + L.nch - 1) / L.nch;
            L.nch = (L.ntiles + L.tpc - 1) / L.tpc;
      }
      L.pf = pair_plan<0>(n);
      L.pv = pair_plan<1>(n);
      L.mixed = mixed;
      L.theta = c.P.par_near_theta > 0. ? c.P.par_near_theta : 0.15;
      L.C = a->checkpoint > 0 ? a->checkpoint : 32;
      L.ncp = (a->nsteps + L.C - 1) / L.C + 1;
      const size_t N = (size_t)n, st = 6 * N + 6, NP = (size_t)L.ntiles * AT;
      const size_t nred = (N + 31) / 32;  // blocks of the final passes
      const size_t rest = 4 * NP + 2 * NP + NP / 2 + 3 * NP / 2 + 2                   // s64 s32 sR32 l32 count
                     + 3 * N * 2 + 2 * N + 6 + 3 * N + 3 * nred                  // X V m sR cm out red
                     + 3 * N * 2 + 6 + N                                         // lx lv LX LV gm
                     + (vjp ? st * L.ncp + (size_t)L.C * (3 * N + 3) : 0)        // checkpoints, segment
                     + (jvp ? 3 * N * 3 + N + 6 + 3 + 3 * N * L.nch : 0)         // tx tv tm tX da dA, partials
                     + 6 * (size_t)L.ntiles                                      // tile boxes
                     + 3 * N + (N + 1) / 2;                                      // stage, perm
      size_t npart;  // the pair sums' rows, fewer at a time where the memory is short
      for (;;) {
            npart = vjp ? std::max(L.pf.doubles, L.pv.doubles) : L.pf.doubles;
            if (rest + npart <= c.lf_cap) break;  // grown when needed, kept for the next call
            if (c.lf_buf) cudaFree(c.lf_buf);
            c.lf_buf = nullptr;
            c.lf_cap = 0;
            const cudaError_t e = cudaMalloc(&c.lf_buf, (rest + npart) * sizeof(double));
            if (e == cudaSuccess) {
                  c.lf_cap = rest + npart;
                  break;
            }
            cudaGetLastError();
            c.lf_buf = nullptr;
            const bool less = pair_halve<0>(L.pf);
            if (!(pair_halve<1>(L.pv) || less)) return cuda_fail(e, "cudaMalloc", __FILE__, __LINE__);
      }
      double *p = c.lf_buf;
      auto take = [&](size_t k) { double *q = p; p += k; return q; };
      L.s64 = (D4 *)take(4 * NP);  // (the widest alignment first)
      L.s32 = (float *)take(2 * NP);
      L.sR32 = (float *)take(NP / 2);
      L.l32 = (float *)take(3 * NP / 2);
      L.count = (unsigned *)take(2);
      L.X = take(3 * N); L.V = take(3 * N); L.m = take(N); L.sR = take(N); L.cm = take(6);
      L.out = take(3 * N); L.part = take(npart); L.red = take(3 * nred);
      L.lx = take(3 * N); L.lv = take(3 * N); L.LX = take(3); L.LV = take(3); L.gm = take(N);
      if (vjp) {
            L.ckpt = take(st * L.ncp);
            L.seg = take((size_t)L.C * (3 * N + 3));
      }
      if (jvp) {
            L.tx = take(3 * N); L.tv = take(3 * N); L.tm = take(N); L.tX = take(6); L.da = take(3 * N); L.dA = take(3);
            L.jpart = take(3 * N * L.nch);
      }
      L.box = take(6 * (size_t)L.ntiles);
      L.stage = take(3 * N);
      int *perm_dev = (int *)take((N + 1) / 2);
      L.perm = perm ? perm_dev : nullptr;
      int status = NCGPU_OK;
      cudaError_t e = cudaSuccess;
      const double h = a->dt / 2.0, dt = a->dt;
      const int nb = (n + 255) / 256;
      if (perm) NCG_CK(cudaMemcpyAsync(perm_dev, perm, sizeof(int) * N, cudaMemcpyHostToDevice, L.st));
      NCG_TRY(rows_in(L, L.X, a->x0, 3));
      NCG_TRY(rows_in(L, L.V, a->v0, 3));
      NCG_TRY(rows_in(L, L.m, a->m, 1));
      NCG_TRY(rows_in(L, L.sR, a->R, 1));
      NCG_CK(cudaMemcpyAsync(L.cm, a->cm, 6 * sizeof(double), cudaMemcpyHostToDevice, L.st));
      NCG_CK(cudaMemsetAsync(L.count, 0, sizeof(unsigned), L.st));
#define LF_TRY(call)                         \
      do {                                   \
            if ((status = (call)) != NCGPU_OK) goto done; \
      } while (0)
#define LF_LAUNCHED()                                                                 \
      do {                                                                            \
            note_launch();                                                            \
            cudaError_t e_ = cudaGetLastError();                                      \
            if (e_ != cudaSuccess) { status = cuda_fail(e_, "launch", __FILE__, __LINE__); goto done; } \
      } while (0)
      k_scale_R<<<(int)((NP + 255) / 256), 256, 0, L.st>>>(L.sR, sp, L.sR, n, L.sR32, (int)NP);
      LF_LAUNCHED();
      // (every input crosses before the first output, which may be the same array)
      if (vjp) LF_TRY(rows_in(L, L.lx, a->adj_x_final, 3));
      if (jvp) {
            LF_TRY(rows_in(L, L.tx, a->tan_x0, 3));
            LF_TRY(rows_in(L, L.tv, a->tan_v0, 3));
            LF_TRY(rows_in(L, L.tm, a->tan_m, 1));
            e = cudaMemsetAsync(L.tX, 0, 6 * sizeof(double), L.st);
            if (e != cudaSuccess) { status = cuda_fail(e, "tangent upload", __FILE__, __LINE__); goto done; }
            k_axpy3<<<nb, 256, 0, L.st>>>(h, L.tv, L.tx, n, n, nullptr, nullptr);
            LF_LAUNCHED();
      }
      // half drift (src/rk4.c:873-880)
      k_axpy3<<<nb, 256, 0, L.st>>>(h, L.V, L.X, n, n, L.cm + 3, L.central ? L.cm : nullptr);
      LF_LAUNCHED();
      for (int s = 0; s < a->nsteps; s++) {
            if (vjp && s % L.C == 0) {
                  double *ck = L.ckpt + st * (s / L.C);
                  e = cudaMemcpyAsync(ck, L.X, sizeof(double) * 6 * N, cudaMemcpyDeviceToDevice, L.st);
                  if (e == cudaSuccess) e = cudaMemcpyAsync(ck + 6 * N, L.cm, 6 * sizeof(double), cudaMemcpyDeviceToDevice, L.st);
                  if (e != cudaSuccess) { status = cuda_fail(e, "checkpoint", __FILE__, __LINE__); goto done; }
            }
            if (jvp) LF_TRY(lf_step_jvp(L, dt));
            else LF_TRY(lf_step(L, dt));
      }
      if (jvp) {
            k_xf<<<nb, 256, 0, L.st>>>(L.tx, L.tv, h, L.da, n);
            LF_LAUNCHED();
            LF_TRY(rows_out(L, a->tan_x_final, L.da, 3));
            e = cudaStreamSynchronize(L.st);
            if (e != cudaSuccess) { status = cuda_fail(e, "tangent download", __FILE__, __LINE__); goto done; }
      }
      if (a->x_final || a->v_final) {
            k_xf<<<nb, 256, 0, L.st>>>(L.X, L.V, h, L.out, n);  // half back-drift of the output (src/rk4.c:929-936)
            LF_LAUNCHED();
            if (a->x_final) LF_TRY(rows_out(L, a->x_final, L.out, 3));
            if (a->v_final) LF_TRY(rows_out(L, a->v_final, L.V, 3));
            e = cudaStreamSynchronize(L.st);
            if (e != cudaSuccess) { status = cuda_fail(e, "leapfrog download", __FILE__, __LINE__); goto done; }
      }
      if (vjp) {
            // x_F = x_n - h v_n
            e = cudaMemsetAsync(L.lv, 0, sizeof(double) * 3 * N, L.st);
            if (e == cudaSuccess) e = cudaMemsetAsync(L.LX, 0, 6 * sizeof(double), L.st);  // LX, LV
            if (e == cudaSuccess) e = cudaMemsetAsync(L.gm, 0, sizeof(double) * N, L.st);
            if (e != cudaSuccess) { status = cuda_fail(e, "adjoint init", __FILE__, __LINE__); goto done; }
            k_axpy3<<<nb, 256, 0, L.st>>>(-h, L.lx, L.lv, n, n, nullptr, nullptr);
            LF_LAUNCHED();
            for (int q = (a->nsteps - 1) / L.C; q >= 0 && a->nsteps > 0; q--) {
                  const int s0 = q * L.C, s1 = std::min(a->nsteps, s0 + L.C);
                  const double *ck = L.ckpt + st * q;
                  e = cudaMemcpyAsync(L.X, ck, sizeof(double) * 6 * N, cudaMemcpyDeviceToDevice, L.st);
                  if (e == cudaSuccess) e = cudaMemcpyAsync(L.cm, ck + 6 * N, 6 * sizeof(double), cudaMemcpyDeviceToDevice, L.st);
                  if (e != cudaSuccess) { status = cuda_fail(e, "restore", __FILE__, __LINE__); goto done; }
                  for (int s = s0; s < s1; s++) {  // recompute, keeping the positions each kick saw
                        LF_TRY(lf_step(L, dt, L.seg + (size_t)(s - s0) * (3 * N + 3)));
                  }
                  for (int s = s1 - 1; s >= s0; s--) {
                        // drift x_{s+1} = x_s + dt v_{s+1}, then kick v_{s+1} = v_s + dt a(x_s)
                        const double *sg = L.seg + (size_t)(s - s0) * (3 * N + 3);
                        LF_TRY(lf_vjp(L, sg, sg + 3 * N, dt));
                  }
            }
            // initial half drift x = x0 + h v0
            k_axpy3<<<nb, 256, 0, L.st>>>(h, L.lx, L.lv, n, n, nullptr, nullptr);
            LF_LAUNCHED();
            LF_TRY(rows_out(L, a->grad_x0, L.lx, 3));
            LF_TRY(rows_out(L, a->grad_v0, L.lv, 3));
            LF_TRY(rows_out(L, a->grad_m, L.gm, 1));
            e = cudaStreamSynchronize(L.st);
            if (e != cudaSuccess) { status = cuda_fail(e, "adjoint download", __FILE__, __LINE__); goto done; }
      }
#undef LF_TRY
#undef LF_LAUNCHED
done:
      cudaStreamSynchronize(L.st);
      return status;
}

// Morton order (30-bit keys from one cubic quantisation of the bounding box)
// of n positions given as 3n AoS doubles: perm[i] = the body at position i.
void morton_order(const double *x, int n, std::vector<int> &perm)
{
      double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
      for (int k = 0; k < n; k++)
            for (int d = 0; d < 3; d++) {
                  lo[d] = std::min(lo[d], x[3 * k + d]);
                  hi[d] = std::max(hi[d], x[3 * k + d]);
            }
      const double ext = std::max(std::max(hi[0] - lo[0], hi[1] - lo[1]), hi[2] - lo[2]);
      auto spread = [](uint32_t v) {  // bits 0..9 to 0, 3, ..., 27
            v = (v | (v << 16)) & 0x030000ffu;
            v = (v | (v << 8)) & 0x0300f00fu;
            v = (v | (v << 4)) & 0x030c30c3u;
            return (v | (v << 2)) & 0x09249249u;
      };
      // a stable radix sort, three digits of 10 bits (16,384 bodies: 0.2 ms; 1.6 ms
      // with the keys bit by bit and a comparison sort)
      constexpr int D = 1024;
      std::vector<uint32_t> key(n), kb(n);
      std::vector<int> pb(n), at(3 * D, 0);
      for (int k = 0; k < n; k++) {
            uint32_t m = 0;
            for (int d = 0; d < 3; d++) {
                  const double f = ext > 0. ? (x[3 * k + d] - lo[d]) / ext : 0.;
                  m |= spread((uint32_t)std::min(std::max((int)(f * 1023.999), 0), 1023)) << d;
            }
            key[k] = m;
            for (int q = 0; q < 3; q++) at[q * D + ((m >> (10 * q)) & (D - 1))]++;
      }
      perm.resize(n);
      for (int k = 0; k < n; k++) perm[k] = k;
      for (int q = 0; q < 3; q++) {
            int *c = &at[q * D], run = 0;
            for (int v = 0; v < D; v++) {
                  const int w = c[v];
                  c[v] = run;
                  run += w;
            }
            for (int k = 0; k < n; k++) {
                  const int to = c[(key[k] >> (10 * q)) & (D - 1)]++;
                  kb[to] = key[k];
                  pb[to] = perm[k];
            }
            key.swap(kb);
            perm.swap(pb);
      }
}

// The MIXED mode runs on the bodies in Morton order of their initial positions.
int lf_run(const struct ncgpu_leapfrog_args *a, int mode)
{
      if (ctx().P.par_gravity_mode != NCGPU_GRAVITY_MIXED) return lf_core(a, mode, false, nullptr);
      if (a->n <= 0 || !a->x0 || !a->v0 || !a->m || !a->R || !a->cm || a->nsteps < 0) return NCGPU_E_ARG;
      std::vector<int> perm;
      morton_order(a->x0, a->n, perm);
      return lf_core(a, mode, true, perm.data());
}

}  // namespace
}  // namespace ncg

using namespace ncg;

extern "C" int ncgpu_leapfrog(const struct ncgpu_leapfrog_args *args)
{
      reset_launches();
      if (!ctx().inited) return NCGPU_E_STATE;
      if (!args) return NCGPU_E_ARG;
      return lf_run(args, 0);
}

extern "C" int ncgpu_leapfrog_vjp(const struct ncgpu_leapfrog_args *args)
{
      reset_launches();
      if (!ctx().inited) return NCGPU_E_STATE;
      if (!args) return NCGPU_E_ARG;
      return lf_run(args, 1);
}

extern "C" int ncgpu_leapfrog_jvp(const struct ncgpu_leapfrog_args *args)
{
      reset_launches();
      if (!ctx().inited) return NCGPU_E_STATE;
      if (!args) return NCGPU_E_ARG;
      return lf_run(args, 2);
}
