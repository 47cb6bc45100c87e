// Pair sums that visit every unordered pair of bodies once: the force on both
// bodies of a pair comes from one difference, one distance and one reciprocal
// square root (Newton's third law).
//
// Bodies come in tiles of PT (Morton-ordered, so that a tile is compact), the
// tiles in blocks of B.  A work unit is a pair of blocks (b, c), c = b + k
// modulo the number of blocks nb, k = 0 .. nb/2 (for even nb and k = nb/2 only
// b < k): every unordered pair of blocks once.  A CTA takes one unit.  A warp
// holds a tile of b in its lanes ("rows", PT/32 bodies a lane) and walks the
// tiles of c ("columns"): at rotation r, lane l meets column body l + r (modulo
// 32; two of them, 32 apart, in the packed FP32 loop), so the lanes always meet
// different bodies, the row sums stay in the lane and the column sums move to the
// next lane with the rotation (a shuffle).  With B row tiles in a CTA, the warp of row tile r takes
// column tile (r + p) mod B in phase p, so no two warps add to one column tile in
// the same phase and the sums need no atomics: their order is fixed.  Each unit
// writes its row sums and its column sums to rows of a partial buffer of their
// own (pair_row), which the final pass adds in order of k: deterministic.
//
// Operations per unordered pair in FP32: 16 lane operations and one rsqrt (and
// 0.75 for the column sums' last addition), against 24 and two when each side is
// summed by itself; in FP64 24 against 40.  Measured, whole force evaluations
// before (each side by itself) and now: mixed 2,109 -> 1,690 us at 65,536 bodies,
// 29.4 -> 22.7 ms at 262,144; FP64 1,164 -> 805 us at 27,000.
#pragma once
#include "common.cuh"

namespace ncg {

constexpr int PT = 128;      // bodies per tile
constexpr int PU = PT / 32;  // row bodies a lane, and 32-body column groups a tile
// The tile pairs summed in FP64 reach 1.45 near_theta here: 1 % of the time at
// 65,536 bodies, for 5 % of the error (see far_group).
constexpr double PAIR_NEAR = 1.45;

struct alignas(16) D4 { double x, y, z, w; };

// The tiles' data: FP64 records (x, y, z, m), softening * radius; the FP32 copy
// relative to each tile's box centre, x[PT] y[PT] z[PT] m[PT] a tile (padding at
// 1e18, massless); the boxes (centre, half extents).
struct PairData {
      const D4 *s64;
      const double *sR64;
      const float *s32;
      const float *sR32;
      const double *box;
      int n, ntiles, nb;
};

// The number of block offsets k of nb blocks.
__host__ __device__ __forceinline__ int pair_offsets(int nb) { return nb / 2 + 1; }

// Whether block b's unit at offset k exists (even nb: the opposite blocks meet once).
__host__ __device__ __forceinline__ bool pair_unit(int nb, int b, int k) { return 2 * k != nb || k == 0 || b < k; }

// Whether the partial row (offset k, side: 0 row sums, 1 column sums) holds a value for block `blk`.
__device__ __forceinline__ bool pair_row(int nb, int blk, int k, int side)
{
      return 2 * k != nb || k == 0 || (side == 0 ? blk < k : blk >= k);
}

// What phase p of a CTA's row tile r does with a unit of offset k: 0 nothing
// (the diagonal unit takes each pair of its tiles once), 1 the tile with
// itself, 2 a pair of tiles.
__device__ __forceinline__ int pair_phase(int B, int k, int r, int p)
{
      if (k != 0) return 2;
      if (p == 0) return 1;
      return 2 * p < B || (2 * p == B && r < p) ? 2 : 0;
}

// One row body (both halves of XT .. MT alike) against two column bodies packed
// in XS .. MS: the row sums get m_c d / D^3, the column sums m_r d / D^3 with d
// from row to column (the column's force is minus its sum).  FIRST: the column
// sums start here.
template <int SM, bool FIRST>
__device__ __forceinline__ void pair_sym(f2 XS, f2 YS, f2 ZS, f2 MS, f2 RS, f2 XT, f2 YT, f2 ZT, f2 MT, f2 RT, f2 E,
                                         f2 (&row)[3], f2 (&col)[3])
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
      const f2 i3 = f2_mul(f2_mul(i, i), i);
      const f2 wr = f2_mul(MS, i3), wc = f2_mul(MT, i3);
      row[0] = f2_fma(wr, dx, row[0]);
      row[1] = f2_fma(wr, dy, row[1]);
      row[2] = f2_fma(wr, dz, row[2]);
      col[0] = FIRST ? f2_mul(wc, dx) : f2_fma(wc, dx, col[0]);
      col[1] = FIRST ? f2_mul(wc, dy) : f2_fma(wc, dy, col[1]);
      col[2] = FIRST ? f2_mul(wc, dz) : f2_fma(wc, dz, col[2]);
}

__device__ __forceinline__ f2 f2_shfl(f2 v, int src)
{
      return __shfl_sync(0xffffffffu, v, src);
}

// A far group's columns in shared memory: slot p the bodies p and p + 32 of the
// 64, every slot twice in a row, so that lane l reads slot (l + r) mod 32 at
// l + r; 16-byte strides (no bank conflicts).
template <int SOFT>
struct PairGroup {
      ulonglong2 xy[64];   // x pair, y pair
      ulonglong2 zm[64];   // z pair, m pair
      f2 R[SOFT == 2 ? 64 : 1];
};

// Far tiles, one group of 64 column bodies against the lane's PU rows.  FP32 sums:
// the rows' over 16 rotations (16 terms a half), the columns' over a visit's four
// rows and then over 8 rotations; both are then added to the FP64 ones (rs, col).
// Those runs and PAIR_NEAR keep the error at or below that of sums of 32 terms a
// half on each side by itself (2-norm against FP64, 8 disks each: 2.3e-9 against
// 2.5e-9 at 65,536 bodies, 2.5e-9 against 2.6e-9 at 250,007); column sums of 32
// terms would be 2 % faster and 6 % less exact.
// Measured on the loop alone, cycles per 4 rows x 32 columns and scheduler (the
// packed arithmetic's floor is 64): 84.9 with the columns packed, 89.5 with the
// rows packed (a shuffle then moves half as much); without the 12 accumulating
// FMAs 53, without shuffles 84, without shared loads and rsqrt 86.
template <int SM>
__device__ __forceinline__ void far_group(const PairGroup<SM> &st, int lane, const f2 (&XT)[PU], const f2 (&YT)[PU],
                                          const f2 (&ZT)[PU], const f2 (&MT)[PU], const f2 (&RT)[PU], f2 E,
                                          double *__restrict__ rs, int rstride, double *__restrict__ col, int cstride)
{
      f2 row[PU][3];
#pragma unroll
      for (int u = 0; u < PU; u++) row[u][0] = row[u][1] = row[u][2] = 0ull;
      const int nxt = (lane + 1) & 31;
#pragma unroll 2
      for (int r0 = 0; r0 < 32; r0 += 8) {
            f2 c[3] = {0ull, 0ull, 0ull};
#pragma unroll
            for (int r = 0; r < 8; r++) {
                  const int p = lane + r0 + r;
                  const ulonglong2 a = st.xy[p], b = st.zm[p];
                  const f2 R = SM == 2 ? st.R[SM == 2 ? p : 0] : 0ull;
                  f2 v[3];
                  pair_sym<SM, true>(a.x, a.y, b.x, b.y, R, XT[0], YT[0], ZT[0], MT[0], RT[0], E, row[0], v);
#pragma unroll
                  for (int u = 1; u < PU; u++)
                        pair_sym<SM, false>(a.x, a.y, b.x, b.y, R, XT[u], YT[u], ZT[u], MT[u], RT[u], E, row[u], v);
#pragma unroll
                  for (int d = 0; d < 3; d++) {
                        c[d] = f2_add(c[d], v[d]);
                        if (r < 7) c[d] = f2_shfl(c[d], nxt);
                  }
            }
            const int j = (lane + r0 + 7) & 31;
#pragma unroll
            for (int d = 0; d < 3; d++) {
                  float lo, hi;
                  f2_unpack(c[d], lo, hi);
                  col[d * cstride + j] -= (double)lo;
                  col[d * cstride + j + 32] -= (double)hi;
            }
            __syncwarp();
            if (r0 & 8) {
#pragma unroll
                  for (int u = 0; u < PU; u++)
#pragma unroll
                        for (int d = 0; d < 3; d++) {
                              float lo, hi;
                              f2_unpack(row[u][d], lo, hi);
                              rs[(3 * u + d) * rstride] += (double)lo + (double)hi;
                              row[u][d] = 0ull;
                        }
            }
      }
}

// FP64 pair sums of one group of 32 column bodies, first body j0.  SELF: the
// row tile's own bodies as columns: row sums only, a body's own term left out.
template <int SOFT, bool SELF>
__device__ __forceinline__ void near_group(const PairData &P, int j0, int i0, int lane, const D4 (&me)[PU],
                                           const double (&rme)[PU], double eps2, double (&acc)[PU][3],
                                           double *__restrict__ col, int cstride)
{
      double c[3] = {0., 0., 0.};
      const int nxt = (lane + 1) & 31;
#pragma unroll 1
      for (int r = 0; r < 32; r++) {
            const int j = j0 + ((lane + r) & 31);
            const bool in = j < P.n;
            D4 s = P.s64[in ? j : 0];
            const double sj = SOFT == 2 ? P.sR64[in ? j : 0] : 0.;
            if (!in) {  // padding: far from everything, massless
                  s.x = s.y = s.z = 1e18;
                  s.w = 0.;
            }
#pragma unroll
            for (int u = 0; u < PU; u++) {
                  const double dx = s.x - me[u].x, dy = s.y - me[u].y, dz = s.z - me[u].z;
                  double r2 = SOFT == 1 ? eps2 : 0.;
                  if (SOFT == 2) {
                        const double e = rme[u] + sj;
                        r2 = e * e;
                  }
                  r2 = fma(dx, dx, fma(dy, dy, fma(dz, dz, r2)));
                  const double ri = rsqrt(r2);
                  const double i3 = ri * ri * ri;
                  const double w = SELF && j == i0 + lane + 32 * u ? 0. : s.w * i3;
                  acc[u][0] = fma(w, dx, acc[u][0]);
                  acc[u][1] = fma(w, dy, acc[u][1]);
                  acc[u][2] = fma(w, dz, acc[u][2]);
                  if (!SELF) {
                        const double wc = me[u].w * i3;
                        c[0] = fma(wc, dx, c[0]);
                        c[1] = fma(wc, dy, c[1]);
                        c[2] = fma(wc, dz, c[2]);
                  }
            }
            if (!SELF)
#pragma unroll
                  for (int d = 0; d < 3; d++) c[d] = __shfl_sync(0xffffffffu, c[d], nxt);
      }
      if (!SELF) {  // after 32 shuffles the sums are back at their own lane
#pragma unroll
            for (int d = 0; d < 3; d++) col[d * cstride + lane] -= c[d];
            __syncwarp();
      }
}

// Shared memory of a unit: the column sums, the lanes' row sums and (MODE 0) the
// column block's FP32 groups.
template <int MODE, int SOFT, int B, int W>
constexpr size_t pair_smem()
{
      return (3 * B * PT + 3 * PU * 32 * W) * sizeof(double) + (MODE == 0 ? 2 * B * sizeof(PairGroup<SOFT>) : 0);
}

// One CTA of W warps = one unit.  MODE 0: mixed (FP32 far tile pairs, FP64 near
// ones), 1: all FP64.  SOFT 0: none, 1: uniform eps^2, 2: eps = sum of the two
// softening * radius.  With fewer row tiles than warps (B < W), two warps share a
// row tile and take a column tile's two groups.
// part: rows of 3 * npad doubles, row 2 (k - k0) the row sums of offset k, row
// 2 (k - k0) + 1 its column sums.
template <int MODE, int SOFT, int B, int W>
__global__ void __launch_bounds__(32 * W, 16 / W) k_pair_sym(PairData P, int k0, double theta, double eps2,
                                                             double *__restrict__ part, long npad)
{
      constexpr int H = W / B;    // warps a row tile: 1 or 2
      constexpr int NG = 2 / H;   // 64-column groups a warp takes of each column tile
      constexpr int NB = B * PT, TH = 32 * W;
      extern __shared__ __align__(16) unsigned char pair_sm[];
      double *col = reinterpret_cast<double *>(pair_sm), *rows = col + 3 * NB;
      PairGroup<SOFT> *st = reinterpret_cast<PairGroup<SOFT> *>(rows + 3 * PU * TH);  // (MODE 0)
      const int b = blockIdx.x, k = k0 + blockIdx.y;
      if (!pair_unit(P.nb, b, k)) return;
      const int c = b + k < P.nb ? b + k : b + k - P.nb;
      const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
      const int r = warp % B, h = warp / B;
      const int I = b * B + r, i0 = I * PT;
      for (int q = tid; q < 3 * NB; q += TH) col[q] = 0.;
      for (int q = 0; q < 3 * PU; q++) rows[q * TH + tid] = 0.;
      if (MODE == 0)
            for (int q = tid; q < 2 * B * 32; q += TH) {
                  const int t = q / 64, g = (q / 32) & 1, s = q & 31, J = c * B + t;
                  if (J >= P.ntiles) continue;
                  const float *v = P.s32 + (size_t)J * 4 * PT + 64 * g + s;
                  PairGroup<SOFT> &G = st[2 * t + g];
                  const ulonglong2 xy = make_ulonglong2(f2_pack(v[0], v[32]), f2_pack(v[PT], v[PT + 32]));
                  const ulonglong2 zm =
                      make_ulonglong2(f2_pack(v[2 * PT], v[2 * PT + 32]), f2_pack(v[3 * PT], v[3 * PT + 32]));
                  G.xy[s] = G.xy[s + 32] = xy;
                  G.zm[s] = G.zm[s + 32] = zm;
                  if (SOFT == 2) {
                        const float *e = P.sR32 + (size_t)J * PT + 64 * g + s;
                        G.R[s] = G.R[SOFT == 2 ? s + 32 : 0] = f2_pack(e[0], e[32]);
                  }
            }
      __syncthreads();
#pragma unroll 1
      for (int p = 0; p < B; p++) {
            const int t = r + p < B ? r + p : r + p - B, J = c * B + t;
            const int what = I < P.ntiles && J < P.ntiles ? pair_phase(B, k, r, p) : 0;
            if (what != 0) {
                  D4 me[PU];
                  double rme[PU];
#pragma unroll
                  for (int u = 0; u < PU; u++) {
                        const int i = i0 + lane + 32 * u;
                        const bool in = i < P.n;
                        me[u] = P.s64[in ? i : 0];
                        rme[u] = SOFT == 2 ? P.sR64[in ? i : 0] : 0.;
                        if (!in) {  // (opposite the columns' padding)
                              me[u].x = me[u].y = me[u].z = -1e18;
                              me[u].w = 0.;
                        }
                  }
                  const double *bj = P.box + 6 * J;
                  double *cl = col + t * PT, *rs = rows + tid;
                  if (MODE == 1 || what == 1 || tiles_near(P.box + 6 * I, bj, PAIR_NEAR * theta)) {
                        double acc[PU][3];
#pragma unroll
                        for (int u = 0; u < PU; u++) acc[u][0] = acc[u][1] = acc[u][2] = 0.;
#pragma unroll 1
                        for (int g = 2 * h * NG; g < 2 * (h + 1) * NG; g++) {
                              if (what == 1)
                                    near_group<SOFT, true>(P, J * PT + 32 * g, i0, lane, me, rme, eps2, acc,
                                                           cl + 32 * g, NB);
                              else
                                    near_group<SOFT, false>(P, J * PT + 32 * g, i0, lane, me, rme, eps2, acc,
                                                            cl + 32 * g, NB);
                        }
#pragma unroll
                        for (int u = 0; u < PU; u++)
#pragma unroll
                              for (int d = 0; d < 3; d++) rs[(3 * u + d) * TH] += acc[u][d];
                  } else {
                        // coordinates relative to the column tile's centre
                        f2 XT[PU], YT[PU], ZT[PU], MT[PU], RT[PU];
#pragma unroll
                        for (int u = 0; u < PU; u++) {
                              const float x = (float)(me[u].x - bj[0]), y = (float)(me[u].y - bj[1]);
                              const float z = (float)(me[u].z - bj[2]), m = (float)me[u].w, e = (float)rme[u];
                              XT[u] = f2_pack(x, x);
                              YT[u] = f2_pack(y, y);
                              ZT[u] = f2_pack(z, z);
                              MT[u] = f2_pack(m, m);
                              RT[u] = SOFT == 2 ? f2_pack(e, e) : 0ull;
                        }
                        const f2 E = f2_pack((float)eps2, (float)eps2);
#pragma unroll 1
                        for (int g = h * NG; g < (h + 1) * NG; g++)
                              far_group<SOFT>(st[2 * t + g], lane, XT, YT, ZT, MT, RT, E, rs, TH, cl + 64 * g, NB);
                  }
            }
            __syncthreads();  // the next phase's warp of each column tile; the sums are complete
      }
      double *prow = part + (size_t)(2 * blockIdx.y) * 3 * npad, *pcol = prow + 3 * npad;
      for (int q = tid; q < NB; q += TH) {
            const int at = (q % 32) + 32 * (q / PT), u = (q % PT) / 32;
            for (int d = 0; d < 3; d++) {
                  double v = rows[(3 * u + d) * TH + at];
                  if (H == 2) v += rows[(3 * u + d) * TH + at + 32 * B];
                  prow[d * npad + (long)b * NB + q] = v;
                  pcol[d * npad + (long)c * NB + q] = col[d * NB + q];
            }
      }
}

// The partial rows of offsets k0 .. k0 + nk - 1 for body q of block blk (32
// bodies a CTA of 256 threads: thread group g adds rows g, g + 8, ...; the
// groups' sums are added in order): v[d] for the threads of group 0.
__device__ __forceinline__ void pair_rows_sum(const double *__restrict__ part, long npad, int nb, int blk, int k0,
                                              int nk, long q, bool live, double (*sh)[8][32], double (&v)[3])
{
      const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
      double s[3] = {0., 0., 0.};
      if (live) {
#pragma unroll 4
            for (int row = g; row < 2 * nk; row += 8) {
                  const bool has = pair_row(nb, blk, k0 + (row >> 1), row & 1);
                  const double *p = part + (size_t)row * 3 * npad + q;
#pragma unroll
                  for (int d = 0; d < 3; d++) s[d] += has ? p[d * npad] : 0.;
            }
      }
#pragma unroll
      for (int d = 0; d < 3; d++) sh[d][g][lane] = s[d];
      __syncthreads();
      if (g == 0)
#pragma unroll
            for (int d = 0; d < 3; d++) {
                  v[d] = sh[d][0][lane];
                  for (int e = 1; e < 8; e++) v[d] += sh[d][e][lane];
            }
}

}  // namespace ncg
