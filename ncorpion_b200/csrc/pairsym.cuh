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
      // OP 1: the adjoint velocities lambda (3 blocks of n) and their FP32 copy,
      // x[PT] y[PT] z[PT] a tile (zero padding)
      const double *l64;
      const float *l32;
};

// 0 for two near tiles (boxes bi, bj; tiles_near's test); for far ones the power of two
// that brings their distances near 1, so that neither the cubes and fifth powers of their
// reciprocals nor their squares leave FP32's range, whatever the caller's unit of length;
// the sums are scaled back as they go to FP64, exact both ways.  1 where the distances
// are near 1 as they are (2^20 either way; 2^12 for the fifth powers), which they are in
// most units: that loop's differences are subtractions, with an operand less (65,536
// bodies 1,675 us a call against 1,718 with the scale in every pair, 262,144 22.8 ms
// against 23.8).  Else the exponent is halfway between those of the smallest and the
// largest distance, softened: 2^42 (2^25) either way of it is in range.  At most 2^64, so
// that the padding at 1e18 stays finite.  eps2: the squared softening length (SOFT 1) or
// its largest (SOFT 2).
template <int SOFT, int OP>
__device__ __forceinline__ float far_scale(const double *__restrict__ bi, const double *__restrict__ bj, double theta,
                                           double eps2)
{
      double g2 = 0., di = 0., dj = 0.;
      int lo = 0, hi = 0;  // high words of the largest gap and the largest distance along an axis
#pragma unroll
      for (int d = 0; d < 3; d++) {
            const double c = fabs(bi[d] - bj[d]), gap = c - bi[3 + d] - bj[3 + d];
            if (gap > 0.) g2 += gap * gap;
            di += bi[3 + d] * bi[3 + d];
            dj += bj[3 + d] * bj[3 + d];
            lo = max(lo, __double2hiint(gap));
            hi = max(hi, __double2hiint(c + (bi[3 + d] + bj[3 + d])));
      }
      if (g2 < theta * theta * (4. * fmax(di, dj))) return 0.f;
      int el = (lo >> 20) - 1023, eh = (hi >> 20) - 1023;
      if (SOFT != 0) {
            const int es = ((__double2hiint(eps2) >> 20) - 1023) >> 1;
            eh = max(eh, es);
            if (SOFT == 1) el = max(el, es);
      }
      constexpr int IN = OP == 0 ? 20 : 12;
      if (el >= -IN && eh < IN) return 1.f;
      if (el <= -1023) el = eh;  // no lower bound
      return __int_as_float((127 - max(-64, min(120, (eh + el) >> 1))) << 23);
}

// What a pair adds.  OP 0: the force, three sums a body.  OP 1: the force's
// vector-Jacobian product with the bodies' lambda, four sums a body: with r from
// row k to column j and w = m_k lambda_j - m_j lambda_k, t = w / D^3 - 3 r (r . w) / D^5
// to the row and -t to the column (the mutual tidal term is antisymmetric), and
// -(lambda_j . r) / D^3 and +(lambda_k . r) / D^3 (the masses' gradients).
template <int OP>
constexpr int PAIR_OUT = OP == 0 ? 3 : 4;
template <int OP>
constexpr int PAIR_ROWS = OP == 0 ? PU : 2;  // rows a lane takes at a time (registers)

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

// The squared distance, softened.  SC: RS in the caller's unit, the rest times S.
template <int SM, bool SC>
__device__ __forceinline__ f2 pair_dist2(f2 dx, f2 dy, f2 dz, f2 RS, f2 RT, f2 E, f2 S)
{
      f2 q;
      if (SM == 0) {
            q = f2_mul(dx, dx);
      } else if (SM == 1) {
            q = f2_fma(dx, dx, E);
      } else {
            const f2 e = SC ? f2_fma(RS, S, RT) : f2_add(RS, RT);
            q = f2_fma(dx, dx, f2_mul(e, e));
      }
      q = f2_fma(dy, dy, q);
      return f2_fma(dz, dz, q);
}

__device__ __forceinline__ f2 f2_shfl(f2 v, int src)
{
      return __shfl_sync(0xffffffffu, v, src);
}

// A far group's columns in shared memory: slot p the bodies p and p + 32 of the
// 64, every slot twice in a row, so that lane l reads slot (l + r) mod 32 at
// l + r; 16-byte strides (no bank conflicts).
template <int SOFT, int OP>
struct PairGroup {
      ulonglong2 xy[64];   // x pair, y pair
      ulonglong2 zm[64];   // z pair, m pair
      ulonglong2 l[OP == 1 ? 64 : 1];  // lambda's x pair, y pair
      f2 lz[OP == 1 ? 64 : 2];
      f2 R[SOFT == 2 ? 64 : 2];
};

// A lane's rows, packed: both halves alike.  -x, -y, -z and R times the tile pair's scale.
template <int OP, int RU>
struct PairRows {
      f2 nx[RU], ny[RU], nz[RU], m[RU], R[RU];
      f2 nlx[RU], nly[RU], nlz[RU];  // -lambda (OP 1)
};

// One row body against two column bodies packed.  OP 0: the row sums get
// m_c d / D^3, the column sums m_r d / D^3 with d from row to column (the column's
// force is minus its sum).  OP 1: t to both; row[3] and col[3] the masses' terms
// (both are subtracted).  FIRST: the column sums start here.  SC: lengths are multiplied
// by the power of two S (far_scale).
template <int SM, int OP, bool SC, bool FIRST, int RU>
__device__ __forceinline__ void pair_sym(ulonglong2 xy, ulonglong2 zm, f2 RS, ulonglong2 l, f2 lz,
                                         const PairRows<OP, RU> &T, int u, f2 E, f2 S,
                                         f2 (&row)[PAIR_OUT<OP>], f2 (&col)[PAIR_OUT<OP>])
{
      const f2 dx = SC ? f2_fma(xy.x, S, T.nx[u]) : f2_add(xy.x, T.nx[u]);
      const f2 dy = SC ? f2_fma(xy.y, S, T.ny[u]) : f2_add(xy.y, T.ny[u]);
      const f2 dz = SC ? f2_fma(zm.x, S, T.nz[u]) : f2_add(zm.x, T.nz[u]);
      const f2 i = f2_rsqrt(pair_dist2<SM, SC>(dx, dy, dz, RS, T.R[u], E, S));
      const f2 ii = f2_mul(i, i), i3 = f2_mul(ii, i);
      if constexpr (OP == 0) {
            const f2 wr = f2_mul(zm.y, i3), wc = f2_mul(T.m[u], i3);
            row[0] = f2_fma(wr, dx, row[0]);
            row[1] = f2_fma(wr, dy, row[1]);
            row[2] = f2_fma(wr, dz, row[2]);
            col[0] = FIRST ? f2_mul(wc, dx) : f2_fma(wc, dx, col[0]);
            col[1] = FIRST ? f2_mul(wc, dy) : f2_fma(wc, dy, col[1]);
            col[2] = FIRST ? f2_mul(wc, dz) : f2_fma(wc, dz, col[2]);
      } else {
            const f2 mj = zm.y, mk = T.m[u], i5 = f2_mul(i3, ii);
            const f2 wx = f2_fma(mj, T.nlx[u], f2_mul(mk, l.x)), wy = f2_fma(mj, T.nly[u], f2_mul(mk, l.y));
            const f2 wz = f2_fma(mj, T.nlz[u], f2_mul(mk, lz));
            const f2 rw = f2_fma(dz, wz, f2_fma(dy, wy, f2_mul(dx, wx)));
            const f2 nc = f2_mul(f2_mul(f2_pack(-3.f, -3.f), rw), i5);
            const f2 tx = f2_fma(dx, nc, f2_mul(wx, i3)), ty = f2_fma(dy, nc, f2_mul(wy, i3));
            const f2 tz = f2_fma(dz, nc, f2_mul(wz, i3));
            const f2 lj = f2_fma(lz, dz, f2_fma(l.y, dy, f2_mul(l.x, dx)));
            const f2 nk = f2_fma(T.nlz[u], dz, f2_fma(T.nly[u], dy, f2_mul(T.nlx[u], dx)));
            row[0] = f2_add(row[0], tx);
            row[1] = f2_add(row[1], ty);
            row[2] = f2_add(row[2], tz);
            row[3] = f2_fma(lj, i3, row[3]);
            col[0] = FIRST ? tx : f2_add(col[0], tx);
            col[1] = FIRST ? ty : f2_add(col[1], ty);
            col[2] = FIRST ? tz : f2_add(col[2], tz);
            col[3] = FIRST ? f2_mul(nk, i3) : f2_fma(nk, i3, col[3]);
      }
}

// Far tiles, one group of 64 column bodies against RU of the lane's rows.  FP32
// sums: the rows' over 16 rotations (16 terms a half), the columns' over a visit's
// rows and then over 8 rotations; both are then added to the FP64 ones (rs, col).
// Those runs and PAIR_NEAR keep the force's error at or below that of sums of 32
// terms a half on each side by itself (2-norm against FP64, 8 disks each: 2.3e-9
// against 2.5e-9 at 65,536 bodies, 2.5e-9 against 2.6e-9 at 250,007); column sums
// of 32 terms would be 2 % faster and 6 % less exact.
// Measured on the force's loop alone, cycles per 4 rows x 32 columns and scheduler
// (the packed arithmetic's floor is 64): 84.9 with the columns packed, 89.5 with
// the rows packed (a shuffle then moves half as much); without the 12 accumulating
// FMAs 53, without shuffles 84, without shared loads and rsqrt 86.
template <int SM, int OP, bool SC, int RU>
__device__ __forceinline__ void far_group(const PairGroup<SM, OP> &st, int lane, const PairRows<OP, RU> &T, f2 E,
                                          f2 S, const double (&back)[2], double *__restrict__ rs, int rstride, double *__restrict__ col, int cstride)
{
      constexpr int NO = PAIR_OUT<OP>;
      f2 row[RU][NO];
#pragma unroll
      for (int u = 0; u < RU; u++)
#pragma unroll
            for (int d = 0; d < NO; d++) row[u][d] = 0ull;
      const int nxt = (lane + 1) & 31;
#pragma unroll(OP == 0 ? 2 : 1)
      for (int r0 = 0; r0 < 32; r0 += 8) {
            f2 c[NO];
#pragma unroll
            for (int d = 0; d < NO; d++) c[d] = 0ull;
#pragma unroll
            for (int r = 0; r < 8; r++) {
                  const int p = lane + r0 + r;
                  const ulonglong2 xy = st.xy[p], zm = st.zm[p];
                  const ulonglong2 l = OP == 1 ? st.l[OP == 1 ? p : 0] : make_ulonglong2(0ull, 0ull);
                  const f2 lz = OP == 1 ? st.lz[OP == 1 ? p : 0] : 0ull;
                  const f2 R = SM == 2 ? st.R[SM == 2 ? p : 0] : 0ull;
                  f2 v[NO];
                  pair_sym<SM, OP, SC, true>(xy, zm, R, l, lz, T, 0, E, S, row[0], v);
#pragma unroll
                  for (int u = 1; u < RU; u++) pair_sym<SM, OP, SC, false>(xy, zm, R, l, lz, T, u, E, S, row[u], v);
#pragma unroll
                  for (int d = 0; d < NO; d++) {
                        c[d] = f2_add(c[d], v[d]);
                        if (r < 7) c[d] = f2_shfl(c[d], nxt);
                  }
            }
            const int j = (lane + r0 + 7) & 31;
#pragma unroll
            for (int d = 0; d < NO; d++) {
                  float lo, hi;
                  f2_unpack(c[d], lo, hi);
                  col[d * cstride + j] -= SC ? (double)lo * back[d / 3] : (double)lo;
                  col[d * cstride + j + 32] -= SC ? (double)hi * back[d / 3] : (double)hi;
            }
            __syncwarp();
            if (r0 & 8) {
#pragma unroll
                  for (int u = 0; u < RU; u++)
#pragma unroll
                        for (int d = 0; d < NO; d++) {
                              float lo, hi;
                              f2_unpack(row[u][d], lo, hi);
                              const double v = SC ? ((double)lo + (double)hi) * back[d / 3] : (double)lo + (double)hi;
                              rs[(NO * u + d) * rstride] += d < 3 ? v : -v;
                              row[u][d] = 0ull;
                        }
            }
      }
}

// RU of a lane's rows in FP64: bodies i + 32 u (padding opposite the columns').
template <int SOFT, int OP, int RU>
struct PairRows64 {
      D4 me[RU];
      double R[RU], l[OP == 1 ? RU : 1][3];

      __device__ __forceinline__ void load(const PairData &P, int i)
      {
#pragma unroll
            for (int u = 0; u < RU; u++) {
                  const int k = i + 32 * u;
                  const bool in = k < P.n;
                  me[u] = P.s64[in ? k : 0];
                  R[u] = SOFT == 2 ? P.sR64[in ? k : 0] : 0.;
                  if (!in) {
                        me[u].x = me[u].y = me[u].z = -1e18;
                        me[u].w = 0.;
                  }
                  if constexpr (OP == 1)
#pragma unroll
                        for (int d = 0; d < 3; d++) l[u][d] = in ? P.l64[(size_t)d * P.n + k] : 0.;
            }
      }
};

// FP64 pair sums of one group of 32 column bodies, first body j0, for the rows of
// T, first body i.  SELF: the row tile's own bodies as columns: row sums only, a
// body's own term left out.
template <int SOFT, int OP, bool SELF, int RU>
__device__ __forceinline__ void near_group(const PairData &P, int j0, int i, int lane,
                                           const PairRows64<SOFT, OP, RU> &T, double eps2,
                                           double (&acc)[RU][PAIR_OUT<OP>], double *__restrict__ col, int cstride)
{
      constexpr int NO = PAIR_OUT<OP>;
      double c[NO];
#pragma unroll
      for (int d = 0; d < NO; d++) c[d] = 0.;
      const int nxt = (lane + 1) & 31;
      // (two rotations at once, the next column's load and shuffle behind the FP64 chain:
      // FP64 65,536 3.78 -> 3.75 ms, 30,011 with general radii 1.03 -> 1.01)
#pragma unroll 2
      for (int r = 0; r < 32; r++) {
            const int j = j0 + ((lane + r) & 31);
            const bool in = j < P.n;
            D4 s = P.s64[in ? j : 0];
            const double sj = SOFT == 2 ? P.sR64[in ? j : 0] : 0.;
            double lx = 0., ly = 0., lz = 0.;
            if (OP == 1 && in) {
                  lx = P.l64[j];
                  ly = P.l64[(size_t)P.n + j];
                  lz = P.l64[2 * (size_t)P.n + j];
            }
            if (!in) {  // padding: far from everything, massless
                  s.x = s.y = s.z = 1e18;
                  s.w = 0.;
            }
#pragma unroll
            for (int u = 0; u < RU; u++) {
                  const double dx = s.x - T.me[u].x, dy = s.y - T.me[u].y, dz = s.z - T.me[u].z;
                  double r2 = SOFT == 1 ? eps2 : 0.;
                  if (SOFT == 2) {
                        const double e = T.R[u] + sj;
                        r2 = e * e;
                  }
                  r2 = fma(dx, dx, fma(dy, dy, fma(dz, dz, r2)));
                  const double ri = rsqrt(r2);
                  const bool own = SELF && j == i + 32 * u;
                  if constexpr (OP == 0) {
                        const double i3 = ri * ri * ri;
                        const double w = own ? 0. : s.w * i3;
                        acc[u][0] = fma(w, dx, acc[u][0]);
                        acc[u][1] = fma(w, dy, acc[u][1]);
                        acc[u][2] = fma(w, dz, acc[u][2]);
                        if (!SELF) {
                              const double wc = T.me[u].w * i3;
                              c[0] = fma(wc, dx, c[0]);
                              c[1] = fma(wc, dy, c[1]);
                              c[2] = fma(wc, dz, c[2]);
                        }
                  } else {
                        const double ii = own ? 0. : ri * ri, i3 = own ? 0. : ii * ri, i5 = i3 * ii;
                        const double mj = s.w, mk = T.me[u].w;
                        const double wx = mk * lx - mj * T.l[u][0], wy = mk * ly - mj * T.l[u][1];
                        const double wz = mk * lz - mj * T.l[u][2];
                        const double cc = 3.0 * (dx * wx + dy * wy + dz * wz) * i5;
                        const double tx = wx * i3 - dx * cc, ty = wy * i3 - dy * cc, tz = wz * i3 - dz * cc;
                        acc[u][0] += tx;
                        acc[u][1] += ty;
                        acc[u][2] += tz;
                        acc[u][3] -= (lx * dx + ly * dy + lz * dz) * i3;
                        if (!SELF) {
                              c[0] += tx;
                              c[1] += ty;
                              c[2] += tz;
                              c[3] -= (T.l[u][0] * dx + T.l[u][1] * dy + T.l[u][2] * dz) * i3;
                        }
                  }
            }
            if (!SELF)
#pragma unroll
                  for (int d = 0; d < NO; d++) c[d] = __shfl_sync(0xffffffffu, c[d], nxt);
      }
      if (!SELF) {  // after 32 shuffles the sums are back at their own lane
#pragma unroll
            for (int d = 0; d < NO; d++) col[d * cstride + lane] -= c[d];
            __syncwarp();
      }
}

// Shared memory of a unit: the column sums, the lanes' row sums and (MODE 0) the
// column block's FP32 groups.
template <int MODE, int SOFT, int OP, int B, int W>
constexpr size_t pair_smem()
{
      return PAIR_OUT<OP> * (B * PT + PU * 32 * W) * sizeof(double) +
             (MODE == 0 ? 2 * B * sizeof(PairGroup<SOFT, OP>) : 0);
}

// One CTA of W warps = one unit.  MODE 0: mixed (FP32 far tile pairs, FP64 near
// ones), 1: all FP64.  SOFT 0: none, 1: uniform eps^2, 2: eps = sum of the two
// softening * radius.  With fewer row tiles than warps (B < W), two or four warps
// share a row tile and the groups of a column tile.
// part: rows of PAIR_OUT * npad doubles, row 2 (k - k0) the row sums of offset k,
// row 2 (k - k0) + 1 its column sums.
template <int MODE, int SOFT, int OP, int B, int W>
__global__ void __launch_bounds__(32 * W, 16 / W) k_pair_sym(PairData P, int k0, double theta, double eps2,
                                                             double *__restrict__ part, long npad)
{
      constexpr int NO = PAIR_OUT<OP>, RU = PAIR_ROWS<OP>;
      constexpr int H = W / B;              // warps a row tile: 1, 2 or 4
      constexpr int NG = H == 1 ? 2 : 1;    // 64-column groups a warp takes of each far column tile
      constexpr int NN = PU / H;            // 32-column groups of each near one
      constexpr int NB = B * PT, TH = 32 * W;
      extern __shared__ __align__(16) unsigned char pair_sm[];
      double *col = reinterpret_cast<double *>(pair_sm), *rows = col + NO * NB;
      PairGroup<SOFT, OP> *st = reinterpret_cast<PairGroup<SOFT, OP> *>(rows + NO * PU * TH);  // (MODE 0)
      const int b = blockIdx.x, k = k0 + blockIdx.y;
      if (!pair_unit(P.nb, b, k)) return;
      const int c = b + k < P.nb ? b + k : b + k - P.nb;
      const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
      const int r = warp % B, h = warp / B;
      const int I = b * B + r;
      for (int q = tid; q < NO * NB; q += TH) col[q] = 0.;
      for (int q = 0; q < NO * PU; q++) rows[q * TH + tid] = 0.;
      // a unit of several tile pairs (row tile, column tile): far_scale of each, by the
      // threads that stage least; one pair's is worked out below, while its rows load
      __shared__ float far_s[B * B];
      if (MODE == 0 && B > 1 && tid >= TH - B * B) {
            const int q = TH - 1 - tid, ti = b * B + q / B, tj = c * B + q % B;
            if (ti < P.ntiles && tj < P.ntiles)
                  far_s[q] = far_scale<SOFT, OP>(P.box + 6 * ti, P.box + 6 * tj, PAIR_NEAR * theta, eps2);
      }
      if (MODE == 0)
            for (int q = tid; q < 2 * B * 32; q += TH) {
                  const int t = q / 64, g = (q / 32) & 1, s = q & 31, J = c * B + t;
                  if (J >= P.ntiles) continue;
                  const float *v = P.s32 + (size_t)J * 4 * PT + 64 * g + s;
                  PairGroup<SOFT, OP> &G = st[2 * t + g];
                  G.xy[s] = G.xy[s + 32] = make_ulonglong2(f2_pack(v[0], v[32]), f2_pack(v[PT], v[PT + 32]));
                  G.zm[s] = G.zm[s + 32] =
                      make_ulonglong2(f2_pack(v[2 * PT], v[2 * PT + 32]), f2_pack(v[3 * PT], v[3 * PT + 32]));
                  if constexpr (OP == 1) {
                        const float *w = P.l32 + (size_t)J * 3 * PT + 64 * g + s;
                        G.l[s] = G.l[s + 32] = make_ulonglong2(f2_pack(w[0], w[32]), f2_pack(w[PT], w[PT + 32]));
                        G.lz[s] = G.lz[s + 32] = f2_pack(w[2 * PT], w[2 * PT + 32]);
                  }
                  if constexpr (SOFT == 2) {
                        const float *e = P.sR32 + (size_t)J * PT + 64 * g + s;
                        G.R[s] = G.R[s + 32] = f2_pack(e[0], e[32]);
                  }
            }
      __syncthreads();
#pragma unroll 1
      for (int p = 0; p < B; p++) {
            const int t = r + p < B ? r + p : r + p - B, J = c * B + t;
            const int what = I < P.ntiles && J < P.ntiles ? pair_phase(B, k, r, p) : 0;
            if (what != 0) {
                  double *cl = col + t * PT;
                  const float sf = MODE == 1 ? 0.f
                                   : B > 1   ? far_s[r * B + t]
                                             : far_scale<SOFT, OP>(P.box + 6 * I, P.box + 6 * J, PAIR_NEAR * theta, eps2);
                  const bool near = MODE == 1 || what == 1 || sf == 0.f;
#pragma unroll 1
                  for (int u0 = 0; u0 < PU; u0 += RU) {
                        const int i = I * PT + lane + 32 * u0;
                        double *rs = rows + NO * u0 * TH + tid;
                        PairRows64<SOFT, OP, RU> T;
                        T.load(P, i);
                        if (near) {
                              double acc[RU][NO];
#pragma unroll
                              for (int u = 0; u < RU; u++)
#pragma unroll
                                    for (int d = 0; d < NO; d++) acc[u][d] = 0.;
#pragma unroll 1
                              for (int g = h * NN; g < (h + 1) * NN; g++) {
                                    if (what == 1)
                                          near_group<SOFT, OP, true>(P, J * PT + 32 * g, i, lane, T, eps2, acc,
                                                                     cl + 32 * g, NB);
                                    else
                                          near_group<SOFT, OP, false>(P, J * PT + 32 * g, i, lane, T, eps2, acc,
                                                                      cl + 32 * g, NB);
                              }
#pragma unroll
                              for (int u = 0; u < RU; u++)
#pragma unroll
                                    for (int d = 0; d < NO; d++) rs[(NO * u + d) * TH] += acc[u][d];
                        } else if (h * NG < 2) {
                              // coordinates relative to the column tile's centre
                              const double *bj = P.box + 6 * J;
                              PairRows<OP, RU> F;
#pragma unroll
                              for (int u = 0; u < RU; u++) {
                                    const float x = -sf * (float)(T.me[u].x - bj[0]);
                                    const float y = -sf * (float)(T.me[u].y - bj[1]);
                                    const float z = -sf * (float)(T.me[u].z - bj[2]), m = (float)T.me[u].w;
                                    F.nx[u] = f2_pack(x, x);
                                    F.ny[u] = f2_pack(y, y);
                                    F.nz[u] = f2_pack(z, z);
                                    F.m[u] = f2_pack(m, m);
                                    const float e = sf * (float)T.R[u];
                                    F.R[u] = SOFT == 2 ? f2_pack(e, e) : 0ull;
                                    if constexpr (OP == 1) {
                                          const float lx = -(float)T.l[u][0], ly = -(float)T.l[u][1];
                                          const float lz = -(float)T.l[u][2];
                                          F.nlx[u] = f2_pack(lx, lx);
                                          F.nly[u] = f2_pack(ly, ly);
                                          F.nlz[u] = f2_pack(lz, lz);
                                    }
                              }
                              const double s = sf;
                              const double back[2] = {OP == 0 ? s * s : s * s * s, s * s};
                              const float es = (float)(eps2 * s * s);
                              const f2 E = f2_pack(es, es), S = f2_pack(sf, sf);
#pragma unroll 1
                              for (int g = h * NG; g < (h + 1) * NG; g++)
                                    if (sf == 1.f)
                                          far_group<SOFT, OP, false, RU>(st[2 * t + g], lane, F, E, S, back, rs, TH,
                                                                         cl + 64 * g, NB);
                                    else
                                          far_group<SOFT, OP, true, RU>(st[2 * t + g], lane, F, E, S, back, rs, TH,
                                                                        cl + 64 * g, NB);
                        }
                  }
            }
            __syncthreads();  // the next phase's warp of each column tile; the sums are complete
      }
      double *prow = part + (size_t)(2 * blockIdx.y) * NO * npad, *pcol = prow + NO * npad;
      for (int q = tid; q < NB; q += TH) {
            const int at = (q % 32) + 32 * (q / PT), u = (q % PT) / 32;
            for (int d = 0; d < NO; d++) {
                  double v = rows[(NO * u + d) * TH + at];
                  for (int e = 1; e < H; e++) v += rows[(NO * u + d) * TH + at + 32 * B * e];
                  prow[d * npad + (long)b * NB + q] = v;
                  pcol[d * npad + (long)c * NB + q] = col[d * NB + q];
            }
      }
}

// The partial rows of offsets k0 .. k0 + nk - 1 for body q of block blk (32
// bodies a CTA of 256 threads: thread group g adds rows g, g + 8, ...; the
// groups' sums are added in order): v[d] for the threads of group 0.
template <int NO>
__device__ __forceinline__ void pair_rows_sum(const double *__restrict__ part, long npad, int nb, int blk, int k0,
                                              int nk, long q, bool live, double (*sh)[8][32], double (&v)[NO])
{
      const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
      double s[NO];
#pragma unroll
      for (int d = 0; d < NO; d++) s[d] = 0.;
      if (live) {
#pragma unroll 4
            for (int row = g; row < 2 * nk; row += 8) {
                  const bool has = pair_row(nb, blk, k0 + (row >> 1), row & 1);
                  const double *p = part + (size_t)row * NO * npad + q;
#pragma unroll
                  for (int d = 0; d < NO; d++) s[d] += has ? p[d * npad] : 0.;
            }
      }
#pragma unroll
      for (int d = 0; d < NO; d++) sh[d][g][lane] = s[d];
      __syncthreads();
      if (g == 0)
#pragma unroll
            for (int d = 0; d < NO; d++) {
                  v[d] = sh[d][0][lane];
                  for (int e = 1; e < 8; e++) v[d] += sh[d][e][lane];
            }
}

// Adds the partial rows of offsets k0 .. k0 + nk - 1 to the sums in base (NO
// blocks of npad; set instead of added to when `first`): for body counts whose
// rows do not fit the partial buffer at once.
template <int NO>
__global__ void __launch_bounds__(256) k_pair_accum(const double *__restrict__ part, long npad, int nb, int k0, int nk,
                                                    int bsize, int n, int first, double *__restrict__ base)
{
      __shared__ double sh[NO][8][32];
      const long q = (long)blockIdx.x * 32 + (threadIdx.x & 31);
      double v[NO];
      pair_rows_sum<NO>(part, npad, nb, (int)(q / bsize), k0, nk, q, q < n, sh, v);
      if (threadIdx.x < 32 && q < n)
            for (int d = 0; d < NO; d++) base[d * npad + q] = first ? v[d] : base[d * npad + q] + v[d];
}

// How the pair sums of n bodies are split: tiles a block, blocks, the offsets of
// one share of the partial rows, and the buffer's doubles (the rows of a share
// and, with several, the sums of the earlier ones behind them).
struct PairPlan {
      int B, nb, nk, per;
      bool few;  // few enough tiles for four warps a unit in the mixed kernel too
      long npad;
      size_t doubles;
};

constexpr size_t PAIR_ROWS_MAX = (size_t)1 << 27;  // doubles of partial rows at once (1 GB)

// At most `most` offsets of pl at once (the shares about equal).
template <int OP>
void pair_share(PairPlan &pl, int most)
{
      const int shares = (pl.nk + most - 1) / most;
      pl.per = (pl.nk + shares - 1) / shares;
      pl.doubles = PAIR_OUT<OP> * (size_t)pl.npad * (2 * pl.per + (pl.per >= pl.nk ? 0 : 1));
}

// Half the offsets at once, for a device whose memory is short; false when there is one.
template <int OP>
bool pair_halve(PairPlan &pl)
{
      if (pl.per <= 1) return false;
      pair_share<OP>(pl, pl.per / 2);
      return true;
}

template <int OP>
PairPlan pair_plan(int n)
{
      PairPlan pl;
      const int ntiles = (n + PT - 1) / PT;
      // Larger blocks write fewer partial rows, smaller ones give more and shorter
      // units.  Whole mixed force calls, equal radii, B = 1 / 2 / 4 (8 is slower
      // everywhere): 204 / 213 / 331 us at 12,345 bodies, 316 / 308 / 398 at 20,011,
      // 520 / 498 / 576 at 30,011, 1,730 / 1,669 / 1,657 at 65,536; FP64 276 / 297 / 352
      // at 12,345, 972 / 958 / 966 at 30,011, 3,935 / 3,882 / 3,808 at 65,536.  (The
      // VJP's larger sums leave room for four CTAs of two tiles.)
      // With one row tile a CTA, four warps share it in the all-FP64 kernel and, up to
      // 96 tiles, in the mixed one, whose near tile pairs are what a unit waits for; two
      // beyond that, where the far ones are and only two of four warps would have a
      // group of them.  Two / four warps, kernel microseconds: mixed 28 / 19 at 2,000
      // bodies, 37 / 31 at 5,000, 54 / 51 at 8,192, 90 / 89 at 12,345, 134 / 139 at
      // 16,384; FP64 28 / 18 at 2,000, 77 / 73 at 8,192, 156 / 148 at 12,345, 267 / 262
      // at 16,384; 24 leapfrog steps and their VJPs, ms: FP64 4.1 / 3.0 at 1,000 bodies,
      // 4.6 / 3.7 at 3,000; mixed 4.3 / 3.0 and 4.75 / 3.75.
      pl.B = ntiles <= 128 ? 1 : ntiles < 384 || OP == 1 ? 2 : 4;
      pl.few = ntiles <= 96;
      pl.nb = (ntiles + pl.B - 1) / pl.B;
      pl.npad = (long)pl.nb * pl.B * PT;
      pl.nk = pair_offsets(pl.nb);
      const size_t row = 2 * PAIR_OUT<OP> * (size_t)pl.npad;  // both sides of an offset
      const int most = (int)(PAIR_ROWS_MAX / row > (size_t)pl.nk ? pl.nk : PAIR_ROWS_MAX / row < 1 ? 1 : PAIR_ROWS_MAX / row);
      pair_share<OP>(pl, most);
      return pl;
}

// What pair_sums left in the partial buffer for the final pass: the rows of
// offsets k0 .. k0 + nk - 1, and the sums of the earlier ones in base (or null).
struct PairRun {
      const double *part, *base;
      int nb, bsize, k0, nk;
      long npad;
};

template <int MODE, int SOFT, int OP, int B, int W>
int pair_launch(const PairData &pd, int k0, int nk, double theta, double eps2, double *part, long npad, cudaStream_t st)
{
      constexpr size_t smem = pair_smem<MODE, SOFT, OP, B, W>();
      static_assert(smem + B * B * sizeof(float) <= 48 * 1024, "no larger carve-out is asked for");
      k_pair_sym<MODE, SOFT, OP, B, W><<<dim3(pd.nb, nk), 32 * W, smem, st>>>(pd, k0, theta, eps2, part, npad);
      NCG_LAUNCHED();
      return NCGPU_OK;
}

template <int MODE, int SOFT, int OP>
int pair_launch_b(const PairPlan &pl, const PairData &pd, int k0, int nk, double theta, double eps2, double *part,
                  long npad, cudaStream_t st)
{
      if constexpr (OP == 0)
            if (pl.B == 4) return pair_launch<MODE, SOFT, OP, 4, 4>(pd, k0, nk, theta, eps2, part, npad, st);
      if (pl.B == 2) return pair_launch<MODE, SOFT, OP, 2, 4>(pd, k0, nk, theta, eps2, part, npad, st);
      if constexpr (MODE == 0)
            if (!pl.few) return pair_launch<MODE, SOFT, OP, 1, 2>(pd, k0, nk, theta, eps2, part, npad, st);
      return pair_launch<MODE, SOFT, OP, 1, 4>(pd, k0, nk, theta, eps2, part, npad, st);
}

// Every unordered pair of pd's bodies once, into part (pl.doubles doubles).
// mode 0: mixed, 1: FP64; soft 0: none, 1: uniform eps2, 2: general.
template <int OP>
int pair_sums(PairData pd, const PairPlan &pl, int mode, int soft, double theta, double eps2, double *part,
              PairRun &run, cudaStream_t st)
{
      pd.nb = pl.nb;
      double *base = pl.per >= pl.nk ? nullptr : part + 2 * PAIR_OUT<OP> * (size_t)pl.npad * pl.per;
      for (int k0 = 0; k0 < pl.nk; k0 += pl.per) {
            const int m = pl.nk - k0 < pl.per ? pl.nk - k0 : pl.per;
            int s;
            if (mode == 0)
                  s = soft == 0   ? pair_launch_b<0, 0, OP>(pl, pd, k0, m, theta, eps2, part, pl.npad, st)
                      : soft == 1 ? pair_launch_b<0, 1, OP>(pl, pd, k0, m, theta, eps2, part, pl.npad, st)
                                  : pair_launch_b<0, 2, OP>(pl, pd, k0, m, theta, eps2, part, pl.npad, st);
            else
                  s = soft == 0   ? pair_launch_b<1, 0, OP>(pl, pd, k0, m, theta, eps2, part, pl.npad, st)
                      : soft == 1 ? pair_launch_b<1, 1, OP>(pl, pd, k0, m, theta, eps2, part, pl.npad, st)
                                  : pair_launch_b<1, 2, OP>(pl, pd, k0, m, theta, eps2, part, pl.npad, st);
            NCG_TRY(s);
            if (k0 + m < pl.nk) {
                  k_pair_accum<PAIR_OUT<OP>><<<(pd.n + 31) / 32, 256, 0, st>>>(part, pl.npad, pl.nb, k0, m, pl.B * PT,
                                                                               pd.n, k0 == 0, base);
                  NCG_LAUNCHED();
            }
            run = PairRun{part, k0 > 0 ? base : nullptr, pl.nb, pl.B * PT, k0, m, pl.npad};
      }
      return NCGPU_OK;
}

}  // namespace ncg
