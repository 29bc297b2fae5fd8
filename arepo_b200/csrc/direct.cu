// direct.cu -- FP64 direct summation over all loaded particles for a set of
// targets: the accuracy instrument of gravity_forcetest_evaluate
// (src/gravity/gravtree_forcetest.c:483-601) without the Ewald terms.  For a
// periodic TreePM run it returns the short-range force with the exact erfc
// factor (u = r / (2 Asmth)); for an isolated run the Newtonian force.  Both
// with the cubic-spline softening of the walk.  Source tiles are dealt out to
// chunks; partial sums are reduced in a fixed order (deterministic).
#include <cub/cub.cuh>

#include "internal.h"

namespace gg
{
namespace
{
#define SF1 10.666666666667
#define SF2 32.0
#define SF3 (-38.4)
#define SF4 (-2.8)
#define SF5 5.333333333333
#define SF6 6.4
#define SF7 (-9.6)
#define SF8 21.333333333333
#define SF9 (-48.0)
#define SF10 38.4
#define SF11 (-10.666666666667)
#define SF12 (-0.066666666667)
#define SF13 (-3.2)
#define SF14 0.066666666667
#define SF15 (-16.0)
#define SF16 9.6
#define SF17 (-2.133333333333)

// Source tiles: 32 consecutive sources in key order and their bounding box (centre, half extents).
constexpr int kTileSrc = 32;
constexpr int kTgt     = 4;  // targets per warp: a source is loaded once for them
struct TileBox
{
  double cx, cy, cz, hx, hy, hz;
};

__global__ void k_tile_box(const double4 *__restrict__ pm, int64_t n, int64_t ntile, TileBox *__restrict__ box)
{
  const int lane = threadIdx.x & 31;
  for(int64_t t = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; t < ntile; t += ((int64_t)gridDim.x * blockDim.x) >> 5)
    {
      const int64_t j = t * kTileSrc + lane;
      const double4 p = pm[j < n ? j : n - 1];
      double lo[3] = {p.x, p.y, p.z}, hi[3] = {p.x, p.y, p.z};
#pragma unroll
      for(int k = 0; k < 3; k++)
        for(int o = 16; o > 0; o >>= 1)
          {
            lo[k] = fmin(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
            hi[k] = fmax(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
          }
      if(lane == 0)
        box[t] = TileBox{0.5 * (lo[0] + hi[0]), 0.5 * (lo[1] + hi[1]), 0.5 * (lo[2] + hi[2]),
                         0.5 * (hi[0] - lo[0]), 0.5 * (hi[1] - lo[1]), 0.5 * (hi[2] - lo[2])};
    }
}

__device__ __forceinline__ double nearest_image(double d, const WalkConst &w)
{
  return !w.periodic ? d : (d > w.half_box) ? d - w.box : ((d < -w.half_box) ? d + w.box : d);
}

// One pair: gravity_forcetest_evaluate's force and potential (src/gravity/gravtree_forcetest.c:483-601).
// u = r / (2 Asmth): beyond kUZero both factors of the split are below 2^-54 of the Newtonian pair, which
// the reference's sums round to no contribution at all (softened pairs excepted); one exponential and
// erfcx serve both factors.
constexpr double kUZero = 6.5;
template <bool PM, bool EWALD>
__device__ __forceinline__ void direct_pair(double dx, double dy, double dz, double r2, double m, double hmax, double uscale,
                                            const WalkConst &w, double4 &a)
{
  const double rinv = r2 > 0 ? rsqrt(r2) : 0.0;
  const double r    = r2 * rinv;
  const double wpn  = -m * rinv;
  const double fn   = -wpn * rinv * rinv;
  double g = 1.0, gp = 1.0;  // force and potential factors of the Newtonian pair
  if(PM)
    {
      const double u = uscale * r, e = exp(-u * u);
      gp             = erfcx(u) * e;
      g              = fma(u * 1.1283791670955126, e, gp);  // 2 / sqrt(pi)
    }
  double fac = fn * g, wp = wpn * gp;
  if(r < hmax)
    {
      const double h_inv = 1.0 / hmax, h3_inv = h_inv * h_inv * h_inv, u = r * h_inv, u2 = u * u;
      if(u < 0.5)
        {
          fac = m * h3_inv * (SF1 + u2 * (SF2 * u + SF3));
          wp  = m * h_inv * (SF4 + u2 * (SF5 + u2 * (SF6 * u + SF7)));
        }
      else
        {
          const double u3 = u2 * u;
          fac = m * h3_inv * (SF8 + SF9 * u + SF10 * u2 + SF11 * u3 + SF12 / u3);
          wp  = m * h_inv * (SF13 + SF14 / u + u2 * (SF1 + u * (SF15 + u * (SF16 + SF17 * u))));
        }
      if(PM)
        {
          fac = fma(fn, g - 1.0, fac);
          wp  = fma(wpn, gp - 1.0, wp);
        }
    }
  a.x = fma(dx, fac, a.x);
  a.y = fma(dy, fac, a.y);
  a.z = fma(dz, fac, a.z);
  a.w += wp;
  if(EWALD)
    {
      // pure periodic tree: every image through the Ewald correction
      double fcorr[3], pcorr;
      ewald_corr(dx, dy, dz, w, fcorr, pcorr);
      a.x += m * fcorr[0];
      a.y += m * fcorr[1];
      a.z += m * fcorr[2];
      a.w += m * pcorr;
    }
}

// A warp sums kTgt targets (consecutive in key order) over the batches of up to 32 tiles blockIdx.y,
// blockIdx.y + gridDim.y, ...: each lane compares one tile's box with the targets, then the warp visits the
// tiles that can hold a pair closer than the split's reach (PM: rskip; else every tile), one source per
// lane.  Lane sums are added over the warp at the end.
constexpr int kDirectWarps = 4;
template <bool PM, bool EWALD>
__global__ void __launch_bounds__(32 * kDirectWarps) k_direct(const double4 *__restrict__ pm, const uint8_t *__restrict__ st, int64_t n,
                                                              const TileBox *__restrict__ box, int64_t ntile, int batch,
                                                              const int32_t *__restrict__ targets, int64_t nt,
                                                              const WalkConst *__restrict__ wcp, int cut, double rskip2,
                                                              double4 *__restrict__ partial)
{
  __shared__ WalkConst w;
  for(int t = threadIdx.x; t < (int)(sizeof(WalkConst) / 4); t += blockDim.x)
    ((int *)&w)[t] = ((const int *)wcp)[t];
  __syncthreads();
  const int lane   = threadIdx.x & 31;
  const int64_t t0 = ((int64_t)blockIdx.x * kDirectWarps + (threadIdx.x >> 5)) * kTgt;
  if(t0 >= nt)
    return;
  const double uscale = PM ? sqrt(w.asmthinv2) : 0.0;  // 1 / (2 Asmth)
  double4 me[kTgt], a[kTgt];
  double h_i[kTgt];
#pragma unroll
  for(int k = 0; k < kTgt; k++)
    {
      const int i = targets[t0 + k < nt ? t0 + k : t0];
      me[k]       = pm[i];
      h_i[k]      = w.soft[st[i]];
      a[k]        = make_double4(0, 0, 0, 0);
    }
  for(int64_t b = (int64_t)blockIdx.y * batch; b < ntile; b += (int64_t)gridDim.y * batch)
    {
      unsigned near = 0;
      if(lane < batch && b + lane < ntile)
        {
          near = (1u << kTgt) - 1u;
          if(PM)
            {
              const TileBox q = box[b + lane];
              near            = 0;
#pragma unroll
              for(int k = 0; k < kTgt; k++)
                {
                  // least distance of the target to any image of the box
                  const double x = fmax(fabs(nearest_image(q.cx - me[k].x, w)) - q.hx, 0.0),
                               y = fmax(fabs(nearest_image(q.cy - me[k].y, w)) - q.hy, 0.0),
                               z = fmax(fabs(nearest_image(q.cz - me[k].z, w)) - q.hz, 0.0);
                  near |= (x * x + y * y + z * z < rskip2 ? 1u : 0u) << k;
                }
            }
        }
      for(unsigned todo = __ballot_sync(0xffffffffu, near != 0); todo; todo &= todo - 1)
        {
          const int q        = __ffs(todo) - 1;
          const unsigned who = __shfl_sync(0xffffffffu, near, q);
          const int64_t j    = (b + q) * kTileSrc + lane;
          const bool valid   = j < n;
          const double4 s    = pm[valid ? j : n - 1];
          const double h_j   = w.soft[st[valid ? j : n - 1]];
#pragma unroll
          for(int k = 0; k < kTgt; k++)
            if(who >> k & 1u)
              {
                const double dx = nearest_image(s.x - me[k].x, w), dy = nearest_image(s.y - me[k].y, w),
                             dz   = nearest_image(s.z - me[k].z, w);
                const double r2   = fma(dx, dx, fma(dy, dy, dz * dz));
                const double hmax = h_j > h_i[k] ? h_j : h_i[k];
                // cut: beyond Rcut lies the part of the force left to the PM mesh
                if(valid && (!PM || (cut ? r2 < w.rcut2 : r2 < rskip2)))
                  direct_pair<PM, EWALD>(dx, dy, dz, r2, s.w, hmax, uscale, w, a[k]);
              }
        }
    }
#pragma unroll
  for(int k = 0; k < kTgt; k++)
    {
      for(int o = 16; o > 0; o >>= 1)
        {
          a[k].x += __shfl_xor_sync(0xffffffffu, a[k].x, o);
          a[k].y += __shfl_xor_sync(0xffffffffu, a[k].y, o);
          a[k].z += __shfl_xor_sync(0xffffffffu, a[k].z, o);
          a[k].w += __shfl_xor_sync(0xffffffffu, a[k].w, o);
        }
      if(lane == 0 && t0 + k < nt)
        partial[(int64_t)blockIdx.y * nt + t0 + k] = a[k];
    }
}

// chunk sums of the t-th target in key order, to its place in the caller's list
__global__ void k_direct_reduce(const double4 *__restrict__ partial, int chunks, int64_t nt, const int32_t *__restrict__ place,
                                double *__restrict__ acc, double *__restrict__ pot)
{
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if(t >= nt)
    return;
  double ax = 0, ay = 0, az = 0, pt = 0;
  for(int c = 0; c < chunks; c++)
    {
      double4 p = partial[(int64_t)c * nt + t];
      ax += p.x;
      ay += p.y;
      az += p.z;
      pt += p.w;
    }
  const int64_t o = place[t];
  acc[3 * o + 0]  = ax;
  acc[3 * o + 1]  = ay;
  acc[3 * o + 2]  = az;
  pot[o]          = pt;
}

__global__ void k_map_targets(const int64_t *__restrict__ tg, int64_t nt, const uint32_t *__restrict__ iperm, int32_t *__restrict__ out,
                              int32_t *__restrict__ place)
{
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if(t < nt)
    {
      out[t]   = (int32_t)iperm[tg[t]];
      place[t] = (int32_t)t;
    }
}
// gravity_direct (src/gravity/gravdirect.c:61-257) with force_evaluate_direct's pair arithmetic
// (src/gravity/forcetree_walk.c:557-708): the n particles are targets and sources; every target's terms
// are the reference's operations (FP64, no contraction) and are added in source order, so the result is
// bit-identical.  Flag bit 1: a softening type >= nsofttypes.
//
// Only the additions have to follow each other; the terms (a square root, divisions, the table) do not.
// A warp takes T targets and 32 sources at a time: every lane computes the terms of its source for the T
// targets into shared memory, then 4 T lanes add them, one sum component each, in source order.  Sets that fill
// the chip with one thread per target have no need of that (k_gravity_direct_wide).
template <bool EWALD, int P>  // P: component pitch of `out`
__device__ __forceinline__ void direct_terms(const double4 s, double h_j, double4 me, double h_i, const WalkConst &w,
                                             double *__restrict__ out)
{
#pragma unroll
  for(int c = 0; c < (EWALD ? 8 : 4); c++)
    out[c * P] = 0.0;
  double hmax = (h_j > h_i) ? h_j : h_i;
  double dx = s.x - me.x, dy = s.y - me.y, dz = s.z - me.z;
  if(w.periodic)
    {
      dx = (dx > w.half_box) ? (dx - w.box) : ((dx < -w.half_box) ? (dx + w.box) : dx);
      dy = (dy > w.half_box) ? (dy - w.box) : ((dy < -w.half_box) ? (dy + w.box) : dy);
      dz = (dz > w.half_box) ? (dz - w.box) : ((dz < -w.half_box) ? (dz + w.box) : dz);
    }
  double r2 = dx * dx + dy * dy + dz * dz;
  double m  = s.w;
  double r  = sqrt(r2);
  double factor_force = 0, factor_pot = 0;
  if(w.pm)
    {
      double tabentry = w.asmthfac * r;
      int tabindex    = (int)tabentry;
      if(tabindex >= kNtab)
        return;
      static_assert((kNtab & (kNtab + 1)) == 0, "all bits set");
      tabindex &= kNtab;  // INT_MIN where r is NaN (a non-finite position): entry 0, and the sums will be NaN
      double tabweight = tabentry - tabindex;
      factor_force     = (1.0 - tabweight) * w.tab_force[tabindex] + tabweight * w.tab_force[tabindex + 1];
      factor_pot       = (1.0 - tabweight) * w.tab_pot[tabindex] + tabweight * w.tab_pot[tabindex + 1];
    }
  double fac, wp;
  if(r >= hmax)
    {
      double rinv  = 1.0 / r;
      double rinv3 = rinv * rinv * rinv;
      if(w.pm)
        {
          fac = rinv3 + rinv * factor_force * w.asmthinv2;
          wp  = rinv * factor_pot;
        }
      else
        {
          fac = rinv3;
          wp  = -rinv;
        }
    }
  else
    {
      double h_inv  = 1.0 / hmax;
      double h3_inv = h_inv * h_inv * h_inv;
      double u      = r * h_inv;
      if(u < 0.5)
        {
          double u2 = u * u;
          fac       = h3_inv * (SF1 + u2 * (SF2 * u + SF3));
          wp        = h_inv * (SF4 + u2 * (SF5 + u2 * (SF6 * u + SF7)));
        }
      else
        {
          double u2 = u * u;
          double u3 = u2 * u;
          fac       = h3_inv * (SF8 + SF9 * u + SF10 * u2 + SF11 * u3 + SF12 / u3);
          wp        = h_inv * (SF13 + SF14 / u + u2 * (SF1 + u * (SF15 + u * (SF16 + SF17 * u))));
        }
      if(w.pm && r > 0)
        {
          double rinv = 1.0 / r;
          fac += rinv * factor_force * w.asmthinv2;
          wp += rinv * (factor_pot + 1.0);
        }
    }
  fac *= m;
  out[0 * P] = dx * fac;
  out[1 * P] = dy * fac;
  out[2 * P] = dz * fac;
  out[3 * P] = m * wp;
  if(EWALD)
    {
      double fcorr[3], pcorr;
      ewald_corr(dx, dy, dz, w, fcorr, pcorr);
      out[4 * P] = m * fcorr[0];
      out[5 * P] = m * fcorr[1];
      out[6 * P] = m * fcorr[2];
      out[7 * P] = m * pcorr;
    }
}

constexpr int kDirWarps        = 4;
constexpr int64_t kDirOneTarget = 8192;
template <int T, bool EWALD>
__global__ void __launch_bounds__(32 * kDirWarps) k_gravity_direct(const double *__restrict__ pos, const double *__restrict__ mass,
                                                                   const uint8_t *__restrict__ st, int64_t n,
                                                                   const WalkConst *__restrict__ wcp, double *__restrict__ acc,
                                                                   double *__restrict__ pot, int *__restrict__ flag)
{
  constexpr int C = EWALD ? 8 : 4;
  static_assert(4 * T <= 32, "one lane per target and component");
  __shared__ WalkConst w;
  __shared__ double term[kDirWarps][T][C][33];
  for(int t = threadIdx.x; t < (int)(sizeof(WalkConst) / 4); t += blockDim.x)
    ((int *)&w)[t] = ((const int *)wcp)[t];
  __syncthreads();
  const int warp   = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t i0 = ((int64_t)blockIdx.x * kDirWarps + warp) * T;
  if(i0 >= n)
    return;
  double4 me[T];
  double h_i[T];
#pragma unroll
  for(int t = 0; t < T; t++)
    {
      const int64_t i = i0 + t < n ? i0 + t : n - 1;  // a target past the end repeats the last one
      const int ty    = st[i];
      if(ty >= w.nsoft)
        atomicOr(flag, 1);
      me[t]  = make_double4(pos[3 * i + 0], pos[3 * i + 1], pos[3 * i + 2], 0.0);
      h_i[t] = w.soft[ty < w.nsoft ? ty : 0];
    }
  const int st_ = lane >> 2, sc = lane & 3;  // this lane's target and component in the additions
  double sum    = 0;
  for(int64_t jb = 0; jb < n && n > 1; jb += 32)
    {
      const int64_t j = jb + lane;
      if(j < n)
        {
          const double4 s  = make_double4(pos[3 * j + 0], pos[3 * j + 1], pos[3 * j + 2], mass[j]);
          const int ty     = st[j];
          const double h_j = w.soft[ty < w.nsoft ? ty : 0];
#pragma unroll
          for(int t = 0; t < T; t++)
            direct_terms<EWALD, 33>(s, h_j, me[t], h_i[t], w, &term[warp][t][0][lane]);
        }
      __syncwarp();
      const int cnt = n - jb < 32 ? (int)(n - jb) : 32;
      if(st_ < T)
        {
          const double *q = &term[warp][st_][sc][0];
          if(cnt == 32)
            {
#pragma unroll
              for(int k = 0; k < 32; k++)
                {
                  sum += q[k];
                  if(EWALD)
                    sum += q[4 * 33 + k];
                }
            }
          else
            for(int k = 0; k < cnt; k++)
              {
                sum += q[k];
                if(EWALD)
                  sum += q[4 * 33 + k];
              }
        }
      __syncwarp();
    }
  if(st_ < T && i0 + st_ < n)
    {
      if(sc < 3)
        acc[3 * (i0 + st_) + sc] = sum;
      else if(pot)
        pot[i0 + st_] = sum;
    }
}

// The same sums, one thread per target over source tiles in shared memory: each thread adds its terms as it
// computes them.
constexpr int kWide = 128;
constexpr int64_t kDirWide = 45000, kDirWideEwald = 110000;  // targets from which it is the faster one
template <bool EWALD>
__global__ void __launch_bounds__(kWide) k_gravity_direct_wide(const double *__restrict__ pos, const double *__restrict__ mass,
                                                               const uint8_t *__restrict__ st, int64_t n,
                                                               const WalkConst *__restrict__ wcp, double *__restrict__ acc,
                                                               double *__restrict__ pot, int *__restrict__ flag)
{
  __shared__ WalkConst w;
  __shared__ double4 src[kWide];
  __shared__ double hsrc[kWide];
  for(int t = threadIdx.x; t < (int)(sizeof(WalkConst) / 4); t += blockDim.x)
    ((int *)&w)[t] = ((const int *)wcp)[t];
  __syncthreads();
  const int64_t i = (int64_t)blockIdx.x * kWide + threadIdx.x, k = i < n ? i : n - 1;  // past the end: the last target
  const int ty    = st[k];
  if(ty >= w.nsoft)
    atomicOr(flag, 1);
  const double4 me = make_double4(pos[3 * k + 0], pos[3 * k + 1], pos[3 * k + 2], 0.0);
  const double h_i = w.soft[ty < w.nsoft ? ty : 0];
  double sum[4]    = {0, 0, 0, 0};
  for(int64_t jb = 0; jb < n; jb += kWide)
    {
      const int64_t j = jb + threadIdx.x;
      __syncthreads();
      if(j < n)
        {
          const int tj      = st[j];
          src[threadIdx.x]  = make_double4(pos[3 * j + 0], pos[3 * j + 1], pos[3 * j + 2], mass[j]);
          hsrc[threadIdx.x] = w.soft[tj < w.nsoft ? tj : 0];
        }
      __syncthreads();
      const int cnt = n - jb < kWide ? (int)(n - jb) : kWide;
      for(int q = 0; q < cnt; q++)
        {
          double term[EWALD ? 8 : 4];
          direct_terms<EWALD, 1>(src[q], hsrc[q], me, h_i, w, term);
#pragma unroll
          for(int c = 0; c < 4; c++)
            {
              sum[c] += term[c];
              if(EWALD)
                sum[c] += term[4 + c];
            }
        }
    }
  if(i < n)
    {
      for(int c = 0; c < 3; c++)
        acc[3 * i + c] = sum[c];
      if(pot)
        pot[i] = sum[3];
    }
}

__global__ void k_fill_i32(int32_t *__restrict__ a, int64_t n, int32_t v)
{
  for(int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    a[i] = v;
}
}  // namespace

cudaError_t gravity_direct_stage(gpugrav_ctx *c, int64_t n, const double *d_pos, const double *d_mass, const uint8_t *d_st,
                                 double *d_acc, double *d_pot, int32_t *d_nint, int *d_flag)
{
  // One target per warp while the chip has room for more warps than targets, then 4, and one per thread once
  // that fills it.  Kernel (ms) with 1 / 4 / one per thread: isolated 3000 0.13 / 0.15 / 0.59, 8000 0.67 / 0.44 /
  // 1.56, 16384 2.6 / 1.8 / 3.2, 40000 15.2 / 8.5 / 8.8, 49152 22.9 / 13.0 / 10.9, 131072 158 / 83 / 54; TreePM 40000
  // 17.4 / 12.9 / 15.9, 49152 26.2 / 19.6 / 19.6, 131072 184 / 128 / 84; Ewald, whose interpolation outweighs the
  // additions, 32768 103 / 103 / 102, 65536 - / 412 / 441, 131072 - / 1642 / 1568.
  const bool ewald = c->prm.periodic && !(c->prm.asmth > 0);
  if(n > (ewald ? kDirWideEwald : kDirWide))
    {
      auto kern = ewald ? k_gravity_direct_wide<true> : k_gravity_direct_wide<false>;
      kern<<<(unsigned)((n + kWide - 1) / kWide), kWide, 0, c->stream>>>(d_pos, d_mass, d_st, n, c->wconst.as<WalkConst>(), d_acc,
                                                                        d_pot, d_flag);
    }
  else
    {
      const int T       = n <= kDirOneTarget ? 1 : 4;
      auto kern         = T == 1 ? (ewald ? k_gravity_direct<1, true> : k_gravity_direct<1, false>)
                                 : (ewald ? k_gravity_direct<4, true> : k_gravity_direct<4, false>);
      const int64_t per = (int64_t)kDirWarps * T;
      kern<<<(unsigned)((n + per - 1) / per), 32 * kDirWarps, 0, c->stream>>>(d_pos, d_mass, d_st, n, c->wconst.as<WalkConst>(), d_acc,
                                                                            d_pot, d_flag);
    }
  if(d_nint)
    k_fill_i32<<<(unsigned)((n + 255) / 256 < 2368 ? (n + 255) / 256 : 2368), 256, 0, c->stream>>>(d_nint, n, (int32_t)n);
  return cudaGetLastError();
}

cudaError_t direct_stage(gpugrav_ctx *c, const WalkConst &wc, int64_t nt, const int64_t *d_targets, int cut, double *d_acc,
                         double *d_pot)
{
  if(nt == 0)
    return cudaSuccess;
  cudaStream_t st     = c->stream;
  const int64_t n     = c->n;
  const int64_t ntile = (n + kTileSrc - 1) / kTileSrc, nwarp = (nt + kTgt - 1) / kTgt;
  // enough warps for several waves whatever the number of targets (at least 8 chunks, at most one
  // batch of tiles each: 32, or down to 4 while there is not a warp per SM, or not eight and few chunks: one
  // target among 3271 sources took 154 us with batches of 32, four warps in all, and 89 with 4; 500 among 2000
  // took 155 with 32 and 93 with 4.  More chunks than that cost the last sum more than they save: one among
  // 100000 162 us with 98 chunks, 180 with 782)
  int batch       = 32;
  auto more_warps = [&]() {
    const int64_t nb = (ntile + batch - 1) / batch, warps = nwarp * nb;
    return warps < 148 || (warps < 8 * 148 && nb < 64);
  };
  while(batch > 4 && more_warps())
    batch /= 2;
  int64_t chunks         = 148 * 128 / nwarp;
  const int64_t nbatch   = (ntile + batch - 1) / batch;
  chunks                 = chunks < 8 ? 8 : chunks;
  chunks                 = chunks > nbatch ? nbatch : chunks;
  // scratch: boxes | chunk sums | sorted positions and places (before and after the sort) | sort space
  size_t tb = 0;
  GG_TRY(cub::DeviceRadixSort::SortPairs(nullptr, tb, (int32_t *)nullptr, (int32_t *)nullptr, (int32_t *)nullptr, (int32_t *)nullptr,
                                         (int)nt, 0, 31, st));
  auto up             = [](size_t b) { return (b + 255) & ~(size_t)255; };
  const size_t bytes  = up(ntile * sizeof(TileBox)) + up((size_t)chunks * nt * sizeof(double4)) + 4 * up(nt * 4) + up(tb);
  GG_TRY(c->dir_buf.ensure(bytes));
  char *q   = c->dir_buf.as<char>();
  auto take = [&](size_t b) { char *r = q; q += up(b); return r; };
  TileBox *box  = (TileBox *)take(ntile * sizeof(TileBox));
  double4 *part = (double4 *)take((size_t)chunks * nt * sizeof(double4));
  int32_t *ts = (int32_t *)take(nt * 4), *ts2 = (int32_t *)take(nt * 4), *pl = (int32_t *)take(nt * 4), *pl2 = (int32_t *)take(nt * 4);
  k_map_targets<<<(unsigned)((nt + 255) / 256), 256, 0, st>>>(d_targets, nt, c->iperm.as<uint32_t>(), ts, pl);
  GG_TRY(cub::DeviceRadixSort::SortPairs(q, tb, ts, ts2, pl, pl2, (int)nt, 0, 31, st));
  // the reach of a pair: Rcut, or where the exact factor vanishes in double precision and no pair is softened
  double hmax = 0;
  for(int i = 0; i < wc.nsoft; i++)
    hmax = wc.soft[i] > hmax ? wc.soft[i] : hmax;
  const double r0 = wc.pm ? kUZero / sqrt(wc.asmthinv2) : 0.0, reach = cut ? wc.rcut : (r0 > hmax ? r0 : hmax);
  if(wc.pm)
    k_tile_box<<<(unsigned)((ntile + 7) / 8 < 2368 ? (ntile + 7) / 8 : 2368), 256, 0, st>>>(c->s_pm.as<double4>(), n, ntile, box);
  auto kern = wc.pm ? k_direct<true, false> : wc.ewald ? k_direct<false, true> : k_direct<false, false>;
  kern<<<dim3((unsigned)((nwarp + kDirectWarps - 1) / kDirectWarps), (unsigned)chunks), 32 * kDirectWarps, 0, st>>>(
      c->s_pm.as<double4>(), c->s_st.as<uint8_t>(), n, box, ntile, batch, ts2, nt, c->wconst.as<WalkConst>(), cut,
      reach * reach * (1.0 + 1e-9), part);
  k_direct_reduce<<<(unsigned)((nt + 255) / 256), 256, 0, st>>>(part, (int)chunks, nt, pl2, d_acc, d_pot);
  return cudaGetLastError();
}
}  // namespace gg
