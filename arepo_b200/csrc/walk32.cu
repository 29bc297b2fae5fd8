// walk32.cu -- FP32 group walk (the fast path).
//
// Physics as in force_treeevaluate (src/gravity/forcetree_walk.c:115-514): the
// tabulated erfc short-range factor cut at Rcut, the cubic-spline softening, the
// periodic nearest image, the relative criterion (ErrTolForceAcc x OldAcc) after
// a Barnes-Hut pass.  Different arithmetic organisation:
//
//  * a warp walks the tree for a group of up to 64 targets that are consecutive in key
//    order (compact in space); nodes are tested 32 at a time, one per lane,
//    against the group's bounding box with the reference's tests made
//    conservative for the whole group (a node is accepted only if every target of
//    the group would accept it), so each target's error is at most that of its
//    own reference walk;
//  * accepted nodes and the particles of opened nodes go to an interaction list
//    in shared memory; the list is evaluated densely -- every lane computes its
//    own target against every entry -- in FP32;
//  * separations: the group centre g is subtracted in FP64 from every list
//    entry and from every target before rounding to FP32, so an FP32 difference
//    never carries the absolute position (error ~ eps32 x |x - g|, not eps32 x |x|);
//  * sums: FP32 within a list batch, batch partials accumulated in FP64.
//
// Layout: the node children of a node contiguous, particles grouped by parent node.
#include <cub/cub.cuh>
#include <thrust/iterator/transform_iterator.h>

#include <type_traits>

#include "internal.h"

namespace gg
{
namespace
{
#ifndef GG_W32_EVAL_AT
#define GG_W32_EVAL_AT 192
#endif
#ifndef GG_W32_UNROLL
#define GG_W32_UNROLL 8
#endif
#ifndef GG_W32_UNROLL2
#define GG_W32_UNROLL2 4
#endif
constexpr int kEvalAt  = GG_W32_EVAL_AT;  // evaluate once this many entries are queued
// list entries in flight per lane in the evaluation loop
template <int TPL>
constexpr int kUnroll = TPL == 2 ? GG_W32_UNROLL2 : GG_W32_UNROLL;
// Launch shape.  The FP32 TreePM walk keeps kCopies copies of the short-range table in shared memory
// (see TabF), 16 KB that one block per SM can afford and six small ones cannot: one block of 24 warps
// with two targets per lane (80 registers a thread), 28 warps with one (72 registers).  The others
// need no table copies: blocks of 4 warps, 6 or 7 (FP64 form: 3) per SM.
template <typename R, bool PERIODIC, int TPL>
struct Shape
{
  static constexpr bool big   = sizeof(R) == 4 && PERIODIC;
  static constexpr int warps  = big ? (TPL == 2 ? 24 : 28) : 4;
  static constexpr int blocks = big ? 1 : (sizeof(R) == 4 ? (TPL == 2 ? 6 : 7) : 3);
};
// capacity (Cap below): accepted nodes (<= 32) join a list holding fewer than kEvalAt entries;
// particles are added at most 32 per round and the list is evaluated first whenever a round could
// overflow it.  Entries inside some target's softening length go to a separate, smaller near list,
// evaluated as soon as it holds kNearAt entries.
constexpr int kNearAt = 64;
constexpr int kStackCap = 16384;  // traversal stack entries per warp (global memory)
// A node that the group-box test opens although it is smaller than 1/kVote of the box's largest side
// and nearer to the box than that is tested against every target of the group instead (opened
// only if some target's own criterion opens it).  For a compact group this never happens; for a
// group whose targets are far apart (outskirts of an isolated system, where consecutive targets
// in key order can lie on both sides of a dense core) the box test alone would open the whole
// core down to single particles.
constexpr float kVote = 16.0f;

// cubic-spline softening coefficients (src/main/allvars.h:557-573), rounded to the walk's type
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

// The arithmetic type R of the evaluation: float (the fast form) or double (the same group walk in
// FP64, the precision ablation of the fast form).  List capacities per type: double entries take
// twice the shared memory.
template <typename R>
struct Cap
{
  static constexpr int eval     = sizeof(R) == 4 ? kEvalAt : 96;
  static constexpr int list     = eval + 64;
  static constexpr int near_at  = sizeof(R) == 4 ? kNearAt : 32;
  static constexpr int near_cap = near_at + 32;
};
template <typename R>
struct V4T;
template <>
struct V4T<float>
{
  typedef float4 type;
};
template <>
struct V4T<double>
{
  typedef double4 type;
};
template <typename R>
using V4 = typename V4T<R>::type;
template <typename R>
__device__ __forceinline__ V4<R> mk4(double x, double y, double z, double m)
{
  V4<R> v;
  v.x = (R)x;
  v.y = (R)y;
  v.z = (R)z;
  v.w = (R)m;
  return v;
}
__device__ __forceinline__ float fmaR(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fmaR(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float maxR(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ double maxR(double a, double b) { return fmax(a, b); }

struct W32Const
{
  double box, half_box;
  float rcut, rcut2, asmthfac;
  float rcut2_all;  // an entry whose farthest distance from the group box is below this is inside Rcut of every target
  float theta2, erracc;
  int periodic, bh;
  float soft[GPUGRAV_MAX_SOFTTYPES + 1];
  const float4 *ewd;       // Ewald correction (fx, fy, fz, pot) per cell corner (pure periodic tree)
  float ewd_fac;           // 2 EN / L
  int mns;                 // MULTIPLE_NODE_SOFTENING: nodes used per softening type
  const float *mpt;        // per-type node masses in layout order, nsoft each
  int nsoft;
  int minangle;            // ACTIVATE_MINIMUM_OPENING_ANGLE
  // FP64 form only (the FP32 kernels do not copy these into shared memory)
  double rcut2_d, asmthfac_d;  // Rcut^2 and the table index factor in double
  double4 tab64[kNtab + 1];    // the table below in double
  // (f[i], f[i+1] - f[i], p[i], p[i+1] - p[i]): force table times 1/Asmth^2, potential table (FP32 form)
  float4 tab[kNtab + 1];
};
// bytes of the constants a kernel of arithmetic type R keeps in shared memory
template <typename R>
constexpr int kW32Bytes = sizeof(R) == 4 ? (int)offsetof(W32Const, rcut2_d) : (int)offsetof(W32Const, tab);

// The FP32 short-range table in shared memory: every pair of the evaluation reads one 16-byte row at an
// index of its own, and a 16-byte load is served a quarter-warp at a time, each lane from one of the 8
// groups of 4 banks.  With one copy of the table the lanes of a quarter collide (measured: about 9
// wavefronts per warp and pair, which bounded the whole walk); with one copy per bank group lane q reads
// copy q mod 8 and a load takes its 4 wavefronts.
constexpr int kCopies = 8;
struct TabF
{
  float4 row[(kNtab + 1) * kCopies];
};
struct TabNone
{
};
// what short_range reads: the lane's copy of the table (FP32), or nothing
struct TabRef
{
  const float4 *row;
};

// ------------------------------------------------------------------------------
// layout
// ------------------------------------------------------------------------------
// Nodes are placed family by family: the node children of a node follow each other in slot order, the
// families in the order of their parents' numbers (which follow the key order); the particle children
// likewise.  Positions come from one scan over the children counts, after the roots.
struct ChildCounts
{
  __device__ __forceinline__ uint64_t operator()(uint8_t c) const { return (uint64_t)(c & 15) | ((uint64_t)(c >> 4) << 32); }
};

// 8 lanes per node, one per slot: every lane moves its child's record to the node's block
__global__ void k_g_fill(int64_t nn, int64_t n, int nroots, const int32_t *__restrict__ suns, const uint8_t *__restrict__ count,
                         const uint64_t *__restrict__ scan, const double4 *__restrict__ sm, const double4 *__restrict__ cl,
                         const uint8_t *__restrict__ maxsoft, const double4 *__restrict__ pm, const uint8_t *__restrict__ st,
                         double4 *__restrict__ g_sm, float4 *__restrict__ g_rel, int4 *__restrict__ g_kids,
                         double4 *__restrict__ g_pm, uint8_t *__restrict__ g_pst, int *err, const double *__restrict__ mpt, int nsoft,
                         float *__restrict__ g_mpt)
{
  auto put = [&](int64_t b, int64_t k) {
    const double4 s  = sm[k], c = cl[k];
    const uint64_t o = scan[k];
    const int m      = count[k];
    g_sm[b]          = s;
    g_rel[b]         = make_float4((float)(c.x - s.x), (float)(c.y - s.y), (float)(c.z - s.z), (float)c.w);
    g_kids[b]        = make_int4((m & 15) ? nroots + (int)(uint32_t)o : -1, (int)(o >> 32), m, (int)maxsoft[k]);
    if(g_mpt)
      for(int q = 0; q < nsoft; q++)
        g_mpt[b * nsoft + q] = (float)mpt[k * nsoft + q];
  };
  const int lane      = threadIdx.x & 31;
  const unsigned below = (1u << (lane & 7)) - 1u;
  for(int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < ((8 * nn + 31) & ~(int64_t)31); i += (int64_t)gridDim.x * blockDim.x)
    {
      const int64_t k    = i >> 3;
      const int32_t c    = k < nn ? suns[i] : -1;
      const unsigned nm  = __ballot_sync(0xffffffffu, c >= n) >> (lane & 24) & below;
      const unsigned pmk = __ballot_sync(0xffffffffu, c >= 0 && c < n) >> (lane & 24) & below;
      if(c >= n)
        put((int64_t)nroots + (uint32_t)scan[k] + __popc(nm), c - n);
      else if(c >= 0)
        {
          const int64_t b = (int64_t)(scan[k] >> 32) + __popc(pmk);
          if(b < n)
            {
              g_pm[b]  = pm[c];
              g_pst[b] = st[c];
            }
        }
      if((lane & 7) == 0 && k < nn)
        {
          if(k < nroots)
            put(k, k);
          // every node but the roots and every particle has exactly one place
          if(k == nn - 1)
            {
              const uint64_t t = scan[k] + ChildCounts()(count[k]);
              if((int64_t)(uint32_t)t != nn - nroots || (int64_t)(t >> 32) != n)
                atomicOr(err, 8);
            }
        }
    }
}

// ------------------------------------------------------------------------------
// walk
// ------------------------------------------------------------------------------
// nearest image (only the few separations beyond half a box take the branch)
template <bool WRAP>
__device__ __forceinline__ double wrapd(double d, const W32Const &w)
{
  if(WRAP && fabs(d) > w.half_box)
    d -= copysign(w.box, d);
  return d;
}

// 32 bytes in one load (32-byte aligned): a double4, and two float4 (load2)
__device__ __forceinline__ double4 load32(const double4 *p)
{
  double4 v;
  asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p));
  return v;
}

__device__ __forceinline__ double wmin(double v)
{
  for(int o = 16; o > 0; o >>= 1)
    v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ double wmax(double v)
{
  for(int o = 16; o > 0; o >>= 1)
    v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float wminf(float v)
{
  for(int o = 16; o > 0; o >>= 1)
    v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float wmaxf(float v)
{
  for(int o = 16; o > 0; o >>= 1)
    v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ int wscan_incl(int v, int lane)
{
  for(int o = 1; o < 32; o <<= 1)
    {
      int u = __shfl_up_sync(0xffffffffu, v, o);
      if(lane >= o)
        v += u;
    }
  return v;
}

// Reciprocal square root of a normal (never subnormal) argument: the hardware approximation
// without the subnormal handling that a general rsqrtf needs (the walk clamps r^2 >= 1e-30).
__device__ __forceinline__ float rsqrt_normal(float x)
{
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ float rsqrtR(float x) { return rsqrt_normal(x); }
__device__ __forceinline__ double rsqrtR(double x) { return rsqrt(x); }
__device__ __forceinline__ float rcut2_of(const W32Const &w, float) { return w.rcut2; }
__device__ __forceinline__ double rcut2_of(const W32Const &w, double) { return w.rcut2_d; }

// Short-range factors of the TreePM split at separation r: linear interpolation of the force
// (scaled by 1/Asmth^2) and potential tables between nodes floor(te) and floor(te) + 1,
// te = r * asmthfac, as the reference does (src/gravity/forcetree_walk.c:366-379).  Adding 1.5 * 2^23 with rounding toward minus
// infinity leaves floor(te) in the low mantissa bits (no conversion instruction).  CLAMP: the index
// is clamped to the last interval, which only entries beyond Rcut reach (they are masked); without
// CLAMP the entry is inside Rcut, so floor(te) <= NTAB (the table has NTAB + 1 rows).
template <bool CLAMP = true>
__device__ __forceinline__ void short_range(float r, const W32Const &w, TabRef tab, float &ff, float &fpt)
{
  const float tr  = __fmaf_rd(r, w.asmthfac, 12582912.0f);
  const float tb0 = CLAMP ? fminf(tr, 12582912.0f + (float)(kNtab - 1)) : tr;
  const float tw  = fmaf(r, w.asmthfac, 12582912.0f - tb0);
  const float4 t  = tab.row[(__float_as_int(tb0) - 0x4B400000) * kCopies];
  ff              = fmaf(tw, t.y, t.x);
  fpt             = fmaf(tw, t.w, t.z);
}
// the same in double: floor(te) by conversion
template <bool CLAMP = true>
__device__ __forceinline__ void short_range(double r, const W32Const &w, TabRef, double &ff, double &fpt)
{
  const double te = r * w.asmthfac_d;
  int i           = (int)te;
  if(CLAMP)
    i = (int)min((unsigned)i, (unsigned)kNtab - 1u);  // also the conversion of a NaN (r2 = 0, no softening)
  const double tw = te - i;
  const double4 t = w.tab64[i];
  ff              = fma(tw, t.y, t.x);
  fpt             = fma(tw, t.w, t.z);
}

// Per-target state of a lane (targets per lane: TPL).
template <typename R>
struct Tgt
{
  R x, y, z, h;             // position relative to the group centre, softening
  R ax, ay, az, pot;        // partial sums of the current list batch (folded into FP64 sums in shared memory)
  int ni;
};

__device__ __forceinline__ void load2(const float4 *p, float4 &a, float4 &b)
{
  asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
      : "l"(p));
}

// Ewald correction (force, potential) for the separation (dx, dy, dz) = source - target:
// the trilinear interpolation and sign flips of ewald_corr (src/gravity/forcetree_ewald.c:268-342)
// in FP32 on the table of cell corners (k_ewald_cells).
__device__ __forceinline__ float4 ewald_corr32(float dx, float dy, float dz, const W32Const &w)
{
  constexpr int n = kEwaldN;
  const float sx = dx < 0.0f ? 1.0f : -1.0f, sy = dy < 0.0f ? 1.0f : -1.0f, sz = dz < 0.0f ? 1.0f : -1.0f;
  float u = fabsf(dx) * w.ewd_fac, v = fabsf(dy) * w.ewd_fac, s = fabsf(dz) * w.ewd_fac;
  const int i = min((int)u, n - 1), j = min((int)v, n - 1), k = min((int)s, n - 1);
  u -= i;
  v -= j;
  s -= k;
  // the cell's corners, two (32 bytes) per load
  const float4 *t = w.ewd + (size_t)((i * n + j) * n + k) * 8;
  float4 a0, a1, a2, a3, b0, b1, b2, b3;
  load2(t, a0, a1);
  load2(t + 2, a2, a3);
  load2(t + 4, b0, b1);
  load2(t + 6, b2, b3);
  const float f1 = (1 - u) * (1 - v) * (1 - s), f2 = (1 - u) * (1 - v) * s, f3 = (1 - u) * v * (1 - s), f4 = (1 - u) * v * s;
  const float f5 = u * (1 - v) * (1 - s), f6 = u * (1 - v) * s, f7 = u * v * (1 - s), f8 = u * v * s;
  float4 r;
  r.x = a0.x * f1 + a1.x * f2 + a2.x * f3 + a3.x * f4 + b0.x * f5 + b1.x * f6 + b2.x * f7 + b3.x * f8;
  r.y = a0.y * f1 + a1.y * f2 + a2.y * f3 + a3.y * f4 + b0.y * f5 + b1.y * f6 + b2.y * f7 + b3.y * f8;
  r.z = a0.z * f1 + a1.z * f2 + a2.z * f3 + a3.z * f4 + b0.z * f5 + b1.z * f6 + b2.z * f7 + b3.z * f8;
  r.w = a0.w * f1 + a1.w * f2 + a2.w * f3 + a3.w * f4 + b0.w * f5 + b1.w * f6 + b2.w * f7 + b3.w * f8;
  return make_float4(sx * r.x, sy * r.y, sz * r.z, r.w);
}

// Separation of a list entry from a target: (dx, dy, dz) = entry - target, r^2, 1/r and r.  A zero
// separation (the target itself) gives a huge 1/r but r = 0 (CLAMP); it lies inside the softening
// length unless that is zero, where the reference's kernel has no finite value either.  far() and
// near() both call this, so they agree on which side of the softening length every pair lies.
template <typename R>
struct Sep
{
  R dx, dy, dz, r2, rinv, r;
};
template <typename R, bool CLAMP = true>
__device__ __forceinline__ Sep<R> separation(const V4<R> e, const Tgt<R> &T)
{
  Sep<R> s;
  s.dx   = e.x - T.x;
  s.dy   = e.y - T.y;
  s.dz   = e.z - T.z;
  s.r2   = fmaR(s.dx, s.dx, fmaR(s.dy, s.dy, s.dz * s.dz));
  s.rinv = rsqrtR(CLAMP ? maxR(s.r2, (R)(sizeof(R) == 4 ? 1.0e-30 : 1.0e-60)) : s.r2);
  s.r    = s.r2 * s.rinv;
  return s;
}

// One target against one list entry, outside the softening length (r >= max(h_i, h_j)): the
// Newtonian kernel, times the TreePM short-range factor when PERIODIC.  MASK: an entry beyond Rcut
// of this target (periodic) is masked, not branched around, so that the interactions of an unrolled
// block schedule together, and the pair is counted only inside Rcut; without MASK the entry is known
// to lie inside Rcut of every target of the group and its interactions are counted per list region.
// CHECK: the entry may lie inside the softening length of this target; such a pair is masked as well
// and reported by the return value, and near() adds the spline kernel for it.  Without CHECK the list
// entry is known to lie outside the softening length of every target of the group.  The Ewald
// correction (EWALD: pure periodic tree, nearest image) is taken here for every pair.
template <typename R, bool PERIODIC, bool POT, bool EWALD = false, bool CHECK = true, bool MASK = true>
__device__ __forceinline__ bool far(const V4<R> e, const R hj, Tgt<R> &T, const W32Const &w, TabRef tab)
{
  constexpr bool PAIRWISE = MASK || CHECK;  // Rcut mask and count per pair
  // outside every target's softening length (no CHECK) r > 0 unless the softening is zero
  const Sep<R> s = separation<R, CHECK>(e, T);
  bool in        = true;
  R ff = 0, fpt = 0;
  if(PERIODIC)
    {
      if(PAIRWISE)
        in = s.r2 < rcut2_of(w, R(0));
      short_range<PAIRWISE>(s.r, w, tab, ff, fpt);
    }
  // force m (1/r^3 + f_s / (r Asmth^2)) = (m/r) (1/r^2 + f_s'), potential (m/r) p_s (Newtonian: -m/r);
  // 1/r^2 stays finite at the clamped r = 0, so masking m/r masks both
  const bool soft = CHECK && s.r < maxR(T.h, hj);
  const R m       = in ? e.w : R(0);
  const R mr      = soft ? R(0) : m * s.rinv;
  const R fm      = mr * (PERIODIC ? fmaR(s.rinv, s.rinv, ff) : s.rinv * s.rinv);
  T.ax            = fmaR(s.dx, fm, T.ax);
  T.ay            = fmaR(s.dy, fm, T.ay);
  T.az            = fmaR(s.dz, fm, T.az);
  if(POT)
    T.pot = PERIODIC ? fmaR(mr, fpt, T.pot) : T.pot - mr;
  if(EWALD)
    {
      const float4 c = ewald_corr32((float)s.dx, (float)s.dy, (float)s.dz, w);
      T.ax           = fmaR(m, (R)c.x, T.ax);
      T.ay           = fmaR(m, (R)c.y, T.ay);
      T.az           = fmaR(m, (R)c.z, T.az);
      if(POT)
        T.pot = fmaR(m, (R)c.w, T.pot);
    }
  if(PAIRWISE)
    T.ni += in ? 1 : 0;  // list entries all have mass != 0
  return soft;
}

// The softened kernel of one target against one list entry, for a pair inside the softening length
// (nothing otherwise): the reference's spline (src/gravity/forcetree_walk.c:421-455), plus the
// TreePM short-range correction of the Newtonian part away from r = 0.
template <typename R, bool PERIODIC, bool POT>
__device__ __forceinline__ void near(const V4<R> e, const R hj, Tgt<R> &T, const W32Const &w, TabRef tab)
{
  const Sep<R> s = separation<R>(e, T);
  const R hmax   = maxR(T.h, hj);
  if(!(s.r < hmax))
    return;
  const R h_inv  = R(1) / hmax;
  const R h3_inv = h_inv * h_inv * h_inv;
  const R u      = s.r * h_inv;
  const R u2     = u * u;
  R fac, wp = 0;
  if(u < R(0.5))
    {
      fac = h3_inv * fmaR(u2, fmaR((R)SF2, u, (R)SF3), (R)SF1);
      if(POT)
        wp = h_inv * fmaR(u2, fmaR(u2, fmaR((R)SF6, u, (R)SF7), (R)SF5), (R)SF4);
    }
  else
    {
      const R u3 = u2 * u;
      fac = h3_inv * ((R)SF8 + (R)SF9 * u + (R)SF10 * u2 + (R)SF11 * u3 + (R)SF12 / u3);
      if(POT)
        wp = h_inv * ((R)SF13 + (R)SF14 / u + u2 * ((R)SF1 + u * ((R)SF15 + u * ((R)SF16 + (R)SF17 * u))));
    }
  bool in = true;
  if(PERIODIC)
    {
      in = s.r2 < rcut2_of(w, R(0));
      if(s.r > R(0))
        {
          R ff, fpt;
          short_range(s.r, w, tab, ff, fpt);
          fac = fmaR(s.rinv, ff, fac);
          if(POT)
            wp = fmaR(s.rinv, fpt + R(1), wp);
        }
    }
  const R m  = in ? e.w : R(0);
  const R fm = fac * m;
  T.ax       = fmaR(s.dx, fm, T.ax);
  T.ay       = fmaR(s.dy, fm, T.ay);
  T.az       = fmaR(s.dz, fm, T.az);
  if(POT)
    T.pot = fmaR(m, wp, T.pot);
}

#ifdef GG_WALK32_STATS
}  // namespace
// measurement build only: [0] list entries evaluated per lane, [1] node tests, [2] particle candidates,
// [3] groups, [4] entries inside Rcut of every target, [5] border entries, [6] warp steps, [7] steps
// with a per-target vote, [8] voting nodes, [9] particle rounds, [10] list evaluations
constexpr int kWalkStats = 12;
__device__ unsigned long long g_walk_stats[kWalkStats];
namespace
{
#define WALK_STAT(i, v)                       \
  do                                          \
    {                                         \
      if((threadIdx.x & 31) == 0)             \
        atomicAdd(&g_walk_stats[i], (unsigned long long)(v)); \
    }                                         \
  while(0)
#else
#define WALK_STAT(i, v) \
  do                    \
    {                   \
    }                   \
  while(0)
#endif

// The lane's TPL targets against one region of the warp's list (each entry read once for all of
// them), in blocks of kUnroll entries evaluated without branches.  CHECK (near list): a block in
// which some pair lies inside the softening length (the targets' own particles, close neighbours)
// is revisited for those pairs.  MASK: per-pair Rcut mask and count (see far()).
template <typename R, bool PERIODIC, bool POT, int TPL, bool EWALD, bool CHECK, bool MASK, int U = kUnroll<TPL>>
__device__ __forceinline__ void evaluate_region(const V4<R> *__restrict__ LP, const R *__restrict__ LH, int nl, Tgt<R> (&T)[TPL],
                                                const W32Const &w, TabRef tab)
{
  int j = 0;
  for(; j + U <= nl; j += U)
    {
      V4<R> e[U];
      R hj[U];
#pragma unroll
      for(int u = 0; u < U; u++)
        {
          e[u]  = LP[j + u];
          hj[u] = CHECK ? LH[j + u] : R(0);
        }
      unsigned soft = 0;
#pragma unroll
      for(int u = 0; u < U; u++)
#pragma unroll
        for(int k = 0; k < TPL; k++)
          soft |= far<R, PERIODIC, POT, EWALD, CHECK, MASK>(e[u], hj[u], T[k], w, tab) ? 1u << (u * TPL + k) : 0u;
      if(CHECK)
        for(; soft; soft &= soft - 1)
          {
            const int b = __ffs(soft) - 1;
            if(TPL == 2 && (b & 1))
              near<R, PERIODIC, POT>(LP[j + b / TPL], LH[j + b / TPL], T[TPL - 1], w, tab);
            else
              near<R, PERIODIC, POT>(LP[j + b / TPL], LH[j + b / TPL], T[0], w, tab);
          }
    }
  for(; j < nl; j++)
    {
      const V4<R> e = LP[j];
      const R hj    = CHECK ? LH[j] : R(0);
#pragma unroll
      for(int k = 0; k < TPL; k++)
        if(far<R, PERIODIC, POT, EWALD, CHECK, MASK>(e, hj, T[k], w, tab) && CHECK)
          near<R, PERIODIC, POT>(e, hj, T[k], w, tab);
    }
}

// ---- packed evaluation: the lane's two targets as the halves of 64-bit register pairs ----
// Blackwell's f32x2 instructions do the same IEEE operation on both halves, so a pair's sums are bitwise
// those of far().  They keep the FP32 pipe's rate (two cycles each) but take one issue slot for two
// operations, which leaves slots to the warps that traverse.  Per entry and two targets, 24 warps per SM,
// measured apart from the walk: scalar 48.3 instructions and 14.2 SM cycles, packed 32.1 and 13.1 (without
// a short-range table 30.3 and 9.0 against 17.3 and 7.6); the FP32 operations alone take 9.5 (6.5).
typedef unsigned long long f2;
__device__ __forceinline__ f2 pk(float a, float b)
{
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void upk(f2 v, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c)
{
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f2 fma2_rd(f2 a, f2 b, f2 c)
{
  f2 r;
  asm("fma.rm.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b)
{
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b)
{
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
struct Sum2
{
  f2 ax, ay, az, pot;
};

// far() for the lane's two targets at once; N: their negated positions.  CHECK (near list, hj the entry's
// softening): bit k of the result says that target k lies inside the softening length (masked here).
template <bool PERIODIC, bool POT, bool MASK, bool CHECK>
__device__ __forceinline__ unsigned far2(const float4 e, const float hj, const f2 (&N)[3], Tgt<float> (&T)[2], Sum2 &S, const W32Const &w,
                                         TabRef tab, f2 afac, f2 big)
{
  const f2 dx = add2(pk(e.x, e.x), N[0]), dy = add2(pk(e.y, e.y), N[1]), dz = add2(pk(e.z, e.z), N[2]);
  const f2 r2 = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
  float r2a, r2b;
  upk(r2, r2a, r2b);
  const float ra = rsqrt_normal(CHECK ? fmaxf(r2a, 1.0e-30f) : r2a), rb = rsqrt_normal(CHECK ? fmaxf(r2b, 1.0e-30f) : r2b);
  const f2 rinv = pk(ra, rb);
  const f2 r    = mul2(r2, rinv);
  float ma = e.w, mb = e.w;
  f2 ff = 0, fpt = pk(-1.0f, -1.0f);
  if(PERIODIC)
    {
      f2 tb = fma2_rd(r, afac, big);
      float ta, tc;
      upk(tb, ta, tc);
      if(MASK)
        {
          const bool ina = r2a < w.rcut2, inb = r2b < w.rcut2;
          ma = ina ? e.w : 0.0f;
          mb = inb ? e.w : 0.0f;
          T[0].ni += ina ? 1 : 0;
          T[1].ni += inb ? 1 : 0;
          ta = fminf(ta, 12582912.0f + (float)(kNtab - 1));
          tc = fminf(tc, 12582912.0f + (float)(kNtab - 1));
          tb = pk(ta, tc);
        }
      const float4 qa = tab.row[(__float_as_int(ta) - 0x4B400000) * kCopies], qb = tab.row[(__float_as_int(tc) - 0x4B400000) * kCopies];
      float wa, wb;
      upk(fma2(r, afac, fma2(tb, pk(-1.0f, -1.0f), big)), wa, wb);
      ff  = pk(fmaf(wa, qa.y, qa.x), fmaf(wb, qb.y, qb.x));
      fpt = pk(fmaf(wa, qa.w, qa.z), fmaf(wb, qb.w, qb.z));
    }
  else if(MASK)
    {
      T[0].ni++;
      T[1].ni++;
    }
  unsigned soft = 0;
  if(CHECK)
    {
      float r_a, r_b;
      upk(r, r_a, r_b);
      const bool sa = r_a < fmaxf(T[0].h, hj), sb = r_b < fmaxf(T[1].h, hj);
      ma   = sa ? 0.0f : ma;
      mb   = sb ? 0.0f : mb;
      soft = (sa ? 1u : 0u) | (sb ? 2u : 0u);
    }
  const f2 mr = mul2(pk(ma, mb), rinv);
  const f2 fm = mul2(mr, PERIODIC ? fma2(rinv, rinv, ff) : mul2(rinv, rinv));
  S.ax        = fma2(dx, fm, S.ax);
  S.ay        = fma2(dy, fm, S.ay);
  S.az        = fma2(dz, fm, S.az);
  if(POT)
    S.pot = fma2(mr, fpt, S.pot);
  return soft;
}

// evaluate_region for two FP32 targets per lane
template <bool PERIODIC, bool POT, bool MASK, bool CHECK>
__device__ __forceinline__ void evaluate_region2(const float4 *__restrict__ LP, const float *__restrict__ LH, int nl, Tgt<float> (&T)[2],
                                                 const W32Const &w, TabRef tab)
{
  constexpr int U = kUnroll<2>;
  Sum2 S;
  auto pack = [&]() {
    S.ax  = pk(T[0].ax, T[1].ax);
    S.ay  = pk(T[0].ay, T[1].ay);
    S.az  = pk(T[0].az, T[1].az);
    S.pot = pk(T[0].pot, T[1].pot);
  };
  auto unpack = [&]() {
    upk(S.ax, T[0].ax, T[1].ax);
    upk(S.ay, T[0].ay, T[1].ay);
    upk(S.az, T[0].az, T[1].az);
    upk(S.pot, T[0].pot, T[1].pot);
  };
  // the pairs of the last entries that lie inside the softening length (bit 2 u + k)
  auto softened = [&](int j, unsigned bits) {
    unpack();
#pragma unroll 1
    for(; bits; bits &= bits - 1)
      {
        const int b = __ffs(bits) - 1;
        if(b & 1)
          near<float, PERIODIC, POT>(LP[j + (b >> 1)], LH[j + (b >> 1)], T[1], w, tab);
        else
          near<float, PERIODIC, POT>(LP[j + (b >> 1)], LH[j + (b >> 1)], T[0], w, tab);
      }
    pack();
  };
  pack();
  const f2 afac = pk(w.asmthfac, w.asmthfac), big = pk(12582912.0f, 12582912.0f);
  const f2 N[3] = {pk(-T[0].x, -T[1].x), pk(-T[0].y, -T[1].y), pk(-T[0].z, -T[1].z)};
  int j         = 0;
  for(; j + U <= nl; j += U)
    {
      float4 e[U];
      float hj[U];
#pragma unroll
      for(int u = 0; u < U; u++)
        {
          e[u]  = LP[j + u];
          hj[u] = CHECK ? LH[j + u] : 0.0f;
        }
      unsigned bits = 0;
#pragma unroll
      for(int u = 0; u < U; u++)
        bits |= far2<PERIODIC, POT, MASK, CHECK>(e[u], hj[u], N, T, S, w, tab, afac, big) << (2 * u);
      if(CHECK && bits)
        softened(j, bits);
    }
  for(; j < nl; j++)
    {
      const unsigned bits = far2<PERIODIC, POT, MASK, CHECK>(LP[j], CHECK ? LH[j] : 0.0f, N, T, S, w, tab, afac, big);
      if(CHECK && bits)
        softened(j, bits);
    }
  unpack();
}

// The warp's interaction list in shared memory.  Main buffer: entries outside the softening length of
// every target of the group, those inside Rcut of every target at the bottom (growing up, `na`),
// the others at the top (growing down, `nb`).  Near buffer (`nn`): entries inside some target's
// softening length, with their softening lengths.
template <typename R>
struct List
{
  V4<R> *P;
  V4<R> *NP;
  R *NH;
  int na, nb, nn;
};

// Evaluates and empties the list, then folds the batch partials into the lane's FP64 sums (shared
// memory, dsum[(4k + c) * 32] for target k and component c = x, y, z, potential).
// NU: entries per block of the near list; a block's softened pairs follow its others, so the order of the
// sums depends on it (a split group keeps that of the whole one).
template <typename R, bool PERIODIC, bool POT, int TPL, bool EWALD, int NU>
__device__ __forceinline__ void evaluate(List<R> &L, Tgt<R> (&T)[TPL], double *dsum, const W32Const &w, TabRef tab)
{
  WALK_STAT(4, L.na);
  WALK_STAT(5, L.nb);
  if constexpr(TPL == 2 && sizeof(R) == 4)
    {
      evaluate_region2<PERIODIC, POT, false, false>(L.P, nullptr, L.na, T, w, tab);
      if(PERIODIC)
        evaluate_region2<PERIODIC, POT, true, false>(L.P + Cap<R>::list - L.nb, nullptr, L.nb, T, w, tab);
      evaluate_region2<PERIODIC, POT, true, true>(L.NP, L.NH, L.nn, T, w, tab);
    }
  else
    {
      evaluate_region<R, PERIODIC, POT, TPL, EWALD, false, false>(L.P, nullptr, L.na, T, w, tab);
      if(PERIODIC)  // without Rcut no entry is a border entry
        evaluate_region<R, PERIODIC, POT, TPL, EWALD, false, true>(L.P + Cap<R>::list - L.nb, nullptr, L.nb, T, w, tab);
      evaluate_region<R, PERIODIC, POT, TPL, EWALD, true, true, NU>(L.NP, L.NH, L.nn, T, w, tab);
    }
#pragma unroll
  for(int k = 0; k < TPL; k++)
    {
      T[k].ni += L.na;
      dsum[(4 * k + 0) * 32] += T[k].ax;
      dsum[(4 * k + 1) * 32] += T[k].ay;
      dsum[(4 * k + 2) * 32] += T[k].az;
      if(POT)
        dsum[(4 * k + 3) * 32] += T[k].pot;
      T[k].ax = T[k].ay = T[k].az = T[k].pot = R(0);
    }
  L.na = L.nb = L.nn = 0;
}

// true when a push round of up to 32 entries could overflow a buffer
template <typename R>
__device__ __forceinline__ bool list_full(const List<R> &L)
{
  return L.na + L.nb + 32 > Cap<R>::list || L.nn + 32 > Cap<R>::near_cap;
}

// Appends one entry per lane that keeps one to the warp's list.  The entry (x, y, z relative to the
// group centre, mass) lies at squared distance d2 from the nearest point of the group box (half
// extents bx, by, bz); hn is the larger of the group's largest softening (with margin) and the
// entry's own.  Closer than hn: near list.  Otherwise, when its farthest distance from the box is
// below Rcut (with margin) or there is no Rcut: inside Rcut of every target; else the border region.
template <typename R, bool PERIODIC>
__device__ __forceinline__ void push(List<R> &L, bool keep, const V4<R> e, R h, float d2, float hn, float bx, float by, float bz,
                                     const W32Const &w, unsigned lt_mask)
{
  const bool nr     = d2 < hn * hn;
  const unsigned kn = __ballot_sync(0xffffffffu, keep && nr);
  keep              = keep && !nr;
  unsigned ka, kb;
  int at;
  if(PERIODIC)
    {
      const float fx = fabsf((float)e.x) + bx, fy = fabsf((float)e.y) + by, fz = fabsf((float)e.z) + bz;
      // the unmasked evaluation indexes the table by r = r2 / sqrt(r2), which takes a normal r2: without
      // softening (hn = 0) a target's own entry goes where the index is clamped
      const bool all = fmaf(fx, fx, fmaf(fy, fy, fz * fz)) < w.rcut2_all && d2 >= 4.0e-38f;
      ka             = __ballot_sync(0xffffffffu, keep && all);
      kb             = __ballot_sync(0xffffffffu, keep && !all);
      at             = all ? L.na + __popc(ka & lt_mask) : Cap<R>::list - 1 - (L.nb + __popc(kb & lt_mask));
      L.nb += __popc(kb);
    }
  else
    {
      ka = __ballot_sync(0xffffffffu, keep);
      at = L.na + __popc(ka & lt_mask);
    }
  if(keep)
    L.P[at] = e;
  L.na += __popc(ka);
  if(kn)
    {
      if(kn >> (threadIdx.x & 31) & 1u)
        {
          const int q = L.nn + __popc(kn & lt_mask);
          L.NP[q]     = e;
          L.NH[q]     = h;
        }
      L.nn += __popc(kn);
    }
}

// A warp's group: centre (FP64), half extents, smallest and (with margin) largest target softening,
// smallest ErrTolForceAcc x |OldAcc|, and the per-target vote's squared size bound.
struct GroupSh
{
  double gx, gy, gz;
  float ex, ey, ez, h_min, h_grp, aold_min, vote_r2;
};

// A warp's shared memory: its list, and cold per-lane and per-warp state kept out of registers -- the
// FP64 sums of the lanes' targets, ErrTolForceAcc x |OldAcc| of the targets (read by the per-target
// vote), the group, the warp's interaction total.
template <typename R, int TPL>
struct WarpSh
{
  V4<R> p[Cap<R>::list];
  V4<R> np[Cap<R>::near_cap];
  R nh[Cap<R>::near_cap];
  double dsum[4 * TPL][32];
  float aold[32 * TPL];
  unsigned long long total;
  GroupSh group;
};
// A block's shared memory (dynamic: the FP32 TreePM walk's block needs 212 KB)
template <typename R, bool PERIODIC, int TPL>
struct BlockSh
{
  WarpSh<R, TPL> warp[Shape<R, PERIODIC, TPL>::warps];
  std::conditional_t<Shape<R, PERIODIC, TPL>::big, TabF, TabNone> tab;
  __align__(16) unsigned char w_raw[kW32Bytes<R>];
};

// SPLIT (two targets per lane, few groups): a group goes to two warps; both make its whole traversal, which
// gives both the same lists, and each evaluates one target per lane.  While there are fewer groups than
// half the warps the walk takes as long as its slowest warp, and the evaluation is most of that.
template <bool PERIODIC, bool POT, int TPL, bool EWALD = false, typename R = float, bool SPLIT = false>
__global__ void __launch_bounds__(32 * Shape<R, PERIODIC, TPL>::warps, Shape<R, PERIODIC, TPL>::blocks)
    k_walk32(const double4 *__restrict__ g_sm, const float4 *__restrict__ g_rel, const int4 *__restrict__ g_kids,
             const double4 *__restrict__ g_pm, const uint8_t *__restrict__ g_pst, const double4 *__restrict__ tpm,
             const uint8_t *__restrict__ tst, const float *__restrict__ oldacc, const int *__restrict__ ngroups_dev,
             const int4 *__restrict__ groups, const int *__restrict__ order, const int32_t *__restrict__ tlist, int slice,
             int nslices, const int64_t *__restrict__ slice_rng, const W32Const *__restrict__ wcp, int *__restrict__ stack_base,
             int *__restrict__ work, double4 *__restrict__ res_out, int32_t *__restrict__ nint_out,
             unsigned long long *__restrict__ total, int *__restrict__ err, const int *__restrict__ layout_err)
{
  constexpr int kWarps = Shape<R, PERIODIC, TPL>::warps;
  constexpr bool WRAP  = PERIODIC || EWALD;  // nearest images in a periodic box
  extern __shared__ __align__(16) unsigned char sh_raw[];
  BlockSh<R, PERIODIC, TPL> &sh = *reinterpret_cast<BlockSh<R, PERIODIC, TPL> *>(sh_raw);
  const W32Const &w             = *reinterpret_cast<const W32Const *>(sh.w_raw);
  static_assert(kW32Bytes<R> % 4 == 0, "constants copied in 4-byte words");
  for(int t = threadIdx.x; t < kW32Bytes<R> / 4; t += blockDim.x)
    ((int *)sh.w_raw)[t] = ((const int *)wcp)[t];
  const int warp         = threadIdx.x >> 5;
  const int lane         = threadIdx.x & 31;
  const unsigned lt_mask = (1u << lane) - 1u;
  TabRef tab{nullptr};
  if constexpr(Shape<R, PERIODIC, TPL>::big)
    {
      for(int t = threadIdx.x; t < (kNtab + 1) * kCopies; t += blockDim.x)
        sh.tab.row[t] = wcp->tab[t / kCopies];
      tab.row = sh.tab.row + lane % kCopies;
    }
  __syncthreads();

  if(*layout_err)
    return;  // the layout's self-check failed: its indices cannot be trusted
  int *stack = stack_base + ((int64_t)blockIdx.x * kWarps + warp) * kStackCap;
  WarpSh<R, TPL> &ws = sh.warp[warp];
  List<R> L;
  L.P  = ws.p;
  L.NP = ws.np;
  L.NH = ws.nh;
  double *dsum = &ws.dsum[0][lane];
  if(lane == 0)
    ws.total = 0;
  // groups of this target slice; the count lives on the device (no host round trip, graph replays)
  const int64_t ng       = *ngroups_dev;
  // (or the cost-balanced range computed on the device, slice_rng[0..1])
  const int g_begin = slice_rng ? (int)slice_rng[0] : (int)(ng * slice / nslices);
  const int g_end   = slice_rng ? (int)slice_rng[1] : (int)(ng * (slice + 1) / nslices);
  // a warp's first unit (group, or half of one) is its number, counted over the blocks first so that a
  // small walk spreads over the SMs; the next ones come from the counter
  constexpr int UPG = SPLIT ? 2 : 1;  // units per group
  constexpr int TE  = TPL / UPG;      // targets per lane that this warp evaluates
  int unit          = warp * (int)gridDim.x + (int)blockIdx.x;

  while(true)
    {
      const int slot = g_begin + unit / UPG, half = SPLIT ? unit & 1 : 0;
      if(slot >= g_end)
        break;
      const int grp = order ? order[slot] : slot;
      // group of up to 32*TPL consecutive targets; lane holds targets t0 + lane + 32k.  A group lies
      // inside one system and walks that system's tree (root).
      const int4 G       = groups[grp];
      const int64_t t0   = G.x;
      const int cnt      = G.y;
      const int root     = G.z;
      const int bh       = G.w >= 0 ? G.w : w.bh;
      WALK_STAT(3, 1);
      double4 p[TPL];
      double mnx = 1e300, mxx = -1e300, mny = 1e300, mxy = -1e300, mnz = 1e300, mxz = -1e300;
      float hmin_l = 3.0e38f, hmax_l = 0.0f, amin_l = 3.0e38f;
#pragma unroll
      for(int k = 0; k < TPL; k++)
        {
          const int s      = lane + 32 * k;
          // idle slots repeat the group's first target; a group of active targets (tlist) holds
          // consecutive entries of the active list
          const int64_t tt = tlist ? (int64_t)tlist[t0 + (s < cnt ? s : 0)] : t0 + (s < cnt ? s : 0);
          p[k]             = tpm[tt];
          const float a_l  = w.erracc * oldacc[tt];
          ws.aold[s] = a_l;
          mnx = fmin(mnx, p[k].x), mxx = fmax(mxx, p[k].x);
          mny = fmin(mny, p[k].y), mxy = fmax(mxy, p[k].y);
          mnz = fmin(mnz, p[k].z), mxz = fmax(mxz, p[k].z);
          hmin_l = fminf(hmin_l, w.soft[tst[tt]]);
          hmax_l = fmaxf(hmax_l, w.soft[tst[tt]]);
          amin_l = fminf(amin_l, a_l);
        }
      // group box (FP64), centre g, half extent (rounded up)
      mnx = wmin(mnx), mxx = wmax(mxx), mny = wmin(mny), mxy = wmax(mxy), mnz = wmin(mnz), mxz = wmax(mxz);
      {
        GroupSh g;
        g.gx = 0.5 * (mnx + mxx), g.gy = 0.5 * (mny + mxy), g.gz = 0.5 * (mnz + mxz);
        g.ex = (float)(0.5 * (mxx - mnx)) * 1.000001f, g.ey = (float)(0.5 * (mxy - mny)) * 1.000001f,
        g.ez = (float)(0.5 * (mxz - mnz)) * 1.000001f;
        g.h_min = wminf(hmin_l);
        // an entry farther than max(h_grp, h_j) from the group box is outside the softening length of
        // every target (the margin covers the rounding of the FP32 separations)
        g.h_grp    = wmaxf(hmax_l) * 1.001f;
        g.aold_min = wminf(amin_l);
        // box side squared over kVote^2: a node smaller than this and closer than it gets the per-target vote
        const float side = 2.0f * fmaxf(g.ex, fmaxf(g.ey, g.ez));
        g.vote_r2        = side * side * (1.0f / (kVote * kVote));
        if(lane == 0)
          ws.group = g;
      }
      __syncwarp();
      // the group's constants are read from shared memory where they are used (out of registers)
      const GroupSh &gs = ws.group;
      const double &gx = gs.gx, &gy = gs.gy, &gz = gs.gz;
      const float &ex = gs.ex, &ey = gs.ey, &ez = gs.ez, &h_min = gs.h_min, &h_grp = gs.h_grp, &aold_min = gs.aold_min,
                  &vote_r2 = gs.vote_r2;
      Tgt<R> T[TPL];
#pragma unroll
      for(int k = 0; k < TPL; k++)
        {
          T[k].x = (R)(p[k].x - gx), T[k].y = (R)(p[k].y - gy), T[k].z = (R)(p[k].z - gz);
          const int sk = lane + 32 * k < cnt ? lane + 32 * k : 0;
          T[k].h       = (R)w.soft[tst[tlist ? (int64_t)tlist[t0 + sk] : t0 + sk]];
        }
      // the targets that this warp evaluates
      Tgt<R> E[TE];
#pragma unroll
      for(int k = 0; k < TE; k++)
        {
          E[k]    = SPLIT && half ? T[TPL - 1] : T[k];
          E[k].ax = E[k].ay = E[k].az = E[k].pot = R(0);
#pragma unroll
          for(int c = 0; c < 4; c++)
            dsum[(4 * k + c) * 32] = 0.0;
          E[k].ni = 0;
        }

      int sp = 1;
      L.na = L.nb = L.nn = 0;
      if(lane == 0)
        stack[0] = root;
      __syncwarp();

      // The walk is a loop over warp-uniform work items, so that the list evaluation has a single
      // (inlined) site: a pending softening-type entry of MULTIPLE_NODE_SOFTENING nodes (t_next <
      // t_end), a pending round of up to 32 particles of opened nodes (q0 < ptot), or a step over
      // up to 32 stack nodes.  The list is evaluated first when the next item could overflow it,
      // when it is full enough at a node step, and at the end.
      int t_next = 0, t_end = 0;  // MULTIPLE_NODE_SOFTENING entries of the last node step
      int q0 = 0, ptot = 0;       // particle rounds of the last node step
      // per-lane state of the last node step, read by the pending items
      int node = -1, action = 0, fp = 0, pinc = 0, pexc = 0;
      bool split = false;
      V4<R> entry  = mk4<R>(0, 0, 0, 0);
      float ent_d2 = 0.0f;  // squared distance of the entry from the group box
      while(true)
        {
          const int queued = L.na + L.nb + L.nn;
          const bool flush = (t_next < t_end || q0 < ptot) ? list_full(L)
                                                           : (sp > 0 ? (queued >= Cap<R>::eval || L.nn >= Cap<R>::near_at)
                                                                     : queued > 0);
          if(flush)
            {
              WALK_STAT(0, queued);
              WALK_STAT(10, 1);
              __syncwarp();  // every lane reads the entries that the others have put
              evaluate<R, PERIODIC, POT, TE, EWALD, kUnroll<TPL>>(L, E, dsum, w, tab);
              __syncwarp();
            }
          if(t_next < t_end)
            {
              // MULTIPLE_NODE_SOFTENING: one entry per softening type with that type's mass and softening
              // (forcetree_walk.c:382-401); for a target whose own softening exceeds the node's largest
              // this equals the single entry, the kernel being linear in the mass
              const int t    = t_next++;
              const float mt = (action == 1 && split) ? w.mpt[(int64_t)node * w.nsoft + t] : 0.0f;
              push<R, PERIODIC>(L, mt != 0.0f, mk4<R>(entry.x, entry.y, entry.z, mt), (R)w.soft[t], ent_d2,
                                fmaxf(h_grp, w.soft[t]), ex, ey, ez, w, lt_mask);
              continue;
            }
          if(q0 < ptot)
            {
              // particles of opened nodes -> list, one particle per lane per round; particles beyond
              // Rcut of the whole group are dropped
              const int q = q0 + lane;
              q0 += 32;
              WALK_STAT(9, 1);
              int owner = 0;  // owner lane: number of lanes whose inclusive prefix is <= q
#pragma unroll
              for(int s = 16; s >= 1; s >>= 1)
                {
                  const int v = __shfl_sync(0xffffffffu, pinc, owner + s - 1);
                  if(v <= q)
                    owner += s;
                }
              owner          = owner < 31 ? owner : 31;
              const int ofp  = __shfl_sync(0xffffffffu, fp, owner);
              const int oexc = __shfl_sync(0xffffffffu, pexc, owner);
              bool keep      = false;
              V4<R> pe       = mk4<R>(0, 0, 0, 0);
              float ph = 0, pd2 = 0;
              if(q < ptot)
                {
                  const int pi     = ofp + (q - oexc);
                  const double4 pp = load32(g_pm + pi);
                  pe   = mk4<R>(wrapd<WRAP>(pp.x - gx, w), wrapd<WRAP>(pp.y - gy, w), wrapd<WRAP>(pp.z - gz, w), pp.w);
                  ph   = w.soft[g_pst[pi]];
                  keep = pp.w != 0.0;
                  const float dmx = fmaxf(fabsf((float)pe.x) - ex, 0.0f), dmy = fmaxf(fabsf((float)pe.y) - ey, 0.0f),
                              dmz = fmaxf(fabsf((float)pe.z) - ez, 0.0f);
                  pd2 = dmx * dmx + dmy * dmy + dmz * dmz;
                  if(PERIODIC)
                    keep = keep && pd2 < w.rcut2;
                }
              push<R, PERIODIC>(L, keep, pe, (R)ph, pd2, fmaxf(h_grp, ph), ex, ey, ez, w, lt_mask);
              continue;
            }
          if(sp == 0)
            break;

          // ---- node step: up to 32 stack nodes, one per lane ----
          const int take = sp < 32 ? sp : 32;
          sp -= take;
          WALK_STAT(1, take);
          WALK_STAT(6, 1);
          node = -1;
          if(lane < take)
            node = stack[sp + lane];
          __syncwarp();

          action = 0;  // 1 accept, 2 open
          entry  = mk4<R>(0, 0, 0, 0);
          ent_d2 = 0.0f;
          split  = false;  // MULTIPLE_NODE_SOFTENING: accepted node listed per type
          float hj = 0;
          int fc = 0, nc = 0, np = 0;
          fp = 0;
          bool vote = false, vote_keep = false;  // per-target vote pending; entry kept if accepted
          float4 vrel = make_float4(0, 0, 0, 0);   // centre - CoM, side of a voting node
          if(node >= 0)
            {
              // the three records of the node are fetched together (one memory round trip)
              const double4 sm = load32(g_sm + node);
              const float4 rel = g_rel[node];
              const int4 kd    = g_kids[node];
              if(sm.w != 0.0)
                {
                  const double dsx = wrapd<WRAP>(sm.x - gx, w), dsy = wrapd<WRAP>(sm.y - gy, w), dsz = wrapd<WRAP>(sm.z - gz, w);
                  const float sx = (float)dsx, sy = (float)dsy, sz = (float)dsz;
                  const float cx = sx + rel.x, cy = sy + rel.y, cz = sz + rel.z;
                  const float L  = rel.w;
                  const float m  = (float)sm.w;
                  hj             = w.soft[kd.w];
                  bool prune     = false;
                  if(PERIODIC)
                    {
                      const float eff = w.rcut + 0.5f * L;
                      prune = (fabsf(cx) - ex > eff) || (fabsf(cy) - ey > eff) || (fabsf(cz) - ez > eff);
                    }
                  if(!prune)
                    {
                      const float dmx = fmaxf(fabsf(sx) - ex, 0.0f), dmy = fmaxf(fabsf(sy) - ey, 0.0f),
                                  dmz = fmaxf(fabsf(sz) - ez, 0.0f);
                      const float rmin2 = dmx * dmx + dmy * dmy + dmz * dmz;
                      const float L2    = L * L;
                      bool open;
                      if(bh)
                        open = L2 > rmin2 * w.theta2;
                      else
                        // with ACTIVATE_MINIMUM_OPENING_ANGLE the mass test also needs the node to span more than
                        // 0.4 radian from the nearest point of the box (conservative for every target)
                        open = (L2 > rmin2 * 1.44f) ||
                               (m * L2 > rmin2 * rmin2 * aold_min && (!w.minangle || L2 > rmin2 * 0.16f)) ||
                               (fabsf(cx) < 0.6f * L + ex && fabsf(cy) < 0.6f * L + ey && fabsf(cz) < 0.6f * L + ez);
                      if(!open && hj > h_min)
                        {
                          // a target's softening is below the node's largest: open inside that
                          // softening, or (MULTIPLE_NODE_SOFTENING) use the node per softening type
                          if(w.mns)
                            split = true;
                          else if(rmin2 < hj * hj)
                            open = true;
                        }
                      if(open)
                        {
                          action = 2;
                          fc     = kd.x;
                          fp     = kd.y;
                          nc     = kd.z & 15;
                          np     = (kd.z >> 4) & 15;
                          if(L2 < vote_r2 && rmin2 < vote_r2)
                            {
                              vote      = true;
                              vote_keep = !PERIODIC || rmin2 < w.rcut2;
                              vrel      = rel;
                              entry     = mk4<R>(dsx, dsy, dsz, sm.w);
                              ent_d2    = rmin2;
                            }
                        }
                      else if(!PERIODIC || rmin2 < w.rcut2)
                        {
                          // accepted; a node whose CoM is beyond Rcut of every target contributes nothing
                          action = 1;
                          entry  = mk4<R>(dsx, dsy, dsz, sm.w);
                          ent_d2 = rmin2;
                        }
                    }
                }
            }
          // per-target vote: the node stays open only if some target's own criterion opens it
          if(const unsigned vm = __ballot_sync(0xffffffffu, vote))
            {
              WALK_STAT(7, 1);
              WALK_STAT(8, __popc(vm));
              // one voting node after the other, every lane testing its own targets
              bool need = false;
              for(unsigned v = vm; v; v &= v - 1)
                {
                  const int b     = __ffs(v) - 1;
                  const float enx = (float)__shfl_sync(0xffffffffu, entry.x, b), eny = (float)__shfl_sync(0xffffffffu, entry.y, b),
                              enz = (float)__shfl_sync(0xffffffffu, entry.z, b), em = (float)__shfl_sync(0xffffffffu, entry.w, b),
                              rx = __shfl_sync(0xffffffffu, vrel.x, b), ry = __shfl_sync(0xffffffffu, vrel.y, b),
                              rz = __shfl_sync(0xffffffffu, vrel.z, b), L = __shfl_sync(0xffffffffu, vrel.w, b),
                              hn = __shfl_sync(0xffffffffu, hj, b);
                  const float L2 = L * L;
                  bool o         = false;
#pragma unroll
                  for(int k = 0; k < TPL; k++)
                    if(lane + 32 * k < cnt)
                      {
                        const float tx = (float)T[k].x, ty = (float)T[k].y, tz = (float)T[k].z, ta = ws.aold[lane + 32 * k];
                        const float dx = enx - tx, dy = eny - ty, dz = enz - tz;
                        const float r2 = dx * dx + dy * dy + dz * dz;
                        if(bh)
                          o |= L2 > r2 * w.theta2;
                        else
                          o |= (L2 > r2 * 1.44f) || (em * L2 > r2 * r2 * ta && (!w.minangle || L2 > r2 * 0.16f)) ||
                               (fabsf(enx + rx - tx) < 0.6f * L && fabsf(eny + ry - ty) < 0.6f * L && fabsf(enz + rz - tz) < 0.6f * L);
                        o |= !w.mns && hn > (float)T[k].h && r2 < hn * hn;
                      }
                  o = __any_sync(0xffffffffu, o);
                  if(lane == b)
                    need = o;
                }
              if(vote && !need)
                {
                  action = vote_keep ? 1 : 0;
                  split  = w.mns && hj > h_min;
                  nc = np = 0;
                }
            }
          // accepted nodes -> list (the list holds fewer than Cap::eval entries, so 32 more fit);
          // nodes used per softening type follow as pending items
          push<R, PERIODIC>(L, action == 1 && !split, entry, (R)hj, ent_d2, fmaxf(h_grp, hj), ex, ey, ez, w, lt_mask);
          t_next = 0;
          t_end  = __ballot_sync(0xffffffffu, action == 1 && split) ? w.nsoft : 0;
          // particles (pending rounds) and node children of opened nodes: one scan of both counts
          // (each below 16, particles in the low half-word)
          const int npx  = (action == 2) ? np : 0;
          const int ncx  = (action == 2) ? nc : 0;
          const int both = wscan_incl(npx | (ncx << 16), lane);
          const int tot  = __shfl_sync(0xffffffffu, both, 31);
          pinc           = both & 0xffff;
          ptot           = tot & 0xffff;
          pexc           = pinc - npx;
          q0             = 0;
          WALK_STAT(2, ptot);
          // node children of opened nodes -> stack (contiguous)
          const int cinc = both >> 16;
          const int ctot = tot >> 16;
          if(sp + ctot <= kStackCap)
            {
              const int cb = sp + cinc - ncx;
              for(int q = 0; q < ncx; q++)
                stack[cb + q] = fc + q;
              sp += ctot;
            }
          else if(lane == 0)
            atomicOr(err, 16);  // stack too small: the walk of this group is incomplete
          __syncwarp();
        }
#pragma unroll
      for(int k = 0; k < TE; k++)
        {
          const int s = lane + 32 * (SPLIT ? half : k);
          if(s < cnt)
            {
              const int64_t t = tlist ? (int64_t)tlist[t0 + s] : t0 + s;
              res_out[t]  = make_double4(dsum[(4 * k + 0) * 32], dsum[(4 * k + 1) * 32], dsum[(4 * k + 2) * 32],
                                         POT ? dsum[(4 * k + 3) * 32] : 0.0);
              nint_out[t] = E[k].ni;
            }
        }
      // the group's interactions (idle slots count none)
      unsigned long long gtot = 0;
#pragma unroll
      for(int k = 0; k < TE; k++)
        gtot += lane + 32 * (SPLIT ? half : k) < cnt ? (unsigned long long)E[k].ni : 0ull;
      for(int o = 16; o > 0; o >>= 1)
        gtot += __shfl_xor_sync(0xffffffffu, gtot, o);
      int nextg = 0;
      if(lane == 0)
        {
          ws.total += gtot;
          nextg = atomicAdd(work, 1);
        }
      unit = kWarps * (int)gridDim.x + __shfl_sync(0xffffffffu, nextg, 0);
    }
  if(lane == 0 && ws.total)
    atomicAdd(total, ws.total);
}

// ---- order of the groups ----
// A walk of several groups per warp ends when its last group does, and the cost of a group under the relative
// criterion varies.  So clustered sets' groups go by falling cost, as far as it can be told before the walk, by the
// binary exponents of the smallest and the largest OldAcc of a run of groups: lo, hi.
//  * TreePM: by lo, which opens the most.  Zoom boxes with OldAcc of a previous pass, key order / this order:
//    2^19 particles 11.3 / 11.1 ms, 2^21 39.6 / 29.4, 2^24 303.9 / 295.1.  It matters most where single groups are far
//    off: with the background's OldAcc also for the few background particles inside the core (180 ms for such a
//    group against 6 for the median) the 2^24 walk takes 331 ms in key order, its last third on 80 of 3552 warps, and
//    249 in this one.
//  * isolated sets, whose cost rises inwards: by hi + 2 (hi - lo), the dear half; the rest follow by key.  By lo the
//    outskirts went first and the core last: Hernquist 2^20 2.34 ms against 1.83 in key order.  Key order / by lo /
//    this order: Plummer 2^18 1.31 / 1.30 / 1.22, 2^20 3.28 / 2.84 / 2.70, 2^22 11.4 / 11.4 / 11.6; Hernquist 2^18 0.71 /
//    0.85 / 0.78, 2^20 1.83 / 2.34 / 1.86 (with OldAcc of a previous pass 2.19 / 2.33 / 2.02), 2^22 12.3 / 11.8 / 10.5.
// Every group's result is its own; the order changes none.
constexpr int kOrderBlock = 256;
constexpr int kOrderRun   = 4;  // consecutive groups that stay together
struct GroupOrder
{
  int hist[256], cursor[256];  // groups per exponent; the scatter's reservations
};
__device__ __forceinline__ void group_range(const int *ngroups_dev, int slice, int nslices, const int64_t *slice_rng, int &b, int &e)
{
  const int64_t ng = *ngroups_dev;
  b                = slice_rng ? (int)slice_rng[0] : (int)(ng * slice / nslices);
  e                = slice_rng ? (int)slice_rng[1] : (int)(ng * (slice + 1) / nslices);
}
__global__ void __launch_bounds__(kOrderBlock) k_order_key(const int *__restrict__ ngroups_dev, int isolated, int slice, int nslices,
                                                           const int64_t *__restrict__ slice_rng, const int4 *__restrict__ groups,
                                                           const int32_t *__restrict__ tlist, const float *__restrict__ oldacc,
                                                           uint8_t *__restrict__ key, GroupOrder *__restrict__ o)
{
  __shared__ int h[256];
  for(int t = threadIdx.x; t < 256; t += blockDim.x)
    h[t] = 0;
  __syncthreads();
  int b, e;
  group_range(ngroups_dev, slice, nslices, slice_rng, b, e);
  const int lane = threadIdx.x & 31, warps = gridDim.x * (kOrderBlock / 32);
  for(int r = blockIdx.x * (kOrderBlock / 32) + (threadIdx.x >> 5); b + r * kOrderRun < e; r += warps)
    {
      const int g0 = b + r * kOrderRun, g1 = g0 + kOrderRun < e ? g0 + kOrderRun : e;
      // consecutive groups hold consecutive targets
      const int4 last = groups[g1 - 1];
      float lo = 3.0e38f, hi = 0.0f;
#pragma unroll 8
      for(int k = groups[g0].x + lane; k < last.x + last.y; k += 32)
        {
          const float a = oldacc[tlist ? tlist[k] : k];
          lo            = fminf(lo, a);
          hi            = fmaxf(hi, a);
        }
      lo = wminf(lo);
      hi = wmaxf(hi);
      if(lane == 0)
        {
          const int eh = (__float_as_int(hi) >> 23) & 255, el = (__float_as_int(lo) >> 23) & 255;
          const int x  = isolated ? 255 - min(max(eh + 2 * min(max(eh - el, 0), 63) - 64, 0), 255) : el;
          key[r]       = (uint8_t)x;
          atomicAdd(&h[x], g1 - g0);
        }
    }
  __syncthreads();
  for(int t = threadIdx.x; t < 256; t += blockDim.x)
    if(h[t])
      atomicAdd(&o->hist[t], h[t]);
}
__global__ void __launch_bounds__(kOrderBlock) k_order_scatter(const int *__restrict__ ngroups_dev, int share, int slice, int nslices,
                                                               const int64_t *__restrict__ slice_rng, const uint8_t *__restrict__ key,
                                                               GroupOrder *__restrict__ o, int *__restrict__ order)
{
  static_assert(kOrderBlock == 256, "one thread per exponent");
  typedef cub::BlockScan<int, kOrderBlock> Scan;
  __shared__ typename Scan::TempStorage tmp;
  __shared__ int cnt[256], base[256], heads, first;  // heads: classes of the dear half; first: groups in them
  const int in_class = o->hist[threadIdx.x];
  int start, b, e;
  Scan(tmp).ExclusiveSum(in_class, start);
  group_range(ngroups_dev, slice, nslices, slice_rng, b, e);
  if(threadIdx.x == 0)
    heads = first = 0;
  __syncthreads();
  if(share * (int64_t)(start + in_class) <= e - b)
    {
      atomicMax(&heads, (int)threadIdx.x + 1);
      atomicMax(&first, start + in_class);
    }
  __syncthreads();
  if(threadIdx.x == 255 && heads < 256)
    start = first;  // the rest share the last class
  const int runs = (e - b + kOrderRun - 1) / kOrderRun;
  for(int r0 = blockIdx.x * kOrderBlock; r0 < runs; r0 += gridDim.x * kOrderBlock)
    {
      cnt[threadIdx.x] = 0;
      __syncthreads();
      const int r = r0 + threadIdx.x, x = r < runs ? (key[r] < heads ? key[r] : 255) : -1;
      const int g0 = b + r * kOrderRun, g1 = g0 + kOrderRun < e ? g0 + kOrderRun : e;
      const int at = x >= 0 ? atomicAdd(&cnt[x], g1 - g0) : 0;
      __syncthreads();
      base[threadIdx.x] = cnt[threadIdx.x] ? b + start + atomicAdd(&o->cursor[threadIdx.x], cnt[threadIdx.x]) : 0;
      __syncthreads();
      if(x >= 0)
        for(int g = g0; g < g1; g++)
          order[base[x] + at + g - g0] = g;
      __syncthreads();
    }
}

// ---- walk groups -------------------------------------------------------------------------
// A group is up to `cap` consecutive targets in Peano-Hilbert order, never spanning two systems.
// cd[i] is the depth of the deepest cell holding particles i and i+1 (-1 across systems and after
// the last particle).  Optionally (slack < 64) groups are also cut between tree cells: pd[i] is the
// depth of the deepest cell around particle i that holds more than cap particles (-1: its whole
// system fits in one group), and consecutive particles stay in one group only while each lies
// inside the other's pd cell (up to `slack` levels above it).  Cell cuts bound a group's box by a
// tree cell at the price of partly filled warps; the per-target vote of the walk already removes
// the cost of loose groups, and plain key-order groups are faster on the measured workloads.
// depth of the deepest cell around sorted particle i that holds more than cap particles (-1: its whole
// system fits in one group), by widening [l, r] one cell at a time along the pair depths
__device__ __forceinline__ int cap_cell_depth(int64_t i, const int8_t *__restrict__ cd, int cap)
{
  int64_t l = i, r = i;  // current cell [l, r]
  while(true)
    {
      const int dl = l > 0 ? cd[l - 1] : -1;
      const int dr = cd[r];
      const int d  = dl > dr ? dl : dr;  // depth of the next larger cell
      if(d < 0)
        return -1;
      while(l > 0 && cd[l - 1] >= d)
        if(r - --l + 1 > cap)
          return d;
      while(cd[r] >= d)
        if(++r - l + 1 > cap)
          return d;
    }
}

__global__ void k_grp_pd(int64_t n, const int8_t *__restrict__ cd, int cap, int8_t *__restrict__ pd)
{
  for(int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    pd[i] = (int8_t)cap_cell_depth(i, cd, cap);
}

// The same for an active list (targets at sorted positions tpos, in key order): the cell depth at each
// target, and the depth of the deepest cell holding consecutive targets k and k + 1 (-1 after the last)
__global__ void k_grp_pd_at(int64_t nt, const int32_t *__restrict__ tpos, const int8_t *__restrict__ cd, int cap,
                            int8_t *__restrict__ apd)
{
  for(int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nt; k += (int64_t)gridDim.x * blockDim.x)
    apd[k] = (int8_t)cap_cell_depth(tpos[k], cd, cap);
}
__global__ void k_active_cd(int64_t nt, const int32_t *__restrict__ tpos, const uint64_t *__restrict__ ix,
                            const uint64_t *__restrict__ iy, const uint64_t *__restrict__ iz, int8_t *__restrict__ acd)
{
  for(int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nt; k += (int64_t)gridDim.x * blockDim.x)
    {
      int d = -1;
      if(k + 1 < nt)
        {
          const int64_t a = tpos[k], b = tpos[k + 1];
          d               = common_depth(ix[a], iy[a], iz[a], ix[b], iy[b], iz[b]);
        }
      acd[k] = (int8_t)d;
    }
}

// segment start candidates: i where a group must begin (system start or a cut before i)
__global__ void k_grp_cut(int64_t n, const int8_t *__restrict__ cd, const int8_t *__restrict__ pd, int slack,
                          int32_t *__restrict__ segv)
{
  for(int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    {
      bool cut = (i == 0);
      if(!cut)
        {
          const int c = cd[i - 1];
          cut         = c < 0;
          if(pd && !cut)
            {
              const int p = pd[i - 1] > pd[i] ? pd[i - 1] : pd[i];
              cut         = c < p - slack;
            }
        }
      segv[i] = cut ? (int32_t)i : 0;
    }
}

__global__ void k_grp_start(int64_t n, const int32_t *__restrict__ seg, int cap, int32_t *__restrict__ flag)
{
  for(int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    flag[i] = ((i - seg[i]) % cap == 0) ? 1 : 0;
}

// group table: (first target, count, root node, -1 = criterion of the walk constants); the groups tile the
// targets, so a count is the distance to the next group's start (k_grp_count)
__global__ void k_grp_fill(int64_t n, const int32_t *__restrict__ flag, const int32_t *__restrict__ gid, const int32_t *__restrict__ sys,
                           int4 *__restrict__ groups, int *__restrict__ ngroups)
{
  for(int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    {
      if(flag[i])
        groups[gid[i]] = make_int4((int)i, 0, sys ? sys[i] : 0, -1);
      if(i == n - 1)
        *ngroups = gid[i] + flag[i];
    }
}
__global__ void k_grp_count(int64_t n, const int *__restrict__ ngroups, int4 *groups)
{
  const int ng = *ngroups;
  for(int g = blockIdx.x * blockDim.x + threadIdx.x; g < ng; g += gridDim.x * blockDim.x)
    groups[g].y = (g + 1 < ng ? groups[g + 1].x : (int)n) - groups[g].x;
}
// one system without cell cuts: consecutive chunks of cap targets
__global__ void k_grp_plain(int64_t n, int cap, int4 *__restrict__ groups, int *__restrict__ ngroups)
{
  const int ng = (int)((n + cap - 1) / cap);
  for(int g = blockIdx.x * blockDim.x + threadIdx.x; g < ng; g += gridDim.x * blockDim.x)
    {
      const int64_t i = (int64_t)g * cap;
      groups[g]       = make_int4((int)i, (int)(n - i < cap ? n - i : cap), 0, -1);
      if(g == 0)
        *ngroups = ng;
    }
}

// outputs (sorted order) of the targets outside this slice set to zero; the slice's target range
// is [start of group g_begin, start of group g_end) with the FP32 group table, else n*s/ns..
__global__ void k_slice_mask(int64_t n, int slice, int nslices, const int4 *__restrict__ groups, const int *__restrict__ ngroups,
                             const int64_t *__restrict__ slice_rng, double4 *__restrict__ res, int32_t *__restrict__ nint)
{
  int64_t t_begin, t_end;
  if(slice_rng)
    {
      t_begin = slice_rng[2];
      t_end   = slice_rng[3];
    }
  else if(groups)
    {
      const int64_t ng = *ngroups;
      const int64_t gb = ng * slice / nslices, ge = ng * (slice + 1) / nslices;
      t_begin          = gb < ng ? groups[gb].x : n;
      t_end            = ge < ng ? groups[ge].x : n;
    }
  else
    {
      t_begin = n * slice / nslices;
      t_end   = n * (slice + 1) / nslices;
    }
  for(int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    if(i < t_begin || i >= t_end)
      {
        res[i]  = make_double4(0, 0, 0, 0);
        nint[i] = 0;
      }
}

struct MaxOp32
{
  __device__ __forceinline__ int32_t operator()(int32_t a, int32_t b) const { return a > b ? a : b; }
};

int grid_for(int64_t n, int threads)
{
  int64_t b = (n + threads - 1) / threads;
  if(b > 148 * 16)
    b = 148 * 16;
  return (int)(b < 1 ? 1 : b);
}

void make_w32(const WalkConst &wc, W32Const *w)
{
  memset(w, 0, sizeof(*w));
  w->box       = wc.box;
  w->half_box  = wc.half_box;
  w->rcut      = (float)wc.rcut;
  // pairs end where the table does, if that is before Rcut (RcutCells x Asmth < Rcut), as tabindex >= NTAB
  // does in the reference; Rcut and the table's end usually agree to rounding
  const double rtab  = wc.pm ? kNtab / wc.asmthfac : wc.rcut;
  const double rcut2 = rtab * (1.0 + 1e-6) < wc.rcut ? rtab * rtab : wc.rcut2;
  w->rcut2     = (float)rcut2;
  w->rcut2_d   = rcut2;
  // margin for the rounding of the FP32 separations and the box extents (relative ~1e-6)
  w->rcut2_all = (float)(rcut2 * (1.0 - 1.0 / 4096.0));
  w->asmthfac  = (float)wc.asmthfac;
  const double finv = wc.pm ? wc.asmthinv2 : 1.0;
  w->theta2    = (float)(wc.theta * wc.theta);
  w->erracc    = (float)wc.erracc;
  w->periodic  = wc.periodic;
  w->bh        = wc.bh;
  w->ewd_fac   = (float)wc.ewd_fac_intp;
  w->mns       = wc.mns;
  w->minangle  = wc.minangle;
  w->nsoft     = wc.nsoft;
  for(int i = 0; i <= GPUGRAV_MAX_SOFTTYPES; i++)
    w->soft[i] = (float)wc.soft[i];
  for(int i = 0; i <= kNtab; i++)
    {
      float f0 = (float)(finv * wc.tab_force[i]), f1 = (float)(finv * ((i < kNtab) ? wc.tab_force[i + 1] : wc.tab_force[i]));
      float p0 = wc.tab_pot[i], p1 = (i < kNtab) ? wc.tab_pot[i + 1] : wc.tab_pot[i];
      w->tab[i] = make_float4(f0, f1 - f0, p0, p1 - p0);
      // FP64 walk: the reference's float table entries, scaled and differenced in double
      const double d0 = finv * wc.tab_force[i], d1 = finv * ((i < kNtab) ? wc.tab_force[i + 1] : wc.tab_force[i]);
      const double q0 = wc.tab_pot[i], q1 = (i < kNtab) ? wc.tab_pot[i + 1] : wc.tab_pot[i];
      w->tab64[i]     = make_double4(d0, d1 - d0, q0, q1 - q0);
    }
  w->asmthfac_d = wc.asmthfac;
}
}  // namespace

// buffers of the FP32 walk layout and group table for n particles and nn nodes
cudaError_t layout32_buffers(gpugrav_ctx *c, int64_t n, int64_t nn)
{
  GG_TRY(c->g_scan.ensure(nn * 8));
  GG_TRY(c->g_sm.ensure(nn * sizeof(double4)));
  GG_TRY(c->g_rel.ensure(nn * sizeof(float4)));
  GG_TRY(c->g_kids.ensure(nn * sizeof(int4)));
  GG_TRY(c->g_pm.ensure(n * sizeof(double4)));
  GG_TRY(c->g_pst.ensure(n + 16));
  GG_TRY(c->g_groups.ensure(n * sizeof(int4)));
  GG_TRY(c->g_ngroups.ensure(16));
  GG_TRY(c->g_gpd.ensure(n + 16));
  GG_TRY(c->g_gseg.ensure(n * 4));
  GG_TRY(c->g_gflag.ensure(n * 4));
  GG_TRY(c->g_gid.ensure(n * 4));
  return cudaSuccess;
}

// layout32_stage's buffers and temporary storage sized once for n particles and nn nodes
cudaError_t layout32_reserve(gpugrav_ctx *c, int64_t n, int64_t nn)
{
  GG_TRY(layout32_buffers(c, n, nn));
  size_t tb = 0, t2 = 0;
  GG_TRY(cub::DeviceScan::ExclusiveSum(nullptr, tb, thrust::make_transform_iterator(c->n_count.as<uint8_t>(), ChildCounts()),
                                       c->g_scan.as<uint64_t>(), (int)nn, c->stream));
  GG_TRY(cub::DeviceScan::InclusiveScan(nullptr, t2, c->g_gflag.as<int32_t>(), c->g_gseg.as<int32_t>(), MaxOp32(), (int)n,
                                        c->stream));
  tb = t2 > tb ? t2 : tb;
  GG_TRY(cub::DeviceScan::ExclusiveSum(nullptr, t2, c->g_gflag.as<int32_t>(), c->g_gid.as<int32_t>(), (int)n, c->stream));
  tb = t2 > tb ? t2 : tb;
  return c->sort_tmp.ensure(tb);
}

// walk group table of the current tree (see k_grp_pd); the group count stays on the device
cudaError_t groups_stage(gpugrav_ctx *c)
{
  const int64_t n = c->n;
  cudaStream_t st = c->stream;
  const int cap    = 32 * walk32_tpl(c);
  c->group_cap     = cap;
  GG_TRY(cudaMemsetAsync(c->g_ngroups.p, 0, sizeof(int), st));
  if(n == 0)
    return cudaSuccess;
  const bool cells = c->group_slack < 64;  // otherwise: cut at system starts only
  if(!cells && !c->multi)
    {
      k_grp_plain<<<grid_for((n + cap - 1) / cap, 256), 256, 0, st>>>(n, cap, c->g_groups.as<int4>(), c->g_ngroups.as<int>());
      return cudaGetLastError();
    }
  if(cells)
    k_grp_pd<<<grid_for(n, 256), 256, 0, st>>>(n, c->s_cd.as<int8_t>(), cap, c->g_gpd.as<int8_t>());
  k_grp_cut<<<grid_for(n, 256), 256, 0, st>>>(n, c->s_cd.as<int8_t>(), cells ? c->g_gpd.as<int8_t>() : nullptr,
                                               c->group_slack, c->g_gflag.as<int32_t>());
  size_t tb = 0;
  GG_TRY(cub::DeviceScan::InclusiveScan(nullptr, tb, c->g_gflag.as<int32_t>(), c->g_gseg.as<int32_t>(), MaxOp32(), (int)n, st));
  GG_TRY(c->sort_tmp.ensure(tb));
  GG_TRY(cub::DeviceScan::InclusiveScan(c->sort_tmp.p, tb, c->g_gflag.as<int32_t>(), c->g_gseg.as<int32_t>(), MaxOp32(), (int)n,
                                        st));
  k_grp_start<<<grid_for(n, 256), 256, 0, st>>>(n, c->g_gseg.as<int32_t>(), cap, c->g_gflag.as<int32_t>());
  tb = 0;
  GG_TRY(cub::DeviceScan::ExclusiveSum(nullptr, tb, c->g_gflag.as<int32_t>(), c->g_gid.as<int32_t>(), (int)n, st));
  GG_TRY(c->sort_tmp.ensure(tb));
  GG_TRY(cub::DeviceScan::ExclusiveSum(c->sort_tmp.p, tb, c->g_gflag.as<int32_t>(), c->g_gid.as<int32_t>(), (int)n, st));
  k_grp_fill<<<grid_for(n, 256), 256, 0, st>>>(n, c->g_gflag.as<int32_t>(), c->g_gid.as<int32_t>(),
                                                c->multi ? c->m_sys.as<int32_t>() : nullptr, c->g_groups.as<int4>(),
                                                c->g_ngroups.as<int>());
  k_grp_count<<<grid_for((n + cap - 1) / cap, 256), 256, 0, st>>>(n, c->g_ngroups.as<int>(), c->g_groups.as<int4>());
  return cudaGetLastError();
}

// walk group table of an active list (gravity_tree(timebin)'s TargetList, sorted positions in key
// order in tpos): up to cap consecutive active targets, also cut where two consecutive targets share
// only a cell more than active_slack levels above the cells of cap particles around them -- active
// targets that follow each other in key order can lie far apart (the background particles on both
// sides of a dense core), and one group box spanning the core would open it for every target.  On the
// zoom box at N = 2^24 the walk of the 2^23 background particles alone takes 55 ms with slack 2
// against 259 ms without cuts; the Plummer particles alone are within 0.6 %.
cudaError_t groups_active_stage(gpugrav_ctx *c, int64_t nt, int cap)
{
  cudaStream_t st = c->stream;
  GG_TRY(c->g_groups.ensure((size_t)(nt + 1) * sizeof(int4)));
  GG_TRY(c->g_ngroups.ensure(16));
  GG_TRY(cudaMemsetAsync(c->g_ngroups.p, 0, sizeof(int), st));
  if(nt == 0)
    return cudaSuccess;
  GG_TRY(c->t_cd.ensure(nt + 16));
  GG_TRY(c->t_pd.ensure(nt + 16));
  GG_TRY(c->g_gseg.ensure(nt * 4));
  GG_TRY(c->g_gflag.ensure(nt * 4));
  GG_TRY(c->g_gid.ensure(nt * 4));
  const int32_t *tpos = c->t_pos_alt.as<int32_t>();
  // every particle active: consecutive targets are neighbours, plain chunks as in the full walk's table
  const bool cells = c->active_slack < 64 && nt < c->n;
  k_active_cd<<<grid_for(nt, 256), 256, 0, st>>>(nt, tpos, c->s_ix.as<uint64_t>(), c->s_iy.as<uint64_t>(), c->s_iz.as<uint64_t>(),
                                                  c->t_cd.as<int8_t>());
  if(cells)
    k_grp_pd_at<<<grid_for(nt, 256), 256, 0, st>>>(nt, tpos, c->s_cd.as<int8_t>(), cap, c->t_pd.as<int8_t>());
  k_grp_cut<<<grid_for(nt, 256), 256, 0, st>>>(nt, c->t_cd.as<int8_t>(), cells ? c->t_pd.as<int8_t>() : nullptr,
                                                c->active_slack, c->g_gflag.as<int32_t>());
  size_t tb = 0;
  GG_TRY(cub::DeviceScan::InclusiveScan(nullptr, tb, c->g_gflag.as<int32_t>(), c->g_gseg.as<int32_t>(), MaxOp32(), (int)nt, st));
  GG_TRY(c->sort_tmp.ensure(tb));
  GG_TRY(cub::DeviceScan::InclusiveScan(c->sort_tmp.p, tb, c->g_gflag.as<int32_t>(), c->g_gseg.as<int32_t>(), MaxOp32(), (int)nt,
                                        st));
  k_grp_start<<<grid_for(nt, 256), 256, 0, st>>>(nt, c->g_gseg.as<int32_t>(), cap, c->g_gflag.as<int32_t>());
  tb = 0;
  GG_TRY(cub::DeviceScan::ExclusiveSum(nullptr, tb, c->g_gflag.as<int32_t>(), c->g_gid.as<int32_t>(), (int)nt, st));
  GG_TRY(c->sort_tmp.ensure(tb));
  GG_TRY(cub::DeviceScan::ExclusiveSum(c->sort_tmp.p, tb, c->g_gflag.as<int32_t>(), c->g_gid.as<int32_t>(), (int)nt, st));
  k_grp_fill<<<grid_for(nt, 256), 256, 0, st>>>(nt, c->g_gflag.as<int32_t>(), c->g_gid.as<int32_t>(), nullptr,
                                                 c->g_groups.as<int4>(), c->g_ngroups.as<int>());
  k_grp_count<<<grid_for((nt + cap - 1) / cap, 256), 256, 0, st>>>(nt, c->g_ngroups.as<int>(), c->g_groups.as<int4>());
  return cudaGetLastError();
}

// the layout above (built once per tree)
cudaError_t layout32_stage(gpugrav_ctx *c)
{
  c->mark(nullptr);
  const int64_t n = c->n, nn = c->num_nodes;
  cudaStream_t st = c->stream;
  GG_TRY(layout32_buffers(c, n, nn));
  const bool mns = c->built_mns;
  if(mns)
    GG_TRY(c->g_mpt.ensure((size_t)(nn + 16) * c->prm.nsofttypes * sizeof(float)));
  auto counts = thrust::make_transform_iterator(c->n_count.as<uint8_t>(), ChildCounts());
  size_t tb   = 0;
  GG_TRY(cub::DeviceScan::ExclusiveSum(nullptr, tb, counts, c->g_scan.as<uint64_t>(), (int)nn, st));
  GG_TRY(c->sort_tmp.ensure(tb));
  GG_TRY(cub::DeviceScan::ExclusiveSum(c->sort_tmp.p, tb, counts, c->g_scan.as<uint64_t>(), (int)nn, st));
  int *err = c->counters.as<int>() + 13;
  GG_TRY(cudaMemsetAsync(err, 0, sizeof(int), st));
  k_g_fill<<<grid_for(8 * nn, 256), 256, 0, st>>>(nn, n, c->multi ? c->ntop : 1, c->n_suns.as<int32_t>(), c->n_count.as<uint8_t>(),
                                                   c->g_scan.as<uint64_t>(), c->n_sm.as<double4>(), c->n_cl.as<double4>(),
                                                   c->n_maxsoft.as<uint8_t>(), c->s_pm.as<double4>(), c->s_st.as<uint8_t>(),
                                                   c->g_sm.as<double4>(), c->g_rel.as<float4>(), c->g_kids.as<int4>(),
                                                   c->g_pm.as<double4>(), c->g_pst.as<uint8_t>(), err,
                                                   mns ? c->n_mpt.as<double>() : nullptr, c->prm.nsofttypes,
                                                   mns ? c->g_mpt.as<float>() : nullptr);
  GG_TRY(cudaGetLastError());
  c->mark("l1 layout32");
  GG_TRY(groups_stage(c));
  c->mark("l2 groups");
  c->layout32_valid = true;
  c->groups_active  = false;
  return cudaSuccess;
}

typedef decltype(&k_walk32<true, true, 1>) Walk32Kernel;

// launch plan of one kernel form: block size and dynamic shared memory
struct Walk32Plan
{
  Walk32Kernel kern;
  int warps;
  size_t smem;
};
template <bool PERIODIC, int TPL, bool EWALD = false, typename R = float, bool SPLIT = false>
Walk32Plan plan_of(bool pot)
{
  return {pot ? k_walk32<PERIODIC, true, TPL, EWALD, R, SPLIT> : k_walk32<PERIODIC, false, TPL, EWALD, R, SPLIT>,
          Shape<R, PERIODIC, TPL>::warps, sizeof(BlockSh<R, PERIODIC, TPL>)};
}

// Everything that must happen before the walk launch and may not be captured in a graph
// (layout, constants upload from host memory, stack allocation, launch shape).
cudaError_t walk32_prepare(gpugrav_ctx *c, const WalkConst &wc)
{
  if(!c->layout32_valid)
    GG_TRY(layout32_stage(c));
  cudaStream_t st = c->stream;
  HostIo *io = c->io();
  if(!io)
    return cudaErrorMemoryAllocation;
  static_assert(sizeof(W32Const) <= sizeof(io->w32), "pinned block");
  W32Const &w = *(W32Const *)io->w32;
  make_w32(wc, &w);
  if(wc.ewald)
    {
      GG_TRY(ewald_ensure(c));
      w.ewd = c->ewd32.as<float4>();
    }
  if(wc.mns)
    w.mpt = c->g_mpt.as<float>();
  GG_TRY(c->scratch.ensure(sizeof(W32Const) + 256));
  GG_TRY(cudaMemcpyAsync(c->scratch.p, &w, sizeof(w), cudaMemcpyHostToDevice, st));
  int dev = 0, sms = 0, per_sm = 0;
  GG_TRY(cudaGetDevice(&dev));
  GG_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const bool periodic = wc.pm != 0;  // TreePM split (Rcut, erfc table)
  const bool pot      = c->want_pot;
  const int tpl       = walk32_tpl(c);
  // the group walk in FP64 arithmetic (precision ablation): TreePM and isolated, one target per lane
  const bool fp64     = c->prm.precision == GPUGRAV_PREC_FP64_GROUP;
  if(fp64 && wc.ewald)
    return cudaErrorNotSupported;
  // two warps per group while all of them run at once (24 warps per SM in either form); an active list may
  // be cut into somewhat more groups, whose second halves then follow in a second round
  const int64_t targets = c->w_ntargets > 0 ? c->w_ntargets : c->n;
  const bool split      = !fp64 && !wc.ewald && tpl == 2 && 2 * ((targets / c->nslices + 63) / 64) <= 24 * sms;
  const Walk32Plan plan =
      fp64 ? (tpl == 2 ? (periodic ? plan_of<true, 2, false, double>(pot) : plan_of<false, 2, false, double>(pot))
                       : (periodic ? plan_of<true, 1, false, double>(pot) : plan_of<false, 1, false, double>(pot)))
      : wc.ewald ? plan_of<false, 1, true>(pot)
      : split    ? (periodic ? plan_of<true, 2, false, float, true>(pot) : plan_of<false, 2, false, float, true>(pot))
      : tpl == 2 ? (periodic ? plan_of<true, 2>(pot) : plan_of<false, 2>(pot))
                 : (periodic ? plan_of<true, 1>(pot) : plan_of<false, 1>(pot));
  GG_TRY(cudaFuncSetAttribute(plan.kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)plan.smem));
  GG_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, plan.kern, 32 * plan.warps, plan.smem));
  if(per_sm < 1)
    per_sm = 1;
  c->w32_kernel  = (void *)plan.kern;
  c->w32_order   = nullptr;
  c->w32_threads = 32 * plan.warps;
  c->w32_smem    = plan.smem;
  c->w32_blocks  = sms * per_sm;
  GG_TRY(c->g_stack.ensure((size_t)c->w32_blocks * plan.warps * kStackCap * sizeof(int)));
  return cudaSuccess;
}

// The walk itself: counter reset + one persistent launch (capturable).  The group table and
// its count live in device memory, so a captured launch serves every tree of the same buffers.
cudaError_t walk32_launch(gpugrav_ctx *c)
{
  cudaStream_t st = c->stream;
  int *work       = c->counters.as<int>() + 20;
  int *err        = c->counters.as<int>() + 14;
  GG_TRY(cudaMemsetAsync(work, 0, sizeof(int), st));
  Walk32Kernel kern = (Walk32Kernel)c->w32_kernel;
  kern<<<c->w32_blocks, c->w32_threads, c->w32_smem, st>>>(
      c->g_sm.as<double4>(), c->g_rel.as<float4>(), c->g_kids.as<int4>(), c->g_pm.as<double4>(), c->g_pst.as<uint8_t>(),
      c->s_pm.as<double4>(), c->s_st.as<uint8_t>(), c->oldacc_s.as<float>(), c->g_ngroups.as<int>(), c->g_groups.as<int4>(),
      c->w32_order, c->w_tlist, c->slice, c->nslices, c->slice_rng_on ? c->slice_rng.as<int64_t>() : nullptr,
      (const W32Const *)c->scratch.p, c->g_stack.as<int>(), work, c->res_s.as<double4>(), c->nint_s.as<int32_t>(),
      (unsigned long long *)(c->counters.as<int>() + 32), err, c->counters.as<int>() + 13);
  return cudaGetLastError();
}

// ---- cost-balanced target slices ----
// Cost of every walk group (FP32) or target (FP64) in key order, from the caller's per-particle cost
// (the previous step's interaction counts, as force_assign_cost_values feeds the reference's domain
// decomposition, src/gravity/forcetree.c:945-1010).
__global__ void k_unit_cost(int64_t nu, int64_t n, const int4 *__restrict__ groups, const uint32_t *__restrict__ perm,
                            const float *__restrict__ cost, double *__restrict__ ucost)
{
  for(int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; u < nu; u += (int64_t)gridDim.x * blockDim.x)
    {
      if(groups)
        {
          const int4 g = groups[u];
          double s     = 0;
          for(int k = 0; k < g.y; k++)
            s += cost[perm[g.x + k]];
          ucost[u] = s;
        }
      else
        ucost[u] = cost[perm[u]];
    }
}

// units [b(s), b(s+1)) with b(s) the first unit whose exclusive cost prefix reaches s/ns of the total
// (equal unit counts when the total is 0); rng = (first group, end group, first target, end target)
__global__ void k_slice_bounds(int64_t nu, int64_t n, const int4 *__restrict__ groups, const double *__restrict__ incl, int slice,
                               int nslices, int64_t *__restrict__ rng)
{
  if(blockIdx.x || threadIdx.x)
    return;
  const double total = nu > 0 ? incl[nu - 1] : 0.0;
  int64_t b[2];
  for(int e = 0; e < 2; e++)
    {
      const int s = slice + e;
      if(s == 0 || nu == 0)
        b[e] = 0;
      else if(s == nslices)
        b[e] = nu;
      else if(!(total > 0))
        b[e] = nu * s / nslices;
      else
        {
          const double want = total * s / nslices;
          int64_t lo = 0, hi = nu;  // first u with exclusive prefix (incl[u-1]) >= want
          while(lo < hi)
            {
              const int64_t mid = (lo + hi) / 2;
              const double ex   = mid > 0 ? incl[mid - 1] : 0.0;
              if(ex >= want)
                hi = mid;
              else
                lo = mid + 1;
            }
          b[e] = lo;
        }
    }
  if(groups)
    {
      rng[0] = b[0];
      rng[1] = b[1];
      rng[2] = b[0] < nu ? groups[b[0]].x : n;
      rng[3] = b[1] < nu ? groups[b[1]].x : n;
    }
  else
    {
      rng[0] = rng[1] = 0;
      rng[2] = b[0];
      rng[3] = b[1];
    }
}

// device-side slice range from the caller's costs (gpugrav_set_target_slice_cost); FP32: in walk
// groups (the group count is read on the host once, here), FP64: in targets
cudaError_t slice_cost_stage(gpugrav_ctx *c, bool fp32)
{
  c->slice_rng_on = false;
  if(c->nslices <= 1 || !c->cost_set)
    return cudaSuccess;
  cudaStream_t st = c->stream;
  int64_t nu      = c->n;
  if(fp32)
    {
      int ng = 0;
      GG_TRY(cudaMemcpyAsync(&ng, c->g_ngroups.p, sizeof(int), cudaMemcpyDeviceToHost, st));
      GG_TRY(cudaStreamSynchronize(st));
      nu = ng;
    }
  GG_TRY(c->slice_rng.ensure(4 * sizeof(int64_t)));
  GG_TRY(c->cost_u.ensure((nu + 1) * sizeof(double)));
  GG_TRY(c->cost_p.ensure((nu + 1) * sizeof(double)));
  const int4 *groups = fp32 ? c->g_groups.as<int4>() : nullptr;
  k_unit_cost<<<grid_for(nu, 256), 256, 0, st>>>(nu, c->n, groups, c->perm.as<uint32_t>(), c->cost_in.as<float>(),
                                                 c->cost_u.as<double>());
  size_t tb = 0;
  GG_TRY(cub::DeviceScan::InclusiveSum(nullptr, tb, c->cost_u.as<double>(), c->cost_p.as<double>(), (int)nu, st));
  GG_TRY(c->sort_tmp.ensure(tb));
  GG_TRY(cub::DeviceScan::InclusiveSum(c->sort_tmp.p, tb, c->cost_u.as<double>(), c->cost_p.as<double>(), (int)nu, st));
  k_slice_bounds<<<1, 32, 0, st>>>(nu, c->n, groups, c->cost_p.as<double>(), c->slice, c->nslices, c->slice_rng.as<int64_t>());
  GG_TRY(cudaGetLastError());
  c->slice_rng_on = true;
  return cudaSuccess;
}

// zero the outputs of the targets outside the current target slice (no-op without slicing)
cudaError_t slice_mask_stage(gpugrav_ctx *c, bool fp32)
{
  if(c->nslices <= 1)
    return cudaSuccess;
  k_slice_mask<<<grid_for(c->n, 256), 256, 0, c->stream>>>(c->n, c->slice, c->nslices, fp32 ? c->g_groups.as<int4>() : nullptr,
                                                           fp32 ? c->g_ngroups.as<int>() : nullptr,
                                                           c->slice_rng_on ? c->slice_rng.as<int64_t>() : nullptr, c->res_s.as<double4>(),
                                                           c->nint_s.as<int32_t>());
  return cudaGetLastError();
}

// the order of the groups of the walk to be launched (k_order_key)
cudaError_t walk32_order(gpugrav_ctx *c, const WalkConst &wc)
{
  // Where some warps take more than one group (a walk that all runs at once needs no order), by the relative
  // criterion (the geometric one, bh, does not look at OldAcc), in a tree deeper by nine levels than an even
  // set's of that size, as zoom boxes and spheres are: displaced grids and random sets, deeper by up to eight,
  // have groups of one cost and lost 0.3 to 5 % by the two kernels' 25 us and the neighbours' cache lines (2^18
  // uniform particles 0.311 -> 0.329 ms, 160^3 of a grid 6.05 -> 6.18).
  const int64_t targets = (c->w_ntargets > 0 ? c->w_ntargets : c->n) / c->nslices;
  if(wc.bh || !deep_tree(c, 9) || targets / (32 * walk32_tpl(c)) <= (int64_t)c->w32_blocks * (c->w32_threads / 32))
    return cudaSuccess;
  GG_TRY(c->g_order.ensure(sizeof(GroupOrder)));
  // the order and the keys take the place of two arrays that only the making of the table uses
  GroupOrder *o      = c->g_order.as<GroupOrder>();
  int *order         = c->g_gflag.as<int>();
  uint8_t *key       = c->g_gpd.as<uint8_t>();
  const int64_t *rng = c->slice_rng_on ? c->slice_rng.as<int64_t>() : nullptr;
  GG_TRY(cudaMemsetAsync(o, 0, sizeof(GroupOrder), c->stream));
  k_order_key<<<148 * 8, kOrderBlock, 0, c->stream>>>(c->g_ngroups.as<int>(), !wc.pm, c->slice, c->nslices, rng,
                                                      c->g_groups.as<int4>(), c->w_tlist, c->oldacc_s.as<float>(), key, o);
  // TreePM: every class in its order; isolated: those of the dear half
  k_order_scatter<<<148, kOrderBlock, 0, c->stream>>>(c->g_ngroups.as<int>(), wc.pm ? 1 : 2, c->slice, c->nslices, rng, key, o,
                                                      order);
  c->w32_order = order;
  return cudaGetLastError();
}
}  // namespace gg

#ifdef GG_WALK32_STATS
// measurement build only: read and reset the walk statistics of the current device
extern "C" int gpugrav_walk_stats(unsigned long long *out)
{
  if(cudaMemcpyFromSymbol(out, gg::g_walk_stats, sizeof(unsigned long long) * gg::kWalkStats) != cudaSuccess)
    return -1;
  unsigned long long z[gg::kWalkStats] = {};
  return cudaMemcpyToSymbol(gg::g_walk_stats, z, sizeof(z)) == cudaSuccess ? 0 : -1;
}
#endif
