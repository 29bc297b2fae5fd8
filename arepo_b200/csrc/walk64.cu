// walk64.cu -- FP64 parity walk.  Compiled with -fmad=false.
//
// force_treeevaluate (src/gravity/forcetree_walk.c:115-514) for every target,
// with the reference's arithmetic operation for operation.  The tree is laid
// out in the reference's traversal order (depth first, slots 0..7), so that
// "nextnode" of an entry is the next entry and "sibling" is the entry after its
// subtree (w_link.x).  A warp takes up to 32 consecutive targets in key order; each
// lane keeps its own position in its own traversal, and the warp always serves
// the smallest position among its lanes: the entry is loaded once for the warp
// and tested by exactly the lanes that are at it.  Every lane therefore sees
// the same interaction sequence, in the same order, as the reference walk for
// its target -- the per-target results are bit-identical to the reference.
#include <type_traits>

#include "internal.h"

namespace gg
{
namespace
{
// cubic-spline softening coefficients, src/main/allvars.h:557-573
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

// GRAVITY_NEAREST_X, src/main/allvars.h:602-608: x - box or x + box beyond half a box; a select, no branches
template <bool PER>
__device__ __forceinline__ double nearest(double x, const WalkConst &w)
{
  return PER ? x - (fabs(x) > w.half_box ? copysign(w.box, x) : 0.0) : x;
}

constexpr int kWarps  = 4;
// Blocks per SM: 6 leave 80 registers a thread, 8 hide more of the loads' latency, 10 hold more warps at once
// (walk64_stage chooses).  Walk (ms) with 6 / 8 / 10: even 48^3 0.99 / 1.11 / 1.37, 53^3 1.75 / 1.34 / 1.70, 57^3
// 2.05 / 2.13 / 1.92, 61^3 2.39 / 2.48 / 2.66, 80^3 5.77 / 5.28 / 5.59, 128^3 19.5 / 17.9 / 18.5; zoom box 150000
// 17.5 / 19.5 / 21.3, 240022 22.4 / 24.9 / 27.2, 2^19 29.3 / 32.7 / 34.9, 2^21 71.5 / 71.4 / 76.3, 2^24 (tolerance 2e-5)
// - / 3868 / -; Plummer 150000 5.7 / 6.1 / 6.2, 2^20 17.5 / 17.2 / 17.3.
constexpr int kBlocks = 6, kBlocksMore = 8, kBlocksMost = 10;
constexpr int kLarge  = 8;  // units per warp from which the walk of a clustered set takes kBlocksMore

// The walk's tests of an internal node, src/gravity/forcetree_walk.c:196-330: opened (go on with the next
// entry), or not -- then skipped with its subtree, and used unless it lies beyond Rcut (out).
template <bool MNS, bool PER>
__device__ __forceinline__ void test_node(double mass, const double4 cl, int type_fl, double r2, double pos_x, double pos_y,
                                          double pos_z, double aold, double h_i, const WalkConst &w, bool &open, bool &out)
{
  // No short-circuit evaluation: the comparisons do not depend on one another and run side by side; a branch
  // for each, taken by some lanes, made the test most of the walk of sets that fill the chip about once
  // (32^3 targets 1.28 ms, 0.87 without; a zoom box of 240022 32 ms, 22 without).
  const double len = cl.w, len2 = len * len;
  const bool beyond = PER && (w.pm != 0) & (r2 > w.rcut2);
  if(w.bh)
    open = len2 > r2 * w.theta * w.theta;
  else
    // ACTIVATE_MINIMUM_OPENING_ANGLE adds a minimum angle to the mass test (forcetree_walk.c:266-271)
    open = (len2 > r2 * (1.2 * 1.2)) | ((mass * len2 > r2 * r2 * aold) & ((w.minangle == 0) | (len2 > r2 * (0.4 * 0.4))));
  if(!MNS)
    {
      const double h_j = w.soft[type_fl & 0xff];
      open             = open | ((h_j > h_i) & (r2 < h_j * h_j));
    }
  const double cx = fabs(nearest<PER>(cl.x - pos_x, w)), cy = fabs(nearest<PER>(cl.y - pos_y, w)),
               cz = fabs(nearest<PER>(cl.z - pos_z, w));
  if(PER)
    {
      const double eff_dist = w.rcut + 0.5 * len;
      out                   = beyond & ((cx > eff_dist) | (cy > eff_dist) | (cz > eff_dist));
    }
  const double in = 0.60 * len;
  open            = (open | (!w.bh & (cx < in) & (cy < in) & (cz < in))) & !out;
}

// One contribution of a walk entry (at dx, dy, dz from the target; type_fl: softening type and node flag) to a
// target, src/gravity/forcetree_walk.c:363-488, added with add(x, y, z, potential); type >= 0: the node's
// mass of that softening type (MULTIPLE_NODE_SOFTENING, forcetree_walk.c:382-401).  False: beyond the table.
template <bool EWALD, bool MNS, class Add>
__device__ __forceinline__ bool interact(uint32_t e, int type, double mass, int type_fl, double dx, double dy, double dz, double r2,
                                         double h_i, const WalkConst &w, Add add)
{
  double r            = sqrt(r2);
  double factor_force = 0, factor_pot = 0;
  if(w.pm)
    {
      double tabentry = w.asmthfac * r;
      int tabindex    = (int)tabentry;
      if(!(tabindex < kNtab))
        return false;
      // INT_MIN where r is NaN (a non-finite mass in the node): entry 0, and the sum will be NaN
      static_assert((kNtab & (kNtab + 1)) == 0, "all bits set");
      tabindex &= kNtab;
      double tabweight = tabentry - tabindex;
      factor_force     = (1.0 - tabweight) * w.tab_force[tabindex] + tabweight * w.tab_force[tabindex + 1];
      factor_pot       = (1.0 - tabweight) * w.tab_pot[tabindex] + tabweight * w.tab_pot[tabindex + 1];
    }
  double h_j = w.soft[type_fl & 0xff];
  if(MNS && type >= 0)
    {
      mass = w.w_mpt[(int64_t)e * w.nsoft + type];
      h_j  = w.soft[type];
      if(!mass)
        return true;
    }
  const double hmax = (h_j > h_i) ? h_j : h_i;
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
  fac *= mass;
  add(dx * fac, dy * fac, dz * fac, mass * wp);
  if(EWALD)
    {
      // all further periodic images, src/gravity/forcetree_walk.c:469-477
      double fcorr[3], pcorr;
      ewald_corr(dx, dy, dz, w, fcorr, pcorr);
      add(mass * fcorr[0], mass * fcorr[1], mass * fcorr[2], mass * pcorr);
    }
  return true;
}

// A warp takes up to 32 targets at a time, its first by number, the next from a counter: the walks of a dense
// core and of the background differ by two orders of magnitude, and blocks of four fixed warps waited for
// their longest.  The chain of one entry after the other bounds it: load, FP64 test, next entry, some 900
// cycles.  Interactions are evaluated where they are found; waiting in queues and evaluated 32 at a time, they
// were 1.2 times faster in a zoom box but 1.5 times slower in an even set of 2^18, whose warps the queues'
// shared memory kept off the SM.
//
// EWALD (pure periodic tree: two contributions per entry), MNS (MULTIPLE_NODE_SOFTENING) and PER (nearest images)
// are compiled in only where used: an isolated sphere of 2^20 particles took 23.6 ms with the selects of PER and
// the separations formed in the test and again in the interaction, 17.2 without.
template <bool EWALD, bool MNS, bool PER, int BLOCKS>
__global__ void __launch_bounds__(32 * kWarps, BLOCKS) k_walk64(const double4 *__restrict__ w_sm, const double4 *__restrict__ w_cl,
                                                        const int2 *__restrict__ w_link, uint32_t n_entries,
                                                        const double4 *__restrict__ tpm, const uint8_t *__restrict__ tst,
                                                        const float *__restrict__ oldacc, int64_t t_begin, int64_t t_end,
                                                        const int32_t *__restrict__ tlist, const WalkConst *__restrict__ wcp,
                                                        int tpu, int *__restrict__ work, double4 *__restrict__ res_out,
                                                        int32_t *__restrict__ nint_out, unsigned long long *__restrict__ total)
{
  __shared__ WalkConst w;
  for(int t = threadIdx.x; t < (int)(sizeof(WalkConst) / 4); t += blockDim.x)
    ((int *)&w)[t] = ((const int *)wcp)[t];
  __syncthreads();

  const int lane           = threadIdx.x & 31;
  const int64_t units      = (t_end - t_begin + tpu - 1) / tpu;
  unsigned long long count = 0;
  for(int64_t u = (int64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x; u < units;)
    {
      // position in the walk's target range; the target itself (sorted particle index) is the same
      // position, or its entry in the list of active targets
      const int64_t slot = t_begin + u * tpu + lane;
      const bool valid   = lane < tpu && slot < t_end;
      const int64_t tgt  = valid && tlist ? (int64_t)tlist[slot] : slot;

      double pos_x = 0, pos_y = 0, pos_z = 0, aold = 0, h_i = 0;
      if(valid)
        {
          double4 p = tpm[tgt];
          pos_x     = p.x;
          pos_y     = p.y;
          pos_z     = p.z;
          aold      = w.erracc * (double)oldacc[tgt];
          h_i       = w.soft[tst[tgt]];
        }
      double acc_x = 0, acc_y = 0, acc_z = 0, pot = 0;
      int ninteractions = 0;
      auto add_own = [&](double tx, double ty, double tz, double tp) {
        acc_x += tx;
        acc_y += ty;
        acc_z += tz;
        pot += tp;
      };
      uint32_t next = valid ? 0u : n_entries;  // entry 0 is the root (Tree_MaxPart)

      while(true)
        {
          const uint32_t i = __reduce_min_sync(0xffffffffu, next);
          if(i >= n_entries)
            break;
          const int2 link  = w_link[i];
          const double4 sm = w_sm[i], cl = w_cl[i];
          const bool node  = (link.y & kNodeFlag) != 0;
          const double dx = nearest<PER>(sm.x - pos_x, w), dy = nearest<PER>(sm.y - pos_y, w), dz = nearest<PER>(sm.z - pos_z, w);
          const double r2 = dx * dx + dy * dy + dz * dz;
          bool open = false, out = false;
          if(node)
            test_node<MNS, PER>(sm.w, cl, link.y, r2, pos_x, pos_y, pos_z, aold, h_i, w, open, out);
          const bool here = next == i, take = here && !open && !out && sm.w != 0;
          if(here)
            next = node && !open ? (uint32_t)link.x : i + 1;
          // MULTIPLE_NODE_SOFTENING: a node is used per softening type, src/gravity/forcetree_walk.c:296-308
          const bool split = MNS && node && w.soft[link.y & 0xff] > h_i;
          if(take)
            {
              bool did = false;
              if(MNS && split)
                for(int t = 0; t < w.nsoft; t++)
                  did = interact<EWALD, MNS>(i, t, sm.w, link.y, dx, dy, dz, r2, h_i, w, add_own);
              else
                did = interact<EWALD, false>(i, -1, sm.w, link.y, dx, dy, dz, r2, h_i, w, add_own);
              ninteractions += did ? 1 : 0;
            }
        }

      if(valid)
        {
          res_out[tgt]  = make_double4(acc_x, acc_y, acc_z, pot);
          nint_out[tgt] = ninteractions;
          count += (unsigned long long)ninteractions;
        }
      int taken = 0;
      if(lane == 0)
        taken = atomicAdd(work, 1);
      u = (int64_t)kWarps * gridDim.x + __shfl_sync(0xffffffffu, taken, 0);
    }
  // interaction total for the timing report
  for(int o = 16; o > 0; o >>= 1)
    count += __shfl_xor_sync(0xffffffffu, count, o);
  if(lane == 0 && count)
    atomicAdd(total, count);
}
}  // namespace

cudaError_t walk64_stage(gpugrav_ctx *c, const WalkConst &wc)
{
  // targets: every particle, or the active list (gpugrav_walk_targets); the slice's range from the
  // device when it is balanced by cost
  const int64_t n = c->w_tlist ? c->w_ntargets : c->n;
  int64_t t_begin = n * c->slice / c->nslices, t_end = n * (c->slice + 1) / c->nslices;
  if(c->slice_rng_on && !c->w_tlist)
    {
      int64_t rng[4];
      GG_TRY(cudaMemcpyAsync(rng, c->slice_rng.p, sizeof(rng), cudaMemcpyDeviceToHost, c->stream));
      GG_TRY(cudaStreamSynchronize(c->stream));
      t_begin = rng[2];
      t_end   = rng[3];
    }
  int sms = 0, per_sm = 0;
  GG_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device));
  auto plan = [&](auto blocks) {
    constexpr int B = decltype(blocks)::value;
    return wc.ewald      ? (wc.mns ? k_walk64<true, true, true, B> : k_walk64<true, false, true, B>)
           : wc.periodic ? (wc.mns ? k_walk64<false, true, true, B> : k_walk64<false, false, true, B>)
                         : (wc.mns ? k_walk64<false, true, false, B> : k_walk64<false, false, false, B>);
  };
  // The warps of an even set all take as long: the fewest blocks that need the fewest rounds of warps, and
  // kBlocksMore beyond two rounds.  A clustered set's differ (its tree is deeper; displaced grids and random sets
  // of 10^5 to 10^6 are deeper than even by up to 5 levels, zoom boxes and spheres by 8 and more), and the long
  // ones want the registers.
  const int64_t warps = (t_end - t_begin + 31) / 32, per_block = (int64_t)kWarps * sms;
  auto rounds         = [&](int b) { return (warps + b * per_block - 1) / (b * per_block); };
  int blocks          = kBlocks;
  if(deep_tree(c, 6))
    blocks = warps >= kLarge * kBlocks * per_block ? kBlocksMore : kBlocks;
  else if(rounds(kBlocks) > 2 || rounds(kBlocksMore) < rounds(kBlocks))
    blocks = kBlocksMore;
  else if(rounds(kBlocksMost) < rounds(kBlocks))
    blocks = kBlocksMost;
  auto kern = blocks == kBlocks       ? plan(std::integral_constant<int, kBlocks>())
              : blocks == kBlocksMore ? plan(std::integral_constant<int, kBlocksMore>())
                                      : plan(std::integral_constant<int, kBlocksMost>());
  GG_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * kWarps, 0));
  // Targets per warp: as few as keep all warps running at once, 4 to 32.  The walk of a set that does not fill
  // the chip takes as long as its longest warp, and that steps on the union of its targets' entries (ms with
  // 4 / 8 / 16 / 32: 4096 targets 0.18 / 0.20 / 0.25 / 0.31, 15625 0.62 / 0.48 / 0.54 / 0.60, 32768
  // 1.56 / 1.25 / 0.84 / 0.95); once there are more warps than fit, shared steps count (110592 targets: 3.75
  // with 16, 2.35 with 32).
  const int64_t resident = (int64_t)sms * (per_sm > 0 ? per_sm : 1) * kWarps, need = (t_end - t_begin + resident - 1) / resident;
  const int tpu          = need < 4 ? 4 : (need > 32 ? 32 : (int)need);
  int *work = c->counters.as<int>() + 20;
  GG_TRY(cudaMemsetAsync(work, 0, sizeof(int), c->stream));
  kern<<<sms * (per_sm > 0 ? per_sm : 1), 32 * kWarps, 0, c->stream>>>(
      c->w_sm.as<double4>(), c->w_cl.as<double4>(), c->w_link.as<int2>(), (uint32_t)c->n_entries, c->s_pm.as<double4>(),
      c->s_st.as<uint8_t>(), c->oldacc_s.as<float>(), t_begin, t_end, c->w_tlist, c->wconst.as<WalkConst>(), tpu, work,
      c->res_s.as<double4>(), c->nint_s.as<int32_t>(), (unsigned long long *)(c->counters.as<int>() + 32));
  return cudaGetLastError();
}
}  // namespace gg
