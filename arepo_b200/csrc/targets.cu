// targets.cu -- walks of an active subset of the particles.
//
// gravity_tree(timebin) walks only the particles of the current gravity time bin: it builds
// TargetList from TimeBinsGravity.ActiveParticleList (src/gravity/gravtree.c:494-520) while the
// tree holds every particle.  Here the caller's list of active particles (caller indices, any order)
// becomes a list of sorted particle positions in Peano-Hilbert order, so that the FP64 walk's warps
// and the FP32 walk's groups take spatially close active targets together; results go back in the
// order of the caller's list.
#include <cub/cub.cuh>

#include "internal.h"

namespace gg
{
namespace
{
int grid_for(int64_t n, int threads)
{
  int64_t b = (n + threads - 1) / threads;
  if(b > 148 * 16)
    b = 148 * 16;
  return (int)(b < 1 ? 1 : b);
}

// sorted position of every listed target (flag bit 1: index out of range)
__global__ void k_target_pos(int64_t nt, const int32_t *__restrict__ targets, int64_t n, const uint32_t *__restrict__ iperm,
                             uint32_t *__restrict__ pos, uint32_t *__restrict__ idx, int *__restrict__ flag)
{
  for(int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < nt; j += (int64_t)gridDim.x * blockDim.x)
    {
      const int32_t t = targets[j];
      if(t < 0 || t >= n)
        {
          atomicOr(flag, 1);
          pos[j] = 0;
        }
      else
        pos[j] = iperm[t];
      idx[j] = (uint32_t)j;
    }
}

// flag bit 2: a particle listed twice
__global__ void k_target_dups(int64_t nt, const uint32_t *__restrict__ pos, int *__restrict__ flag)
{
  for(int64_t j = 1 + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < nt; j += (int64_t)gridDim.x * blockDim.x)
    if(pos[j] == pos[j - 1])
      atomicOr(flag, 2);
}

// results of the active list back to the caller's list order; entries outside this target slice
// (another rank's) are written as zero.  The slice is a range of walk groups where the walk has them
// (groups not null; their number is known on the device only), else of targets.
__global__ void k_scatter_targets(int64_t nt, const uint32_t *__restrict__ tpos, const uint32_t *__restrict__ tidx, int slice,
                                  int nslices, const int4 *__restrict__ groups, const int *__restrict__ ngroups,
                                  const double4 *__restrict__ res_s, const int32_t *__restrict__ nint_s,
                                  double *__restrict__ acc, double *__restrict__ pot, int32_t *__restrict__ nint)
{
  int64_t a = nt * slice / nslices, b = nt * (slice + 1) / nslices;
  if(groups)
    {
      const int64_t ng = *ngroups, ga = ng * slice / nslices, gb = ng * (slice + 1) / nslices;
      a = ga < ng ? groups[ga].x : nt;
      b = gb < ng ? groups[gb].x : nt;
    }
  for(int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nt; i += (int64_t)gridDim.x * blockDim.x)
    {
      const int64_t o = tidx[i], s = tpos[i];
      const bool in   = i >= a && i < b;
      const double4 r = in ? res_s[s] : make_double4(0, 0, 0, 0);
      acc[3 * o + 0]  = r.x;
      acc[3 * o + 1]  = r.y;
      acc[3 * o + 2]  = r.z;
      if(pot)
        pot[o] = r.w;
      if(nint)
        nint[o] = in ? nint_s[s] : 0;
    }
}
}  // namespace

// Sorted positions of the caller's active list in key order (t_pos_alt) and their places in the
// list (t_idx_alt); flags: bit 1 an index outside [0, n), bit 2 a particle listed twice.
cudaError_t targets_stage(gpugrav_ctx *c, int64_t nt, const int32_t *d_targets, int *flags)
{
  cudaStream_t st = c->stream;
  const int64_t n = c->n;
  GG_TRY(c->t_pos.ensure(nt * sizeof(uint32_t) + 16));
  GG_TRY(c->t_pos_alt.ensure(nt * sizeof(uint32_t) + 16));
  GG_TRY(c->t_idx.ensure(nt * sizeof(uint32_t) + 16));
  GG_TRY(c->t_idx_alt.ensure(nt * sizeof(uint32_t) + 16));
  int *flag = c->counters.as<int>() + 16;
  GG_TRY(cudaMemsetAsync(flag, 0, sizeof(int), st));
  k_target_pos<<<grid_for(nt, 256), 256, 0, st>>>(nt, d_targets, n, c->iperm.as<uint32_t>(), c->t_pos.as<uint32_t>(),
                                                  c->t_idx.as<uint32_t>(), flag);
  int bits = 1;
  while(bits < 32 && ((int64_t)1 << bits) < n)
    bits++;
  size_t tb = 0;
  GG_TRY(cub::DeviceRadixSort::SortPairs(nullptr, tb, c->t_pos.as<uint32_t>(), c->t_pos_alt.as<uint32_t>(),
                                         c->t_idx.as<uint32_t>(), c->t_idx_alt.as<uint32_t>(), (int)nt, 0, bits, st));
  GG_TRY(c->sort_tmp.ensure(tb));
  GG_TRY(cub::DeviceRadixSort::SortPairs(c->sort_tmp.p, tb, c->t_pos.as<uint32_t>(), c->t_pos_alt.as<uint32_t>(),
                                         c->t_idx.as<uint32_t>(), c->t_idx_alt.as<uint32_t>(), (int)nt, 0, bits, st));
  k_target_dups<<<grid_for(nt, 256), 256, 0, st>>>(nt, c->t_pos_alt.as<uint32_t>(), flag);
  GG_TRY(cudaGetLastError());
  GG_TRY(cudaMemcpyAsync(flags, flag, sizeof(int), cudaMemcpyDeviceToHost, st));
  GG_TRY(cudaStreamSynchronize(st));
  return cudaSuccess;
}

cudaError_t targets_scatter(gpugrav_ctx *c, int64_t nt, bool groups, double *acc, double *pot, int32_t *nint)
{
  k_scatter_targets<<<grid_for(nt, 256), 256, 0, c->stream>>>(nt, c->t_pos_alt.as<uint32_t>(), c->t_idx_alt.as<uint32_t>(), c->slice,
                                                             c->nslices, groups ? c->g_groups.as<int4>() : nullptr,
                                                             groups ? c->g_ngroups.as<int>() : nullptr, c->res_s.as<double4>(),
                                                             c->nint_s.as<int32_t>(), acc, pot, nint);
  return cudaGetLastError();
}
}  // namespace gg
