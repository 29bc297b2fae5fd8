// domain.cu -- domain stage: periodic wrap, extent, Peano-Hilbert keys, stable
// key sort, gather into the sorted structure-of-arrays.  Compiled with
// -fmad=false: every double operation rounds like the reference's C.
//
//   wrap      do_box_wrapping          src/domain/domain_box.c:259-300
//   extent    domain_findExtent        src/domain/domain_box.c:107-197
//   keys      domain_double_to_int + peano_hilbert_key
//                                      src/domain/domain.c:361-370, src/domain/peano.c:374-390
//   sort      peano_hilbert_order      src/domain/peano.c:74-133 (stable: radix sort)
#include <cub/cub.cuh>

#include "internal.h"
#include "ph.cuh"

namespace gg
{
namespace
{
__constant__ PhTable c_ph;
bool g_ph_ready = false;

__device__ __forceinline__ uint64_t mant52(double d) { return (uint64_t)__double_as_longlong(d) & 0xFFFFFFFFFFFFFull; }

// do_box_wrapping: repeated +/- box until inside [0, box); bounded, reports failure
__device__ __forceinline__ bool wrap_coord(double &x, double box)
{
  int it = 0;
  while(x < 0 && it < 64)
    {
      x = __dadd_rn(x, box);
      it++;
    }
  while(x >= box && it < 128)
    {
      x = __dsub_rn(x, box);
      it++;
    }
  return x >= 0 && x < box;
}

__device__ __forceinline__ uint64_t to_int52(double x, double corner, double inv_len)
{
  return mant52(__dadd_rn(__dmul_rn(__dsub_rn(x, corner), inv_len), 1.0));
}

struct MinOp
{
  __device__ double operator()(double u, double v) const { return fmin(u, v); }
};
struct MaxOp
{
  __device__ double operator()(double u, double v) const { return fmax(u, v); }
};

// ---- extent: per-block min/max, then a single-block finalisation ----
constexpr int kExtBlocks  = 296;
constexpr int kExtThreads = 256;

__global__ void k_extent_partial(const double *__restrict__ pos, int64_t n, int periodic, double box, double *partial,
                                 int *flags)
{
  double mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
  int bad      = 0;
  for(int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    {
      for(int j = 0; j < 3; j++)
        {
          double x = pos[3 * i + j];
          if(!isfinite(x))
            {
              bad = 1;
              continue;
            }
          if(periodic && !wrap_coord(x, box))
            bad = 1;
          mn[j] = fmin(mn[j], x);
          mx[j] = fmax(mx[j], x);
        }
    }
  typedef cub::BlockReduce<double, kExtThreads> BR;
  __shared__ typename BR::TempStorage tmp;
  for(int j = 0; j < 3; j++)
    {
      double a = BR(tmp).Reduce(mn[j], MinOp());
      __syncthreads();
      double b = BR(tmp).Reduce(mx[j], MaxOp());
      __syncthreads();
      if(threadIdx.x == 0)
        {
          partial[blockIdx.x * 6 + j]     = a;
          partial[blockIdx.x * 6 + 3 + j] = b;
        }
    }
  if(bad)
    atomicOr(flags, 2);
}

// one warp per bound (6 warps), the rest by one thread
__global__ void k_extent_final(const double *partial, int nblocks, BuildConst *bc)
{
  __shared__ double ext[6];
  const int k = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double v = k < 3 ? INFINITY : -INFINITY;
  for(int b = lane; b < nblocks; b += 32)
    v = k < 3 ? fmin(v, partial[b * 6 + k]) : fmax(v, partial[b * 6 + k]);
  for(int o = 16; o > 0; o >>= 1)
    {
      const double u = __shfl_xor_sync(0xffffffffu, v, o);
      v              = k < 3 ? fmin(v, u) : fmax(v, u);
    }
  if(lane == 0)
    ext[k] = v;
  __syncthreads();
  if(threadIdx.x != 0)
    return;
  double xmin[3], xmax[3];
  for(int j = 0; j < 3; j++)
    {
      // preset to the simulation box (src/domain/domain_box.c:113-118)
      xmin[j] = 0;
      xmax[j] = bc->box;
      if(xmin[j] > ext[j])
        xmin[j] = ext[j];
      if(xmax[j] < ext[3 + j])
        xmax[j] = ext[3 + j];
    }
  double len = 0;
  for(int j = 0; j < 3; j++)
    if(__dsub_rn(xmax[j], xmin[j]) > len)
      len = __dsub_rn(xmax[j], xmin[j]);
  len = __dmul_rn(len, bc->periodic ? 1.00001 : 1.2);
  for(int j = 0; j < 3; j++)
    {
      bc->dom.center[j] = __dmul_rn(0.5, __dadd_rn(xmin[j], xmax[j]));
      bc->dom.corner[j] = __dsub_rn(__dmul_rn(0.5, __dadd_rn(xmin[j], xmax[j])), __dmul_rn(0.5, len));
    }
  bc->dom.len         = len;
  bc->dom.inverse_len = __ddiv_rn(1.0, len);
  bc->dom.big_fac     = __ddiv_rn(len, 4503599627370496.0); /* 2^52 */
}

// ---- keys ----
__global__ void k_keys(const double *__restrict__ pos, int64_t n, const BuildConst *__restrict__ bc, u128 *__restrict__ key,
                       uint64_t *__restrict__ lead, uint32_t *__restrict__ idx, int *flags)
{
  __shared__ uint16_t tab[48 * 8];
  for(int t = threadIdx.x; t < 48 * 8; t += blockDim.x)
    tab[t] = c_ph.e[t];
  __syncthreads();
  const int periodic = bc->periodic;
  const double box   = bc->box;
  const double inv   = bc->dom.inverse_len;
  const double len   = bc->dom.len;
  for(int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    {
      uint64_t ip[3];
      int bad = 0;
      for(int j = 0; j < 3; j++)
        {
          double x = pos[3 * i + j];
          if(periodic)
            wrap_coord(x, box);
          double c = bc->dom.corner[j];
          // particle must lie in [DomainCorner, DomainCorner + DomainLen) (src/gravity/forcetree.c:411-415)
          if(!(x >= c && x < __dadd_rn(c, len)))
            bad = 1;
          ip[j] = to_int52(x, c, inv);
        }
      if(bad)
        atomicOr(flags, 1);
      const u128 k = ph_key_dev(tab, ip[0] >> (52 - kBits), ip[1] >> (52 - kBits), ip[2] >> (52 - kBits), kBits);
      key[i]       = k;
      lead[i]      = (uint64_t)(k >> (3 * kBits - 64));
      idx[i]       = (uint32_t)i;
    }
}

// ---- the key order from the leading 64 key bits ----
// Sorting 126-bit keys takes 16 radix passes over 20 bytes a particle; their leading 64 bits (21 levels
// of the curve, a cell of 5e-7 of the domain) take 8 over 12 bytes and leave few particles in runs of
// equal leading bits, which are ordered here by their full keys.  A run longer than kMaxRun (coincident
// or nearly coincident points, the centre of a deep zoom) sets flag 8: the caller then sorts the full keys, and
// goes on with these for the next sets of the context until k_long_runs finds none (2^22 particles with such a
// clump: 2.0 ms for both sorts and gathers, 1.2 for the full sort alone; 2^24 7.5 and 4.2).
constexpr int kMaxRun = 32;
__global__ void k_sort_ties(int64_t n, const uint64_t *__restrict__ lead, const u128 *__restrict__ key, uint32_t *__restrict__ perm,
                            int *__restrict__ flags)
{
  for(int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i + 1 < n; i += (int64_t)gridDim.x * blockDim.x)
    {
      const uint64_t p = lead[i];
      if(lead[i + 1] != p || (i > 0 && lead[i - 1] == p))
        continue;  // not the first of a run
      int64_t e = i + 2;
      while(e < n && e - i <= kMaxRun && lead[e] == p)
        e++;
      if(e - i > kMaxRun)
        {
          atomicOr(flags, 8);
          continue;
        }
      // insertion by the full key; the radix sort left equal keys in the caller's order
      for(int64_t a = i + 1; a < e; a++)
        {
          const uint32_t o = perm[a];
          const u128 k     = key[o];
          int64_t b        = a;
          for(; b > i && key[perm[b - 1]] > k; b--)
            perm[b] = perm[b - 1];
          perm[b] = o;
        }
    }
}

// flag 8: the sorted keys hold a run of more than kMaxRun equal leading bits (k >> shift)
__global__ void k_long_runs(int64_t n, const u128 *__restrict__ key, int shift, int *__restrict__ flags)
{
  bool found = false;
  for(int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i + kMaxRun < n; i += (int64_t)gridDim.x * blockDim.x)
    found |= (uint64_t)(key[i] >> shift) == (uint64_t)(key[i + kMaxRun] >> shift);
  if(found)
    atomicOr(flags, 8);
}

// ---- gather into sorted SoA ----
__global__ void k_gather(const double *__restrict__ pos, const double *__restrict__ mass, const uint8_t *__restrict__ st,
                         const uint32_t *__restrict__ perm, int64_t n, const BuildConst *__restrict__ bc,
                         uint32_t *__restrict__ iperm, double4 *__restrict__ s_pm, uint64_t *__restrict__ s_ix, uint64_t *__restrict__ s_iy,
                         uint64_t *__restrict__ s_iz, uint8_t *__restrict__ s_st, int *flags)
{
  const int nsoft    = bc->nsoft;
  const int periodic = bc->periodic;
  const double box   = bc->box;
  const double inv   = bc->dom.inverse_len;
  for(int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    {
      uint32_t o = perm[i];
      iperm[o]   = (uint32_t)i;
      double x = pos[3 * (int64_t)o + 0], y = pos[3 * (int64_t)o + 1], z = pos[3 * (int64_t)o + 2];
      if(periodic)
        {
          wrap_coord(x, box);
          wrap_coord(y, box);
          wrap_coord(z, box);
        }
      s_pm[i] = make_double4(x, y, z, mass[o]);
      s_ix[i] = to_int52(x, bc->dom.corner[0], inv);
      s_iy[i] = to_int52(y, bc->dom.corner[1], inv);
      s_iz[i] = to_int52(z, bc->dom.corner[2], inv);
      uint8_t t = st[o];
      s_st[i]   = t;
      // a softening type must index ForceSoftening[0 .. nsofttypes-1]
      if(t >= nsoft)
        atomicOr(flags, 4);
    }
}

int grid_for(int64_t n, int threads)
{
  int64_t b = (n + threads - 1) / threads;
  if(b > 148 * 16)
    b = 148 * 16;
  return (int)(b < 1 ? 1 : b);
}
}  // namespace

cudaError_t domain_stage(gpugrav_ctx *c, bool compute_extent)
{
  cudaError_t e;
  if(!g_ph_ready)
    {
      PhTable t = ph_make_table();
      if((e = cudaMemcpyToSymbolAsync(c_ph, &t, sizeof(t), 0, cudaMemcpyHostToDevice, c->stream)) != cudaSuccess ||
         (e = cudaStreamSynchronize(c->stream)) != cudaSuccess)  // other contexts' streams read it from now on
        return e;
      g_ph_ready = true;
    }
  const int64_t n = c->n;
  if((e = c->scratch.ensure(kExtBlocks * 6 * sizeof(double) + 64)) != cudaSuccess)
    return e;
  if((e = c->counters.ensure(kCounters * sizeof(int))) != cudaSuccess)
    return e;
  if((e = c->key.ensure(n * sizeof(u128))) != cudaSuccess || (e = c->key_alt.ensure(n * sizeof(u128))) != cudaSuccess ||
     (e = c->idx.ensure(n * sizeof(uint32_t))) != cudaSuccess || (e = c->perm.ensure(n * sizeof(uint32_t))) != cudaSuccess)
    return e;
  int *flags = c->counters.as<int>();
  cudaMemsetAsync(flags, 0, sizeof(int), c->stream);
  BuildConst *bc = c->bconst.as<BuildConst>();
  if(compute_extent)
    {
      k_extent_partial<<<kExtBlocks, kExtThreads, 0, c->stream>>>(c->pos_in.as<double>(), n, c->prm.periodic, c->prm.box_size,
                                                                  c->scratch.as<double>(), flags);
      k_extent_final<<<1, 192, 0, c->stream>>>(c->scratch.as<double>(), kExtBlocks, bc);
    }
  k_keys<<<grid_for(n, 256), 256, 0, c->stream>>>(c->pos_in.as<double>(), n, bc, c->key.as<u128>(), c->key_alt.as<uint64_t>(),
                                                 c->idx.as<uint32_t>(), flags);
  return cudaGetLastError();
}

// Order of the n keys in c->key (perm) from their leading bits, which the caller put into the first half of
// c->key_alt; flag 8 of *flags: sort_full_stage is needed.
cudaError_t sort_lead_stage(gpugrav_ctx *c, int64_t n, int *flags)
{
  uint64_t *lead = c->key_alt.as<uint64_t>();
  size_t tb      = 0;
  GG_TRY(cub::DeviceRadixSort::SortPairs(nullptr, tb, lead, lead + n, c->idx.as<uint32_t>(), c->perm.as<uint32_t>(), (int)n, 0, 64,
                                         c->stream));
  GG_TRY(c->sort_tmp.ensure(tb));
  GG_TRY(cub::DeviceRadixSort::SortPairs(c->sort_tmp.p, tb, lead, lead + n, c->idx.as<uint32_t>(), c->perm.as<uint32_t>(), (int)n, 0, 64,
                                         c->stream));
  k_sort_ties<<<grid_for(n, 256), 256, 0, c->stream>>>(n, lead + n, c->key.as<u128>(), c->perm.as<uint32_t>(), flags);
  return cudaGetLastError();
}

// stable LSD radix sort over key bits [0, bits): equal keys keep the caller order, as the merge sort of
// peano_hilbert_order does
cudaError_t sort_full_stage(gpugrav_ctx *c, int64_t n, int bits)
{
  size_t tb = 0;
  GG_TRY(cub::DeviceRadixSort::SortPairs(nullptr, tb, c->key.as<u128>(), c->key_alt.as<u128>(), c->idx.as<uint32_t>(),
                                         c->perm.as<uint32_t>(), (int)n, 0, bits, c->stream));
  GG_TRY(c->sort_tmp.ensure(tb));
  return cub::DeviceRadixSort::SortPairs(c->sort_tmp.p, tb, c->key.as<u128>(), c->key_alt.as<u128>(), c->idx.as<uint32_t>(),
                                         c->perm.as<uint32_t>(), (int)n, 0, bits, c->stream);
}

// after sort_full_stage: whether sort_lead_stage, on leading bits k >> shift, would have needed it (flag 8 of *flags)
cudaError_t sort_runs_stage(gpugrav_ctx *c, int64_t n, int shift, int *flags)
{
  k_long_runs<<<grid_for(n, 256), 256, 0, c->stream>>>(n, c->key_alt.as<u128>(), shift, flags);
  return cudaGetLastError();
}

cudaError_t gather_stage(gpugrav_ctx *c)
{
  const int64_t n = c->n;
  cudaError_t e;
  if((e = c->s_pm.ensure(n * sizeof(double4))) != cudaSuccess || (e = c->s_ix.ensure(n * 8)) != cudaSuccess ||
     (e = c->s_iy.ensure(n * 8)) != cudaSuccess || (e = c->s_iz.ensure(n * 8)) != cudaSuccess ||
     (e = c->s_st.ensure(n + 16)) != cudaSuccess || (e = c->iperm.ensure(n * sizeof(uint32_t))) != cudaSuccess)
    return e;
  k_gather<<<grid_for(n, 256), 256, 0, c->stream>>>(c->pos_in.as<double>(), c->mass_in.as<double>(), c->st_in.as<uint8_t>(),
                                                   c->perm.as<uint32_t>(), n, c->bconst.as<BuildConst>(),
                                                   c->iperm.as<uint32_t>(), c->s_pm.as<double4>(),
                                                   c->s_ix.as<uint64_t>(), c->s_iy.as<uint64_t>(), c->s_iz.as<uint64_t>(),
                                                   c->s_st.as<uint8_t>(), c->counters.as<int>());
  return cudaGetLastError();
}
}  // namespace gg
