// tree.cu -- top-level tree, octree build, multipole moments, threading and the
// depth-first walk layout.  Compiled with -fmad=false (bit-exact doubles).
//
// The reference inserts particles one at a time in Peano-Hilbert order
// (force_treebuild_insert_single_point, src/gravity/forcetree.c:835-938).  The
// resulting octree is canonical: below the top-level skeleton, a node exists for
// every cell that holds at least two particles (down to MAX_TREE_LEVEL), and the
// node for a cell is created while inserting the second particle of that cell.
// Because the particles of any cell are contiguous in key order, that particle is
// (first particle of the cell) + 1, and the reference's node numbering is the
// order of (inserting particle, depth).  Here every adjacent pair (j-1, j) of the
// sorted particles contributes the nodes for the cells holding both j-1 and j that
// are deeper than the cells holding j-2 and j-1: counted, prefix-summed and filled
// in parallel.  Cells at MAX_TREE_LEVEL that hold several particles follow the
// reference's slot-shifting rule (src/gravity/forcetree.c:861-877), which depends
// on insertion order: those cells are replayed sequentially, one thread each.
//
// Moments (force_update_node_recursive, src/gravity/forcetree.c:1217-1429) are
// accumulated bottom-up in one launch: a node is summed, its eight slots in order
// 0..7 exactly as the recursion does, by the thread that finished its last child.
// The nextnode/sibling threading and depth-first positions, which the FP64 walk
// and the exports need, follow from the subtree sizes along each node's ancestors.
#include <cub/cub.cuh>

#include "internal.h"
#include "ph.cuh"

namespace gg
{
namespace
{
__constant__ PhTable c_ph_tree;
int g_ph_tree_ready[64] = {0};

__device__ __forceinline__ int morton_slot(uint64_t x, uint64_t y, uint64_t z, int depth)
{
  // child index inside a node of depth (depth-1): bits 52-depth, x | y<<1 | z<<2 (src/gravity/forcetree.c:854-855)
  int b = 52 - depth;
  return (int)(((x >> b) & 1) | (((y >> b) & 1) << 1) | (((z >> b) & 1) << 2));
}

struct TreeArgs
{
  int64_t n;
  int32_t ntop;
  const double4 *pm;
  const uint64_t *ix, *iy, *iz;
  const uint8_t *st;
  const int8_t *cd;      // n entries, cd[n-1] = -1
  const uint8_t *tl;     // top-leaf depth
  const int32_t *tlnode; // top-leaf node (relative index)
  const int32_t *base;   // n+1
  const gpugrav_domain *dom;
  const int32_t *sys;           // several independent systems: system of each sorted particle (else null)
  const gpugrav_domain *doms;   // ... and the domain of each system
  int64_t nn;            // node capacity (known after the numbering scan; 0 before)
  int *err;              // self-check flag: set instead of writing out of bounds
};

// domain whose integer grid particle j lives on
__device__ __forceinline__ const gpugrav_domain *dom_of(const TreeArgs &a, int64_t j) { return a.sys ? &a.doms[a.sys[j]] : a.dom; }

// node index self-check: every computed node index must lie in [0, nn)
__device__ __forceinline__ bool node_ok(const TreeArgs &a, int64_t k)
{
  if(k >= 0 && k < a.nn)
    return true;
  atomicOr(a.err, 1);
  return false;
}

__device__ __forceinline__ int CD(const TreeArgs &a, int64_t i) { return (i < 0 || i >= a.n - 1) ? -1 : (int)a.cd[i]; }
__device__ __forceinline__ int cap30(int d) { return d < kMaxTreeLevel ? d : kMaxTreeLevel; }

// first depth of the canonical nodes created while inserting particle j (pair j-1, j)
__device__ __forceinline__ int dstart_of(const TreeArgs &a, int64_t j)
{
  int t = a.tl[j - 1], p = cap30(CD(a, j - 2));
  return (t > p ? t : p) + 1;
}
__device__ __forceinline__ int canon_count(const TreeArgs &a, int64_t j)
{
  if(j <= 0)
    return 0;
  int c = cap30(CD(a, j - 1)) - dstart_of(a, j) + 1;
  return c > 0 ? c : 0;
}
__device__ __forceinline__ int delta(const TreeArgs &a, int64_t p, int64_t q)
{
  if(a.sys && a.sys[p] != a.sys[q])
    return -1;  // different systems share no cell
  return common_depth(a.ix[p], a.iy[p], a.iz[p], a.ix[q], a.iy[q], a.iz[q]);
}
// smallest s <= i with delta(s, i) >= d  (start of the depth-d cell containing i)
__device__ int64_t cell_start(const TreeArgs &a, int64_t i, int d)
{
  int64_t lo_ok = i, step = 1, lo_bad = -1;
  while(true)
    {
      int64_t c = i - step;
      if(c < 0)
        {
          lo_bad = -1;
          break;
        }
      if(delta(a, c, i) >= d)
        {
          lo_ok = c;
          step <<= 1;
        }
      else
        {
          lo_bad = c;
          break;
        }
    }
  // answer in (lo_bad, lo_ok]
  while(lo_ok - lo_bad > 1)
    {
      int64_t m = lo_bad + (lo_ok - lo_bad) / 2;
      if(delta(a, m, i) >= d)
        lo_ok = m;
      else
        lo_bad = m;
    }
  return lo_ok;
}
// largest e >= s with delta(s, e) >= d
__device__ int64_t cell_end(const TreeArgs &a, int64_t s, int d)
{
  int64_t hi_ok = s, step = 1, hi_bad = a.n;
  while(true)
    {
      int64_t c = s + step;
      if(c >= a.n)
        {
          hi_bad = a.n;
          break;
        }
      if(delta(a, s, c) >= d)
        {
          hi_ok = c;
          step <<= 1;
        }
      else
        {
          hi_bad = c;
          break;
        }
    }
  while(hi_bad - hi_ok > 1)
    {
      int64_t m = hi_ok + (hi_bad - hi_ok) / 2;
      if(delta(a, s, m) >= d)
        hi_ok = m;
      else
        hi_bad = m;
    }
  return hi_ok;
}
// relative index of the canonical node of depth d whose cell starts at particle s
__device__ __forceinline__ int64_t node_of(const TreeArgs &a, int64_t s, int d)
{
  return (int64_t)a.ntop + a.base[s + 1] + (d - dstart_of(a, s + 1));
}

// ------------------------------------------------------------------------------
// Top-level tree for one rank (domain_determineTopTree, src/domain/domain_toplevel.c:111-269,
// domain_do_local_refine :280-368, domain_walktoptree :381-393), work load = count / N.
// One block: the candidates are ranked in parallel and a warp searches the sorted keys for each new
// cell's first particle (a serial search took 0.1 to 0.3 ms); the choice itself is one thread's loop.
// ------------------------------------------------------------------------------
struct TopTmp
{
  u128 size, start;
  int64_t count, pindex;
  int32_t daughter, leaf;
  double work;
};

// first position in [lo, hi) whose key is not below k; the whole warp probes 32 positions at a time
__device__ int64_t lower_bound_key(const u128 *keys, const uint32_t *perm, int64_t lo, int64_t hi, u128 k)
{
  const int lane = threadIdx.x & 31;
  while(hi > lo)
    {
      const int64_t len = hi - lo;
      if(len <= 32)
        return lo + __popc(__ballot_sync(0xffffffffu, lane < len && keys[perm[lo + (lane < len ? lane : 0)]] < k));
      const int c = __popc(__ballot_sync(0xffffffffu, keys[perm[lo + (lane + 1) * len / 33]] < k));
      const int64_t l = lo;
      lo              = c > 0 ? l + c * len / 33 + 1 : l;
      hi              = c < 32 ? l + (c + 1) * len / 33 : hi;
    }
  return lo;
}

__device__ bool top_less(const TopTmp *T, int a, int b)
{
  if(T[a].work > T[b].work)
    return true;
  if(T[a].work < T[b].work)
    return false;
  return a < b;
}

constexpr int kTopThreads = 256;
__global__ void __launch_bounds__(kTopThreads)
    k_toptree(const u128 *__restrict__ keys, const uint32_t *__restrict__ perm, int64_t n, double tnf, int mdom, TopTmp *T, int *queue,
              int *list, int *sorted, gpugrav_topnode *out, int max_top, int *result)
{
  const int ntask = 1;
  int a = 1 + (ntask / 7 + 1) * 8, b = (int)(tnf * mdom * ntask);
  int limit_ntop = 2 * (a > b ? a : b);
  if(limit_ntop + 8 > max_top)
    {
      if(threadIdx.x == 0)
        *result = -1;
      return;
    }
  double limit = 1.0 / (tnf * mdom * ntask);
  __shared__ int s_count, s_nq;
  int nq = 1, ntop = 1, nleaves = 1;
  if(threadIdx.x == 0)
    {
      T[0].daughter = -1;
      T[0].size     = (u128)1 << (3 * kBits);
      T[0].start    = 0;
      T[0].pindex   = 0;
      T[0].count    = n;
      T[0].work     = 1.0;
      queue[0]      = 0;
    }
  __syncthreads();
  while(true)
    {
      // the queue by decreasing work, then index
      for(int q = threadIdx.x; q < nq; q += kTopThreads)
        {
          const int me = queue[q];
          int rank     = 0;
          for(int p = 0; p < nq; p++)
            rank += top_less(T, queue[p], me) ? 1 : 0;
          sorted[rank] = me;
        }
      __syncthreads();
      for(int q = threadIdx.x; q < nq; q += kTopThreads)
        queue[q] = sorted[q];
      if(threadIdx.x == 0)
        {
          int count             = 0;
          double first_workload = 0;
          for(int q = 0; q < nq; q++)
            if(T[sorted[q]].size >= 8)
              {
                first_workload = T[sorted[q]].work;
                break;
              }
          for(int q = 0; q < nq; q++)
            {
              int np = sorted[q];
              if(T[np].work < 0.125 * first_workload)
                break;
              if(ntop + 8 * (count + 1) >= limit_ntop)
                break;
              if(T[np].work > limit || (nleaves < mdom * ntask && count == 0))
                {
                  if(T[np].size < 8)
                    {
                      count = -1;  // the reference stops here: PEANOGRID not fine enough
                      break;
                    }
                  list[count++] = np;
                }
            }
          s_count = count;
        }
      __syncthreads();
      const int count = s_count;
      if(count < 0)
        {
          if(threadIdx.x == 0)
            *result = -2;
          return;
        }
      if(count == 0)
        break;
      // eight daughters each: first particle of every daughter (a warp per daughter), then the counts
      for(int it = threadIdx.x >> 5; it < 8 * count; it += kTopThreads / 32)
        {
          const int i = list[it >> 3], j = it & 7, sub = ntop + it;
          const u128 size  = T[i].size >> 3;
          const u128 start = T[i].start + (u128)j * size;
          const int64_t f  = lower_bound_key(keys, perm, T[i].pindex, T[i].pindex + T[i].count, start);
          if((threadIdx.x & 31) == 0)
            {
              T[sub].daughter = -1;
              T[sub].size     = size;
              T[sub].start    = start;
              T[sub].pindex   = f;
            }
        }
      __syncthreads();
      for(int it = threadIdx.x; it < 8 * count; it += kTopThreads)
        {
          const int i = list[it >> 3], sub = ntop + it;
          const int64_t next = (it & 7) < 7 ? T[sub + 1].pindex : T[i].pindex + T[i].count;
          T[sub].count       = next - T[sub].pindex;
          T[sub].work        = (double)T[sub].count / (double)n;
          if((it & 7) == 0)
            T[i].daughter = sub;
        }
      __syncthreads();
      if(threadIdx.x == 0)
        {
          int w = 0;
          for(int q = 0; q < nq; q++)
            if(T[queue[q]].daughter < 0)
              queue[w++] = queue[q];
          for(int it = 0; it < 8 * count; it++)
            queue[w++] = ntop + it;
          s_nq = w;
        }
      ntop += 8 * count;
      nleaves += 7 * count;
      __syncthreads();
      nq = s_nq;
    }
  __syncthreads();

  // leaf numbering in Peano-Hilbert order (domain_walktoptree): the leaves partition the key space, so
  // a leaf's number is the count of leaves that start before it
  for(int i = threadIdx.x; i < ntop; i += kTopThreads)
    if(T[i].daughter < 0)
      {
        int leaf = 0;
        for(int l = 0; l < ntop; l++)
          leaf += (T[l].daughter < 0 && T[l].start < T[i].start) ? 1 : 0;
        T[i].leaf = leaf;
      }

  for(int i = threadIdx.x; i < ntop; i += kTopThreads)
    {
      out[i].start_key_hi = (uint64_t)(T[i].start >> 64);
      out[i].start_key_lo = (uint64_t)T[i].start;
      out[i].size_hi      = (uint64_t)(T[i].size >> 64);
      out[i].size_lo      = (uint64_t)T[i].size;
      out[i].daughter     = T[i].daughter;
      out[i].leaf         = T[i].daughter < 0 ? T[i].leaf : 0;
      // MortonToPeanoSubnode: Hilbert state after the node's key digits, then digit per octant
      int levels = 0;
      u128 s     = T[i].size;
      while(s < ((u128)1 << (3 * kBits)))
        {
          s <<= 3;
          levels++;
        }
      unsigned state = 0;
      for(int l = 0; l < levels; l++)
        {
          unsigned digit = (unsigned)((T[i].start >> (3 * (kBits - 1 - l))) & 7);
          unsigned oct   = 0;
          while(oct < 8 && (c_ph_tree.e[state * 8 + oct] & 7) != digit)
            oct++;
          state = c_ph_tree.e[state * 8 + (oct & 7)] >> 3;
        }
      for(unsigned oct = 0; oct < 8; oct++)
        {
          unsigned morton             = ((oct >> 2) & 1) | (((oct >> 1) & 1) << 1) | ((oct & 1) << 2);
          out[i].morton_to_peano[morton] = (uint8_t)(c_ph_tree.e[state * 8 + oct] & 7);
        }
    }
  if(threadIdx.x == 0)
    *result = ntop;
}

// ------------------------------------------------------------------------------
// Skeleton: force_create_empty_nodes (src/gravity/forcetree.c:1131-1180), iteratively,
// creating nodes in the same order (i, j, k loops, depth first).  Relative node 0 is the root (len
// DomainLen, centre DomainCenter).  One block: the depth-first creation is one thread's, on shared copies
// of the top nodes, of the cells and of the leaf table where they fit (the chain of dependent reads took
// 35 us from global memory); validation and output are everyone's.
// ------------------------------------------------------------------------------
constexpr int kSkelThreads = 128, kSkelShared = 256;
__global__ void __launch_bounds__(kSkelThreads)
    k_skeleton(const gpugrav_topnode *__restrict__ top_g, int ntop, const int *__restrict__ ntop_dev, const BuildConst *__restrict__ bc,
               int32_t *__restrict__ suns, double4 *__restrict__ cl_g, uint8_t *__restrict__ depth, int32_t *__restrict__ father,
               int32_t *__restrict__ leafnode, int32_t *__restrict__ nodetop, SkelInfo *info)
{
  __shared__ gpugrav_topnode top_sh[kSkelShared];
  __shared__ double4 cl_sh[kSkelShared];
  __shared__ int s_leaves, s_bad;
  if(ntop_dev)
    ntop = *ntop_dev;  // the library's top tree
  const bool fits            = ntop <= kSkelShared;
  const gpugrav_topnode *top = fits ? top_sh : top_g;
  double4 *cl                = fits ? cl_sh : cl_g;
  if(threadIdx.x == 0)
    s_leaves = s_bad = 0;
  __syncthreads();
  for(int t = threadIdx.x; t < ntop; t += kSkelThreads)
    {
      const gpugrav_topnode tn = top_g[t];
      if(fits)
        top_sh[t] = tn;
      if(tn.daughter < 0)
        atomicAdd(&s_leaves, 1);
      else if(tn.daughter <= t || tn.daughter + 8 > ntop)
        s_bad = 1;
    }
  __syncthreads();
  const int nleaves = s_leaves;
  for(int t = threadIdx.x; t < ntop; t += kSkelThreads)
    if(top[t].daughter < 0 && (top[t].leaf < 0 || top[t].leaf >= nleaves))
      s_bad = 1;
  for(int l = threadIdx.x; l < nleaves; l += kSkelThreads)
    leafnode[l] = -1;
  for(int64_t q = threadIdx.x; q < 8 * (int64_t)ntop; q += kSkelThreads)
    suns[q] = -1;
  __syncthreads();
  if(s_bad || ntop < 1)
    {
      if(threadIdx.x == 0)
        info->status = -2;
      return;
    }
  if(threadIdx.x == 0)
    {
      const gpugrav_domain dom = bc->dom;
      const int64_t n          = bc->n;
      cl[0]                    = make_double4(dom.center[0], dom.center[1], dom.center[2], dom.len);
      depth[0]                 = 0;
      father[0]                = -1;
      nodetop[0]               = 0;
      int numnodes = 1, maxd = 0, bad = 0;
      if(top[0].daughter < 0)
        leafnode[top[0].leaf] = 0;
      struct Frame
      {
        int no, topnode, state, ijk;  // state: of the Peano-Hilbert curve in the node's cell
      };
      Frame st[3 * kBits + 8];
      int sp   = 0;
      st[sp++] = Frame{0, 0, 0, 0};
      while(sp > 0)
        {
          Frame &f = st[sp - 1];
          if(top[f.topnode].daughter < 0 || f.ijk == 8)
            {
              sp--;
              continue;
            }
          int i = (f.ijk >> 2) & 1, j = (f.ijk >> 1) & 1, k = f.ijk & 1;
          const unsigned e = c_ph_tree.e[f.state * 8 + f.ijk];  // octant (x << 2) | (y << 1) | z
          f.ijk++;
          if(numnodes >= ntop || sp >= 3 * kBits + 8)
            {
              bad = 1;
              break;
            }
          int count = i + 2 * j + 4 * k;
          int nf    = numnodes++;
          suns[8 * f.no + count] = (int32_t)(nf + n);  // slots hold global indices: nodes start at n
          father[nf]             = (int32_t)(f.no + n);
          double4 p      = cl[f.no];
          double lenhalf = __dmul_rn(0.25, p.w);
          cl[nf] = make_double4(__dadd_rn(p.x, __dmul_rn((double)(2 * i - 1), lenhalf)),
                                __dadd_rn(p.y, __dmul_rn((double)(2 * j - 1), lenhalf)),
                                __dadd_rn(p.z, __dmul_rn((double)(2 * k - 1), lenhalf)), __dmul_rn(0.5, p.w));
          depth[nf] = (uint8_t)sp;  // the parent's depth is sp - 1
          maxd      = sp > maxd ? sp : maxd;
          int d       = top[f.topnode].daughter + (int)(e & 7);
          nodetop[nf] = d;
          if(top[d].daughter == -1)
            leafnode[top[d].leaf] = nf;
          st[sp++] = Frame{nf, d, (int)(e >> 3), 0};
        }
      s_bad               = bad;
      info->ntop_nodes    = numnodes;
      info->nleaves       = nleaves;
      info->max_top_depth = maxd;
      s_leaves            = numnodes;
    }
  __syncthreads();
  if(!ntop_dev)
    // a caller's top tree: particles descend by its morton_to_peano, nodes were made by the curve
    for(int k = threadIdx.x; k < s_leaves; k += kSkelThreads)
      {
        const gpugrav_topnode &tn = top[nodetop[k]];
        for(int q = 0; q < 8 && tn.daughter >= 0 && !s_bad; q++)
          {
            const int64_t c = suns[8 * (int64_t)k + q] - bc->n;
            if(c < 1 || c >= s_leaves || nodetop[c] != tn.daughter + tn.morton_to_peano[q])
              s_bad = 1;
          }
      }
  __syncthreads();
  for(int l = threadIdx.x; l < nleaves; l += kSkelThreads)
    if(leafnode[l] < 0)
      s_bad = 1;
  if(fits)
    for(int t = threadIdx.x; t < s_leaves; t += kSkelThreads)
      cl_g[t] = cl_sh[t];
  __syncthreads();
  if(threadIdx.x == 0)
    info->status = s_bad ? -2 : 0;
}

// top leaf of every sorted particle: walk TopNodes with MortonToPeanoSubnode
// (src/gravity/forcetree.c:507-522)
__global__ void k_topleaf(const gpugrav_topnode *__restrict__ top, const int32_t *__restrict__ leafnode,
                          const SkelInfo *__restrict__ info, int64_t n,
                          const uint64_t *__restrict__ ix, const uint64_t *__restrict__ iy, const uint64_t *__restrict__ iz,
                          uint8_t *__restrict__ tl, int32_t *__restrict__ tlnode)
{
  for(int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    {
      uint64_t x = ix[i], y = iy[i], z = iz[i];
      int no = 0, levels = 0;
      if(info->status < 0)
        {
          // invalid top tree: the build stops after the host has read the status
          tl[i]     = 0;
          tlnode[i] = 0;
          continue;
        }
      while(top[no].daughter >= 0 && levels < 52)
        {
          int b      = 51 - levels;
          int sub    = (int)(((x >> b) & 1) | (((y >> b) & 1) << 1) | (((z >> b) & 1) << 2));
          levels++;
          no = top[no].daughter + top[no].morton_to_peano[sub];
        }
      tl[i]     = (uint8_t)levels;
      tlnode[i] = leafnode[top[no].leaf];
    }
}

__global__ void k_pairdepth(int64_t n, const uint64_t *__restrict__ ix, const uint64_t *__restrict__ iy,
                            const uint64_t *__restrict__ iz, const int32_t *__restrict__ sys, int8_t *__restrict__ cd)
{
  // particles of different systems share no cell
  for(int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    cd[i] = (i + 1 < n && (!sys || sys[i] == sys[i + 1]))
                ? (int8_t)common_depth(ix[i], iy[i], iz[i], ix[i + 1], iy[i + 1], iz[i + 1])
                : (int8_t)-1;
}

// several systems: node s is the root of system s (len DomainLen, centre DomainCenter of that system)
__global__ void k_roots(int nsys, const gpugrav_domain *__restrict__ doms, int32_t *__restrict__ suns, double4 *__restrict__ cl,
                        uint8_t *__restrict__ depth, int32_t *__restrict__ father)
{
  for(int s = blockIdx.x * blockDim.x + threadIdx.x; s < nsys; s += gridDim.x * blockDim.x)
    {
      for(int q = 0; q < 8; q++)
        suns[8 * (int64_t)s + q] = -1;
      cl[s]     = make_double4(doms[s].center[0], doms[s].center[1], doms[s].center[2], doms[s].len);
      depth[s]  = 0;
      father[s] = -1;
    }
}

// several systems: every particle's "top leaf" is its system's root, at depth 0
__global__ void k_tl_roots(int64_t n, const int32_t *__restrict__ sys, uint8_t *__restrict__ tl, int32_t *__restrict__ tlnode)
{
  for(int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    {
      tl[i]     = 0;
      tlnode[i] = sys[i];
    }
}

// canonical node count per inserting particle + detection of replayed (coincident) cells
__global__ void k_count(TreeArgs a, int32_t *__restrict__ cnt, int32_t *__restrict__ hack_start, int *counters)
{
  for(int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j <= a.n; j += (int64_t)gridDim.x * blockDim.x)
    {
      if(j == a.n)
        {
          cnt[j] = 0;
          continue;
        }
      cnt[j] = canon_count(a, j);
      // cell at MAX_TREE_LEVEL with >= 2 particles starting at j (below a shallower top leaf) ...
      bool h = (a.tl[j] < kMaxTreeLevel) && (CD(a, j) >= kMaxTreeLevel) && (CD(a, j - 1) < kMaxTreeLevel);
      // ... or a top leaf at or below MAX_TREE_LEVEL (its first particle)
      h = h || (a.tl[j] >= kMaxTreeLevel && (j == 0 || a.tlnode[j - 1] != a.tlnode[j]));
      if(h)
        {
          int slot = atomicAdd(&counters[1], 1);
          hack_start[slot] = (int32_t)j;
        }
    }
}

// ---- replay of cells where the MAX_TREE_LEVEL rule applies ----
struct HackCell
{
  int64_t s, e;      // particle range (sorted indices, inclusive)
  int64_t scratch;   // offset into the scratch node pool (count pass)
  int32_t level;     // depth of the cell's node
  int32_t top_leaf;  // 1: the cell is a top leaf
};

__global__ void k_hack_range(TreeArgs a, const int32_t *__restrict__ hack_start, int nh, HackCell *cells, int64_t *sizes)
{
  int h = blockIdx.x * blockDim.x + threadIdx.x;
  if(h >= nh)
    return;
  int64_t s = hack_start[h];
  HackCell c;
  c.s = s;
  if(a.tl[s] >= kMaxTreeLevel)
    {
      int64_t e = s;
      while(e + 1 < a.n && a.tlnode[e + 1] == a.tlnode[s])
        e++;
      c.e        = e;
      c.level    = a.tl[s];
      c.top_leaf = 1;
    }
  else
    {
      c.e        = cell_end(a, s, kMaxTreeLevel);
      c.level    = kMaxTreeLevel;
      c.top_leaf = 0;
    }
  c.scratch = 0;
  cells[h]  = c;
  sizes[h]  = c.e - c.s + 1;
}

template <bool FILL>
__device__ void replay_cell(const TreeArgs &a, const HackCell &c, int32_t *suns, int32_t *scratch_suns, int32_t *cnt,
                            double4 *cl, uint8_t *depth, int32_t *father)
{
  // node storage: FILL -> the real node arrays (relative indices); count pass -> a local pool
  // whose entry 0 is the cell node itself
  const int64_t n = a.n;
  int64_t cellnode;
  if(FILL)
    cellnode = c.top_leaf ? (int64_t)a.tlnode[c.s] : node_of(a, c.s, kMaxTreeLevel);
  else
    cellnode = 0;
  int32_t *S    = FILL ? suns : scratch_suns;
  int64_t local = 1;
  // node storage capacity: the whole node array, or one pool entry per particle of the cell
  // (each insertion below MAX_TREE_LEVEL creates at most one node)
  const int64_t cap = FILL ? a.nn : (c.e - c.s + 1);
  if(cellnode < 0 || cellnode >= cap)
    {
      atomicOr(a.err, 2);
      return;
    }
  auto SUN = [&](int64_t node, int slot) -> int32_t & { return S[8 * node + slot]; };
  if(!FILL)
    for(int q = 0; q < 8; q++)
      SUN(0, q) = -1;

  // the first particle takes its natural slot (node creation, src/gravity/forcetree.c:921-924,
  // or the first insertion into an empty top leaf)
  SUN(cellnode, morton_slot(a.ix[c.s], a.iy[c.s], a.iz[c.s], c.level + 1)) = (int32_t)c.s;

  for(int64_t q = c.s + 1; q <= c.e; q++)
    {
      const uint64_t xxb = a.ix[q], yyb = a.iy[q], zzb = a.iz[q];
      int levels         = c.level;
      uint64_t mask      = 1ull << (51 - levels);
      int shiftx = 51 - levels, shifty = 50 - levels, shiftz = 49 - levels;
      int64_t centermask = (int64_t)0xFFF0000000000000ull;
      centermask >>= levels;
      int64_t th = cellnode + n;  // node handle: >= n is a node
      int64_t parent = -1;
      int subnode    = 0;
      int created    = 0;
      int64_t fbase  = FILL ? ((int64_t)a.ntop + a.base[q] + canon_count(a, q)) : 0;
      auto shr = [](uint64_t v, int s) -> uint64_t { return (s < 0 || s > 63) ? 0 : (v >> s); };
      for(int guard = 0; guard < 4096; guard++)
        {
          if(th >= n)
            {
              int64_t nd = th - n;
              subnode    = (int)(shr(xxb & mask, shiftx) | shr(yyb & mask, shifty) | shr(zzb & mask, shiftz));
              shiftx--;
              shifty--;
              shiftz--;
              centermask >>= 1;
              mask >>= 1;
              levels++;
              if(levels > kMaxTreeLevel)
                {
                  for(int jj = 0; jj < 8; jj++)
                    {
                      if(SUN(nd, subnode) < 0)
                        break;
                      subnode++;
                      if(subnode >= 8)
                        subnode = 7;
                    }
                }
              int32_t nn = SUN(nd, subnode);
              if(nn >= 0)
                {
                  parent = nd;
                  th     = nn;
                }
              else
                {
                  SUN(nd, subnode) = (int32_t)q;
                  break;
                }
            }
          else
            {
              int64_t nf = FILL ? (fbase + created) : (local++);
              if(nf < 0 || nf >= cap || th < 0 || th >= n)
                {
                  atomicOr(a.err, 2);
                  return;
                }
              SUN(parent, subnode) = (int32_t)(nf + n);
              if(FILL)
                {
                  const gpugrav_domain *dm = dom_of(a, q);
                  const double bf          = dm->big_fac;
                  double len               = __dmul_rn((double)(mask << 1), bf);
                  double cx = __dadd_rn(__dmul_rn((double)((xxb & (uint64_t)centermask) | mask), bf), dm->corner[0]);
                  double cy = __dadd_rn(__dmul_rn((double)((yyb & (uint64_t)centermask) | mask), bf), dm->corner[1]);
                  double cz = __dadd_rn(__dmul_rn((double)((zzb & (uint64_t)centermask) | mask), bf), dm->corner[2]);
                  cl[nf]     = make_double4(cx, cy, cz, len);
                  depth[nf]  = (uint8_t)(levels > 255 ? 255 : levels);
                  father[nf] = (int32_t)(parent + n);
                }
              for(int jj = 0; jj < 8; jj++)
                SUN(nf, jj) = -1;
              int sub2 = (int)(shr(a.ix[th] & mask, shiftx) | shr(a.iy[th] & mask, shifty) | shr(a.iz[th] & mask, shiftz));
              SUN(nf, sub2) = (int32_t)th;
              th            = nf + n;
              created++;
            }
        }
      if(!FILL)
        cnt[q] += created;
    }
}

__global__ void k_hack_count(TreeArgs a, const HackCell *cells, const int64_t *offsets, int nh, int32_t *scratch, int32_t *cnt)
{
  int h = blockIdx.x * blockDim.x + threadIdx.x;
  if(h >= nh)
    return;
  HackCell c = cells[h];
  replay_cell<false>(a, c, nullptr, scratch + 8 * offsets[h], cnt, nullptr, nullptr, nullptr);
}

__global__ void k_hack_fill(TreeArgs a, const HackCell *cells, int nh, int32_t *suns, double4 *cl, uint8_t *depth,
                            int32_t *father)
{
  int h = blockIdx.x * blockDim.x + threadIdx.x;
  if(h >= nh)
    return;
  HackCell c = cells[h];
  replay_cell<true>(a, c, suns, nullptr, nullptr, cl, depth, father);
}

// ---- canonical nodes: centre/len (src/gravity/forcetree.c:903-911), parent slot ----
__global__ void k_nodes(TreeArgs a, int32_t *__restrict__ suns, double4 *__restrict__ cl, uint8_t *__restrict__ depth)
{
  for(int64_t j = 1 + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < a.n; j += (int64_t)gridDim.x * blockDim.x)
    {
      int cnt = canon_count(a, j);
      if(cnt <= 0)
        continue;
      int d0          = dstart_of(a, j);
      int64_t k0      = (int64_t)a.ntop + a.base[j];
      uint64_t x = a.ix[j], y = a.iy[j], z = a.iz[j];
      const gpugrav_domain *dm = dom_of(a, j);
      const double bf          = dm->big_fac;
      for(int t = 0; t < cnt; t++)
        {
          int d      = d0 + t;
          int64_t k  = k0 + t;
          uint64_t m = 1ull << (51 - d);
          uint64_t keep = ~((1ull << (52 - d)) - 1ull);
          double len = __dmul_rn((double)(m << 1), bf);
          double cx  = __dadd_rn(__dmul_rn((double)((x & keep) | m), bf), dm->corner[0]);
          double cy  = __dadd_rn(__dmul_rn((double)((y & keep) | m), bf), dm->corner[1]);
          double cz  = __dadd_rn(__dmul_rn((double)((z & keep) | m), bf), dm->corner[2]);
          cl[k]      = make_double4(cx, cy, cz, len);
          depth[k]   = (uint8_t)d;
          for(int q = 0; q < 8; q++)
            suns[8 * k + q] = -1;
        }
    }
}

// link canonical nodes into their parents' slots
__global__ void k_link_nodes(TreeArgs a, int32_t *__restrict__ suns, int32_t *__restrict__ father)
{
  for(int64_t j = 1 + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < a.n; j += (int64_t)gridDim.x * blockDim.x)
    {
      int cnt = canon_count(a, j);
      if(cnt <= 0)
        continue;
      int d0     = dstart_of(a, j);
      int64_t k0 = (int64_t)a.ntop + a.base[j];
      uint64_t x = a.ix[j], y = a.iy[j], z = a.iz[j];
      // first node: parent is the top leaf or a canonical node of an earlier particle
      int pd = d0 - 1;
      int64_t parent;
      if(pd == a.tl[j - 1])
        parent = a.tlnode[j - 1];
      else
        parent = node_of(a, cell_start(a, j - 1, pd), pd);
      if(!node_ok(a, parent) || !node_ok(a, k0 + cnt - 1))
        continue;
      suns[8 * parent + morton_slot(x, y, z, d0)] = (int32_t)(k0 + a.n);
      father[k0]                                  = (int32_t)(parent + a.n);
      for(int t = 1; t < cnt; t++)
        {
          suns[8 * (k0 + t - 1) + morton_slot(x, y, z, d0 + t)] = (int32_t)(k0 + t + a.n);
          father[k0 + t]                                        = (int32_t)(k0 + t - 1 + a.n);
        }
    }
}

// particles into the slot of their deepest node
__global__ void k_leaves(TreeArgs a, int32_t *__restrict__ suns)
{
  for(int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < a.n; i += (int64_t)gridDim.x * blockDim.x)
    {
      int tl = a.tl[i];
      if(tl >= kMaxTreeLevel)
        continue;  // replayed
      int dp = cap30(CD(a, i - 1)), dn = cap30(CD(a, i));
      int D  = dp > dn ? dp : dn;
      int64_t parent;
      if(D <= tl)
        {
          parent = a.tlnode[i];
          D      = tl;
        }
      else if(D >= kMaxTreeLevel)
        continue;  // replayed
      else if(dn == D && CD(a, i - 1) < D)
        parent = node_of(a, i, D);
      else
        parent = node_of(a, cell_start(a, i, D), D);
      if(!node_ok(a, parent))
        continue;
      suns[8 * parent + morton_slot(a.ix[i], a.iy[i], a.iz[i], D + 1)] = (int32_t)i;
    }
}

// ---- children ----
__device__ __forceinline__ void load_suns(const int32_t *__restrict__ suns, int64_t k, int32_t (&c)[8])
{
  const int4 a = ((const int4 *)suns)[2 * k], b = ((const int4 *)suns)[2 * k + 1];
  c[0] = a.x, c[1] = a.y, c[2] = a.z, c[3] = a.w, c[4] = b.x, c[5] = b.y, c[6] = b.z, c[7] = b.w;
}

// counts of every node (node children | particle children << 4), arrival counters of the upward pass
// cleared, deepest level
__global__ void k_children(int64_t nn, int32_t n, const int32_t *__restrict__ suns, const uint8_t *__restrict__ depth,
                           uint8_t *__restrict__ count, int32_t *__restrict__ arrived, int *__restrict__ deepest)
{
  int d = 0;
  for(int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nn; k += (int64_t)gridDim.x * blockDim.x)
    {
      int32_t c[8];
      load_suns(suns, k, c);
      int nc = 0, np = 0;
#pragma unroll
      for(int q = 0; q < 8; q++)
        {
          nc += c[q] >= n ? 1 : 0;
          np += c[q] >= 0 && c[q] < n ? 1 : 0;
        }
      count[k]   = (uint8_t)(nc | (np << 4));
      arrived[k] = 0;
      d          = depth[k] > d ? depth[k] : d;
    }
  d = __reduce_max_sync(0xffffffffu, d);
  if((threadIdx.x & 31) == 0 && d > 0)
    atomicMax(deepest, d);
}

constexpr int kChildren = 4;  // records that k_moments reads at a time
// ancestors of a node: a replayed cell's chain has up to 4096 (replay_cell's bound), below the tree's levels
constexpr int kMaxChain = 4096 + 64;

// ---- moments (force_update_node_recursive, src/gravity/forcetree.c:1266-1392) ----
// Every thread starts at a node without node children and goes up as long as it is the last to arrive at
// the parent, so that the whole tree takes one launch; what other threads wrote is read from L2.  One
// launch per level (two dozen) left the narrow upper levels to pay a launch and a memory latency chain
// each: 0.15 ms on 4099 particles against 0.05.  Bound by latency -- a warp's lanes go up at different times, each
// step a round trip to the children, one to the counter --, hence by the warps in flight: the children are read
// four at a time, which leaves 64 registers and eight blocks per SM, and the counter's addition carries the ordering
// (release of this node's record, acquire of the siblings') instead of two fences around it.  With all eight
// children at once (104 registers) and fences the build of the 2^24 zoom box took 4.26 ms, of 256^3 targets 2.21, of
// 2^20 0.38; now 2.96, 1.86 and 0.30 (level by level 1.3 of it were moments, in one launch 2.7, now 1.3).
template <bool MNS>
__global__ void __launch_bounds__(128, 8)
    k_moments(int64_t nn, int32_t n, const int32_t *__restrict__ suns, const uint8_t *__restrict__ count, int32_t *__restrict__ arrived,
              const int32_t *__restrict__ father, const double4 *__restrict__ pm, const uint8_t *__restrict__ st,
              const double4 *__restrict__ cl, double4 *sm, uint8_t *maxsoft, int32_t *size, const BuildConst *__restrict__ bc,
              double *mpt, int *err)
{
  int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  // after a failed self-check some fathers and children are not set: the build ends without following any
  if(k >= nn || *err || (count[k] & 15) != 0)
    return;
  for(int g = 0; g < kMaxChain; g++)
    {
      int32_t c[8];
      load_suns(suns, k, c);
      if(MNS)
        {
          // ExtNodes[].mass_per_type (MULTIPLE_NODE_SOFTENING, src/gravity/forcetree.c:1256-1308): per type,
          // the particle masses and the child sums of slots 0..7 in order
          const int ns = bc->nsoft;
          double acc[GPUGRAV_MAX_SOFTTYPES];
          for(int q = 0; q < ns; q++)
            acc[q] = 0.0;
          for(int q = 0; q < 8; q++)
            {
              if(c[q] < 0)
                continue;
              if(c[q] < n)
                {
                  const int s = st[c[q]];
                  acc[s]      = __dadd_rn(acc[s], pm[c[q]].w);
                }
              else
                for(int u = 0; u < ns; u++)
                  acc[u] = __dadd_rn(acc[u], __ldcg(&mpt[(int64_t)(c[q] - n) * ns + u]));
            }
          for(int q = 0; q < ns; q++)
            mpt[k * ns + q] = acc[q];
        }
      double mass = 0, sx = 0, sy = 0, sz_ = 0;
      int ms    = bc->nsoft;  // NSOFTTYPES + NSOFTTYPES_HYDRO: the entry whose softening is 0
      int total = 1;
#pragma unroll
      for(int h = 0; h < 8; h += kChildren)
        {
          // some children's records, fetched together
          double4 m[kChildren];
          int ts[kChildren], sz[kChildren];
#pragma unroll
          for(int q = 0; q < kChildren; q++)
            {
              const int32_t v = c[h + q];
              m[q]            = make_double4(0, 0, 0, 0);
              ts[q] = sz[q] = 0;
              if(v >= n)
                {
                  const double2 *r = (const double2 *)(sm + (v - n));
                  const double2 a = __ldcg(r), b = __ldcg(r + 1);
                  m[q]  = make_double4(a.x, a.y, b.x, b.y);
                  ts[q] = __ldcg(maxsoft + (v - n));
                  sz[q] = __ldcg(size + (v - n));
                }
              else if(v >= 0)
                {
                  m[q]  = pm[v];
                  ts[q] = st[v];
                  sz[q] = 1;
                }
            }
#pragma unroll
          for(int q = 0; q < kChildren; q++)
            if(c[h + q] >= 0)
              {
                mass = __dadd_rn(mass, m[q].w);
                sx   = __dadd_rn(sx, __dmul_rn(m[q].w, m[q].x));
                sy   = __dadd_rn(sy, __dmul_rn(m[q].w, m[q].y));
                sz_  = __dadd_rn(sz_, __dmul_rn(m[q].w, m[q].z));
                if(bc->soft[ms] < bc->soft[ts[q]])
                  ms = ts[q];
                total += sz[q];
              }
        }
      if(mass != 0)
        {
          sx  = __ddiv_rn(sx, mass);
          sy  = __ddiv_rn(sy, mass);
          sz_ = __ddiv_rn(sz_, mass);
        }
      else
        {
          const double4 q = cl[k];
          sx  = q.x;
          sy  = q.y;
          sz_ = q.z;
        }
      sm[k]           = make_double4(sx, sy, sz_, mass);
      maxsoft[k]      = (uint8_t)ms;
      size[k]         = total;
      const int32_t p = father[k];
      if(p < n)
        return;  // a root
      k = p - n;
      int before;
      asm volatile("atom.add.acq_rel.gpu.global.s32 %0, [%1], 1;" : "=r"(before) : "l"(arrived + k) : "memory");
      if(before + 1 < (count[k] & 15))
        return;
    }
  atomicOr(err, 16);  // no root above: the build's self-check
}

// ---- threading and depth-first positions ----
constexpr int32_t kInherit = -2;     // the link is the father's sibling

// per node: its children's offsets from its own position and the links among them
__global__ void k_offsets(int64_t nn, int32_t n, const int32_t *__restrict__ suns, const int32_t *__restrict__ size,
                          const int32_t *__restrict__ father, int32_t *__restrict__ noff, int32_t *__restrict__ nsib,
                          int32_t *__restrict__ nnext, int32_t *__restrict__ poff, int32_t *__restrict__ pnext,
                          int32_t *__restrict__ pfather, const int *__restrict__ err)
{
  if(*err)
    return;
  for(int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nn; k += (int64_t)gridDim.x * blockDim.x)
    {
      int32_t c[8];
      load_suns(suns, k, c);
      int32_t off = 1, first = kInherit, last = -1;
#pragma unroll
      for(int q = 0; q < 8; q++)
        if(c[q] >= 0)
          {
            // the previous child's link is this one
            if(last < 0)
              first = c[q];
            else if(last < n)
              pnext[last] = c[q];
            else
              nsib[last - n] = c[q];
            last = c[q];
            if(c[q] < n)
              {
                poff[c[q]]    = off;
                pfather[c[q]] = (int32_t)(k + n);
                off += 1;
              }
            else
              {
                noff[c[q] - n] = off;
                off += size[c[q] - n];
              }
          }
      if(last >= n)
        nsib[last - n] = kInherit;
      else if(last >= 0)
        pnext[last] = kInherit;
      nnext[k] = first;
      if(father[k] < 0)
        {
          noff[k] = 0;
          nsib[k] = -1;
        }
    }
}

// per node: position = offsets of the node and its ancestors; an inherited sibling is that of the nearest
// ancestor that has one (a concurrent thread may have resolved it already: the same value)
__global__ void k_thread(int64_t nn, int32_t n, const int32_t *__restrict__ father, const int32_t *__restrict__ noff, int32_t *nsib,
                         int32_t *__restrict__ nnext, int32_t *__restrict__ ndfs, int *err)
{
  if(*err)
    return;
  for(int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nn; k += (int64_t)gridDim.x * blockDim.x)
    {
      int32_t pos = noff[k], sib = nsib[k];
      int32_t p   = father[k];
      for(int g = 0; p >= 0 && g < kMaxChain; g++)
        {
          pos += noff[p - n];
          if(sib == kInherit)
            sib = __ldcg(nsib + (p - n));
          p = father[p - n];
        }
      if(p >= 0)
        atomicOr(err, 16);
      ndfs[k] = pos;
      nsib[k] = sib;
      if(nnext[k] == kInherit)
        nnext[k] = sib;
    }
}

// ---- walk layout in depth-first order ----
__global__ void k_layout(int64_t n, int64_t nn, const double4 *__restrict__ pm, const uint8_t *__restrict__ st,
                         const int32_t *__restrict__ poff, const int32_t *__restrict__ pfather, int32_t *__restrict__ pnext,
                         const int32_t *__restrict__ nsib, const double4 *__restrict__ sm, const double4 *__restrict__ cl,
                         const uint8_t *__restrict__ maxsoft, const int32_t *__restrict__ size,
                         const int32_t *__restrict__ ndfs, double4 *__restrict__ w_sm, double4 *__restrict__ w_cl,
                         int2 *__restrict__ w_link, int *err, const double *__restrict__ mpt, int nsoft,
                         double *__restrict__ w_mpt)
{
  const int64_t ne = n + nn;
  for(int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n + nn; t += (int64_t)gridDim.x * blockDim.x)
    {
      if(t < n)
        {
          const int64_t f = pfather[t] - n;
          const int32_t e = f >= 0 && f < nn ? ndfs[f] + poff[t] : -1;
          if(e < 0 || e >= ne)
            {
              atomicOr(err, 4);
              continue;
            }
          if(pnext[t] == kInherit)
            pnext[t] = nsib[f];
          w_sm[e]   = pm[t];
          w_cl[e]   = make_double4(0, 0, 0, 0);
          w_link[e] = make_int2(e + 1, (int)st[t]);
        }
      else
        {
          int64_t k = t - n;
          int32_t e = ndfs[k];
          if(e < 0 || e >= ne || e + size[k] > ne)
            {
              atomicOr(err, 4);
              continue;
            }
          w_sm[e]   = sm[k];
          w_cl[e]   = cl[k];
          w_link[e] = make_int2(e + size[k], (int)maxsoft[k] | kNodeFlag);
          if(w_mpt)
            for(int q = 0; q < nsoft; q++)
              w_mpt[(int64_t)e * nsoft + q] = mpt[k * nsoft + q];
        }
    }
}

int grid_for(int64_t n, int threads)
{
  int64_t b = (n + threads - 1) / threads;
  if(b > 148 * 16)
    b = 148 * 16;
  return (int)(b < 1 ? 1 : b);
}

cudaError_t ensure_ph(int device, cudaStream_t st)
{
  if(device >= 0 && device < 64 && g_ph_tree_ready[device])
    return cudaSuccess;
  PhTable t     = ph_make_table();
  cudaError_t e = cudaMemcpyToSymbolAsync(c_ph_tree, &t, sizeof(t), 0, cudaMemcpyHostToDevice, st);
  if(e == cudaSuccess)
    e = cudaStreamSynchronize(st);  // other contexts' streams read it from now on
  if(e == cudaSuccess && device >= 0 && device < 64)
    g_ph_tree_ready[device] = 1;
  return e;
}
}  // namespace

// The node count stays on the device (counters[kTopCount]); the host allocates for the bound.
cudaError_t toptree_stage(gpugrav_ctx *c, int *status)
{
  GG_TRY(ensure_ph(c->device, c->stream));
  const int max_top = kMaxTop;
  const int a = 1 + 2 * 4, b = (int)(c->prm.top_node_factor * c->prm.multiple_domains);
  c->ntop_cap = 2 * (a > b ? a : b) + 8;  // k_toptree's limit and one refinement more
  *status     = GPUGRAV_OK;
  if(c->ntop_cap > max_top)
    {
      *status = GPUGRAV_ERR_TOPNODES;
      return cudaSuccess;
    }
  GG_TRY(c->top.ensure(max_top * sizeof(gpugrav_topnode)));
  GG_TRY(c->scratch.ensure(max_top * (sizeof(TopTmp) + 3 * sizeof(int)) + 256));
  GG_TRY(c->counters.ensure(kCounters * sizeof(int)));
  char *s     = (char *)c->scratch.p;
  TopTmp *T   = (TopTmp *)s;
  int *queue  = (int *)(s + max_top * sizeof(TopTmp));
  int *list   = queue + max_top;
  k_toptree<<<1, kTopThreads, 0, c->stream>>>(c->key.as<u128>(), c->perm.as<uint32_t>(), c->n, c->prm.top_node_factor,
                                              c->prm.multiple_domains, T, queue, list, list + max_top, c->top.as<gpugrav_topnode>(),
                                              max_top, c->counters.as<int>() + kTopCount);
  c->top_dev = true;
  return cudaGetLastError();
}

// Builds the whole tree: skeleton, nodes, moments, threading, walk layout.
// node arrays for nn nodes
cudaError_t node_arrays(gpugrav_ctx *c, int64_t nn)
{
  cudaError_t e;
  if((e = c->n_suns.ensure(nn * 8 * sizeof(int32_t))) != cudaSuccess)
    return e;
  if((e = c->n_depth.ensure(nn + 16)) != cudaSuccess)
    return e;
  if((e = c->n_cl.ensure(nn * sizeof(double4))) != cudaSuccess)
    return e;
  if((e = c->n_sm.ensure(nn * sizeof(double4))) != cudaSuccess)
    return e;
  if((e = c->n_maxsoft.ensure(nn + 16)) != cudaSuccess)
    return e;
  if((e = c->n_size.ensure(nn * sizeof(int32_t))) != cudaSuccess)
    return e;
  if((e = c->n_father.ensure(nn * sizeof(int32_t))) != cudaSuccess)
    return e;
  if((e = c->n_count.ensure(nn + 16)) != cudaSuccess)
    return e;
  if((e = c->n_arrived.ensure(nn * sizeof(int32_t))) != cudaSuccess)
    return e;
  return cudaSuccess;
}

// every buffer of build_stage sized for n particles, nn nodes and ntop top nodes (or systems), so
// that a long-lived caller allocates once
cudaError_t build_reserve(gpugrav_ctx *c, int64_t n, int64_t nn, int32_t ntop)
{
  GG_TRY(c->s_cd.ensure(n + 16));
  GG_TRY(c->s_tl.ensure(n + 16));
  GG_TRY(c->s_tlnode.ensure((n + 16) * sizeof(int32_t)));
  GG_TRY(c->cnt.ensure((n + 16) * sizeof(int32_t)));
  GG_TRY(c->base.ensure((n + 16) * sizeof(int32_t)));
  GG_TRY(c->hack_list.ensure((n + 16) * sizeof(int32_t)));
  GG_TRY(c->counters.ensure(kCounters * sizeof(int)));
  GG_TRY(c->skel.ensure(sizeof(SkelInfo) + (size_t)(ntop + 8) * 2 * sizeof(int32_t)));
  GG_TRY(node_arrays(c, nn + 16));
  size_t tb = 0;
  GG_TRY(cub::DeviceScan::ExclusiveSum(nullptr, tb, c->cnt.as<int32_t>(), c->base.as<int32_t>(), (int)(n + 1), c->stream));
  return c->sort_tmp.ensure(tb);
}

// nextnode/sibling threading, fathers of the particles and the FP64 walk's layout of the built tree
cudaError_t thread_stage(gpugrav_ctx *c)
{
  const int64_t n = c->n, nn = c->num_nodes, ne = n + nn;
  cudaStream_t st = c->stream;
  const bool mns  = c->built_mns;
  GG_TRY(c->n_off.ensure((nn + 16) * sizeof(int32_t)));
  GG_TRY(c->n_sibling.ensure((nn + 16) * sizeof(int32_t)));
  GG_TRY(c->n_next.ensure((nn + 16) * sizeof(int32_t)));
  GG_TRY(c->n_dfs.ensure((nn + 16) * sizeof(int32_t)));
  GG_TRY(c->p_next.ensure((n + 16) * sizeof(int32_t)));
  GG_TRY(c->p_father.ensure((n + 16) * sizeof(int32_t)));
  GG_TRY(c->p_off.ensure((n + 16) * sizeof(int32_t)));
  GG_TRY(c->w_sm.ensure(ne * sizeof(double4)));
  GG_TRY(c->w_cl.ensure(ne * sizeof(double4)));
  GG_TRY(c->w_link.ensure(ne * sizeof(int2)));
  if(mns)
    GG_TRY(c->w_mpt.ensure((size_t)ne * c->prm.nsofttypes * sizeof(double)));
  k_offsets<<<grid_for(nn, 256), 256, 0, st>>>(nn, (int32_t)n, c->n_suns.as<int32_t>(), c->n_size.as<int32_t>(),
                                               c->n_father.as<int32_t>(), c->n_off.as<int32_t>(), c->n_sibling.as<int32_t>(),
                                               c->n_next.as<int32_t>(), c->p_off.as<int32_t>(), c->p_next.as<int32_t>(),
                                               c->p_father.as<int32_t>(), c->counters.as<int>() + 12);
  k_thread<<<grid_for(nn, 256), 256, 0, st>>>(nn, (int32_t)n, c->n_father.as<int32_t>(), c->n_off.as<int32_t>(),
                                              c->n_sibling.as<int32_t>(), c->n_next.as<int32_t>(), c->n_dfs.as<int32_t>(),
                                              c->counters.as<int>() + 12);
  k_layout<<<grid_for(ne, 256), 256, 0, st>>>(n, nn, c->s_pm.as<double4>(), c->s_st.as<uint8_t>(), c->p_off.as<int32_t>(),
                                               c->p_father.as<int32_t>(), c->p_next.as<int32_t>(), c->n_sibling.as<int32_t>(),
                                               c->n_sm.as<double4>(), c->n_cl.as<double4>(), c->n_maxsoft.as<uint8_t>(),
                                               c->n_size.as<int32_t>(), c->n_dfs.as<int32_t>(), c->w_sm.as<double4>(),
                                               c->w_cl.as<double4>(), c->w_link.as<int2>(), c->counters.as<int>() + 12,
                                               mns ? c->n_mpt.as<double>() : nullptr, c->prm.nsofttypes,
                                               mns ? c->w_mpt.as<double>() : nullptr);
  c->threaded = true;
  return cudaGetLastError();
}

// the same for a tree that was built for the group walk
cudaError_t thread_ensure(gpugrav_ctx *c)
{
  if(c->threaded)
    return cudaSuccess;
  int *err = c->counters.as<int>() + 12;
  GG_TRY(cudaMemsetAsync(err, 0, sizeof(int), c->stream));
  GG_TRY(thread_stage(c));
  int e = 0;
  GG_TRY(cudaMemcpyAsync(&e, err, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
  GG_TRY(cudaStreamSynchronize(c->stream));
  c->threaded = e == 0;
  return e == 0 ? cudaSuccess : cudaErrorUnknown;
}

cudaError_t build_stage(gpugrav_ctx *c, int *status)
{
  GG_TRY(ensure_ph(c->device, c->stream));
  const int64_t n    = c->n;
  const bool lib_top = !c->multi && c->top_dev;      // top tree built by toptree_stage: its size is on the device
  int32_t ntop       = lib_top ? c->ntop_cap : c->ntop;  // ... and this its bound until the host has read it
  cudaStream_t st    = c->stream;
  int launches       = 0;
  *status            = GPUGRAV_OK;
  HostIo *io         = c->io();
  if(!io)
    return cudaErrorMemoryAllocation;
  c->mark(nullptr);

  GG_TRY(c->s_cd.ensure(n + 16));
  GG_TRY(c->s_tl.ensure(n + 16));
  GG_TRY(c->s_tlnode.ensure((n + 16) * sizeof(int32_t)));
  GG_TRY(c->cnt.ensure((n + 16) * sizeof(int32_t)));
  GG_TRY(c->base.ensure((n + 16) * sizeof(int32_t)));
  GG_TRY(c->hack_list.ensure((n + 16) * sizeof(int32_t)));
  GG_TRY(c->counters.ensure(kCounters * sizeof(int)));
  GG_TRY(c->skel.ensure(sizeof(SkelInfo) + (size_t)(ntop + 8) * 2 * sizeof(int32_t)));
  int *counters     = c->counters.as<int>();
  SkelInfo *sinfo   = (SkelInfo *)c->skel.p;
  int32_t *leafnode = (int32_t *)((char *)c->skel.p + sizeof(SkelInfo));
  int32_t *nodetop  = leafnode + ntop + 4;

  // skeleton needs node storage for the first ntop nodes; size node arrays for ntop now, grow later
  auto ensure_nodes = [&](int64_t nn) { return node_arrays(c, nn); };

  // 1. per-particle top leaf, pair depths (skeleton first: it validates the top tree and maps leaves to nodes)
  const int32_t *msys            = c->multi ? c->m_sys.as<int32_t>() : nullptr;
  const gpugrav_domain *mdoms    = c->multi ? c->m_doms.as<gpugrav_domain>() : nullptr;
  GG_TRY(ensure_nodes(ntop + 16));
  if(c->multi)
    {
      // independent systems: one root per system, no top-level skeleton below it
      k_roots<<<grid_for(ntop, 128), 128, 0, st>>>(ntop, mdoms, c->n_suns.as<int32_t>(), c->n_cl.as<double4>(),
                                                    c->n_depth.as<uint8_t>(), c->n_father.as<int32_t>());
      k_tl_roots<<<grid_for(n, 256), 256, 0, st>>>(n, msys, c->s_tl.as<uint8_t>(), c->s_tlnode.as<int32_t>());
      c->nleaves = ntop;
      launches += 2;
    }
  else
    {
      k_skeleton<<<1, kSkelThreads, 0, st>>>(c->top.as<gpugrav_topnode>(), ntop, lib_top ? counters + kTopCount : nullptr,
                                    c->bconst.as<BuildConst>(), c->n_suns.as<int32_t>(), c->n_cl.as<double4>(),
                                    c->n_depth.as<uint8_t>(), c->n_father.as<int32_t>(), leafnode, nodetop, sinfo);
      launches++;
      GG_TRY(cudaMemcpyAsync(&io->skel, sinfo, sizeof(SkelInfo), cudaMemcpyDeviceToHost, st));
      k_topleaf<<<grid_for(n, 256), 256, 0, st>>>(c->top.as<gpugrav_topnode>(), leafnode, sinfo, n, c->s_ix.as<uint64_t>(),
                                                   c->s_iy.as<uint64_t>(), c->s_iz.as<uint64_t>(), c->s_tl.as<uint8_t>(),
                                                   c->s_tlnode.as<int32_t>());
      launches++;
    }
  k_pairdepth<<<grid_for(n, 256), 256, 0, st>>>(n, c->s_ix.as<uint64_t>(), c->s_iy.as<uint64_t>(), c->s_iz.as<uint64_t>(), msys,
                                                 c->s_cd.as<int8_t>());
  launches++;

  TreeArgs a;
  a.n      = n;
  a.ntop   = ntop;
  a.pm     = c->s_pm.as<double4>();
  a.ix     = c->s_ix.as<uint64_t>();
  a.iy     = c->s_iy.as<uint64_t>();
  a.iz     = c->s_iz.as<uint64_t>();
  a.st     = c->s_st.as<uint8_t>();
  a.cd     = c->s_cd.as<int8_t>();
  a.tl     = c->s_tl.as<uint8_t>();
  a.tlnode = c->s_tlnode.as<int32_t>();
  a.base   = c->base.as<int32_t>();
  a.dom    = &c->bconst.as<BuildConst>()->dom;
  a.sys    = msys;
  a.doms   = mdoms;
  a.nn     = 0;
  a.err    = counters + 12;

  c->mark("b1 roots+pairdepth");
  // 2. node counts per inserting particle, replayed cells
  GG_TRY(cudaMemsetAsync(counters, 0, 16 * sizeof(int), st));
  k_count<<<grid_for(n + 1, 256), 256, 0, st>>>(a, c->cnt.as<int32_t>(), c->hack_list.as<int32_t>(), counters);
  launches++;
  // numbering: exclusive scan of the per-particle node counts (again where cells are replayed below)
  auto number_nodes = [&]() -> cudaError_t {
    size_t tb = 0;
    GG_TRY(cub::DeviceScan::ExclusiveSum(nullptr, tb, c->cnt.as<int32_t>(), c->base.as<int32_t>(), (int)(n + 1), st));
    GG_TRY(c->sort_tmp.ensure(tb));
    GG_TRY(cub::DeviceScan::ExclusiveSum(c->sort_tmp.p, tb, c->cnt.as<int32_t>(), c->base.as<int32_t>(), (int)(n + 1), st));
    launches++;
    return cudaMemcpyAsync(&io->mdyn, c->base.as<int32_t>() + n, sizeof(int32_t), cudaMemcpyDeviceToHost, st);
  };
  GG_TRY(number_nodes());
  int *hc = io->counters;
  GG_TRY(cudaMemcpyAsync(hc, counters, kCounters * sizeof(int), cudaMemcpyDeviceToHost, st));
  GG_TRY(cudaStreamSynchronize(st));
  if(!c->multi)
    {
      if(lib_top)
        ntop = c->ntop = hc[kTopCount];
      if(ntop < 1 || io->skel.status < 0 || io->skel.ntop_nodes != ntop)
        {
          *status = GPUGRAV_ERR_TOPNODES;
          return cudaSuccess;
        }
      c->nleaves = io->skel.nleaves;
      a.ntop     = ntop;
    }
  if(c->multi && hc[kSortFlag])
    {
      *status = kNeedFullSort;  // the serving loop sorts the full keys and builds again
      return cudaSuccess;
    }
  const int nh  = hc[1];
  c->hack_cells = nh;
  HackCell *cells = nullptr;
  if(nh > 0)
    {
      GG_TRY(c->hcnt.ensure((size_t)nh * (sizeof(HackCell) + 2 * sizeof(int64_t)) + 64));
      cells            = (HackCell *)c->hcnt.p;
      int64_t *sizes   = (int64_t *)(cells + nh);
      int64_t *offsets = sizes + nh;
      k_hack_range<<<(nh + 127) / 128, 128, 0, st>>>(a, c->hack_list.as<int32_t>(), nh, cells, sizes);
      size_t tb = 0;
      GG_TRY(cub::DeviceScan::ExclusiveSum(nullptr, tb, sizes, offsets, nh, st));
      GG_TRY(c->sort_tmp.ensure(tb));
      GG_TRY(cub::DeviceScan::ExclusiveSum(c->sort_tmp.p, tb, sizes, offsets, nh, st));
      int64_t last[2];
      GG_TRY(cudaMemcpyAsync(&last[0], sizes + nh - 1, 8, cudaMemcpyDeviceToHost, st));
      GG_TRY(cudaMemcpyAsync(&last[1], offsets + nh - 1, 8, cudaMemcpyDeviceToHost, st));
      GG_TRY(cudaStreamSynchronize(st));
      int64_t pool = last[0] + last[1];
      GG_TRY(c->hack_scratch.ensure((size_t)pool * 8 * sizeof(int32_t) + 64));
      k_hack_count<<<(nh + 127) / 128, 128, 0, st>>>(a, cells, offsets, nh, c->hack_scratch.as<int32_t>(), c->cnt.as<int32_t>());
      launches += 2;
    }

  if(nh > 0)
    {
      GG_TRY(number_nodes());
      GG_TRY(cudaStreamSynchronize(st));
    }
  const int32_t mdyn = io->mdyn;
  c->mark("b2 count+scan");
  // 3. node storage
  const int64_t nn = (int64_t)ntop + mdyn;
  if(n + nn >= (int64_t)INT32_MAX)
    {
      *status = GPUGRAV_ERR_TREE_FULL;
      return cudaSuccess;
    }
  c->num_nodes = nn;
  c->n_entries = n + nn;
  a.nn         = nn;

  // grow node arrays, keeping the skeleton written by k_skeleton
  if((size_t)nn * 8 * sizeof(int32_t) > c->n_suns.cap || (size_t)nn * sizeof(double4) > c->n_cl.cap ||
     (size_t)nn + 16 > c->n_depth.cap || (size_t)nn * sizeof(int32_t) > c->n_father.cap)
    {
      // the skeleton is cheap: re-create after growth
      gg::DevBuf *bufs[] = {&c->n_suns, &c->n_depth, &c->n_cl, &c->n_sm, &c->n_maxsoft, &c->n_size,
                            &c->n_father, &c->n_count, &c->n_arrived};
      for(auto *b : bufs)
        b->release();
      GG_TRY(ensure_nodes(nn + 16));
      if(c->multi)
        k_roots<<<grid_for(ntop, 128), 128, 0, st>>>(ntop, mdoms, c->n_suns.as<int32_t>(), c->n_cl.as<double4>(),
                                                      c->n_depth.as<uint8_t>(), c->n_father.as<int32_t>());
      else
        k_skeleton<<<1, kSkelThreads, 0, st>>>(c->top.as<gpugrav_topnode>(), ntop, nullptr, c->bconst.as<BuildConst>(),
                                      c->n_suns.as<int32_t>(), c->n_cl.as<double4>(), c->n_depth.as<uint8_t>(),
                                      c->n_father.as<int32_t>(), leafnode, nodetop, sinfo);
      launches++;
    }

  c->mark("b3b grow");
  // 4. fill canonical nodes, link, place particles, replay coincident cells
  k_nodes<<<grid_for(n, 256), 256, 0, st>>>(a, c->n_suns.as<int32_t>(), c->n_cl.as<double4>(), c->n_depth.as<uint8_t>());
  k_link_nodes<<<grid_for(n, 256), 256, 0, st>>>(a, c->n_suns.as<int32_t>(), c->n_father.as<int32_t>());
  k_leaves<<<grid_for(n, 256), 256, 0, st>>>(a, c->n_suns.as<int32_t>());
  launches += 3;
  if(nh > 0)
    {
      k_hack_fill<<<(nh + 127) / 128, 128, 0, st>>>(a, cells, nh, c->n_suns.as<int32_t>(), c->n_cl.as<double4>(),
                                                     c->n_depth.as<uint8_t>(), c->n_father.as<int32_t>());
      launches++;
    }
  GG_TRY(cudaGetLastError());

  c->mark("b4 nodes+link+leaves");
  // 5. moments bottom-up (with MULTIPLE_NODE_SOFTENING also the per-type masses)
  const bool mns = (c->prm.flags & GPUGRAV_FLAG_MULTIPLE_NODE_SOFTENING) != 0;
  if(mns)
    GG_TRY(c->n_mpt.ensure((size_t)(nn + 16) * c->prm.nsofttypes * sizeof(double)));
  k_children<<<grid_for(nn, 256), 256, 0, st>>>(nn, (int32_t)n, c->n_suns.as<int32_t>(), c->n_depth.as<uint8_t>(),
                                                 c->n_count.as<uint8_t>(), c->n_arrived.as<int32_t>(), counters + 4);
  auto moments = mns ? k_moments<true> : k_moments<false>;
  moments<<<(unsigned)((nn + 127) / 128), 128, 0, st>>>(nn, (int32_t)n, c->n_suns.as<int32_t>(), c->n_count.as<uint8_t>(),
                                                        c->n_arrived.as<int32_t>(), c->n_father.as<int32_t>(), c->s_pm.as<double4>(),
                                                        c->s_st.as<uint8_t>(), c->n_cl.as<double4>(), c->n_sm.as<double4>(),
                                                        c->n_maxsoft.as<uint8_t>(), c->n_size.as<int32_t>(),
                                                        c->bconst.as<BuildConst>(), mns ? c->n_mpt.as<double>() : nullptr, a.err);
  launches += 2;
  c->mark("b5 moments");
  // 6. threading and the layout of the FP64 walk; the group walk needs neither (several systems are
  // walked by the group walk only)
  c->threaded  = false;
  c->built_mns = mns;
  if(!c->multi && c->prm.precision == GPUGRAV_PREC_FP64)
    {
      GG_TRY(thread_stage(c));
      launches += 3;
    }
  c->mark("b6 threading+layout64");
  c->timings.build_kernel_launches = launches;
  GG_TRY(cudaGetLastError());
  cudaEventRecord(c->ev[6], st);
  // counters[4]: deepest level, [12]: self-check flags
  GG_TRY(cudaMemcpyAsync(io->counters, counters, kCounters * sizeof(int), cudaMemcpyDeviceToHost, st));
  GG_TRY(cudaStreamSynchronize(st));
  c->max_depth  = io->counters[4];
  const int err = io->counters[12];
  if(err)
    {
      c->err  = "tree build self-check failed (flags " + std::to_string(err) + ")";
      *status = GPUGRAV_ERR_TREE_FULL;
    }
  return cudaSuccess;
}
}  // namespace gg
