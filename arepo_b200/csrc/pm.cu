// pm.cu -- periodic particle-mesh long-range force on the GPU.
//
// Replaces pmforce_periodic(0, NULL) (src/gravity/pm/pm_periodic.c:1572-1936, the uniform data
// path of pmforce_uniform_optimized_prepare_density / _readout_forces_or_potential, :720-1538):
//   1. CIC mass assignment onto a PMGRID^3 mesh (node-based: cell (int)(PMGRID/L x), weights
//      1-dx and dx, periodic, :1090-1165), FP64 atomics;
//   2. real-to-complex FFT (cuFFT, FP64);
//   3. Green's function -exp(-k^2 Asmth^2) / k^2 times the CIC deconvolution
//      (sin(k d/2) / (k d/2))^-4 per axis, zero mode cleared (:1620-1704); both factors separate
//      into per-axis tables;
//   4. complex-to-real FFT: the potential mesh (unnormalised, as the FFTW backward transform);
//   5. the force mesh: the 4-point finite differences of the potential,
//      fac ((4/3)(phi[-1] - phi[+1]) - (1/6)(phi[-2] - phi[+2])), fac = 4 pi G / L^3 / (2 d)
//      (:1735-1800), the three components and the potential side by side, read at the 8 CIC nodes of
//      every particle and CIC-weighted (:1322-1538), the potential with 4 pi G / L^3; for large sets
//      in brick order both in one pass, without that mesh.
// G = 1 (accelerations without the factor G, like the tree walk).  The mesh is FP64 (the reference's
// default fft_real is float; FP64 costs little here next to the tree walk).

#include <cub/cub.cuh>
#include <cufft.h>

#include <cmath>
#include <vector>

#include "internal.h"

namespace gg
{
namespace
{
// (int)(f x) and its offset as in the reference; cells wrapped into the mesh.  A position that is
// not finite or absurdly far outside the box sets *bad and is placed at cell 0 with weight 0, so
// that no index ever leaves the mesh.
__device__ __forceinline__ void cic_axis(double x, double f, int n, int &c0, int &c1, double &w, int *bad)
{
  const double xs = f * x;
  if(!(xs > -1.0e15 && xs < 1.0e15))
    {
      atomicOr(bad, 1);
      c0 = 0;
      c1 = 1 % n;
      w  = 0.0;
      return;
    }
  const double s = floor(xs);  // positions in [0, L): the reference's (int) truncation
  w              = xs - s;
  int c          = (int)(s - (double)n * floor(s / n));  // in [0, n)
  c              = c < 0 ? 0 : (c >= n ? n - 1 : c);
  c0             = c;
  c1             = c0 + 1 == n ? 0 : c0 + 1;
}

// ---- particle order ----
// Particles come in the caller's order; on a mesh larger than L2 the eight nodes of a particle are then
// fetched from memory one sector at a time.  For large sets the particles are first brought into the order
// of bricks of 16^3 cells (a sort of 15 bits at 512^3), so that those running together share the mesh's
// lines; results are written in that order and read back by the caller's.  With 2^24 particles on 512^3 the
// call went from 9.36 to 7.63 ms for a zoom box and from 11.3 to 7.6 ms for an even set.  The sort and the
// two permutations cost 80 us per 2^20 particles: on meshes that fit in L2, or with few particles per brick, the
// caller's order stays.  Caller's / brick order (ms), zoom box and even set: 256^3 with 2^22 particles 1.64 / 1.90 and
// 1.66 / 1.28, 2^23 2.6 either way for the zoom box; 512^3 with 2^20 5.43 / 5.59 and 5.57 / 5.08, 2^21 5.69 / 5.47 and
// 5.93 / 5.05, 2^22 6.20 / 5.68 and 6.70 / 5.34.  The line below is 256^3's; on larger meshes it could lie at 2^21.
constexpr int kBrick             = 4;    // log2 of a brick's side in cells
constexpr int kSortMesh          = 256;  // from 128 MB of potential, which is the L2's size
constexpr int64_t kSortParticles = 1 << 23;
__global__ void k_pm_brick(int64_t np, const double *__restrict__ pos, int n, double f, int nb, uint32_t *__restrict__ key,
                           uint32_t *__restrict__ idx, int *bad)
{
  for(int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < np; i += (int64_t)gridDim.x * blockDim.x)
    {
      int c[3], c1;
      double w;
#pragma unroll
      for(int a = 0; a < 3; a++)
        cic_axis(pos[3 * i + a], f, n, c[a], c1, w, bad);
      key[i] = (uint32_t)(((c[0] >> kBrick) * nb + (c[1] >> kBrick)) * nb + (c[2] >> kBrick));
      idx[i] = (uint32_t)i;
    }
}
// the inverse order, and where every brick's particles begin (key: sorted)
__global__ void k_pm_starts(int64_t np, const uint32_t *__restrict__ key, const uint32_t *__restrict__ perm, int bricks,
                            uint32_t *__restrict__ iperm, uint32_t *__restrict__ start)
{
  for(int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i <= np; i += (int64_t)gridDim.x * blockDim.x)
    {
      const int64_t from = i > 0 ? (int64_t)key[i - 1] + 1 : 0, to = i < np ? (int64_t)key[i] : bricks;
      for(int64_t k = from; k <= to; k++)
        start[k] = (uint32_t)i;
      if(i < np)
        iperm[perm[i]] = (uint32_t)i;
    }
}
// particles into brick order: read in order and written a whole 32-byte sector each (the other way round,
// three sectors fetched per particle, took 1.03 ms for 2^24 particles)
__global__ void k_pm_scatter(int64_t np, const uint32_t *__restrict__ iperm, const double *__restrict__ pos, const double *__restrict__ mass,
                             double4 *__restrict__ pm)
{
  for(int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; o < np; o += (int64_t)gridDim.x * blockDim.x)
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(pm + iperm[o]), "d"(pos[3 * o]), "d"(pos[3 * o + 1]), "d"(pos[3 * o + 2]),
                 "d"(mass[o])
                 : "memory");
}
// SORTED: positions and masses in brick order (pm), else the caller's arrays
template <bool SORTED>
__global__ void k_pm_deposit(int64_t np, const double *__restrict__ pos, const double *__restrict__ mass, const double4 *__restrict__ pm, int n,
                             double f, double *__restrict__ rho, int *bad)
{
  for(int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < np; i += (int64_t)gridDim.x * blockDim.x)
    {
      int x0, x1, y0, y1, z0, z1;
      double dx, dy, dz;
      const double4 p = SORTED ? pm[i] : make_double4(pos[3 * i + 0], pos[3 * i + 1], pos[3 * i + 2], mass[i]);
      cic_axis(p.x, f, n, x0, x1, dx, bad);
      cic_axis(p.y, f, n, y0, y1, dy, bad);
      cic_axis(p.z, f, n, z0, z1, dz, bad);
      const double m = p.w;
      const int64_t N = n;
      atomicAdd(&rho[(x0 * N + y0) * N + z0], m * (1.0 - dx) * (1.0 - dy) * (1.0 - dz));
      atomicAdd(&rho[(x0 * N + y0) * N + z1], m * (1.0 - dx) * (1.0 - dy) * dz);
      atomicAdd(&rho[(x0 * N + y1) * N + z0], m * (1.0 - dx) * dy * (1.0 - dz));
      atomicAdd(&rho[(x0 * N + y1) * N + z1], m * (1.0 - dx) * dy * dz);
      atomicAdd(&rho[(x1 * N + y0) * N + z0], m * dx * (1.0 - dy) * (1.0 - dz));
      atomicAdd(&rho[(x1 * N + y0) * N + z1], m * dx * (1.0 - dy) * dz);
      atomicAdd(&rho[(x1 * N + y1) * N + z0], m * dx * dy * (1.0 - dz));
      atomicAdd(&rho[(x1 * N + y1) * N + z1], m * dx * dy * dz);
    }
}


// mesh of the forward transform: n x n x (n/2 + 1), last index fastest.  The Gaussian and the CIC
// deconvolution factor per axis: tab[i] = (exp(-k_i^2 Asmth^2), 1 / sinc(k_i d / 2)^4) for the wave
// number k_i of mesh index i, so that an entry costs one product and one division.
__global__ void k_pm_green(int n, double kfac, const double2 *__restrict__ tab, cufftDoubleComplex *__restrict__ rk)
{
  const int nz      = n / 2 + 1;
  const int64_t tot = (int64_t)n * n * nz;
  for(int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < tot; i += (int64_t)gridDim.x * blockDim.x)
    {
      const int z = (int)(i % nz);
      const int y = (int)((i / nz) % n);
      const int x = (int)(i / ((int64_t)nz * n));
      const int xx = x >= n / 2 ? x - n : x, yy = y >= n / 2 ? y - n : y, zz = z >= n / 2 ? z - n : z;
      const double kx = kfac * xx, ky = kfac * yy, kz = kfac * zz;
      const double k2 = kx * kx + ky * ky + kz * kz;
      double g        = 0.0;  // the zero mode carries the mean density: no force
      if(k2 > 0)
        {
          const double2 a = tab[x], b = tab[y], c = tab[z];
          g               = -(a.x * b.x * c.x) * (a.y * b.y * c.y) / k2;
        }
      rk[i].x *= g;
      rk[i].y *= g;
    }
}

// one component of the force mesh: the 4-point difference of the potential along `dim`.  One block
// per mesh row (x, y), threads along z: coordinates without a per-point division, coalesced rows.
__global__ void k_pm_fd(int n, int dim, double fac, const double *__restrict__ phi, double *__restrict__ force)
{
  const int64_t N = n;
  auto wrap       = [n](int q) { return q < 0 ? q + n : (q >= n ? q - n : q); };
  for(int64_t row = blockIdx.x; row < N * N; row += gridDim.x)
    {
      const int x = (int)(row / N), y = (int)(row % N);
      const double *r0 = phi + row * N;
      // the rows (dim 0: x +- 1, 2; dim 1: y +- 1, 2) or this row (dim 2) holding the four neighbours
      const double *rm1 = r0, *rp1 = r0, *rm2 = r0, *rp2 = r0;
      if(dim == 0)
        {
          rm1 = phi + (wrap(x - 1) * N + y) * N;
          rp1 = phi + (wrap(x + 1) * N + y) * N;
          rm2 = phi + (wrap(x - 2) * N + y) * N;
          rp2 = phi + (wrap(x + 2) * N + y) * N;
        }
      else if(dim == 1)
        {
          rm1 = phi + (x * N + wrap(y - 1)) * N;
          rp1 = phi + (x * N + wrap(y + 1)) * N;
          rm2 = phi + (x * N + wrap(y - 2)) * N;
          rp2 = phi + (x * N + wrap(y + 2)) * N;
        }
      for(int z = threadIdx.x; z < n; z += blockDim.x)
        {
          const int zm1 = dim == 2 ? wrap(z - 1) : z, zp1 = dim == 2 ? wrap(z + 1) : z;
          const int zm2 = dim == 2 ? wrap(z - 2) : z, zp2 = dim == 2 ? wrap(z + 2) : z;
          force[row * N + z] = fac * ((4.0 / 3) * (rm1[zm1] - rp1[zp1]) - (1.0 / 6) * (rm2[zm2] - rp2[zp2]));
        }
    }
}

// CIC readout of one mesh at every particle: out[ostride * i + ooff] = scale * sum_nodes w mesh
__global__ void k_pm_cic_read(int64_t np, const double *__restrict__ pos, int n, double f, const double *__restrict__ mesh,
                              double scale, double *__restrict__ out, int ostride, int ooff, int *bad)
{
  const int64_t N = n;
  for(int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < np; i += (int64_t)gridDim.x * blockDim.x)
    {
      int c[3][2];
      double w[3][2];
      for(int a = 0; a < 3; a++)
        {
          double d;
          cic_axis(pos[3 * i + a], f, n, c[a][0], c[a][1], d, bad);
          w[a][0] = 1.0 - d;
          w[a][1] = d;
        }
      double v = 0;
      for(int ix = 0; ix < 2; ix++)
        for(int iy = 0; iy < 2; iy++)
          for(int iz = 0; iz < 2; iz++)
            v += mesh[(c[0][ix] * N + c[1][iy]) * N + c[2][iz]] * (w[0][ix] * w[1][iy] * w[2][iz]);
      out[ostride * i + ooff] = v * scale;
    }
}

// The three force components and the potential of every mesh point in one 32-byte record, so that a
// particle's read of a node is one sector: 8 per particle instead of 8 per component.  One pass over the
// mesh, a block per mesh row as in k_pm_fd.  At 2^24 particles and 512^3 points the three differences and
// four reads took 5.55 ms together.
__global__ void k_pm_fd4(int n, double fac, const double *__restrict__ phi, double4 *__restrict__ force)
{
  const int64_t N = n;
  auto wrap       = [n](int q) { return q < 0 ? q + n : (q >= n ? q - n : q); };
  for(int64_t row = blockIdx.x; row < N * N; row += gridDim.x)
    {
      const int x = (int)(row / N), y = (int)(row % N);
      const double *r0  = phi + row * N;
      const double *xm1 = phi + (wrap(x - 1) * N + y) * N, *xp1 = phi + (wrap(x + 1) * N + y) * N,
                   *xm2 = phi + (wrap(x - 2) * N + y) * N, *xp2 = phi + (wrap(x + 2) * N + y) * N;
      const double *ym1 = phi + (x * N + wrap(y - 1)) * N, *yp1 = phi + (x * N + wrap(y + 1)) * N,
                   *ym2 = phi + (x * N + wrap(y - 2)) * N, *yp2 = phi + (x * N + wrap(y + 2)) * N;
      for(int z = threadIdx.x; z < n; z += blockDim.x)
        {
          const int zm1 = wrap(z - 1), zp1 = wrap(z + 1), zm2 = wrap(z - 2), zp2 = wrap(z + 2);
          double4 f;
          f.x = fac * ((4.0 / 3) * (xm1[z] - xp1[z]) - (1.0 / 6) * (xm2[z] - xp2[z]));
          f.y = fac * ((4.0 / 3) * (ym1[z] - yp1[z]) - (1.0 / 6) * (ym2[z] - yp2[z]));
          f.z = fac * ((4.0 / 3) * (r0[zm1] - r0[zp1]) - (1.0 / 6) * (r0[zm2] - r0[zp2]));
          f.w = r0[z];
          asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(force + row * N + z), "d"(f.x), "d"(f.y), "d"(f.z), "d"(f.w)
                       : "memory");
        }
    }
}

// Call (ms) with the records / component by component on 512^3: 1000 and 2^16 particles 5.20 / 5.07, 2^20 of a zoom
// box 5.46 / 5.45, of an even set 5.59 / 5.71, 2^22 6.25 / 6.57 and 6.75 / 7.50; on 384^3 and smaller meshes the records
// are never behind (1000 particles 3.00 / 3.01, on 256^3 0.69 / 0.77).
constexpr int kFewMesh  = 384;
constexpr int kFewShare = 128;  // few: less than one particle to so many mesh points

// CIC readout of the records: accelerations and (pot not null) potentials scaled by `scale`
__global__ void __launch_bounds__(256) k_pm_read4(int64_t np, const double *__restrict__ pos, int n, double f, const double4 *__restrict__ mesh,
                                                  double scale, double *__restrict__ acc, double *__restrict__ pot, int *bad)
{
  const int64_t N = n;
  for(int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < np; i += (int64_t)gridDim.x * blockDim.x)
    {
      int c[3][2];
      double w[3][2];
#pragma unroll
      for(int a = 0; a < 3; a++)
        {
          double d;
          cic_axis(pos[3 * i + a], f, n, c[a][0], c[a][1], d, bad);
          w[a][0] = 1.0 - d;
          w[a][1] = d;
        }
      double4 m[8];
#pragma unroll
      for(int q = 0; q < 8; q++)
        asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
            : "=d"(m[q].x), "=d"(m[q].y), "=d"(m[q].z), "=d"(m[q].w)
            : "l"(mesh + (c[0][q >> 2] * N + c[1][q >> 1 & 1]) * N + c[2][q & 1]));
      double4 v = make_double4(0, 0, 0, 0);
#pragma unroll
      for(int q = 0; q < 8; q++)
        {
          const double g = w[0][q >> 2] * w[1][q >> 1 & 1] * w[2][q & 1];
          v.x += m[q].x * g;
          v.y += m[q].y * g;
          v.z += m[q].z * g;
          v.w += m[q].w * g;
        }
      acc[3 * i + 0] = v.x;
      acc[3 * i + 1] = v.y;
      acc[3 * i + 2] = v.z;
      if(pot)
        pot[i] = v.w * scale;
    }
}

// Finite differences and CIC readout in one pass for particles in brick order: a block takes kReadChunk of
// them, lays the potential of one brick after the other with its halo (2 cells below, 3 above) into shared
// memory and forms the 8 nodes' differences there from 56 values per particle.  The mesh of records (32
// bytes a point, written once and read eight times per particle) took 2.6 ms of 9.1 at 512^3 with 2^24
// particles; this pass only reads the potential.  Bound by shared memory: 56 scattered 8-byte reads per
// particle and 74 KB loaded per brick.  Chunks of a fixed number of particles and not of bricks, so that a
// dense brick is shared by many blocks.
constexpr int kTile      = (1 << kBrick) + 5;
constexpr int kReadChunk = 2048;
__global__ void __launch_bounds__(256) k_pm_read_brick(int64_t np, const double4 *__restrict__ pm, const uint32_t *__restrict__ start, int n,
                                                       int nb, double f, const double *__restrict__ phi, double fac, double scale,
                                                       double4 *__restrict__ res, int *bad)
{
  extern __shared__ double tile[];  // kTile^3
  const int64_t N  = n;
  const int64_t c0 = blockIdx.x * (int64_t)kReadChunk, c1 = c0 + kReadChunk < np ? c0 + kReadChunk : np;
  for(int64_t i0 = c0; i0 < c1;)
    {
      int o[3], up;
      double w;
      const double4 first = pm[i0];
      cic_axis(first.x, f, n, o[0], up, w, bad);
      cic_axis(first.y, f, n, o[1], up, w, bad);
      cic_axis(first.z, f, n, o[2], up, w, bad);
#pragma unroll
      for(int a = 0; a < 3; a++)
        o[a] >>= kBrick;
      const int64_t last = start[(o[0] * nb + o[1]) * nb + o[2] + 1], i1 = last < c1 ? last : c1;
#pragma unroll
      for(int a = 0; a < 3; a++)
        o[a] = (o[a] << kBrick) - 2;
      __syncthreads();
#pragma unroll 6
      for(int t = threadIdx.x; t < kTile * kTile * kTile; t += 256)
        {
          int x = o[0] + t / (kTile * kTile), y = o[1] + t / kTile % kTile, z = o[2] + t % kTile;
          x       = x < 0 ? x + n : (x >= n ? x - n : x);
          y       = y < 0 ? y + n : (y >= n ? y - n : y);
          z       = z < 0 ? z + n : (z >= n ? z - n : z);
          tile[t] = phi[(x * N + y) * N + z];
        }
      __syncthreads();
      for(int64_t i = i0 + threadIdx.x; i < i1; i += 256)
        {
          const double4 p = pm[i];
          int c[3];
          double g[3][2];
          cic_axis(p.x, f, n, c[0], up, g[0][1], bad);
          cic_axis(p.y, f, n, c[1], up, g[1][1], bad);
          cic_axis(p.z, f, n, c[2], up, g[2][1], bad);
#pragma unroll
          for(int a = 0; a < 3; a++)
            g[a][0] = 1.0 - g[a][1];
          const double *t = tile + ((c[0] - o[0]) * kTile + c[1] - o[1]) * kTile + c[2] - o[2];
          double v[2][2][2];
          double4 r = make_double4(0, 0, 0, 0);
#pragma unroll
          for(int q = 0; q < 8; q++)
            {
              v[q >> 2][q >> 1 & 1][q & 1] = t[(q >> 2) * kTile * kTile + (q >> 1 & 1) * kTile + (q & 1)];
              r.w += v[q >> 2][q >> 1 & 1][q & 1] * (g[0][q >> 2] * g[1][q >> 1 & 1] * g[2][q & 1]);
            }
          // the difference at the lower and the upper node of a line m2 m1 lo up p2 p3, weighted
          auto line = [](const double *b, int st, double lo, double hi, double wl, double wh) {
            const double m2 = b[-2 * st], m1 = b[-st], p2 = b[2 * st], p3 = b[3 * st];
            return wl * ((4.0 / 3) * (m1 - hi) - (1.0 / 6) * (m2 - p2)) + wh * ((4.0 / 3) * (lo - p2) - (1.0 / 6) * (m1 - p3));
          };
#pragma unroll
          for(int q = 0; q < 4; q++)
            {
              const int a = q >> 1, b = q & 1;
              r.x += g[1][a] * g[2][b] * line(t + a * kTile + b, kTile * kTile, v[0][a][b], v[1][a][b], g[0][0], g[0][1]);
              r.y += g[0][a] * g[2][b] * line(t + a * kTile * kTile + b, kTile, v[a][0][b], v[a][1][b], g[1][0], g[1][1]);
              r.z += g[0][a] * g[1][b] * line(t + a * kTile * kTile + b * kTile, 1, v[a][b][0], v[a][b][1], g[2][0], g[2][1]);
            }
          res[i] = make_double4(fac * r.x, fac * r.y, fac * r.z, scale * r.w);
        }
      i0 = i1;
    }
}

int blocks_for(int64_t n)
{
  int64_t b = (n + 255) / 256;
  return (int)(b < 1 ? 1 : (b > 148 * 32 ? 148 * 32 : b));
}
}  // namespace

// PM force for np particles (device arrays pos n*3, mass n) into acc (n*3) and pot (n, may be null)
cudaError_t pm_stage(gpugrav_ctx *c, int pmgrid, int64_t np, const double *pos, const double *mass, double *acc, double *pot,
                     int *cufft_status)
{
  cudaStream_t st  = c->stream;
  const int n      = pmgrid;
  const int64_t N3 = (int64_t)n * n * n, NC = (int64_t)n * n * (n / 2 + 1);
  *cufft_status    = CUFFT_SUCCESS;
  if(c->pm_grid != n)
    {
      if(c->pm_grid > 0)
        {
          cufftDestroy((cufftHandle)c->pm_plan_f);
          cufftDestroy((cufftHandle)c->pm_plan_b);
          c->pm_grid = 0;
        }
      cufftHandle pf, pb;
      cufftResult r = cufftPlan3d(&pf, n, n, n, CUFFT_D2Z);
      if(r != CUFFT_SUCCESS)
        {
          *cufft_status = r;
          return cudaSuccess;
        }
      r = cufftPlan3d(&pb, n, n, n, CUFFT_Z2D);
      if(r != CUFFT_SUCCESS)
        {
          cufftDestroy(pf);
          *cufft_status = r;
          return cudaSuccess;
        }
      c->pm_plan_f = (int)pf;
      c->pm_plan_b = (int)pb;
      c->pm_grid   = n;
    }
  GG_TRY(c->pm_rho.ensure(N3 * sizeof(double)));
  GG_TRY(c->pm_rhok.ensure(NC * sizeof(cufftDoubleComplex)));
  if(c->pm_tab_n != n || c->pm_tab_box != c->prm.box_size || c->pm_tab_asmth != c->prm.asmth)
  {
    // per-axis factors of the Green's function (host, n entries), kept while mesh, box and Asmth stay
    const double bx = c->prm.box_size, dd = bx / n, kf = 2.0 * M_PI / bx, a2 = c->prm.asmth * c->prm.asmth;
    std::vector<double2> tab(n);
    for(int i = 0; i < n; i++)
      {
        const int ii   = i >= n / 2 ? i - n : i;
        const double k = kf * ii;
        double s       = 1.0;
        if(ii != 0)
          {
            const double a = k * 0.5 * dd;
            s              = sin(a) / a;
          }
        const double f = 1.0 / s;
        tab[i]         = make_double2(exp(-k * k * a2), f * f * f * f);
      }
    GG_TRY(c->pm_tab.ensure(n * sizeof(double2)));
    GG_TRY(cudaMemcpyAsync(c->pm_tab.p, tab.data(), n * sizeof(double2), cudaMemcpyHostToDevice, st));
    GG_TRY(cudaStreamSynchronize(st));  // `tab` lives on this stack frame
    c->pm_tab_n     = n;
    c->pm_tab_box   = bx;
    c->pm_tab_asmth = c->prm.asmth;
  }
  cufftSetStream((cufftHandle)c->pm_plan_f, st);
  cufftSetStream((cufftHandle)c->pm_plan_b, st);
  const double box = c->prm.box_size, d = box / n, f = n / box;
  GG_TRY(cudaMemsetAsync(c->pm_rho.p, 0, N3 * sizeof(double), st));
  int *bad = c->counters.as<int>() + 15;
  GG_TRY(cudaMemsetAsync(bad, 0, sizeof(int), st));
  // brick order for large sets on large meshes (kSortMesh); without room for it the caller's order
  const int nb = (n + (1 << kBrick) - 1) >> kBrick;
  bool sorted  = n >= kSortMesh && np >= kSortParticles && np < (int64_t)1 << 31;
  double4 *s_pm = nullptr, *s_res = nullptr;
  uint32_t *iperm = nullptr, *start = nullptr;
  if(sorted)
    {
      int bits = 1;
      while((1 << bits) < nb * nb * nb)
        bits++;
      size_t tb = 0;
      GG_TRY(cub::DeviceRadixSort::SortPairs(nullptr, tb, (uint32_t *)nullptr, (uint32_t *)nullptr, (uint32_t *)nullptr, (uint32_t *)nullptr,
                                             (int)np, 0, bits, st));
      // particles | (keys, places: before and after the sort; later the results) | inverse order | starts | sort space
      const int bricks  = nb * nb * nb;
      const size_t need = (size_t)np * (32 + 32 + 4) + (size_t)(bricks + 1) * 4 + 1024 + tb;
      size_t free_b = 0, total_b = 0;
      sorted = c->pm_sort.cap >= need || (cudaMemGetInfo(&free_b, &total_b) == cudaSuccess && need <= free_b / 4 &&
                                          c->pm_sort.ensure(need) == cudaSuccess);
      if(!sorted)
        cudaGetLastError();
      else
        {
          char *q = c->pm_sort.as<char>();
          auto at = [&](size_t b) { char *r = q; q += (b + 255) & ~(size_t)255; return r; };
          s_pm  = (double4 *)at(np * 32);
          s_res = (double4 *)at(np * 32);
          iperm = (uint32_t *)at(np * 4);
          start = (uint32_t *)at((size_t)(bricks + 1) * 4);
          uint32_t *key = (uint32_t *)s_res, *key2 = key + np, *idx = key2 + np, *perm = idx + np;
          k_pm_brick<<<blocks_for(np), 256, 0, st>>>(np, pos, n, f, nb, key, idx, bad);
          GG_TRY(cub::DeviceRadixSort::SortPairs(q, tb, key, key2, idx, perm, (int)np, 0, bits, st));
          k_pm_starts<<<blocks_for(np + 1), 256, 0, st>>>(np, key2, perm, bricks, iperm, start);
          k_pm_scatter<<<blocks_for(np), 256, 0, st>>>(np, iperm, pos, mass, s_pm);
        }
    }
  if(sorted)
    k_pm_deposit<true><<<blocks_for(np), 256, 0, st>>>(np, nullptr, nullptr, s_pm, n, f, c->pm_rho.as<double>(), bad);
  else
    k_pm_deposit<false><<<blocks_for(np), 256, 0, st>>>(np, pos, mass, nullptr, n, f, c->pm_rho.as<double>(), bad);
  GG_TRY(cudaGetLastError());
  cufftResult r = cufftExecD2Z((cufftHandle)c->pm_plan_f, c->pm_rho.as<double>(), c->pm_rhok.as<cufftDoubleComplex>());
  if(r == CUFFT_SUCCESS)
    {
      k_pm_green<<<blocks_for(NC), 256, 0, st>>>(n, 2.0 * M_PI / box, c->pm_tab.as<double2>(),
                                                  c->pm_rhok.as<cufftDoubleComplex>());
      GG_TRY(cudaGetLastError());
      r = cufftExecZ2D((cufftHandle)c->pm_plan_b, c->pm_rhok.as<cufftDoubleComplex>(), c->pm_rho.as<double>());
    }
  if(r != CUFFT_SUCCESS)
    {
      *cufft_status = r;
      return cudaSuccess;
    }
  const double fac_pot = 4.0 * M_PI / (box * box * box);
  const int64_t rows   = (int64_t)n * n;
  if(sorted)
    {
      const int smem = kTile * kTile * kTile * (int)sizeof(double);
      GG_TRY(cudaFuncSetAttribute(k_pm_read_brick, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      k_pm_read_brick<<<(int)((np + kReadChunk - 1) / kReadChunk), 256, smem, st>>>(np, s_pm, start, n, nb, f, c->pm_rho.as<double>(),
                                                                                    fac_pot / (2.0 * d), fac_pot, s_res, bad);
      return results_out(st, np, s_res, nullptr, iperm, acc, pot, nullptr);
    }
  // The records take 32 bytes per mesh point, written once.  Few particles on a large mesh (kFewMesh, kFewShare) do
  // not pay for that, and where the records would take more than a quarter of the device's free memory there is
  // no room: then one component after the other in the complex buffer, which is free after the inverse transform.
  const bool few = n > kFewMesh && np * kFewShare < N3;
  bool records   = !few && c->pm_force.cap >= N3 * sizeof(double4);
  if(!few && !records)
    {
      size_t free_b = 0, total_b = 0;
      records = cudaMemGetInfo(&free_b, &total_b) == cudaSuccess && N3 * sizeof(double4) <= free_b / 4 &&
                c->pm_force.ensure(N3 * sizeof(double4)) == cudaSuccess;
      if(!records)
        cudaGetLastError();
    }
  if(records)
    {
      k_pm_fd4<<<(int)(rows < 148 * 16 ? rows : 148 * 16), 256, 0, st>>>(n, fac_pot / (2.0 * d), c->pm_rho.as<double>(),
                                                                           c->pm_force.as<double4>());
      k_pm_read4<<<blocks_for(np), 256, 0, st>>>(np, pos, n, f, c->pm_force.as<double4>(), fac_pot, acc, pot, bad);
      return cudaGetLastError();
    }
  double *force = (double *)c->pm_rhok.p;  // n^2 (n/2+1) complex >= n^3 doubles
  for(int dim = 0; dim < 3; dim++)
    {
      k_pm_fd<<<(int)(rows < 148 * 16 ? rows : 148 * 16), 256, 0, st>>>(n, dim, fac_pot / (2.0 * d), c->pm_rho.as<double>(),
                                                                          force);
      k_pm_cic_read<<<blocks_for(np), 256, 0, st>>>(np, pos, n, f, force, 1.0, acc, 3, dim, bad);
    }
  if(pot)
    k_pm_cic_read<<<blocks_for(np), 256, 0, st>>>(np, pos, n, f, c->pm_rho.as<double>(), fac_pot, pot, 1, 0, bad);
  return cudaGetLastError();
}

void pm_release(gpugrav_ctx *c)
{
  if(c->pm_grid > 0)
    {
      cufftDestroy((cufftHandle)c->pm_plan_f);
      cufftDestroy((cufftHandle)c->pm_plan_b);
      c->pm_grid = 0;
    }
  c->pm_rho.release();
  c->pm_rhok.release();
  c->pm_tab.release();
  spare_take(&c->pm_force);
  spare_take(&c->pm_sort);
  c->pm_force.release();
  c->pm_sort.release();
  c->pm_tab_n = 0;
}
}  // namespace gg
