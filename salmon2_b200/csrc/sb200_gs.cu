// sb200_gs.cu -- ground state on real orbitals (one k-point): real hpsi
// (dstencil + dpseudo), the band-by-band preconditioned CG eigensolver of
// gscg_rwf, classical Gram-Schmidt and the subspace diagonalisation, all on
// the device.  Orbitals use the resident layout psi[o][z][y][x] (double),
// o = ispin + nspin*io, with the context's grid, V_local and projector tables.
//
// Every reduction is deterministic: per-CTA partial sums in a fixed order,
// then a fixed-order sum of the partials by the consumer.
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <vector>

#include "sb200_gs.cuh"
#include "sb200_internal.cuh"

namespace sb200 {
namespace {

constexpr int RT = 256;            // threads of the reduction kernels
constexpr int DOT_PTS = RT * 8;    // points per reduction CTA

// ---------------------------------------------------------------------------
// real hpsi: 25-point Laplacian + V_local (stencil.f90:30-80) and the KB term
// (nonlocal_potential.f90:26-171; tables from the complex path: pmap entries
// carry uV)
// ---------------------------------------------------------------------------
struct RArgs {
  int nx, ny, nz, periodic, nspin, nlma, natom, nps, totpts, hz;
  long npts;
  double lap0, lapt[12];
  const double* vloc;
  const int *pmap, *ent_lma;
  const double* ent_uv;
  int pairs;           // 1: the (point, atom) pair form applies
  const int *pmap2, *pair_lma;
  const double* pair_uv;
  const double* proj;  // [norb][nlma]
  const int *atom_start, *mps, *lma_start, *nproj, *pt_lin;
  const double *uv, *rinv;
};

__device__ __forceinline__ int wrap(int q, int n, int periodic, bool& ok) {
  if (periodic) {
    q = q < 0 ? q + n : (q >= n ? q - n : q);
    ok = true;
  } else {
    ok = (q >= 0) && (q < n);
  }
  return q;
}

// Block-wide sums of NV values per thread (NT threads); every thread gets the
// totals (fixed order: butterfly in the warp, then the warps in order).
template <int NV, int NT>
__device__ __forceinline__ void block_totals(double (&v)[NV], double (*red)[NT / 32]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < NV; ++i)
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], off);
  __syncthreads();
  if (lane == 0)
    for (int i = 0; i < NV; ++i) red[i][warp] = v[i];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    v[i] = red[i][0];
    for (int w = 1; w < NT / 32; ++w) v[i] += red[i][w];
  }
}

// Sum over the blocks of one orbital's partial sums part[n][NV], by every block
// that needs it (no launch of its own for a scalar).
template <int NV>
__device__ __forceinline__ void part_totals(const double* __restrict__ part, int n, double scale, double (&v)[NV],
                                            double (*red)[RT / 32]) {
#pragma unroll
  for (int i = 0; i < NV; ++i) v[i] = 0.0;
  for (int b = threadIdx.x; b < n; b += RT)
#pragma unroll
    for (int i = 0; i < NV; ++i) v[i] += part[(long)b * NV + i];
  block_totals<NV, RT>(v, red);
#pragma unroll
  for (int i = 0; i < NV; ++i) v[i] *= scale;
}

// Launches of one CTA per 32 x 8 tile x hz planes of an orbital: a thread owns
// an (x, y) column, no index division per point.
constexpr int HX = 32, HY = 8;
__device__ __forceinline__ bool tile_column(int nx, int ny, int& x, int& y) {
  const int ntx = (nx + HX - 1) / HX;
  x = (int)(blockIdx.x % ntx) * HX + (int)(threadIdx.x % HX);
  y = (int)(blockIdx.x / ntx) * HY + (int)(threadIdx.x / HX);
  return x < nx && y < ny;
}
__device__ __forceinline__ long tile_block() { return (long)blockIdx.y * gridDim.x + blockIdx.x; }

// H of real orbitals: each column marches up hz planes with the nine z neighbours
// in registers; x and y neighbours from the plane's tile with its 4-point halo
// (zero outside an isolated grid) in shared memory, the next plane's loads
// issued before this one's sums.  (Neighbours through L1 took a test, a select
// and an address each: 200 instructions a point and plane, 45 of them FP64.)
// The KB term by (point, atom) pairs from projections staged in shared memory,
// the point map read a plane ahead.  scale: null, or an orbital's partial sums
// of <in|in> (nscale blocks): the result is that of in / sqrt(<in|in>).  DOT:
// partial sums of <x|out> and <in scaled|out> in part[o][block][2].
constexpr int HMAX_NLMA = 1024;
template <bool DOT>
__global__ void __launch_bounds__(HX* HY) k_dhpsi(const double* __restrict__ in, double* __restrict__ out, RArgs a,
                                                  const double* __restrict__ scale, int nscale, double hvol,
                                                  const double* __restrict__ xk, double* __restrict__ part) {
  __shared__ double red[2][RT / 32];
  __shared__ double sproj[HMAX_NLMA];
  const int o = blockIdx.z;
  int x, y;
  const bool act = tile_column(a.nx, a.ny, x, y);
  const int z0 = blockIdx.y * a.hz, z1 = min(a.nz, z0 + a.hz);
  const double* pj = a.proj + (long)o * a.nlma;
  if (a.nlma > 0 && a.nlma <= HMAX_NLMA) {
    for (int i = threadIdx.x; i < a.nlma; i += HX * HY) sproj[i] = pj[i];
    pj = sproj;
  }
  double f = 1.0;
  if (scale) {
    double t[1];
    part_totals<1>(scale + (long)o * nscale, nscale, hvol, t, red);
    f = 1.0 / sqrt(t[0]);
  }
  __syncthreads();
  double d[2] = {0.0, 0.0};
  const double* src = in + (long)o * a.npts;
  const int plane = a.nx * a.ny, col = act ? x + a.nx * y : 0;
  constexpr int SX = HX + 2 * ND, NS = SX * (HY + 2 * ND), SL = (NS + HX * HY - 1) / (HX * HY);
  __shared__ double tile[2][NS];
  const int x0 = x - (int)(threadIdx.x % HX), y0 = y - (int)(threadIdx.x / HX);
  int goff[SL];  // plane offset of the tile values this thread loads, -1: zero
#pragma unroll
  for (int i = 0; i < SL; ++i) {
    const int e = threadIdx.x + i * HX * HY;
    int gx = x0 - ND + e % SX, gy = y0 - ND + e / SX;
    goff[i] = -1;
    if (e >= NS) continue;
    if (a.periodic) {
      gx = gx % a.nx;
      gy = gy % a.ny;
      gx = gx < 0 ? gx + a.nx : gx;
      gy = gy < 0 ? gy + a.ny : gy;
    }
    if (gx >= 0 && gx < a.nx && gy >= 0 && gy < a.ny) goff[i] = gx + a.nx * gy;
  }
  auto ldz = [&](int z) -> double {
    bool in_grid;
    const int q = wrap(z, a.nz, a.periodic, in_grid);
    return in_grid && act ? __ldg(src + (long)q * plane + col) : 0.0;
  };
  const int* map = a.pairs ? a.pmap2 : a.pmap;
  double w[2 * ND + 1], v[SL];
#pragma unroll
  for (int i = 0; i < 2 * ND; ++i) w[i] = ldz(z0 - ND + i);
#pragma unroll
  for (int i = 0; i < SL; ++i) v[i] = goff[i] >= 0 ? __ldg(src + (long)z0 * plane + goff[i]) : 0.0;
  const double* V = a.vloc + (long)(o % a.nspin) * a.npts;
  int pn = a.nlma > 0 && act ? __ldg(map + (long)z0 * plane + col) : -1;
  const int ctr = (threadIdx.x / HX + ND) * SX + threadIdx.x % HX + ND;
  for (int z = z0; z < z1; ++z) {
    double* T = tile[z & 1];
#pragma unroll
    for (int i = 0; i < SL; ++i)
      if (threadIdx.x + i * HX * HY < NS) T[threadIdx.x + i * HX * HY] = v[i];
    __syncthreads();
    w[2 * ND] = ldz(z + ND);
    const int p = z * plane + col;
    const int pm = pn;
    if (z + 1 < z1) {
      if (a.nlma > 0 && act) pn = __ldg(map + p + plane);
#pragma unroll
      for (int i = 0; i < SL; ++i) v[i] = goff[i] >= 0 ? __ldg(src + (long)(z + 1) * plane + goff[i]) : 0.0;
    }
    if (act) {
      const double vl = __ldg(V + p);
      double vx = 0.0, vy = 0.0, vz = 0.0;
#pragma unroll
      for (int s = 0; s < ND; ++s) {
        vx += a.lapt[s] * (T[ctr + s + 1] + T[ctr - s - 1]);
        vy += a.lapt[ND + s] * (T[ctr + (s + 1) * SX] + T[ctr - (s + 1) * SX]);
        vz += a.lapt[2 * ND + s] * (w[ND + 1 + s] + w[ND - 1 - s]);
      }
      const double c = w[ND];
      double h = (vl + a.lap0) * c - 0.5 * (vz + (vy + vx));
      if (pm >= 0) {
        const int e1 = (pm >> 8) + (pm & 255);
        if (a.pairs) {
          for (int e = pm >> 8; e < e1; ++e) {
            const int lm = __ldg(a.pair_lma + e);
            const double2 u0 = __ldg((const double2*)a.pair_uv + 2 * e), u1 = __ldg((const double2*)a.pair_uv + 2 * e + 1);
            const double* q = pj + (lm & 0xffffff);
            const int np = lm >> 24;
            h += q[0] * u0.x;
            if (np > 1) h += q[1] * u0.y;
            if (np > 2) h += q[2] * u1.x;
            if (np > 3) h += q[3] * u1.y;
          }
        } else {
          for (int e = pm >> 8; e < e1; ++e) h += pj[__ldg(a.ent_lma + e)] * __ldg(a.ent_uv + e);
        }
      }
      h *= f;
      out[(long)o * a.npts + p] = h;
      if (DOT) {
        d[0] = fma(__ldg(xk + (long)o * a.npts + p), h, d[0]);
        d[1] = fma(f * c, h, d[1]);
      }
    }
#pragma unroll
    for (int i = 0; i < 2 * ND; ++i) w[i] = w[i + 1];
  }
  if (DOT) {
    block_totals<2, HX * HY>(d, red);
    if (threadIdx.x < 2)
      part[((long)o * gridDim.x * gridDim.y + tile_block()) * 2 + threadIdx.x] = d[threadIdx.x];
  }
}

// real projections uVpsi = rinv * sum_j uV(j,ilma) psi(jxyz): CTA of four warps
// per (orbital, atom)
__global__ void __launch_bounds__(128) k_dproject(const double* __restrict__ in, double* __restrict__ proj, RArgs a) {
  __shared__ double red[4][4];
  const int atom = blockIdx.x, o = blockIdx.y;
  const double* psi = in + (long)o * a.npts;
  const int start = a.atom_start[atom], m = a.mps[atom];
  const int lma0 = a.lma_start[atom], np = a.nproj[atom];
  for (int q0 = 0; q0 < np; q0 += 4) {
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 2
    for (int j = threadIdx.x; j < m; j += 128) {
      const double v = __ldg(psi + a.pt_lin[start + j]);
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (q0 + q < np) acc[q] += __ldg(a.uv + (long)(lma0 + q0 + q) * a.nps + j) * v;
    }
    block_totals<4, 128>(acc, red);
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if ((int)threadIdx.x == q && q0 + q < np)
        proj[(long)o * a.nlma + lma0 + q0 + q] = acc[q] * a.rinv[lma0 + q0 + q];
  }
}

// ---------------------------------------------------------------------------
// The band-by-band CG (conjugate_gradient.f90) as six launches per iteration,
// each one pass over the orbitals that forms the scalars it needs from the
// partial sums the launch before left (per orbital, fixed order) and leaves its
// own: the scalars cost no launch and no vector is read only for a dot.
// state [o][CG_NC]: <x|H|x> and <g|g> of the last two iterations.
// ---------------------------------------------------------------------------
struct CgArgs {
  long npts;
  int nx, ny, nz, periodic, hz;
  double hvol;
  double* state;
};

// g = hx - <x|H|x> x, and its low-pass filter (preconditioning.f90:25-77) when
// LOWPASS: dir = the (filtered) gradient and partial sums of <dir|g>.  Before
// that, for iterations past the first, psi = x / sqrt(<x|x>) of the iteration
// before (when 1e-16 < |<x|x>| <= 1e30).  prev: [nprev][2] sums <x|H|x>, <x|x>.
template <bool LOWPASS>
__global__ void __launch_bounds__(HX* HY) k_cg_gradient(CgArgs c, const double* __restrict__ x,
                                                        const double* __restrict__ hx,
                                                        const double* __restrict__ prev, int nprev,
                                                        double* __restrict__ psi, double* __restrict__ dir,
                                                        double rx2, double ry2, double rz2, double omega_d,
                                                        double* __restrict__ part) {
  __shared__ double red[2][RT / 32];
  const int o = blockIdx.z;
  int ix, iy;
  const bool act = tile_column(c.nx, c.ny, ix, iy);
  const int z0 = blockIdx.y * c.hz, z1 = min(c.nz, z0 + c.hz);
  double v[2];
  part_totals<2>(prev + (long)o * nprev * 2, nprev, c.hvol, v, red);
  const double e = v[0];
  if (tile_block() == 0 && threadIdx.x == 0) c.state[CG_NC * o + CG_XKHXK] = e;
  const bool keep = psi && 1e-16 < fabs(v[1]) && fabs(v[1]) <= 1e30;
  const double root = sqrt(v[1]);
  double s[1] = {0.0};
  if (act) {
    const int plane = c.nx * c.ny;
    const long col = (long)o * c.npts + ix + (long)c.nx * iy;
    auto grad = [&](long i, bool ok) -> double { return ok ? __ldg(hx + i) - e * x[i] : 0.0; };
    bool kxp, kxm, kyp, kym, kz;
    const int xp = wrap(ix + 1, c.nx, c.periodic, kxp) - ix, xm = wrap(ix - 1, c.nx, c.periodic, kxm) - ix;
    const int yp = (wrap(iy + 1, c.ny, c.periodic, kyp) - iy) * c.nx, ym = (wrap(iy - 1, c.ny, c.periodic, kym) - iy) * c.nx;
    int q = wrap(z0 - 1, c.nz, c.periodic, kz);
    double gm = LOWPASS ? grad(col + (long)q * plane, kz) : 0.0, g = grad(col + (long)z0 * plane, true);
    for (int z = z0; z < z1; ++z) {
      const long i = col + (long)z * plane;
      double gp = 0.0, d = g;
      if (LOWPASS) {
        q = wrap(z + 1, c.nz, c.periodic, kz);
        gp = grad(col + (long)q * plane, kz);
        const double lap = (grad(i + xp, kxp) - 2.0 * g + grad(i + xm, kxm)) * rx2 +
                           (grad(i + yp, kyp) - 2.0 * g + grad(i + ym, kym)) * ry2 + (gp - 2.0 * g + gm) * rz2;
        d = omega_d * (2.0 * g - omega_d * (-0.5 * lap));
      } else if (z + 1 < z1) {
        gp = grad(i + plane, true);
      }
      if (keep) psi[i] = x[i] / root;
      dir[i] = d;
      s[0] = fma(d, g, s[0]);
      gm = g;
      g = gp;
    }
  }
  block_totals<1, HX * HY>(s, red);
  if (threadIdx.x == 0) part[(long)o * gridDim.x * gridDim.y + tile_block()] = s[0];
}

// partial sums of <u|v>
__global__ void __launch_bounds__(RT) k_cg_dot(CgArgs c, const double* __restrict__ u, const double* __restrict__ v,
                                               double* __restrict__ part) {
  __shared__ double red[1][RT / 32];
  const long base = (long)blockIdx.y * c.npts;
  double s[1] = {0.0};
  for (int it = 0; it < DOT_PTS / RT; ++it) {
    const long p = (long)blockIdx.x * DOT_PTS + it * RT + threadIdx.x;
    if (p < c.npts) s[0] = fma(u[base + p], v[base + p], s[0]);
  }
  block_totals<1, RT>(s, red);
  if (threadIdx.x == 0) part[(long)blockIdx.y * gridDim.x + blockIdx.x] = s[0];
}

// pk = dir + uk pk (uk = 0 where restart) and partial sums of <x|pk>; pgg: the
// sums of <dir|g>, kept in the state for the next iteration
__global__ void __launch_bounds__(RT) k_cg_direction(CgArgs c, const double* __restrict__ dir,
                                                     const double* __restrict__ x, const double* __restrict__ pgg,
                                                     int ngg, int iter, int restart, double* __restrict__ pk,
                                                     double* __restrict__ part) {
  __shared__ double red[1][RT / 32];
  const int o = blockIdx.y;
  const long base = (long)o * c.npts;
  double v[1];
  part_totals<1>(pgg + (long)o * ngg, ngg, c.hvol, v, red);
  double uk = 0.0;
  if (!restart) {
    const double old = c.state[CG_NC * o + CG_GG0 + ((iter + 1) & 1)];
    uk = fabs(old) > 1e-16 ? v[0] / old : 0.0;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) c.state[CG_NC * o + CG_GG0 + (iter & 1)] = v[0];
  double s[1] = {0.0};
  for (int it = 0; it < DOT_PTS / RT; ++it) {
    const long p = (long)blockIdx.x * DOT_PTS + it * RT + threadIdx.x;
    if (p >= c.npts) break;
    const double q = restart ? dir[base + p] : dir[base + p] + uk * pk[base + p];
    pk[base + p] = q;
    s[0] = fma(x[base + p], q, s[0]);
  }
  block_totals<1, RT>(s, red);
  if (threadIdx.x == 0) part[(long)o * gridDim.x + blockIdx.x] = s[0];
}

// pko = pk - <x|pk> x and partial sums of <pko|pko>
__global__ void __launch_bounds__(RT) k_cg_orthogonal(CgArgs c, const double* __restrict__ pk,
                                                      const double* __restrict__ x, const double* __restrict__ pxp,
                                                      double* __restrict__ pko, double* __restrict__ part) {
  __shared__ double red[1][RT / 32];
  const int o = blockIdx.y;
  const long base = (long)o * c.npts;
  double v[1];
  part_totals<1>(pxp + (long)o * gridDim.x, gridDim.x, c.hvol, v, red);
  double s[1] = {0.0};
  for (int it = 0; it < DOT_PTS / RT; ++it) {
    const long p = (long)blockIdx.x * DOT_PTS + it * RT + threadIdx.x;
    if (p >= c.npts) break;
    const double q = pk[base + p] - v[0] * x[base + p];
    pko[base + p] = q;
    s[0] = fma(q, q, s[0]);
  }
  block_totals<1, RT>(s, red);
  if (threadIdx.x == 0) part[(long)o * gridDim.x + blockIdx.x] = s[0];
}

// 2 x 2 Rayleigh-Ritz of x and pko / sqrt(<pko|pko>): x and hx rotated to the
// lower state (xin may be psi in the first iteration), partial sums of <x|H|x>, <x|x>
__global__ void __launch_bounds__(RT) k_cg_rotate(CgArgs c, const double* xin, double* xout,
                                                  double* __restrict__ hx, const double* __restrict__ pko,
                                                  const double* __restrict__ hwf, const double* __restrict__ ppp,
                                                  const double* __restrict__ ph, int nph,
                                                  double* __restrict__ part) {
  __shared__ double red[2][RT / 32];
  const int o = blockIdx.y;
  const long base = (long)o * c.npts;
  double n[1], v[2];
  part_totals<1>(ppp + (long)o * gridDim.x, gridDim.x, c.hvol, n, red);
  part_totals<2>(ph + (long)o * nph * 2, nph, c.hvol, v, red);
  const double f = 1.0 / sqrt(n[0]);
  const double xkHxk = c.state[CG_NC * o + CG_XKHXK], xkHpk = v[0], pkHpk = v[1];
  const double ev = 0.5 * ((xkHxk + pkHpk) -
                           sqrt((xkHxk - pkHpk) * (xkHxk - pkHpk) + 4.0 * fabs(xkHpk) * fabs(xkHpk)));
  double cx = 1.0, cp = 0.0;
  if (fabs(ev - xkHxk) > 1e-16) {
    cx = xkHpk / (ev - xkHxk);
    cp = 1.0 / sqrt(1.0 + fabs(cx) * fabs(cx));
    cx = cx * cp;
  }
  double s[2] = {0.0, 0.0};
  for (int it = 0; it < DOT_PTS / RT; ++it) {
    const long p = (long)blockIdx.x * DOT_PTS + it * RT + threadIdx.x;
    if (p >= c.npts) break;
    const double xn = cx * xin[base + p] + cp * (f * pko[base + p]);
    const double hn = cx * hx[base + p] + cp * hwf[base + p];
    xout[base + p] = xn;
    hx[base + p] = hn;
    s[0] = fma(xn, hn, s[0]);
    s[1] = fma(xn, xn, s[1]);
  }
  block_totals<2, RT>(s, red);
  if (threadIdx.x < 2) part[((long)o * gridDim.x + blockIdx.x) * 2 + threadIdx.x] = s[threadIdx.x];
}

// psi = x / sqrt(<x|x>) after the last iteration; esp[o] = <x|H|x> / <x|x>
__global__ void __launch_bounds__(RT) k_cg_end(CgArgs c, const double* __restrict__ x,
                                               const double* __restrict__ prev, int nprev, double* __restrict__ psi,
                                               double* __restrict__ esp) {
  __shared__ double red[2][RT / 32];
  const int o = blockIdx.y;
  const long base = (long)o * c.npts;
  double v[2];
  part_totals<2>(prev + (long)o * nprev * 2, nprev, c.hvol, v, red);
  if (blockIdx.x == 0 && threadIdx.x == 0) esp[o] = v[0] / v[1];
  if (!(1e-16 < fabs(v[1]) && fabs(v[1]) <= 1e30)) return;
  const double root = sqrt(v[1]);
  for (int it = 0; it < DOT_PTS / RT; ++it) {
    const long p = (long)blockIdx.x * DOT_PTS + it * RT + threadIdx.x;
    if (p < c.npts) psi[base + p] = x[base + p] / root;
  }
}

// low-pass preconditioner (preconditioning.f90:25-77), 3-point Laplacian
__global__ void k_precond(const double* __restrict__ g, double* __restrict__ pre, RArgs a, double hx2, double hy2,
                          double hz2, double omega_d) {
  const long p = blockIdx.x * 256L + threadIdx.x;
  if (p >= a.npts) return;
  const int o = blockIdx.y;
  const int x = (int)(p % a.nx), y = (int)((p / a.nx) % a.ny), z = (int)(p / ((long)a.nx * a.ny));
  const double* t = g + (long)o * a.npts;
  const double c = t[p];
  auto nb = [&](int q, int n, int cc, long st) -> double {
    bool ok;
    const int w = wrap(q, n, a.periodic, ok);
    return ok ? t[p + (w - cc) * st] : 0.0;
  };
  const double v = (nb(x + 1, a.nx, x, 1) - 2.0 * c + nb(x - 1, a.nx, x, 1)) / hx2 +
                   (nb(y + 1, a.ny, y, a.nx) - 2.0 * c + nb(y - 1, a.ny, y, a.nx)) / hy2 +
                   (nb(z + 1, a.nz, z, (long)a.nx * a.ny) - 2.0 * c + nb(z - 1, a.nz, z, (long)a.nx * a.ny)) / hz2;
  pre[(long)o * a.npts + p] = omega_d * (2.0 * c - omega_d * (-0.5 * v));
}

// ---------------------------------------------------------------------------
// Tall-skinny products for Gram-Schmidt and the subspace matrix:
//   part[b][i][j] = sum_{p in chunk b} A[i][p] * B[j][p], i < m, j < n
// One CTA = one 32 x 32 output tile over a point chunk; its four groups of 64
// threads take the chunk's 16-point slabs in turn (4 x 4 outputs a thread: 8
// shared loads per 16 FMA, the LSU and FP64 pipes even) and are added in group
// order.  Bound by reading A and B; the chunks are cut so that about four CTAs
// per SM run (24 orbitals of 48^3: 7 CTAs of 16384 points took 649 us a product).
// upper: tiles below the diagonal are left out (their part is not written).
// ---------------------------------------------------------------------------
constexpr int GT = 32, GK = 16;
__global__ void __launch_bounds__(256) k_gram_part(const double* __restrict__ A, int m, const double* __restrict__ B,
                                                   int n, long npts, long chunk, int upper,
                                                   double* __restrict__ part) {
  const int ti = blockIdx.x, tj = blockIdx.y, b = blockIdx.z;
  if (upper && ti > tj) return;
  __shared__ double S[2][4][GT][GK + 1];  // slabs of A and B per group; the sums reuse them
  const int g = threadIdx.x >> 6, u = threadIdx.x & 63, tx = u & 7, ty = u >> 3;
  const int kl = u & (GK - 1), rl = u / GK;
  const long p0 = (long)b * chunk, p1 = min(npts, p0 + chunk);
  double acc[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[r][c] = 0.0;
  for (long pp = p0 + g * GK; pp < p0 + chunk; pp += 4 * GK) {
    const long p = pp + kl;
#pragma unroll
    for (int r = rl; r < GT; r += 64 / GK) {
      const int i = ti * GT + r, j = tj * GT + r;
      S[0][g][r][kl] = (i < m && p < p1) ? A[(long)i * npts + p] : 0.0;
      S[1][g][r][kl] = (j < n && p < p1) ? B[(long)j * npts + p] : 0.0;
    }
    __syncthreads();
#pragma unroll 4
    for (int k = 0; k < GK; ++k) {
      double x[4], y[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        x[r] = S[0][g][ty + 8 * r][k];
        y[r] = S[1][g][tx + 8 * r][k];
      }
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][c] = fma(x[r], y[c], acc[r][c]);
    }
    __syncthreads();
  }
  double* sum = &S[0][0][0][0];  // [4][32 x 32] of the 2 x 4 x 32 x 17 doubles
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) sum[g * GT * GT + (ty + 8 * r) * GT + tx + 8 * c] = acc[r][c];
  __syncthreads();
  for (int q = threadIdx.x; q < GT * GT; q += 256) {
    const int i = ti * GT + q / GT, j = tj * GT + q % GT;
    if (i < m && j < n)
      part[((long)b * m + i) * n + j] = ((sum[q] + sum[GT * GT + q]) + sum[2 * GT * GT + q]) + sum[3 * GT * GT + q];
  }
}

// out[q] = scale * sum_b part[b][q]: 32 entries x 32 slices of the chunks per
// block, the slices added in order
__global__ void __launch_bounds__(1024) k_gram_final(const double* __restrict__ part, int nb, long mn, double scale,
                                                     double* __restrict__ out) {
  __shared__ double red[32][33];
  const long q = blockIdx.x * 32L + threadIdx.x;
  double s = 0.0;
  if (q < mn)
    for (int b = threadIdx.y; b < nb; b += 32) s += part[(long)b * mn + q];
  red[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y == 0 && q < mn) {
    double t = 0.0;
    for (int k = 0; k < 32; ++k) t += red[k][threadIdx.x];
    out[q] = t * scale;
  }
}

// ---------------------------------------------------------------------------
// Column Gram-Schmidt of all orbitals at once: with G = X^T X hvol the
// coefficients of every column follow from G alone.  k_gs_coeff (one CTA)
// eliminates row after row: row i < j of column j holds T(i, j), the part of
// the original orbital i in the orthonormal orbital j, rows i >= j what is left
// of G, so one n x n matrix W (row-major) carries both.  Q^T Q = T^T G T carries
// the rounding of G times the square of the growth g = |T_ij| |x_i|: up to
// 4 g^2 2^-52 in groups of 5 columns about one other, growth 10 to 70, in 8 to 64
// of 5814 points; column by column (classical Gram-Schmidt) loses the same square,
// 1 to 5 times as much there.  When g passes GS_GROWTH (orbitals close to linear
// dependence, or a zero or non-finite one) *bad is set and the caller takes the
// column-by-column form instead.  24
// orbitals of 48^3: 115 launches, 15.7 ms column by column; 5 launches here
// (a solver iteration with CG and subspace rotation 18.8 -> 2.1 ms).
// ---------------------------------------------------------------------------
constexpr double GS_GROWTH = 100.0;  // largest |T_ij| |x_i|: its square is four digits of the 16
constexpr int GC_THREADS = 512;
constexpr int GC_SMEM_N = 150;  // W kept in shared memory up to here (180 KB)

__global__ void __launch_bounds__(GC_THREADS) k_gs_coeff(double* __restrict__ G, int n, int in_smem,
                                                         double* __restrict__ T, double* __restrict__ work,
                                                         int* __restrict__ bad) {
  extern __shared__ double gsm[];
  double* nrm = work;        // [n] G_ii
  double* rb = work + n;     // [n] R(j, k) of the current row
  double* W = G;
  if (in_smem) {
    W = gsm;
    nrm = gsm + (size_t)n * n;
    rb = nrm + n;
    for (int q = threadIdx.x; q < n * n; q += GC_THREADS) W[q] = G[q];
  }
  __shared__ int sbad;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, NWP = GC_THREADS / 32;
  if (threadIdx.x == 0) sbad = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += GC_THREADS) nrm[i] = W[(size_t)i * n + i];
  __syncthreads();
  for (int j = 0; j < n; ++j) {
    const double d = W[(size_t)j * n + j];
    const double r = 1.0 / sqrt(d);  // a negative or NaN d is caught by the growth test
    for (int k = j + 1 + threadIdx.x; k < n; k += GC_THREADS) rb[k] = W[(size_t)j * n + k] * r;
    __syncthreads();
    // row j turns from what is left of G into T; column j of T is scaled
    for (int i = threadIdx.x; i <= j; i += GC_THREADS) W[(size_t)i * n + j] = (i == j) ? r : W[(size_t)i * n + j] * r;
    for (int k = j + 1 + threadIdx.x; k < n; k += GC_THREADS) W[(size_t)j * n + k] = 0.0;
    __syncthreads();
    // T(:, k) -= R(j, k) T(:, j) for rows i <= j; G(i, k) -= R(j, i) R(j, k) for j < i <= k
    for (int i = warp; i < n; i += NWP) {
      const double f = i <= j ? W[(size_t)i * n + j] : rb[i];
      for (int k = max(i, j + 1) + lane; k < n; k += 32) W[(size_t)i * n + k] = fma(-f, rb[k], W[(size_t)i * n + k]);
    }
    __syncthreads();
  }
  int b = 0;
  for (int i = warp; i < n; i += NWP)
    for (int j = lane; j < n; j += 32) {
      const double v = j >= i ? W[(size_t)i * n + j] : 0.0;
      T[(size_t)j * n + i] = v;  // column-major for k_gs_apply
      if (!(v * v * nrm[i] <= GS_GROWTH * GS_GROWTH)) b = 1;
    }
  if (b) sbad = 1;
  __syncthreads();
  if (threadIdx.x == 0) *bad = sbad;
}

// Sum of 32 values over the 32 lanes of a warp by reduce-scatter: lane L gets
// the total of value L (31 shuffles, fixed order).
__device__ __forceinline__ double warp_scatter32(double (&v)[32], int lane) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const bool upper = (lane & off) != 0;
#pragma unroll
    for (int i = 0; i < off; ++i) {
      const double keep = upper ? v[off + i] : v[i];
      const double send = upper ? v[i] : v[off + i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
  }
  return v[0];
}

// X(p, j) <- sum_{i <= j} X(p, i) T(i, j) in place (a thread owns its point;
// column tiles from the last to the first), and the sums of squares of every
// new column over the block's points in part[j][block].  Each X value is read
// once per column tile and feeds 32 FMA against T broadcast from shared memory.
constexpr int GA_THREADS = 128;
__global__ void __launch_bounds__(GA_THREADS) k_gs_apply(double* __restrict__ X, int n, const double* __restrict__ T,
                                                         long npts, double* __restrict__ part,
                                                         const int* __restrict__ bad) {
  if (*bad) return;
  __shared__ __align__(16) double Ts[GT][GT];
  __shared__ double red[GA_THREADS / 32][GT];
  const long p = blockIdx.x * (long)GA_THREADS + threadIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int j0 = (n - 1) / GT * GT; j0 >= 0; j0 -= GT) {
    double acc[GT];
#pragma unroll
    for (int u = 0; u < GT; ++u) acc[u] = 0.0;
    const int iend = min(n, j0 + GT);
    for (int i0 = 0; i0 < iend; i0 += GT) {
      __syncthreads();
      for (int c = threadIdx.x; c < GT * GT; c += GA_THREADS) {
        const int ii = c % GT, jj = c / GT;
        Ts[ii][jj] = (i0 + ii < n && j0 + jj < n) ? T[(size_t)(j0 + jj) * n + i0 + ii] : 0.0;
      }
      __syncthreads();
      if (p < npts) {
        const int im = min(GT, n - i0);
#pragma unroll 4
        for (int ii = 0; ii < im; ++ii) {
          const double x = X[(long)(i0 + ii) * npts + p];
#pragma unroll
          for (int u = 0; u < GT; ++u) acc[u] = fma(x, Ts[ii][u], acc[u]);
        }
      }
    }
#pragma unroll
    for (int u = 0; u < GT; ++u) {
      if (p < npts && j0 + u < n) X[(long)(j0 + u) * npts + p] = acc[u];
      acc[u] *= acc[u];
    }
    const double s = warp_scatter32(acc, lane);
    red[warp][lane] = s;
    __syncthreads();
    if (threadIdx.x < GT && j0 + threadIdx.x < n) {
      double t = red[0][threadIdx.x];
      for (int w = 1; w < GA_THREADS / 32; ++w) t += red[w][threadIdx.x];
      part[(long)(j0 + threadIdx.x) * gridDim.x + blockIdx.x] = t;
    }
  }
}

// Y[j][p] = beta * Y[j][p] + alpha * sum_i X[i][p] * M[i][j]; M column-major m x n
__global__ void __launch_bounds__(256) k_rotate(const double* __restrict__ X, int m, const double* __restrict__ M,
                                                int n, long npts, double alpha, double beta, double* __restrict__ Y) {
  __shared__ double Ms[GT][GT + 1];
  const long p = blockIdx.x * 256L + threadIdx.x;
  const int j0 = blockIdx.y * GT;
  double acc[GT];
#pragma unroll
  for (int u = 0; u < GT; ++u) acc[u] = 0.0;
  for (int i0 = 0; i0 < m; i0 += GT) {
    for (int c = threadIdx.x; c < GT * GT; c += 256) {
      const int ii = c / GT, jj = c % GT;
      Ms[ii][jj] = (i0 + ii < m && j0 + jj < n) ? M[(long)(j0 + jj) * m + (i0 + ii)] : 0.0;
    }
    __syncthreads();
    if (p < npts) {
      for (int ii = 0; ii < GT && i0 + ii < m; ++ii) {
        const double x = X[(long)(i0 + ii) * npts + p];
#pragma unroll
        for (int u = 0; u < GT; ++u) acc[u] += x * Ms[ii][u];
      }
    }
    __syncthreads();
  }
  if (p < npts)
    for (int u = 0; u < GT; ++u)
      if (j0 + u < n) {
        const long q = (long)(j0 + u) * npts + p;
        Y[q] = alpha * acc[u] + (beta != 0.0 ? beta * Y[q] : 0.0);
      }
}

// partial sums of squares of columns blockIdx.y of y, then every column scaled by
// 1/sqrt(hvol * sum): all columns in one launch each
__global__ void __launch_bounds__(RT) k_sq_part(const double* __restrict__ y, long n, double* __restrict__ part) {
  __shared__ double red[RT];
  double s = 0.0;
  const long p0 = (long)blockIdx.x * DOT_PTS;
  const double* yc = y + blockIdx.y * n;
  for (int it = 0; it < DOT_PTS / RT; ++it) {
    const long p = p0 + it * RT + threadIdx.x;
    if (p >= n) break;
    s += yc[p] * yc[p];
  }
  red[threadIdx.x] = s;
  __syncthreads();
  for (int st = RT / 2; st > 0; st >>= 1) {
    if (threadIdx.x < st) red[threadIdx.x] += red[threadIdx.x + st];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[(long)blockIdx.y * gridDim.x + blockIdx.x] = red[0];
}

// bad: null, or a device flag that makes the launch return at once
__global__ void __launch_bounds__(RT) k_scale_norm(const double* y, double* out, long n,
                                                   const double* __restrict__ part, int nblk, double hvol,
                                                   const int* __restrict__ bad) {
  if (bad && *bad) return;
  __shared__ double red[RT];
  const double* pc = part + (long)blockIdx.y * nblk;
  double s = 0.0;
  for (int b = threadIdx.x; b < nblk; b += RT) s += pc[b];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int st = RT / 2; st > 0; st >>= 1) {
    if (threadIdx.x < st) red[threadIdx.x] += red[threadIdx.x + st];
    __syncthreads();
  }
  const double f = 1.0 / sqrt(red[0] * hvol);
  const long p0 = (long)blockIdx.x * DOT_PTS, base = blockIdx.y * n;
  for (int it = 0; it < DOT_PTS / RT; ++it) {
    const long p = p0 + it * RT + threadIdx.x;
    if (p < n) out[base + p] = f * y[base + p];
  }
}

__global__ void k_relayout_real(const double* __restrict__ src, double* __restrict__ dst, int nx, int ny, int nz,
                                int nxa, int nya, long vola, int ox, int oy, int oz, int norb, int to_ref) {
  const long npts = (long)nx * ny * nz;
  const long total = npts * norb;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const long o = i / npts, p = i % npts;
    const int x = (int)(p % nx), y = (int)((p / nx) % ny), z = (int)(p / ((long)nx * ny));
    const long r = o * vola + (x + ox) + (long)nxa * ((y + oy) + (long)nya * (z + oz));
    if (to_ref) dst[r] = src[i];
    else dst[i] = src[r];
  }
}

int gridsz(long n) {
  long b = (n + 255) / 256;
  if (b > 148L * 32) b = 148L * 32;
  return (int)(b < 1 ? 1 : b);
}

}  // namespace

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
static RArgs rargs(sb200_ctx* c) {
  RArgs a;
  a.nx = c->g.nx;
  a.ny = c->g.ny;
  a.nz = c->g.nz;
  a.periodic = c->g.periodic;
  a.hz = 1;
  a.nspin = c->orb.nspin;
  a.nlma = c->pp.nlma;
  a.natom = c->pp.natom;
  a.nps = c->pp.nps;
  a.totpts = c->pp.totpts;
  a.npts = c->g.npts;
  a.lap0 = c->g.coef_lap0;
  for (int i = 0; i < 12; ++i) a.lapt[i] = c->g.coef_lap[i];
  a.vloc = c->d_vloc;
  a.pmap = c->pp.d_pmap;
  a.ent_lma = c->pp.d_ent_lma;
  a.ent_uv = c->pp.d_ent_uv;
  a.pairs = c->pp.npair > 0 ? 1 : 0;
  a.pmap2 = c->pp.d_pmap2;
  a.pair_lma = c->pp.d_pair_lma;
  a.pair_uv = c->pp.d_pair_uv;
  a.proj = c->gs.d_proj;
  a.atom_start = c->pp.d_atom_start;
  a.mps = c->pp.d_mps;
  a.lma_start = c->pp.d_lma_start;
  a.nproj = c->pp.d_nproj;
  a.pt_lin = c->pp.d_pt_lin;
  a.uv = c->pp.d_uv;
  a.rinv = c->pp.d_rinv;
  return a;
}

// one CTA per 32 x 8 tile x hz planes and orbital; hz from 1 (small grids: latency)
// to 16 (a column reads 8 planes more than it has), about six CTAs per SM
int dhpsi_hz(const sb200_ctx* c) {
  const GridInfo& g = c->g;
  const long planes = (long)((g.nx + HX - 1) / HX) * ((g.ny + HY - 1) / HY) * g.nz * c->orb.norb;
  const long hz = planes / (148 * 6);
  return (int)(hz < 1 ? 1 : (hz > 16 ? 16 : hz));
}
dim3 dhpsi_grid(const sb200_ctx* c) {
  const GridInfo& g = c->g;
  const int hz = dhpsi_hz(c);
  return dim3((unsigned)(((g.nx + HX - 1) / HX) * ((g.ny + HY - 1) / HY)), (unsigned)((g.nz + hz - 1) / hz),
              (unsigned)c->orb.norb);
}

int gs_ensure(sb200_ctx* c, bool cg_work) {
  GSState& s = c->gs;
  const long n = c->g.npts * c->orb.norb;
  const int norb = c->orb.norb;
  const int nblk = (int)((c->g.npts + DOT_PTS - 1) / DOT_PTS);
  const dim3 hg = dhpsi_grid(c);
  const size_t per = 6 * (size_t)nblk + 3 * (size_t)hg.x * hg.y;  // partial sums of an orbital
  const size_t npart = per * norb, nproj = (size_t)norb * (c->pp.nlma > 0 ? c->pp.nlma : 1);
  if (s.n != n || s.norb != norb || s.npart < npart || s.nproj < nproj) {
    dfree(s.d_proj);
    dfree(s.d_part);
    dfree(s.d_dots);
    dfree(s.d_coef);
    dfree(s.d_work);
    s.n = 0;
    s.have_work = false;
    TRY_GS(dalloc(&s.d_proj, nproj));
    TRY_GS(dalloc(&s.d_part, npart));
    TRY_GS(dalloc(&s.d_dots, (size_t)norb));
    TRY_GS(dalloc(&s.d_coef, (size_t)norb * CG_NC));
    s.n = n;
    s.norb = norb;
    s.nblk = nblk;
    s.npart = npart;
    s.nproj = nproj;
  }
  s.nblk = nblk;
  if (cg_work && !s.have_work) {
    TRY_GS(dalloc(&s.d_work, (size_t)n * 7));
    s.have_work = true;
  }
  return SB200_OK;
}

// out = H in; with part: partial sums of <x|out> and <in|out>; with scale
// (partial sums of <in|in>): of in / sqrt(<in|in>)
int gs_hpsi(sb200_ctx* c, const double* in, double* out, const double* scale = nullptr, const double* x = nullptr,
            double* part = nullptr) {
  RArgs a = rargs(c);
  a.hz = dhpsi_hz(c);
  if (a.nlma > 0) {
    dim3 g(a.natom, c->orb.norb);
    k_dproject<<<g, 128, 0, c->stream>>>(in, c->gs.d_proj, a);
    SB_LAUNCH_CHECK("k_dproject");
  }
  const dim3 g = dhpsi_grid(c);
  if (part)
    k_dhpsi<true><<<g, HX * HY, 0, c->stream>>>(in, out, a, scale, c->gs.nblk, c->g.hvol, x, part);
  else
    k_dhpsi<false><<<g, HX * HY, 0, c->stream>>>(in, out, a, scale, c->gs.nblk, c->g.hvol, nullptr, nullptr);
  SB_LAUNCH_CHECK("k_dhpsi");
  return SB200_OK;
}

int gs_precond(sb200_ctx* c, const double* g, double* pre, double alpha) {
  RArgs a = rargs(c);
  const double h0 = c->g.hgs[0], h1 = c->g.hgs[1], h2 = c->g.hgs[2];
  const double omega = 2.0 * (1.0 - alpha);
  const double d = -0.5 * ((-2.0) / (h0 * h0) + (-2.0) / (h1 * h1) + (-2.0) / (h2 * h2));
  dim3 gr((unsigned)((a.npts + 255) / 256), c->orb.norb);
  k_precond<<<gr, 256, 0, c->stream>>>(g, pre, a, h0 * h0, h1 * h1, h2 * h2, omega / d);
  SB_LAUNCH_CHECK("k_precond");
  return SB200_OK;
}

// ---- complex column Gram-Schmidt (gram_schmidt_col_complex8) -------------
// Orbitals io of one (k, spin) group sit `stride` complex values apart.
// part[io2][b] = sum over the points of block b of conj(psi_io2) psi_io1
__global__ void __launch_bounds__(RT) k_zgs_dots(const double2* __restrict__ psi, long stride, int io1, long npts,
                                                 double2* __restrict__ part, int nb) {
  __shared__ double rr[RT], ri[RT];
  const int io2 = blockIdx.y;
  const double2* a = psi + stride * io2;
  const double2* b = psi + stride * io1;
  double sr = 0.0, si = 0.0;
  const long p0 = (long)blockIdx.x * DOT_PTS;
  for (int it = 0; it < DOT_PTS / RT; ++it) {
    const long p = p0 + it * RT + threadIdx.x;
    if (p < npts) {
      const double2 x = a[p], y = b[p];
      sr += x.x * y.x + x.y * y.y;
      si += x.x * y.y - x.y * y.x;
    }
  }
  rr[threadIdx.x] = sr;
  ri[threadIdx.x] = si;
  __syncthreads();
  for (int st = RT / 2; st > 0; st >>= 1) {
    if (threadIdx.x < st) {
      rr[threadIdx.x] += rr[threadIdx.x + st];
      ri[threadIdx.x] += ri[threadIdx.x + st];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) part[(long)io2 * nb + blockIdx.x] = make_double2(rr[0], ri[0]);
}

// coeff[io2] = hvol * sum_b part[io2][b] (blocks in order)
__global__ void k_zgs_coeff(const double2* __restrict__ part, int nb, int m, double hvol,
                            double2* __restrict__ coeff) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  double sr = 0.0, si = 0.0;
  for (int b = 0; b < nb; ++b) {
    sr += part[(long)i * nb + b].x;
    si += part[(long)i * nb + b].y;
  }
  coeff[i] = make_double2(sr * hvol, si * hvol);
}

// psi_io1 <- psi_io1 - sum_{io2 < io1} coeff[io2] psi_io2 (exclusion term
// accumulated in io2 order, then subtracted)
__global__ void k_zgs_sub(double2* __restrict__ psi, long stride, int io1, const double2* __restrict__ coeff,
                          long npts) {
  for (long p = blockIdx.x * 256L + threadIdx.x; p < npts; p += (long)gridDim.x * 256) {
    double2 exc = make_double2(0.0, 0.0);
    for (int io2 = 0; io2 < io1; ++io2) {
      const double2 cf = coeff[io2], x = psi[stride * io2 + p];
      exc = make_double2(cf.x * x.x - cf.y * x.y + exc.x, cf.x * x.y + cf.y * x.x + exc.y);
    }
    double2* w = psi + stride * io1 + p;
    *w = make_double2(-exc.x + w->x, -exc.y + w->y);
  }
}

// part[b] = sum over block b of |psi|^2
__global__ void __launch_bounds__(RT) k_zsq_part(const double2* __restrict__ y, long n, double* __restrict__ part) {
  __shared__ double r[RT];
  double s = 0.0;
  const long p0 = (long)blockIdx.x * DOT_PTS;
  for (int it = 0; it < DOT_PTS / RT; ++it) {
    const long p = p0 + it * RT + threadIdx.x;
    if (p < n) s += y[p].x * y[p].x + y[p].y * y[p].y;
  }
  r[threadIdx.x] = s;
  __syncthreads();
  for (int st = RT / 2; st > 0; st >>= 1) {
    if (threadIdx.x < st) r[threadIdx.x] += r[threadIdx.x + st];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = r[0];
}

// y <- y / sqrt(hvol * sum_b part[b])
__global__ void k_zscale_norm(double2* __restrict__ y, long n, const double* __restrict__ part, int nb, double hvol) {
  double s = 0.0;
  for (int b = 0; b < nb; ++b) s += part[b];
  const double sc = 1.0 / sqrt(s * hvol);
  for (long p = blockIdx.x * 256L + threadIdx.x; p < n; p += (long)gridDim.x * 256)
    y[p] = make_double2(sc * y[p].x, sc * y[p].y);
}

// C (m x n, row-major [i][j]) = scale * A(m orbitals) . B(n orbitals); upper:
// entries of 32 x 32 tiles below the diagonal are left undefined
int gs_gram(sb200_ctx* c, const double* A, int m, const double* B, int n, double scale, double* C_dev,
            bool upper = false) {
  const long npts = c->g.npts;
  const long ti = (m + GT - 1) / GT, tj = (n + GT - 1) / GT;
  // about four CTAs per SM, each with at least 256 points
  long nb = (148L * 4 + ti * tj - 1) / (ti * tj);
  if (nb > (npts + 255) / 256) nb = (npts + 255) / 256;
  if (nb < 1) nb = 1;
  const long chunk = ((npts + nb - 1) / nb + 4 * GK - 1) / (4 * GK) * (4 * GK);
  nb = (npts + chunk - 1) / chunk;
  const size_t need = (size_t)nb * m * n;
  if (c->gs.gram_cap < need) {
    dfree(c->gs.d_gram);
    c->gs.gram_cap = 0;
    TRY_GS(dalloc(&c->gs.d_gram, need));
    c->gs.gram_cap = need;
  }
  dim3 g((unsigned)ti, (unsigned)tj, (unsigned)nb);
  k_gram_part<<<g, 256, 0, c->stream>>>(A, m, B, n, npts, chunk, upper ? 1 : 0, c->gs.d_gram);
  SB_LAUNCH_CHECK("k_gram_part");
  const long mn = (long)m * n;
  k_gram_final<<<(unsigned)((mn + 31) / 32), dim3(32, 32), 0, c->stream>>>(c->gs.d_gram, (int)nb, mn, scale, C_dev);
  SB_LAUNCH_CHECK("k_gram_final");
  return SB200_OK;
}

int gs_relayout(sb200_ctx* c, const double* src, double* dst, int norb, bool to_ref) {
  const GridInfo& g = c->g;
  const int nxa = g.ie_array[0] - g.is_array[0] + 1;
  const int nya = g.ie_array[1] - g.is_array[1] + 1;
  k_relayout_real<<<gridsz(g.npts * norb), 256, 0, c->stream>>>(src, dst, g.nx, g.ny, g.nz, nxa, nya,
                                                                 g.vol_array(), g.is[0] - g.is_array[0],
                                                                 g.is[1] - g.is_array[1], g.is[2] - g.is_array[2],
                                                                 norb, to_ref ? 1 : 0);
  SB_LAUNCH_CHECK("k_relayout_real");
  return SB200_OK;
}

int gs_rotate(sb200_ctx* c, const double* X, int m, const double* M_dev, int n, double beta, double* Y) {
  dim3 g((unsigned)((c->g.npts + 255) / 256), (n + GT - 1) / GT);
  k_rotate<<<g, 256, 0, c->stream>>>(X, m, M_dev, n, c->g.npts, 1.0, beta, Y);
  SB_LAUNCH_CHECK("k_rotate");
  return SB200_OK;
}

// y <- y - sum_i coeff[i] * X_i  (exc accumulated in i order, then subtracted)
// Y -= X (X^T Y) hvol for Y of n orbitals: removes from every column of Y its
// components along the m orthonormal orbitals X (scratch: the small-matrix area)
int gs_project_out(sb200_ctx* c, const double* X, int m, double* Y, int n) {
  if (c->gs.mat_cap < (size_t)m * n) {
    dfree(c->gs.d_mat);
    TRY_GS(dalloc(&c->gs.d_mat, (size_t)m * n));
    c->gs.mat_cap = (size_t)m * n;
  }
  // gs_gram(Y, X) stores <Y_j, X_i> at j*m + i: the column-major M(i, j) k_rotate reads
  TRY_GS(gs_gram(c, Y, n, X, m, c->g.hvol, c->gs.d_mat));
  dim3 g((unsigned)((c->g.npts + 255) / 256), (n + GT - 1) / GT);
  k_rotate<<<g, 256, 0, c->stream>>>(X, m, c->gs.d_mat, n, c->g.npts, -1.0, 1.0, Y);
  SB_LAUNCH_CHECK("k_rotate");
  return SB200_OK;
}

int gs_rotate_sub(sb200_ctx* c, const double* X, int m, const double* coeff_dev, double* y) {
  dim3 g((unsigned)((c->g.npts + 255) / 256), 1);
  k_rotate<<<g, 256, 0, c->stream>>>(X, m, coeff_dev, 1, c->g.npts, -1.0, 1.0, y);
  SB_LAUNCH_CHECK("k_rotate");
  return SB200_OK;
}

// out_j <- y_j / sqrt(hvol * sum y_j^2) for nc orbitals, deterministic
int gs_norm_scale(sb200_ctx* c, const double* y, double* out, int nc) {
  const long n = c->g.npts;
  const int nblk = (int)((n + DOT_PTS - 1) / DOT_PTS);
  dim3 g(nblk, nc);
  k_sq_part<<<g, RT, 0, c->stream>>>(y, n, c->gs.d_part);
  SB_LAUNCH_CHECK("k_sq_part");
  k_scale_norm<<<g, RT, 0, c->stream>>>(y, out, n, c->gs.d_part, nblk, c->g.hvol, nullptr);
  SB_LAUNCH_CHECK("k_scale_norm");
  return SB200_OK;
}

// Gram-Schmidt of the n contiguous orbitals X at once (k_gs_coeff); *bad (device)
// says that X was left as it was and needs the column form.  mat: 2 n^2 + 2 n
// doubles.
int gs_orthonormalise(sb200_ctx* c, double* X, int n, double* mat, int* bad) {
  const long npts = c->g.npts;
  double* G = mat;
  double* T = mat + (size_t)n * n;
  double* work = T + (size_t)n * n;
  TRY_GS(gs_gram(c, X, n, X, n, c->g.hvol, G, true));
  const int in_smem = n <= GC_SMEM_N;
  const size_t smem = in_smem ? ((size_t)n * n + 2 * n) * sizeof(double) : 0;
  SB_CUDA(cudaFuncSetAttribute(k_gs_coeff, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (GC_SMEM_N * GC_SMEM_N + 2 * GC_SMEM_N) * (int)sizeof(double)));
  k_gs_coeff<<<1, GC_THREADS, smem, c->stream>>>(G, n, in_smem, T, work, bad);
  SB_LAUNCH_CHECK("k_gs_coeff");
  const int nblk = (int)((npts + GA_THREADS - 1) / GA_THREADS);
  const size_t need = (size_t)nblk * n;  // the sums of squares share the Gram partials' buffer
  if (c->gs.gram_cap < need) {
    dfree(c->gs.d_gram);
    c->gs.gram_cap = 0;
    TRY_GS(dalloc(&c->gs.d_gram, need));
    c->gs.gram_cap = need;
  }
  k_gs_apply<<<nblk, GA_THREADS, 0, c->stream>>>(X, n, T, npts, c->gs.d_gram, bad);
  SB_LAUNCH_CHECK("k_gs_apply");
  k_scale_norm<<<dim3((unsigned)((npts + DOT_PTS - 1) / DOT_PTS), n), RT, 0, c->stream>>>(X, X, npts, c->gs.d_gram,
                                                                                       nblk, c->g.hvol, bad);
  SB_LAUNCH_CHECK("k_scale_norm");
  return SB200_OK;
}

}  // namespace sb200

// ---------------------------------------------------------------------------
// C ABI of the ground-state path
// ---------------------------------------------------------------------------
using namespace sb200;

namespace {

int gs_ready(sb200_ctx* c) {
  if (!c) return set_error(SB200_ERR_INVALID_ARG, "null ctx");
  if (!c->g.set || !c->orb.set || !c->vloc_set)
    return set_error(SB200_ERR_STATE, "ground state needs sb200_set_grid / _set_orbitals / _set_vlocal first");
  if (c->orb.nk != 1) return set_error(SB200_ERR_UNSUPPORTED, "real-orbital ground state takes one k-point");
  return SB200_OK;
}

struct DevGuard {
  int prev = -1;
  explicit DevGuard(int dev) {
    if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
    if (prev != dev) cudaSetDevice(dev);
  }
  ~DevGuard() {
    if (prev >= 0) cudaSetDevice(prev);
  }
};

int gs_mat(sb200_ctx* c, size_t n) {
  if (c->gs.mat_cap >= n) return SB200_OK;
  dfree(c->gs.d_mat);
  TRY_GS(dalloc(&c->gs.d_mat, n));
  c->gs.mat_cap = n;
  return SB200_OK;
}

int gs_relayout_all(sb200_ctx* c, const double* src_ref, double* dst_dev, double* dst_ref, const double* src_dev,
                    bool to_ref) {
  const size_t blk = (size_t)c->g.vol_array() * sizeof(double);
  const int norb = c->orb.norb;
  int chunk = (int)((size_t)(256u << 20) / blk);
  if (chunk < 1) chunk = 1;
  if (chunk > norb) chunk = norb;
  if (c->stage_bytes < blk * chunk) {
    if (c->d_stage) cudaFree(c->d_stage);
    c->d_stage = nullptr;
    c->stage_bytes = 0;
    SB_CUDA(cudaMalloc(&c->d_stage, blk * chunk));
    c->stage_bytes = blk * chunk;
  }
  for (int o0 = 0; o0 < norb; o0 += chunk) {
    const int n = (o0 + chunk <= norb) ? chunk : norb - o0;
    if (!to_ref) {
      SB_CUDA(cudaMemcpyAsync(c->d_stage, (const char*)src_ref + blk * o0, blk * n, cudaMemcpyDefault, c->stream));
      TRY_GS(gs_relayout(c, (const double*)c->d_stage, dst_dev + c->g.npts * o0, n, false));
    } else {
      SB_CUDA(cudaMemsetAsync(c->d_stage, 0, blk * n, c->stream));
      TRY_GS(gs_relayout(c, src_dev + c->g.npts * o0, (double*)c->d_stage, n, true));
      SB_CUDA(cudaMemcpyAsync((char*)dst_ref + blk * o0, c->d_stage, blk * n, cudaMemcpyDefault, c->stream));
    }
    SB_CUDA(cudaStreamSynchronize(c->stream));
  }
  return SB200_OK;
}

}  // namespace

extern "C" {

int sb200_gs_from_ref(sb200_ctx* c, const double* rwf_ref, double* psi_dev) {
  TRY_GS(gs_ready(c));
  if (!rwf_ref || !psi_dev) return set_error(SB200_ERR_INVALID_ARG, "null orbital pointer");
  DevGuard dg(c->device);
  return gs_relayout_all(c, rwf_ref, psi_dev, nullptr, nullptr, false);
}

int sb200_gs_to_ref(sb200_ctx* c, const double* psi_dev, double* rwf_ref) {
  TRY_GS(gs_ready(c));
  if (!rwf_ref || !psi_dev) return set_error(SB200_ERR_INVALID_ARG, "null orbital pointer");
  DevGuard dg(c->device);
  return gs_relayout_all(c, nullptr, nullptr, rwf_ref, psi_dev, true);
}

int sb200_hpsi_real(sb200_ctx* c, const double* tpsi, double* htpsi) {
  TRY_GS(gs_ready(c));
  if (!tpsi || !htpsi || tpsi == htpsi) return set_error(SB200_ERR_INVALID_ARG, "tpsi/htpsi null or aliased");
  DevGuard dg(c->device);
  TRY_GS(gs_ensure(c, false));
  return gs_hpsi(c, tpsi, htpsi);
}

int sb200_gscg(sb200_ctx* c, double* psi, int ncg, int precondition, double alpha_pre, double* esp) {
  TRY_GS(gs_ready(c));
  if (!psi || ncg < 1 || precondition < SB200_PRECOND_NONE || precondition > SB200_PRECOND_LEARNED)
    return set_error(SB200_ERR_INVALID_ARG, "sb200_gscg: bad argument");
  if (precondition == SB200_PRECOND_LEARNED && !c->learned_set)
    return set_error(SB200_ERR_STATE, "learned preconditioner weights not set");
  DevGuard dg(c->device);
  TRY_GS(gs_ensure(c, true));
  const long n = c->gs.n;
  double* w = c->gs.d_work;
  double *xk = w, *hxk = w + n, *pk = w + 2 * n, *gk = w + 3 * n, *pre = w + 4 * n, *pko = w + 5 * n,
         *hwf = w + 6 * n;
  const int norb = c->orb.norb, nblk = c->gs.nblk;
  const dim3 grid(nblk, norb), hg = dhpsi_grid(c);
  const int nh = (int)(hg.x * hg.y);
  // partial sums: <dir|g>, <x|pk>, <pko|pko>, the two of H, the two of the rotated x
  const size_t ob = (size_t)norb * nblk;
  double *p_xp = c->gs.d_part, *p_pp = p_xp + ob, *p_x = p_pp + ob, *p_h = p_x + 2 * ob, *p_gg = p_h + 2 * (size_t)norb * nh;
  CgArgs a;
  a.npts = c->g.npts;
  a.nx = c->g.nx;
  a.ny = c->g.ny;
  a.nz = c->g.nz;
  a.periodic = c->g.periodic;
  a.hz = dhpsi_hz(c);
  a.hvol = c->g.hvol;
  a.state = c->gs.d_coef;
  const double h0 = c->g.hgs[0], h1 = c->g.hgs[1], h2 = c->g.hgs[2];
  const double omega_d = 2.0 * (1.0 - alpha_pre) /
                         (-0.5 * ((-2.0) / (h0 * h0) + (-2.0) / (h1 * h1) + (-2.0) / (h2 * h2)));
  const double* x = psi;  // the first iteration reads psi, later ones the rotated xk
  TRY_GS(gs_hpsi(c, x, hxk, nullptr, x, p_h));
  for (int iter = 1; iter <= ncg; ++iter) {
    const double* prev = iter == 1 ? p_h : p_x;
    const int nprev = iter == 1 ? nh : nblk;
    double* keep = iter == 1 ? nullptr : psi;
    double* dir = precondition == SB200_PRECOND_LEARNED ? gk : pre;
    if (precondition == SB200_PRECOND_LOWPASS)
      k_cg_gradient<true><<<hg, HX * HY, 0, c->stream>>>(a, x, hxk, prev, nprev, keep, dir, 1.0 / (h0 * h0),
                                                         1.0 / (h1 * h1), 1.0 / (h2 * h2), omega_d, p_gg);
    else
      k_cg_gradient<false><<<hg, HX * HY, 0, c->stream>>>(a, x, hxk, prev, nprev, keep, dir, 1.0, 1.0, 1.0, 0.0,
                                                          p_gg);
    SB_LAUNCH_CHECK("k_cg_gradient");
    int ngg = nh;
    if (precondition == SB200_PRECOND_LEARNED) {
      ngg = nblk;
      TRY_GS(learned_precond_apply(c, gk, x, pre));
      k_cg_dot<<<grid, RT, 0, c->stream>>>(a, pre, gk, p_gg);
      SB_LAUNCH_CHECK("k_cg_dot");
      dir = pre;
    }
    // the network direction is not a fixed linear preconditioner: with it the
    // conjugation restarts every iteration (uk = 0, as in the first iteration)
    const int restart = iter == 1 || precondition == SB200_PRECOND_LEARNED;
    k_cg_direction<<<grid, RT, 0, c->stream>>>(a, dir, x, p_gg, ngg, iter, restart, pk, p_xp);
    SB_LAUNCH_CHECK("k_cg_direction");
    k_cg_orthogonal<<<grid, RT, 0, c->stream>>>(a, pk, x, p_xp, pko, p_pp);
    SB_LAUNCH_CHECK("k_cg_orthogonal");
    TRY_GS(gs_hpsi(c, pko, hwf, p_pp, x, p_h));
    k_cg_rotate<<<grid, RT, 0, c->stream>>>(a, x, xk, hxk, pko, hwf, p_pp, p_h, nh, p_x);
    SB_LAUNCH_CHECK("k_cg_rotate");
    x = xk;
  }
  k_cg_end<<<grid, RT, 0, c->stream>>>(a, x, p_x, nblk, psi, c->gs.d_dots);
  SB_LAUNCH_CHECK("k_cg_end");
  if (esp) SB_CUDA(cudaMemcpyAsync(esp, c->gs.d_dots, norb * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
  SB_CUDA(cudaStreamSynchronize(c->stream));
  return SB200_OK;
}

// gram_schmidt_col_real8 (gram_schmidt_orth.f90:59-230): classical GS, the
// coefficients of orbital io1 taken against its original vector.
int sb200_gram_schmidt_real(sb200_ctx* c, double* psi) {
  TRY_GS(gs_ready(c));
  if (!psi) return set_error(SB200_ERR_INVALID_ARG, "null psi");
  DevGuard dg(c->device);
  TRY_GS(gs_ensure(c, false));
  const int nspin = c->orb.nspin, no = c->orb.no;
  const long npts = c->g.npts;
  const size_t nn = (size_t)no * no;
  TRY_GS(gs_mat(c, 2 * nn + 2 * (size_t)no + 8));
  double* coeff = c->gs.d_mat;
  int* bad = (int*)(c->gs.d_mat + 2 * nn + 2 * (size_t)no);
  // orbitals of one spin are strided by nspin blocks: gather per spin
  double* buf = nullptr;
  if (nspin > 1) {
    TRY_GS(gs_ensure(c, true));
    buf = c->gs.d_work;  // [no][npts] of the current spin + 1 scratch block
  }
  for (int is = 0; is < nspin; ++is) {
    double* P = psi;
    if (nspin > 1) {
      for (int io = 0; io < no; ++io)
        SB_CUDA(cudaMemcpyAsync(buf + npts * io, psi + npts * ((long)io * nspin + is), sizeof(double) * npts,
                                cudaMemcpyDeviceToDevice, c->stream));
      P = buf;
    }
    TRY_GS(gs_orthonormalise(c, P, no, c->gs.d_mat, bad));
    int hbad = 0;
    SB_CUDA(cudaMemcpyAsync(&hbad, bad, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    SB_CUDA(cudaStreamSynchronize(c->stream));
    for (int io1 = 0; hbad && io1 < no; ++io1) {  // close to linear dependence: column by column
      double* w1 = P + npts * io1;
      if (io1 > 0) {
        // coeff(io2) = hvol <psi_io2 | psi_io1>, io2 < io1 ; w1 -= sum coeff * psi_io2
        TRY_GS(gs_gram(c, P, io1, w1, 1, c->g.hvol, coeff));
        TRY_GS(gs_rotate_sub(c, P, io1, coeff, w1));
      }
      TRY_GS(gs_norm_scale(c, w1, w1, 1));
    }
    if (nspin > 1)
      for (int io = 0; io < no; ++io)
        SB_CUDA(cudaMemcpyAsync(psi + npts * ((long)io * nspin + is), buf + npts * io, sizeof(double) * npts,
                                cudaMemcpyDeviceToDevice, c->stream));
  }
  SB_CUDA(cudaStreamSynchronize(c->stream));
  return SB200_OK;
}

}  // extern "C"

namespace sb200 {
// scratch of gs_complex_issue: part [no][nb], coeff [no]
size_t gs_complex_part_len(const sb200_ctx* c) {
  const long nb = (c->g.npts + DOT_PTS - 1) / DOT_PTS;
  return (size_t)c->orb.no * (size_t)nb;
}

// gram_schmidt_col_complex8's launches for every (k, spin) group, on the
// context's stream, with caller-given scratch: no allocation, no host wait
// (also issued inside the time loop's CUDA graph)
int gs_complex_issue(sb200_ctx* c, double2* z, double2* part, double2* coeff) {
  const int nspin = c->orb.nspin, no = c->orb.no, nk = c->orb.nk;
  const long npts = c->g.npts;
  const int nb = (int)((npts + DOT_PTS - 1) / DOT_PTS);
  const long stride = (long)nspin * npts;
  for (int ik = 0; ik < nk; ++ik)
    for (int is = 0; is < nspin; ++is) {
      double2* base = z + npts * ((long)is + (long)nspin * no * ik);
      for (int io1 = 0; io1 < no; ++io1) {
        double2* w1 = base + stride * io1;
        if (io1 > 0) {
          k_zgs_dots<<<dim3(nb, io1), RT, 0, c->stream>>>(base, stride, io1, npts, part, nb);
          k_zgs_coeff<<<(io1 + 127) / 128, 128, 0, c->stream>>>(part, nb, io1, c->g.hvol, coeff);
          k_zgs_sub<<<gridsz(npts), 256, 0, c->stream>>>(base, stride, io1, coeff, npts);
        }
        k_zsq_part<<<nb, RT, 0, c->stream>>>(w1, npts, (double*)part);
        k_zscale_norm<<<gridsz(npts), 256, 0, c->stream>>>(w1, npts, (const double*)part, nb, c->g.hvol);
      }
      const cudaError_t e = cudaGetLastError();
      if (e != cudaSuccess) return cuda_error(e, "complex Gram-Schmidt");
    }
  return SB200_OK;
}
}  // namespace sb200

extern "C" {

// gram_schmidt_col_complex8 (gram_schmidt_orth.f90:1069-1242) for every
// (k, spin) group of the complex orbital block, orbitals in order.
int sb200_gram_schmidt_complex(sb200_ctx* c, double* psi) {
  if (!c) return set_error(SB200_ERR_INVALID_ARG, "null ctx");
  if (!c->g.set || !c->orb.set) return set_error(SB200_ERR_STATE, "sb200_set_grid / _set_orbitals first");
  if (!psi) return set_error(SB200_ERR_INVALID_ARG, "null psi");
  DevGuard dg(c->device);
  const int nspin = c->orb.nspin, no = c->orb.no, nk = c->orb.nk;
  const long npts = c->g.npts;
  const int nb = (int)((npts + DOT_PTS - 1) / DOT_PTS);
  double2* part = nullptr;
  double2* coeff = nullptr;
  TRY_GS(dalloc(&part, (size_t)no * nb));
  int r = dalloc(&coeff, (size_t)no);
  (void)nspin;
  (void)nk;
  if (r == SB200_OK) r = gs_complex_issue(c, (double2*)psi, part, coeff);
  if (r == SB200_OK) {
    const cudaError_t e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) r = cuda_error(e, "complex Gram-Schmidt");
  }
  dfree(part);
  dfree(coeff);
  return r;
}

// ssdg_rwf (subspace_diagonalization.f90:62-238): H_sub = <psi_i|H|psi_j>,
// its eigenvectors on the GPU (sb200_eigh.cu), psi <- psi V, normalised.
// evals(no*nspin) host.
int sb200_subspace_diag_real(sb200_ctx* c, double* psi, double* evals) {
  TRY_GS(gs_ready(c));
  if (!psi) return set_error(SB200_ERR_INVALID_ARG, "null psi");
  DevGuard dg(c->device);
  TRY_GS(gs_ensure(c, true));
  const int nspin = c->orb.nspin, no = c->orb.no;
  if (nspin != 1) return set_error(SB200_ERR_UNSUPPORTED, "subspace diagonalisation implemented for nspin = 1");
  double* hpsi = c->gs.d_work;
  double* rot = c->gs.d_work + c->gs.n;
  TRY_GS(gs_hpsi(c, psi, hpsi));
  // work: M (no^2), V (no^2), eigensolver scratch (2 no^2), w (no), info
  const size_t nn = (size_t)no * no;
  TRY_GS(gs_mat(c, 4 * nn + no + 8));
  double* M = c->gs.d_mat;
  double* V = M + nn;
  double* ework = M + 2 * nn;
  double* w = M + 4 * nn;
  int* info = (int*)(w + no);
  TRY_GS(gs_gram(c, psi, no, hpsi, no, c->g.hvol, M, true));
  // M[i][j] row-major = <psi_i|H psi_j>; the eigensolver reads its upper
  // triangle (dsyev with uplo = 'U'), on the GPU
  TRY_GS(launch_eigh(c, M, no, ework, V, w, info));
  TRY_GS(gs_rotate(c, psi, no, V, no, 0.0, rot));
  TRY_GS(gs_norm_scale(c, rot, psi, no));
  std::vector<double> hw(no + 1);
  SB_CUDA(cudaMemcpyAsync(hw.data(), w, sizeof(double) * (no + 1), cudaMemcpyDeviceToHost, c->stream));
  SB_CUDA(cudaStreamSynchronize(c->stream));
  int hinfo = 0;
  std::memcpy(&hinfo, &hw[no], sizeof(int));
  if (hinfo != 0) return set_error(SB200_ERR_UNSUPPORTED, "subspace eigensolver: QL iterations did not converge");
  if (evals)
    for (int i = 0; i < no; ++i) evals[i] = hw[i];
  return SB200_OK;
}

}  // extern "C"
