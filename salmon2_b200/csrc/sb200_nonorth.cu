// sb200_nonorth.cu -- H psi on a non-orthogonal lattice (zstencil_nonorthogonal,
// stencil.f90:120-214, called from hamiltonian.f90:306-357) in one sweep:
//
//   h = (V + k_lap0) psi - 1/2 sum_d F_d v_d - i sum_d Bk_d w_d
//       - 1/2 (F_4 d_z w_y + F_5 d_z w_x + F_6 d_x w_y),   Bk = B (k + A)
//
// with v_d the lattice-axis Laplacian sums and w_d the first derivatives, then
// the KB term and the Taylor epilogue of MODE (modes of sb200_internal.cuh).
//
// A CTA owns a w x h column tile of one orbital, a thread a column, and takes the
// planes of a z chunk in order, each brought with its wrapped 4-point halo by
// cp.async into a ring of four.  Everything a plane contributes within itself is
// formed when it arrives: v_x, v_y, w_x, w_y of the thread's column; w_y (halo
// columns included) also goes to shared memory, from which the next step takes
// d_x w_y (the reference's d_y w_x is the same sum), so a step has one barrier.
// Its part in the z sums of the four planes below and above, with -1/2 F_3 v_z on
// psi and d_z on g = -i Bk_z psi - 1/2 (F_4 w_y + F_5 w_x), is added to nine
// running values of h that rotate through registers, and the plane four below is
// then done.  The chunk's halo planes take w_x and w_y only.  So psi is read about
// once and nothing but h and the accumulator is written, where two passes over
// stored derivatives moved nine blocks (24^3 x 128 orbitals: 120 -> 67 us a term).  Bound by
// the instructions and shared-memory loads of a point (26 of 16 bytes); the tile
// is the one of the least time by a model of both (tile_shape).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "sb200_internal.cuh"
#include "sb200_stencil.cuh"
#include "sb200_tiled_body.cuh"

namespace sb200 {
namespace {

using namespace tiled;

constexpr int MAX_NT = 256;  // two CTAs an SM, 128 registers a thread (112 spill: 84 -> 67 us below)
constexpr int REGS = 128;
constexpr int RING = 4;      // planes resident or in flight
constexpr int SLOTS = 4;     // plane values a thread copies at most
constexpr int SMEM_LIMIT = 200 * 1024;  // of every tile: the kernel's limit is shared by all contexts

struct NoArgs {
  int w, h;  // tile
  double F[6];
  double lz[ND];  // -1/2 F_3 coef_lap along the third axis
};

__device__ __forceinline__ void copy16(double2* dst, const double2* src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

template <int MODE>
__global__ void __launch_bounds__(MAX_NT, 2) k_hpsi_no(const double2* __restrict__ in, double2* __restrict__ hout,
                                                      double2* __restrict__ acc, const __grid_constant__ TiledArgs a,
                                                      const __grid_constant__ NoArgs n) {
  extern __shared__ __align__(16) double2 sm[];
  const int NT = blockDim.x, t = threadIdx.x;
  const int SX = n.w + 2 * ND, PLANE = SX * (n.h + 2 * ND), ROWS = SX * n.h;
  double2* wybuf = sm + RING * PLANE;  // w_y of the tile's rows, halo columns included, of two planes
  const bool mine = t < n.w * n.h;
  const int ty = mine ? t / n.w : 0, tx = mine ? t - ty * n.w : 0;
  const int ntx = (a.nx + n.w - 1) / n.w;
  const int x0 = ((int)blockIdx.x % ntx) * n.w, y0 = ((int)blockIdx.x / ntx) * n.h;
  const int x = x0 + tx, y = y0 + ty;
  const bool active = mine && x < a.nx && y < a.ny;
  const int zc0 = blockIdx.y * a.zchunk, zc1 = min(a.nz, zc0 + a.zchunk);
  const int ntot = zc1 - zc0 + 2 * ND;  // input planes zc0 - 4 .. zc1 + 3
  const int o = blockIdx.z, ik = o / a.nspin_no, ispin = o % a.nspin;
  const double* kc = a.kcoef + (long)KC * ik;
  const double Bx = kc[16], By = kc[17], Bz = kc[18], lap0 = kc[3];
  const int plane = a.nx * a.ny, pxy = active ? y * a.nx + x : 0;
  const double2* src = in + (long)o * a.npts;
  int goff[SLOTS];
#pragma unroll
  for (int i = 0; i < SLOTS; ++i) {
    const int e = t + i * NT, hx = e % SX, hy = e / SX;
    int gx = (x0 - ND + hx) % a.nx, gy = (y0 - ND + hy) % a.ny;
    if (gx < 0) gx += a.nx;
    if (gy < 0) gy += a.ny;
    goff[i] = gy * a.nx + gx;
  }
  int zi = (zc0 - ND) % a.nz;  // plane of the next copy, wrapped
  if (zi < 0) zi += a.nz;
  auto issue = [&](int p) {
    if (p < ntot) {
      const double2* s = src + (long)zi * plane;
      zi = zi + 1 < a.nz ? zi + 1 : 0;
      double2* d = sm + (p & (RING - 1)) * PLANE;
#pragma unroll
      for (int i = 0; i < SLOTS; ++i)
        if (t + i * NT < PLANE) copy16(d + t + i * NT, s + goff[i]);
    }
    copy_commit();
  };
  for (int p = 0; p < RING - 1; ++p) issue(p);
  const double* V = a.vloc + (long)ispin * a.npts;
  const double2* pair_ph = a.use_pairs ? a.pair_ph + (long)ik * a.npair : nullptr;
  const double2* proj = a.nlma > 0 ? a.proj + (long)o * a.nlma : nullptr;
  int pm_n = a.nlma > 0 ? __ldg(a.pmap + (long)zc0 * plane + pxy) : -1;
  Pair1<double> f1;
  f1.lm = 0;
  if (a.use_pairs) load_pair1<double>(f1, pm_n, a, pair_ph);
  const int row = ty * SX + tx + ND, ctr = row + ND * SX;
  const double hF0 = -0.5 * n.F[0], hF1 = -0.5 * n.F[1], hF5 = -0.5 * n.F[5];
  const double hF3 = -0.5 * n.F[3], hF4 = -0.5 * n.F[4];
  double2 h[2 * ND + 1];  // h of planes p - 4 .. p + 4 so far
#pragma unroll
  for (int i = 0; i < 2 * ND + 1; ++i) h[i] = make_double2(0.0, 0.0);
  auto potential = [&](int p) {  // V of input plane p at this thread's point
    const int z = min(max(zc0 - ND + p, 0), a.nz - 1);
    return __ldg(V + (long)z * plane + pxy);
  };
  double vl_n = potential(0);
#pragma unroll 1
  for (int p = 0; p < ntot; ++p) {
    const int z = zc0 + p - 2 * ND;  // the output plane of this step (from p = 8 on)
    const bool emit = p >= 2 * ND && active;
    const long gi = (long)o * a.npts + (long)z * plane + pxy;
    double2 ac = make_double2(0.0, 0.0);
    int pm = -1;
    if (emit) {
      if (MODE == 2 || MODE == 3) ac = acc[gi];
      if (MODE == 1 || MODE == 4) ac = __ldg(in + gi);
      pm = pm_n;
      if (a.nlma > 0 && z + 1 < zc1) pm_n = __ldg(a.pmap + (long)(z + 1) * plane + pxy);
    }
    const double dg = vl_n + lap0;
    vl_n = potential(p + 1);
    copy_wait<RING - 2>();
    __syncthreads();  // plane p and w_y of plane p - 1 are there; every warp is done with plane p - 1
    issue(p + RING - 1);
    const double2* P = sm + (p & (RING - 1)) * PLANE;
    double2* W = wybuf + (p & 1) * ROWS;
    const bool inner = p >= ND && p < ntot - ND;  // an output plane, not a halo plane of the chunk
    double2 wx = make_double2(0.0, 0.0), wy = wx;
    const double2 c = P[ctr];
    if (inner) {
      double2 vx = wx, vy = wx;
#pragma unroll
      for (int s = 1; s <= ND; ++s) {
        const double2 xp = P[ctr + s], xm = P[ctr - s], yp = P[ctr + s * SX], ym = P[ctr - s * SX];
        vx = cfma(a.lapt[s - 1], cadd(xp, xm), vx);
        wx = cfma(a.nab[s - 1], csub(xp, xm), wx);
        vy = cfma(a.lapt[3 + s], cadd(yp, ym), vy);
        wy = cfma(a.nab[3 + s], csub(yp, ym), wy);
      }
      if (mine) W[row] = wy;
      for (int e = t; e < 2 * ND * n.h; e += NT) {  // the rows' halo columns
        const int hy = e / (2 * ND), hx = e % (2 * ND), hr = hy * SX + (hx < ND ? hx : n.w + hx);
        const double2* Q = P + ND * SX + hr;
        double2 wh = make_double2(0.0, 0.0);
#pragma unroll
        for (int s = 1; s <= ND; ++s) wh = cfma(a.nab[3 + s], csub(Q[s * SX], Q[-s * SX]), wh);
        W[hr] = wh;
      }
      const double2 bw = cfma(By, wy, cscal(Bx, wx));
      double2 r = cfma(dg, c, cfma(hF1, vy, cscal(hF0, vx)));
      r.x += bw.y;
      r.y -= bw.x;
      h[ND] = cadd(h[ND], r);
    } else {
#pragma unroll
      for (int s = 1; s <= ND; ++s) {
        wx = cfma(a.nab[s - 1], csub(P[ctr + s], P[ctr - s]), wx);
        wy = cfma(a.nab[3 + s], csub(P[ctr + s * SX], P[ctr - s * SX]), wy);
      }
    }
    if (p > ND && p <= ntot - ND) {  // the mixed derivative of plane p - 1
      const double2* M = wybuf + ((p - 1) & 1) * ROWS + row;
      double2 mix = make_double2(0.0, 0.0);
#pragma unroll
      for (int s = 1; s <= ND; ++s) mix = cfma(a.nab[s - 1], csub(M[s], M[-s]), mix);
      h[ND - 1] = cfma(hF5, mix, h[ND - 1]);
    }
    const double2 g = make_double2(fma(Bz, c.y, fma(hF4, wx.x, hF3 * wy.x)),
                                   fma(-Bz, c.x, fma(hF4, wx.y, hF3 * wy.y)));
    h[2 * ND] = make_double2(0.0, 0.0);
#pragma unroll
    for (int s = 1; s <= ND; ++s) {
      const double nz = a.nab[7 + s];
      h[ND - s] = cfma(nz, g, cfma(n.lz[s - 1], c, h[ND - s]));
      h[ND + s] = cfma(-nz, g, cfma(n.lz[s - 1], c, h[ND + s]));
    }
    if (emit) {
      double2 r = h[0];
      if (pm >= 0) {
        if (a.use_pairs) {
          r = kb_pairs_ahead<double>(r, pm, proj, a, ik, f1);
        } else {
          const double2* zk = a.ent_zk + (long)ik * a.nent;
          const int e1 = (pm >> 8) + (pm & 255);
          for (int e = pm >> 8; e < e1; ++e) r = cadd(r, cmul(proj[__ldg(a.ent_lma + e)], __ldg(zk + e)));
        }
      }
      if (MODE <= 2) hout[gi] = r;
      if (MODE != 0) acc[gi] = cadd(ac, cmul(a.zc, r));
      if (a.use_pairs && z + 1 < zc1) load_pair1<double>(f1, pm_n, a, pair_ph);
    }
#pragma unroll
    for (int i = 0; i < 2 * ND; ++i) h[i] = h[i + 1];
  }
}

// The tile and z chunk of the least time: per wave, planes (8 halo planes each chunk)
// x a chain of 1.3 us, longer with the warps behind the CTA's barrier, with the SM's
// warps, the values it copies a plane, and the warps whose groups of eight threads
// straddle rows of the tile (bank conflicts: tiles as wide as the row or a multiple
// of eight wide are the better ones).  The weights are a fit to 2600 pairs of tile
// and chunk on 13 lattices from 9 x 11 x 30 to 40^3, 1 to 200 orbitals; the tile
// chosen is 1.3 % slower than the best of them on average, 10 % at most.  A thread copies at most SLOTS values of a plane, so
// narrow tiles get some threads without a column.  H psi, us, the best tile and the
// one of the least waves x warps x planes with four planes a chunk at least: 26^3 x
// 2 orbitals 17.5 and 26, x 32 45 and 53; 20^3 x 64 43 and 53; 24^3 x 128 83 both
// (8 x 8, whole columns).
NonorthTile tile_shape(const GridInfo& g, int norb) {
  NonorthTile best;
  double least = 0.0;
  for (int kx = (g.nx + 63) / 64; kx <= 1 + g.nx / 8; ++kx) {
    const int w = (g.nx + kx - 1) / kx;
    for (int ky = (g.ny * w + MAX_NT - 1) / MAX_NT, h1 = 0; ky <= g.ny; ++ky) {
      const int h = (g.ny + ky - 1) / ky;
      if (h == h1) continue;
      h1 = h;
      NonorthTile k;
      k.w = w;
      k.h = h;
      const int area = (w + 2 * ND) * (h + 2 * ND);
      k.NT = (std::max(w * h, (area + SLOTS - 1) / SLOTS) + 31) / 32 * 32;
      k.smem = ((size_t)RING * area + 2 * (size_t)(w + 2 * ND) * h) * sizeof(double2);
      if (k.NT > MAX_NT) continue;
      const int per_sm = std::min(std::min(32, 65536 / (REGS * k.NT)), (int)(SMEM_LIMIT / k.smem));
      const int groups = std::max(1, w * h / 8);
      int straddle = 0;
      for (int i = 0; i < groups; ++i) straddle += i * 8 / w != (i * 8 + 7) / w;
      const double per_cta = 0.005 * (k.NT / 32) + 0.2e-3 * area + 0.013 * ((w * h + 31) / 32) * straddle / groups;
      const double chain = 1.3 + 0.014 * (k.NT / 32);
      const long tiles = (long)((g.nx + w - 1) / w) * ((g.ny + h - 1) / h), slots = 148L * per_sm;
      for (int nchunk = 1, zc1 = 0; nchunk <= g.nz; ++nchunk) {
        const int zc = (g.nz + nchunk - 1) / nchunk;
        if (zc == zc1) continue;
        zc1 = zc;
        k.nchunk = nchunk;
        const long ctas = tiles * norb * ((g.nz + zc - 1) / zc), rest = ctas % slots;
        const double cost = (zc + 2 * ND) * ((double)(ctas / slots) * (chain + per_sm * per_cta) +
                                             (rest > 0 ? chain + (double)((rest + 147) / 148) * per_cta : 0.0));
        if (best.w == 0 || cost < least) {
          least = cost;
          best = k;
        }
      }
    }
  }
  return best;
}

template <int MODE>
int launch_mode(const HpsiLaunch& L, const TiledArgs& a, const NoArgs& n, const NonorthTile& k, dim3 grid, cudaStream_t st) {
  SB_CUDA(cudaFuncSetAttribute(k_hpsi_no<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT));
  k_hpsi_no<MODE><<<grid, k.NT, k.smem, st>>>((const double2*)L.in, (double2*)L.hout, L.out, a, n);
  SB_LAUNCH_CHECK("k_hpsi_no");
  return SB200_OK;
}

}  // namespace

int launch_hpsi_nonorth(sb200_ctx* c, const HpsiLaunch& L) {
  if (L.mode > 4) return set_error(SB200_ERR_UNSUPPORTED, "the non-orthogonal hpsi has no mixed-precision modes");
  TiledArgs a = make_tiled_args(c, L.zc);
  const GridInfo& g = c->g;
  if (c->no_tile.w == 0) c->no_tile = tile_shape(g, c->orb.norb);
  const NonorthTile& k = c->no_tile;
  NoArgs n;
  n.w = k.w;
  n.h = k.h;
  for (int i = 0; i < 6; ++i) n.F[i] = g.coefF[i];
  for (int i = 0; i < ND; ++i) n.lz[i] = -0.5 * g.coefF[2] * g.coef_lap[8 + i];
  a.zchunk = (g.nz + k.nchunk - 1) / k.nchunk;
  const long tiles = (long)((g.nx + k.w - 1) / k.w) * ((g.ny + k.h - 1) / k.h);
  const dim3 grid((unsigned)tiles, (unsigned)((g.nz + a.zchunk - 1) / a.zchunk), (unsigned)c->orb.norb);
  switch (L.mode) {
    case 0: return launch_mode<0>(L, a, n, k, grid, c->stream);
    case 1: return launch_mode<1>(L, a, n, k, grid, c->stream);
    case 2: return launch_mode<2>(L, a, n, k, grid, c->stream);
    case 3: return launch_mode<3>(L, a, n, k, grid, c->stream);
    default: return launch_mode<4>(L, a, n, k, grid, c->stream);
  }
}

}  // namespace sb200
