// sb200_orbital_any.cu -- the fused Taylor step for periodic orthogonal grids
// of any extents whose orbital fits in the shared memory of a cluster of at
// most eight CTAs, taken where it is faster than the sweeps (any_us, sweep_us; 16^3
// grids have their own, sb200_orbital_blk.cu).
//
// One thread-block cluster applies all n_hamil terms of taylor.f90:47-117 to
// one orbital.  CTA r of the C in the cluster holds planes r nz / C ..
// (r + 1) nz / C - 1 of h_{n-1} in shared memory.  A thread owns an (x, y)
// column of the slab and marches up z with the nine z neighbours in registers;
// x and y neighbours come from the CTA's own planes, the four planes below and
// above the slab from the neighbour CTAs' shared memory (read once per column
// and term).  The stencil of a point goes to the thread's lane of tensor memory
// (TMEM), which also holds the Taylor accumulator psi_out, so neither registers
// nor shared memory carry them: orbitals of up to 8192 points a CTA fit.
//
// Per term: partial Kleinman-Bylander projections of the slab's sphere points
// (warps per atom; each atom's points are sorted by grid point, so a slab's
// part is one run) and the stencil sweep; cluster barrier; every CTA adds the C
// partial sums (a lane to each rank's), forms the contribution of each of its
// (point, atom) pairs, and the owners finish h_n = stencil + pairs, update
// psi_out and overwrite h_{n-1}; cluster barrier.  After the last term the
// observables of psi(t+dt), added over the cluster in rank order by CTA 0; its
// nonlocal current from the projections P of psi(t+dt), pair by pair:
// sum_j r_j Im(conj(e_j psi_j) sum_q uV_qj P_q), which is the sum over q of
// Im(conj(<r beta_q|psi>) P_q).  HBM: psi in, psi_out out.
//
// The KB tables are read twice a term, from L2 where they are large; STAGE keeps
// the slab's in shared memory (60 bytes a pair) where they fit beside the
// orbital: small cells, where a term is a chain of latencies (12^3 x 32 orbitals,
// a step with its observables: 41.5 -> 33 us).
//
// Bound inside the SM: per point and term 96 FP64 operations of the stencil
// (64 lanes a cycle) against 18 shared-memory loads of 16 bytes (128 bytes a
// cycle).
//
// Reference: zstencil_typical_seq (zstencil_core/typical/seq.f90:65-122),
// zpseudo (nonlocal_potential.f90:351-382), taylor (taylor.f90:47-117),
// stencil_current and calc_current_nonlocal (density_matrix.f90:465-591),
// calc_dip (dip.f90:114-225).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>
#include <vector>

#include "sb200_internal.cuh"
#include "sb200_orbital.cuh"
#include "sb200_tma.cuh"
#include "sb200_tmem.cuh"

namespace cg = cooperative_groups;

namespace sb200 {
namespace {

constexpr int MAX_NT = 512;
constexpr int MAX_NW = MAX_NT / 32;

struct AnyArgs {
  int nx, ny, nz, ncol;  // ncol = nx ny columns
  int rounds, dmax;      // columns per thread, largest slab
  int hmode;             // 1: out = H in (one term), 0: Taylor step
  unsigned tcols;        // TMEM columns of the CTA
  int tw;                // TMEM words per thread
  int npart;             // warps per atom in the projections
  long npts;
  int nspin, nspin_no, natom, nlma, totpts;
  double mhl[12], nab[12], off[3];  // -coef_lap / 2, coef_nab, dipole coordinate offsets
  const double* kcoef;
  const double* vloc;
  const int* pst;        // [natom][nz + 1] first flat sphere point of the atom at or above each plane
  const int* ppl;        // [nz + 1] first (point, atom) pair at or above each plane
  const int* pt_lin;
  const int* apj;        // [totpts] pair of each sphere point
  const double* uv4;     // [totpts][4]
  const double2* phase;  // [nk][totpts]
  const int *lma_start, *nproj;
  const double* rinv;
  int npair;
  const double2* pair_ph;  // [nk][npair]
  const double* pair_uv;   // [npair][4]
  const int* pair_lma;     // [npair] lma0 | nproj << 24
  const int* pair_pt;      // [npair] grid point
  const double* pair_r;    // [npair][3] coordinates
  const int* pmap2;        // [npts] (first pair << 8) | count, or -1
  int ahead;               // clusters at work at a time: the orbital that many on is fetched into L2
  double* obs;             // [norb][OBS_NQ]
  double* jw;              // [norb][3] or null
  int* err;
  // byte offsets into dynamic shared memory (after the slab)
  unsigned o_pc, o_part, o_proj, o_atom, o_ptab, o_rinv, o_pm, o_tab, o_idx;
  int maxpairs;            // most pairs of a slab
};
constexpr int NB = 4;     // sphere points, pairs or grid points of a thread in flight at once
constexpr int NSUM = 10;  // sums of an orbital: OBS_NQ and the nonlocal current

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// h += A (tp + tm) - i B (tp - tm)
__device__ __forceinline__ void pair_acc(double2& h, const double2 tp, const double2 tm, const double A,
                                         const double B) {
  const double sx = tp.x + tm.x, sy = tp.y + tm.y, dx = tp.x - tm.x, dy = tp.y - tm.y;
  h.x = fma(A, sx, h.x);
  h.y = fma(A, sy, h.y);
  h.x = fma(B, dy, h.x);
  h.y = fma(-B, dx, h.y);
}
__device__ __forceinline__ double cur_term(const double nab, const double2 c, const double2 t) {
  return nab * (c.x * t.y - c.y * t.x);
}

// sum of NV values over the warp by reduce-scatter: lane L ends with value
// L >> (5 - log2 NV) (fixed order)
template <int NV>
__device__ __forceinline__ double warp_scatter(double (&v)[NV], int lane) {
#pragma unroll
  for (int lev = 0; lev < 5; ++lev) {
    const int off = 16 >> lev, n = NV >> lev;
    if (n > 1) {
      const bool upper = (lane & off) != 0;
#pragma unroll
      for (int i = 0; i < n / 2; ++i) {
        const double keep = upper ? v[n / 2 + i] : v[i];
        const double send = upper ? v[i] : v[n / 2 + i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
      }
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
    }
  }
  return v[0];
}

__device__ __forceinline__ void cluster_barrier(int C) {
  if (C > 1) cg::this_cluster().sync();
  else __syncthreads();
}

// f(integral_constant<J>, k0 + J) for J = J0 .. N-1 while k0 + J < n
template <int J, int N, typename F>
__device__ __forceinline__ void unrolled(F& f, int k0, int n) {
  if constexpr (J < N) {
    if (k0 + J >= n) return;
    f(std::integral_constant<int, J>{}, k0 + J);
    unrolled<J + 1, N>(f, k0, n);
  }
}

// STAGE: the slab's KB tables stay in shared memory for the whole step
template <bool OBS, bool STAGE>
__global__ void __launch_bounds__(MAX_NT, 1) k_step_any(const double2* __restrict__ in, double2* __restrict__ out,
                                                        const __grid_constant__ AnyArgs a,
                                                        const __grid_constant__ StepZC zc, int nterm) {
  extern __shared__ __align__(128) unsigned char sraw[];
  double2* buf = (double2*)sraw;                   // [D][ncol] h_{n-1} of the slab
  double2* pc = (double2*)(sraw + a.o_pc);         // contribution of each of the slab's pairs
  double* ppart = (double*)(sraw + a.o_part);      // [natom npart][8] partial projections
  double2* sproj = (double2*)(sraw + a.o_proj);    // [nlma] projections
  int4* satm = (int4*)(sraw + a.o_atom);           // [natom] run of the slab (first, end), first ilma, projectors
  const double2** ptab = (const double2**)(sraw + a.o_ptab);  // [nz] plane pointers, own and the neighbours'
  double* srinv = (double*)(sraw + a.o_rinv);      // [nlma]
  int* spm = (int*)(sraw + a.o_pm);                // [D][ncol] point map of the slab
  // STAGE: per pair of the slab the phase and the four uV (three runs of 16 bytes)
  // and first ilma | projectors << 24; per sphere point its pair and its point
  double2* te = (double2*)(sraw + a.o_tab);
  double2* tu0 = te + a.maxpairs;
  double2* tu1 = tu0 + a.maxpairs;
  int* tlm = (int*)(tu1 + a.maxpairs);
  int2* tix = (int2*)(sraw + a.o_idx);
  int* sbase = (int*)ppart;  // (before the first projections)
  __shared__ uint32_t s_tmem;
  __shared__ __align__(16) double kn[12];
  __shared__ double red[NSUM][MAX_NW];
  __shared__ double osum[NSUM];
  __shared__ __align__(8) uint64_t s_bar;

  cg::cluster_group cl = cg::this_cluster();
  const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int NT = blockDim.x, NW = NT >> 5;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int o = (int)blockIdx.x / C;
  const int z0 = rank * a.nz / C, D = (rank + 1) * a.nz / C - z0;
  const int ncol = a.ncol;
  const int ik = o / a.nspin_no, ispin = o % a.nspin;
  const double* kc = a.kcoef + (long)KC * ik;
  const bool kb = a.nlma > 0;

  if (warp == 0) tmem::alloc(&s_tmem, a.tcols);
  if (t == 0) {
    tma::mbar_init(&s_bar, 1);
    tma::fence_barrier_init();
    const unsigned bytes = (unsigned)(D * ncol) * 16u;
    const double2* src = in + (long)o * a.npts + (long)z0 * ncol;
    tma::mbar_arrive_expect_tx(&s_bar, bytes);
    tma::bulk_load(buf, src, bytes, &s_bar);
    if (a.ahead > 0 && (o + a.ahead + 1) * C <= (int)gridDim.x)
      tma::bulk_prefetch_l2(src + (long)a.ahead * a.npts, bytes);
  }
  if (t < 12) kn[t] = __ldg(kc + 4 + t);
  if (kb) {
    for (int i = t; i < a.natom; i += NT) {
      const int* ps = a.pst + (long)i * (a.nz + 1);
      const int np = __ldg(a.nproj + i), j0 = __ldg(ps + z0);  // (no projectors: no pairs, an empty run)
      satm[i] = make_int4(j0, np > 0 ? __ldg(ps + z0 + D) : j0, __ldg(a.lma_start + i), np);
    }
    for (int i = t; i < a.nlma; i += NT) srinv[i] = __ldg(a.rinv + i);
#pragma unroll 8
    for (int i = t; i < D * ncol; i += NT) spm[i] = __ldg(a.pmap2 + (long)z0 * ncol + i);
  }
  for (int z = t; z < a.nz; z += NT) {
    int r = 0;
    while ((r + 1) * a.nz / C <= z) ++r;
    double2* mine = buf + (long)(z - r * a.nz / C) * ncol;  // the offset in rank r's slab
    ptab[z] = C > 1 ? cl.map_shared_rank(mine, r) : mine;
  }
  tmem::fence_before_sync();
  __syncthreads();
  tmem::fence_after_sync();
  const uint32_t tb = tmem::warp_addr(s_tmem, warp, (uint32_t)(warp >> 2) * (uint32_t)a.tw);
  const int pb0 = kb ? __ldg(a.ppl + z0) : 0, pb1 = kb ? __ldg(a.ppl + z0 + D) : 0;
  if (STAGE && kb) {
    for (int i = t; i < pb1 - pb0; i += NT) {
      const int pr = pb0 + i;
      te[i] = __ldg(a.pair_ph + (long)ik * a.npair + pr);
      tu0[i] = __ldg((const double2*)a.pair_uv + 2 * pr);
      tu1[i] = __ldg((const double2*)a.pair_uv + 2 * pr + 1);
      tlm[i] = __ldg(a.pair_lma + pr);
    }
    // the runs of the atoms one after the other; satm then counts in tix
    for (int atom = warp; atom < a.natom; atom += NW) {
      int n = 0;
      for (int i = lane; i < atom; i += 32) n += satm[i].y - satm[i].x;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) n += __shfl_xor_sync(0xffffffffu, n, off);
      const int4 at = satm[atom];
      for (int j = at.x + lane; j < at.y; j += 32)
        tix[n + j - at.x] = make_int2(__ldg(a.apj + j) - pb0, __ldg(a.pt_lin + j) - z0 * ncol);
      if (lane == 0) sbase[atom] = n;
    }
    __syncthreads();
    for (int i = t; i < a.natom; i += NT) {
      const int4 at = satm[i];
      satm[i] = make_int4(sbase[i], sbase[i] + at.y - at.x, at.z, at.w);
    }
  }
  const double2* ph = kb ? a.phase + (long)ik * a.totpts : nullptr;
  const double2* pph = kb ? a.pair_ph + (long)ik * a.npair : nullptr;
  if (!tma::mbar_wait(&s_bar, 0)) {  // bounded; the step goes on to its barriers with the flag set
    if (t == 0) atomicExch(a.err, 1);
    tma::mbar_wait(&s_bar, 0);
  }
  cluster_barrier(C);

  const double lap0 = __ldg(kc + 3);
  const double* vsl = a.vloc + (long)ispin * a.npts + (long)z0 * ncol;
  double2* osl = out + (long)o * a.npts + (long)z0 * ncol;

  // partial projections of the orbital in buf over the slab's sphere points
  auto project = [&]() {
    for (int task = warp; task < a.natom * a.npart; task += NW) {
      const int atom = task / a.npart, part = task - atom * a.npart;
      const int4 at = satm[atom];
      double v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = 0.0;
      // NB table loads in flight (past the run's end: its last point, weight zero)
      for (int j0 = at.x + 32 * part + lane; j0 < at.y; j0 += NB * 32 * a.npart) {
        double2 ev[NB], u0[NB], u1[NB];
#pragma unroll
        for (int i = 0; i < NB; ++i) {
          const int j = min(j0 + i * 32 * a.npart, at.y - 1);
          if (STAGE) {
            const int2 x = tix[j];
            ev[i] = cmul(te[x.x], buf[x.y]);
            u0[i] = tu0[x.x];
            u1[i] = tu1[x.x];
          } else {
            ev[i] = cmul(__ldg(ph + j), buf[__ldg(a.pt_lin + j) - z0 * ncol]);
            u0[i] = __ldg((const double2*)a.uv4 + 2 * j);
            u1[i] = __ldg((const double2*)a.uv4 + 2 * j + 1);
          }
        }
#pragma unroll
        for (int i = 0; i < NB; ++i) {
          if (j0 + i * 32 * a.npart >= at.y) ev[i] = make_double2(0.0, 0.0);
          v[0] = fma(u0[i].x, ev[i].x, v[0]);
          v[1] = fma(u0[i].x, ev[i].y, v[1]);
          v[2] = fma(u0[i].y, ev[i].x, v[2]);
          v[3] = fma(u0[i].y, ev[i].y, v[3]);
          v[4] = fma(u1[i].x, ev[i].x, v[4]);
          v[5] = fma(u1[i].x, ev[i].y, v[5]);
          v[6] = fma(u1[i].y, ev[i].x, v[6]);
          v[7] = fma(u1[i].y, ev[i].y, v[7]);
        }
      }
      const double r = warp_scatter<8>(v, lane);
      if ((lane & 3) == 0) ppart[8 * task + (lane >> 2)] = r;
    }
  };
  // the projections from the cluster's partial sums (after a cluster barrier)
  auto gather = [&]() {
    // C lanes to a projection, one per rank: the remote loads of all in flight at
    // once; added by butterfly over the ranks
    const int items = 4 * a.natom * C, r = t & (C - 1);
    const double* pr = C > 1 ? cl.map_shared_rank(ppart, r) : ppart;
    for (int i0 = warp * 32; i0 < items; i0 += NT) {
      const int i = (i0 + lane) / C, atom = i >> 2, q = i & 3;
      const int4 at = i0 + lane < items ? satm[atom] : make_int4(0, 0, 0, 0);
      double2 s = make_double2(0.0, 0.0);
      if (q < at.w)
        for (int p = 0; p < a.npart; ++p) {
          const double2 v = *(const double2*)(pr + 8 * (atom * a.npart + p) + 2 * q);
          s = make_double2(s.x + v.x, s.y + v.y);
        }
      for (int off = 1; off < C; off <<= 1) {
        s.x += __shfl_xor_sync(0xffffffffu, s.x, off);
        s.y += __shfl_xor_sync(0xffffffffu, s.y, off);
      }
      if (r == 0 && q < at.w) {
        const double rv = srinv[at.z + q];
        sproj[at.z + q] = make_double2(rv * s.x, rv * s.y);
      }
    }
    __syncthreads();
  };
  struct Pair {
    int lm;
    double2 e, u0, u1;
  };
  auto load_pair = [&](Pair& f, int pr) {
    if (STAGE) {
      f.lm = tlm[pr - pb0];
      f.e = te[pr - pb0];
      f.u0 = tu0[pr - pb0];
      f.u1 = tu1[pr - pb0];
      return;
    }
    f.lm = __ldg(a.pair_lma + pr);
    f.e = __ldg(pph + pr);
    f.u0 = __ldg((const double2*)a.pair_uv + 2 * pr);
    f.u1 = __ldg((const double2*)a.pair_uv + 2 * pr + 1);
  };
  // sum_q uV_q P_q of a pair
  auto pair_sum = [&](const Pair& f) {
    const double2* P = sproj + (f.lm & 0xffffff);
    const int np = f.lm >> 24;
    double2 s = make_double2(f.u0.x * P[0].x, f.u0.x * P[0].y);
    if (np > 1) s = make_double2(fma(f.u0.y, P[1].x, s.x), fma(f.u0.y, P[1].y, s.y));
    if (np > 2) s = make_double2(fma(f.u1.x, P[2].x, s.x), fma(f.u1.x, P[2].y, s.y));
    if (np > 3) s = make_double2(fma(f.u1.y, P[3].x, s.x), fma(f.u1.y, P[3].y, s.y));
    return s;
  };

  for (int nn = 0; nn < nterm; ++nn) {
    // h = -1/2 lap - i (k + A).grad + (V + lap0) of h_{n-1} into TMEM
    auto sweep = [&]() {
      for (int rd = 0; rd < a.rounds; ++rd) {
        const int c = min(rd * NT + t, ncol - 1);
        const int y = c / a.nx, x = c - y * a.nx;
        int xo[ND], yo[ND];  // element offsets of the neighbours + s (low half) and - s (high half)
#pragma unroll
        for (int s = 1; s <= ND; ++s) {
          const int xp = x + s < a.nx ? s : s - a.nx, xm = x - s >= 0 ? -s : a.nx - s;
          const int yp = (y + s < a.ny ? s : s - a.ny) * a.nx, ym = (y - s >= 0 ? -s : a.ny - s) * a.nx;
          xo[s - 1] = (xp & 0xffff) | (int)((unsigned)xm << 16);
          yo[s - 1] = (yp & 0xffff) | (int)((unsigned)ym << 16);
        }
        double2 w[2 * ND + 1];  // rolls through registers (steps unrolled by 3 or 9 cost more in fetches: 35, 40 : 33 us)
#pragma unroll
        for (int i = 0; i < 2 * ND; ++i) {
          int z = z0 - ND + i;
          z = z < 0 ? z + a.nz : (z >= a.nz ? z - a.nz : z);
          w[i] = ptab[z][c];
        }
        double dn = __ldg(vsl + c);
#pragma unroll 1
        for (int k = 0; k < D; ++k) {
          int z = z0 + k + ND;
          z = z >= a.nz ? z - a.nz : z;
          w[2 * ND] = ptab[z][c];
          const double2* P = buf + k * ncol + c;
          const double2 cv = w[ND];
          const double dg = dn + lap0;
          dn = __ldg(vsl + min(k + 1, D - 1) * ncol + c);
          // one accumulator per axis: chains of 8 dependent FMA instead of 24
          double2 hz = make_double2(dg * cv.x, dg * cv.y), hx = make_double2(0.0, 0.0), hy = hx;
#pragma unroll
          for (int s = 0; s < ND; s += 2) {  // the k-dependent coefficients two to a load
            const double2 kx = *(const double2*)(kn + s), ky = *(const double2*)(kn + 4 + s);
            const double2 kz = *(const double2*)(kn + 8 + s);
            pair_acc(hx, P[(short)xo[s]], P[xo[s] >> 16], a.mhl[s], kx.x);
            pair_acc(hy, P[(short)yo[s]], P[yo[s] >> 16], a.mhl[4 + s], ky.x);
            pair_acc(hz, w[ND + 1 + s], w[ND - 1 - s], a.mhl[8 + s], kz.x);
            pair_acc(hx, P[(short)xo[s + 1]], P[xo[s + 1] >> 16], a.mhl[s + 1], kx.y);
            pair_acc(hy, P[(short)yo[s + 1]], P[yo[s + 1] >> 16], a.mhl[5 + s], ky.y);
            pair_acc(hz, w[ND + 2 + s], w[ND - 2 - s], a.mhl[9 + s], kz.y);
          }
          const double2 h = make_double2((hx.x + hy.x) + hz.x, (hx.y + hy.y) + hz.y);
          const uint32_t ta = tb + 8 * (rd * a.dmax + k);
          if (nn == 0) {  // psi_out starts as psi
            const uint32_t hw[8] = {tmem::lo_word(h.x),  tmem::hi_word(h.x),  tmem::lo_word(h.y),  tmem::hi_word(h.y),
                                    tmem::lo_word(cv.x), tmem::hi_word(cv.x), tmem::lo_word(cv.y), tmem::hi_word(cv.y)};
            tmem::st8_async(ta, hw);
          } else {
            const uint32_t hw[4] = {tmem::lo_word(h.x), tmem::hi_word(h.x), tmem::lo_word(h.y), tmem::hi_word(h.y)};
            tmem::st4_async(ta, hw);
          }
#pragma unroll
          for (int i = 0; i < 2 * ND; ++i) w[i] = w[i + 1];
        }
      }
    };
    if (kb) project();
    sweep();
    tmem::st_wait();
    cluster_barrier(C);  // every read of h_{n-1} is done, every partial projection is there
    if (kb) {
      gather();
      for (int p0 = pb0 + t; p0 < pb1; p0 += NB * NT) {
        Pair f[NB];
#pragma unroll
        for (int i = 0; i < NB; ++i) load_pair(f[i], min(p0 + i * NT, pb1 - 1));
#pragma unroll
        for (int i = 0; i < NB; ++i) {
          const double2 v = cmul(make_double2(f[i].e.x, -f[i].e.y), pair_sum(f[i]));
          if (p0 + i * NT < pb1) pc[p0 + i * NT - pb0] = v;
        }
      }
      __syncthreads();
    }
    // ---- h_n, the Taylor update, h_n over h_{n-1} ----
    const bool last = nn == nterm - 1;
    double2 zn = zc.v[0];
#pragma unroll
    for (int q = 1; q < STEP_MAX_NTERM; ++q)
      if (nn == q) zn = zc.v[q];
    for (int rd = 0; rd < a.rounds; ++rd) {
      const int ci = rd * NT + t, c = min(ci, ncol - 1);
      const bool act = ci < ncol;
      auto finish = [&](auto nc, const int k) {
        constexpr int N = decltype(nc)::value;
        uint32_t w[8 * N];
        int pm[N];
        double2 c1[N];  // each point's first pair, loaded before any is used
        const uint32_t ta = tb + 8 * (rd * a.dmax + k);
        if constexpr (N == 4) tmem::ld32(ta, w);
        else tmem::ld8(ta, w);
#pragma unroll
        for (int i = 0; i < N; ++i) pm[i] = kb ? spm[(k + i) * ncol + c] : -1;
#pragma unroll
        for (int i = 0; i < N; ++i) c1[i] = pm[i] >= 0 ? pc[(pm[i] >> 8) - pb0] : make_double2(0.0, 0.0);
#pragma unroll
        for (int i = 0; i < N; ++i) {
          const int p = (k + i) * ncol + c;
          double2 h = make_double2(tmem::as_double(w[8 * i], w[8 * i + 1]) + c1[i].x,
                                   tmem::as_double(w[8 * i + 2], w[8 * i + 3]) + c1[i].y);
          if (pm[i] >= 0 && (pm[i] & 255) > 1) {  // the point's other pairs, atoms in ilma order
            const int p0 = (pm[i] >> 8) - pb0, p1 = p0 + (pm[i] & 255);
            for (int pr = p0 + 1; pr < p1; ++pr) h = make_double2(h.x + pc[pr].x, h.y + pc[pr].y);
          }
          const double2 ao = make_double2(tmem::as_double(w[8 * i + 4], w[8 * i + 5]),
                                          tmem::as_double(w[8 * i + 6], w[8 * i + 7]));
          const double2 an = make_double2(fma(zn.x, h.x, fma(-zn.y, h.y, ao.x)),
                                          fma(zn.x, h.y, fma(zn.y, h.x, ao.y)));
          if (last) {
            if (act) {
              osl[p] = a.hmode ? h : an;
              if (OBS) buf[p] = an;
            }
          } else {
            if (act) buf[p] = h;
            const uint32_t aw[4] = {tmem::lo_word(an.x), tmem::hi_word(an.x), tmem::lo_word(an.y),
                                    tmem::hi_word(an.y)};
            tmem::st4_async(ta + 8 * i + 4, aw);
          }
        }
      };
      int k = 0;
      for (; k + NB <= D; k += NB) finish(std::integral_constant<int, NB>{}, k);
      for (; k < D; ++k) finish(std::integral_constant<int, 1>{}, k);
    }
    tmem::st_wait();
    cluster_barrier(C);  // h_n (or psi(t + dt)) complete; the partial projections are free
  }

  if (OBS) {
    double q[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) q[i] = 0.0;
    auto local = [&]() {
      for (int rd = 0; rd < a.rounds; ++rd) {
        const int c = rd * NT + t;
        if (c >= ncol) continue;
        const int y = c / a.nx, x = c - y * a.nx;
        int xp[ND], yp[ND];
#pragma unroll
        for (int s = 1; s <= ND; ++s) {
          xp[s - 1] = x + s < a.nx ? s : s - a.nx;
          yp[s - 1] = (y + s < a.ny ? s : s - a.ny) * a.nx;
        }
        double2 w[ND + 1];
#pragma unroll
        for (int i = 0; i < ND; ++i) {
          const int z = z0 + i;
          w[i] = ptab[z >= a.nz ? z - a.nz : z][c];
        }
        const double fx = (double)x + a.off[0], fy = (double)y + a.off[1];
        auto step = [&](auto jc, const int k) {
          constexpr int j = decltype(jc)::value;
          const int z = z0 + k + ND;
          w[(j + ND) % (ND + 1)] = ptab[z >= a.nz ? z - a.nz : z][c];
          const double2* P = buf + k * ncol + c;
          const double2 cv = w[j];
          const double r2 = cv.x * cv.x + cv.y * cv.y;
          q[0] += r2;
          double jx = 0.0, jy = 0.0, jz = 0.0;
#pragma unroll
          for (int s = 0; s < ND; ++s) {
            jx += cur_term(a.nab[s], cv, P[xp[s]]);
            jy += cur_term(a.nab[4 + s], cv, P[yp[s]]);
            jz += cur_term(a.nab[8 + s], cv, w[(j + 1 + s) % (ND + 1)]);
          }
          q[1] += jx;
          q[2] += jy;
          q[3] += jz;
          q[4] = fma(fx, r2, q[4]);
          q[5] = fma(fy, r2, q[5]);
          q[6] = fma((double)(z0 + k) + a.off[2], r2, q[6]);
        };
        for (int k0 = 0; k0 < D; k0 += ND + 1) unrolled<0, ND + 1>(step, k0, D);
      }
    };
    if (kb) project();
    local();
    if (kb) {
      cluster_barrier(C);
      gather();
      for (int p0 = pb0 + t; p0 < pb1; p0 += NB * NT) {
        Pair f[NB];
        double2 ev[NB];
#pragma unroll
        for (int i = 0; i < NB; ++i) {
          const int pr = min(p0 + i * NT, pb1 - 1);
          load_pair(f[i], pr);
          ev[i] = cmul(f[i].e, buf[__ldg(a.pair_pt + pr) - z0 * ncol]);
        }
#pragma unroll
        for (int i = 0; i < NB; ++i) {
          const int pr = min(p0 + i * NT, pb1 - 1);
          const double2 s = pair_sum(f[i]);
          const double im = p0 + i * NT < pb1 ? ev[i].x * s.y - ev[i].y * s.x : 0.0;
          q[7] = fma(__ldg(a.pair_r + 3L * pr), im, q[7]);
          q[8] = fma(__ldg(a.pair_r + 3L * pr + 1), im, q[8]);
          q[9] = fma(__ldg(a.pair_r + 3L * pr + 2), im, q[9]);
        }
      }
    }
    const double r = warp_scatter<16>(q, lane);
    if ((lane & 1) == 0 && (lane >> 1) < NSUM) red[lane >> 1][warp] = r;
    __syncthreads();
    if (t < NSUM) {
      double s = 0.0;
      for (int w = 0; w < NW; ++w) s += red[t][w];
      osum[t] = s;
    }
    cluster_barrier(C);
    if (rank == 0 && t < NSUM) {
      double s = 0.0;
      for (int r2 = 0; r2 < C; ++r2) s += *(C > 1 ? cl.map_shared_rank(&osum[t], r2) : &osum[t]);
      if (t < OBS_NQ) a.obs[(long)o * OBS_NQ + t] = s;
      else if (a.jw != nullptr) a.jw[3L * o + t - OBS_NQ] = s;
    }
    cluster_barrier(C);  // no CTA leaves while CTA 0 reads its sums
  }
  tmem::fence_before_sync();
  __syncthreads();
  tmem::fence_after_sync();
  if (warp == 0) tmem::dealloc(s_tmem, a.tcols);
}

// Shape of the launch with clusters of C CTAs: false when the orbital does not fit.
struct AnyShape {
  int C = 0, NT = 0, rounds = 0, dmax = 0, tw = 0, npart = 1;
  bool stage = false;
  int maxpairs = 0;
  unsigned tcols = 0, o_tab = 0, o_idx = 0, o_pc = 0, o_part = 0, o_proj = 0, o_atom = 0, o_ptab = 0, o_rinv = 0, o_pm = 0;
  size_t smem = 0;
};

bool any_shape(const sb200_ctx* c, int C, bool stage, AnyShape* s) {
  const GridInfo& g = c->g;
  const PPInfo& pp = c->pp;
  if (C > g.nz) return false;
  const int ncol = g.nx * g.ny;
  s->C = C;
  s->dmax = (g.nz + C - 1) / C;
  s->rounds = (ncol + MAX_NT - 1) / MAX_NT;
  s->NT = ((ncol + s->rounds - 1) / s->rounds + 31) / 32 * 32;
  const int quads = (s->NT / 32 + 3) / 4;
  s->tw = 8 * s->rounds * s->dmax;
  s->tcols = 32;
  while ((int)s->tcols < quads * s->tw) s->tcols *= 2;
  if (s->tcols > 512) return false;
  const bool kb = pp.nlma > 0;
  const int natom = kb ? pp.natom : 0;
  s->npart = natom > 0 ? std::max(1, std::min(4, (s->NT / 32) / natom)) : 1;
  size_t pairs = 0;
  if (kb)
    for (int r = 0; r < C; ++r)
      pairs = std::max(pairs, (size_t)(pp.h_ppl[(r + 1) * g.nz / C] - pp.h_ppl[r * g.nz / C]));
  auto up = [](size_t v) { return (v + 15) & ~(size_t)15; };
  size_t off = (size_t)s->dmax * ncol * 16;
  s->o_pc = (unsigned)off;
  off += pairs * 16;
  s->o_part = (unsigned)off;
  off += up((size_t)natom * s->npart * 64);
  s->o_proj = (unsigned)off;
  off += up((size_t)(kb ? pp.nlma : 0) * 16);
  s->o_atom = (unsigned)off;
  off += (size_t)natom * 16;
  s->o_ptab = (unsigned)off;
  off += up((size_t)g.nz * 8);
  s->o_rinv = (unsigned)off;
  off += up((size_t)(kb ? pp.nlma : 0) * 8);
  s->o_pm = (unsigned)off;
  off += up(kb ? (size_t)s->dmax * ncol * 4 : 0);
  s->stage = stage && kb;
  s->maxpairs = (int)pairs;
  if (s->stage) {  // pairs and sphere points are one to one
    s->o_tab = (unsigned)off;
    off += up(pairs * 52);
    s->o_idx = (unsigned)off;
    off += up(pairs * 8);
  }
  // CTAs that share an SM share its 512 TMEM columns: each takes at least the
  // same share of its 228 KB of shared memory (1 KB of it the system's, some
  // static), so that an allocation never waits for another CTA's columns
  s->smem = std::max(off, (size_t)(228 * 1024) * s->tcols / 512 - 1024 - (size_t)c->any_static);
  return s->smem <= (size_t)c->any_smem_cap;
}

cudaLaunchConfig_t any_config(const AnyShape& s, int norb, cudaStream_t st, cudaLaunchAttribute* at) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(norb * s.C));
  cfg.blockDim = dim3((unsigned)s.NT);
  cfg.dynamicSmemBytes = s.smem;
  cfg.stream = st;
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = (unsigned)s.C;
  at->val.clusterDim.y = 1;
  at->val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}

// shared memory of the kernel: what a CTA may take at run time and its static part
// (the same for every device of this architecture)
void any_limits(sb200_ctx* c) {
  static const int stat = [] {
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, k_step_any<true, false>) != cudaSuccess) {
      cudaGetLastError();
      return -1;
    }
    return (int)fa.sharedSizeBytes;
  }();
  int optin = 0;
  if (stat < 0 || cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device) != cudaSuccess ||
      cudaFuncSetAttribute(k_step_any<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - stat) != cudaSuccess ||
      cudaFuncSetAttribute(k_step_any<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - stat) != cudaSuccess ||
      cudaFuncSetAttribute(k_step_any<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - stat) != cudaSuccess ||
      cudaFuncSetAttribute(k_step_any<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - stat) != cudaSuccess) {
    cudaGetLastError();
    c->any_smem_cap = 0;
    return;
  }
  c->any_static = stat;
  c->any_smem_cap = optin - stat;
}

// Clusters of the shape at work at a time (a cluster stays within a GPC, and GPUs
// differ in the SMs of theirs: 15 clusters of eight and 33 of four with one CTA per
// SM on the GPU of the figures below); 0: none.
int any_resident_clusters(const AnyShape& s, int norb, size_t smem) {
  cudaLaunchAttribute at;
  cudaLaunchConfig_t cfg = any_config(s, norb, nullptr, &at);
  cfg.dynamicSmemBytes = smem;
  int n = 0;
  const cudaError_t e = s.stage ? cudaOccupancyMaxActiveClusters(&n, k_step_any<true, true>, &cfg)
                                : cudaOccupancyMaxActiveClusters(&n, k_step_any<true, false>, &cfg);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

// Microseconds of a time step of four terms with its observables [0], or of one H psi
// [1], in clusters (any_us) and by the sweeps (sweep_us), from a fit to both over 12
// grids from 14^3 to 36^3 with 8 and 64 atoms, 1 to 300 orbitals.  In clusters,
// each wave: the barriers; per column of a thread the planes of the slab and eight of
// the neighbours', each bound by its own chain of loads (0.7) or by the shared-memory
// loads of the SM's warps; three passes over the slab's points; the turns of the
// warps over the atoms.  By the sweeps: waves of two CTAs an SM x planes with their
// halo, slower once psi and H psi leave L2, and the sphere points of the projections.
// Rms error 6 and 9 %.  Both sides meet where the last wave is nearly empty or where
// few large orbitals leave most SMs idle (us, clusters : sweeps, a step): 24^3 32
// orbitals 113 : 177, 34 orbitals 208 : 177; 36^3 1 orbital 149 : 132, 8 orbitals
// 148 : 211.  One H psi has a term only to pay for the cluster's prologue: 32^3
// 8 orbitals 29 : 23; 24^3 300 orbitals 283 : 202; 28^3 300 orbitals 303 : 329.
double any_us(const sb200_ctx* c, const AnyShape& s, int resident, int alone, int one) {
  static constexpr double K[2][7] = {{8.5, 0.5, 2.5, 13.6, 4.5, 3.2, 4.1}, {3.2, 2.0, 0.9, 3.4, 0.46, 0.9, 0.4}};
  const double* k = K[one];
  const int warps = s.NT / 32, natom = c->pp.nlma > 0 ? c->pp.natom : 0, ncol = c->g.nx * c->g.ny;
  const int turns = (natom * s.npart + warps - 1) / warps;
  auto wave = [&](int n) {  // of n clusters; more than `alone` share SMs
    const double share = n > alone ? 1.0 + 0.4 * ((resident + alone - 1) / alone - 1) : 1.0;
    const double plane = std::max(0.7, 0.07 * warps * share);
    return k[0] + (s.C > 1 ? k[1] : 0.0) + s.rounds * plane * (k[2] * s.dmax + k[3]) +
           share * (k[4] * 1e-3 * s.dmax * ncol + k[s.stage ? 5 : 6] * turns);
  };
  const int norb = c->orb.norb, rest = norb % resident;
  return (one ? 3.5 : 16.5) + (norb / resident) * wave(resident) + (rest > 0 ? wave(rest) : 0.0);
}

double sweep_us(const sb200_ctx* c, int one) {
  const int norb = c->orb.norb;
  const bool tma = tma_sweep_applies(c);
  const SweepShape s = tma ? tma_sweep_shape(c->g, norb, 296) : tiled_sweep_shape(c->g, norb);
  const long ctas = (long)s.ntiles * s.nzc * norb, rest = ctas % 296;
  const double waves = (double)(ctas / 296) + (rest == 0 ? 0.0 : (rest > 148 ? 1.0 : 0.8));
  const double out = std::min(1.0, std::max(0.0, (32.0 * norb * (double)c->g.npts - 60e6) / 126e6));
  const double points = 1e-6 * norb * (double)c->pp.totpts;
  const double h = (c->pp.nlma > 0 ? 0.0 : -3.5) +  // (no launch of projections)
                   (tma ? 9.0 + waves * (s.zchunk + 8) * (0.9 + 0.35 * out) + 25.0 * points
                        : 12.0 + waves * (s.zchunk + 8) * (1.1 + 0.5 * out) + 12.0 * points);
  return one ? h : 5.05 * h;
}

// Cluster sizes for the context's grid, orbitals and projectors, chosen at the first
// step after one of them was set.
void any_plan(sb200_ctx* c) {
  c->any_C[0] = c->any_C[1] = 0;
  const GridInfo& g = c->g;
  if (!g.set || !c->orb.set || !g.periodic) return;
  if (g.nx == 16 && g.ny == 16 && g.nz == 16) return;  // sb200_orbital_blk.cu
  const PPInfo& pp = c->pp;
  if (pp.nlma > 0 && (pp.npair <= 0 || pp.d_pst == nullptr)) return;  // no (point, atom) pair form
  if ((long)g.nx * g.ny > 4096) return;  // neighbour offsets in 16 bits
  const int asked = c->cluster_asked;  // this size wherever it fits; 0: the sweeps
  if (asked == 0) return;
  any_limits(c);
  if (c->any_smem_cap == 0) return;
  double best[2] = {sweep_us(c, 0), sweep_us(c, 1)};
  if (asked > 0) best[0] = best[1] = 1e30;
  for (int C = 1; C <= 8; C *= 2) {
    AnyShape s;
    if (asked > 0 && asked != C) continue;
    // with the tables in shared memory where they fit
    if (!any_shape(c, C, true, &s) && !any_shape(c, C, false, &s)) continue;
    const int resident = any_resident_clusters(s, c->orb.norb, s.smem);
    const int alone = any_resident_clusters(s, c->orb.norb, (size_t)c->any_smem_cap);  // one CTA per SM
    if (resident < 1 || alone < 1) continue;
    for (int one = 0; one < 2; ++one) {
      const double us = any_us(c, s, resident, alone, one);
      if (us < best[one]) {
        best[one] = us;
        c->any_C[one] = C;
        c->any_resident[one] = resident;
      }
    }
  }
}

}  // namespace

bool step_any_applies(sb200_ctx* c, int n_hamil) {
  if (c->g.nonorth || c->microac || c->cap_on || c->stencil_variant != 1 || c->sweep_asked ||
      c->project_variant != 1 || c->precision != SB200_PREC_FP64 || n_hamil < 1 || n_hamil > STEP_MAX_NTERM)
    return false;
  if (c->any_C[0] < 0) any_plan(c);
  return c->any_C[n_hamil == 1] > 0;
}

// hmode: out = H in; else the Taylor step, with_obs: its observables too
int launch_step_any(sb200_ctx* c, const double2* in, double2* out, const double2* zc, int n_hamil, bool with_obs,
                    bool hmode) {
  AnyShape s;
  const int one = n_hamil == 1, C = c->any_C[one];
  if (!any_shape(c, C, true, &s) && !any_shape(c, C, false, &s))
    return set_error(SB200_ERR_BAD_SHAPE, "fused step: the orbital does not fit");
  const GridInfo& g = c->g;
  const PPInfo& pp = c->pp;
  AnyArgs a;
  a.nx = g.nx;
  a.ny = g.ny;
  a.nz = g.nz;
  a.ncol = g.nx * g.ny;
  a.rounds = s.rounds;
  a.dmax = s.dmax;
  a.hmode = hmode ? 1 : 0;
  a.tcols = s.tcols;
  a.tw = s.tw;
  a.npart = s.npart;
  a.npts = g.npts;
  a.nspin = c->orb.nspin;
  a.nspin_no = c->orb.nspin * c->orb.no;
  a.natom = pp.nlma > 0 ? pp.natom : 0;
  a.nlma = pp.nlma;
  a.totpts = pp.totpts;
  for (int i = 0; i < 12; ++i) {
    a.mhl[i] = -0.5 * g.coef_lap[i];
    a.nab[i] = g.coef_nab[i];
  }
  for (int d = 0; d < 3; ++d) a.off[d] = (double)g.is[d] - ((g.lg_num[d] % 2 == 1) ? 0.0 : 0.5);
  a.kcoef = c->d_kcoef;
  a.vloc = c->d_vloc;
  a.pst = pp.d_pst;
  a.ppl = pp.d_ppl;
  a.pt_lin = pp.d_pt_lin;
  a.uv4 = pp.d_uv4;
  a.phase = pp.d_phase;
  a.lma_start = pp.d_lma_start;
  a.nproj = pp.d_nproj;
  a.rinv = pp.d_rinv;
  a.npair = pp.npair;
  a.pair_ph = pp.d_pair_ph;
  a.pair_uv = pp.d_pair_uv;
  a.pair_lma = pp.d_pair_lma;
  a.pmap2 = pp.d_pmap2;
  a.obs = with_obs ? c->d_obs : nullptr;
  a.jw = (with_obs && pp.nlma > 0) ? c->d_jw : nullptr;
  a.err = c->d_err;
  a.o_pc = s.o_pc;
  a.o_part = s.o_part;
  a.o_proj = s.o_proj;
  a.o_atom = s.o_atom;
  a.o_ptab = s.o_ptab;
  a.o_tab = s.o_tab;
  a.o_idx = s.o_idx;
  a.maxpairs = s.maxpairs;
  a.apj = pp.d_apj;
  a.o_rinv = s.o_rinv;
  a.o_pm = s.o_pm;
  a.pair_pt = pp.d_pair_pt;
  a.pair_r = pp.d_pair_r;
  a.ahead = c->any_resident[one];
  StepZC z;
  for (int i = 0; i < STEP_MAX_NTERM; ++i) z.v[i] = (zc && i < n_hamil) ? zc[i] : make_double2(0.0, 0.0);
  cudaLaunchAttribute at;
  const cudaLaunchConfig_t cfg = any_config(s, c->orb.norb, c->stream, &at);
  void (*fn)(const double2*, double2*, AnyArgs, StepZC, int) =
      with_obs ? (s.stage ? k_step_any<true, true> : k_step_any<true, false>)
               : (s.stage ? k_step_any<false, true> : k_step_any<false, false>);
  SB_CUDA(cudaLaunchKernelEx(&cfg, fn, in, out, a, z, n_hamil));
  return SB200_OK;
}

}  // namespace sb200
