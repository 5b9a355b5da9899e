// sb200_tma_body.cuh -- the TMA-fed tiled hpsi sweep as a device function,
// shared by the per-system kernel (sb200_tma_stencil.cu) and the batched
// persistent kernel (sb200_batch.cu).  See sb200_tma_stencil.cu for the design.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "sb200_internal.cuh"
#include "sb200_stencil.cuh"
#include "sb200_tiled_body.cuh"
#include "sb200_tma.cuh"

namespace sb200 {
namespace tmak {


using namespace tiled;

constexpr int TX = 32, TY = 8, NT = TX * TY, HALO = ND;
constexpr int RING = 8;   // input planes resident / in flight
constexpr int ARING = 4;  // accumulator planes in flight
constexpr int TMA_PLANES = 2;  // planes per step on isolated grids
constexpr int TMA_UNROLL = 2;  // plane steps unrolled in the FP64 modes of periodic grids
constexpr int TMA_MAX_NLMA = 512;  // projections staged in shared memory (else read from global)

struct TmaMaps {
  CUtensorMap in;    // input planes: (2 SX) x SY box, or (2 TX) x TY for the periodic centre rows
  CUtensorMap inh;   // periodic: (2 TX) x 4 halo rows
  CUtensorMap acc;   // FP64 accumulator tile (2 TX) x TY
  CUtensorMap d32;   // FP32 correction tile (2 TX) x TY
};

template <int MODE, bool PER>
struct Geo {
  using R = typename ModeT<MODE>::R;
  using C2 = typename Cx<R>::T;
  static constexpr int SX = PER ? TX : TX + 2 * HALO;
  static constexpr int SY = TY + 2 * HALO;
  static constexpr int PLANE = SX * SY;  // complex values per ring slot
  static constexpr unsigned PLANE_BYTES = PLANE * sizeof(C2);
  // psi_out by tensor copy; isolated grids (two planes a step) load it at the step's
  // start instead: a ring deep enough for two planes a step would not fit twice
  static constexpr bool ACC64 = ((MODE == 2 || MODE == 3) && PER) || MODE == 8;
  static constexpr bool ACC_LD = (MODE == 2 || MODE == 3) && !PER;
  static constexpr bool D32 = (MODE == 7 || MODE == 8);                 // reads the FP32 correction
  static constexpr unsigned ACC_BYTES = ACC64 ? NT * 16u : 0u;
  static constexpr unsigned D32_BYTES = D32 ? NT * 8u : 0u;
  static constexpr size_t RING_OFF = 0;
  static constexpr size_t ACC_OFF = RING_OFF + (size_t)RING * PLANE_BYTES;
  static constexpr size_t D32_OFF = ACC_OFF + (size_t)ARING * ACC_BYTES;
  static constexpr size_t BAR_OFF = D32_OFF + (size_t)ARING * D32_BYTES;
  static constexpr size_t PS_OFF = BAR_OFF + 256;  // projections of the item's orbital
  static constexpr size_t SMEM = PS_OFF + (size_t)TMA_MAX_NLMA * 16 + 128;  // + alignment slack
};

template <int MODE, bool PER>
__device__ __forceinline__ void issue_plane(const TmaMaps& m, unsigned char* base, uint64_t* pbar, int r, int q,
                                            int x0, int y0, int o, int nz, int ny) {
  using G = Geo<MODE, PER>;
  const int slot = r & (RING - 1);
  unsigned char* dst = base + G::RING_OFF + (size_t)slot * G::PLANE_BYTES;
  tma::mbar_arrive_expect_tx(&pbar[slot], G::PLANE_BYTES);
  if (!PER) {
    tma::tensor_load_4d(dst, &m.in, 2 * (x0 - HALO), y0 - HALO, q, o, &pbar[slot]);
  } else {
    int qz = q % nz;
    if (qz < 0) qz += nz;
    const int ya = y0 - HALO < 0 ? y0 - HALO + ny : y0 - HALO;
    const int yb = y0 + TY >= ny ? y0 + TY - ny : y0 + TY;
    constexpr size_t ROW = (size_t)TX * sizeof(typename G::C2);
    tma::tensor_load_4d(dst, &m.inh, 0, ya, qz, o, &pbar[slot]);
    tma::tensor_load_4d(dst + HALO * ROW, &m.in, 0, y0, qz, o, &pbar[slot]);
    tma::tensor_load_4d(dst + (HALO + TY) * ROW, &m.inh, 0, yb, qz, o, &pbar[slot]);
  }
}

template <int MODE, bool PER>
__device__ __forceinline__ void issue_acc(const TmaMaps& m, unsigned char* base, uint64_t* abar, int k, int z,
                                          int x0, int y0, int o) {
  using G = Geo<MODE, PER>;
  const int slot = k & (ARING - 1);
  tma::mbar_arrive_expect_tx(&abar[slot], G::ACC_BYTES + G::D32_BYTES);
  if (G::ACC64) tma::tensor_load_4d(base + G::ACC_OFF + (size_t)slot * G::ACC_BYTES, &m.acc, 2 * x0, y0, z, o, &abar[slot]);
  if (G::D32) tma::tensor_load_4d(base + G::D32_OFF + (size_t)slot * G::D32_BYTES, &m.d32, 2 * x0, y0, z, o, &abar[slot]);
}

// f(integral_constant<J>, k0 + J) for J = J0, J0 + KS .. N-1 while k0 + J < nsteps;
// false as soon as one call returns false
template <int J, int N, int KS, typename F>
__device__ __forceinline__ bool run_steps(F& f, int k0, int nsteps) {
  if constexpr (J < N) {
    if (k0 + J >= nsteps) return true;
    if (!f(std::integral_constant<int, J>{}, k0 + J)) return false;
    return run_steps<J + KS, N, KS>(f, k0, nsteps);
  } else {
    return true;
  }
}

// One work item: tile bx, z chunk by, orbital bz.  `base` is the 128-byte
// aligned shared-memory area of Geo<MODE, PER>; its barriers are initialised
// by the caller and keep their phases across items in pmask / amask / emask
// (bit s = parity of the next completion of slot s).
// Periodic grids (LOOSE): no CTA barrier in the sweep.  A warp that has finished
// plane step k arrives on ebar[k % RING], and thread 0 refills the slots of step
// k - 1 at its own step k once every warp has arrived there, so the warps drift
// apart and the stencil of one hides the waits of another (32^3 x 512 orbitals,
// mixed terms 1, 2, 3, 4: 501, 341, 415, 423 us with a barrier per plane, 435,
// 318, 388, 368 without).  Isolated grids, whose steps without gradient are
// shorter, keep the barrier, which lets the refill start a step earlier (64^3 x
// 5 orbitals: 33.4 us a term, 36.2 loose).  Returns false when a copy did not
// arrive in time (err is set and the CTA's other copies are drained).
template <int MODE, bool PER>
__device__ __forceinline__ bool tma_body(const TmaMaps& maps, void* __restrict__ hout, double2* __restrict__ acc,
                                         float2* __restrict__ d32, const TiledArgs& a, int* __restrict__ err,
                                         int bx, int by, int bz, unsigned char* base, uint32_t& pmask,
                                         uint32_t& amask, uint32_t& emask) {
  using G = Geo<MODE, PER>;
  using R = typename G::R;
  using C2 = typename G::C2;
  constexpr int SX = G::SX;
  const C2* ring = (const C2*)(base + G::RING_OFF);
  const double2* accr = (const double2*)(base + G::ACC_OFF);
  const float2* d32r = (const float2*)(base + G::D32_OFF);
  uint64_t* pbar = (uint64_t*)(base + G::BAR_OFF);
  double2* psm = (double2*)(base + G::PS_OFF);
  uint64_t* abar = pbar + RING;
  uint64_t* ebar = abar + ARING;  // LOOSE: all warps have finished a step

  const int t = threadIdx.x;
  const int tx = t & (TX - 1), ty = t / TX;
  const int ntx = (a.nx + TX - 1) / TX;
  const int x0 = (bx % ntx) * TX, y0 = (bx / ntx) * TY;
  const int x = x0 + tx, y = y0 + ty;
  const bool active = (x < a.nx) && (y < a.ny);
  const int zc0 = by * a.zchunk;
  const int zc1 = min(a.nz, zc0 + a.zchunk);
  const int nsteps = zc1 - zc0;
  const int ntot = nsteps + 2 * HALO;  // input planes zc0-4 .. zc1+3
  const int o = bz;
  const int ik = o / a.nspin_no;
  const int ispin = o % a.nspin;
  const double* kc = a.kcoef + (long)KC * ik;
  const R kx = (R)kc[0], ky = (R)kc[1], kz = (R)kc[2], lap0 = (R)kc[3];
  const int ctr = (ty + HALO) * SX + (PER ? tx : tx + HALO);
  const long sz = (long)a.nx * a.ny;
  const long pxy = (long)y * a.nx + x;
  constexpr bool GRAD = PER;

  // copies issued / waited, tracked identically by every thread
  int p_issued = 0, p_waited = 0, a_issued = 0, a_waited = 0;
  const int pro = ntot < RING ? ntot : RING;
  if (t == 0) {
    tma::fence_proxy_async_smem();  // the previous item's reads of the rings come first
    for (int r = 0; r < pro; ++r)
      issue_plane<MODE, PER>(maps, base, pbar, r, zc0 - HALO + r, x0, y0, o, a.nz, a.ny);
    if (G::ACC64 || G::D32)
      for (int k = 0; k < ARING && k < nsteps; ++k) issue_acc<MODE, PER>(maps, base, abar, k, zc0 + k, x0, y0, o);
  }
  p_issued = pro;
  if (G::ACC64 || G::D32) a_issued = nsteps < ARING ? nsteps : ARING;

  // projections of this orbital into shared memory (read before the first
  // barrier below; the previous item's readers have all passed its last barrier)
  const bool ps_smem = a.nlma > 0 && a.nlma <= TMA_MAX_NLMA;
  if (ps_smem)
    for (int i = t; i < a.nlma; i += NT) psm[i] = a.proj[(long)o * a.nlma + i];
  bool ok = true;
  // KS planes per step: its waits, barrier and refill are shared by KS planes
  // (isolated grids: 348 instructions a warp and plane, 65 of them FP64, with 1).
  // Plane j of a group of U reads w[j .. j + 8].
  constexpr bool LOOSE = PER;
  constexpr int KS = LOOSE ? 1 : TMA_PLANES, U = (KS > 1) ? KS : (MODE < 6 ? TMA_UNROLL : 1);
  C2 w[2 * HALO + U];
  // window planes zc0-4 .. zc0+3
#pragma unroll
  for (int r = 0; r < 2 * HALO; ++r) {
    ok = tma::mbar_wait(&pbar[r], (pmask >> r) & 1u) && ok;
    pmask ^= 1u << r;
    w[r] = ring[(size_t)r * G::PLANE + ctr];
  }
  p_waited = 2 * HALO;
  bool all_ok = __syncthreads_and(ok);  // the same in every thread
  if (all_ok) {
    if (t == 0) {  // the four pre-window slots take planes zc0+4 .. zc0+7
      tma::fence_proxy_async_smem();
      for (int r = RING; r < RING + HALO && r < ntot; ++r)
        issue_plane<MODE, PER>(maps, base, pbar, r, zc0 - HALO + r, x0, y0, o, a.nz, a.ny);
    }
    p_issued = ntot < RING + HALO ? ntot : RING + HALO;

    const C2 czc = Cx<R>::make((R)a.zc.x, (R)a.zc.y);
    const R* vsrc;
    if (sizeof(R) == 8) vsrc = (const R*)(a.vloc + (long)ispin * a.npts);
    else vsrc = (const R*)(a.vloc32 + (long)ispin * a.npts);
    R vl_n[KS];  // V, point map and first pair of the next step's planes
    int pm_n[KS];
    const int sz32 = (int)sz;
    int off = zc0 * sz32 + (int)pxy;  // this thread's point of the step's first plane
    auto load_next = [&](int k) {
#pragma unroll
      for (int i = 0; i < KS; ++i) {
        vl_n[i] = (R)0;
        pm_n[i] = -1;
        if (active && k + i < nsteps) {
          const int p = off + (i + (k > 0 ? KS : 0)) * sz32;
          vl_n[i] = __ldg(vsrc + p);
          if (a.nlma > 0) pm_n[i] = __ldg(a.pmap + p);
        }
      }
    };
    load_next(0);
    void* hbase;
    if (ModeT<MODE>::h32) hbase = (float2*)hout + (long)o * a.npts;
    else hbase = (double2*)hout + (long)o * a.npts;
    double2* abase = acc + (long)o * a.npts;
    float2* dbase = d32 + (long)o * a.npts;
    // pair form of the KB scatter: the first pair of the next plane's point
    // is loaded at the end of each step, from pm_n (loaded at its start), on
    // periodic grids (isolated ones have few points in spheres)
    constexpr bool AHEAD = PER && (MODE <= 3 || MODE >= 6) && MODE != 0;
    const bool pairs = AHEAD && a.nlma > 0 && a.use_pairs;
    const double2* pair_ph = pairs ? a.pair_ph + (a.phase_per_k ? (long)ik * a.npair : 0L) : nullptr;
    Pair1<R> f1[KS];
#pragma unroll
    for (int i = 0; i < KS; ++i) {
      f1[i].lm = 0;
      if (pairs) load_pair1<R>(f1[i], pm_n[i], a, pair_ph);
    }
    // The window of z neighbours moves down by U registers after every U planes.
    auto step = [&](auto jc, const int k) -> bool {
      constexpr int j0 = decltype(jc)::value;
#pragma unroll
      for (int i = 0; i < KS; ++i) {
        if (k + i >= nsteps) break;
        const int rf = k + i + 2 * HALO;  // plane z+4 feeds the window
        ok = tma::mbar_wait(&pbar[rf & (RING - 1)], (pmask >> (rf & (RING - 1))) & 1u) && ok;
        pmask ^= 1u << (rf & (RING - 1));
        w[j0 + i + 2 * HALO] = ring[(size_t)(rf & (RING - 1)) * G::PLANE + ctr];
        p_waited = rf + 1;
        if (G::ACC64 || G::D32) {
          const int as = (k + i) & (ARING - 1);
          ok = tma::mbar_wait(&abar[as], (amask >> as) & 1u) && ok;
          amask ^= 1u << as;
          a_waited = k + i + 1;
        }
      }
      if (LOOSE && !__all_sync(0xffffffffu, ok)) {  // the other warps give up at the same copy
        ok = false;
        return false;
      }
      R vl_k[KS];
      int pm_k[KS];
#pragma unroll
      for (int i = 0; i < KS; ++i) {
        vl_k[i] = vl_n[i];
        pm_k[i] = pm_n[i];
      }
      if (k + KS < nsteps) load_next(k + KS);
      double2 acl[KS];
      if (G::ACC_LD) {
#pragma unroll
        for (int i = 0; i < KS; ++i)
          acl[i] = active && k + i < nsteps ? __ldcg(abase + off + i * sz32) : make_double2(0.0, 0.0);
      }
      auto point = [&](auto ic) {
        constexpr int i = decltype(ic)::value, j = j0 + i;
        const int kk = k + i;
        if (!active || kk >= nsteps) return;
        const R vl = vl_k[i];
        const int pm = pm_k[i];
        const C2* P = ring + (size_t)((kk + HALO) & (RING - 1)) * G::PLANE;
        C2 vx = Cx<R>::make(0, 0), wx = vx, vy = vx, wy = vx, vz = vx, wz = vx;
#pragma unroll
        for (int s = 1; s <= HALO; ++s) {
          C2 tp, tm;
          if (PER) {
            tp = P[(ty + HALO) * SX + ((tx + s) & (TX - 1))];
            tm = P[(ty + HALO) * SX + ((tx - s) & (TX - 1))];
          } else {
            tp = P[ctr + s];
            tm = P[ctr - s];
          }
          vx = cfma((R)a.lapt[s - 1], cadd(tp, tm), vx);
          if (GRAD) wx = cfma((R)a.nab[s - 1], csub(tp, tm), wx);
        }
#pragma unroll
        for (int s = 1; s <= HALO; ++s) {
          const C2 tp = P[ctr + s * SX], tm = P[ctr - s * SX];
          vy = cfma((R)a.lapt[4 + s - 1], cadd(tp, tm), vy);
          if (GRAD) wy = cfma((R)a.nab[4 + s - 1], csub(tp, tm), wy);
        }
#pragma unroll
        for (int s = 0; s < HALO; ++s) {
          const C2 tp = w[j + HALO + 1 + s], tm = w[j + HALO - 1 - s];
          vz = cfma((R)a.lapt[8 + s], cadd(tp, tm), vz);
          if (GRAD) wz = cfma((R)a.nab[8 + s], csub(tp, tm), wz);
        }
        const C2 v = cadd(vz, cadd(vy, vx));
        const C2 c = w[j + HALO];
        C2 h;  // stencil value, then + KB term
        h = hcore(vl, lap0, c, v);
        if (GRAD) {
          const C2 ww = cfma(kz, wz, cfma(ky, wy, cscal(kx, wx)));
          h.x += ww.y;
          h.y -= ww.x;
        }
        if (a.nlma > 0 && pm >= 0 && a.use_pairs) {
          if (AHEAD) h = kb_pairs_ahead<R>(h, pm, ps_smem ? psm : a.proj + (long)o * a.nlma, a, ik, f1[i]);
          else h = kb_pairs<R>(h, pm, ps_smem ? psm : a.proj + (long)o * a.nlma, a, ik);
        } else if (a.nlma > 0 && pm >= 0) {
          const double2* pj = ps_smem ? psm : a.proj + (long)o * a.nlma;
          const double2* zk = a.ent_zk + (a.phase_per_k ? (long)ik * a.nent : 0L);
          const int e0 = pm >> 8, e1 = e0 + (pm & 255);
          for (int e = e0; e < e1; e += 8) {  // entries eight at a time, summed in entry order
            int l[8];
            double2 zv[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const int ee = min(e + i, e1 - 1);
              l[i] = __ldg(a.ent_lma + ee);
              zv[i] = __ldg(zk + ee);
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
              if (e + i < e1) {
                const double2 pv = pj[l[i]];
                h = cadd(h, cmul(Cx<R>::make((R)pv.x, (R)pv.y), Cx<R>::make((R)zv[i].x, (R)zv[i].y)));
              }
          }
        }
        const int gi = off + i * sz32;
        const int ti = (kk & (ARING - 1)) * NT + t;
        if (ModeT<MODE>::store_h) {
          if (ModeT<MODE>::h32) ((float2*)hbase)[gi] = make_float2((float)h.x, (float)h.y);
          else ((double2*)hbase)[gi] = make_double2((double)h.x, (double)h.y);
        }
        if (MODE == 1 || MODE == 4 || MODE == 5) {
          const double2 cd = make_double2((double)c.x, (double)c.y);
          const double2 hd = make_double2((double)h.x, (double)h.y);
          abase[gi] = cadd(cd, cmul(a.zc, hd));
        } else if (MODE == 2 || MODE == 3) {
          const double2 hd = make_double2((double)h.x, (double)h.y);
          abase[gi] = cadd(G::ACC_LD ? acl[i] : accr[ti], cmul(a.zc, hd));
        } else if (MODE == 6) {
          const C2 tt = cmul(czc, h);
          dbase[gi] = make_float2((float)tt.x, (float)tt.y);
        } else if (MODE == 7) {
          const float2 dd = d32r[ti];
          const C2 tt = cadd(Cx<R>::make((R)dd.x, (R)dd.y), cmul(czc, h));
          dbase[gi] = make_float2((float)tt.x, (float)tt.y);
        } else if (MODE == 8) {
          const float2 dd = d32r[ti];
          const C2 tt = cadd(Cx<R>::make((R)dd.x, (R)dd.y), cmul(czc, h));
          abase[gi] = cadd(accr[ti], make_double2((double)tt.x, (double)tt.y));
        }
        if (pairs && k + KS + i < nsteps) load_pair1<R>(f1[i], pm_n[i], a, pair_ph);
      };
      point(std::integral_constant<int, 0>{});
      if constexpr (KS > 1) point(std::integral_constant<int, 1>{});
      off += KS * sz32;
      if constexpr (LOOSE) {
        __syncwarp();
        if ((t & 31) == 0) tma::mbar_arrive(&ebar[k & (RING - 1)]);
        if (t == 0 && k > 0) {  // the slots of step k - 1, once every warp is done with it
          const int k1 = k - 1;
          ok = tma::mbar_wait(&ebar[k1 & (RING - 1)], (emask >> (k1 & (RING - 1))) & 1u) && ok;
          emask ^= 1u << (k1 & (RING - 1));
          if (ok) {
            tma::fence_proxy_async_smem();
            const int rn = k1 + RING + HALO;
            if (rn < ntot) {
              issue_plane<MODE, PER>(maps, base, pbar, rn, zc0 - HALO + rn, x0, y0, o, a.nz, a.ny);
              p_issued = rn + 1;
            }
            if ((G::ACC64 || G::D32) && k1 + ARING < nsteps) {
              issue_acc<MODE, PER>(maps, base, abar, k1 + ARING, zc0 + k1 + ARING, x0, y0, o);
              a_issued = k1 + ARING + 1;
            }
          }
        }
      } else {
        // warp 0 waits for the next step's copies before the step barrier, so the
        // other warps find them complete at their own (first) try-wait and
        // block in the barrier instead of polling
        if (t < 32) {
#pragma unroll
          for (int i = 0; i < KS; ++i) {
            if (k + KS + i >= nsteps) break;
            const int rf1 = (k + KS + i + 2 * HALO) & (RING - 1), as = (k + KS + i) & (ARING - 1);
            ok = tma::mbar_wait(&pbar[rf1], (pmask >> rf1) & 1u) && ok;
            if (G::ACC64 || G::D32) ok = tma::mbar_wait(&abar[as], (amask >> as) & 1u) && ok;
          }
        }
        all_ok = __syncthreads_and(ok);
        if (!all_ok) return false;
        if (t == 0) tma::fence_proxy_async_smem();
#pragma unroll
        for (int i = 0; i < KS; ++i) {  // refill the slots of plane z + i and of accumulator k + i
          const int rn = k + i + RING + HALO, an = k + i + ARING;  // plane z+8
          if (rn < ntot) {
            if (t == 0) issue_plane<MODE, PER>(maps, base, pbar, rn, zc0 - HALO + rn, x0, y0, o, a.nz, a.ny);
            p_issued = rn + 1;
          }
          if ((G::ACC64 || G::D32) && an < nsteps) {
            if (t == 0) issue_acc<MODE, PER>(maps, base, abar, an, zc0 + an, x0, y0, o);
            a_issued = an + 1;
          }
        }
      }
      return true;
    };
    for (int k0 = 0; k0 < nsteps; k0 += U) {
      if (!run_steps<0, U, KS>(step, k0, nsteps)) break;
#pragma unroll
      for (int i = 0; i < 2 * HALO; ++i) w[i] = w[i + U];
    }
  }
  // LOOSE: every warp is done with the rings and the projections of this item
  if (LOOSE && all_ok) {
    all_ok = __syncthreads_and(ok);
    if (t == 0 && all_ok) {
      const int k1 = nsteps - 1;
      tma::mbar_wait(&ebar[k1 & (RING - 1)], (emask >> (k1 & (RING - 1))) & 1u);  // complete: all have arrived
      emask ^= 1u << (k1 & (RING - 1));
    }
  }
  if (!all_ok) {
    // a copy did not arrive in time: flag it, wait (bounded) for the copies
    // still in flight into this CTA's shared memory, and leave
    if (t == 0) {
      atomicExch(err, 1);
      for (int r = p_waited; r < p_issued; ++r) {
        tma::mbar_wait(&pbar[r & (RING - 1)], (pmask >> (r & (RING - 1))) & 1u);
        pmask ^= 1u << (r & (RING - 1));
      }
      for (int k = a_waited; k < a_issued; ++k) {
        tma::mbar_wait(&abar[k & (ARING - 1)], (amask >> (k & (ARING - 1))) & 1u);
        amask ^= 1u << (k & (ARING - 1));
      }
    }
    __syncthreads();
  }
  return all_ok;
}


// barriers of a Geo<MODE, PER> area, initialised once per CTA
template <int MODE, bool PER>
__device__ __forceinline__ void tma_init_barriers(unsigned char* base) {
  using G = Geo<MODE, PER>;
  if (threadIdx.x == 0) {
    uint64_t* bar = (uint64_t*)(base + G::BAR_OFF);
    for (int i = 0; i < RING + ARING; ++i) tma::mbar_init(&bar[i], 1);
    for (int i = 0; i < RING; ++i) tma::mbar_init(&bar[RING + ARING + i], NT / 32);
    tma::fence_barrier_init();
  }
  __syncthreads();
}

__device__ __forceinline__ unsigned char* tma_area(unsigned char* raw) {
  return (unsigned char*)(((uintptr_t)raw + 127) & ~(uintptr_t)127);
}

}  // namespace tmak

// 4-D map over an orbital block [norb][nz][ny][2 nx] of FP64 or FP32 reals
// with the given box; false when the copy engine cannot address it.
bool make_tma_map(CUtensorMap* m, const void* base, bool f32, const GridInfo& g, int norb, int box0, int box1);

}  // namespace sb200
