// Verlet list, WCA core forces and cluster bonds -- the GPU form of
// neigh_list / check_list (v25/functions.cpp:1298-1394), force_sc
// (:1397-1553) and the cluster criterion of clust_conf (:2987-3016), plus
// an energy criterion for clusters (pair energy below a threshold).
//
// List: each particle keeps every partner (both directions, ascending
// index) whose segment distance is below r_list = max(2^(1/6) sigma_max,
// sigma_max + min_s) + skin.  It is rebuilt when any rod end may have moved
// by more than skin/2 since the last build (centre displacement plus half
// the length times the axis change); the reference's own test looks at the
// centres only (v25/functions.cpp:1386-1387), which is not enough once the
// list radius is tight.  The build scans every particle of the system in
// FP32 (fixed-point separations, exact minimum image).  Systems of
// kCellMinRods rods or more whose box holds at least 3 cells along every
// axis bin their rods into cells no smaller than the largest reach of a
// list entry and scan only the 27 cells around each rod's own: O(N) per
// build instead of O(N^2).  A cell's rods are staged in cell order (the
// fixed-point position with the rod's index, and the axis with the
// length), and the two warps of a cell read each neighbour cell's slots
// together, the same address across the warp.  The tests are the same FP32
// expressions on the same values as the all-pairs scan, and each list is
// sorted by index before it is written, so both scans give the same lists.
//
// WCA: the force is non-zero only for segment distance < 2^(1/6) sigma_ij.
// A pair is first screened in FP32; pairs that pass are evaluated exactly as
// the reference does, in FP64 and with the reference's segment-distance
// routine and sentinels, always with the lower index as particle i so both
// members of a pair see the same numbers.  Each particle sums its own pairs
// in ascending partner order -- the order in which force_sc adds them.
#include "mdsc_dev.cuh"
#include "reduce.cuh"
#include "seg_dist.cuh"

namespace mdsc {

// Does the system build its list this step?  From the largest displacement
// measure of the new configuration (particle_kernel), the same in every block.
// A list asked for is built unless one was built at this very configuration:
// the neighbour pass's lists also fix the order of its FP32 sums.
__device__ __forceinline__ bool list_due(const Batch& b, const SysDev& P, const SysState& S, int s, int force_all) {
  if (at_limit(b, s)) return false;
  return force_all || (S.force_list && (!S.list_ok || S.dmax != 0)) || 2.0 * soft_f2d(__int_as_float(S.dmax)) > P.skin;
}

// cell of a fixed-point position: floor(fraction x cells), exact
__device__ __forceinline__ int cell_of(const SysDev& P, uint32_t ux, uint32_t uy, uint32_t uz) {
  const int cx = (int)(((unsigned long long)ux * (unsigned)P.cnx) >> 32);
  const int cy = (int)(((unsigned long long)uy * (unsigned)P.cny) >> 32);
  const int cz = (int)(((unsigned long long)uz * (unsigned)P.cnz) >> 32);
  return (cz * P.cny + cy) * P.cnx + cx;
}

// Each rod of a rebuilding cell system into a slot of its cell (any order; the
// counts were cleared with the working copies).
__global__ void __launch_bounds__(kPartBlock) cell_bin_kernel(Batch b, int force_all) {
  const int2 bk = b.blk[blockIdx.x];
  const SysDev& P = b.sys[bk.x];
  SysState& S = b.st[bk.x];
  if (P.ncell == 0 || !list_due(b, P, S, bk.x, force_all)) return;
  const int i = bk.y + threadIdx.x;
  if (i >= P.part_off + P.n) return;
  const int N = b.ntot;
  const uint32_t ux = b.pfx[i], uy = b.pfx[N + i], uz = b.pfx[2 * N + i];
  const int c = P.cell_off + cell_of(P, ux, uy, uz);
  const int slot = atomicAdd(&b.ccnt[c], 1);
  if (slot < kCellSlots) {
    b.cpos[(long long)c * kCellSlots + slot] = make_uint4(ux, uy, uz, (uint32_t)i);
    b.cax[(long long)c * kCellSlots + slot] = b.pax[i];
  } else {
    atomicExch(&S.cell_ovf, 1);
  }
}

// ascending insertion sort of a short list
template <class A>
__device__ __forceinline__ void sort_small(A& v, int n) {
  for (int a = 1; a < n; ++a) {
    const int x = v[a];
    int c = a - 1;
    while (c >= 0 && v[c] > x) {
      v[c + 1] = v[c];
      --c;
    }
    v[c + 1] = x;
  }
}

// A fixed grid looks through the rows for those that are due: most steps
// rebuild few systems, and a block per row held the registers of the SMs from
// the tiles that start at the same time.
constexpr int kListBlocks = 4 * kSMs;

// The cell scan: blocks of two cells (two warps each), a thread per slot.
__device__ void list_cells(const Batch& b, int force_all) {
  const int2 cb = b.cellblk[blockIdx.x - kListBlocks];
  const SysDev& P = b.sys[cb.x];
  SysState& S = b.st[cb.x];
  if (P.ncell == 0 || S.cell_ovf || !list_due(b, P, S, cb.x, force_all)) return;
  const int c = cb.y + (threadIdx.x >> 6);
  if (c >= P.ncell) return;
  const int t = threadIdx.x & 63;
  const int cnt0 = b.ccnt[P.cell_off + c];
  const bool ok = t < cnt0;
  uint4 me = make_uint4(0u, 0u, 0u, 0u);
  float4 ai = make_float4(0.f, 0.f, 1.f, 0.f);
  if (ok) {
    me = b.cpos[(long long)(P.cell_off + c) * kCellSlots + t];
    ai = b.cax[(long long)(P.cell_off + c) * kCellSlots + t];
  }
  const int i = (int)me.w;
  const float rl = (float)P.r_list;
  const float rl2 = rl * rl;
  const float Lx = P.Lfix[0], Ly = P.Lfix[1], Lz = P.Lfix[2];
  const bool rcut = P.rc_real > 0.0;
  int lst[kMaxNb];
  int cnt = 0, rcnt = 0;
  int* rout = b.rnb + (long long)i * kMaxR;
  const int cx = c % P.cnx, cy = (c / P.cnx) % P.cny, cz = c / (P.cnx * P.cny);
  for (int dz = -1; dz <= 1; ++dz) {
    const int qz = (cz + dz + P.cnz) % P.cnz;
    for (int dy = -1; dy <= 1; ++dy) {
      const int qy = (cy + dy + P.cny) % P.cny;
      for (int dx0 = -1; dx0 <= 1; ++dx0) {
        const int qx = (cx + dx0 + P.cnx) % P.cnx;
        const long long q = P.cell_off + (qz * P.cny + qy) * P.cnx + qx;
        const int m = b.ccnt[q];
        const uint4* cp = b.cpos + q * kCellSlots;
        const float4* ca = b.cax + q * kCellSlots;
        for (int k = 0; k < m; ++k) {
          const uint4 pj = cp[k];
          const float4 aj = ca[k];
          if (!ok || pj.w == me.w) continue;
          const float dx = fix_diff(me.x, pj.x, Lx);
          const float dy = fix_diff(me.y, pj.y, Ly);
          const float dz2 = fix_diff(me.z, pj.z, Lz);
          const float r2 = dx * dx + dy * dy + dz2 * dz2;
          if (rcut && r2 < P.rl_r2) {
            if (rcnt < kMaxR) rout[rcnt] = (int)pj.w;
            ++rcnt;
          }
          const float reach = rl + 0.5f * (ai.w + aj.w);
          if (!(r2 < reach * reach)) continue;
          const float d2 = seg_dist_fast(dx, dy, dz2, ai.x, ai.y, ai.z, ai.w, aj.x, aj.y, aj.z, aj.w);
          if (d2 < rl2) {
            if (cnt < kMaxNb) lst[cnt] = (int)pj.w;
            ++cnt;
          }
        }
      }
    }
  }
  if (!ok) return;
  int err = (cnt > kMaxNb || rcnt > kMaxR) ? kErrListOverflow : 0;
  cnt = min(cnt, kMaxNb);
  sort_small(lst, cnt);
  int* out = b.nb + (long long)i * kMaxNb;
  int lower = 0;
  for (int k = 0; k < cnt; ++k) {
    out[k] = lst[k];
    lower += lst[k] < i ? 1 : 0;
  }
  b.nbc[i] = cnt;
  b.nblo[i] = lower;
  if (rcut) {
    rcnt = min(rcnt, kMaxR);
    sort_small(rout, rcnt);
    b.rnbc[i] = rcnt;
  }
  if (err) atomicOr(&S.status, err);
  const int N = b.ntot;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    b.fsave[3 * i + a] = b.pfx[a * N + i];
    b.usave[3 * i + a] = a == 0 ? ai.x : (a == 1 ? ai.y : ai.z);
  }
}

// The list build: blocks below nwblk scan all pairs for 32 rods (systems
// without cells, or whose cells overflowed this build); the rest scan cells.
// A few systems rebuild at a time, so the scan is a latency: the four warps
// of a block hold the same 32 rods and take a quarter each of every chunk of
// 128 candidates, whose hits they place in ascending order.
// Averaged over the steps of 64 systems of 128 to 2048 rods: 35 us a launch with
// a lane per rod over whole chunks (and its decision kernel), 19 this way.
__device__ void list_row(const Batch& b, int2 bk) {
  __shared__ uint32_t sx[kPartBlock], sy[kPartBlock], sz[kPartBlock];
  __shared__ float4 sa[kPartBlock];
  __shared__ uint32_t sm[2][4][32], sr[2][4][32];  // hits per (buffer, warp, rod): Verlet and real-space lists
  const SysDev& P = b.sys[bk.x];
  SysState& S = b.st[bk.x];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = bk.y + lane;
  const bool ok = i < P.part_off + P.n;
  const int N = b.ntot;
  uint32_t ux = 0, uy = 0, uz = 0;
  float4 ai = make_float4(0.f, 0.f, 1.f, 0.f);
  if (ok) {
    ux = b.pfx[i];
    uy = b.pfx[N + i];
    uz = b.pfx[2 * N + i];
    ai = b.pax[i];
  }
  const float rl = (float)P.r_list;
  const float rl2 = rl * rl;
  const float Lx = P.Lfix[0], Ly = P.Lfix[1], Lz = P.Lfix[2];
  const int first = P.part_off, n = P.n;
  int cnt = 0;
  int* out = b.nb + (long long)i * kMaxNb;
  // real-space neighbours (systems with a real-space cutoff): every rod whose
  // centre is within rl_r2, in ascending order, both directions
  const bool rcut = P.rc_real > 0.0;
  int rcnt = 0;
  int* rout = b.rnb + (long long)i * kMaxR;
  int buf = 0, lower = 0;
  for (int q0 = 0; q0 < n; q0 += kPartBlock, buf ^= 1) {
    const int nq = min(kPartBlock, n - q0);
    __syncthreads();
    if (threadIdx.x < nq) {
      const int q = first + q0 + threadIdx.x;
      sx[threadIdx.x] = b.pfx[q];
      sy[threadIdx.x] = b.pfx[N + q];
      sz[threadIdx.x] = b.pfx[2 * N + q];
      sa[threadIdx.x] = b.pax[q];
    }
    __syncthreads();
    // 1. centre distance against the reach of the two rods, branch-free,
    //    into a mask of the warp's 32 candidates: nearly every warp has a
    //    lane with some candidate in reach, so testing the segments inside
    //    this loop would run the segment routine for every candidate
    uint32_t bits = 0u, rbits = 0u;
#pragma unroll 8
    for (int kk = 0; kk < 32; ++kk) {
      const int k = 32 * w + kk;
      const float dx = fix_diff(ux, sx[k], Lx);
      const float dy = fix_diff(uy, sy[k], Ly);
      const float dz = fix_diff(uz, sz[k], Lz);
      const float reach = rl + 0.5f * (ai.w + sa[k].w);
      const float r2 = dx * dx + dy * dy + dz * dz;
      const bool other = ok && k < nq && first + q0 + k != i;
      bits |= (uint32_t)(other && r2 < reach * reach) << kk;
      if (rcut) rbits |= (uint32_t)(other && r2 < P.rl_r2) << kk;
    }
    // 2. segment distance of the candidates in reach
    uint32_t hits = 0u;
    for (uint32_t m = bits; m; m &= m - 1u) {
      const int kk = __ffs(m) - 1, k = 32 * w + kk;
      const float dx = fix_diff(ux, sx[k], Lx);
      const float dy = fix_diff(uy, sy[k], Ly);
      const float dz = fix_diff(uz, sz[k], Lz);
      const float4 aj = sa[k];
      const float d2 = seg_dist_fast(dx, dy, dz, ai.x, ai.y, ai.z, ai.w, aj.x, aj.y, aj.z, aj.w);
      if (d2 < rl2) hits |= 1u << kk;
    }
    // 3. into the lists, after the lower warps' hits
    sm[buf][w][lane] = hits;
    if (rcut) sr[buf][w][lane] = rbits;
    __syncthreads();
    int at = cnt, rat = rcnt;
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const uint32_t h = sm[buf][v][lane];
      const int c = __popc(h), below = i - (first + q0 + 32 * v);  // candidates of lower index
      at += v < w ? c : 0;
      cnt += c;
      lower += __popc(below >= 32 ? h : (below > 0 ? h & ((1u << below) - 1u) : 0u));
      if (rcut) {
        const int rc = __popc(sr[buf][v][lane]);
        rat += v < w ? rc : 0;
        rcnt += rc;
      }
    }
    for (uint32_t m = hits; m; m &= m - 1u, ++at)
      if (at < kMaxNb) out[at] = first + q0 + 32 * w + __ffs(m) - 1;
    for (uint32_t m = rbits; m; m &= m - 1u, ++rat)
      if (rat < kMaxR) rout[rat] = first + q0 + 32 * w + __ffs(m) - 1;
  }
  if (!ok || w > 0) return;
  int err = (cnt > kMaxNb || rcnt > kMaxR) ? kErrListOverflow : 0;
  b.nbc[i] = min(cnt, kMaxNb);
  b.nblo[i] = min(lower, kMaxNb);
  if (rcut) b.rnbc[i] = min(rcnt, kMaxR);
  if (err) atomicOr(&S.status, err);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    b.fsave[3 * i + a] = b.pfx[a * N + i];
    b.usave[3 * i + a] = a == 0 ? ai.x : (a == 1 ? ai.y : ai.z);
  }
}

__global__ void __launch_bounds__(kPartBlock) list_build_kernel(Batch b, int force_all) {
  __shared__ int due_rows[kPartBlock], ndue;
  if ((int)blockIdx.x >= kListBlocks) {
    list_cells(b, force_all);
    return;
  }
  for (int r0 = blockIdx.x; r0 < b.nwblk; r0 += kListBlocks * kPartBlock) {
    if (threadIdx.x == 0) ndue = 0;
    __syncthreads();
    const int r = r0 + threadIdx.x * kListBlocks;
    if (r < b.nwblk) {
      const int2 bk = b.wblk[r];
      const SysDev& P = b.sys[bk.x];
      SysState& S = b.st[bk.x];
      const bool due = list_due(b, P, S, bk.x, force_all);
      if (bk.y == P.part_off) S.rebuild = due ? 1 : 0;
      if (due && !(b.cells && P.ncell > 0 && !S.cell_ovf)) due_rows[atomicAdd(&ndue, 1)] = r;
    }
    __syncthreads();
    const int nd = ndue;
    for (int k = 0; k < nd; ++k) list_row(b, b.wblk[due_rows[k]]);
    __syncthreads();
  }
}

__device__ __forceinline__ void load_rod(const Batch& b, int i, RodD& R) {
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    R.r[a] = b.r[3 * i + a];
    R.o[a] = b.O[9 * i + 6 + a];
  }
  R.len = b.len[i];
}

// WCA pair (v25/functions.cpp:1438-1540) for A < B; returns false when the
// pair does not interact.  fA: force on A; tA, tB: torques; ev: U, W and
// the pressure tensor.  This file is compiled without FMA contraction (the
// cluster test must repeat the reference's roundings); the force path asks
// for its FMAs explicitly.
__device__ bool wca_pair(const Batch& b, const SysDev& P, int A, int B, double* fA, double* tA,
                         double* tB, double* ev, int& err) {
  RodD ra, rb;
  load_rod(b, A, ra);
  load_rod(b, B, rb);
  const double shA0 = ra.len, shB0 = rb.len;
  const double sigma = (b.dia[A] + b.dia[B]) / 2;
  const double sig_sq = sigma * sigma;
  const double srt = 1.122462048309373;   // 2^(1/6)
  const double rsh = srt * srt * sig_sq;
  double rij[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    rij[a] = ra.r[a] - rb.r[a];
    rij[a] = fma(-P.L[a], floor(fma(rij[a], P.invL[a], 0.5)), rij[a]);
  }
  const double rsq = fma(rij[2], rij[2], fma(rij[1], rij[1], rij[0] * rij[0]));
  double dij[3], st[2];
  const double dsq = seg_dist_wca(ra, rb, P.L, rij, dij, st);
  if (dsq < 0.49 * sig_sq || dsq > rsq * 1.00001) err |= kErrOverlap;
  if (!(dsq < rsh)) return false;
  // one reciprocal instead of the reference's three divisions; FIJ = W / ddr
  // reduces to 6 (pot + 4 SR6^2) / dsq, NaN where ddr = 0 as in the reference
  const double inv_dsq = 1.0 / dsq;
  const double SR2s = sig_sq * inv_dsq;
  const double SR6s = SR2s * SR2s * SR2s;
  const double pot = fma(4 * SR6s, SR6s, -4 * SR6s);
  const double ddr = fma(rij[2], dij[2], fma(rij[1], dij[1], rij[0] * dij[0]));
  const double fw = 6 * fma(4 * SR6s, SR6s, pot) * inv_dsq;
  const double FIJ = (ddr != 0.0) ? fw : __longlong_as_double(0x7ff8000000000000LL);
  if (!(fabs(FIJ) < 1e300)) err |= kErrNan;
  ev[0] = pot + 1.;
  ev[1] = fw * ddr;
#pragma unroll
  for (int a = 0; a < 3; ++a) fA[a] = FIJ * dij[a];
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int c = 0; c < 3; ++c) ev[2 + 3 * a + c] = rij[a] * fA[c];
  const double *oi = ra.o, *oj = rb.o;
  const double icroj[3] = {fma(oi[1], oj[2], -oi[2] * oj[1]), fma(oi[2], oj[0], -oi[0] * oj[2]),
                           fma(oi[0], oj[1], -oi[1] * oj[0])};
  const double icror[3] = {fma(oi[1], rij[2], -oi[2] * rij[1]), fma(oi[2], rij[0], -oi[0] * rij[2]),
                           fma(oi[0], rij[1], -oi[1] * rij[0])};
  const double jcror[3] = {fma(oj[1], rij[2], -oj[2] * rij[1]), fma(oj[2], rij[0], -oj[0] * rij[2]),
                           fma(oj[0], rij[1], -oj[1] * rij[0])};
  double fact1 = (st[0] - 0.5) * shA0;
  double fact2 = -(st[1] - 0.5) * shB0;
  if (st[0] == -1.e+6) fact1 = fact2 = 0.;
  // as in the reference, -3e10 is tested twice (v25/functions.cpp:1526,1529),
  // so the (-/+) end-point sentinel keeps the lever arms computed above
  if (st[0] == -1.e+10) {
    fact1 = 0.5 * shA0;
    fact2 = 0.5 * shB0;
  } else if (st[0] == -2.e+10) {
    fact1 = -0.5 * shA0;
    fact2 = -0.5 * shB0;
  } else if (st[0] == -3.e+10) {
    fact1 = 0.5 * shA0;
    fact2 = -0.5 * shB0;
  }
  const double fmul = fact1 * fact2;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    tA[a] = FIJ * fma(fact1, icror[a], fmul * icroj[a]);
    tB[a] = FIJ * fma(fact2, jcror[a], -fmul * icroj[a]);
  }
  return true;
}

// WCA in two kernels.  (1) wca_screen: each particle's partners of higher
// index (each pair once) are screened in FP32 against 2^(1/3) sigma^2 with a
// margin; the candidates go to the particle's slots (wcand) in ascending
// index and (slot, system) items to a work list, one atomic per warp.  (2) wca_eval: every thread of a fixed
// grid takes list items and evaluates them in FP64 -- only pairs that can
// touch reach the FP64 unit (1/64 of the FP32 rate on this GPU), densely
// packed, with no block-wide synchronisation.  Each item writes its own
// share (force and torque on the lower index), its partner's share and its
// energy/virial terms to the candidate's slot.  The finalize kernel adds a
// particle's own shares in slot order and its partners' shares in partner
// order, and the per-system reduction adds the slots' energies in particle
// and slot order, so the list order (which depends on warp timing) does not
// reach any result.
//
// The screen takes LANES lanes per rod: the lanes test LANES list entries of
// higher index at a time (each a chain of gathers, so one
// lane per rod waited for its whole list), a ballot puts the entries that
// pass into the rod's slots in list order -- ascending partners -- and each
// partner learns where its share of the pair will be (win, wincnt).
template <int LANES>
__global__ void __launch_bounds__(128) wca_screen_kernel(Batch b) {
  constexpr int kPer = 32 * LANES / 128;  // blocks per row of 32 rods
  const int2 bk = b.wblk[blockIdx.x / kPer];
  const int s = bk.x;
  if (at_limit(b, s)) return;
  const SysDev& P = b.sys[s];
  const int lane = threadIdx.x & 31, sub = lane % LANES, grp = lane / LANES;
  const int i = bk.y + (blockIdx.x % kPer * 128 + threadIdx.x) / LANES;
  const bool ok = i < P.part_off + P.n;
  const int N = b.ntot;
  int nl = 0, lo = 0, nc = 0, err = 0;
  uint32_t ux = 0, uy = 0, uz = 0;
  float4 ai = make_float4(0.f, 0.f, 1.f, 0.f);
  float di = 0.f;
  if (ok) {
    nl = b.nbc[i];
    lo = b.nblo[i];  // the list ascends: entries from here on are above i
    ux = b.pfx[i];
    uy = b.pfx[N + i];
    uz = b.pfx[2 * N + i];
    ai = b.pax[i];
    di = b.pdia[i];
  }
  const int* lst = b.nb + (long long)i * kMaxNb;
  for (int k = lo + sub; __any_sync(0xffffffffu, k < nl); k += LANES) {
    bool cand = false;
    int q = -1;
    if (k < nl) {
      q = lst[k];
      const float dx = fix_diff(ux, b.pfx[q], P.Lfix[0]);
      const float dy = fix_diff(uy, b.pfx[N + q], P.Lfix[1]);
      const float dz = fix_diff(uz, b.pfx[2 * N + q], P.Lfix[2]);
      const float4 aj = b.pax[q];
      const float sg = 0.5f * (di + b.pdia[q]);
      const float d2 = seg_dist_fast(dx, dy, dz, ai.x, ai.y, ai.z, ai.w, aj.x, aj.y, aj.z, aj.w);
      // 2^(1/3) sigma^2, with a margin for the FP32 screen
      cand = !(d2 >= 1.2599211f * sg * sg * 1.002f);  // NaN (no length) is left to the FP64 evaluation
    }
    const uint32_t mask = (__ballot_sync(0xffffffffu, cand) >> (grp * LANES)) & ((1u << LANES) - 1u);
    if (cand) {
      const int slot = nc + __popc(mask & ((1u << sub) - 1u));
      if (slot < kMaxC) {
        b.wcand[(long long)i * kMaxC + slot] = q;
        const int t = atomicAdd(&b.wincnt[q], 1);
        if (t < kMaxC)
          b.win[(long long)q * kMaxC + t] = i * kMaxC + slot;
        else
          err |= kErrListOverflow;
      }
    }
    nc += __popc(mask);
  }
  if (nc > kMaxC) {
    err |= kErrListOverflow;
    nc = kMaxC;
  }
  if (ok && sub == 0) b.wcnt[i] = nc;
  // room on the work list for the warp's candidates: one atomic per warp
  int at = 0, tot = 0;
#pragma unroll
  for (int g = 0; g < 32 / LANES; ++g) {
    const int c = __shfl_sync(0xffffffffu, nc, g * LANES);
    at += g < grp ? c : 0;
    tot += c;
  }
  int base = 0;
  if (lane == 0 && tot > 0) base = atomicAdd(b.wlist_n, tot);
  at += __shfl_sync(0xffffffffu, base, 0);
  for (int k = sub; k < nc; k += LANES) b.wlist[at + k] = make_int2(i * kMaxC + k, s);
  if (err) atomicOr(&b.st[s].status, err);
}

__global__ void __launch_bounds__(128) wca_eval_kernel(Batch b) {
  const int n = *(volatile const int*)b.wlist_n;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    const int2 it = b.wlist[e];
    const int slot = it.x, s = it.y;
    const int p = slot / kMaxC;
    const SysDev& P = b.sys[s];
    const int q = b.wcand[slot];
    int err = 0;
    double fA[3], tA[3], tB[3], ev[11];
    if (!wca_pair(b, P, p, q, fA, tA, tB, ev, err)) {
#pragma unroll
      for (int a = 0; a < 3; ++a) fA[a] = tA[a] = tB[a] = 0.0;
#pragma unroll
      for (int c = 0; c < 11; ++c) ev[c] = 0.0;
    }
    double* own = b.wown + (long long)slot * 6;
    double* rec = b.wrec + (long long)slot * 6;
    double* evo = b.wev + (long long)slot * 11;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      own[a] = fA[a];
      own[3 + a] = tA[a];
      rec[a] = -fA[a];
      rec[3 + a] = tB[a];
    }
#pragma unroll
    for (int c = 0; c < 11; ++c) evo[c] = ev[c];
    if (err) atomicOr(&b.st[s].status, err);
  }
}

// The same on four lanes per pair, for batches whose contacts leave the FP64
// units idle: an FP64 instruction takes a warp 64 cycles whatever its lanes do,
// and the pair's 210 of them are the time.  Lane 0 to 2 take the components of
// vectors, or one of three values of the same form each (products, candidate
// points, crosses), exchanged by shuffles: 100 instructions, the same operations
// on the same values as wca_pair with seg_dist_wca, and so the same bits: 10.4 us
// a launch in the step of 256 rods on one lane, 7.6 on four.
__device__ __forceinline__ double quad(double v, int from) { return __shfl_sync(0xffffffffu, v, from, 4); }
__device__ __forceinline__ double sel(const double (&v)[3], int k) { return k == 0 ? v[0] : (k == 1 ? v[1] : v[2]); }

__global__ void __launch_bounds__(128) wca_eval4_kernel(Batch b) {
  const int n = *(volatile const int*)b.wlist_n;
  const int lane = threadIdx.x & 31, c = lane & 3, cc = min(c, 2);
  for (int w0 = (blockIdx.x * 4 + (threadIdx.x >> 5)) * 8; w0 < n; w0 += gridDim.x * 32) {
    const bool ok = w0 + (lane >> 2) < n;
    const int2 it = b.wlist[ok ? w0 + (lane >> 2) : n - 1];  // spare lanes repeat the last pair and store nothing
    const int slot = it.x, A = slot / kMaxC, B = b.wcand[slot];
    const SysDev& P = b.sys[it.y];
    double oA[3], oB[3], rij[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      oA[q] = b.O[9 * A + 6 + q];
      oB[q] = b.O[9 * B + 6 + q];
    }
    const double lA = b.len[A], lB = b.len[B];
    const double sigma = (b.dia[A] + b.dia[B]) / 2;
    const double sig_sq = sigma * sigma;
    double x = b.r[3 * A + cc] - b.r[3 * B + cc];
    x = fma(-P.L[cc], floor(fma(x, P.invL[cc], 0.5)), x);
#pragma unroll
    for (int q = 0; q < 3; ++q) rij[q] = quad(x, q);
    // oA.oB, rij.oA, rij.oB, rij.rij
    double u[3], v[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      u[q] = c == 0 ? oA[q] : rij[q];
      v[q] = c == 1 ? oA[q] : (c == 3 ? rij[q] : oB[q]);
    }
    x = fma(u[2], v[2], fma(u[1], v[1], u[0] * v[0]));
    const double doto = quad(x, 0), dotrA = quad(x, 1), dotrB = quad(x, 2), rsq = quad(x, 3);
    // lA^2, lB^2, (oA.oB) lA
    x = (c == 0 ? lA : (c == 1 ? lB : doto)) * (c == 1 ? lB : lA);
    const double a2 = quad(x, 0), c2 = quad(x, 1), bb = quad(x, 2) * lB;
    // d, e
    const double hb = 0.5 * bb;
    x = fma(c == 0 ? dotrA : dotrB, c == 0 ? lA : lB, (c == 0 ? -0.5 : 0.5) * (c == 0 ? a2 : c2));
    x = x + (c == 0 ? hb : -hb);
    const double d = quad(x, 0), e = quad(x, 1);
    // s, t, det
    x = fma(c == 0 ? bb : a2, c < 2 ? e : c2, -(c == 0 ? c2 : bb) * (c < 2 ? d : bb));
    const double s = quad(x, 0), t = quad(x, 1), det = quad(x, 2);
    const bool par = !(det > 1.e-12);
    const double dets = par ? 1.0 : det;
    const double ac = a2 * c2;
    const double inv = 1.0 / (dets * ac);
    // 1 / det, 1 / c, 1 / a: what the lane's candidate needs
    const double scale = inv * (c == 0 ? ac : dets) * (c == 0 ? 1.0 : (c == 1 ? a2 : c2));
    double laA[3], lbB[3];
    x = lA * sel(oA, cc);
    const double y = lB * sel(oB, cc);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      laA[q] = quad(x, q);
      lbB[q] = quad(y, q);
    }
    const double lo = c == 0 ? det : (c == 1 ? det : (c == 2 ? s : t));
    const double hi = c == 0 ? s : (c == 1 ? t : 0.0);
    const unsigned f = (__ballot_sync(0xffffffffu, lo < hi) >> (lane & 28)) & 15u;
    const bool sbig = f & 1, tbig = f & 2, sneg = f & 4, tneg = f & 8;
    const double S = sbig ? 1.0 : 0.0, T = tbig ? 1.0 : 0.0;
    // the candidates: lane 0 the interior point, 1 s held, 2 t held
    x = (c == 0 ? s : fma(bb, c == 1 ? S : T, c == 1 ? e : -d)) * scale;
    const double tI = t * scale;
    const double xc = x > 1.0 ? 1.0 : (x < 0.0 ? 0.0 : x);
    const double sv = c == 0 ? x : (c == 1 ? S : xc), tv = c == 0 ? tI : (c == 1 ? xc : T);
    const double sm = sv - 0.5, tm = 0.5 - tv;
    double o[3], dij[3], st[2];
#pragma unroll
    for (int q = 0; q < 3; ++q) o[q] = fma(tm, lbB[q], fma(sm, laA[q], rij[q]));
    x = fma(o[2], o[2], fma(o[1], o[1], o[0] * o[0]));
    const double dI = quad(x, 0), dS = quad(x, 1), dT = quad(x, 2);
    const bool sout = sneg || sbig, tout = tneg || tbig;
    int pick;
    if (!sout && !tout) pick = 0;
    else if (!tout) pick = 1;
    else if (!sout) pick = 2;
    else if (sbig) pick = (dT < dS) ? 2 : 1;
    else pick = (dS < dT) ? 1 : 2;
#pragma unroll
    for (int q = 0; q < 3; ++q) dij[q] = quad(o[q], pick);
    st[0] = quad(sv, pick);
    st[1] = quad(tv, pick);
    double dsq = quad(x, pick);
    if (par || dI < 1.e-12) {  // parallel or intersecting axes: every lane of the pair alike
      RodD ra, rb;
      load_rod(b, A, ra);
      load_rod(b, B, rb);
      dsq = seg_dist_ref<false>(ra, rb, P.L, rij, dij, st);
    }
    __syncwarp();
    const double srt = 1.122462048309373;  // 2^(1/6)
    const double lim = (c == 0 ? 0.49 : (c == 1 ? srt * srt : 1.00001)) * (c < 2 ? sig_sq : rsq);
    const unsigned g =
        (__ballot_sync(0xffffffffu, c == 2 ? lim < dsq : dsq < lim) >> (lane & 28)) & 7u;
    int err = (g & 5u) ? kErrOverlap : 0;
    const bool in = g & 2u;
    double fA = 0.0, tA = 0.0, tB = 0.0, row[3] = {0.0, 0.0, 0.0}, e0 = 0.0, e1 = 0.0;
    if (__any_sync(0xffffffffu, in)) {
      const double inv_dsq = 1.0 / dsq;
      const double SR2s = sig_sq * inv_dsq;
      const double SR6s = SR2s * SR2s * SR2s;
      const double q4 = 4 * SR6s;
      const double pot = fma(q4, SR6s, -q4);
      const double ddr = fma(rij[2], dij[2], fma(rij[1], dij[1], rij[0] * dij[0]));
      const double fw = 6 * fma(q4, SR6s, pot) * inv_dsq;
      const double FIJ = (ddr != 0.0) ? fw : __longlong_as_double(0x7ff8000000000000LL);
      if (in && !(fabs(FIJ) < 1e300)) err |= kErrNan;
      const double fc = FIJ * sel(dij, cc);
      const int k1 = cc == 2 ? 0 : cc + 1, k2 = cc == 0 ? 2 : cc - 1;
      const double oi1 = sel(oA, k1), oi2 = sel(oA, k2), oj1 = sel(oB, k1), oj2 = sel(oB, k2);
      const double r1 = sel(rij, k1), r2 = sel(rij, k2), rc = sel(rij, cc);
      const double icroj = fma(oi1, oj2, -oi2 * oj1);
      const double icror = fma(oi1, r2, -oi2 * r1);
      const double jcror = fma(oj1, r2, -oj2 * r1);
      x = (c == 0 ? st[0] : st[1]) - 0.5;
      x = (c == 0 ? x : -x) * (c == 0 ? lA : lB);
      double fact1 = quad(x, 0), fact2 = quad(x, 1);
      if (st[0] < -1.e+5) {  // the sentinels, as wca_pair
        if (st[0] == -1.e+6) fact1 = fact2 = 0.;
        if (st[0] == -1.e+10) {
          fact1 = 0.5 * lA;
          fact2 = 0.5 * lB;
        } else if (st[0] == -2.e+10) {
          fact1 = -0.5 * lA;
          fact2 = -0.5 * lB;
        } else if (st[0] == -3.e+10) {
          fact1 = 0.5 * lA;
          fact2 = -0.5 * lB;
        }
      }
      __syncwarp();
      const double fmul = fact1 * fact2;
      const double ta = FIJ * fma(fact1, icror, fmul * icroj), tb = FIJ * fma(fact2, jcror, -fmul * icroj);
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const double fq = quad(fc, q);
        if (in) row[q] = rc * fq;
      }
      if (in) {
        fA = fc;
        tA = ta;
        tB = tb;
        e0 = pot + 1.;
        e1 = fw * ddr;
      }
    }
    if (!ok) continue;
    double* evo = b.wev + (long long)slot * 11;
    if (c < 3) {
      double* own = b.wown + (long long)slot * 6;
      double* rec = b.wrec + (long long)slot * 6;
      own[c] = fA;
      own[3 + c] = tA;
      rec[c] = -fA;
      rec[3 + c] = tB;
#pragma unroll
      for (int q = 0; q < 3; ++q) evo[2 + 3 * c + q] = row[q];
    } else {
      evo[0] = e0;
      evo[1] = e1;
      if (err) atomicOr(&b.st[it.y].status, err);
    }
  }
}

// ---- clusters (v25/functions.cpp:2987-3016,3282-3324) ----------------
// Bond flags for list entries q > i: segment distance < (D_i + D_j)/2 + min_s
// in FP64 with the reference's routine (lower index first).  An FP32 distance,
// the smallest one between the segments, decides first where it is the
// routine's as well (bond_clear) and more than half a percent from the
// threshold.  What is left takes the FP64 routine (~20,000 cycles of a warp).
// Eight lanes per rod: 32,768 rods 237 us a launch with one lane and FP64 for
// every entry, 17 this way.
//
// The routine's distance is the smallest one, to FP32 accuracy, unless the axes
// are nearly parallel (it then takes the distance of the lines, or of the ends),
// the axis lines meet (an end point's distance to the other segment, whichever
// of the ends it tries first: coplanar rods within the threshold by their
// smallest distance can be beyond it by the routine's), or a rod has hardly any
// length (parallel to everything).  Bounds well inside its own (a^2 c^2 sin^2 <
// 1e-12, lines within 1e-6): sin^2 above 1e-4, lengths' product above 1e-3 and
// lines more than 0.001 apart; the distance of the lines in FP32 is good to ~5e-7
// |r| / sin, which the last term covers.  And the axes of unit length, which the
// routine takes for granted.  r: between the centres.
__device__ __forceinline__ bool bond_clear(float rx, float ry, float rz, float4 ai, float4 aj) {
  const float cx = ai.y * aj.z - ai.z * aj.y, cy = ai.z * aj.x - ai.x * aj.z, cz = ai.x * aj.y - ai.y * aj.x;
  const float sin2 = cx * cx + cy * cy + cz * cz, h = rx * cx + ry * cy + rz * cz;
  const float ni = ai.x * ai.x + ai.y * ai.y + ai.z * ai.z, nj = aj.x * aj.x + aj.y * aj.y + aj.z * aj.z;
  return fmaxf(fabsf(ni - 1.f), fabsf(nj - 1.f)) < 1e-5f && sin2 > 1e-4f && ai.w * aj.w > 1e-3f &&
         h * h > 1e-6f * sin2 + 1e-11f * (rx * rx + ry * ry + rz * rz);
}
__device__ __forceinline__ bool bonded_ref(const Batch& b, const SysDev& P, int i, int q) {
  RodD ri, rq;
  load_rod(b, i, ri);
  load_rod(b, q, rq);
  const double sigma = (b.dia[i] + b.dia[q]) / 2 + P.min_s;
  double rij[3], dij[3], st[2];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    rij[a] = ri.r[a] - rq.r[a];
    rij[a] -= P.L[a] * floor(rij[a] / P.L[a] + 0.5);
  }
  return seg_dist_ref<true>(ri, rq, P.L, rij, dij, st) < sigma * sigma;
}

constexpr int kBondLanes = 8;
__global__ void __launch_bounds__(128) cluster_bonds_kernel(Batch b) {
  constexpr int kPer = 32 * kBondLanes / 128;  // blocks per row of 32 rods
  const int2 bk = b.wblk[blockIdx.x / kPer];
  const SysDev& P = b.sys[bk.x];
  const int i = bk.y + (blockIdx.x % kPer * 128 + threadIdx.x) / kBondLanes, sub = threadIdx.x % kBondLanes;
  if (i >= P.part_off + P.n) return;
  if (sub == 0) b.comp[i] = i;
  if (sub == 0 && i == P.part_off) b.st[bk.x].dmax = 0;  // the list of this configuration stands
  if (P.cl_mode) return;  // energy criterion: ebond_eval_kernel
  const int nc = b.nbc[i];
  const int* lst = b.nb + (long long)i * kMaxNb;
  unsigned char* fl = b.eflag + (long long)i * kMaxNb;
  const int N = b.ntot;
  const uint32_t ux = b.pfx[i], uy = b.pfx[N + i], uz = b.pfx[2 * N + i];
  const float4 ai = b.pax[i];
  const float di = b.pdia[i], ms = (float)P.min_s;
  for (int k = b.nblo[i] + sub; k < nc; k += kBondLanes) {
    const int q = lst[k];
    const float4 aj = b.pax[q];
    const float dx = fix_diff(ux, b.pfx[q], P.Lfix[0]), dy = fix_diff(uy, b.pfx[N + q], P.Lfix[1]),
                dz = fix_diff(uz, b.pfx[2 * N + q], P.Lfix[2]);
    const float d2 = seg_dist_fast(dx, dy, dz, ai.x, ai.y, ai.z, ai.w, aj.x, aj.y, aj.z, aj.w);
    const float sg = 0.5f * (di + b.pdia[q]) + ms, thr = sg * sg;
    bool bond = d2 < 0.995f * thr;
    if (!((bond || d2 > 1.005f * thr) && bond_clear(dx, dy, dz, ai, aj))) bond = bonded_ref(b, P, i, q);
    fl[k] = bond ? 1 : 0;
  }
}

// ---- energy criterion (an extension; the reference's test is geometric) --
// U_pair = the WCA pair energy of force_sc (v25/functions.cpp:1436-1483) +
// the bare dipole-dipole energy of every dipole pair of the two rods at the
// minimum image of the sites, mu_a mu_b (o_a.o_b - 3 (o_a.r)(o_b.r)/r^2)/r^3,
// in FP64 with the operations in the oracle's order (A < B; this file is
// compiled without FMA contraction, and sqrt and division round correctly).
__device__ void dip_lab_ref(const Batch& b, const SysDev& P, int i, int w, double pos[3], double ori[3],
                            double* mu) {
  const int g = P.dip_off + (i - P.part_off) * P.nd + w;
  const double* O = b.O + 9 * (long long)i;
  const double d0 = b.dpc[g];
#pragma unroll
  for (int a = 0; a < 3; ++a) pos[a] = b.r[3 * i + a] + d0 * O[6 + a];
#pragma unroll
  for (int m = 0; m < 3; ++m) {  // transpose(O) times the body direction, summed from 0
    double acc = 0.;
    acc += O[m] * b.dob[3 * g];
    acc += O[3 + m] * b.dob[3 * g + 1];
    acc += O[6 + m] * b.dob[3 * g + 2];
    ori[m] = acc;
  }
  *mu = b.dmu[g];
}

__device__ double pair_energy_ref(const Batch& b, const SysDev& P, int A, int B) {
  RodD ra, rb;
  load_rod(b, A, ra);
  load_rod(b, B, rb);
  double rij[3], dij[3], st[2];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    rij[a] = ra.r[a] - rb.r[a];
    rij[a] -= P.L[a] * floor(rij[a] / P.L[a] + 0.5);
  }
  const double dsq = seg_dist_ref<true>(ra, rb, P.L, rij, dij, st);
  const double sigma = (b.dia[A] + b.dia[B]) / 2;
  const double sig_sq = sigma * sigma;
  const double srt = 1.122462048309373;  // 2^(1/6)
  double U = 0.;
  if (dsq < srt * srt * sig_sq) {
    const double SR2s = sig_sq / dsq;
    const double SR6s = SR2s * SR2s * SR2s;
    U = 4 * SR6s * (SR6s - 1.) + 1.;
  }
  for (int a = 0; a < P.nd; ++a) {
    double pa[3], oa[3], ma;
    dip_lab_ref(b, P, A, a, pa, oa, &ma);
    if (ma == 0.) continue;
    for (int c = 0; c < P.nd; ++c) {
      double pb[3], ob[3], mb;
      dip_lab_ref(b, P, B, c, pb, ob, &mb);
      if (mb == 0.) continue;
      double r[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) r[k] = dmimg(pa[k] - pb[k], P.L[k]);
      const double r2 = ddot(r, r);
      const double ir = 1. / sqrt(r2);
      const double ir3 = ir * ir * ir;
      const double dd = ddot(oa, ob), da = ddot(oa, r), db = ddot(ob, r);
      U += ma * mb * (dd - 3. * da * db / r2) * ir3;
    }
  }
  return U;
}

// Candidates for bonds U_pair < -cl_ubond among the higher indices of the
// system: an FP32 screen on the centres (fixed-point minimum image) keeps
// the pairs that can bond, |U_dd| <= 2 M_i M_j / (r - e_i - e_j)^3 with M
// the sum of a rod's moments and e its largest dipole offset, U_WCA >= 0.
// ebond_eval_kernel evaluates them exactly; their order reaches no result.
//
// That bound is a distance, so a system with a cell grid (systems of
// kCellMinRods rods or more) bins its rods and screens the 27 cells around
// each, where the bound of its largest M and e fits a cell; the others, and
// systems with an overfull cell, screen all pairs.  32,768 rods, screen and
// evaluation: 3470 us over all pairs with the bounds formed anew for every
// pair of blocks and one lane per rod evaluating, 128 this way; 3000 rods
// (all pairs) 356 and 83.
__device__ __forceinline__ bool ebond_near(float2 mi, float2 mj, float dx, float dy, float dz, float thr,
                                           float reach2) {
  const float r2 = dx * dx + dy * dy + dz * dz;
  if (r2 > reach2) return false;
  const float gap = sqrtf(r2) * 0.9999f - mi.y - mj.y;
  return mj.x != 0.f && (gap <= 0.f || 2.f * mi.x * mj.x >= thr * gap * gap * gap);
}
// no pair of the system passes that test beyond this distance
__device__ __forceinline__ float ebond_reach(const SysDev& P) {
  return (cbrtf(2.f * P.cl_mmax * P.cl_mmax / ((float)P.cl_ubond * 0.999f)) + 2.f * P.cl_emax) * 1.001f;
}
__device__ __forceinline__ bool ebond_on_cells(const Batch& b, const SysDev& P) {
  return b.cells && P.ncell > 0 &&
         ebond_reach(P) <= fminf(P.Lf[0] / P.cnx, fminf(P.Lf[1] / P.cny, P.Lf[2] / P.cnz));
}

// (M, e) of every rod, to scratch (the WCA terms' slots, read by the force
// assembly only), the bond counts cleared, and the rods into their cells
__global__ void __launch_bounds__(kPartBlock) ebond_prep_kernel(Batch b) {
  const int2 bk = b.blk[blockIdx.x];
  const SysDev& P = b.sys[bk.x];
  const int i = bk.y + threadIdx.x;
  if (P.cl_mode != 1 || i >= P.part_off + P.n) return;
  float m = 0.f, e = 0.f;
  for (int w = 0; w < P.nd; ++w) {
    const int g = P.dip_off + (i - P.part_off) * P.nd + w;
    const float ob = (float)sqrt(b.dob[3 * g] * b.dob[3 * g] + b.dob[3 * g + 1] * b.dob[3 * g + 1] +
                                 b.dob[3 * g + 2] * b.dob[3 * g + 2]);
    m += fabsf((float)b.dmu[g]) * ob;
    e = fmaxf(e, fabsf((float)b.dpc[g]));
  }
  const float2 me = make_float2(m * 1.0001f, e * 1.0001f);
  reinterpret_cast<float2*>(b.wev)[i] = me;
  b.ecnt[i] = 0;
  b.ebcnt[i] = 0;
  if (!ebond_on_cells(b, P)) return;
  const int N = b.ntot;
  const uint32_t ux = b.pfx[i], uy = b.pfx[N + i], uz = b.pfx[2 * N + i];
  const int c = P.cell_off + cell_of(P, ux, uy, uz);
  const int slot = atomicAdd(&b.ccnt[c], 1);
  if (slot < kCellSlots) {
    b.cpos[(long long)c * kCellSlots + slot] = make_uint4(ux, uy, uz, (uint32_t)i);
    b.cax[(long long)c * kCellSlots + slot] = make_float4(me.x, me.y, 0.f, 0.f);
  } else {
    atomicExch(&b.st[bk.x].cell_ovf, 1);
  }
}

__device__ void ebond_cells(const Batch& b) {
  const int2 cb = b.cellblk[blockIdx.x - b.nwblk];
  const SysDev& P = b.sys[cb.x];
  if (P.cl_mode != 1 || b.st[cb.x].cell_ovf || !ebond_on_cells(b, P)) return;
  const int c = cb.y + (threadIdx.x >> 6);
  if (c >= P.ncell) return;
  const int t = threadIdx.x & 63;
  const bool ok = t < b.ccnt[P.cell_off + c];
  uint4 me = make_uint4(0u, 0u, 0u, 0u);
  float4 mi = make_float4(0.f, 0.f, 0.f, 0.f);
  if (ok) {
    me = b.cpos[(long long)(P.cell_off + c) * kCellSlots + t];
    mi = b.cax[(long long)(P.cell_off + c) * kCellSlots + t];
  }
  const float thr = (float)P.cl_ubond * 0.999f, reach = ebond_reach(P), reach2 = reach * reach;
  const float Lx = P.Lfix[0], Ly = P.Lfix[1], Lz = P.Lfix[2];
  int* out = b.ecand + (long long)me.w * kMaxE;
  int cnt = 0;
  const int cx = c % P.cnx, cy = (c / P.cnx) % P.cny, cz = c / (P.cnx * P.cny);
  for (int n = 0; n < 27; ++n) {
    const int qx = (cx + n % 3 - 1 + P.cnx) % P.cnx, qy = (cy + n / 3 % 3 - 1 + P.cny) % P.cny,
              qz = (cz + n / 9 - 1 + P.cnz) % P.cnz;
    const long long q = P.cell_off + (qz * P.cny + qy) * P.cnx + qx;
    const int m = b.ccnt[q];
#pragma unroll 4
    for (int k = 0; k < m; ++k) {
      const uint4 pj = b.cpos[q * kCellSlots + k];
      const float4 mj = b.cax[q * kCellSlots + k];
      if (ok && pj.w > me.w && mi.x != 0.f &&
          ebond_near(make_float2(mi.x, mi.y), make_float2(mj.x, mj.y), fix_diff(me.x, pj.x, Lx),
                     fix_diff(me.y, pj.y, Ly), fix_diff(me.z, pj.z, Lz), thr, reach2)) {
        if (cnt < kMaxE) out[cnt] = (int)pj.w;
        ++cnt;
      }
    }
  }
  if (!ok) return;
  b.ecnt[me.w] = min(cnt, kMaxE);
  if (cnt > kMaxE) atomicOr(&b.eovf[cb.x], 1);
}

// blocks below nwblk: 32 rods against all higher indices of their system, the
// four warps a quarter each of every 128; the rest: cells
__global__ void __launch_bounds__(kPartBlock) ebond_screen_kernel(Batch b) {
  __shared__ uint32_t sx[kPartBlock], sy[kPartBlock], sz[kPartBlock];
  __shared__ float2 sme[kPartBlock];
  __shared__ int cnt[32];
  if ((int)blockIdx.x >= b.nwblk) {
    ebond_cells(b);
    return;
  }
  const int2 bk = b.wblk[blockIdx.x];
  const int s = bk.x;
  const SysDev& P = b.sys[s];
  if (P.cl_mode != 1 || (ebond_on_cells(b, P) && !b.st[s].cell_ovf)) return;  // the same for the whole block
  const int first = P.part_off, n = P.n, N = b.ntot;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = bk.y + lane;
  const bool ok = i < first + n;
  const float2* scr = reinterpret_cast<const float2*>(b.wev);
  uint32_t ux = 0, uy = 0, uz = 0;
  float2 mi = make_float2(0.f, 0.f);
  if (ok) {
    ux = b.pfx[i];
    uy = b.pfx[N + i];
    uz = b.pfx[2 * N + i];
    mi = scr[i];
  }
  if (w == 0) cnt[lane] = 0;
  const float Lx = P.Lfix[0], Ly = P.Lfix[1], Lz = P.Lfix[2];
  const float thr = (float)P.cl_ubond * 0.999f, reach = ebond_reach(P), reach2 = reach * reach;
  int* out = b.ecand + (long long)i * kMaxE;
  for (int q0 = (bk.y - first) / kPartBlock * kPartBlock; q0 < n; q0 += kPartBlock) {
    __syncthreads();
    if (q0 + (int)threadIdx.x < n) {
      const int q = first + q0 + threadIdx.x;
      sx[threadIdx.x] = b.pfx[q];
      sy[threadIdx.x] = b.pfx[N + q];
      sz[threadIdx.x] = b.pfx[2 * N + q];
      sme[threadIdx.x] = scr[q];
    }
    __syncthreads();
    if (!ok || mi.x == 0.f) continue;
    const int k1 = min(32 * w + 32, n - q0);
#pragma unroll 4
    for (int t = 32 * w; t < k1; ++t) {
      const int j = first + q0 + t;
      if (j > i && ebond_near(mi, sme[t], fix_diff(ux, sx[t], Lx), fix_diff(uy, sy[t], Ly), fix_diff(uz, sz[t], Lz),
                              thr, reach2)) {
        const int k = atomicAdd(&cnt[lane], 1);
        if (k < kMaxE) out[k] = j;
      }
    }
  }
  __syncthreads();
  if (ok && w == 0) {
    b.ecnt[i] = min(cnt[lane], kMaxE);
    if (cnt[lane] > kMaxE) atomicOr(&b.eovf[s], 1);
  }
}

// The screened candidates, exactly: a bond where the FP64 pair energy
// (pair_energy_ref, lower index first) is below -cl_ubond.  A block packs the
// candidates of its rods one per thread (few rods have any, and a pair is
// ~400 FP64 instructions of a warp however many of its lanes take part).
__global__ void __launch_bounds__(kPartBlock) ebond_eval_kernel(Batch b) {
  __shared__ int pre[kPartBlock + 1];
  __shared__ int wsum[kPartBlock / 32];
  const int2 bk = b.blk[blockIdx.x];
  const int s = bk.x;
  const SysDev& P = b.sys[s];
  if (P.cl_mode != 1) return;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const int nc = bk.y + t < P.part_off + P.n ? b.ecnt[bk.y + t] : 0;
  int inc = nc;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) inc += v;
  }
  if (lane == 31) wsum[w] = inc;
  __syncthreads();
  for (int v = 0; v < w; ++v) inc += wsum[v];
  pre[t + 1] = inc;
  if (t == 0) pre[0] = 0;
  __syncthreads();
  const int tot = pre[kPartBlock];
  for (int e = t; e < tot; e += kPartBlock) {
    int lo = 0;  // the rod of item e: the last with pre <= e
#pragma unroll
    for (int d = kPartBlock / 2; d; d >>= 1)
      if (pre[lo + d] <= e) lo += d;
    const int i = bk.y + lo, j = b.ecand[(long long)i * kMaxE + (e - pre[lo])];
    if (pair_energy_ref(b, P, i, j) < -P.cl_ubond) {
      const int k = atomicAdd(&b.ebcnt[i], 1);
      if (k < kMaxC) b.ebond[(long long)i * kMaxC + k] = j;
      else atomicOr(&b.eovf[s], 1);
    }
  }
}

__device__ __forceinline__ int find_root(const int* comp, int x) {
  int p = __ldcg(comp + x);
  while (p != x) {
    x = p;
    p = __ldcg(comp + x);
  }
  return x;
}

// Hook: for every bond, attach the larger root to the smaller one.  A bond
// retries until its ends share a root: where another bond took the larger
// root first, atomicMin leaves it at the smaller of the two new parents and
// the loop goes on to join the other, so one pass over the bonds joins them
// all and a component's root is its smallest index.
__global__ void __launch_bounds__(kPartBlock) cluster_hook_kernel(Batch b) {
  const int2 bk = b.blk[blockIdx.x];
  const SysDev& P = b.sys[bk.x];
  const int i = bk.y + threadIdx.x;
  if (i >= P.part_off + P.n) return;
  const bool en = P.cl_mode == 1;
  const int nc = en ? min(b.ebcnt[i], kMaxC) : b.nbc[i];
  const int* lst = en ? b.ebond + (long long)i * kMaxC : b.nb + (long long)i * kMaxNb;
  const unsigned char* fl = en ? nullptr : b.eflag + (long long)i * kMaxNb;
  for (int k = en ? 0 : b.nblo[i]; k < nc; ++k) {
    if (fl && !fl[k]) continue;
    int ra = find_root(b.comp, i), rb = find_root(b.comp, lst[k]);
    while (ra != rb) {
      const int hi = max(ra, rb), lo = min(ra, rb);
      const int old = atomicMin(&b.comp[hi], lo);
      if (old == hi) break;
      ra = find_root(b.comp, old);
      rb = find_root(b.comp, lo);
    }
  }
}

__global__ void __launch_bounds__(kPartBlock) cluster_compress_kernel(Batch b) {
  const int2 bk = b.blk[blockIdx.x];
  const SysDev& P = b.sys[bk.x];
  const int i = bk.y + threadIdx.x;
  if (i >= P.part_off + P.n) return;
  b.comp[i] = find_root(b.comp, i);
}

void launch_list_build(const Batch& b, int force_all, cudaStream_t s) {
  if (!b.nwblk) return;
  const int ncb = b.cells ? b.ncellblk : 0;
  if (ncb) cell_bin_kernel<<<b.nblk, kPartBlock, 0, s>>>(b, force_all);
  list_build_kernel<<<kListBlocks + ncb, kPartBlock, 0, s>>>(b, force_all);
}
// once per device: the step's memory split
cudaError_t prepare_wca() {
  return set_carveout(cell_bin_kernel, list_build_kernel, wca_screen_kernel<4>, wca_screen_kernel<8>,
                      wca_eval_kernel, wca_eval4_kernel);
}

// rows of 32 rods up to which the screen takes 8 lanes per rod
constexpr int kScreenWideMax = 1200;
// Batches of at most this many rows evaluate a pair on four lanes.  us per step on
// one lane and on four: 256 rods 34.4 and 33.2, 333 rods 35.8 and 33.5, 700 rods
// 37.5 and 34.3, 1500 rods with a cutoff 37.5 and 36.3, 2048 and 32,768 rods (1024
// rows) the same; 64 systems (1800 rows) 196.6 and 199, 192 systems 528 and 536,
// whose contacts fill the FP64 units.
constexpr int kEvalQuadMax = 1200;

// The WCA screen and evaluation.  The work list's length and the partners'
// slot counts are cleared with the working copies of every new configuration
// (particle_kernel); clear: here, for a screen that runs again without one.
void launch_wca(const Batch& b, bool clear, cudaStream_t s) {
  if (!b.nwblk) return;
  if (clear) {
    cudaMemsetAsync(b.wlist_n, 0, sizeof(int), s);
    cudaMemsetAsync(b.wincnt, 0, sizeof(int) * b.ntot, s);
  }
  if (b.nwblk <= kScreenWideMax)
    wca_screen_kernel<8><<<2 * b.nwblk, 128, 0, s>>>(b);
  else
    wca_screen_kernel<4><<<b.nwblk, 128, 0, s>>>(b);
  // a fixed grid (chosen by the autotuner); each thread loops over the list
  if (b.nwblk <= kEvalQuadMax)
    wca_eval4_kernel<<<b.tune.wca_blocks, 128, 0, s>>>(b);
  else
    wca_eval_kernel<<<b.tune.wca_blocks, 128, 0, s>>>(b);
}
void launch_cluster_bonds(const Batch& b, cudaStream_t s) {
  if (b.nwblk) cluster_bonds_kernel<<<b.nwblk * (32 * kBondLanes / 128), 128, 0, s>>>(b);
}
void launch_ebond(const Batch& b, cudaStream_t s) {
  if (!b.nblk || !b.ecand) return;
  const int ncb = b.cells ? b.ncellblk : 0;
  if (ncb) cudaMemsetAsync(b.ccnt, 0, sizeof(int) * b.ncellcap, s);
  ebond_prep_kernel<<<b.nblk, kPartBlock, 0, s>>>(b);
  ebond_screen_kernel<<<b.nwblk + ncb, kPartBlock, 0, s>>>(b);
  ebond_eval_kernel<<<b.nblk, kPartBlock, 0, s>>>(b);
}
void launch_cluster_hook(const Batch& b, cudaStream_t s) {
  if (b.nblk) cluster_hook_kernel<<<b.nblk, kPartBlock, 0, s>>>(b);
}
void launch_cluster_compress(const Batch& b, cudaStream_t s) {
  if (b.nblk) cluster_compress_kernel<<<b.nblk, kPartBlock, 0, s>>>(b);
}

}  // namespace mdsc
