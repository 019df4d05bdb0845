// Integrator, force assembly and per-system reductions -- the GPU form of
// moveTher / moveP / moveX / renorm / ext_field and of the driver's
// bookkeeping (v25/functions.cpp:1992-2025,2071-2218; v25/classes.cpp:228-325;
// v25/main.cpp:558-649).
//
// Precision: the master state (r, p, l, O, F, T) is FP64.  FP64 runs at a
// small fraction of the FP32 rate on this GPU, so the free-rotor update
// (five plane rotations in the body frame, J. Chem. Phys. 107, 5840, as
// Spherocyl::rotate does) is composed in FP32 as M = I + D, with every
// rotation entered as cos-1 = -2 sin^2(a/2) and sin a so that D keeps full
// FP32 *relative* precision (|D| ~ 1e-3 -> ~1e-10 absolute), and is applied
// to the FP64 orientation as O += D O.  Kicks, drifts and the thermostat
// scalars stay in FP64.
#include <algorithm>
#include <climits>
#include <type_traits>
#include <vector>

#include "mdsc_dev.cuh"
#include "reduce.cuh"

namespace mdsc {

// Spherocyl::renorm, v25/classes.cpp:307-325
__device__ __forceinline__ void renorm_O(double* o) {
  double norm = sqrt(o[6] * o[6] + o[7] * o[7] + o[8] * o[8]);
  o[6] /= norm; o[7] /= norm; o[8] /= norm;
  const double Up[3] = {o[6] + o[3], o[7] + o[4], o[8] + o[5]};
  const double d = Up[0] * o[6] + Up[1] * o[7] + Up[2] * o[8];
  o[3] = Up[0] - d * o[6];
  o[4] = Up[1] - d * o[7];
  o[5] = Up[2] - d * o[8];
  norm = sqrt(o[3] * o[3] + o[4] * o[4] + o[5] * o[5]);
  o[3] /= norm; o[4] /= norm; o[5] /= norm;
  o[0] = o[4] * o[8] - o[7] * o[5];
  o[1] = o[5] * o[6] - o[8] * o[3];
  o[2] = o[3] * o[7] - o[6] * o[4];
}

// one plane rotation of the composition: rows/components (i, j) turn by a
__device__ __forceinline__ void plane_rot(float a, int i, int j, float* lb, float* D) {
  float sh, ch;
  sincosf(0.5f * a, &sh, &ch);
  const float s = 2.f * sh * ch;
  const float cm1 = -2.f * sh * sh;  // cos a - 1 with full relative precision
  const float li = lb[i], lj = lb[j];
  lb[i] = li + (cm1 * li - s * lj);
  lb[j] = lj + (s * li + cm1 * lj);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const float di = D[3 * i + c], dj = D[3 * j + c];
    float ni = di + (cm1 * di - s * dj);
    float nj = dj + (s * di + cm1 * dj);
    if (c == i) { ni += cm1; nj += s; }
    if (c == j) { ni -= s; nj += cm1; }
    D[3 * i + c] = ni;
    D[3 * j + c] = nj;
  }
}

// K_r = l^T (O^T I^-1 O) l = sum_a (O l)_a^2 / I_a  (v25/functions.cpp:2123-2148)
__device__ __forceinline__ double rot_kin(const Batch& b, int i, const double* O, const double* l) {
  double kr = 0.0;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const double lb = O[3 * a] * l[0] + O[3 * a + 1] * l[1] + O[3 * a + 2] * l[2];
    kr += lb * lb * b.invI[3 * i + a];
  }
  return kr;
}

// ---------------------------------------------------------------------
// One rod on three lanes.  An FP64 instruction occupies a warp for 64 cycles
// here, however many independent ones follow it, so the per-particle kernels
// take a block of 32 rods and three warps, warp a the component a of every
// vector and row a of the orientation; what a component needs of the others
// goes through shared memory.  A third of the instructions per warp on three
// times the warps: one system's step waits for ~20 of them instead of ~60,
// and a batch that fills the GPU keeps the FP64 unit as busy as before.
// ---------------------------------------------------------------------
constexpr int kRows = 32;           // rods per block
constexpr int kRowBlock = 3 * kRows;

struct Shared3 {
  double l[3][kRows];
  double ax[3][kRows];
  double p[3][kRows];
  double lb2[3][kRows];
  float O[9][kRows];   // orientation before the move
  float O2[9][kRows];  // and after it
  float d2[3][kRows];
};

// Working copies of component a: fixed-point position, dipole positions and
// moment vectors, and (warp 2, which holds the rod axis) the FP32 axis and
// length; sh.O2 and sh.ax hold the new orientation.  Returns, in warp 2, how
// far the rod's ends may have moved since the last list build: the centre's
// move from the fixed-point coordinates (exact minimum image) plus half the
// length times the axis change (u_built, ax_built: its position component and
// axis at that build, loaded with the rest of the state).
__device__ __forceinline__ float derive_comp(const Batch& b, const SysDev& P, Shared3& sh, int a, int lane, int i,
                                             bool ok, double r, const double* O, uint32_t u_built,
                                             const float* ax_built) {
  const int N = b.ntot, ND = b.ndtot;
  const uint32_t u = to_fix(r, P.invL32[a]);
#pragma unroll
  for (int c = 0; c < 3; ++c) sh.O2[3 * a + c][lane] = soft_d2f_rn(O[c]);
  if (a == 2) {
#pragma unroll
    for (int c = 0; c < 3; ++c) sh.ax[c][lane] = O[c];
  }
  {
    const float d = fix_diff(u, u_built, P.Lfix[a]);
    sh.d2[a][lane] = d * d;
  }
  __syncthreads();
  float disp = 0.f;
  if (ok) {
    b.pfx[a * N + i] = u;
    const int nd = P.nd;
    const int g0 = P.dip_off + (i - P.part_off) * nd;
    const float o0 = sh.O2[a][lane], o1 = sh.O2[3 + a][lane], o2 = sh.O2[6 + a][lane];
    for (int w = 0; w < nd; ++w) {
      const int g = g0 + w;
      const double pc = b.dpc[g];
      b.dfx[a * ND + g] = pc == 0.0 ? u : to_fix(r + pc * sh.ax[a][lane], P.invL32[a]);
      // lab direction O^T o_body (Spherocyl::set_dip, v25/classes.cpp:166-170), times the moment
      const float ox = soft_d2f_rn(b.dob[3 * g]), oy = soft_d2f_rn(b.dob[3 * g + 1]),
                  oz = soft_d2f_rn(b.dob[3 * g + 2]);
      b.dm[a * ND + g] = soft_d2f_rn(b.dmu[g]) * (o0 * ox + o1 * oy + o2 * oz);
    }
    if (a == 2) {
      const float ln = soft_d2f_rn(b.len[i]);
      const float x[3] = {sh.O2[6][lane], sh.O2[7][lane], sh.O2[8][lane]};
      b.pax[i] = make_float4(x[0], x[1], x[2], ln);
      b.pdia[i] = soft_d2f_rn(b.dia[i]);
      float du2 = 0.f;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const float q = x[c] - ax_built[c];
        du2 += q * q;
      }
      disp = sqrtf(sh.d2[0][lane] + sh.d2[1][lane] + sh.d2[2][lane]) + 0.5f * ln * sqrtf(du2);
    }
  }
  return disp;
}

// the block's largest displacement measure, from warp 2 (non-negative, so its
// bits order as integers)
__device__ __forceinline__ void store_disp(const Batch& b, SysState& S, int row, int a, float disp) {
  if (a != 2) return;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) disp = fmaxf(disp, __shfl_xor_sync(0xffffffffu, disp, off));
  if ((threadIdx.x & 31) == 0) {
    b.dmax[row] = disp;
    atomicMax(&S.dmax, __float_as_int(disp));
  }
}

// A particle's kinetic energies, doubled: translational from its momentum,
// rotational, sum_a (O l)_a^2 / I_a (v25/functions.cpp:2123-2148), from the
// squares; each by one warp, in the order of the components.
__device__ __forceinline__ double kin_t(const double (&p)[3][kRows], int lane, double invm) {
  double psq = 0.0;
#pragma unroll
  for (int c = 0; c < 3; ++c) psq += p[c][lane] * p[c][lane];
  return psq * invm;
}
__device__ __forceinline__ double kin_r(const Batch& b, const double (&lb2)[3][kRows], int lane, int i) {
  double k = 0.0;
#pragma unroll
  for (int c = 0; c < 3; ++c) k += lb2[c][lane] * b.invI[3 * i + c];
  return k;
}

// The row's kinetic energies, translational by warp 0 and rotational by warp
// 1, after the rest of the kernel: nothing before the second half kick reads
// them.
__device__ __forceinline__ void store_kin(const Batch& b, const Shared3& sh, int row, int a, int lane, int i, bool ok) {
  if (a == 2) return;
  const double v = !ok ? 0.0 : a == 0 ? kin_t(sh.p, lane, b.invm[i]) : kin_r(b, sh.lb2, lane, i);
  const FF k = ff_warp_sum(ff_from(v));
  if (lane == 0) b.krow[2 * row + a] = make_float2(k.hi, k.lo);
}

// the free-rotor move of the step (Spherocyl::rotate, v25/classes.cpp:240-304):
// row a of the increment D O from the FP32 orientation and angular momentum;
// every warp composes the rotation
__device__ __forceinline__ void rotor_row(const Batch& b, const Shared3& sh, int a, int lane, int i, double dt,
                                          float* inc) {
  const float iI0 = soft_d2f_rn(b.invI[3 * i]), iI1 = soft_d2f_rn(b.invI[3 * i + 1]),
              iI2 = soft_d2f_rn(b.invI[3 * i + 2]);
  const float fdt = soft_d2f_rn(dt), h = 0.5f * fdt;
  const float lf[3] = {soft_d2f_rn(sh.l[0][lane]), soft_d2f_rn(sh.l[1][lane]), soft_d2f_rn(sh.l[2][lane])};
  float Of[9], lb[3], D[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) Of[k] = sh.O[k][lane];
#pragma unroll
  for (int k = 0; k < 3; ++k) lb[k] = Of[3 * k] * lf[0] + Of[3 * k + 1] * lf[1] + Of[3 * k + 2] * lf[2];
#pragma unroll
  for (int k = 0; k < 9; ++k) D[k] = 0.f;
  plane_rot(-lb[0] * h * iI0, 1, 2, lb, D);   // Rx
  plane_rot(-lb[1] * h * iI1, 2, 0, lb, D);   // Ry
  plane_rot(-lb[2] * fdt * iI2, 0, 1, lb, D); // Rz
  plane_rot(-lb[1] * h * iI1, 2, 0, lb, D);   // Ry
  plane_rot(-lb[0] * h * iI0, 1, 2, lb, D);   // Rx
  // O += D O: the increment (|D| ~ 1e-3) in FP32, ~1e-10 absolute like D
  // itself, added to the FP64 orientation
  const float d0 = a == 0 ? D[0] : (a == 1 ? D[3] : D[6]), d1 = a == 0 ? D[1] : (a == 1 ? D[4] : D[7]),
              d2 = a == 0 ? D[2] : (a == 1 ? D[5] : D[8]);
#pragma unroll
  for (int c = 0; c < 3; ++c) inc[c] = d0 * Of[c] + d1 * Of[3 + c] + d2 * Of[6 + c];
}

// ---------------------------------------------------------------------
// first half of the step: moveTher(0), [renorm], moveP(first), moveX
// (v25/functions.cpp:2071-2149); kPartMoveX: moveX alone; kPartDerive: only the
// working copies and the displacement measure; kPartCopies: only the copies, for
// calls that decide no list (the system's maximum counts up until a pass that
// reads the lists clears it)
// ---------------------------------------------------------------------
// Measured against one lane per rod in blocks of 128 (with the force assembly
// below and the per-system sums on lanes): a step of 256 rods 62.4 -> 51.8 us,
// of 4096 rods 113 -> 93.7, of 32,768 rods 2205 -> 2135, of 64 systems 223 ->
// 215, of 256 systems 688 -> 688 (FP64 throughput and the state's reads).
enum : int { kPartDerive = 0, kPartMoveX = 1, kPartStep = 2, kPartCopies = 3 };

template <int MODE>
__global__ void __launch_bounds__(kRowBlock) particle_kernel(Batch b) {
  __shared__ Shared3 sh;
  __shared__ double sfac[2];
  const int2 bk = b.wblk[blockIdx.x];
  const int s = bk.x;
  if (blockIdx.x == 0 && threadIdx.x == 0) *b.wlist_n = 0;
  if (MODE == kPartStep && at_limit(b, s)) return;
  const SysDev& P = b.sys[s];
  SysState& S = b.st[s];
  const int a = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool ok = bk.y + lane < P.part_off + P.n;
  const int i = ok ? bk.y + lane : bk.y;  // lanes past the end repeat the first rod and store nothing
  const int row = P.w_off + (bk.y - P.part_off) / kRows;
  // what the lists and the WCA screen of the new configuration count up from:
  // the partners' slots, and the cells (at most one per 8 rods)
  if (a == 0 && ok) b.wincnt[i] = 0;
  if (a == 1 && bk.y == P.part_off && lane == 0 && S.rebuild) S.list_ok = 1;
  if (P.ncell > 0 && a == 1) {
    const int c = (bk.y - P.part_off) / 8 + lane;
    if (lane < kRows / 8 && c < P.ncell) b.ccnt[P.cell_off + c] = 0;
    if (bk.y == P.part_off && lane == 0) S.cell_ovf = 0;
  }
  double r = b.r[3 * i + a], O[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) O[c] = b.O[9 * i + 3 * a + c];
  const uint32_t u_built = b.fsave[3 * i + a];
  float ax_built[3] = {0.f, 0.f, 0.f};
  if (a == 2) {
#pragma unroll
    for (int c = 0; c < 3; ++c) ax_built[c] = b.usave[3 * i + c];
  }
  if constexpr (MODE == kPartMoveX || MODE == kPartStep) {
    double p = b.p[3 * i + a], l = b.l[3 * i + a];
    const double im = b.invm[i];
    if constexpr (MODE == kPartStep) {
      const double h = 0.5 * P.dt, F = b.F[3 * i + a], T = b.T[3 * i + a];
      if (threadIdx.x < 2) {
        // moveTher mode 0 (v25/functions.cpp:2193-2202); noise drawn on the host
        const double* nz = b.noise + ((long long)S.iter * b.nsys + s) * 4;
        const double x = P.ex1 * S.xi[threadIdx.x] + P.cnoise * nz[2 * threadIdx.x];
        sfac[threadIdx.x] = 1.0 / (1.0 + 0.5 * P.dt * x);
      }
      if (S.step % 100 == 0) {  // v25/main.cpp:556-563
        double A[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) A[k] = b.O[9 * i + k];
        renorm_O(A);
#pragma unroll
        for (int c = 0; c < 3; ++c) O[c] = a == 0 ? A[c] : (a == 1 ? A[3 + c] : A[6 + c]);
      }
      __syncthreads();
      // moveP first half (v25/functions.cpp:2129-2149)
      p = (p + h * F) * sfac[0];
      l = (l + h * T) * sfac[1];
    }
    sh.l[a][lane] = l;
#pragma unroll
    for (int c = 0; c < 3; ++c) sh.O[3 * a + c][lane] = soft_d2f_rn(O[c]);
    __syncthreads();
    if constexpr (MODE == kPartStep) {
      // the kinetic energies before the move, in store_kin
      const double lb = O[0] * sh.l[0][lane] + O[1] * sh.l[1][lane] + O[2] * sh.l[2][lane];
      sh.p[a][lane] = p;
      sh.lb2[a][lane] = lb * lb;
      if (ok) {
        b.p[3 * i + a] = p;
        b.l[3 * i + a] = l;
      }
    }
    // moveX (v25/functions.cpp:2071-2092)
    r += P.dt * p * im;
    float inc[3];
    rotor_row(b, sh, a, lane, i, P.dt, inc);
#pragma unroll
    for (int c = 0; c < 3; ++c) O[c] += soft_f2d(inc[c]);
    if (ok) {
      b.r[3 * i + a] = r;
#pragma unroll
      for (int c = 0; c < 3; ++c) b.O[9 * i + 3 * a + c] = O[c];
    }
  }
  const float disp = derive_comp(b, P, sh, a, lane, i, ok, r, O, u_built, ax_built);
  if constexpr (MODE == kPartDerive || MODE == kPartStep) store_disp(b, S, row, a, disp);
  if constexpr (MODE == kPartStep) store_kin(b, sh, row, a, lane, i, ok);
}

// Thermostat coordinates of the second half kick, moveTher 0 then 1
// (v25/functions.cpp:2193-2206), from the first-half kinetic energies: a
// block per system, beside the force chains (only the second kick reads them).
// The rows of 128 particles are added in float-float and those sums in FP64,
// in order: the thermostat feeds back on every momentum, so its last bits stay
// what they were when a block of 128 threads summed its particles.
__global__ void __launch_bounds__(128) xi_mid_kernel(Batch b) {
  __shared__ double sh[2][128];
  const int s = blockIdx.x;
  const SysDev& P = b.sys[s];
  SysState& S = b.st[s];
  const bool off = at_limit(b, s);
  if (threadIdx.x == 0) S.stepping = !off;
  if (off) return;
  const int nb = cdiv(P.nw, 4), c = threadIdx.x;
  double K = 0.0, x1 = 0.0;
  if (c < 2) x1 = P.ex1 * S.xi[c] + P.cnoise * b.noise[((long long)S.iter * b.nsys + s) * 4 + 2 * c];
  for (int b0 = 0; b0 < nb; b0 += 128) {
    const int blk = b0 + threadIdx.x;
    if (blk < nb) {
      const float4* in = reinterpret_cast<const float4*>(b.krow) + P.w_off + 4 * blk;
      float4 x[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) x[q] = 4 * blk + q < P.nw ? in[q] : make_float4(0.f, 0.f, 0.f, 0.f);
      FF t{x[0].x, x[0].y}, r{x[0].z, x[0].w};
#pragma unroll
      for (int q = 1; q < 4; ++q) {
        t = ff_add(t, FF{x[q].x, x[q].y});
        r = ff_add(r, FF{x[q].z, x[q].w});
      }
      sh[0][threadIdx.x] = soft_f2d(t.hi) + soft_f2d(t.lo);
      sh[1][threadIdx.x] = soft_f2d(r.hi) + soft_f2d(r.lo);
    }
    __syncthreads();
    if (c < 2) {
#pragma unroll 8
      for (int k = 0; k < min(128, nb - b0); ++k) K += sh[c][k];
    }
    __syncthreads();
  }
  if (c >= 2) return;
  const double Kf = 0.5 * K;
  S.K_first[c] = Kf;
  S.xi_mid[c] = x1 + P.dt * (2. * Kf - P.ntemp3) / P.Q;
}

// ---------------------------------------------------------------------
// oo_params' terms (v25/functions.cpp:2720-2760, Qmat_3d :3426-3445) per
// particle block, from the FP32 working copies of this step's orientations:
// the rod axis o, o o^T and the dipole vectors mu o_dipole, float-float
// block sums.  Its own small kernel, early in the step on the WCA stream:
// widening finalize's sums cost that kernel occupancy.
__device__ __forceinline__ void order_terms_block(const Batch& b, int block) {
  __shared__ double sh[12 * kPartBlock / 32];
  const int2 bk = b.blk[block];
  if (at_limit(b, bk.x)) return;
  const SysDev& P = b.sys[bk.x];
  const int i = bk.y + threadIdx.x;
  FF v[12];
#pragma unroll
  for (int c = 0; c < 12; ++c) v[c].hi = v[c].lo = 0.f;
  if (i < P.part_off + P.n) {
    const float4 q = b.pax[i];
    const float t[9] = {q.x, q.y, q.z, q.x * q.x, q.x * q.y, q.x * q.z, q.y * q.y, q.y * q.z, q.z * q.z};
#pragma unroll
    for (int c = 0; c < 9; ++c) v[c] = ff_of(t[c]);
    const int ND = b.ndtot, g0 = P.dip_off + (i - P.part_off) * P.nd;
    for (int w = 0; w < P.nd; ++w) {
#pragma unroll
      for (int a = 0; a < 3; ++a) v[9 + a] = ff_add(v[9 + a], ff_of(b.dm[a * ND + g0 + w]));
    }
  }
  double tot[12];
  block_sum<12, kPartBlock>(v, sh, tot);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int c = 0; c < 12; ++c) b.obk[12 * blk_slot(P, bk) + c] = tot[c];
  }
}

__global__ void __launch_bounds__(kPartBlock) order_terms_kernel(Batch b) { order_terms_block(b, blockIdx.x); }

// ---------------------------------------------------------------------
// force assembly (+ ext_field) and optionally moveP(last): three lanes per
// rod as above, twice.  Warps 3 to 5 add the WCA pairs' shares while warps 0
// to 2 add the dipoles' real- and reciprocal-space parts and then, from both,
// make the kick: a chain of dependent reads each (records by slot; partials by
// tile), one behind the other 10.0 us a launch for 256 rods, side by side 6.9.
// Each warp leaves its sums for the per-system reduction as float-float rows:
// krow2 (K_t or K_r, two kinetic pressure terms, U_ext) and wrow (the WCA terms
// a, a + 3, ... of U, W, PT of the rods' own pairs).
// ---------------------------------------------------------------------
constexpr int kKinCols = 4, kWcaCols = 4;
// kinetic pressure terms of warp a: (xx, xy), (yy, yz), (zz, zx)

// warps 0 to 2 only
__device__ __forceinline__ void sync_rows() { asm volatile("bar.sync 1, %0;" ::"n"(kRowBlock) : "memory"); }

// k-space force and torque of dipole w (g) of rod i, component a, from the k
// tiles' sums: the force, and the torque m x G of the second triple with the
// FP32 moment, as the gather forms them where it walks all tiles.  Called by
// all of warps 0 to 2.
__device__ __forceinline__ void ktile_force(const Batch& b, const SysDev& P, FF (&sg)[3][kRows], int i, int g, int w,
                                            int a, int lane, FF& kf, FF& kt) {
  const int a1 = a == 2 ? 0 : a + 1, a2 = a == 0 ? 2 : a - 1;
  const float* set = ktile_set(b, P, i, 0) + (w * 6 + a) * kPartBlock;
  FF q[2];
  ktile_sums<6>(set, P.nkt, P.nd * kSet, 3 * kPartBlock, P.kgs, q);
  kf = q[0];
  const float m1 = b.dm[a1 * b.ndtot + g], m2 = b.dm[a2 * b.ndtot + g];
  sync_rows();
  sg[a][lane] = q[1];
  sync_rows();
  kt = ff_cross(m1, sg[a2][lane], m2, sg[a1][lane]);
}

// ORDER: the order-parameter blocks (their first kPartBlock threads) in the same
// launch, behind the rows: the function-level calls run one kernel after
// another, and a kernel for the order terms was 5.4 us of each of them.
// TWO: the two halves side by side (warps 3 to 5 the pairs), else one behind the
// other by three warps (kFinalizeTwoMax).
template <bool ORDER, bool TWO>
__global__ void __launch_bounds__((TWO ? 2 : 1) * kRowBlock, TWO ? 5 : 10) finalize_kernel(Batch b, int mode) {
  if constexpr (ORDER) {
    if ((int)blockIdx.x >= b.nwblk) {
      if (threadIdx.x < kPartBlock) order_terms_block(b, blockIdx.x - b.nwblk);
      return;
    }
  }
  __shared__ double sw[2][3][TWO ? kRows : 1];  // F, T with the WCA pairs' shares
  __shared__ double sl[3][kRows], sv[3][kRows], sf[3][kRows];
  __shared__ float sp[3][kRows];
  __shared__ double sk[2][3][kRows];  // p; (O l)_a^2
  __shared__ FF sg[3][kRows];
  const int2 bk = b.wblk[blockIdx.x];
  const int s = bk.x;
  if (at_limit(b, s)) return;
  const SysDev& P = b.sys[s];
  SysState& S = b.st[s];
  const bool pairs = TWO && threadIdx.x >= kRowBlock;  // the same for a warp
  const int a = (threadIdx.x >> 5) - (pairs ? 3 : 0), lane = threadIdx.x & 31;
  const bool ok = bk.y + lane < P.part_off + P.n;
  const int i = ok ? bk.y + lane : bk.y;
  const int row = 3 * (P.w_off + (bk.y - P.part_off) / kRows) + a;
  double F = 0.0, T = 0.0;
  if (!TWO || pairs) {
    if (bk.y == P.part_off && a == 0 && lane == 0) S.dmax = 0;  // the lists of this configuration stand
    F = (mode & kFlagAccum) ? b.F[3 * i + a] : 0.0;
    T = (mode & kFlagAccum) ? b.T[3 * i + a] : 0.0;
    FF w[kWcaCols];
#pragma unroll
    for (int c = 0; c < kWcaCols; ++c) w[c] = ff_of(0.f);
    if ((mode & kMaskWca) && ok) {
      const int nc = b.wcnt[i];
      const int nin = min(b.wincnt[i], kMaxC);
      const int4* win = reinterpret_cast<const int4*>(b.win + (long long)i * kMaxC);
      int v[kMaxC];
#pragma unroll
      for (int q = 0; q < kMaxC / 4; ++q) {
        const int4 x = 4 * q < nin ? win[q] : make_int4(0, 0, 0, 0);
        v[4 * q] = 4 * q < nin ? x.x : INT_MAX;
        v[4 * q + 1] = 4 * q + 1 < nin ? x.y : INT_MAX;
        v[4 * q + 2] = 4 * q + 2 < nin ? x.z : INT_MAX;
        v[4 * q + 3] = 4 * q + 3 < nin ? x.w : INT_MAX;
      }
      // its own shares of its candidate pairs (higher-index partners), in
      // slot order, as force_sc adds them
      const double* own = b.wown + (long long)i * kMaxC * 6;
      const double* ev = b.wev + (long long)i * kMaxC * 11;
      for (int c = 0; c < nc; ++c) {
        F += own[6 * c + a];
        T += own[6 * c + 3 + a];
#pragma unroll
        for (int q = 0; q < kWcaCols; ++q)
          if (a + 3 * q < 11) w[q] = ff_add(w[q], ff_from(ev[11 * c + a + 3 * q]));
      }
      // shares of the pairs this particle forms with lower-index partners,
      // left by the WCA kernel in the partner's records.  The screen listed
      // their slots here in arrival order; taken in ascending order the slots
      // ascend with the partner (slot = partner * kMaxC + c), the order
      // force_sc adds them.
      int last = -1;
      for (int k = 0; k < nin; ++k) {
        int m = INT_MAX;
#pragma unroll
        for (int q = 0; q < kMaxC; ++q) m = min(m, v[q] > last ? v[q] : INT_MAX);
        const double* rec = b.wrec + (long long)m * 6;
        F += rec[a];
        T += rec[3 + a];
        last = m;
      }
    }
    if constexpr (TWO) {
      sw[0][a][lane] = F;
      sw[1][a][lane] = T;
      __syncthreads();
    }
    if (mode & kMaskWca) {
#pragma unroll
      for (int c = 0; c < kWcaCols; ++c) {
        w[c] = ff_warp_sum(w[c]);
        if (lane == 0) b.wrow[kWcaCols * row + c] = make_float2(w[c].hi, w[c].lo);
      }
    }
    if constexpr (TWO) return;
  }
  const int a1 = a == 2 ? 0 : a + 1, a2 = a == 0 ? 2 : a - 1;  // the cyclic next and previous component
  const bool kick = mode & kFlagMoveP;
  double p = 0.0, l = 0.0, im = 0.0, O[3] = {0.0, 0.0, 0.0};
  if (kick) {  // asked for ahead of the forces
    p = b.p[3 * i + a];
    l = b.l[3 * i + a];
    im = b.invm[i];
#pragma unroll
    for (int c = 0; c < 3; ++c) O[c] = b.O[9 * i + 3 * a + c];
  }
  const int nd = P.nd;
  // the field term needs the FP64 moment; without a field it adds nothing
  const bool ext = (mode & kMaskExt) && (P.B[0] != 0.0 || P.B[1] != 0.0 || P.B[2] != 0.0);
  double uext = 0.0;
  for (int w = 0; w < max(nd, 1); ++w) {
    double f = 0.0, t = 0.0;
    if (w < nd) {
      const int g = P.dip_off + (i - P.part_off) * nd + w;
      const double pc = b.dpc[g];
      // real- and reciprocal-space force and torque of this dipole in
      // float-float (FP32 instructions), one conversion to FP64 at the end
      FF qf = ff_of(0.f), qt = ff_of(0.f);
      if (mode & kMaskReal) {
        // this dipole's tile partials summed over all partner strips: here, or
        // by real_sum_kernel (or near_pass_kernel) before
        if (P.rc_real <= 0.0 && P.nstrip <= kStripRows) {
          const int loc = g - P.dip_off;
          const float* part = b.rpart + P.pp_off + ((long long)(loc / kTile) * P.nstrip * 6 + a) * kTile + loc % kTile;
          FF q[2];
          strip_sums<8>(part, P.nstrip, 6 * kTile, 3 * kTile, q);
          qf = q[0];
          qt = q[1];
        } else {
          const float2 x = b.rsum[(long long)a * b.ndtot + g], y = b.rsum[(long long)(3 + a) * b.ndtot + g];
          qf = FF{x.x, x.y};
          qt = FF{y.x, y.y};
        }
      }
      if (mode & kMaskK) {
        FF kf, kt;
        if (P.kgt > 1) {
          ktile_force(b, P, sg, i, g, w, a, lane, kf, kt);
        } else {
          const float2 x = b.Fk[3 * g + a], y = b.Tk[3 * g + a];
          kf = FF{x.x, x.y};
          kt = FF{y.x, y.y};
        }
        qf = ff_add(qf, kf);
        qt = ff_add(qt, kt);
      }
      f = soft_f2d(qf.hi) + soft_f2d(qf.lo);
      t = soft_f2d(qt.hi) + soft_f2d(qt.lo);
      if (ext) {
        // ext_field: torque mu o x B, energy -mu o.B (v25/functions.cpp:2014-2020),
        // with the dipole vector mu O^T o_body in FP64
        const double* Oi = b.O + 9 * i;
        const double m = b.dmu[g] * (Oi[a] * b.dob[3 * g] + Oi[3 + a] * b.dob[3 * g + 1] + Oi[6 + a] * b.dob[3 * g + 2]);
        sync_rows();
        sv[a][lane] = m;
        sync_rows();
        t += sv[a1][lane] * P.B[a2] - sv[a2][lane] * P.B[a1];
        // by one warp: the three products cancel in FP64, not in the rows' 48 bits
        if (a == 0) uext -= sv[0][lane] * P.B[0] + sv[1][lane] * P.B[1] + sv[2][lane] * P.B[2];
      }
      // lever arm of an off-centre dipole: d x f (v25/classes.hpp:135-136)
      sync_rows();
      sf[a][lane] = f;
      sync_rows();
      if (pc != 0.0) t += pc * b.O[9 * i + 6 + a1] * sf[a2][lane] - pc * b.O[9 * i + 6 + a2] * sf[a1][lane];
    }
    if (TWO && w == 0) {
      __syncthreads();  // the pairs' shares come first
      F = sw[0][a][lane];
      T = sw[1][a][lane];
    }
    if (w < nd) {
      F += f;
      T += t;
    }
  }
  // warp 0: K_t, warp 1: K_r; then two terms of the pressure tensor, U_ext
  FF k[kKinCols];
#pragma unroll
  for (int c = 0; c < kKinCols; ++c) k[c] = ff_of(0.f);
  k[3] = ff_from(ok ? uext : 0.0);
  if (ok) {
    b.F[3 * i + a] = F;
    b.T[3 * i + a] = T;
  }
  if (kick) {
    // moveP last half (v25/functions.cpp:2150-2173), with xi after moveTher
    // 0 and 1 (xi_mid_kernel)
    const double h = 0.5 * P.dt;
    // (the products' roundings written out: both kicks keep their last bits)
    p = __fma_rn(p, 1. - h * S.xi_mid[0], h * F);
    l = __fma_rn(l, 1. - h * S.xi_mid[1], h * T);
    sl[a][lane] = l;
    sp[a][lane] = soft_d2f_rn(p);
    sk[0][a][lane] = p;
    sync_rows();
    const double lb = O[0] * sl[0][lane] + O[1] * sl[1][lane] + O[2] * sl[2][lane];
    sk[1][a][lane] = lb * lb;
    if (ok) {
      b.p[3 * i + a] = p;
      b.l[3 * i + a] = l;
      if (a == 0) k[0] = ff_from(kin_t(sk[0], lane, im));
      // kinetic pressure tensor p_a p_b / m: FP32 products, float-float sums
      const float imf = soft_d2f_rn(im), pf = sp[a][lane];
      k[1] = ff_of(pf * pf * imf);
      k[2] = ff_of(pf * sp[a1][lane] * imf);
    }
    sync_rows();
    if (ok && a == 1) k[0] = ff_from(kin_r(b, sk[1], lane, i));
  }
#pragma unroll
  for (int c = 0; c < kKinCols; ++c) {
    k[c] = ff_warp_sum(k[c]);
    if (lane == 0) b.krow2[kKinCols * row + c] = make_float2(k[c].hi, k[c].lo);
  }
}

// ---------------------------------------------------------------------
// per-system sums and the thermostat's last update.  kRedGroups blocks per
// system, one per group of sums (real-space tiles, k tiles, WCA pairs,
// kinetic terms, order parameters), each in float-float with a fixed order;
// the kinetic block also closes the step's thermostat and bookkeeping.  The
// warps' sums are added and converted one value per lane: an FP64 addition
// per value in one thread would cost 64 cycles each.
constexpr int kRedThreads = 128;
// HOME: into the host's observables as well (a step's kernel without it: 1 us
// shorter).
template <bool HOME>
__global__ void __launch_bounds__(kRedThreads) reduce_obs_kernel(Batch b, int mode) {
  constexpr int NV = 12;
  __shared__ FF sh[NV][kRedThreads / 32];
  const int s = blockIdx.x / kRedGroups, grp = blockIdx.x % kRedGroups;
  const SysDev& P = b.sys[s];
  SysState& S = b.st[s];
  SysObs& ob = b.obs[s];
  // In a step not by the step count, which the kinetic block advances: a block
  // of the same system that started behind it would take the last step before
  // the limit for one beyond it.
  if ((mode & kRedStep) ? !S.stepping : at_limit(b, s)) return;
  FF v[NV];
#pragma unroll
  for (int c = 0; c < NV; ++c) v[c] = ff_of(0.f);
  if (grp == 2) {
    // columns q of warp a of every row: term a + 3 q of U, W, PT
    for (int t = threadIdx.x; t < P.nw; t += kRedThreads) {
      const float2* w = b.wrow + (long long)(P.w_off + t) * 3 * kWcaCols;
#pragma unroll
      for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int q = 0; q < kWcaCols; ++q)
          if (a + 3 * q < 11) v[a + 3 * q] = ff_add(v[a + 3 * q], FF{w[kWcaCols * a + q].x, w[kWcaCols * a + q].y});
    }
  } else if (grp == 3) {
    // K_t, K_r, then (xx xy)(yy yz)(zz zx), U_ext.  K_t and K_r by blocks of
    // 128 particles, as in xi_mid_kernel
    const float2* k = b.krow2 + (long long)P.w_off * 3 * kKinCols;
    for (int t = threadIdx.x; t < cdiv(P.nw, 4); t += kRedThreads) {
      float2 x[4][2];
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int c = 0; c < 2; ++c)
          x[q][c] = 4 * t + q < P.nw ? k[((4 * t + q) * 3 + c) * kKinCols] : make_float2(0.f, 0.f);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        FF y{x[0][c].x, x[0][c].y};
#pragma unroll
        for (int q = 1; q < 4; ++q) y = ff_add(y, FF{x[q][c].x, x[q][c].y});
        v[c] = ff_add(v[c], ff_from(soft_f2d(y.hi) + soft_f2d(y.lo)));
      }
    }
    // from the last thread down: in small systems beside the sums above
    for (int t = kRedThreads - 1 - threadIdx.x; t < P.nw; t += kRedThreads) {
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const float2* q = k + (3 * t + a) * kKinCols;
        v[2 + 2 * a] = ff_add(v[2 + 2 * a], FF{q[1].x, q[1].y});
        v[3 + 2 * a] = ff_add(v[3 + 2 * a], FF{q[2].x, q[2].y});
        v[8] = ff_add(v[8], FF{q[3].x, q[3].y});
      }
    }
  } else {
    // the rows of one per-system table, column by column: real-space tiles
    // (U, PT; FP32), in large systems strips (each strip's tiles summed by
    // strip_energy) or the neighbour pass's blocks, k tiles (U, PT) or
    // order-parameter blocks, through one code path
    const float* fsrc = nullptr;
    const double* dsrc = nullptr;
    int nrow, ncol = 10;
    if (grp == 0 && P.rc_real > 0.0) {
      dsrc = b.rlE + (long long)P.blk_off * 10;
      nrow = P.nblk;
    } else if (grp == 0 && P.nstrip > kStripRows) {
      dsrc = b.stripE + (long long)P.strip_off * 10;
      nrow = P.nstrip;
    } else if (grp == 0) {
      fsrc = b.tileE + (long long)P.tile_off * 10;
      nrow = P.ntile;
    } else if (grp == 1) {
      dsrc = b.kE + (long long)P.kt_off * 10;
      nrow = P.nkt;
    } else {
      dsrc = b.obk + (long long)P.blk_off * 12;
      nrow = P.nblk;
      ncol = 12;
    }
    for (int t = threadIdx.x; t < nrow; t += kRedThreads) {
#pragma unroll
      for (int c = 0; c < NV; ++c) {
        if (c < ncol) {
          const long long e = (long long)t * ncol + c;
          v[c] = ff_add(v[c], fsrc ? ff_of(fsrc[e]) : ff_from(dsrc[e]));
        }
      }
    }
  }
#pragma unroll
  for (int c = 0; c < NV; ++c) {
    v[c] = ff_warp_sum(v[c]);
    if ((threadIdx.x & 31) == 0) sh[c][threadIdx.x >> 5] = v[c];
  }
  __syncthreads();
  const int c = threadIdx.x;
  if (c >= 32) return;
  double x = 0.0;
  if (c < NV) {
    const FF t = ff_add(ff_add(ff_add(sh[c][0], sh[c][1]), sh[c][2]), sh[c][3]);
    x = soft_f2d(t.hi) + soft_f2d(t.lo);
  }
  auto put = [&](auto& field, auto v) {
    field = v;
    if constexpr (HOME) {
      const long long home = (char*)(b.obs_host + s) - (char*)&ob;
      *reinterpret_cast<std::remove_reference_t<decltype(field)>*>((char*)&field + home) = v;
    }
  };
  if (grp == 0) {
    if (c == 0) put(ob.U_dipR, x);
    else if (c < 10) put(ob.PT_dipR[c - 1], x);
  } else if (grp == 1) {
    if (c == 0) put(ob.U_dipK, x);
    else if (c < 10) put(ob.PT_dipK[c - 1], x);
  } else if (grp == 2) {
    if (c == 0) put(ob.U_ss, x);
    else if (c == 1) put(ob.W_ss, x);
    else if (c < 11) put(ob.PT_ss[c - 2], x);
  } else if (grp == 4) {
    if (c < 12) put(ob.osum[c], x);
  } else {
    if (c == 8) {
      put(ob.U_ext, x);
      put(ob.U_self, P.Uself);
    }
    if (mode & kRedStep) {
      if (c < 2) {
        put(ob.K[c], 0.5 * x);
        // moveTher mode 2 (v25/functions.cpp:2207-2213) closes the step
        const double g = b.noise[((long long)S.iter * b.nsys + s) * 4 + 2 * c + 1];
        const double xi = P.ex1 * S.xi_mid[c] + P.cnoise * g;
        S.xi[c] = xi;
        S.strn[c] = g;
        put(ob.xi[c], xi);
      } else if (c < 8) {
        // (xx xy)(yy yz)(zz zx) to their places and mirrors
        const int a = (c - 2) >> 1, q = (c & 1) ? (a + 1) % 3 : a;
        put(ob.PT_kin[3 * a + q], x);
        put(ob.PT_kin[3 * q + a], x);
      }
      __syncwarp();
      if (c == 0) {
        S.step += 1;
        S.iter += 1;
        // a list asked for counts with the step that would have built it, also
        // where a force evaluation of the same state had built it already
        if (S.rebuild || S.force_list) S.list_builds += 1;
        S.force_list = 0;
      }
      __syncwarp();
    } else if (c < 2) {
      put(ob.xi[c], S.xi[c]);
    }
    if (c == 0) {
      put(ob.step, S.step);
      put(ob.status, S.status);
      put(ob.list_builds, S.list_builds);
    }
  }
}

// ---------------------------------------------------------------------
// function-level entry points
// ---------------------------------------------------------------------
__global__ void __launch_bounds__(kPartBlock) renorm_kernel(Batch b) {
  const int2 bk = b.blk[blockIdx.x];
  const SysDev& P = b.sys[bk.x];
  const int i = bk.y + threadIdx.x;
  if (i >= P.part_off + P.n) return;
  double O[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) O[k] = b.O[9 * i + k];
  renorm_O(O);
#pragma unroll
  for (int k = 0; k < 9; ++k) b.O[9 * i + k] = O[k];
}

// moveP with caller-given thermostat coordinates xi[2*sys]; partial sums
// K_t, K_r, PT (6) per block into kin2
__global__ void __launch_bounds__(kPartBlock) movep_kernel(Batch b, const double* __restrict__ xi,
                                                          int last) {
  __shared__ double sh[9 * kPartBlock / 32];
  const int2 bk = b.blk[blockIdx.x];
  const int s = bk.x;
  const SysDev& P = b.sys[s];
  const int i = bk.y + threadIdx.x;
  double acc[9];
#pragma unroll
  for (int c = 0; c < 9; ++c) acc[c] = 0.0;
  if (i < P.part_off + P.n) {
    const double h = 0.5 * P.dt;
    double p[3], l[3], O[9];
    double psq = 0.0;
#pragma unroll
    for (int k = 0; k < 9; ++k) O[k] = b.O[9 * i + k];
    const double xt = xi[2 * s], xr = xi[2 * s + 1];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const double p0 = b.p[3 * i + a], l0 = b.l[3 * i + a];
      const double f = b.F[3 * i + a], t = b.T[3 * i + a];
      if (!last) {
        p[a] = (p0 + h * f) / (1. + h * xt);
        l[a] = (l0 + h * t) / (1. + h * xr);
      } else {
        p[a] = p0 * (1. - h * xt) + h * f;
        l[a] = l0 * (1. - h * xr) + h * t;
      }
      psq += p[a] * p[a];
      b.p[3 * i + a] = p[a];
      b.l[3 * i + a] = l[a];
    }
    const double im = b.invm[i];
    acc[0] = psq * im;
    acc[1] = rot_kin(b, i, O, l);
    if (last) {
      acc[2] = p[0] * p[0] * im;
      acc[3] = p[0] * p[1] * im;
      acc[4] = p[0] * p[2] * im;
      acc[5] = p[1] * p[1] * im;
      acc[6] = p[1] * p[2] * im;
      acc[7] = p[2] * p[2] * im;
    }
  }
  double tot[9];
  block_sum<9, kPartBlock>(acc, sh, tot);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int c = 0; c < 9; ++c) b.kin2[9 * blk_slot(P, bk) + c] = tot[c];
  }
}

// Opens a run of steps; a short run's noise comes with the launch (a copy of it
// took 2 us of the stream and as much of the host) into `noise`.
__global__ void reset_iter_kernel(Batch b, double* noise, NoiseArgs a) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s < b.nsys) b.st[s].iter = 0;
  if (s < a.n) noise[s] = a.v[s];
}

// The arrays of a small batch's state, to or from the host in one launch: six
// copies of 333 rods' arrays take 12.5 us of the stream, one launch 4.2 (2048
// rods 15 and 6.2, 8192 15 and 11.7; above, the copy engine's 205 GB/s against
// 150 here decide).
__global__ void __launch_bounds__(256) copy_arrays_kernel(ArrayCopies c) {
  const int q = blockIdx.y;
  const double* src = c.src[q];
  double* dst = c.dst[q];
  for (long long i = blockIdx.x * 256 + threadIdx.x; i < c.n[q]; i += (long long)gridDim.x * 256) dst[i] = src[i];
}

// ---------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------
void launch_reset_iter(const Batch& b, double* noise, const NoiseArgs& a, cudaStream_t s) {
  if (b.nsys) reset_iter_kernel<<<cdiv(std::max(b.nsys, a.n), 128), 128, 0, s>>>(b, noise, a);
}
void launch_copy_arrays(const ArrayCopies& c, cudaStream_t s) {
  long long most = 0;
  for (int q = 0; q < c.k; ++q) most = std::max(most, c.n[q]);
  if (most) copy_arrays_kernel<<<dim3((unsigned)std::min<long long>((most + 255) / 256, kSMs), c.k), 256, 0, s>>>(c);
}
void launch_derive(const Batch& b, cudaStream_t s) {
  if (b.nwblk) particle_kernel<kPartDerive><<<b.nwblk, kRowBlock, 0, s>>>(b);
}
void launch_copies(const Batch& b, cudaStream_t s) {
  if (b.nwblk) particle_kernel<kPartCopies><<<b.nwblk, kRowBlock, 0, s>>>(b);
}
void launch_integrate_first(const Batch& b, cudaStream_t s) {
  if (b.nwblk) particle_kernel<kPartStep><<<b.nwblk, kRowBlock, 0, s>>>(b);
}
void launch_xi_mid(const Batch& b, cudaStream_t s) {
  if (b.nsys) xi_mid_kernel<<<b.nsys, 128, 0, s>>>(b);
}
// Batches of at most this many rows of 32 rods run the force assembly's halves
// side by side.  us per step one behind the other and side by side: 4096 rods (128
// rows) 82.5 and 80.0, 24 systems (680) 97.4 and 95.4; 32,768 rods (1024) 2101 and
// 2106, 64 systems (1800) 192 and 194.5, 192 systems 520 and 531, 256 systems (5700)
// 682 and 698: twice the warps hold the registers of the next rows.
constexpr int kFinalizeTwoMax = 1000;
void launch_finalize(const Batch& b, int mode, cudaStream_t s) {
  if (!b.nwblk) return;
  if (b.nwblk <= kFinalizeTwoMax)
    finalize_kernel<false, true><<<b.nwblk, 2 * kRowBlock, 0, s>>>(b, mode);
  else
    finalize_kernel<false, false><<<b.nwblk, kRowBlock, 0, s>>>(b, mode);
}
void launch_finalize_order(const Batch& b, int mode, cudaStream_t s) {
  if (b.nwblk) finalize_kernel<true, true><<<b.nwblk + b.nblk, 2 * kRowBlock, 0, s>>>(b, mode);
}
void launch_order_terms(const Batch& b, cudaStream_t s) {
  if (b.nblk) order_terms_kernel<<<b.nblk, kPartBlock, 0, s>>>(b);
}
void launch_reduce_obs(const Batch& b, int mode, cudaStream_t s) {
  if (!b.nsys) return;
  if (b.obs_host)
    reduce_obs_kernel<true><<<kRedGroups * b.nsys, kRedThreads, 0, s>>>(b, mode);
  else
    reduce_obs_kernel<false><<<kRedGroups * b.nsys, kRedThreads, 0, s>>>(b, mode);
}
void launch_movex(const Batch& b, cudaStream_t s) {
  if (b.nwblk) particle_kernel<kPartMoveX><<<b.nwblk, kRowBlock, 0, s>>>(b);
}
void launch_renorm(const Batch& b, cudaStream_t s) {
  if (b.nblk) renorm_kernel<<<b.nblk, kPartBlock, 0, s>>>(b);
}
void launch_movep(const Batch& b, const double* xi, int last, cudaStream_t s) {
  if (b.nblk) movep_kernel<<<b.nblk, kPartBlock, 0, s>>>(b, xi, last);
}

}  // namespace mdsc

// ---------------------------------------------------------------------
// systems moved between batches (mdsc_transfer_many): the particle state,
// forces, shapes and dipoles of each (destination slot, source slot) pair,
// the dipole owners for the destination's layout, and the mutable state
// with a list rebuild requested.  One launch per kTransferChunk pairs,
// grid.y over the pairs.
// ---------------------------------------------------------------------
namespace mdsc {

constexpr int kTransferChunk = 256;
struct TransferPairs {
  int n;
  int2 p[kTransferChunk];  // (destination system, source system)
};

__global__ void transfer_kernel(Batch dst, Batch src, TransferPairs tp) {
  const int k = blockIdx.y;
  if (k >= tp.n) return;
  const int d = tp.p[k].x, q = tp.p[k].y;
  const SysDev& Pd = dst.sys[d];
  const SysDev& Ps = src.sys[q];
  const int n = Pd.n, ndip = Pd.ndip;
  const long long is = Ps.part_off, id = Pd.part_off, gs = Ps.dip_off, gd = Pd.dip_off;
  const int stride = gridDim.x * blockDim.x;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < 9 * n; t += stride) {
    dst.O[9 * id + t] = src.O[9 * is + t];
    if (t < 3 * n) {
      dst.r[3 * id + t] = src.r[3 * is + t];
      dst.p[3 * id + t] = src.p[3 * is + t];
      dst.l[3 * id + t] = src.l[3 * is + t];
      dst.F[3 * id + t] = src.F[3 * is + t];
      dst.T[3 * id + t] = src.T[3 * is + t];
      dst.inert[3 * id + t] = src.inert[3 * is + t];
      dst.invI[3 * id + t] = src.invI[3 * is + t];
    }
    if (t < n) {
      dst.len[id + t] = src.len[is + t];
      dst.dia[id + t] = src.dia[is + t];
      dst.mass[id + t] = src.mass[is + t];
      dst.invm[id + t] = src.invm[is + t];
    }
    if (t < 3 * ndip) dst.dob[3 * gd + t] = src.dob[3 * gs + t];
    if (t < ndip) {
      dst.dpc[gd + t] = src.dpc[gs + t];
      dst.dmu[gd + t] = src.dmu[gs + t];
      dst.downer[gd + t] = (int)id + t / max(Pd.nd, 1);
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    SysState st = src.st[q];
    st.force_list = 1;
    st.list_ok = 0;
    st.rebuild = 0;
    st.iter = 0;
    dst.st[d] = st;
  }
}

cudaError_t launch_transfer(const Batch& dst, const Batch& src, const std::vector<int2>& pairs, cudaStream_t s) {
  for (size_t k0 = 0; k0 < pairs.size(); k0 += kTransferChunk) {
    TransferPairs tp;
    tp.n = (int)std::min<size_t>(kTransferChunk, pairs.size() - k0);
    for (int k = 0; k < tp.n; ++k) tp.p[k] = pairs[k0 + k];
    // enough threads for the largest system of the batch: 9 values per rod
    const int grid_x = std::min(64, cdiv(9 * std::max(dst.ntot, 1), 256));
    transfer_kernel<<<dim3(grid_x, tp.n), 256, 0, s>>>(dst, src, tp);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace mdsc
