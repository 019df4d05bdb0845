// Reciprocal-space Ewald dipolar sum -- the GPU form of force_dipK
// (v25/functions.cpp:1706-1961) with wave_v's prefactors (:1963-1990).
//
// k-set.  The reference loops n_x, n_y, n_z in [0, K_max-1] with four sign
// patterns (+-k_x, +-k_y, +k_z) and divides by 2 or 4 where components are
// zero (:1725-1744,1845-1850); that visits every distinct +-k pair of the
// cube exactly once with weight 2*Kvec/V.  The host enumerates the same
// distinct vectors once each (one representative per +-k pair) with that
// weight, optionally masked to |n|^2 <= ksq_max.
//
// Per k the structure factor is S(k) = k . U(k) with
// U_c(k) = sum_dipoles mu o_c exp(-i k.r) (the reference's uve); the
// reference removes each particle's own interaction per k with
// self(k) = sum_i |S_i(k)|^2 and uvslf_c(k) = sum_i Re(conj(S_i) U_ic).
//
// Phases.  Dipole positions are 32-bit box fractions u, so for
// k = 2 pi n / L the phase k.r = 2 pi (n . u) / 2^32 and the integer n . u
// wraps modulo 2^32 exactly: the phase is reduced exactly to [-pi, pi) for
// any box size and any k, and only the final sine/cosine is rounded.
//
// Kernels: ksum (partial sums over chunks of kKChunk particles), kstruct
// (chunks -> FP64 sums per k and val S(k), all the gather waits for), kenergy
// (energy and pressure tensor of each k tile, beside the gather), kgather (per
// particle over all k: force and torque).
#include <initializer_list>

#include "mdsc_dev.cuh"
#include "reduce.cuh"

namespace mdsc {

// Batches of at most this many structure-factor blocks (4 per SM) run ksum1s:
// a system of 256 rods 65.7 us per step with ksum1 and 62.4 with ksum1s, 24
// systems of 128 to 2048 rods (330 blocks) 144 and 135; 64 systems (900) 229
// and 226, 256 systems 693 and 696.
constexpr int kKsumScalarMax = 4 * kSMs;

// (int)ph * 2^-31 * pi: the phase, already reduced to [-pi, pi); the
// hardware sine/cosine is accurate to ~4e-7 absolute on that range
__device__ __forceinline__ float phase_rad(uint32_t ph) { return (float)(int32_t)ph * 1.4629180792671596e-09f; }
__device__ __forceinline__ void phase_cs(uint32_t ph, float& c, float& s) { __sincosf(phase_rad(ph), &s, &c); }
__device__ __forceinline__ uint32_t phase_of(uint32_t ux, uint32_t uy, uint32_t uz, int4 n) {
  return (uint32_t)n.x * ux + (uint32_t)n.y * uy + (uint32_t)n.z * uz;
}
__device__ __forceinline__ void phase_exp(uint32_t ux, uint32_t uy, uint32_t uz, int4 n, float& c,
                                          float& s) {
  phase_cs(phase_of(ux, uy, uz, n), c, s);
}
// the gathers walk their k-vectors in order: where a k-vector is the last
// one plus (1, 0, 0) (n.w = 1, marked at layout) the phase advances by u_x,
// the same integer modulo 2^32 as the three products
__device__ __forceinline__ uint32_t phase_next(uint32_t ph, bool have, uint32_t ux, uint32_t uy, uint32_t uz,
                                               int4 n) {
  return (have && n.w) ? ph + ux : phase_of(ux, uy, uz, n);
}

// The moment tensor of one particle chunk, sum of m m^T (one dipole per
// particle), for the self terms of kenergy, by a warp of its own block (work
// items of k tile -1).  FP64: the products exact, the sums to 53 bits.  An FP64
// instruction holds a warp 64 cycles, ~5000 cycles for a chunk, beside the waves
// of the other items, which take longer: ksum1s of 256 rods 7.8 us a launch, 7.6
// with float-float sums (48 bits); the step 31.4 us either way, of 4096 rods 75.5
// and 77.3.
__device__ __forceinline__ void chunk_tensor(const Batch& b, const SysDev& P, int chunk) {
  if (threadIdx.x >= 32) return;
  const int N = b.ndtot, p0 = chunk * kKChunk, np = min(kKChunk, P.n - p0);
  double g[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll 4
  for (int q = threadIdx.x; q < np; q += 32) {
    const int d = P.dip_off + p0 + q;
    const double x = soft_f2d(b.dm[d]), y = soft_f2d(b.dm[N + d]), z = soft_f2d(b.dm[2 * N + d]);
    const double u[6] = {x, x, x, y, y, z}, v[6] = {x, y, z, y, z, z};
#pragma unroll
    for (int c = 0; c < 6; ++c) g[c] = fma(u[c], v[c], g[c]);
  }
#pragma unroll
  for (int c = 0; c < 6; ++c) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) g[c] += __shfl_xor_sync(0xffffffffu, g[c], off);
    if (threadIdx.x == c) b.kG[((long long)P.gch_off + chunk) * 6 + c] = g[c];
  }
}

// Structure-factor partials, component-major so that a warp's 32 k-vectors
// are consecutive: partial c of k-vector kl in a chunk, nv values per k.
__device__ __forceinline__ float* ksum_part(const Batch& b, const SysDev& P, int chunk, int nv) {
  return b.kpart + ((long long)P.kchunk_off * 10 + (long long)chunk * P.nk * nv);
}

// Several dipoles per particle: one block per (system, particle chunk, k
// tile) of the work list kwork, one k per thread.  The particle's own terms
// per k (S_i over its dipoles) need the per-k work here.
template <int ND>
__global__ void __launch_bounds__(kKBlock) ksum_kernel(Batch b, const int4* __restrict__ kwork) {
  __shared__ uint32_t sx[kKChunk * ND], sy[kKChunk * ND], sz[kKChunk * ND];
  __shared__ float smx[kKChunk * ND], smy[kKChunk * ND], smz[kKChunk * ND];
  const int4 w = kwork[blockIdx.x];
  const SysDev& P = b.sys[w.x];
  if (P.nd <= 1 || at_limit(b, w.x)) return;  // single-dipole systems: ksum1_kernel, ksum1s_kernel
  const int chunk = w.y;
  const int kl = w.z * kKBlock + threadIdx.x;
  const int ND_all = b.ndtot;
  const int p0 = chunk * kKChunk;
  const int np = min(kKChunk, P.n - p0);
  const int nd = P.nd;
  for (int q = threadIdx.x; q < np * nd; q += kKBlock) {
    const int g = P.dip_off + p0 * nd + q;
    sx[q] = b.dfx[g];
    sy[q] = b.dfx[ND_all + g];
    sz[q] = b.dfx[2 * ND_all + g];
    smx[q] = b.dm[g];
    smy[q] = b.dm[ND_all + g];
    smz[q] = b.dm[2 * ND_all + g];
  }
  __syncthreads();
  if (kl >= P.nk) return;
  const int4 n = b.kn[P.k_off + kl];
  const float4 kv = b.kv[P.k_off + kl];
  float acc[10];
#pragma unroll
  for (int c = 0; c < 10; ++c) acc[c] = 0.f;
  for (int p = 0; p < np; ++p) {
    float Sr = 0.f, Si = 0.f, Ur[3] = {0.f, 0.f, 0.f}, Ui[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int d = 0; d < ND; ++d) {
      if (d < nd) {
        const int q = p * nd + d;
        float c, s;
        phase_exp(sx[q], sy[q], sz[q], n, c, s);
        const float mx = smx[q], my = smy[q], mz = smz[q];
        const float a = mx * kv.x + my * kv.y + mz * kv.z;
        Sr += a * c;
        Si -= a * s;
        Ur[0] += mx * c; Ui[0] -= mx * s;
        Ur[1] += my * c; Ui[1] -= my * s;
        Ur[2] += mz * c; Ui[2] -= mz * s;
      }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      acc[2 * c] += Ur[c];
      acc[2 * c + 1] += Ui[c];
      acc[7 + c] += Sr * Ur[c] + Si * Ui[c];
    }
    acc[6] += Sr * Sr + Si * Si;
  }
  float* out = ksum_part(b, P, chunk, 10) + kl;
#pragma unroll
  for (int c = 0; c < 10; ++c) out[(long long)c * P.nk] = acc[c];
}

// The same sums for batches that leave SMs idle: a block takes 32 k-vectors of
// a work item, its ten warps the particles in turn -- each forms one particle's
// sums over its dipoles and leaves them in shared memory -- and then each warp
// adds one of the ten components over those particles, in particle order, so
// every sum keeps its order.  One thread's walk over the chunk was the time:
// 1500 rods of two dipoles (24 work items) 39 us a launch beside the tiles, 13
// this way.
constexpr int kSumWarps = 10;
constexpr int kSumTerms = 8;  // U (3 real and imaginary pairs), S
template <int ND>
__global__ void __launch_bounds__(32 * kSumWarps) ksum_split_kernel(Batch b, const int4* __restrict__ kwork) {
  __shared__ uint32_t sx[kKChunk * ND], sy[kKChunk * ND], sz[kKChunk * ND];
  __shared__ float smx[kKChunk * ND], smy[kKChunk * ND], smz[kKChunk * ND];
  __shared__ float term[2][kSumWarps][kSumTerms][32];
  const int4 wk = kwork[blockIdx.x / (kKBlock / 32)];
  const SysDev& P = b.sys[wk.x];
  if (P.nd <= 1 || at_limit(b, wk.x)) return;  // single-dipole systems: ksum1_kernel, ksum1s_kernel
  const int k0 = wk.z * kKBlock + (blockIdx.x % (kKBlock / 32)) * 32;
  if (k0 >= P.nk) return;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kl = min(k0 + lane, P.nk - 1);
  const int N = b.ndtot, nd = P.nd;
  const int p0 = wk.y * kKChunk, np = min(kKChunk, P.n - p0);
  for (int q = threadIdx.x; q < np * nd; q += 32 * kSumWarps) {
    const int g = P.dip_off + p0 * nd + q;
    sx[q] = b.dfx[g];
    sy[q] = b.dfx[N + g];
    sz[q] = b.dfx[2 * N + g];
    smx[q] = b.dm[g];
    smy[q] = b.dm[N + g];
    smz[q] = b.dm[2 * N + g];
  }
  const int4 n = b.kn[P.k_off + kl];
  const float4 kv = b.kv[P.k_off + kl];
  float acc = 0.f;
  __syncthreads();
  for (int r = 0, buf = 0; r < np; r += kSumWarps, buf ^= 1) {
    if (r + w < np) {
      float S[2] = {0.f, 0.f}, U[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int d = 0; d < ND; ++d) {
        if (d < nd) {
          const int q = (r + w) * nd + d;
          float c, s;
          phase_exp(sx[q], sy[q], sz[q], n, c, s);
          const float m[3] = {smx[q], smy[q], smz[q]};
          const float a = m[0] * kv.x + m[1] * kv.y + m[2] * kv.z;
          S[0] += a * c;
          S[1] -= a * s;
#pragma unroll
          for (int e = 0; e < 3; ++e) {
            U[2 * e] += m[e] * c;
            U[2 * e + 1] -= m[e] * s;
          }
        }
      }
#pragma unroll
      for (int e = 0; e < 6; ++e) term[buf][w][e][lane] = U[e];
      term[buf][w][6][lane] = S[0];
      term[buf][w][7][lane] = S[1];
    }
    // one barrier a round: a buffer is written again only after the next one,
    // which every warp reaches with its reads of this one done
    __syncthreads();
    const int cnt = min(kSumWarps, np - r);
    const float(*t)[kSumTerms][32] = term[buf];
    if (w < 6) {
#pragma unroll
      for (int q = 0; q < kSumWarps; ++q)
        if (q < cnt) acc = __fadd_rn(acc, t[q][w][lane]);
    } else {
      // w = 6: |S_i|^2; 7 to 9: Re(conj(S_i) U_i)
      const int ur = w == 6 ? 6 : 2 * (w - 7), ui = ur + 1;
#pragma unroll
      for (int q = 0; q < kSumWarps; ++q)
        if (q < cnt) acc = __fadd_rn(acc, __fmaf_rn(t[q][6][lane], t[q][ur][lane], __fmul_rn(t[q][7][lane], t[q][ui][lane])));
    }
  }
  if (k0 + lane < P.nk) ksum_part(b, P, wk.y, 10)[(long long)w * P.nk + kl] = acc;
}

// Single-dipole systems.  The particle's own terms need no per-k work:
// |S_i(k)|^2 = (m_i.k)^2 and Re(conj(S_i) U_ic) = (m_i.k) m_ic, so
// self(k) = k^T G k and uvslf(k) = G k with G = sum_i m_i m_i^T
// (chunk_tensor).
//
// Two forms, the same IEEE operations in the same order per (particle, k)
// and so the same bits.  ksum1: two k-vectors per thread (kl and kl + 64 of
// the block's k tile) in the halves of float2 values, so every particle
// read from shared memory serves two k's and the six multiply-adds of U(k)
// issue once for both -- for batches that fill the GPU.  ksum1s: one k per
// thread, the cosine sums and the sine sums on different warps -- for the
// others, where one warp's walk over the chunk is the time (the special-
// function unit takes a warp 8 cycles per sine or cosine): 256 rods 10.7 us a
// launch with both sums on one warp, 7.9 this way.
constexpr int kAhead = 8;  // waves formed ahead of their sums
struct KChunk {
  uint4 u[kKChunk];   // fixed-point x, y, z
  float4 m[kKChunk];  // moment
};

template <int NT>
__device__ __forceinline__ int stage_chunk(const Batch& b, const SysDev& P, int4 w, KChunk& c) {
  const int N = b.ndtot, p0 = w.y * kKChunk;
  const int np = min(kKChunk, P.n - p0);
  for (int q = threadIdx.x; q < np; q += NT) {
    const int g = P.dip_off + p0 + q;
    c.u[q] = make_uint4(b.dfx[g], b.dfx[N + g], b.dfx[2 * N + g], 0u);
    c.m[q] = make_float4(b.dm[g], b.dm[N + g], b.dm[2 * N + g], 0.f);
  }
  __syncthreads();
  return np;
}

__global__ void __launch_bounds__(kKBlock / 2) ksum1_kernel(Batch b, const int4* __restrict__ kwork) {
  __shared__ KChunk ck;
  const int4 w = kwork[blockIdx.x];
  const SysDev& P = b.sys[w.x];
  if (P.nd != 1 || at_limit(b, w.x)) return;  // other systems: ksum_kernel<ND>
  if (w.z < 0) {
    chunk_tensor(b, P, w.y);
    return;
  }
  const int np = stage_chunk<kKBlock / 2>(b, P, w, ck);
  const int kl0 = w.z * kKBlock + threadIdx.x, kl1 = kl0 + kKBlock / 2;
  const bool v0 = kl0 < P.nk, v1 = kl1 < P.nk;
  if (!v0) return;
  const int4 n0 = b.kn[P.k_off + kl0];
  const int4 n1 = v1 ? b.kn[P.k_off + kl1] : n0;
  float2 acc[6];
#pragma unroll
  for (int c = 0; c < 6; ++c) acc[c] = make_float2(0.f, 0.f);
#pragma unroll 2
  for (int p = 0; p < np; ++p) {
    float c0, s0, c1, s1;
    const uint4 u = ck.u[p];
    phase_exp(u.x, u.y, u.z, n0, c0, s0);
    phase_exp(u.x, u.y, u.z, n1, c1, s1);
    const float2 c = make_float2(c0, c1), sn = make_float2(-s0, -s1);
    // E = exp(-i k.r) = (c, -s); U_c += m_c E
    const float4 m = ck.m[p];
    acc[0] = __ffma2_rn(make_float2(m.x, m.x), c, acc[0]);
    acc[1] = __ffma2_rn(make_float2(m.x, m.x), sn, acc[1]);
    acc[2] = __ffma2_rn(make_float2(m.y, m.y), c, acc[2]);
    acc[3] = __ffma2_rn(make_float2(m.y, m.y), sn, acc[3]);
    acc[4] = __ffma2_rn(make_float2(m.z, m.z), c, acc[4]);
    acc[5] = __ffma2_rn(make_float2(m.z, m.z), sn, acc[5]);
  }
  float* out = ksum_part(b, P, w.y, 6);
#pragma unroll
  for (int c = 0; c < 6; ++c) {
    out[(long long)c * P.nk + kl0] = acc[c].x;
    if (v1) out[(long long)c * P.nk + kl1] = acc[c].y;
  }
}

__global__ void __launch_bounds__(2 * kKBlock) ksum1s_kernel(Batch b, const int4* __restrict__ kwork) {
  __shared__ KChunk ck;
  const int4 w = kwork[blockIdx.x];
  const SysDev& P = b.sys[w.x];
  if (P.nd != 1 || at_limit(b, w.x)) return;  // other systems: ksum_kernel<ND>
  if (w.z < 0) {
    chunk_tensor(b, P, w.y);
    return;
  }
  const int np = stage_chunk<2 * kKBlock>(b, P, w, ck);
  const bool sine = threadIdx.x >= kKBlock;  // the same for a warp
  const int kl = w.z * kKBlock + (threadIdx.x & (kKBlock - 1));
  if (kl >= P.nk) return;
  const int4 n = b.kn[P.k_off + kl];
  float acc[3] = {0.f, 0.f, 0.f};
  auto walk = [&](auto&& wave) {
    int p = 0;
#pragma unroll 1
    for (; p + kAhead <= np; p += kAhead) {
      float v[kAhead];
#pragma unroll
      for (int q = 0; q < kAhead; ++q) v[q] = wave(p + q);
#pragma unroll
      for (int q = 0; q < kAhead; ++q) {
        const float4 m = ck.m[p + q];
        acc[0] = __fmaf_rn(m.x, v[q], acc[0]);
        acc[1] = __fmaf_rn(m.y, v[q], acc[1]);
        acc[2] = __fmaf_rn(m.z, v[q], acc[2]);
      }
    }
#pragma unroll 1
    for (; p < np; ++p) {
      const float v = wave(p);
      const float4 m = ck.m[p];
      acc[0] = __fmaf_rn(m.x, v, acc[0]);
      acc[1] = __fmaf_rn(m.y, v, acc[1]);
      acc[2] = __fmaf_rn(m.z, v, acc[2]);
    }
  };
  // E = exp(-i k.r) = (c, -s); U_c += m_c E
  if (sine)
    walk([&](int p) { return -__sinf(phase_rad(phase_of(ck.u[p].x, ck.u[p].y, ck.u[p].z, n))); });
  else
    walk([&](int p) { return __cosf(phase_rad(phase_of(ck.u[p].x, ck.u[p].y, ck.u[p].z, n))); });
  float* out = ksum_part(b, P, w.y, 6) + (sine ? P.nk : 0) + kl;
#pragma unroll
  for (int c = 0; c < 3; ++c) out[(long long)2 * c * P.nk] = acc[c];
}

template <int ND>
static void launch_ksum(const Batch& b, const int4* kwork, int nkwork, cudaStream_t s) {
  // every single-dipole system through a single-dipole kernel, in any
  // batch, so that it gives the same bits alone and beside multi-dipole ones
  if (!b.ones)
    ;
  else if (nkwork <= kKsumScalarMax)
    ksum1s_kernel<<<nkwork, 2 * kKBlock, 0, s>>>(b, kwork);
  else
    ksum1_kernel<<<nkwork, kKBlock / 2, 0, s>>>(b, kwork);
  if constexpr (ND > 1) {
    if (b.sum_split)
      ksum_split_kernel<ND><<<nkwork * (kKBlock / 32), 32 * kSumWarps, 0, s>>>(b, kwork);
    else
      ksum_kernel<ND><<<nkwork, kKBlock, 0, s>>>(b, kwork);
  }
}

// The totals of NC components of a system's k-vector, c0, c0 + 1, ..., over the
// chunks, in chunk order (float-float; W loads of each in flight): the gathers'
// input keeps one order of its sums.
template <int W, int NC>
__device__ __forceinline__ void ksum_totals(const Batch& b, const SysDev& P, int kl, int c0, int nv, double (&s)[NC]) {
  const float* in = ksum_part(b, P, 0, nv) + (long long)c0 * P.nk + kl;
  FF sf[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) sf[c] = ff_of(0.f);
  for (int ch = 0; ch < P.nkchunk; ch += W) {
    float x[W][NC];
#pragma unroll
    for (int q = 0; q < W; ++q)
#pragma unroll
      for (int c = 0; c < NC; ++c) x[q][c] = ch + q < P.nkchunk ? in[((long long)(ch + q) * nv + c) * P.nk] : 0.f;
#pragma unroll
    for (int q = 0; q < W; ++q)
      if (ch + q < P.nkchunk) {
#pragma unroll
        for (int c = 0; c < NC; ++c) sf[c] = ff_add(sf[c], ff_of(x[q][c]));
      }
  }
#pragma unroll
  for (int c = 0; c < NC; ++c) s[c] = soft_f2d(sf[c].hi) + soft_f2d(sf[c].lo);
}

// val S(k) from the six totals (the roundings written out: two kernels form it)
__device__ __forceinline__ float2 val_S(const Batch& b, long long k, const double (&s)[6]) {
  const double kx = b.kvec[3 * k], ky = b.kvec[3 * k + 1], kz = b.kvec[3 * k + 2];
  const double val = b.kval[k];
  const double Sr = __fma_rn(kz, s[4], __fma_rn(kx, s[0], __dmul_rn(ky, s[2])));
  const double Si = __fma_rn(kz, s[5], __fma_rn(kx, s[1], __dmul_rn(ky, s[3])));
  return make_float2(soft_d2f_rn(val * Sr), soft_d2f_rn(val * Si));
}

// Chunk sums per k and val S(k): all the gather needs, nothing more.  A block
// takes 32 consecutive k-vectors of the batch; warp w totals components w, w +
// kStructWarps, ..., and warp 0 forms val S(k).  Five blocks an SM: with 128
// registers a thread its blocks waited for the tiles of 4096 rods to leave, 15
// us of the 82 of a step.
constexpr int kStructWarps = 6;
__global__ void __launch_bounds__(32 * kStructWarps, 5) kstruct_kernel(Batch b, const int2* __restrict__ kowner) {
  __shared__ double sh[6][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int k = blockIdx.x * 32 + lane;
  bool on = k < b.nktot;
  const int2 ow = on ? kowner[k] : make_int2(0, 0);  // (system, k index within the system)
  on = on && !at_limit(b, ow.x);
  const SysDev& P = b.sys[ow.x];
  const int nv = P.nd == 1 ? 6 : 10;
  if (on) {
    for (int c = w; c < nv; c += kStructWarps) {
      double s[1];
      ksum_totals<8>(b, P, ow.y, c, nv, s);
      b.ksum[(long long)k * 10 + c] = s[0];
      if (c < 6) sh[c][lane] = s[0];
    }
  }
  __syncthreads();
  if (w > 0 || !on) return;
  double s[6];
#pragma unroll
  for (int c = 0; c < 6; ++c) s[c] = sh[c][lane];
  b.kS[k] = val_S(b, k, s);
}

// Energy and pressure tensor of one k tile (v25/functions.cpp:1839-1952),
// the tile's k-vectors summed in float-float into one row of kE.  Off the
// path the forces wait for: it runs beside the gather.
__global__ void __launch_bounds__(kKBlock) kenergy_kernel(Batch b) {
  __shared__ double sh[10 * kKBlock / 32];
  __shared__ double sG[6];
  const int2 kt = b.ktile[blockIdx.x];  // (system, k tile)
  if (at_limit(b, kt.x)) return;
  const SysDev& P = b.sys[kt.x];
  const bool one = P.nd == 1;
  if (one) {  // the moment tensor over the system's chunks, in chunk order
    if (threadIdx.x < 6) {
      const double* in = b.kG + (long long)P.gch_off * 6 + threadIdx.x;
      double g = 0.0;
#pragma unroll 8
      for (int ch = 0; ch < P.nkchunk; ++ch) g += in[6 * ch];
      sG[threadIdx.x] = g;
    }
    __syncthreads();
  }
  FF e[10];
#pragma unroll
  for (int c = 0; c < 10; ++c) e[c] = ff_of(0.f);
  const int kl = kt.y * kKBlock + threadIdx.x;
  if (kl < P.nk) {
    const long long k = P.k_off + kl;
    const double* ks = b.ksum + k * 10;
    const double kk[3] = {b.kvec[3 * k], b.kvec[3 * k + 1], b.kvec[3 * k + 2]};
    double s[6], slf, uv[3];
#pragma unroll
    for (int c = 0; c < 6; ++c) s[c] = ks[c];
    if (one) {
      uv[0] = sG[0] * kk[0] + sG[1] * kk[1] + sG[2] * kk[2];
      uv[1] = sG[1] * kk[0] + sG[3] * kk[1] + sG[4] * kk[2];
      uv[2] = sG[2] * kk[0] + sG[4] * kk[1] + sG[5] * kk[2];
      slf = kk[0] * uv[0] + kk[1] * uv[1] + kk[2] * uv[2];
    } else {
      slf = ks[6];
#pragma unroll
      for (int c = 0; c < 3; ++c) uv[c] = ks[7 + c];
    }
    const double Sr = kk[0] * s[0] + kk[1] * s[2] + kk[2] * s[4];
    const double Si = kk[0] * s[1] + kk[1] * s[3] + kk[2] * s[5];
    const double val = b.kval[k];
    // val/2 ((delta_jq - pval k_j k_q)(|S|^2 - self) + 2 re_j k_q) with
    // re_j = Re(conj(S) U_j) - uvslf_j
    const double en = val * 0.5 * (Sr * Sr + Si * Si - slf);
    const double pen = b.kpre[k] * en;
    e[0] = ff_from(en);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const double re = Sr * s[2 * j] + Si * s[2 * j + 1] - uv[j];
      const double row = val * re - pen * kk[j];
#pragma unroll
      for (int q = 0; q < 3; ++q) e[1 + 3 * j + q] = ff_from(j == q ? row * kk[q] + en : row * kk[q]);
    }
  }
  double out[10];
  block_sum<10, kKBlock>(e, sh, out);
  if (threadIdx.x == 0) {
    double* dst = b.kE + (long long)blockIdx.x * 10;
#pragma unroll
    for (int c = 0; c < 10; ++c) dst[c] = out[c];
  }
}

// k-space results of one dipole from its Kahan sums (sum = fo - fc): the
// force as float-float, and the torque m x G (G the second triple) with the
// FP32 moment -- as accurate as the FP32 sums it is built from
__device__ __forceinline__ void store_tk(const Batch& b, int g, const float* go, const float* gc, float mx, float my,
                                         float mz) {
  const FF G[3] = {{go[0], -gc[0]}, {go[1], -gc[1]}, {go[2], -gc[2]}};
  const float m[3] = {mx, my, mz};
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const FF t = ff_cross(m[(c + 1) % 3], G[(c + 2) % 3], m[(c + 2) % 3], G[(c + 1) % 3]);
    b.Tk[3 * g + c] = make_float2(t.hi, t.lo);
  }
}
__device__ __forceinline__ void store_kout(const Batch& b, int g, const float* fo, const float* fc,
                                           float mx, float my, float mz) {
#pragma unroll
  for (int c = 0; c < 3; ++c) b.Fk[3 * g + c] = make_float2(fo[c], -fc[c]);
  store_tk(b, g, fo + 3, fc + 3, mx, my, mz);
}

// The gathers: per particle over all k of its system, force and torque
// (:1853-1925).  The sums of a k tile are plain FP32, the tiles are added in
// order (Kahan), and a system of SysDev::kgs > 1 parts adds its parts'
// sums the same way -- the order of every addition is the system's own.
//
// The work of one particle block goes to one block (it walks every tile and
// leaves force and torque, store_kout) or to one block per tile (SysDev::kgt >
// 1): each leaves its tile's sums in the partial set of (particle block, tile)
// and the force assembly adds the tiles, in the same order (ktile_sums).  The
// block that finished last added them before: with the fences, the count and
// one thread per rod for all six sums, 14.5 us a launch for 256 rods in the
// step and 23 for 4096 with 9 tiles; one thread per rod and waves ahead as well
// as this, 6.3 and 9.5.
// the k-vectors of a work item: tile wk.y, or all of them (wk.y < 0)
__device__ __forceinline__ void ktile_range(const SysDev& P, int2 wk, int& kb, int& ke) {
  kb = wk.y < 0 ? 0 : wk.y * kKBlock;
  ke = wk.y < 0 ? P.nk : min(P.nk, kb + kKBlock);
}

struct KTile {
  int4 n[kKBlock];
  float4 v[kKBlock];  // kx, ky, kz, val
  float2 S[kKBlock];  // val * S(k)
};
// TOTALS (Batch::stage_k): val S(k) formed here; a template because its registers
// (kgather1 80 -> 128) cost the large batches 8 us of the gather's 96
template <int NT, bool TOTALS>
__device__ __forceinline__ int stage_ktile(const Batch& b, const SysDev& P, int k0, int ke, KTile& kt) {
  const int nk = min(kKBlock, ke - k0);
  __syncthreads();
  for (int q = threadIdx.x; q < nk; q += NT) {
    kt.n[q] = b.kn[P.k_off + k0 + q];
    kt.v[q] = b.kv[P.k_off + k0 + q];
    if constexpr (TOTALS) {
      double s[6];
      ksum_totals<4>(b, P, k0 + q, 0, P.nd == 1 ? 6 : 10, s);
      kt.S[q] = val_S(b, P.k_off + k0 + q, s);
    } else {
      kt.S[q] = b.kS[P.k_off + k0 + q];
    }
  }
  __syncthreads();
  return nk;
}

// several dipoles per particle, one particle per thread
template <int ND, bool TOTALS>
__global__ void __launch_bounds__(kPartBlock) kgather_kernel(Batch b) {
  __shared__ KTile kt;
  const int2 wk = b.kgwork[blockIdx.x];  // (particle block, tile)
  const int2 bk = b.blk[wk.x];
  const SysDev& P = b.sys[bk.x];
  if (P.nd <= 1 || at_limit(b, bk.x)) return;  // single-dipole systems: kgather1 / kgather1s
  const int i = bk.y + threadIdx.x;  // batch particle index
  const bool ok = i < P.part_off + P.n;
  const int nd = P.nd;
  const int ND_all = b.ndtot;
  uint32_t ux[ND], uy[ND], uz[ND];
  float mx[ND], my[ND], mz[ND];
  const int gd0 = P.dip_off + (i - P.part_off) * nd;
#pragma unroll
  for (int d = 0; d < ND; ++d) {
    const bool v = ok && d < nd;
    const int g = v ? gd0 + d : 0;
    ux[d] = b.dfx[g];
    uy[d] = b.dfx[ND_all + g];
    uz[d] = b.dfx[2 * ND_all + g];
    mx[d] = v ? b.dm[g] : 0.f;
    my[d] = v ? b.dm[ND_all + g] : 0.f;
    mz[d] = v ? b.dm[2 * ND_all + g] : 0.f;
  }
  float fo[ND][6], fc[ND][6], ft[ND][6];
#pragma unroll
  for (int d = 0; d < ND; ++d)
#pragma unroll
    for (int c = 0; c < 6; ++c) fo[d][c] = fc[d][c] = ft[d][c] = 0.f;

  uint32_t ph[ND];
#pragma unroll
  for (int d = 0; d < ND; ++d) ph[d] = 0u;
  bool have = false;
  int kb, ke;
  ktile_range(P, wk, kb, ke);
  for (int k0 = kb; k0 < ke; k0 += kKBlock) {
    const int nk = stage_ktile<kPartBlock, TOTALS>(b, P, k0, ke, kt);
#pragma unroll
    for (int d = 0; d < ND; ++d)
#pragma unroll
      for (int c = 0; c < 6; ++c) ft[d][c] = 0.f;
    for (int q = 0; q < nk; ++q) {
      const int4 n = kt.n[q];
      const float4 kv = kt.v[q];
      const float2 vS = kt.S[q];
      float Ec[ND], Es[ND], a[ND];
      float Sr = 0.f, Si = 0.f;
#pragma unroll
      for (int d = 0; d < ND; ++d) {
        if (d < nd) {
          ph[d] = phase_next(ph[d], have, ux[d], uy[d], uz[d], n);
          phase_cs(ph[d], Ec[d], Es[d]);
          a[d] = mx[d] * kv.x + my[d] * kv.y + mz[d] * kv.z;
          Sr += a[d] * Ec[d];
          Si -= a[d] * Es[d];
        }
      }
      have = true;
      // D = conj(val S) - val conj(S_i)
      const float Dr = vS.x - kv.w * Sr;
      const float Di = -vS.y + kv.w * Si;
#pragma unroll
      for (int d = 0; d < ND; ++d) {
        if (d < nd) {
          // Z = E D with E = (c, -s)
          const float Zr = Ec[d] * Dr + Es[d] * Di;
          const float Zi = Ec[d] * Di - Es[d] * Dr;
          const float fF = -a[d] * Zi;
          const float fT = -Zr;
          ft[d][0] += fF * kv.x;
          ft[d][1] += fF * kv.y;
          ft[d][2] += fF * kv.z;
          ft[d][3] += fT * kv.x;
          ft[d][4] += fT * kv.y;
          ft[d][5] += fT * kv.z;
        }
      }
    }
#pragma unroll
    for (int d = 0; d < ND; ++d)
#pragma unroll
      for (int c = 0; c < 6; ++c) kahan(fo[d][c], fc[d][c], ft[d][c]);
  }
  if (!ok) return;
  if (wk.y >= 0) {  // one tile: leave its sums
    float* mine = ktile_set(b, P, i, wk.y);
#pragma unroll
    for (int d = 0; d < ND; ++d)
      if (d < nd) {
#pragma unroll
        for (int c = 0; c < 6; ++c) mine[d * kSet + c * kPartBlock] = ft[d][c];
      }
    return;
  }
#pragma unroll
  for (int d = 0; d < ND; ++d)
    if (d < nd) store_kout(b, gd0 + d, fo[d], fc[d], mx[d], my[d], mz[d]);
}

// The same for batches that leave SMs idle: a block takes 32 particles of the
// work item, a lane each; its four warps form the terms of the k-vectors in
// turn (force and torque factor of each dipole) and leave them in shared
// memory, and each then adds its dipoles' force or torque sums over those
// k-vectors, in order: a thread's walk over a k tile was the time (700 rods of
// two dipoles 53.8 us per step, 49.7 this way).
constexpr int kGatherWarps = 4, kGatherTurn = 4;  // k-vectors a warp forms per round
template <int ND, bool TOTALS>
__global__ void __launch_bounds__(32 * kGatherWarps) kgather_split_kernel(Batch b) {
  constexpr int kRound = kGatherWarps * kGatherTurn;
  constexpr int kMine = (2 * ND + kGatherWarps - 1) / kGatherWarps;  // sums (dipole; force or torque) of a warp
  __shared__ KTile kt;
  __shared__ float term[2][kRound][2 * ND][32];
  const int2 wk = b.kgwork[blockIdx.x / (kPartBlock / 32)];  // (particle block, tile)
  const int2 bk = b.blk[wk.x];
  const SysDev& P = b.sys[bk.x];
  if (P.nd <= 1 || at_limit(b, bk.x)) return;  // single-dipole systems: kgather1 / kgather1s
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r0 = bk.y + (blockIdx.x % (kPartBlock / 32)) * 32, end = P.part_off + P.n;
  if (r0 >= end) return;
  const bool ok = r0 + lane < end;
  const int i = ok ? r0 + lane : r0;
  const int nd = P.nd, N = b.ndtot;
  const int g0 = P.dip_off + (i - P.part_off) * nd;
  uint32_t ux[ND], uy[ND], uz[ND];
  float mx[ND], my[ND], mz[ND];
#pragma unroll
  for (int d = 0; d < ND; ++d) {
    const int g = d < nd ? g0 + d : g0;
    ux[d] = b.dfx[g];
    uy[d] = b.dfx[N + g];
    uz[d] = b.dfx[2 * N + g];
    mx[d] = b.dm[g];
    my[d] = b.dm[N + g];
    mz[d] = b.dm[2 * N + g];
  }
  float fo[kMine][3], fc[kMine][3], ft[kMine][3];
#pragma unroll
  for (int m = 0; m < kMine; ++m)
#pragma unroll
    for (int c = 0; c < 3; ++c) fo[m][c] = fc[m][c] = 0.f;
  int kb, ke, buf = 0;
  ktile_range(P, wk, kb, ke);
  for (int k0 = kb; k0 < ke; k0 += kKBlock) {
    const int nk = stage_ktile<32 * kGatherWarps, TOTALS>(b, P, k0, ke, kt);
#pragma unroll
    for (int m = 0; m < kMine; ++m)
#pragma unroll
      for (int c = 0; c < 3; ++c) ft[m][c] = 0.f;
    for (int q0 = 0; q0 < nk; q0 += kRound, buf ^= 1) {
#pragma unroll
      for (int u = 0; u < kGatherTurn; ++u) {
        const int q = q0 + u * kGatherWarps + w;
        if (q < nk) {
          const int4 n = kt.n[q];
          const float4 kv = kt.v[q];
          const float2 vS = kt.S[q];
          float Ec[ND], Es[ND], a[ND];
          float Sr = 0.f, Si = 0.f;
#pragma unroll
          for (int d = 0; d < ND; ++d) {
            if (d < nd) {
              phase_exp(ux[d], uy[d], uz[d], n, Ec[d], Es[d]);
              a[d] = mx[d] * kv.x + my[d] * kv.y + mz[d] * kv.z;
              Sr += a[d] * Ec[d];
              Si -= a[d] * Es[d];
            }
          }
          // D = conj(val S) - val conj(S_i)
          const float Dr = vS.x - kv.w * Sr;
          const float Di = -vS.y + kv.w * Si;
#pragma unroll
          for (int d = 0; d < ND; ++d) {
            if (d < nd) {
              // Z = E D with E = (c, -s)
              const float Zr = Ec[d] * Dr + Es[d] * Di;
              const float Zi = Ec[d] * Di - Es[d] * Dr;
              term[buf][q - q0][2 * d][lane] = -a[d] * Zi;
              term[buf][q - q0][2 * d + 1][lane] = -Zr;
            }
          }
        }
      }
      // one barrier a round, as in ksum_split_kernel
      __syncthreads();
      const int cnt = min(kRound, nk - q0);
#pragma unroll
      for (int m = 0; m < kMine; ++m) {
        const int j = w + m * kGatherWarps;
        if (j < 2 * nd) {
#pragma unroll
          for (int q = 0; q < kRound; ++q)
            if (q < cnt) {
              const float4 kv = kt.v[q0 + q];
              const float f = term[buf][q][j][lane];
              ft[m][0] = __fmaf_rn(f, kv.x, ft[m][0]);
              ft[m][1] = __fmaf_rn(f, kv.y, ft[m][1]);
              ft[m][2] = __fmaf_rn(f, kv.z, ft[m][2]);
            }
        }
      }
    }
#pragma unroll
    for (int m = 0; m < kMine; ++m)
#pragma unroll
      for (int c = 0; c < 3; ++c) kahan(fo[m][c], fc[m][c], ft[m][c]);
  }
  if (!ok) return;
#pragma unroll
  for (int m = 0; m < kMine; ++m) {
    const int j = w + m * kGatherWarps, d = j >> 1, g = g0 + d;
    if (j >= 2 * nd) continue;
    if (wk.y >= 0) {  // one tile: leave its sums
      float* mine = ktile_set(b, P, i, wk.y) + d * kSet + (j & 1) * 3 * kPartBlock;
#pragma unroll
      for (int c = 0; c < 3; ++c) mine[c * kPartBlock] = ft[m][c];
    } else if (j & 1) {
      store_tk(b, g, fo[m], fc[m], b.dm[g], b.dm[N + g], b.dm[2 * N + g]);
    } else {
#pragma unroll
      for (int c = 0; c < 3; ++c) b.Fk[3 * g + c] = make_float2(fo[m][c], -fc[m][c]);
    }
  }
}

// Single-dipole systems: a thread takes two particles, i and i + 64 of its
// block, and runs them side by side in the halves of float2 values with
// the paired FP32 instructions, so every k read from shared memory serves
// two particles and the force/torque arithmetic issues once for both.
// With D = conj(val S) - val conj(S_i) (S_i = a e^{-ik.r}, a = m.k) the
// k-term is Z = e^{-ik.r} D; fF = -a Im Z, fT = -Re Z, written below with
// Dr = Re(val S) - val a cos, Dn = Im(val S) + val a sin.
namespace {
__device__ __forceinline__ float2 pk(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ float2 bc(float a) { return make_float2(a, a); }
}  // namespace

__global__ void __launch_bounds__(kPartBlock / 2) kgather1_kernel(Batch b) {
  __shared__ KTile kt;
  const int2 wk = b.kgwork[blockIdx.x];  // (particle block, tile)
  const int2 bk = b.blk[wk.x];
  const SysDev& P = b.sys[bk.x];
  if (P.nd != 1 || at_limit(b, bk.x)) return;  // other systems: kgather_kernel<ND>
  int kb, ke;
  ktile_range(P, wk, kb, ke);
  const int t = threadIdx.x;
  const int i0 = bk.y + t, i1 = i0 + kPartBlock / 2;
  const int iend = P.part_off + P.n;
  const bool ok0 = i0 < iend, ok1 = i1 < iend;
  const int ND_all = b.ndtot;
  // single dipole: dipole index = dip_off + (particle - part_off)
  const int g0 = ok0 ? P.dip_off + (i0 - P.part_off) : 0;
  const int g1 = ok1 ? P.dip_off + (i1 - P.part_off) : 0;
  const uint32_t ux0 = b.dfx[g0], uy0 = b.dfx[ND_all + g0], uz0 = b.dfx[2 * ND_all + g0];
  const uint32_t ux1 = b.dfx[g1], uy1 = b.dfx[ND_all + g1], uz1 = b.dfx[2 * ND_all + g1];
  const float2 mx = pk(ok0 ? b.dm[g0] : 0.f, ok1 ? b.dm[g1] : 0.f);
  const float2 my = pk(ok0 ? b.dm[ND_all + g0] : 0.f, ok1 ? b.dm[ND_all + g1] : 0.f);
  const float2 mz = pk(ok0 ? b.dm[2 * ND_all + g0] : 0.f, ok1 ? b.dm[2 * ND_all + g1] : 0.f);
  // outer accumulators (Kahan-compensated) of the per-tile sums
  float2 fo[6], fc[6], ft[6];
#pragma unroll
  for (int c = 0; c < 6; ++c) fo[c] = fc[c] = ft[c] = bc(0.f);

  uint32_t ph0 = 0u, ph1 = 0u;
  bool have = false;  // a phase from the previous k-vector (the first of the range computes its own)
  for (int k0 = kb; k0 < ke; k0 += kKBlock) {
    const int nk = stage_ktile<kPartBlock / 2, false>(b, P, k0, ke, kt);
#pragma unroll
    for (int c = 0; c < 6; ++c) ft[c] = bc(0.f);
#pragma unroll 2
    for (int q = 0; q < nk; ++q) {
      const int4 n = kt.n[q];
      const float4 kv = kt.v[q];
      const float2 vS = kt.S[q];
      float c0, s0, c1, s1;
      ph0 = phase_next(ph0, have, ux0, uy0, uz0, n);
      ph1 = phase_next(ph1, have, ux1, uy1, uz1, n);
      have = true;
      phase_cs(ph0, c0, s0);
      phase_cs(ph1, c1, s1);
      const float2 c = pk(c0, c1), sn = pk(s0, s1);
      const float2 a = __ffma2_rn(mz, bc(kv.z), __ffma2_rn(my, bc(kv.y), __fmul2_rn(mx, bc(kv.x))));
      const float2 va = __fmul2_rn(bc(kv.w), a);
      const float2 Dr = __ffma2_rn(pk(-va.x, -va.y), c, bc(vS.x));
      const float2 Dn = __ffma2_rn(va, sn, bc(vS.y));
      const float2 fF = __fmul2_rn(a, __ffma2_rn(c, Dn, __fmul2_rn(sn, Dr)));
      const float2 fT = __ffma2_rn(sn, Dn, __fmul2_rn(pk(-c.x, -c.y), Dr));
      ft[0] = __ffma2_rn(fF, bc(kv.x), ft[0]);
      ft[1] = __ffma2_rn(fF, bc(kv.y), ft[1]);
      ft[2] = __ffma2_rn(fF, bc(kv.z), ft[2]);
      ft[3] = __ffma2_rn(fT, bc(kv.x), ft[3]);
      ft[4] = __ffma2_rn(fT, bc(kv.y), ft[4]);
      ft[5] = __ffma2_rn(fT, bc(kv.z), ft[5]);
    }
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      const float2 y = __fadd2_rn(ft[c], pk(-fc[c].x, -fc[c].y));
      const float2 tt = __fadd2_rn(fo[c], y);
      fc[c] = __fadd2_rn(__fadd2_rn(tt, pk(-fo[c].x, -fo[c].y)), pk(-y.x, -y.y));
      fo[c] = tt;
    }
  }
  if (wk.y >= 0) {  // one tile: leave its sums
    float *s0 = ktile_set(b, P, i0, wk.y), *s1 = s0 + kPartBlock / 2;
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      if (ok0) s0[c * kPartBlock] = ft[c].x;
      if (ok1) s1[c * kPartBlock] = ft[c].y;
    }
    return;
  }
  float a0[6], c0[6], a1[6], c1[6];
#pragma unroll
  for (int c = 0; c < 6; ++c) {
    a0[c] = fo[c].x;
    c0[c] = fc[c].x;
    a1[c] = fo[c].y;
    c1[c] = fc[c].y;
  }
  if (ok0) store_kout(b, g0, a0, c0, mx.x, my.x, mz.x);
  if (ok1) store_kout(b, g1, a1, c1, mx.y, my.y, mz.y);
}

// The same gather with one particle per thread (128 threads per block):
// twice the warps of the packed form and no paired instructions.  Every
// particle goes through the same IEEE operations in the same order as in
// the packed kernel (explicit _rn intrinsics, no contraction), so the two
// forms give identical bits and the autotuner may pick either.  kWavesAhead
// waves are formed before their sums: in the small batches this form is for, a
// warp often has its scheduler to itself and a k-vector's chain (phase, sine,
// four dependent multiply-adds) would be the time.
constexpr int kWavesAhead = 8;
template <bool TOTALS>
__global__ void __launch_bounds__(kPartBlock) kgather1s_kernel(Batch b) {
  __shared__ KTile kt;
  const int2 wk = b.kgwork[blockIdx.x];  // (particle block, tile)
  const int2 bk = b.blk[wk.x];
  const SysDev& P = b.sys[bk.x];
  if (P.nd != 1 || at_limit(b, bk.x)) return;  // other systems: kgather_kernel<ND>
  int kb, ke;
  ktile_range(P, wk, kb, ke);
  const int t = threadIdx.x;
  const int i0 = bk.y + t;
  const bool ok0 = i0 < P.part_off + P.n;
  const int ND_all = b.ndtot;
  const int g0 = ok0 ? P.dip_off + (i0 - P.part_off) : 0;
  const uint32_t ux0 = b.dfx[g0], uy0 = b.dfx[ND_all + g0], uz0 = b.dfx[2 * ND_all + g0];
  const float mx = ok0 ? b.dm[g0] : 0.f, my = ok0 ? b.dm[ND_all + g0] : 0.f,
              mz = ok0 ? b.dm[2 * ND_all + g0] : 0.f;
  float fo[6], fc[6], ft[6];
#pragma unroll
  for (int c = 0; c < 6; ++c) fo[c] = fc[c] = ft[c] = 0.f;
  for (int k0 = kb; k0 < ke; k0 += kKBlock) {
    const int nk = stage_ktile<kPartBlock, TOTALS>(b, P, k0, ke, kt);
#pragma unroll
    for (int c = 0; c < 6; ++c) ft[c] = 0.f;
    auto add = [&](int q, float c, float sn) {
      const float4 kv = kt.v[q];
      const float2 vS = kt.S[q];
      const float a = __fmaf_rn(mz, kv.z, __fmaf_rn(my, kv.y, __fmul_rn(mx, kv.x)));
      const float va = __fmul_rn(kv.w, a);
      const float Dr = __fmaf_rn(-va, c, vS.x);
      const float Dn = __fmaf_rn(va, sn, vS.y);
      const float fF = __fmul_rn(a, __fmaf_rn(c, Dn, __fmul_rn(sn, Dr)));
      const float fT = __fmaf_rn(sn, Dn, __fmul_rn(-c, Dr));
      ft[0] = __fmaf_rn(fF, kv.x, ft[0]);
      ft[1] = __fmaf_rn(fF, kv.y, ft[1]);
      ft[2] = __fmaf_rn(fF, kv.z, ft[2]);
      ft[3] = __fmaf_rn(fT, kv.x, ft[3]);
      ft[4] = __fmaf_rn(fT, kv.y, ft[4]);
      ft[5] = __fmaf_rn(fT, kv.z, ft[5]);
    };
    int q0 = 0;
#pragma unroll 1
    for (; q0 + kWavesAhead <= nk; q0 += kWavesAhead) {
      float c[kWavesAhead], sn[kWavesAhead];
#pragma unroll
      for (int q = 0; q < kWavesAhead; ++q) phase_exp(ux0, uy0, uz0, kt.n[q0 + q], c[q], sn[q]);
#pragma unroll
      for (int q = 0; q < kWavesAhead; ++q) add(q0 + q, c[q], sn[q]);
    }
#pragma unroll 1
    for (; q0 < nk; ++q0) {
      float c, sn;
      phase_exp(ux0, uy0, uz0, kt.n[q0], c, sn);
      add(q0, c, sn);
    }
#pragma unroll
    for (int c = 0; c < 6; ++c) kahan(fo[c], fc[c], ft[c]);
  }
  if (!ok0) return;
  if (wk.y >= 0) {  // one tile: leave its sums
    float* mine = ktile_set(b, P, i0, wk.y);
#pragma unroll
    for (int c = 0; c < 6; ++c) mine[c * kPartBlock] = ft[c];
    return;
  }
  store_kout(b, g0, fo, fc, mx, my, mz);
}

template <int ND, bool TOTALS>
static void launch_kgather(const Batch& b, cudaStream_t s) {
  if (b.nkgwork == 0) return;  // k-vectors, but no rods
  if (b.ones) {
    if (b.tune.kg_scalar || TOTALS)  // the form that forms val S(k) itself is the one-rod one
      kgather1s_kernel<TOTALS><<<b.nkgwork, kPartBlock, 0, s>>>(b);
    else
      kgather1_kernel<<<b.nkgwork, kPartBlock / 2, 0, s>>>(b);
  }
  if constexpr (ND > 1) {
    if (b.gather_split)
      kgather_split_kernel<ND, TOTALS><<<b.nkgwork * (kPartBlock / 32), 32 * kGatherWarps, 0, s>>>(b);
    else
      kgather_kernel<ND, TOTALS><<<b.nkgwork, kPartBlock, 0, s>>>(b);
  }
}

template <int ND>
static void kspace_part_nd(const Batch& b, const int4* kwork, int nkwork, const int2* kowner, int part,
                           cudaStream_t s) {
  if (b.nktot == 0) return;
  if (part == 0 && nkwork > 0) launch_ksum<ND>(b, kwork, nkwork, s);
  if (part == 1) kstruct_kernel<<<cdiv(b.nktot, 32), 32 * kStructWarps, 0, s>>>(b, kowner);
  if (part == 2 && b.stage_k) launch_kgather<ND, true>(b, s);
  if (part == 2 && !b.stage_k) launch_kgather<ND, false>(b, s);
  if (part == 3) kenergy_kernel<<<b.nktile, kKBlock, 0, s>>>(b);
}

// one of the four k-space stages (0: ksum, 1: kstruct, 2: kgather, 3:
// kenergy; 2 and 3 need 0 and 1 before them, and may run side by side)
void launch_kspace_parts(const Batch& b, int maxnd, const int4* kwork, int nkwork, const int2* kowner, int part,
                         cudaStream_t s) {
  if (maxnd <= 1)
    kspace_part_nd<1>(b, kwork, nkwork, kowner, part, s);
  else if (maxnd == 2)
    kspace_part_nd<2>(b, kwork, nkwork, kowner, part, s);
  else
    kspace_part_nd<4>(b, kwork, nkwork, kowner, part, s);
}

// once per device: the step's memory split
cudaError_t prepare_kspace() {
  return set_carveout(ksum1_kernel, ksum1s_kernel, ksum_kernel<2>, ksum_kernel<4>, ksum_split_kernel<2>,
                      ksum_split_kernel<4>, kstruct_kernel, kenergy_kernel, kgather1_kernel, kgather1s_kernel<false>,
                      kgather1s_kernel<true>, kgather_kernel<2, false>, kgather_kernel<2, true>,
                      kgather_kernel<4, false>, kgather_kernel<4, true>, kgather_split_kernel<2, false>,
                      kgather_split_kernel<2, true>, kgather_split_kernel<4, false>, kgather_split_kernel<4, true>);
}

void launch_kspace(const Batch& b, int maxnd, const int4* kwork, int nkwork, const int2* kowner, cudaStream_t s) {
  for (int part : {0, 1, 3, 2}) launch_kspace_parts(b, maxnd, kwork, nkwork, kowner, part, s);
}

}  // namespace mdsc
