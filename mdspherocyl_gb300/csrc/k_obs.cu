// Observables outside the step -- the GPU form of acc_correl
// (v25/functions.cpp:2400-2470) and of the sums behind oo_params
// (:2702-2748, Qmat_3d :3426-3445).
//
// Pair histograms (acc_correl): every unordered pair of particles adds its
// terms to its distance bin floor(r / bar_w) of the functions 000, 110, 112
// and 220 -- 2, 2 dot, 2 (3 doti dotj - dot), 3 dot^2 - 1 to its species'
// histogram when both particles are of one species, and 1, dot,
// 3 doti dotj - dot, (3 dot^2 - 1) / 2 to the histogram of the species pair
// otherwise.  Species are contiguous blocks of particles, as the reference
// numbers them (calc_II / rev_II); a system's histograms are its nc species
// blocks, then the nc (nc - 1) / 2 pair blocks in the order (0,1), (0,2), ...,
// (1,2), ..., each 4 x nbins.
//
// Work: the pair triangle of a system in tiles of 128 x 128 particles (I <= J).
// A fixed grid of blocks takes runs of tiles; a thread holds one particle of
// the I strip and meets half of the J strip from shared memory.  The sums are
// integers -- the counts exactly, the three others in fixed point with 2^24
// units -- so they are the same whatever order the atomics land in.  A block
// keeps its histogram in shared memory as 32-bit words, the fixed-point terms
// split in two (v = hi 2^16 + lo): native shared atomics, where 64-bit ones
// are loops, and no sum can leave its word within kCorrFlush tiles, after
// which the block adds its words to the global 64-bit histogram.  Histograms
// that do not fit (kCorrSmemBins) add to global memory directly.
//
// 4096 particles of two species at 0.1 (3 x 330 bins): one block per 128
// particles with a 64-bit histogram took 1650 us (32 blocks, most atomics in
// global memory), this 69.
//
#include "mdsc_dev.cuh"
#include "reduce.cuh"

namespace mdsc {

constexpr int kCorrWords = 7;        // 32-bit words per bin: count, then (lo, hi) of the three sums
constexpr int kCorrSmemBins = 7000;  // most bins of a histogram in shared memory (196 KB)
constexpr int kCorrFlush = 4;        // tiles between flushes: 2^16 pairs of a block at most
constexpr int kCorrThreads = 256;
constexpr float kCorrScale = 16777216.f;  // 2^24: fixed-point unit of the non-count sums

// a block's shared histogram into the system's global one, and cleared
__device__ void corr_flush(uint32_t* sh, int nblocks, int nbins, unsigned long long* __restrict__ gh) {
  __syncthreads();
  const int bins = nblocks * nbins;
  for (int k = threadIdx.x; k < bins; k += kCorrThreads) {
    const uint32_t c = sh[k];
    if (c == 0u) continue;
    unsigned long long* g = gh + (size_t)(k / nbins) * 4 * nbins + k % nbins;
    atomicAdd(g, (unsigned long long)c);
    sh[k] = 0u;
#pragma unroll
    for (int f = 0; f < 3; ++f) {
      const long long v = ((long long)(int32_t)sh[(2 * f + 2) * bins + k] << 16) + sh[(2 * f + 1) * bins + k];
      atomicAdd(g + (f + 1) * nbins, (unsigned long long)v);
      sh[(2 * f + 1) * bins + k] = sh[(2 * f + 2) * bins + k] = 0u;
    }
  }
  __syncthreads();
}

template <bool SMEM>
__global__ void __launch_bounds__(kCorrThreads) corr_kernel(Batch b, const CorrSys* __restrict__ cs,
                                                            const unsigned char* __restrict__ species, double bar_w,
                                                            int ntiles, unsigned long long* __restrict__ hist) {
  extern __shared__ uint32_t shist[];
  __shared__ uint32_t sx[kPartBlock], sy[kPartBlock], sz[kPartBlock];
  __shared__ float4 sa[kPartBlock];
  __shared__ unsigned char ssp[kPartBlock];
  const int per = cdiv(ntiles, gridDim.x);
  const int t0 = blockIdx.x * per, t1 = min(ntiles, t0 + per);
  if (t0 >= t1) return;
  int s = 0;
  while (t0 >= cs[s].tile_off + cs[s].ntiles) ++s;
  CorrSys C = cs[s];
  int nblocks = C.nsp + C.nsp * (C.nsp - 1) / 2, bins = nblocks * C.nbins;
  if (SMEM) {
    for (int k = threadIdx.x; k < kCorrWords * bins; k += kCorrThreads) shist[k] = 0u;
  }
  const int N = b.ntot;
  const float ibw = (float)(1.0 / bar_w);
  int since = 0;
  for (int tile = t0; tile < t1; ++tile) {
    if (tile >= C.tile_off + C.ntiles || since == kCorrFlush) {
      if (SMEM) corr_flush(shist, nblocks, C.nbins, hist + C.off);
      since = 0;
      if (tile >= C.tile_off + C.ntiles) {
        while (tile >= cs[s].tile_off + cs[s].ntiles) ++s;
        C = cs[s];
        nblocks = C.nsp + C.nsp * (C.nsp - 1) / 2;
        bins = nblocks * C.nbins;
        if (SMEM)
          for (int k = threadIdx.x; k < kCorrWords * bins; k += kCorrThreads) shist[k] = 0u;
      }
    }
    ++since;
    const SysDev& P = b.sys[s];
    const int nbins = C.nbins, nc = C.nsp;
    // tile -> strips (I, J), I <= J, row by row of the upper triangle
    const int ns = cdiv(P.n, kPartBlock);
    int I = 0, q = tile - C.tile_off;
    while (q >= ns - I) q -= ns - I++;
    const int J = I + q;
    const int iend = P.part_off + P.n;
    const int i = P.part_off + I * kPartBlock + (threadIdx.x & (kPartBlock - 1));
    const int j0 = P.part_off + J * kPartBlock;
    const int nj = min(kPartBlock, iend - j0);
    const bool ok = i < iend;
    // how far the FP32 t = r / bar_w may be from the reference's: ~8 roundings
    // relative (bounded by 1e-6 t) plus the fixed-point quantum of each
    // coordinate difference (L / 2^32 per axis, doubled)
    const float q0 = (float)(4.0 * fmax(P.L[0], fmax(P.L[1], P.L[2])) / 4294967296.0 / bar_w) + 1e-6f;
    __syncthreads();
    if (threadIdx.x < nj) {
      const int p = j0 + threadIdx.x;
      sx[threadIdx.x] = b.pfx[p];
      sy[threadIdx.x] = b.pfx[N + p];
      sz[threadIdx.x] = b.pfx[2 * N + p];
      sa[threadIdx.x] = b.pax[p];
      ssp[threadIdx.x] = species[p];
    }
    __syncthreads();
    if (!ok) continue;
    const uint32_t ux = b.pfx[i], uy = b.pfx[N + i], uz = b.pfx[2 * N + i];
    const float4 ai = b.pax[i];
    const int spi = species[i];
    const int k1 = min(nj, (threadIdx.x >> 7) * 64 + 64);
    for (int k = (threadIdx.x >> 7) * 64; k < k1; ++k) {
      const int j = j0 + k;
      if (j <= i) continue;
      const float dx = fix_diff(ux, sx[k], P.Lfix[0]);
      const float dy = fix_diff(uy, sy[k], P.Lfix[1]);
      const float dz = fix_diff(uz, sz[k], P.Lfix[2]);
      const float4 aj = sa[k];
      float r = sqrtf(dx * dx + dy * dy + dz * dz);
      const float t = r * ibw;
      int bin = (int)floorf(t);
      const float fr = t - (float)bin;
      const float edge = 1e-6f * t + q0;
      if (fr < edge || fr > 1.f - edge) {
        // near a bin edge: the reference's distance in FP64, rounded step
        // by step as it is (no fused multiply-adds)
        double D[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const double X = __dsub_rn(b.r[3 * i + a], b.r[3 * j + a]);
          D[a] = __dsub_rn(X, __dmul_rn(P.L[a], floor(__dadd_rn(X / P.L[a], 0.5))));
        }
        const double R = sqrt(__dadd_rn(__dadd_rn(__dmul_rn(D[0], D[0]), __dmul_rn(D[1], D[1])),
                                        __dmul_rn(D[2], D[2])));
        bin = (int)floor(R / bar_w);
      }
      if (bin < 0 || bin >= nbins) continue;
      const float dot = ai.x * aj.x + ai.y * aj.y + ai.z * aj.z;
      const float ir = r > 0.f ? 1.f / r : 0.f;
      const float doti = (ai.x * dx + ai.y * dy + ai.z * dz) * ir;
      const float dotj = (aj.x * dx + aj.y * dy + aj.z * dz) * ir;
      // i < j and species ascend with the index, so spi <= spj
      const int spj = ssp[k];
      const bool intra = spi == spj;
      // pair block (m, n), m < n: after the nc species blocks, in row order
      const int blkno = intra ? spi : nc + spi * (2 * nc - spi - 1) / 2 + (spj - spi - 1);
      const float w = intra ? 2.f : 1.f;
      const int v110 = __float2int_rn(w * dot * kCorrScale);
      const int v112 = __float2int_rn(w * (3.f * doti * dotj - dot) * kCorrScale);
      const int v220 = __float2int_rn(0.5f * w * (3.f * dot * dot - 1.f) * kCorrScale);
      if (SMEM) {
        uint32_t* h = shist + blkno * nbins + bin;
        atomicAdd(h, intra ? 2u : 1u);
        atomicAdd(h + 1 * bins, (uint32_t)v110 & 0xffffu);
        atomicAdd(h + 2 * bins, (uint32_t)(v110 >> 16));
        atomicAdd(h + 3 * bins, (uint32_t)v112 & 0xffffu);
        atomicAdd(h + 4 * bins, (uint32_t)(v112 >> 16));
        atomicAdd(h + 5 * bins, (uint32_t)v220 & 0xffffu);
        atomicAdd(h + 6 * bins, (uint32_t)(v220 >> 16));
      } else {
        unsigned long long* hb = hist + C.off + (size_t)blkno * 4 * nbins;
        atomicAdd(&hb[0 * nbins + bin], intra ? 2ull : 1ull);
        atomicAdd(&hb[1 * nbins + bin], (unsigned long long)(long long)v110);
        atomicAdd(&hb[2 * nbins + bin], (unsigned long long)(long long)v112);
        atomicAdd(&hb[3 * nbins + bin], (unsigned long long)(long long)v220);
      }
    }
  }
  if (SMEM) corr_flush(shist, nblocks, C.nbins, hist + C.off);
}

// Per particle block: sum of the rod axes (3), of their outer products (6,
// the Q tensor's input) and of the dipole moment vectors mu O^T o_body (3),
// in FP64, then float-float over the block.
__global__ void __launch_bounds__(kPartBlock) order_sums_kernel(Batch b, double* __restrict__ out) {
  __shared__ double sh[12 * kPartBlock / 32];
  const int2 bk = b.blk[blockIdx.x];
  const SysDev& P = b.sys[bk.x];
  const int i = bk.y + threadIdx.x;
  double v[12];
#pragma unroll
  for (int c = 0; c < 12; ++c) v[c] = 0.0;
  if (i < P.part_off + P.n) {
    const double* O = b.O + 9 * i;
    const double o0 = O[6], o1 = O[7], o2 = O[8];
    v[0] = o0;
    v[1] = o1;
    v[2] = o2;
    v[3] = o0 * o0;
    v[4] = o0 * o1;
    v[5] = o0 * o2;
    v[6] = o1 * o1;
    v[7] = o1 * o2;
    v[8] = o2 * o2;
    const int g0 = P.dip_off + (i - P.part_off) * P.nd;
    for (int w = 0; w < P.nd; ++w) {
      const int g = g0 + w;
      const double ox = b.dob[3 * g], oy = b.dob[3 * g + 1], oz = b.dob[3 * g + 2], mu = b.dmu[g];
      v[9] += mu * (O[0] * ox + O[3] * oy + O[6] * oz);
      v[10] += mu * (O[1] * ox + O[4] * oy + O[7] * oz);
      v[11] += mu * (O[2] * ox + O[5] * oy + O[8] * oz);
    }
  }
  double tot[12];
  block_sum<12, kPartBlock>(v, sh, tot);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int c = 0; c < 12; ++c) out[12 * blk_slot(P, bk) + c] = tot[c];
  }
}

// ntiles: 128 x 128 tiles over all systems (CorrSys); max_bins: the largest
// (species blocks + pair blocks) x nbins of any system
cudaError_t launch_correlations(const Batch& b, const CorrSys* c, const unsigned char* species, double bar_w,
                                int ntiles, int max_bins, unsigned long long* hist, cudaStream_t s) {
  if (ntiles <= 0) return cudaSuccess;
  // two blocks per SM: a run of tiles pays for a block's clearing and flush
  const int grid = ntiles < 2 * kSMs ? ntiles : 2 * kSMs;
  if (max_bins <= kCorrSmemBins) {
    const int bytes = kCorrWords * max_bins * (int)sizeof(uint32_t);
    const cudaError_t e = cudaFuncSetAttribute(corr_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               kCorrWords * kCorrSmemBins * (int)sizeof(uint32_t));
    if (e != cudaSuccess) return e;
    corr_kernel<true><<<grid, kCorrThreads, bytes, s>>>(b, c, species, bar_w, ntiles, hist);
  } else {
    corr_kernel<false><<<grid, kCorrThreads, 0, s>>>(b, c, species, bar_w, ntiles, hist);
  }
  return cudaGetLastError();
}

void launch_order_sums(const Batch& b, double* out, cudaStream_t s) {
  if (b.nblk) order_sums_kernel<<<b.nblk, kPartBlock, 0, s>>>(b, out);
}

}  // namespace mdsc
