// Headless picture of a system -- the GPU replacement of the reference's
// SDL/OpenGL viewer (v25/graphic.cpp), which needs a display and a GL stack.
// The scene is the viewer's (v25/graphic.cpp:183-330,612-680):
//   * each rod a spherocylinder of its length and diameter, grey by species
//     (tone_list), with a blue tip on the +axis cap (latitude sin > 0.8) and
//     red and green meridians on the cylinder marking the body x and y axes;
//   * each dipole a pair of segments through its position, blue behind and
//     red ahead, 1.5 radii long each;
//   * the box edges in (0.6, 0.3, 0.3), around [-L/2, L/2]^3;
//   * optionally the 26 periodic images, optionally one cluster only;
//   * white background, the viewer's camera: gluLookAt from
//     usr = dist (sin t cos p, sin t sin p, cos t) to ref with z up, then
//     moved back |usr| along the view (computeLocation, :405-415), a
//     60-degree vertical field; ambient 0.5 plus a directional light of 0.7
//     from usr (:612-624).
// Lines of the viewer (dipoles 2 pixels wide, box edges 1) become capsules
// of that width at the distance looked at.
// It is ray cast instead of rasterised: one thread per pixel, blocks of 16 x 8
// pixels.  A block first keeps the capsules (rods, dipole segments, box edges)
// whose bounding sphere meets the cone around its rays, in scene order, and
// its pixels test those.  Output: 8-bit RGB, rows from the top.
#include "mdsc_dev.cuh"

namespace mdsc {

// a capsule of the scene: segment a..b, radius, shading data
struct Capsule {
  float ax, ay, az, bx, by, bz;
  float rad;
  float ex, ey, ez;     // body x axis (rods), for the meridians
  float tone;           // grey of the species (rods); < 0: flat colour r, g, b below
  float cr, cg, cb;     // flat colour (segments)
  int kind;             // 0 rod, 1 segment
};

struct RenderView {
  int width, height;
  float eye[3], fwd[3], right[3], up[3];
  float tan_half;   // tan(fov / 2)
  float light[3];   // unit vector towards the light
};

__constant__ float kTone[5] = {1.f, 0.4f, 0.6f, 0.2f, 0.8f};

// a sphere that holds the capsule (centre, radius); radius < 0: nothing to hit
__device__ __forceinline__ float4 ball_of(const Capsule& c) {
  const float dx = 0.5f * (c.bx - c.ax), dy = 0.5f * (c.by - c.ay), dz = 0.5f * (c.bz - c.az);
  return make_float4(0.5f * (c.ax + c.bx), 0.5f * (c.ay + c.by), 0.5f * (c.az + c.bz),
                     c.rad > 0.f ? sqrtf(dx * dx + dy * dy + dz * dz) + c.rad : -1.f);
}

// per particle: its rod (and its periodic images) and its dipoles' segments
__global__ void scene_kernel(Batch b, int sys, const unsigned char* __restrict__ species,
                             const int* __restrict__ keep, int images, int dipoles, float seg_rad,
                             Capsule* __restrict__ rods, Capsule* __restrict__ segs, float4* __restrict__ ball,
                             int seg0, int* __restrict__ counts) {
  const SysDev& P = b.sys[sys];
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= P.n) return;
  if (keep && !keep[k]) return;
  const int i = P.part_off + k;
  const double* O = b.O + 9 * i;
  const double* r = b.r + 3 * i;
  const float h = (float)(0.5 * b.len[i]), rad = (float)(0.5 * b.dia[i]);
  const float u[3] = {(float)O[6], (float)O[7], (float)O[8]};
  const int nimg = images ? 27 : 1;
  const int ri = atomicAdd(&counts[0], nimg);
  const int nd = dipoles ? P.nd : 0;
  const int si = atomicAdd(&counts[1], 2 * nd * nimg);
  for (int m = 0; m < nimg; ++m) {
    const float sh[3] = {images ? (float)(P.L[0] * (m % 3 - 1)) : 0.f,
                         images ? (float)(P.L[1] * ((m / 3) % 3 - 1)) : 0.f,
                         images ? (float)(P.L[2] * (m / 9 - 1)) : 0.f};
    const float c[3] = {(float)r[0] + sh[0], (float)r[1] + sh[1], (float)r[2] + sh[2]};
    // the ends' roundings written out: which of two capsules that meet a pixel has
    // hangs on their last bits, and the bounding spheres share their terms
    Capsule q;
    q.ax = __fsub_rn(c[0], __fmul_rn(h, u[0]));
    q.ay = __fsub_rn(c[1], __fmul_rn(h, u[1]));
    q.az = __fsub_rn(c[2], __fmul_rn(h, u[2]));
    q.bx = __fadd_rn(c[0], __fmul_rn(h, u[0]));
    q.by = __fadd_rn(c[1], __fmul_rn(h, u[1]));
    q.bz = __fadd_rn(c[2], __fmul_rn(h, u[2]));
    q.rad = rad;
    q.ex = (float)O[0];
    q.ey = (float)O[1];
    q.ez = (float)O[2];
    q.tone = kTone[species[k] % 5];
    q.cr = q.cg = q.cb = 0.f;
    q.kind = 0;
    rods[ri + m] = q;
    ball[ri + m] = ball_of(q);
    // dipoles: lab position r + offset * axis, direction O^T o_body
    for (int w = 0; w < nd; ++w) {
      const int g = P.dip_off + k * nd + w;
      if (b.dmu[g] == 0.0) {
        // a padding dipole: an empty segment
        for (int s = 0; s < 2; ++s) {
          Capsule z{};
          z.rad = 0.f;
          z.kind = 1;
          z.tone = -1.f;
          segs[si + 2 * (m * nd + w) + s] = z;
          ball[seg0 + si + 2 * (m * nd + w) + s] = ball_of(z);
        }
        continue;
      }
      const double pc = b.dpc[g];
      const float p[3] = {c[0] + (float)(pc * O[6]), c[1] + (float)(pc * O[7]), c[2] + (float)(pc * O[8])};
      const double ox = b.dob[3 * g], oy = b.dob[3 * g + 1], oz = b.dob[3 * g + 2];
      const float d[3] = {(float)(O[0] * ox + O[3] * oy + O[6] * oz), (float)(O[1] * ox + O[4] * oy + O[7] * oz),
                          (float)(O[2] * ox + O[5] * oy + O[8] * oz)};
      const float mlt = 1.5f * rad, thick = seg_rad;
      for (int s = 0; s < 2; ++s) {
        Capsule z;
        const float s0 = s == 0 ? -mlt : 0.f, s1 = s == 0 ? 0.f : mlt;
        z.ax = __fmaf_rn(s0, d[0], p[0]);
        z.ay = __fmaf_rn(s0, d[1], p[1]);
        z.az = __fmaf_rn(s0, d[2], p[2]);
        z.bx = __fmaf_rn(s1, d[0], p[0]);
        z.by = __fmaf_rn(s1, d[1], p[1]);
        z.bz = __fmaf_rn(s1, d[2], p[2]);
        z.rad = thick;
        z.ex = z.ey = z.ez = 0.f;
        z.tone = -1.f;
        z.cr = s == 0 ? 0.f : 1.f;
        z.cg = 0.f;
        z.cb = s == 0 ? 1.f : 0.f;
        z.kind = 1;
        segs[si + 2 * (m * nd + w) + s] = z;
        ball[seg0 + si + 2 * (m * nd + w) + s] = ball_of(z);
      }
    }
  }
}

// distance along the unit ray o + t d to the capsule surface, or -1
__device__ __forceinline__ float hit_capsule(const float o[3], const float d[3], const Capsule& c) {
  if (c.rad <= 0.f) return -1.f;
  const float ba[3] = {c.bx - c.ax, c.by - c.ay, c.bz - c.az};
  const float oa[3] = {o[0] - c.ax, o[1] - c.ay, o[2] - c.az};
  const float baba = ba[0] * ba[0] + ba[1] * ba[1] + ba[2] * ba[2];
  const float bard = ba[0] * d[0] + ba[1] * d[1] + ba[2] * d[2];
  const float baoa = ba[0] * oa[0] + ba[1] * oa[1] + ba[2] * oa[2];
  const float rdoa = d[0] * oa[0] + d[1] * oa[1] + d[2] * oa[2];
  const float oaoa = oa[0] * oa[0] + oa[1] * oa[1] + oa[2] * oa[2];
  const float r2 = c.rad * c.rad;
  // the cylinder: |(oa + t d) - ((oa + t d).ba / baba) ba|^2 = r^2, a quadratic in t
  const float qa = baba - bard * bard;
  const float qb = baba * rdoa - baoa * bard;
  const float qc = baba * oaoa - baoa * baoa - r2 * baba;
  if (qa > 1e-12f * baba) {
    const float disc = qb * qb - qa * qc;
    if (disc >= 0.f) {
      const float t = (-qb - sqrtf(disc)) / qa;
      const float y = baoa + t * bard;  // along the axis, 0..baba on the body
      if (t > 0.f && y > 0.f && y < baba) return t;
    }
  }
  // the end spheres: the nearer of the two intersections
  float best = -1.f;
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const float oc[3] = {e ? o[0] - c.bx : oa[0], e ? o[1] - c.by : oa[1], e ? o[2] - c.bz : oa[2]};
    const float hb = d[0] * oc[0] + d[1] * oc[1] + d[2] * oc[2];
    const float hc = oc[0] * oc[0] + oc[1] * oc[1] + oc[2] * oc[2] - r2;
    const float disc = hb * hb - hc;
    if (disc >= 0.f) {
      const float t = -hb - sqrtf(disc);
      if (t > 0.f && (best < 0.f || t < best)) best = t;
    }
  }
  return best;
}

constexpr int kRenderTile = 128;

// the unit ray through the centre of a pixel
__device__ __forceinline__ void pixel_ray(const RenderView& v, int px, int py, float d[3]) {
  const float aspect = (float)v.width / (float)v.height;
  const float sx = (2.f * (px + 0.5f) / v.width - 1.f) * v.tan_half * aspect;
  const float sy = (1.f - 2.f * (py + 0.5f) / v.height) * v.tan_half;
  float nrm = 0.f;
  for (int a = 0; a < 3; ++a) {
    d[a] = v.fwd[a] + sx * v.right[a] + sy * v.up[a];
    nrm += d[a] * d[a];
  }
  nrm = rsqrtf(nrm);
  for (int a = 0; a < 3; ++a) d[a] *= nrm;
}

__device__ __forceinline__ float cross_norm(const float a[3], const float b[3]) {
  const float x = a[1] * b[2] - a[2] * b[1], y = a[2] * b[0] - a[0] * b[2], z = a[0] * b[1] - a[1] * b[0];
  return sqrtf(x * x + y * y + z * z);
}

// A picture of 2000 rods with their dipoles (6012 capsules, 480 x 480): every
// ray against every capsule took 3310 us, bound by the hit tests' FP32; with
// the cone test below 73.
__global__ void __launch_bounds__(kRenderTile) render_kernel(RenderView v, const Capsule* __restrict__ rods,
                                                             const Capsule* __restrict__ segs,
                                                             const float4* __restrict__ ball, int seg0,
                                                             const int* __restrict__ counts,
                                                             unsigned char* __restrict__ rgb) {
  __shared__ Capsule sc[kRenderTile];
  __shared__ int keep[2 * kRenderTile];
  __shared__ int wcnt[kRenderTile / 32];
  const int px0 = blockIdx.x * 16, py0 = blockIdx.y * 8;
  const int px = px0 + (threadIdx.x & 15), py = py0 + (threadIdx.x >> 4);
  const bool on = px < v.width && py < v.height;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float d[3];
  pixel_ray(v, px, py, d);
  // the cone: its axis between two opposite corner rays, its angle that of the
  // widest of the four (the others lie between them, as long as that is below a
  // right angle: a block of a low, wide picture can span more, and then its rays
  // are tested against everything)
  float axis[3], sn = 0.f, cs = 1.f;
  {
    float c[4][3], nrm = 0.f;
    for (int k = 0; k < 4; ++k) pixel_ray(v, px0 + (k & 1 ? 15 : 0), py0 + (k & 2 ? 7 : 0), c[k]);
    for (int a = 0; a < 3; ++a) {
      axis[a] = c[0][a] + c[3][a];
      nrm += axis[a] * axis[a];
    }
    nrm = rsqrtf(nrm);
    for (int a = 0; a < 3; ++a) axis[a] *= nrm;
    for (int k = 0; k < 4; ++k) {
      sn = fmaxf(sn, cross_norm(axis, c[k]));
      cs = fminf(cs, axis[0] * c[k][0] + axis[1] * c[k][1] + axis[2] * c[k][2]);
    }
    sn *= 1.0001f;
  }
  const bool wide = !(cs > 0.1f);
  float tmin = 3.0e38f;
  int hit_k = -1, hit_list = 0;
  for (int list = 0; list < 2; ++list) {
    const Capsule* src = list ? segs : rods;
    const float4* bl = ball + (list ? seg0 : 0);
    const int n = counts[list];
    int have = 0;
    for (int c0 = 0; c0 < n; c0 += kRenderTile) {
      // the capsules of this chunk that the cone may meet, in order
      const int q = c0 + (int)threadIdx.x;
      bool in = false;
      if (q < n) {
        const float4 s = bl[q];
        const float w[3] = {s.x - v.eye[0], s.y - v.eye[1], s.z - v.eye[2]};
        const float t = w[0] * axis[0] + w[1] * axis[1] + w[2] * axis[2], perp = cross_norm(w, axis);
        // room for the rounding of t and perp
        const float r = s.w * 1.001f + 1e-5f * (fabsf(t) + perp);
        // outside: behind the eye, or further from the cone than its radius
        // (the distance to the cone's edge line is never above that to the cone)
        in = s.w >= 0.f && (wide || !(t < -r || perp * cs - t * sn > r));
      }
      const uint32_t m = __ballot_sync(0xffffffffu, in);
      if (lane == 0) wcnt[warp] = __popc(m);
      __syncthreads();
      int at = have;
      for (int k = 0; k < kRenderTile / 32; ++k) {
        at += k < warp ? wcnt[k] : 0;
        have += wcnt[k];
      }
      if (in) keep[at + __popc(m & ((1u << lane) - 1u))] = q;
      __syncthreads();
      // test a full chunk of kept capsules, or what is left at the end
      while (have >= kRenderTile || (have > 0 && c0 + kRenderTile >= n)) {
        const int cnt = min(have, kRenderTile);
        if ((int)threadIdx.x < cnt) sc[threadIdx.x] = src[keep[threadIdx.x]];
        __syncthreads();
        if (on)
          for (int k = 0; k < cnt; ++k) {
            const float t = hit_capsule(v.eye, d, sc[k]);
            if (t > 0.f && t < tmin) {
              tmin = t;
              hit_k = keep[k];
              hit_list = list;
            }
          }
        __syncthreads();
        const int rest = have - cnt;  // below kRenderTile
        const int mv = (int)threadIdx.x < rest ? keep[cnt + threadIdx.x] : 0;
        __syncthreads();
        if ((int)threadIdx.x < rest) keep[threadIdx.x] = mv;
        have = rest;
        __syncthreads();
      }
    }
  }
  const bool any = hit_k >= 0;
  Capsule hit{};
  if (any) hit = (hit_list ? segs : rods)[hit_k];
  if (!on) return;
  float col[3] = {1.f, 1.f, 1.f};  // the background
  if (any) {
    const float p[3] = {v.eye[0] + tmin * d[0], v.eye[1] + tmin * d[1], v.eye[2] + tmin * d[2]};
    if (hit.kind == 1) {
      col[0] = hit.cr;
      col[1] = hit.cg;
      col[2] = hit.cb;
    } else {
      // the nearest point of the axis segment gives the normal
      const float ba[3] = {hit.bx - hit.ax, hit.by - hit.ay, hit.bz - hit.az};
      const float len2 = ba[0] * ba[0] + ba[1] * ba[1] + ba[2] * ba[2];
      const float pa[3] = {p[0] - hit.ax, p[1] - hit.ay, p[2] - hit.az};
      float s = len2 > 0.f ? (pa[0] * ba[0] + pa[1] * ba[1] + pa[2] * ba[2]) / len2 : 0.f;
      s = fminf(fmaxf(s, 0.f), 1.f);
      float nv[3];
      for (int a = 0; a < 3; ++a) nv[a] = (pa[a] - s * ba[a]) / hit.rad;
      const float il = len2 > 0.f ? rsqrtf(len2) : 0.f;
      const float u[3] = {ba[0] * il, ba[1] * il, ba[2] * il};
      float base[3] = {hit.tone, hit.tone, hit.tone};
      if (s >= 1.f) {
        // the +axis cap: blue above latitude sin = 0.8
        const float z = nv[0] * u[0] + nv[1] * u[1] + nv[2] * u[2];
        if (z > 0.8f) base[0] = base[1] = 0.f, base[2] = 1.f;
      } else if (s > 0.f) {
        // the cylinder: red and green meridians at the body x and y axes,
        // fading over one facet of the viewer's 12 (30 degrees) on each side
        const float ey[3] = {u[1] * hit.ez - u[2] * hit.ey, u[2] * hit.ex - u[0] * hit.ez,
                             u[0] * hit.ey - u[1] * hit.ex};
        const float cx = nv[0] * hit.ex + nv[1] * hit.ey + nv[2] * hit.ez;
        const float cy = nv[0] * ey[0] + nv[1] * ey[1] + nv[2] * ey[2];
        const float phi = atan2f(cy, cx);
        const float facet = 3.14159265f / 6.f;
        const float wr = fmaxf(0.f, 1.f - fabsf(phi) / facet);
        const float wg = fmaxf(0.f, 1.f - fabsf(phi - 1.57079633f) / facet);
        const float wt = 1.f - wr - wg;
        base[0] = wt * hit.tone + wr;
        base[1] = wt * hit.tone + wg;
        base[2] = wt * hit.tone;
      }
      const float lam = fmaxf(0.f, nv[0] * v.light[0] + nv[1] * v.light[1] + nv[2] * v.light[2]);
      const float shade = 0.5f + 0.7f * lam;
      for (int a = 0; a < 3; ++a) col[a] = fminf(1.f, base[a] * shade);
    }
  }
  const size_t o = 3 * ((size_t)py * v.width + px);
  for (int a = 0; a < 3; ++a) rgb[o + a] = (unsigned char)__float2int_rn(255.f * fminf(fmaxf(col[a], 0.f), 1.f));
}

// the box's 12 edges as flat segments
__global__ void box_kernel(Batch b, int sys, float thick, Capsule* __restrict__ segs, float4* __restrict__ ball,
                           int seg0, int* __restrict__ counts) {
  const int e = threadIdx.x;
  if (e >= 12) return;
  const SysDev& P = b.sys[sys];
  const float h[3] = {(float)(0.5 * P.L[0]), (float)(0.5 * P.L[1]), (float)(0.5 * P.L[2])};
  const int axis = e / 4, corner = e % 4;
  float a[3], c[3];
  const int o1 = (axis + 1) % 3, o2 = (axis + 2) % 3;
  a[axis] = -h[axis];
  c[axis] = h[axis];
  a[o1] = c[o1] = (corner & 1) ? h[o1] : -h[o1];
  a[o2] = c[o2] = (corner & 2) ? h[o2] : -h[o2];
  const int base = atomicAdd(&counts[1], 0);  // the dipole segments are written first
  Capsule z;
  z.ax = a[0];
  z.ay = a[1];
  z.az = a[2];
  z.bx = c[0];
  z.by = c[1];
  z.bz = c[2];
  z.rad = thick;
  z.ex = z.ey = z.ez = 0.f;
  z.tone = -1.f;
  z.cr = 0.6f;
  z.cg = 0.3f;
  z.cb = 0.3f;
  z.kind = 1;
  segs[base + e] = z;
  ball[seg0 + base + e] = ball_of(z);
  __syncthreads();
  if (e == 0) counts[1] = base + 12;
}

size_t render_scratch_bytes(int n, int nd, int images) {
  const size_t nimg = images ? 27 : 1;
  return (sizeof(Capsule) + sizeof(float4)) * ((size_t)n * nimg + (size_t)2 * n * nd * nimg + 12) + 128;
}

// scratch: render_scratch_bytes(n, nd, images) bytes of device memory;
// eye, fwd, right, up: the camera frame; light: unit vector to the light;
// seg_rad, box_rad: radii of the dipole and box-edge capsules
void launch_render(const Batch& b, int sys, int n, int nd, const unsigned char* species, const int* keep, int images,
                   int dipoles, int draw_box, float seg_rad, float box_rad, const float* eye, const float* fwd,
                   const float* right, const float* up, const float* light, float tan_half, int width,
                   int height, void* scratch, unsigned char* rgb, cudaStream_t s) {
  char* base = static_cast<char*>(scratch);
  int* counts = reinterpret_cast<int*>(base);
  Capsule* rods = reinterpret_cast<Capsule*>(base + 64);
  const size_t nimg = images ? 27 : 1;
  Capsule* segs = rods + (size_t)n * nimg;
  const size_t total = (size_t)n * nimg + (size_t)2 * n * nd * nimg + 12;
  float4* ball = reinterpret_cast<float4*>(base + (64 + sizeof(Capsule) * total + 15) / 16 * 16);
  const int seg0 = (int)((size_t)n * nimg);
  cudaMemsetAsync(counts, 0, 64, s);
  if (n > 0)
    scene_kernel<<<cdiv(n, 128), 128, 0, s>>>(b, sys, species, keep, images, dipoles, seg_rad, rods, segs, ball, seg0,
                                              counts);
  if (draw_box) box_kernel<<<1, 32, 0, s>>>(b, sys, box_rad, segs, ball, seg0, counts);
  RenderView v;
  v.width = width;
  v.height = height;
  for (int a = 0; a < 3; ++a) {
    v.eye[a] = eye[a];
    v.fwd[a] = fwd[a];
    v.right[a] = right[a];
    v.up[a] = up[a];
    v.light[a] = light[a];
  }
  v.tan_half = tan_half;
  dim3 grid(cdiv(width, 16), cdiv(height, 8));
  render_kernel<<<grid, kRenderTile, 0, s>>>(v, rods, segs, ball, seg0, counts, rgb);
}

}  // namespace mdsc
