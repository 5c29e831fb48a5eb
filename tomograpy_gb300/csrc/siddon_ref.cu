// Double-precision projector that follows the reference's arithmetic step by
// step, and the unit-vector / intersection-parameter diagnostics.
//
// This translation unit is compiled with --fmad=false: the reference is
// built without FMA contraction, and every expression below is evaluated in
// the reference's order, so with the same ray direction the f64 GPU path
// reproduces the reference's double-precision results (differences come only
// from the last bits of CUDA's sin / cos versus the host libm).
//
//   conic_image_projector  tomograpy/C_siddon.c.template:500-528
//   ray_projector          :530-580
//   voxel (merge step)     :811-912
//   pj / bpj / pjt / bpjt  :914-944
//   in_map / sun           :947-961
#include "siddon_geom.cuh"

namespace tg {

// What bounds it: the FP64 pipe (1/64 of the FP32 rate), so every FP64
// instruction that is not one of the reference's own additions and products is
// kept off the walk, with the same results:
//  * comparisons: after the first step every plane distance is positive, and
//    positive doubles order like their bit patterns, so the minimum and the
//    ties are integer comparisons (the reference's 6 per step);
//  * the obstacle test (12 per step): |M + ac u|^2 > 1 holds for certain
//    outside the parameter window in which |r|^2 <= 1 + 1e-5, which is set up
//    once per ray; the upper words of ac and of the window's ends decide it,
//    and inside the window the reference's test runs;
//  * four rows per CTA, not eight, to even out the SMs' shares of small launches;
//  * the product of a step is added one step later (same order), so its gather
//    is not waited for.
// Measured on GB300, P then P^T in float64 at 48^3 x 12 x 64^2, sun: 633 ->
// 262 us (352 us with eight rows per CTA, 246 us with two, whose tables weigh
// more in larger launches).

// Parameter window outside which |M + ac u|^2 > 1 for certain, as the upper
// words of its ends; negative parameters are always tested.
struct SunWindow {
  int lo, span;
  __device__ __forceinline__ bool test(double ac) const {
    const int h = __double2hiint(ac);
    return h < 0 || (unsigned)(h - lo) <= (unsigned)span;
  }
};

__device__ __forceinline__ SunWindow sun_window(const double M[3], const double u[3]) {
  // |M + s u|^2 - 1 = (s + b)^2 - disc + s^2 (uu - 1): for a unit vector u at
  // most 1e-5 within sqrt(disc + 1e-5) of -b.  Inside the sphere |s u| <= |M| + 1,
  // so the last term is below 2 (mm + 1) |uu - 1|, at most 2e-6 here; the
  // rounding of disc (about 1e-15 mm) and of the single-precision root is at
  // most 1e-6 together for |M| < 1e4.  The 1e-5 covers them.  Directions
  // further off unit length (the matrix of a header with few decimals: 1e-9 is
  // 5e-5 at 215 radii) are tested everywhere.
  const double uu = u[0] * u[0] + u[1] * u[1] + u[2] * u[2];
  const double mm = M[0] * M[0] + M[1] * M[1] + M[2] * M[2];
  if (!((float)mm < 1e8f && fabs(uu - 1.0) * (mm + 1.0) < 1e-6)) return {0, 0x7fffffff};
  const double b = M[0] * u[0] + M[1] * u[1] + M[2] * u[2];
  const float disc = (float)(b * b - mm + 1.0) + 1e-5f;
  if (disc < 0.f) return {0x7fffffff, 0};
  const double sq = (double)sqrtf(disc);
  const int lo = __double2hiint(-b - sq), hi = __double2hiint(sq - b);
  if (hi < 0) return {0x7fffffff, 0};
  return {max(lo, 0), hi - max(lo, 0)};
}

template <int MODE, bool SUN>
__global__ void __launch_bounds__(kThreads)
ref64_kernel(const Geometry G, const double *__restrict__ xin, double *__restrict__ xout) {
  constexpr bool PJ = (MODE == TG_PJ || MODE == TG_PJT);
  constexpr bool T4 = (MODE == TG_PJT || MODE == TG_BPJT);
  __shared__ TrigTables T;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int t = G.view0 + blockIdx.z;
  const tg_image_header &V = G.views[t];
  const int col0 = (G.bx0 + blockIdx.x) * 32, row0 = (G.by0 + blockIdx.y) * (blockDim.x >> 5);
  fill_trig(T, V, col0, row0);
  __syncthreads();
  const int i = row0 + warp, j = col0 + lane;
  if (i >= G.n1 || j >= G.n2) return;
  if (G.ray_i >= 0 && (i != G.ray_i || j != G.ray_j)) return;
  if (masked(G, i, j, t)) return;
  long long fbase = 0;
  if (T4) {
    const int f = V.frame;
    if (f < 0 || f >= G.nframes) return;
    fbase = (long long)f * G.ms[3];
  }
  const long long po = (long long)i * G.ds[0] + (long long)j * G.ds[1] + (long long)t * G.ds[2];
  const double M[3] = {V.M[0], V.M[1], V.M[2]};
  double u[3];
  ray_direction(T.cl[lane], T.sl[lane], T.cg[warp], T.sg[warp], V.R, u);
  RefWalk w;
  if (!ref_setup(G.mh, G.n, M, u, w)) return;
  const double *cin = PJ ? xin + fbase : nullptr;
  double *cout = PJ ? nullptr : xout + fbase;
  double acc = PJ ? xout[po] : 0.0;
  const double yv = PJ ? 0.0 : xin[po];
  double ac = w.amin;
  int guard = G.n[0] + G.n[1] + G.n[2] + 8;
  SunWindow win = {0, 0};
  if (SUN) win = sun_window(M, u);

  // The first step in the reference's own comparisons (a distance may come out
  // of the set-up negative or as NaN); `later` and `v` are its product's factors.
  bool walks = w.iv[0] >= 0 && w.iv[0] < G.n[0] && w.iv[1] >= 0 && w.iv[1] < G.n[1] && w.iv[2] >= 0 &&
               w.iv[2] < G.n[2];
  if (!walks || (SUN && !ref_outside_sun(M, u, ac))) return;
  double dmin = w.D[0];
  if (w.D[1] < dmin) dmin = w.D[1];
  if (w.D[2] < dmin) dmin = w.D[2];
  if (dmin != dmin) return;
  long long off = (long long)w.iv[0] * G.ms[0] + (long long)w.iv[1] * G.ms[1] + (long long)w.iv[2] * G.ms[2];
  const long long st[3] = {w.upd[0] * (long long)G.ms[0], w.upd[1] * (long long)G.ms[1],
                           w.upd[2] * (long long)G.ms[2]};
  bool bits = true;  // distances comparable by their bit patterns from here on
#pragma unroll
  for (int k = 0; k < 3; ++k) bits = bits && w.D[k] == w.D[k] && w.pabs[k] == w.pabs[k];
  double later = 0.0, v = 0.0;
  for (bool first = true; guard-- > 0; first = false) {
    if (!first) {
      if (!((unsigned)w.iv[0] < (unsigned)G.n[0] && (unsigned)w.iv[1] < (unsigned)G.n[1] &&
            (unsigned)w.iv[2] < (unsigned)G.n[2]))
        break;
      if (SUN && win.test(ac) && !ref_outside_sun(M, u, ac)) break;
      if (bits) {
        long long m = __double_as_longlong(w.D[0]);
        m = min(m, __double_as_longlong(w.D[1]));
        m = min(m, __double_as_longlong(w.D[2]));
        dmin = __longlong_as_double(m);
      } else {
        dmin = w.D[0];
        if (w.D[1] < dmin) dmin = w.D[1];
        if (w.D[2] < dmin) dmin = w.D[2];
        if (dmin != dmin) break;
      }
    }
    if (SUN) ac = __dadd_rn(ac, dmin);
    if (PJ) {
      const double next = cin[off];
      if (!first) acc = __dadd_rn(acc, __dmul_rn(later, v));
      later = dmin;
      v = next;
    } else {
      atomicAdd(cout + off, __dmul_rn(dmin, yv));
    }
    bool hit[3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
      hit[k] = (bits && !first) ? __double_as_longlong(w.D[k]) == __double_as_longlong(dmin) : w.D[k] == dmin;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      if (hit[k]) {
        w.iv[k] += w.upd[k];
        off += st[k];
        w.D[k] = w.pabs[k];
      } else {
        w.D[k] = __dsub_rn(w.D[k], dmin);
      }
    }
  }
  if (PJ) xout[po] = __dadd_rn(acc, __dmul_rn(later, v));
}

// Unit vectors of the pixel rays in the arithmetic of C type CT (float or
// double): angles and rotation in CT, cosines / sines in double
// (tomograpy/C_siddon.c.template:618-648,1013-1046).  NaN data pixels are left
// untouched.
template <typename CT>
__device__ __forceinline__ void ct_direction(const tg_image_header &V, int i, int j, CT u0[3]) {
  const CT s0 = (CT)V.crpix[0], p0 = (CT)V.cdelt[0], v0 = (CT)V.crval[0];
  const CT s1 = (CT)V.crpix[1], p1 = (CT)V.cdelt[1], v1 = (CT)V.crval[1];
  const CT gam = ((CT)(unsigned int)i - s0 + (CT)1) * p0 + v0;
  const CT lam = ((CT)(unsigned int)j - s1 + (CT)1) * p1 + v1;
  CT u2[3];
  u2[0] = (CT)(cos((double)lam) * cos((double)gam));
  u2[1] = (CT)(cos((double)lam) * sin((double)gam));
  u2[2] = (CT)sin((double)lam);
#pragma unroll
  for (int k = 0; k < 3; ++k)
    u0[k] = (CT)V.R[3 * k] * u2[0] + (CT)V.R[3 * k + 1] * u2[1] + (CT)V.R[3 * k + 2] * u2[2];
}

template <typename CT>
__global__ void unit_vector_kernel(const Geometry G, const CT *__restrict__ data, double *__restrict__ u,
                                   long long us0, long long us1, long long us2, long long us3) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = blockIdx.y;
  const int t = G.view0 + blockIdx.z;
  if (i >= G.n1 || j >= G.n2) return;
  const CT v = data[(long long)i * G.ds[0] + (long long)j * G.ds[1] + (long long)t * G.ds[2]];
  if (v != v) return;
  CT u0[3];
  ct_direction<CT>(G.views[t], i, j, u0);
  const long long o = (long long)i * us0 + (long long)j * us1 + (long long)t * us2;
#pragma unroll
  for (int k = 0; k < 3; ++k) u[o + k * us3] = (double)u0[k];
}

template <typename CT>
__global__ void intersection_kernel(const Geometry G, const double *__restrict__ u, double *__restrict__ a1,
                                    double *__restrict__ an, long long us0, long long us1, long long us2,
                                    long long us3) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = blockIdx.y;
  const int t = G.view0 + blockIdx.z;
  if (i >= G.n1 || j >= G.n2) return;
  const tg_image_header &V = G.views[t];
  const long long o = (long long)i * us0 + (long long)j * us1 + (long long)t * us2;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const CT uk = (CT)u[o + k * us3];
    const CT Mk = (CT)V.M[k];
    CT b1, bn;
    if (uk != (CT)0) {
      b1 = ((CT)G.mh.mmin[k] - Mk) / uk;
      bn = ((CT)G.mh.mmax[k] - Mk) / uk;
    } else {
      b1 = -(CT)kRefInf;
      bn = (CT)kRefInf;
    }
    a1[o + k * us3] = (double)b1;
    an[o + k * us3] = (double)bn;
  }
}

cudaError_t launch_ref_f64(const Geometry &G, int mode, int obstacle, double *data, double *map, int rows, int gx,
                           int gy, int gz, cudaStream_t s) {
  dim3 grid(gx, gy, gz), block(32 * rows);
  const bool sun = obstacle == TG_OBSTACLE_SUN;
  switch (mode) {
  case TG_PJ:
    if (sun) ref64_kernel<TG_PJ, true><<<grid, block, 0, s>>>(G, map, data);
    else ref64_kernel<TG_PJ, false><<<grid, block, 0, s>>>(G, map, data);
    break;
  case TG_BPJ:
    if (sun) ref64_kernel<TG_BPJ, true><<<grid, block, 0, s>>>(G, data, map);
    else ref64_kernel<TG_BPJ, false><<<grid, block, 0, s>>>(G, data, map);
    break;
  case TG_PJT:
    if (sun) ref64_kernel<TG_PJT, true><<<grid, block, 0, s>>>(G, map, data);
    else ref64_kernel<TG_PJT, false><<<grid, block, 0, s>>>(G, map, data);
    break;
  default:
    if (sun) ref64_kernel<TG_BPJT, true><<<grid, block, 0, s>>>(G, data, map);
    else ref64_kernel<TG_BPJT, false><<<grid, block, 0, s>>>(G, data, map);
    break;
  }
  return cudaGetLastError();
}

cudaError_t launch_unit_vector(const Geometry &G, int ctype_f64, const void *data, double *u,
                               const long long us[4], int gx, int gy, int gz, cudaStream_t s) {
  dim3 grid(gx, gy, gz), block(128);
  if (ctype_f64)
    unit_vector_kernel<double><<<grid, block, 0, s>>>(G, (const double *)data, u, us[0], us[1], us[2], us[3]);
  else
    unit_vector_kernel<float><<<grid, block, 0, s>>>(G, (const float *)data, u, us[0], us[1], us[2], us[3]);
  return cudaGetLastError();
}

cudaError_t launch_intersection_parameters(const Geometry &G, int ctype_f64, const double *u,
                                           const long long us[4], double *a1, double *an, int gx, int gy,
                                           int gz, cudaStream_t s) {
  dim3 grid(gx, gy, gz), block(128);
  if (ctype_f64)
    intersection_kernel<double><<<grid, block, 0, s>>>(G, u, a1, an, us[0], us[1], us[2], us[3]);
  else
    intersection_kernel<float><<<grid, block, 0, s>>>(G, u, a1, an, us[0], us[1], us[2], us[3]);
  return cudaGetLastError();
}

}  // namespace tg
