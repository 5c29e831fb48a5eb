// Packed multi-job launches: many independent reconstructions (each with its
// own cube size, view count, image size and geometry) traced by ONE kernel
// launch, and the per-job (segmented) vector kernels of a batched CG.
//
// A plan is a device buffer holding the first CTA tile of every job (int64,
// ascending) followed by one PackedJob record per job (the job's kernel
// Geometry and its data / cube pointers), sorted by decreasing work.  A CTA
// finds its job by binary search on the compact tile array, copies the job's
// record into shared memory and runs the same tile body as the single-job
// kernel.
#include "packed_kernel.cuh"

namespace tg {

template <int MODE, typename IDX, int RPW, bool DET>
static void launch_packed_rpw(const long long *tile0, const PackedJob *jobs, int n_jobs, long long tiles, bool sun,
                              unsigned char *ws, cudaStream_t s) {
  if (sun) packed_kernel<MODE, true, IDX, RPW, DET><<<(unsigned)tiles, kThreads, 0, s>>>(tile0, jobs, n_jobs, ws);
  else packed_kernel<MODE, false, IDX, RPW, DET><<<(unsigned)tiles, kThreads, 0, s>>>(tile0, jobs, n_jobs, ws);
}

template <int MODE, typename IDX, bool DET = false>
static void launch_packed_mode(const long long *tile0, const PackedJob *jobs, int n_jobs, long long tiles, int rpw,
                               bool sun, cudaStream_t s, unsigned char *ws = nullptr) {
  if (rpw == 1) launch_packed_rpw<MODE, IDX, 1, DET>(tile0, jobs, n_jobs, tiles, sun, ws, s);
  else if (rpw == 2) launch_packed_rpw<MODE, IDX, 2, DET>(tile0, jobs, n_jobs, tiles, sun, ws, s);
  else launch_packed_rpw<MODE, IDX, 4, DET>(tile0, jobs, n_jobs, tiles, sun, ws, s);
}

// Deterministic packed backprojection, per job (blockIdx.y): max |y|, scale,
// and the final scaled add of the accumulator into the job's cube.
constexpr int kDetBlocks = 64;  // blocks per job of the prepass / finalize

__global__ void packed_det_prepass(const PackedJob *__restrict__ jobs, unsigned char *__restrict__ ws) {
  const PackedJob &J = jobs[blockIdx.y];
  det_prepass_range(J.G, J.data, J.G.n_views, reinterpret_cast<DetScale *>(ws + J.ws_off),
                    blockIdx.x * (long long)blockDim.x + threadIdx.x, (long long)gridDim.x * blockDim.x);
}

__global__ void packed_det_scale(const PackedJob *__restrict__ jobs, int n_jobs, unsigned char *__restrict__ ws) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n_jobs) return;
  const PackedJob &J = jobs[k];
  det_scale(reinterpret_cast<DetScale *>(ws + J.ws_off), J.rays, J.lmax);
}

__global__ void packed_det_finalize(const PackedJob *__restrict__ jobs, unsigned char *__restrict__ ws) {
  const PackedJob &J = jobs[blockIdx.y];
  det_finalize_range(J.G, reinterpret_cast<const long long *>(ws + J.ws_off + 256),
                     reinterpret_cast<const DetScale *>(ws + J.ws_off), J.cube,
                     blockIdx.x * (long long)blockDim.x + threadIdx.x, (long long)gridDim.x * blockDim.x);
}

size_t packed_records_offset(int n_jobs) { return packed_records_offset_of(n_jobs); }

cudaError_t launch_packed(const void *plan, int n_jobs, long long tiles, int rpw, bool idx64, int mode, int obstacle,
                          int lane_axis, int batch, cudaStream_t s) {
  const long long *tile0 = (const long long *)plan;
  const PackedJob *jobs = (const PackedJob *)((const unsigned char *)plan + packed_records_offset(n_jobs));
  const bool sun = obstacle == TG_OBSTACLE_SUN;
  if (lane_axis != 1 || batch != 0)  // the plan builder keeps 64-bit plans on the default schedule
    return launch_packed_tuned(tile0, jobs, n_jobs, tiles, rpw, mode, sun, lane_axis, batch, s);
  if (idx64) {
    switch (mode) {
    case TG_PJ: launch_packed_mode<TG_PJ, long long>(tile0, jobs, n_jobs, tiles, rpw, sun, s); break;
    case TG_BPJ: launch_packed_mode<TG_BPJ, long long>(tile0, jobs, n_jobs, tiles, rpw, sun, s); break;
    case TG_PJT: launch_packed_mode<TG_PJT, long long>(tile0, jobs, n_jobs, tiles, rpw, sun, s); break;
    default: launch_packed_mode<TG_BPJT, long long>(tile0, jobs, n_jobs, tiles, rpw, sun, s); break;
    }
  } else {
    switch (mode) {
    case TG_PJ: launch_packed_mode<TG_PJ, int>(tile0, jobs, n_jobs, tiles, rpw, sun, s); break;
    case TG_BPJ: launch_packed_mode<TG_BPJ, int>(tile0, jobs, n_jobs, tiles, rpw, sun, s); break;
    case TG_PJT: launch_packed_mode<TG_PJT, int>(tile0, jobs, n_jobs, tiles, rpw, sun, s); break;
    default: launch_packed_mode<TG_BPJT, int>(tile0, jobs, n_jobs, tiles, rpw, sun, s); break;
    }
  }
  return cudaGetLastError();
}

cudaError_t launch_packed_det(const void *plan, int n_jobs, long long tiles, int rpw, bool idx64, bool four_d,
                              int obstacle, void *workspace, size_t ws_bytes, cudaStream_t s) {
  const long long *tile0 = (const long long *)plan;
  const PackedJob *jobs = (const PackedJob *)((const unsigned char *)plan + packed_records_offset(n_jobs));
  unsigned char *ws = (unsigned char *)workspace;
  const bool sun = obstacle == TG_OBSTACLE_SUN;
  cudaError_t e = cudaMemsetAsync(workspace, 0, ws_bytes, s);
  if (e != cudaSuccess) return e;
  packed_det_prepass<<<dim3(kDetBlocks, n_jobs), 256, 0, s>>>(jobs, ws);
  packed_det_scale<<<(n_jobs + 127) / 128, 128, 0, s>>>(jobs, n_jobs, ws);
  if (idx64) {
    if (four_d) launch_packed_mode<TG_BPJT, long long, true>(tile0, jobs, n_jobs, tiles, rpw, sun, s, ws);
    else launch_packed_mode<TG_BPJ, long long, true>(tile0, jobs, n_jobs, tiles, rpw, sun, s, ws);
  } else {
    if (four_d) launch_packed_mode<TG_BPJT, int, true>(tile0, jobs, n_jobs, tiles, rpw, sun, s, ws);
    else launch_packed_mode<TG_BPJ, int, true>(tile0, jobs, n_jobs, tiles, rpw, sun, s, ws);
  }
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  packed_det_finalize<<<dim3(kDetBlocks, n_jobs), 256, 0, s>>>(jobs, ws);
  return cudaGetLastError();
}

size_t packed_job_bytes() { return sizeof(PackedJob); }

void packed_fill(void *dst, const Geometry &G, float *data, float *cube, long long tile0, int gx, int gy,
                 long long ws_off) {
  PackedJob *J = (PackedJob *)dst;
  J->G = G;
  J->data = data;
  J->cube = cube;
  J->tile0 = tile0;
  J->gx = gx;
  J->gy = gy;
  J->ws_off = ws_off;
  det_acc_strides(G, J->acc_ms);
  J->rays = (double)G.n1 * G.n2 * G.n_views;
  J->lmax = det_lmax(G);
}

// ---------------------------------------------------------------------------
// segmented vector kernels of the batched CG: segment s = [seg[2s], seg[2s+1])

// What bounds them: memory, and in the inner products the FP64 pipe (two
// conversions and a multiply-add per element; 64 cycles of an SM per warp, as
// tg_dot_f32 on 1216 CTAs shows too).  Every
// thread takes four consecutive elements at a time (one 16-byte access per
// vector where the segment's start allows it).  The updates take as many
// blocks as fill the GPU.  An inner product has 32 partials per segment, each
// the sum of 8 parts.  Where few segments would leave the GPU empty, a CTA
// computes one part (wide: so that one segment reaches all SMs), else all parts
// of a partial in turn; the sums are formed in the same order either way, so a
// segment's result depends on its length only.  The parts go through the
// caller's workspace: a kernel of its own adds them anyway, and the end of the
// first launch is all the ordering they need.  Measured on GB300, one segment
// of 64^3 / 256^3 elements, us before -> after: inner product 11.4 -> 8.0 /
// 527 -> 115 (107 of FP64), x and r 12.6 -> 7.0 / 1824 -> 62, p 8.8 -> 8.0 /
// 934 -> 30, lam term 6.8 -> 1.9 / 911 -> 26; the whole solve of 4 iterations at
// 64^3 x 60 x 128^2 1357 -> 1289.
constexpr int kSegBlocks = 32;  // partials of an inner product per segment
constexpr int kSegParts = 8;    // parts of a partial
// Segments from which a CTA takes all parts of a partial: a wide launch is 256
// CTAs per segment, most of them empty for small segments (+1.1 us each), and
// their workspace eight times as large.  Wide / not, us: 1 segment of 32^3 5.2 /
// 24, of 128^3 18 / 68; 15 segments of 32^3 17.5 / 43, of 64^3 63 / 80.
constexpr int kSegMany = 16;
constexpr int kSegThreads = 256;

// blocks per segment of the updates
static int seg_update_blocks(int n_seg) {
  const int b = 8 * 152 / n_seg;
  return b < kSegBlocks ? kSegBlocks : b;
}

__device__ __forceinline__ bool aligned16(const void *p) { return ((uintptr_t)p & 15u) == 0; }

// elements i .. i + 3 of a vector of n (zeros behind its end)
__device__ __forceinline__ float4 load4(const float *__restrict__ p, long long i, long long n, bool vec) {
  if (vec && i + 4 <= n) return *reinterpret_cast<const float4 *>(p + i);
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (i < n) v.x = p[i];
  if (i + 1 < n) v.y = p[i + 1];
  if (i + 2 < n) v.z = p[i + 2];
  if (i + 3 < n) v.w = p[i + 3];
  return v;
}

__device__ __forceinline__ void store4(float *__restrict__ p, long long i, long long n, bool vec, float4 v) {
  if (vec && i + 4 <= n) {
    *reinterpret_cast<float4 *>(p + i) = v;
    return;
  }
  if (i < n) p[i] = v.x;
  if (i + 1 < n) p[i + 1] = v.y;
  if (i + 2 < n) p[i + 2] = v.z;
  if (i + 3 < n) p[i + 3] = v.w;
}

__device__ __forceinline__ double dot4(float4 a, float4 b, double acc) {
  acc = fma((double)a.x, (double)b.x, acc);
  acc = fma((double)a.y, (double)b.y, acc);
  acc = fma((double)a.z, (double)b.z, acc);
  return fma((double)a.w, (double)b.w, acc);
}

// Share b of segment s is the b-th of 32 interleaved ones.  WIDE: a CTA per
// part, partial[(s * 32 + b) * 8 + q] = part q; else a CTA per share,
// partial[s * 32 + b] = the sum of its parts (float64).
template <bool WIDE>
__global__ void __launch_bounds__(kSegThreads) seg_dot_partial(const float *__restrict__ a,
                                                               const float *__restrict__ b,
                                                               const long long *__restrict__ off,
                                                               double *__restrict__ partial) {
  __shared__ double sh[kSegThreads / 32];
  const int s = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long lo = off[2 * s], n = off[2 * s + 1] - lo;
  a += lo;
  b += lo;
  const bool va = aligned16(a), vb = aligned16(b);
  const int share = WIDE ? blockIdx.x / kSegParts : blockIdx.x;
  const int q0 = WIDE ? blockIdx.x % kSegParts : 0, q1 = WIDE ? q0 + 1 : kSegParts;
  const long long step = 4LL * kSegThreads * kSegParts * kSegBlocks;
  double sum = 0.0;
  for (int q = q0; q < q1; ++q) {
    const long long first = 4LL * kSegThreads * (share * kSegParts + q);
    double v = 0.0;
    if (first < n) {  // uniform over the CTA
      double w = 0.0;
      for (long long i = first + 4 * threadIdx.x; i < n; i += 2 * step) {
        const float4 x0 = load4(a, i, n, va), y0 = load4(b, i, n, vb);
        const float4 x1 = load4(a, i + step, n, va), y1 = load4(b, i + step, n, vb);
        v = dot4(x0, y0, v);
        w = dot4(x1, y1, w);
      }
      v += w;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      __syncthreads();
      if (lane == 0) sh[warp] = v;
      __syncthreads();
      v = lane < kSegThreads / 32 ? sh[lane] : 0.0;
#pragma unroll
      for (int o = kSegThreads / 64; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    }
    sum = q == q0 ? v : sum + v;
  }
  if (threadIdx.x == 0) partial[s * (long long)gridDim.x + blockIdx.x] = sum;
}

// out[s] = sum of segment s's partials, one warp per segment in a fixed order
template <bool WIDE>
__global__ void seg_dot_final(const double *__restrict__ partial, int n_seg, double *__restrict__ out) {
  static_assert(kSegBlocks == 32, "one partial per lane");
  const int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (s >= n_seg) return;
  double v;
  if (WIDE) {
    const double *part = partial + ((long long)s * kSegBlocks + lane) * kSegParts;
    v = part[0];
#pragma unroll
    for (int q = 1; q < kSegParts; ++q) v += part[q];
  } else {
    v = partial[(long long)s * kSegBlocks + lane];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (lane == 0) out[s] = v;
}

// x += alpha_s p, r -= alpha_s Ap with alpha_s = rr_s / pAp_s
__global__ void __launch_bounds__(kSegThreads) seg_cg_x(float *__restrict__ x, float *__restrict__ r,
                                                        const float *__restrict__ p, const float *__restrict__ Ap,
                                                        const double *__restrict__ rr,
                                                        const double *__restrict__ pAp,
                                                        const long long *__restrict__ off) {
  const int s = blockIdx.y;
  const double den = pAp[s];
  const float alpha = (den != 0.0) ? (float)(rr[s] / den) : 0.f;
  const long long lo = off[2 * s], n = off[2 * s + 1] - lo;
  x += lo, r += lo, p += lo, Ap += lo;
  const bool vec = aligned16(x) && aligned16(r) && aligned16(p) && aligned16(Ap);
  for (long long i = 4LL * ((long long)blockIdx.x * kSegThreads + threadIdx.x); i < n;
       i += 4LL * kSegThreads * gridDim.x) {
    const float4 vp = load4(p, i, n, vec), va = load4(Ap, i, n, vec);
    float4 vx = load4(x, i, n, vec), vr = load4(r, i, n, vec);
    vx.x = fmaf(alpha, vp.x, vx.x), vx.y = fmaf(alpha, vp.y, vx.y);
    vx.z = fmaf(alpha, vp.z, vx.z), vx.w = fmaf(alpha, vp.w, vx.w);
    vr.x = fmaf(-alpha, va.x, vr.x), vr.y = fmaf(-alpha, va.y, vr.y);
    vr.z = fmaf(-alpha, va.z, vr.z), vr.w = fmaf(-alpha, va.w, vr.w);
    store4(x, i, n, vec, vx);
    store4(r, i, n, vec, vr);
  }
}

// p = r + beta_s p with beta_s = rr_new_s / rr_s
__global__ void __launch_bounds__(kSegThreads) seg_cg_p(float *__restrict__ p, const float *__restrict__ r,
                                                        const double *__restrict__ rr,
                                                        const double *__restrict__ rr_new,
                                                        const long long *__restrict__ off) {
  const int s = blockIdx.y;
  const double den = rr[s];
  const float beta = (den != 0.0) ? (float)(rr_new[s] / den) : 0.f;
  const long long lo = off[2 * s], n = off[2 * s + 1] - lo;
  p += lo, r += lo;
  const bool vec = aligned16(p) && aligned16(r);
  for (long long i = 4LL * ((long long)blockIdx.x * kSegThreads + threadIdx.x); i < n;
       i += 4LL * kSegThreads * gridDim.x) {
    const float4 vr = load4(r, i, n, vec);
    float4 v = load4(p, i, n, vec);
    v.x = fmaf(beta, v.x, vr.x), v.y = fmaf(beta, v.y, vr.y);
    v.z = fmaf(beta, v.z, vr.z), v.w = fmaf(beta, v.w, vr.w);
    store4(p, i, n, vec, v);
  }
}

// y[i] = alpha * x[i] + beta * y[i] over the segments (beta = 0: y = alpha x)
__global__ void __launch_bounds__(kSegThreads) seg_axpby(float *__restrict__ y, const float *__restrict__ x, float alpha,
                                                         float beta, const long long *__restrict__ off) {
  const int s = blockIdx.y;
  const long long lo = off[2 * s], n = off[2 * s + 1] - lo;
  y += lo;
  if (x) x += lo;
  const bool vec = aligned16(y) && aligned16(x);
  for (long long i = 4LL * ((long long)blockIdx.x * kSegThreads + threadIdx.x); i < n;
       i += 4LL * kSegThreads * gridDim.x) {
    const float4 vx = x ? load4(x, i, n, vec) : make_float4(0.f, 0.f, 0.f, 0.f);
    float4 v;
    if (beta == 0.f) {
      v = x ? make_float4(alpha * vx.x, alpha * vx.y, alpha * vx.z, alpha * vx.w) : vx;
    } else {
      v = load4(y, i, n, vec);
      v = make_float4(fmaf(alpha, vx.x, beta * v.x), fmaf(alpha, vx.y, beta * v.y), fmaf(alpha, vx.z, beta * v.z),
                      fmaf(alpha, vx.w, beta * v.w));
    }
    store4(y, i, n, vec, v);
  }
}

cudaError_t launch_seg_axpby(float *y, const float *x, float alpha, float beta, const long long *off, int n_seg,
                             cudaStream_t st) {
  seg_axpby<<<dim3(seg_update_blocks(n_seg), n_seg), kSegThreads, 0, st>>>(y, x, alpha, beta, off);
  return cudaGetLastError();
}

__global__ void seg_copy(double *__restrict__ dst, const double *__restrict__ src, int n) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s < n) dst[s] = src[s];
}

cudaError_t launch_seg_dot(const float *a, const float *b, const long long *off, int n_seg, double *partial,
                           size_t bytes, double *out, cudaStream_t st) {
  const unsigned blocks = (unsigned)(n_seg + 3) / 4;
  if (n_seg < kSegMany && bytes >= seg_workspace_bytes(n_seg)) {
    seg_dot_partial<true><<<dim3(kSegBlocks * kSegParts, n_seg), kSegThreads, 0, st>>>(a, b, off, partial);
    seg_dot_final<true><<<blocks, 128, 0, st>>>(partial, n_seg, out);
  } else {
    seg_dot_partial<false><<<dim3(kSegBlocks, n_seg), kSegThreads, 0, st>>>(a, b, off, partial);
    seg_dot_final<false><<<blocks, 128, 0, st>>>(partial, n_seg, out);
  }
  return cudaGetLastError();
}

cudaError_t launch_seg_cg_x(float *x, float *r, const float *p, const float *Ap, const double *rr, const double *pAp,
                            const long long *off, int n_seg, cudaStream_t st) {
  seg_cg_x<<<dim3(seg_update_blocks(n_seg), n_seg), kSegThreads, 0, st>>>(x, r, p, Ap, rr, pAp, off);
  return cudaGetLastError();
}

cudaError_t launch_seg_cg_p(float *p, const float *r, double *rr, const double *rr_new, const long long *off,
                            int n_seg, cudaStream_t st) {
  seg_cg_p<<<dim3(seg_update_blocks(n_seg), n_seg), kSegThreads, 0, st>>>(p, r, rr, rr_new, off);
  seg_copy<<<(n_seg + 127) / 128, 128, 0, st>>>(rr, rr_new, n_seg);
  return cudaGetLastError();
}

size_t seg_workspace_least(int n_seg) { return (size_t)n_seg * kSegBlocks * sizeof(double); }
size_t seg_workspace_bytes(int n_seg) { return seg_workspace_least(n_seg) * (n_seg < kSegMany ? kSegParts : 1); }

}  // namespace tg
