// Row walk: the fast walk for views whose image axis 1 (lambda) runs along the
// cube's axis 2, i.e. whose rotation matrix has R[0][2] = R[1][2] = 0 (an
// observer in the equatorial plane, no roll).
//
// Directions are w = A_row + tan(lambda) R[:, 2] (siddon_fast.cuh), so in such
// a view all rays of an image row have the same w_x and w_y: they cross the
// planes of axes 0 and 1 at the same parameters and pass the same (x, y) cells;
// only their position along axis 2 differs, and over the cube they cross a few
// planes of that axis (|w_z| is the pixel's angle from the row's centre).
// The general walk spends ~19 instructions per voxel on each ray's own
// three-way merge of crossings and is bound by instruction issue.  Here a
// warp, 32 neighbouring rays of one row, does
//  * once per row of the tile (row_setup, one lane per row): entry into the
//    (x, y) rectangle, first crossings and spacings of the two families, in
//    double-float as in the general set-up;
//  * once per ray (row_ray): its interval inside the cube, its obstacle stop
//    and its crossings of axis 2.  Parts of row segments at the ray's ends are
//    added at once; in between it has a run of whole row segments, along which
//    its z changes at a few "cuts", the segments that hold a plane of axis 2:
//    their parts are added at once too, and the run leaves them out;
//  * for 32 row segments at a time: each lane computes one segment of the
//    merged (x, y) path in closed form (length and cell offset, to shared
//    memory), then all lanes walk the 32 segments together in two groups: per
//    segment half a 16-byte broadcast read, a compare and a predicated move of
//    the offset along axis 2, one address, one gather and one FMA (or one
//    product and one red), which leaves out the cut.
// All lanes are in the same (x, y) cell at a time, so a gather touches one run
// of axis 2: 2.9 sectors per request at 256^3 x 512^2, where the general
// walk's lanes drift apart with their numbers of plane crossings (4.6).
//
// Measured on GB300 at 256^3 x 360 x 512^2, sun, general walk -> row walk:
// projection 15.73 -> 12.47 ms (1.08e9 warp-instructions per 36 views against
// 1.53e9; bound by issue, 68 % active, and the gathers' latency),
// backprojection 18.07 -> 14.75 ms (bound by the L2's red traffic: 5.4 sectors
// per request, since two rays in one voxel take two passes);
// 128^3 x 28 frames x 784 x 256^2: 5.59 -> 4.41 and 6.44 -> 4.79 ms.  Of the
// projection's time 0.2 ms are the parts of cut segments, 0.25 the low words of
// axis 2, 0.3 the short rays and 0.1 the entry's cells.
// Groups of 8 / 16 / 32 segments between looks at the cuts, on a form with whole
// cut segments: projection 14.35 / 11.95 / 15.18 ms (16: the gathers of a group
// are in flight together; 32 spill).
// Slower than the general walk where planes of axis 2 are close together (below
// 20 row segments a plane: 32 x 32 x 512, 90 x 192^2, projection 216 -> 264 us):
// several cuts in a group are walked segment by segment.  Kept there as well,
// for its exact lengths: a path of 1e-3 radii behind a plane is 4e-6 off on the
// general walk, below 1e-6 here.
#pragma once

namespace tg {

// Planes of axis 2 that a ray of the row walk may cross.  Each costs ~50
// instructions beside the walk, about three voxels of the general walk, and
// its cut list lives in shared memory; rows whose bound (row_setup) is above
// it take the general walk.
constexpr int kRowCross = 8;
constexpr int kRowWin = 32;                // row segments listed at a time
#ifndef TG_ROW_GROUP
#define TG_ROW_GROUP 16
#endif
constexpr int kRowGroup = TG_ROW_GROUP;    // segments between looks at the cuts
constexpr int kRowNever = 0xffff;          // no cut / no segment
constexpr float kRowBig = 1e30f;           // crossing of a family that the row never crosses

enum RowMode { kRowGeneral = 0, kRowWalk = 1, kRowMiss = 2 };

// Per row of the tile.  Crossing i of a family (0: the first one after the
// entry) is at fma(i - m0, p, d), measured from the row's chord midpoint, as in
// Walk; the cell after i crossings is entry + i.
struct RowTables {
  int mode[kFastRows];
  int off0[kFastRows];                       // entry cell's offset
  int iv[2][kFastRows];                      // entry cell
  float p[2][kFastRows], d[2][kFastRows], m0[2][kFastRows];
  float ip[2][kFastRows];                    // 1 / p
  float top[2][kFastRows];                   // cells ahead of the entry cell
  float q1[kFastRows], q0[kFastRows];        // cell of segment r: floor((r + 1) q1 + q0)
  float h[kFastRows], texit[kFastRows];      // half chord, exit parameter
  // first crossing from the entry (hi + lo) and the spacing's low word, for
  // rays that take an origin of their own
  float dh[2][kFastRows], dl[2][kFastRows], pl[2][kFastRows];
  float bh[kFastRows], bl[kFastRows];        // entry parameter, double-float
  float e[2][kFastRows];                     // entry point
};

struct RowShared {
  RowTables R;
  int4 list[kRows][kRowWin / 2];             // per warp, two segments each: (length, cell offset)
  unsigned short ev[kRows][kRowCross + 2][32];  // per ray: its cuts, kRowNever twice
};

__device__ __forceinline__ bool df_less(df a, df b) { return a.hi < b.hi || (a.hi == b.hi && a.lo < b.lo); }

// Bound of the double-float arithmetic's error (2^-45 per operation), relative
// to the terms that are added: rows that it cannot tell from a miss or from an
// entry at an edge take the general walk, which decides in double precision.
constexpr float kRowTol = 3.6e-12f;  // 2^-38

// Crossing i of family k of the row, as the walk computes it.
__device__ __forceinline__ float row_cross(float i, float m0, float p, float d) { return fmaf(i - m0, p, d); }

// Set-up of one row of the tile by one lane.  zmax: bound of |tan lambda| over
// the image (not the tile, so that a ray's walk does not depend on the tile
// that traces it).
__device__ __forceinline__ void row_setup(const Geometry &G, const tg_image_header &V, const FastTables &T, int slot,
                                          float zmax, RowTables &R) {
  int mode = kRowWalk;
  df wd[2], inv[2], bin = {-3e38f, 0.f}, bout = {3e38f, 0.f};
  int upd[2], kin = -1;
  df ain[2] = {};
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    wd[k] = {T.ah[slot][k], T.al[slot][k]};
    upd[k] = (wd[k].hi >= 1e-14f) ? 1 : ((wd[k].hi <= -1e-14f) ? -1 : 0);
    inv[k] = {0.f, 0.f};
    if (upd[k]) {
      inv[k] = df_rcp(wd[k]);
      const int in = upd[k] > 0 ? 0 : 1;
      const df a = df_mul({T.fh[k][in], T.fl[k][in]}, inv[k]);
      const df b = df_mul({T.fh[k][1 - in], T.fl[k][1 - in]}, inv[k]);
      ain[k] = a;
      if (kin < 0 || df_less(bin, a)) {
        bin = a;
        kin = k;
      }
      if (df_less(b, bout)) bout = b;
    }
  }
  const float tol = kRowTol * (fabsf(bin.hi) + fabsf(bout.hi));
  if (kin < 0) mode = kRowGeneral;                       // a ray along axis 2
  else if (fabsf(df_add(bout, {-bin.hi, -bin.lo}).hi) <= tol) mode = kRowGeneral;
  else if (!df_less(bin, bout)) mode = kRowMiss;
  else if (upd[0] && upd[1] && fabsf(df_add(ain[0], {-ain[1].hi, -ain[1].lo}).hi) <= tol) mode = kRowGeneral;
  float dk[2], pk[2], dl[2], pl[2], ce[2];
  int iv[2];
  float texit0 = kRowBig;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const df C = {G.cdeltf[k], G.cdeltl[k]};
    const df iaw = upd[k] < 0 ? df{-inv[k].hi, -inv[k].lo} : inv[k];
    const df pd = df_mul(C, iaw);
    pk[k] = pd.hi;
    pl[k] = pd.lo;
    if (upd[k] == 0) {
      // in the plane: the index holds for the whole chord (as in setup_ray)
      const double ep = __dsub_rn(V.M[k], G.mh.mmin[k]);
      iv[k] = ref_utrunc(__ddiv_rn(ep, G.mh.cdelt[k])) - ref_utrunc(__ddiv_rn(ep, G.mh.pshape[k]));
      R.e[k][slot] = G.mminf[k] + (float)ep;
      dk[k] = kRowBig;
      pk[k] = 2.f * kRowBig;
      dl[k] = pl[k] = 0.f;
    } else if (k == kin) {
      iv[k] = upd[k] > 0 ? 0 : G.n[k] - 1;
      R.e[k][slot] = upd[k] > 0 ? G.mminf[k] : G.mminf[k] + (float)G.mh.pshape[k];
      dk[k] = pk[k];
      dl[k] = pl[k];
    } else {
      // entry point and its voxel by a floor division against the exact plane
      // positions, remainder and first crossing in double-float (setup_ray)
      const df e = df_add({T.mh[k], T.ml[k]}, df_mul(bin, wd[k]));
      const df mC = {-C.hi, -C.lo};
      const float q = floorf((e.hi + e.lo) * G.inv_cdeltf[k]);
      const df qc = df_mul({q, 0.f}, C);
      df r = df_add(e, {-qc.hi, -qc.lo});
      int qi = (int)q;
      if (r.hi < 0.f || (r.hi == 0.f && r.lo < 0.f)) {
        qi -= 1;
        r = df_add(r, C);
      } else {
        const df rc = df_add(r, mC);
        if (rc.hi > 0.f || (rc.hi == 0.f && rc.lo >= 0.f)) {
          qi += 1;
          r = rc;
        }
      }
      if (qi == -1) {
        qi = 0;
        r = df_add(r, mC);
      } else if (qi == G.n[k]) {
        qi = G.n[k] - 1;
        r = df_add(r, C);
      }
      iv[k] = qi;
      const df dd = df_mul(upd[k] > 0 ? df_add(C, {-r.hi, -r.lo}) : r, iaw);
      dk[k] = dd.hi;
      dl[k] = dd.lo;
      R.e[k][slot] = G.mminf[k] + (e.hi + e.lo);
    }
    if (iv[k] < 0 || iv[k] >= G.n[k]) mode = mode == kRowWalk ? (int)kRowMiss : mode;
    ce[k] = (float)(upd[k] > 0 ? G.n[k] - iv[k] : (upd[k] < 0 ? iv[k] + 1 : 1));
    if (upd[k]) texit0 = fminf(texit0, fmaf(ce[k] - 1.f, pk[k], dk[k]));
  }
  // origin at the chord midpoint, crossings counted from the nearest one (setup_ray)
  const float h = 0.5f * texit0;
  float texit = kRowBig;
  float x0[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    float m0 = 0.f;
    R.dh[k][slot] = dk[k];
    R.dl[k][slot] = dl[k];
    R.pl[k][slot] = pl[k];
    if (upd[k]) {
      m0 = fminf(fmaxf(rintf(__fdividef(h - dk[k], pk[k])), 0.f), ce[k] - 1.f);
      const float p = __fmul_rn(m0, pk[k]);
      const float err = fmaf(m0, pk[k], -p) + fmaf(m0, pl[k], dl[k]);
      dk[k] = ((p - h) + dk[k]) + err;                   // the small term last: exact next to the midpoint
      texit = fminf(texit, row_cross(ce[k] - 1.f, m0, pk[k], dk[k]));
    }
    R.p[k][slot] = pk[k];
    R.d[k][slot] = dk[k];
    R.m0[k][slot] = m0;
    R.ip[k][slot] = upd[k] ? __frcp_rn(pk[k]) : 0.f;
    R.top[k][slot] = ce[k] - 1.f;
    R.iv[k][slot] = iv[k];
    x0[k] = row_cross(-1.f, m0, pk[k], dk[k]);           // the plane the entry cell was entered by
  }
  const float is = __fdividef(1.f, pk[0] + pk[1]);
  R.q1[slot] = pk[1] * is;
  R.q0[slot] = (x0[1] - x0[0]) * is;
  R.h[slot] = h;
  R.texit[slot] = texit;
  R.bh[slot] = bin.hi;
  R.bl[slot] = bin.lo;
  R.off0[slot] = iv[0] * (int)G.ms[0] + iv[1] * (int)G.ms[1];
  // planes of axis 2 that any ray of the image's row can cross
  const float wz = fabsf(T.ah[slot][2]) + zmax * fabsf(T.B[2]);
  const float drift = texit0 * wz * G.inv_cdeltf[2];
  if (mode == kRowWalk && !(drift + 0.5f < (float)kRowCross && ce[0] + ce[1] < 65000.f)) mode = kRowGeneral;
  R.mode[slot] = mode;
}

// One row's crossings in registers.
struct RowPath {
  float px, dx, mx, py, dy, my, ipx, ipy, tx, ty;  // p, d, m0 per family; 1 / p; cells ahead
  float t0;                                        // the row's entry
  int off0, sx, sy;
  __device__ __forceinline__ float cx(float i) const { return row_cross(i, mx, px, dx); }
  __device__ __forceinline__ float cy(float j) const { return row_cross(j, my, py, dy); }
  // Where cell (i, j) begins.  The cells of the entry begin at t0: crossing -1 of
  // a family is as far from the midpoint as its spacing, which can be a hundred
  // times the chord (a row that clips an edge of the cube), and rounded so.
  __device__ __forceinline__ float start(float i, float j) const {
    return fmaxf(i > 0.f ? cx(i - 1.f) : t0, j > 0.f ? cy(j - 1.f) : t0);
  }
  // cells passed at parameter t: the numbers of crossings <= t
  __device__ __forceinline__ void at(float t, float &i, float &j) const {
    i = floorf(fmaf(t - dx, ipx, mx)) + 1.f;
    j = floorf(fmaf(t - dy, ipy, my)) + 1.f;
    // the quotient is at most one off
    i += (cx(i) <= t ? 1.f : 0.f) - (cx(i - 1.f) > t ? 1.f : 0.f);
    j += (cy(j) <= t ? 1.f : 0.f) - (cy(j - 1.f) > t ? 1.f : 0.f);
    i = fminf(fmaxf(i, 0.f), tx);
    j = fminf(fmaxf(j, 0.f), ty);
  }
  __device__ __forceinline__ int cell(float i, float j) const { return off0 + (int)i * sx + (int)j * sy; }
};

// A gather / an add that only happens where `on` (predicated, so that the
// others of a group are in flight with it).
__device__ __forceinline__ float row_load_if(const float *p, bool on) {
  float v;
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %2, 0;\n\tmov.f32 %0, 0f00000000;\n\t"
               "@p ld.global.nc.f32 %0, [%1];\n\t}"
               : "=f"(v)
               : "l"(__cvta_generic_to_global(p)), "r"((int)on));
  return v;
}

// kRowGroup segments of the row: those before `cut` at offset zo along axis 2,
// those behind it at zn, and not the cut itself, whose parts row_ray adds: it
// is taken at zn, a voxel the ray passes, and a projection leaves it out of the
// sum, a backprojection adds 0 there (a predicated red for each segment costs
// 3 to 8 % of the backprojection, the select 1 to 4 %).  The projection tests
// the cut's bit: 11.8 ms at 256^3 x 360 x 512^2, 12.7 with a second compare.
// EDGE: only segments lo <= s < hi are this ray's.  A projection's gathers are
// issued before its sums.
template <int MODE, bool DET, bool EDGE>
__device__ __forceinline__ void row_group(const int4 *__restrict__ list4, int zo, int zn, int cut, int lo, int hi,
                                          const float *cin, float *cout, unsigned long long *aout, float yv, float yq,
                                          float qs, float &part) {
  constexpr bool PJ = (MODE == TG_PJ || MODE == TG_PJT);
  int4 q[kRowGroup / 2];
#pragma unroll
  for (int s = 0; s < kRowGroup / 2; ++s) q[s] = list4[s];
  int z = zo;
  float v[kRowGroup];
#pragma unroll
  for (int s = 0; s < kRowGroup; ++s) {
    if (s == cut) z = zn;
    const int o = (s & 1 ? q[s >> 1].w : q[s >> 1].y) + z;
    if (PJ) {
      if (EDGE) v[s] = row_load_if(cin + o, s >= lo && s < hi);
      else v[s] = __ldg(cin + o);
    } else if (!EDGE || (s >= lo && s < hi)) {
      accumulate<MODE, DET, int>(__int_as_float(s & 1 ? q[s >> 1].z : q[s >> 1].x), o, cin, cout, aout,
                                 s == cut ? 0.f : yv, s == cut ? 0.f : yq, qs, part);
    }
  }
  if (PJ) {
    const unsigned keep = ~((unsigned)cut < 32u ? 1u << cut : 0u);
#pragma unroll
    for (int s = 0; s < kRowGroup; ++s)
      if ((keep >> s) & 1u) part = fmaf(__int_as_float(s & 1 ? q[s >> 1].z : q[s >> 1].x), v[s], part);
  }
}

// One ray of the row: its run [js, je) of whole row segments, the voxel of
// axis 2 it starts the run in and the direction it goes there, and how many
// cuts (the segment of each plane of axis 2) its list holds.
struct RowRay {
  int js, je, z0, uz, cuts;
};

// Rays whose chord is below this fraction of their row's are measured from the
// middle of their own chord and walked alone (row_alone).  The row's parameters have their
// origin at the row's midpoint, so a crossing is rounded at 2^-24 of the row's
// half chord wherever the ray is: a ray that leaves through a face of axis 2
// soon after it entered would carry that on a short path (2e-5 of 3e-3 radii,
// 5e-6 of 1/29 of the row).  At 1/8 it is below 1e-6 of the path; four rows of
// 512 pixels in five have such a ray (256^3 x 360 x 512^2 12.36 -> 12.42 ms from
// 1/32 to 1/8).  Out of line: inlined, the second walk costs 2 to 8 % more.
constexpr float kRowShort = 1.f / 8.f;

__device__ __forceinline__ RowPath row_path(const Geometry &G, const FastTables &T, const RowTables &R, int slot) {
  RowPath P;
  P.px = R.p[0][slot], P.dx = R.d[0][slot], P.mx = R.m0[0][slot], P.ipx = R.ip[0][slot], P.tx = R.top[0][slot];
  P.py = R.p[1][slot], P.dy = R.d[1][slot], P.my = R.m0[1][slot], P.ipy = R.ip[1][slot], P.ty = R.top[1][slot];
  P.t0 = -R.h[slot];
  P.off0 = R.off0[slot];
  P.sx = T.ah[slot][0] > 0.f ? (int)G.ms[0] : -(int)G.ms[0];
  P.sy = T.ah[slot][1] > 0.f ? (int)G.ms[1] : -(int)G.ms[1];
  return P;
}

// The row's crossings measured from the point o behind its entry (row_setup
// does the same for the midpoint).
__device__ __forceinline__ void row_origin(const RowTables &R, int slot, float o, RowPath &P) {
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const float pk = k ? P.py : P.px, dh = R.dh[k][slot];
    if (pk > kRowBig) continue;                          // never crossed
    const float m0 = fminf(fmaxf(rintf(__fdividef(o - dh, pk)), 0.f), k ? P.ty : P.tx);
    const float p = __fmul_rn(m0, pk);
    const float d = ((p - o) + dh) + (fmaf(m0, pk, -p) + fmaf(m0, R.pl[k][slot], R.dl[k][slot]));
    (k ? P.dy : P.dx) = d;
    (k ? P.my : P.mx) = m0;
  }
}

template <int MODE, bool SUN, bool DET>
__device__ float row_alone(const Geometry &G, const tg_image_header &V, const FastTables &T, const RowTables &R,
                           int cidx, int slot, const float *cin, float *cout, unsigned long long *aout, float yv,
                           float yq, float qs);

// Set-up of the ray of column cidx of the CTA's tables: interval inside the
// cube, obstacle stop, crossings of axis 2 (to ev, a list with stride 32);
// what its run leaves out is added here.  False when it has no run.  Whether a
// ray enters through a face of axis 2 is decided in double-float, to 2^-45 of
// |M - MMIN| (1e-13 radii): nearer to an edge the first voxel is either one.
// ALONE: a short ray, walked here as a whole.
template <int MODE, bool SUN, bool DET, bool ALONE>
__device__ __forceinline__ bool row_ray(const Geometry &G, const tg_image_header &V, const FastTables &T,
                                        const RowTables &R, RowPath P, int cidx, int slot, const float *cin,
                                        float *cout, unsigned long long *aout, float yv, float yq, float qs,
                                        unsigned short (*ev)[32], RowRay &ray, float &acc) {
  // ---- the ray's crossings of axis 2, its interval inside the cube
  float h = R.h[slot];                                 // the origin, from the row's entry
  const df bin = {R.bh[slot], R.bl[slot]};
  df wz = df_add({T.ah[slot][2], T.al[slot][2]}, df_mul({T.th[cidx], T.tl[cidx]}, {T.B[2], T.Bl[2]}));
  float tin = -h, tend = R.texit[slot];
  float pz = 2.f * kRowBig, dz = kRowBig, mz = 0.f;    // crossing m at fma(m - mz, pz, dz)
  const auto cz = [&](float m) { return fmaf(m - mz, pz, dz); };
  float ez;                                            // z - MMIN at the row's entry
  int iz, uz = 0;
  if (fabsf(wz.hi) < 1e-14f) {
    wz = {0.f, 0.f};
    const double ep = __dsub_rn(V.M[2], G.mh.mmin[2]);
    iz = ref_utrunc(__ddiv_rn(ep, G.mh.cdelt[2])) - ref_utrunc(__ddiv_rn(ep, G.mh.pshape[2]));
    ez = (float)ep;
    if (iz < 0 || iz >= G.n[2]) return false;
  } else {
    uz = wz.hi > 0.f ? 1 : -1;
    const df C = {G.cdeltf[2], G.cdeltl[2]};
    const df e = df_add({T.mh[2], T.ml[2]}, df_mul(bin, wz));
    const df iaw = df_rcp(uz > 0 ? wz : df{-wz.hi, -wz.lo});
    const df pd = df_mul(C, iaw);
    pz = pd.hi;
    ez = e.hi + e.lo;
    df dd;                                             // first crossing, from the row's entry
    // distance to go before the entry face of axis 2 (MMIN upwards, MMAX downwards)
    const df fu = df_add({T.fh[2][1], T.fl[2][1]}, {T.mh[2], T.ml[2]});   // MMAX - MMIN
    const df gap = uz > 0 ? df{-e.hi, -e.lo} : df_add(e, {-fu.hi, -fu.lo});
    const float a = gap.hi * iaw.hi, len = 2.f * h, in = fmaxf(a, 0.f);
    const float chord = fminf(len, fmaf(fu.hi, iaw.hi, a)) - in;
    if (ALONE) {
      h = fmaf(0.5f, chord, in);
      tin = -h;
      row_origin(R, slot, h, P);
      tend = fminf(P.cx(P.tx), P.cy(P.ty));
    } else if (chord < kRowShort * len) {
      if (chord > -1e-2f * len)                        // not a clear miss
        acc = row_alone<MODE, SUN, DET>(G, V, T, R, cidx, slot, cin, cout, aout, yv, yq, qs);
      return false;
    }
    if (gap.hi > 0.f) {                                // enters through that face
      const df tf = df_mul(gap, iaw);
      iz = uz > 0 ? 0 : G.n[2] - 1;
      tin = (tf.hi - h) + tf.lo;
      dd = df_add(tf, pd);
    } else {
      const df mC = {-C.hi, -C.lo};
      const float q = floorf((e.hi + e.lo) * G.inv_cdeltf[2]);
      const df qc = df_mul({q, 0.f}, C);
      df r = df_add(e, {-qc.hi, -qc.lo});
      int qi = (int)fminf(fmaxf(q, -2.f), (float)G.n[2] + 1.f);
      if (r.hi < 0.f || (r.hi == 0.f && r.lo < 0.f)) {
        qi -= 1;
        r = df_add(r, C);
      } else {
        const df rc = df_add(r, mC);
        if (rc.hi > 0.f || (rc.hi == 0.f && rc.lo >= 0.f)) {
          qi += 1;
          r = rc;
        }
      }
      // on the entry face (the gap above decides who is outside)
      if (uz > 0 && qi == -1) {
        qi = 0;
        r = df_add(r, mC);
      } else if (uz < 0 && qi == G.n[2]) {
        qi = G.n[2] - 1;
        r = df_add(r, C);
      }
      iz = qi;
      dd = df_mul(uz > 0 ? df_add(C, {-r.hi, -r.lo}) : r, iaw);
      if (iz < 0 || iz >= G.n[2]) return false;
    }
    // counted from the crossing nearest the midpoint, as the row's
    const float left = (float)(uz > 0 ? G.n[2] - iz : iz + 1) - 1.f;
    mz = fminf(fmaxf(rintf(__fdividef(h - dd.hi, pz)), 0.f), left);
    const float p = __fmul_rn(mz, pz);
    dz = ((p - h) + dd.hi) + (fmaf(mz, pz, -p) + fmaf(mz, pd.lo, dd.lo));
    tend = fminf(tend, cz(left));
  }
  if (!(tin < tend)) return false;

  // ---- obstacle: the first voxel entry inside the sphere stops the ray.
  // Only entries within the parameter window where |r|^2 - 1 can be below
  // the decision threshold are looked at (|r|^2 - 1 = ww (s - sc)^2 -
  // disc / ww; 3e-5 covers the threshold and the float rounding of disc).
  if (SUN) {
    const float wx = T.ah[slot][0], wy = T.ah[slot][1], w2 = wz.hi;
    const float ex = R.e[0][slot], ey = R.e[1][slot], e2 = G.mminf[2] + ez;
    const float ww = fmaf(wx, wx, fmaf(wy, wy, w2 * w2));
    const float b = fmaf(ex, wx, fmaf(ey, wy, e2 * w2));
    const float c = fmaf(ex, ex, fmaf(ey, ey, e2 * e2)) - 1.f;
    const float disc = fmaf(b, b, -ww * c);
    if (disc > -2e-5f * ww) {
      const float iw = __frcp_rn(ww);
      const float hw = sqrtf(fmaf(fmaxf(disc, 0.f), iw, 3e-5f) * iw);
      const float lo = fmaf(-b, iw, -hw) - h, hi = fmaf(-b, iw, hw) - h;
      float fi, fj, m = 0.f, tc;
      if (lo <= tin) {
        tc = tin;                                      // the entry voxel is tested too
        P.at(tin, fi, fj);
      } else {
        P.at(lo, fi, fj);
        while (m < (float)kRowCross && cz(m) <= lo) m += 1.f;
        tc = min3f(P.cx(fi), P.cy(fj), cz(m));
      }
      while (tc < tend && tc <= hi) {
        if (P.cx(fi) == tc) fi += 1.f;
        if (P.cy(fj) == tc) fj += 1.f;
        if (cz(m) == tc) m += 1.f;
        const float se = tc + h;
        const float rx = fmaf(se, wx, ex), ry = fmaf(se, wy, ey), rz = fmaf(se, w2, e2);
        const float dd = fmaf(rx, rx, fmaf(ry, ry, rz * rz)) - 1.f;
        bool outside = dd > kSunTh;
        if (!outside && dd >= -kSunTh) {
          const int ivn[3] = {R.iv[0][slot] + (wx > 0.f ? (int)fi : -(int)fi),
                              R.iv[1][slot] + (wy > 0.f ? (int)fj : -(int)fj), iz + uz * (int)m};
          outside = exact_outside(G, V, T, cidx, slot, ivn);
        }
        if (!outside) {
          tend = tc;
          break;
        }
        tc = min3f(P.cx(fi), P.cy(fj), cz(m));
      }
      if (!(tin < tend)) return false;
    }
  }

  // ---- the run [js, je) of whole row segments, with the segment from which
  // each next plane of axis 2 is behind the ray (its cuts); the parts of
  // segments at the ray's ends are added here
  {
    const int sz = uz * (int)G.ms[2];
    int zo = iz * (int)G.ms[2];
    float ai, aj, bi, bj;
    P.at(tin, ai, aj);
    if (ALONE) {
      int guard = (int)(P.tx + P.ty) + kRowCross + 4;
      float m = 0.f;
      while (tin < tend && guard-- > 0) {
        const float tx = P.cx(ai), ty = P.cy(aj), tz = cz(m);
        const float tn = fminf(min3f(tx, ty, tz), tend);
        if (tn > tin) accumulate<MODE, DET, int>(tn - tin, P.cell(ai, aj) + zo, cin, cout, aout, yv, yq, qs, acc);
        tin = tn;
        if (tx == tn) ai += 1.f;
        if (ty == tn) aj += 1.f;
        if (tz == tn) {
          m += 1.f;
          zo += sz;
        }
      }
      return false;
    }
    P.at(tend, bi, bj);
    ray.js = (int)(ai + aj);
    ray.je = (int)(bi + bj);
    ray.uz = uz;
    const float tsb = P.start(bi, bj);
    int m = 0, ne = 0, z = iz;
    float tz = cz(0.f);
    bool tail = true;
    if (tin > P.start(ai, aj)) {
      // enters inside a segment (through a face of axis 2)
      const float te = fminf(fminf(P.cx(ai), P.cy(aj)), tend);
      const int ca = P.cell(ai, aj);
      float ta = tin;
      while (tz < te && m < kRowCross) {
        if (tz > ta) accumulate<MODE, DET, int>(tz - ta, ca + zo, cin, cout, aout, yv, yq, qs, acc);
        ta = tz;
        zo += sz;
        z += uz;
        tz = cz((float)++m);
      }
      if (te > ta) accumulate<MODE, DET, int>(te - ta, ca + zo, cin, cout, aout, yv, yq, qs, acc);
      tail = ray.je != ray.js;
      ray.js += 1;
    }
    ray.z0 = z;
    // Planes crossed inside the run: the segment a plane lies in is left out
    // of the run and added here, part by part.
    float tp = -kRowBig;                                 // the plane before
    while (tz < fminf(tsb, tend) && m < kRowCross) {
      float ci, cj;
      P.at(tz, ci, cj);
      const int c = P.cell(ci, cj) + zo;
      const float ts = P.start(ci, cj), te = fminf(P.cx(ci), P.cy(cj));
      const float tn = cz((float)++m);
      if (ts >= tp && tz > ts) accumulate<MODE, DET, int>(tz - ts, c, cin, cout, aout, yv, yq, qs, acc);
      accumulate<MODE, DET, int>(fminf(te, tn) - tz, c + sz, cin, cout, aout, yv, yq, qs, acc);
      ev[ne++][0] = (unsigned short)(int)(ci + cj);
      zo += sz;
      tp = tz;
      tz = tn;
    }
    ray.cuts = ne;
    if (tail && tend > tsb) {
      const int cb = P.cell(bi, bj);
      float ta = tsb;
      while (tz < tend && m < kRowCross) {
        if (tz > ta) accumulate<MODE, DET, int>(tz - ta, cb + zo, cin, cout, aout, yv, yq, qs, acc);
        ta = tz;
        zo += sz;
        tz = cz((float)++m);
      }
      accumulate<MODE, DET, int>(tend - ta, cb + zo, cin, cout, aout, yv, yq, qs, acc);
    }
  }
  return true;
}

// A short ray, out of line.
template <int MODE, bool SUN, bool DET>
__device__ __noinline__ float row_alone(const Geometry &G, const tg_image_header &V, const FastTables &T,
                                        const RowTables &R, int cidx, int slot, const float *cin, float *cout,
                                        unsigned long long *aout, float yv, float yq, float qs) {
  RowRay ray;
  float acc = 0.f;
  row_ray<MODE, SUN, DET, true>(G, V, T, R, row_path(G, T, R, slot), cidx, slot, cin, cout, aout, yv, yq, qs, nullptr,
                                ray, acc);
  return acc;
}

// Trace the 32 rays (row i, columns j = col0 + lane) of view t, each lane a ray.
// The whole warp calls it.
template <int MODE, bool SUN, bool DET>
__device__ __forceinline__ void row_trace(const Geometry &G, const tg_image_header &V, const FastTables &T,
                                          RowShared &S, int i, int cidx, int col0, int t, int slot,
                                          const float *__restrict__ xin, float *__restrict__ xout,
                                          unsigned long long *__restrict__ acc64,
                                          const DetScale *__restrict__ dsc) {
  constexpr bool PJ = (MODE == TG_PJ || MODE == TG_PJT);
  constexpr bool T4 = (MODE == TG_PJT || MODE == TG_BPJT);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int j = col0 + lane;
  const RowTables &R = S.R;
  bool live = j < G.n2 && !(G.ray_i >= 0 && (i != G.ray_i || j != G.ray_j));
  const long long po = (long long)i * G.ds[0] + (long long)j * G.ds[1] + (long long)t * G.ds[2];
  const bool ovw = PJ && G.overwrite && live;
  if (live && masked(G, i, j, t)) live = false;
  long long fbase = 0;
  if (T4) {
    const int f = V.frame;
    if (f < 0 || f >= G.nframes) live = false;
    else fbase = (long long)f * G.ms[3];
  }
  float yv = 0.f;
  if (!PJ && live) {
    yv = xin[po];
    if (yv == 0.f) live = false;
  }
  if (R.mode[slot] == kRowMiss) live = false;
  if (!__any_sync(0xffffffffu, live)) {
    if (ovw) xout[po] = 0.f;
    return;
  }
  const float *cin = PJ ? xin + fbase : nullptr;
  float *cout = PJ ? nullptr : xout + fbase;
  unsigned long long *aout = DET ? acc64 + fbase : nullptr;
  const float lscale = T.icl[cidx + lane];
  yv *= lscale;
  const float yq = DET ? yv * dsc->yscale : 0.f;
  const float qs = DET ? dsc->qscale : 0.f;
  float acc = 0.f;
  const RowPath P = row_path(G, T, R, slot);
  unsigned short(*ev)[32] = S.ev[warp];
  RowRay ray = {kRowNever, kRowNever, 0, 0, 0};
  const bool hit = live && row_ray<MODE, SUN, DET, false>(
                               G, V, T, R, P, cidx + lane, slot, cin, cout, aout, yv, yq, qs,
                               reinterpret_cast<unsigned short(*)[32]>(&ev[0][lane]), ray, acc);
  if (!hit || ray.js >= ray.je) ray.js = ray.je = kRowNever;
  else ev[ray.cuts][lane] = ev[ray.cuts + 1][lane] = kRowNever;
  const int js = ray.js, je = ray.je, dz = ray.uz * (int)G.ms[2];
  int zo = ray.z0 * (int)G.ms[2];                        // offset along axis 2
  const int first = __reduce_min_sync(0xffffffffu, js);
  const int last = __reduce_max_sync(0xffffffffu, je == kRowNever ? -1 : je);
  if (last > 0) {
    // ---- the run: whole row segments, all lanes on the same segment
    int2 *list = reinterpret_cast<int2 *>(S.list[warp]);
    const int4 *list4 = S.list[warp];
    const float q1 = R.q1[slot], q0 = R.q0[slot];
    int c1 = kRowNever, c2 = kRowNever;                  // the next two cuts
    const unsigned short *pe = &ev[2][lane];
    if (js != kRowNever) {
      c1 = ev[0][lane];
      if (c1 != kRowNever) c2 = ev[1][lane];
    }
    // Windows start at multiples of kRowWin of the row's own count, and a sum
    // is kept per window: a ray's rounding does not depend on the rays beside it.
    for (int base = first & ~(kRowWin - 1); base < last; base += kRowWin) {
      {
        // segment r of the merged path: i crossings of axis 0, r - i of axis 1
        const float r = (float)(base + lane);
        float fi = floorf(fmaf(r + 1.f, q1, q0)), fj = r - fi;
        float ui = fi - P.mx, uj = fj - P.my;
        float x0 = fmaf(ui - 1.f, P.px, P.dx), x1 = fmaf(ui, P.px, P.dx);
        float y0 = fmaf(uj - 1.f, P.py, P.dy), y1 = fmaf(uj, P.py, P.dy);
        if (fi <= 0.f) x0 = P.t0;  // as RowPath::start
        if (fj <= 0.f) y0 = P.t0;
        if (x0 > y1 || y0 > x1) {  // rounding next to a crossing of both: one cell off
          const float d = x0 > y1 ? -1.f : 1.f;
          fi += d;
          fj -= d;
          x0 = y0 = P.start(fi, fj), x1 = P.cx(fi), y1 = P.cy(fj);
        }
        float L = fminf(x1, y1) - fmaxf(x0, y0);
        if (!(L > 0.f)) {
          // both families crossed at once: the corner's cell is not passed; its
          // slot goes to the cell before it, which every ray with this slot in
          // its run has passed (a run begins behind a corner or at the end of
          // a part that row_ray added), with a length of no weight (0 would
          // turn an infinite voxel there into NaN)
          if (y1 <= x1) fi -= 1.f;
          else fj -= 1.f;
          L = 1e-37f;
        }
        fi = fminf(fmaxf(fi, 0.f), P.tx);
        fj = fminf(fmaxf(fj, 0.f), P.ty);
        __syncwarp();
        list[lane] = make_int2(__float_as_int(L), P.cell(fi, fj));
        __syncwarp();
      }
      float part = 0.f;
      const int4 *l4 = list4;
      const int wend = min(base + kRowWin, last);
#pragma unroll 1
      for (int b = base; b < wend; b += kRowGroup, l4 += kRowGroup / 2) {
        const int e = b + kRowGroup;
        const bool in = js < e && je > b;
        if (!__any_sync(0xffffffffu, in && (js > b || je < e || c2 < e))) {
          if (in) row_group<MODE, DET, false>(l4, zo, zo + dz, c1 - b, 0, 0, cin, cout, aout, yv, yq, qs, part);
        } else if (!__any_sync(0xffffffffu, in && c2 < e)) {
          if (in) row_group<MODE, DET, true>(l4, zo, zo + dz, c1 - b, js - b, je - b, cin, cout, aout, yv, yq, qs, part);
        } else if (in) {
          // rays with several cuts in the group: segment by segment
#pragma unroll 1
          for (int s = 0; s < kRowGroup; ++s) {
            bool at_cut = false;
            while (c1 <= b + s) {
              at_cut = c1 == b + s;
              zo += dz;
              c1 = c2;
              if (c2 != kRowNever) {
                c2 = *pe;
                pe += 32;
              }
            }
            const int2 q = reinterpret_cast<const int2 *>(l4)[s];
            if (!at_cut && b + s >= js && b + s < je)
              accumulate<MODE, DET, int>(__int_as_float(q.x), q.y + zo, cin, cout, aout, yv, yq, qs, part);
          }
        }
        if (c1 < e) {                                    // at most one left in the group
          zo += dz;
          c1 = c2;
          if (c2 != kRowNever) {
            c2 = *pe;
            pe += 32;
          }
        }
      }
      acc += part;
    }
  }
  if (ovw) xout[po] = acc * lscale;
  else if (PJ && acc != 0.f) xout[po] += acc * lscale;
}

}  // namespace tg
