// hxg_fp64.cuh -- the FP64 (parity) shell kernel: every value of the ray, the
// fields, the emissivity and the sums in FP64.
//
// Speed.  The sample loop is bound by the FP64 pipe, so it is written for few
// FP64 instructions at unchanged precision:
//   - everything is expressed in the frame turned by the ray's azimuth, where
//     the ray stays at constant Y: the position is X(d), Y, z(d), the field is
//     (B_X, B_Y, B_z), B_par = st B_X + ct B_z, and the sky components are
//     -(ct B_X - st B_z) and -B_Y; no Cartesian position or versor products;
//   - grid coordinates are linear in the distance, one FMA each, split with
//     one round-down add; the 8 corners are summed with weights, each record
//     read with one 32-byte load (two 16-byte loads each take the L1 data
//     stage twice as long);
//   - a ray's window is trimmed with the cut test itself, so the samples
//     between its ends need no test (without an inner radius), and the window,
//     not the whole ray, is cut into the chunks of a pixel's lanes;
//   - divisions by model parameters are products with their reciprocals, the
//     remaining functions come from hxg_math64.cuh, two exponentials of one
//     product are one, and launch constants multiply the sums once; constants
//     whose rounding would act on every sample alike (reciprocals, the
//     observer's grid coordinates, the emissivity scale) are kept in two parts
//     or made in extended precision, so that the maps are as near to the exact
//     ones as with the reference's operations, which round sample by sample;
//   - |B_perp|^2 of CRE index 3 needs neither root nor power, and the angle's
//     cos 2ipa, sin 2ipa never divide by |B_perp|^2;
//   - up to three frequency passes of one geometry share the traversal: a
//     further pass adds its phase and Q, U sums, 23 FP64 instructions.
//
// Measured (B200, two passes over Nside 64/128/256 to 30 kpc on 256^3 grids):
// 34.4 ms before these, 19.4 ms with the sample arithmetic, 14.4 ms with the
// window cut into chunks and the coefficients as constant operands (30 of 32
// lanes active against 20), 13.1 ms with quarter warps of neighbouring rays at
// 128 x 5, 11.6 ms with 32-byte record loads, all pass by pass; 6.7 ms with the two
// passes fused.  A sample is 170 FP64
// instructions, 85 clocks of an SM's FP64 pipes, and about as many of its L1
// data stage (8 records of 32 bytes for each of 32 lanes); the two together
// bound the loop, each about 60 % busy.
#pragma once

#include "hxg_dispatch.cuh"
#include "hxg_integrate.cuh"

// Launch shape of the FP64 shell kernels: threads per block and the resident
// blocks per SM their register allocation must allow.  128 x 5 (96 registers,
// 20 warps, no spills with one grid) runs the case above pass by pass in 11.6 ms
// against 12.4 ms at 128 x 4 and 12.1 ms at 128 x 6 (80 registers, spills).
#ifndef HXG_FP64_THREADS
#define HXG_FP64_THREADS 128
#endif
#ifndef HXG_FP64_MIN_BLOCKS
#define HXG_FP64_MIN_BLOCKS 5
#endif
// With the Jaffe / JF12 / YMW16 models 128 x 4 (128 registers): the masked JF12
// pass of hxg_models_ext.cuh in 2.03 ms against 2.10 ms at 128 x 5; 1 to 3 passes over
// Nside 32/64/128 with Jaffe, JF12, YMW16 and their combinations, with and without a
// grid, within 3 % of 128 x 5 either way and 3-14 % faster than 128 x 3.
#ifndef HXG_FP64_EXT_MIN_BLOCKS
#define HXG_FP64_EXT_MIN_BLOCKS 4
#endif
// The fused kernels: three passes over Nside 128-1024 on 512^3 grids 91.7 ms (94.4 at
// 128 x 4, 95.4 at 128 x 6), two passes over the case above 6.8 ms (7.2, 7.1); 92.5 and
// 6.7 ms now (211 and 11.8 pass by pass).
#ifndef HXG_FP64_MULTI_MIN_BLOCKS
#define HXG_FP64_MULTI_MIN_BLOCKS 5
#endif

namespace hxg {

// Sample range [i0, i1) of chunk c of a ray: the ray window (ray_window) trimmed
// with the cut test itself, |pos| <= r_max and z_min <= z <= z_max
// (integrator.cc:179-182), then cut into equal parts.  Ball and slab are
// convex, so the passing samples are one run and need no further test (but
// for an inner radius).  Equal parts of the window, not of the whole ray: a
// warp's chunks end together, where parts of the ray left the outer chunks of
// the outer shells empty.  The adjoint takes the same ranges.
__device__ __forceinline__ void chunk_range64(const ShellLaunch &P, const double u[3], int c,
                                              int &i0, int &i1) {
  const auto pass = [&](long long i) {
    const double d = fma((double)i + 0.5, P.delta, P.d_start);
    const double px = fma(u[0], d, P.obs[0]), py = fma(u[1], d, P.obs[1]),
                 pz = fma(u[2], d, P.obs[2]);
    const double len = sqrt(px * px + py * py + pz * pz);
    return !(len > P.gc_r_max || pz < P.gc_z_min || pz > P.gc_z_max);
  };
  long long lo, hi;
  ray_window(P, u[0], u[1], u[2], lo, hi);
  while (lo < hi && !pass(lo)) ++lo;
  while (hi > lo && !pass(hi - 1)) --hi;
  // sample indices fit 32 bits (checked on the host)
  const long long n = max(hi - lo, 0ll);
  i0 = (int)(lo + ((n * c) >> P.log2_chunks));
  i1 = (int)(lo + ((n * (c + 1)) >> P.log2_chunks));
}

// The observer in the frame turned by the ray's azimuth, (oX, Y): r^2 along the ray
// is X^2 + YY with X = st d + oX, never 0, so that 1/r is finite; csY and ssY are Y
// times the cos and sin of the spiral's pitch.  Rounding of oX and Y moves every
// sample of the ray alike, so their second parts go into the constants: into csY, ssY
// and Y^2 exactly, 2 X oXl into YY with the X of the middle of the samples [i0, i1).
// Error of Q, U at 1.4 GHz against an extended-precision integral (Nside 4/8/16, 32^3
// grids, mean of 24 skies): 4.4e-15, 4.5e-15 without, 3.8e-15, 4.2e-15 with.
__device__ __forceinline__ void turned_observer(const ShellLaunch &P, double st, double cp,
                                                double sp, int i0, int i1, double &oX,
                                                double &YY, double &csY, double &ssY) {
  const FastModels &F = P.fast;
  double oXl, Y, Yl;
  dot2_64(cp, P.obs[0], sp, P.obs[1], oX, oXl);
  dot2_64(cp, P.obs[1], -sp, P.obs[0], Y, Yl);
  const double Xm = fma(st, fma(0.5 * ((double)i0 + (double)i1), P.delta, P.d_start), oX);
  YY = fmax(fma(Y, Y, 2. * fma(Y, Yl, Xm * oXl)), 1e-280);
  csY = fma(F.sp_cos, Y, fma(F.sp_cos, Yl, -(F.sp_sin * oXl)));
  ssY = fma(F.sp_sin, Y, fma(F.sp_sin, Yl, F.sp_cos * oXl));
}

// Grid coordinate k of the ray at distance d: (observer - lo + u d) scale, the
// rounding of observer - lo, which would move every sample of every ray the
// same way, added back.
__device__ __forceinline__ double grid_at64(const DevGridGroup &G, double u, int k, double d) {
  return fma(fma(u, d, G.ol[k]), G.scale[k], G.gl[k]);
}

// The samples [ga, gb) of [i0, i1) of a ray that lie inside a grid group's box
// (0 < g < n - 1 on every axis, breg.cc:34-54): the slab intersections, widened
// by two samples and trimmed with the test itself (the rounded grid coordinate
// is monotone in d).
__device__ __forceinline__ void grid_range64(const ShellLaunch &P, const DevGridGroup &G,
                                             const double u[3], int i0, int i1, int &ga,
                                             int &gb) {
  double g0[3], gv[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    g0[k] = G.ol[k] * G.scale[k];
    gv[k] = u[k] * G.scale[k];
  }
  grid_window(P, G, g0, gv, i0, i1, ga, gb);
  const auto in = [&](int i) {
    const double d = fma((double)i + 0.5, P.delta, P.d_start);
    bool ok = true;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double g = grid_at64(G, u[k], k, d);
      ok = ok && g > 0. && g < G.gmax[k];
    }
    return ok;
  };
  while (ga < gb && !in(ga)) ++ga;
  while (gb > ga && !in(gb - 1)) --gb;
}

// Cell and fraction of a grid coordinate 0 < g < 2^31: adding 2^52 rounded
// down leaves floor(g) in the low word.
__device__ __forceinline__ void cell64(double g, int &cell, double &frac) {
  const double t = __dadd_rd(g, kC64.floor52);
  cell = __double2loint(t);
  frac = g - (t - kC64.floor52);
}

// One voxel record (32 bytes, aligned to 32) in one load.
__device__ __forceinline__ void load_rec32(const double2 *p, double2 &a, double2 &b) {
  asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
      : "=d"(a.x), "=d"(a.y), "=d"(b.x), "=d"(b.y)
      : "l"(p));
}

// The cell of a sample: record index of its corner 000 (32 bits: larger grids take
// the kernel for several grids, fp64_groups), the (x, y) weights and the z weights.
struct Cell64 {
  unsigned key;
  double w4[4], ez, fz;
};
__device__ __forceinline__ void cell_of64(const DevGridGroup &G, const double u[3], double d,
                                          Cell64 &W) {
  int cx, cy, cz;
  double fx, fy;
  cell64(grid_at64(G, u[0], 0, d), cx, fx);
  cell64(grid_at64(G, u[1], 1, d), cy, fy);
  cell64(grid_at64(G, u[2], 2, d), cz, W.fz);
  W.key = ((unsigned)cx * (unsigned)G.ny + (unsigned)cy) * (unsigned)G.nz + (unsigned)cz;
  const double ex = 1. - fx, ey = 1. - fy;
  W.ez = 1. - W.fz;
  W.w4[0] = ex * ey;
  W.w4[1] = ex * fy;
  W.w4[2] = fx * ey;
  W.w4[3] = fx * fy;
}

// Trilinear sample of the FP64 records (breg.cc:58-96): the 8 corner records
// summed with their weights.  out = bx, by, bz, n_e.
__device__ __forceinline__ void trilinear64(const DevGridGroup &G, const Cell64 &W,
                                            double out[4]) {
  const double2 *p = reinterpret_cast<const double2 *>(G.rec) + 2 * (size_t)W.key;
  const size_t sy = 2 * (size_t)G.nz, sx = sy * (size_t)G.ny;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const double2 *q = p + (k & 1 ? sy : 0) + (k & 2 ? sx : 0);
    double2 a0, a1, b0, b1;
    load_rec32(q, a0, a1);
    load_rec32(q + 2, b0, b1);
    const double wa = W.w4[k] * W.ez, wb = W.w4[k] * W.fz;
    if (k == 0) {
      out[0] = wa * a0.x;
      out[1] = wa * a0.y;
      out[2] = wa * a1.x;
      out[3] = wa * a1.y;
    } else {
      out[0] = fma(wa, a0.x, out[0]);
      out[1] = fma(wa, a0.y, out[1]);
      out[2] = fma(wa, a1.x, out[2]);
      out[3] = fma(wa, a1.y, out[3]);
    }
    out[0] = fma(wb, b0.x, out[0]);
    out[1] = fma(wb, b0.y, out[1]);
    out[2] = fma(wb, b1.x, out[2]);
    out[3] = fma(wb, b1.y, out[3]);
  }
}

// (rs - r) / r_s - |z| / h_s of the spiral, -(r / r_s + |z| / h_s) of the disk,
// with reciprocals in two parts.
__device__ __forceinline__ double spiral_arg64(const FastModels &F, double r, double az) {
  const double s = F.sp_rsun - r;
  const double t = fma(az, F.sp_ihs_l, fma(-s, F.sp_irs_l, az * F.sp_ihs));
  return fma(s, F.sp_irs, -t);
}
__device__ __forceinline__ double disk_arg64(const FastModels &F, double r, double az) {
  const double t = fma(az, F.ex_ihn_l, fma(r, F.ex_irn_l, az * F.ex_ihn));
  return -fma(r, F.ex_irn, t);
}

// CRE_ana spatial profile exp((R0 - r)/r0) sech^2(z/z0) (cre_ana.cc:11-63):
//   = e^((R0 - r)/r0 - 2|z|/z0) (2 / (1 + t))^2, t = e^(-2|z|/z0).
template <bool kRange>
__device__ __forceinline__ double cre_ana_prof64(const FastModels &F, double r, double az) {
  const double a = az * F.cre64_2iz0;
  const double t = exp64<kRange>(-a);
  const double e = exp64<kRange>(fma(F.cre64_R0 - r, F.cre64_ir0, -a));
  const double i = rcp64(fma(t, 0.5, 0.5));
  return e * (i * i);
}

// |B_perp|^pe of the constant-index emissivity, b2 = |B_perp|^2 in units of
// 2^-40 G^2 (k_t and k_p carry the unit), so that the logarithm stays small.
// With an exponent e = (index + 1)/2 above 0 the reference's A^e |B_perp| at
// zero field is inf * 0.
__device__ __forceinline__ double bperp_pow64(const ShellLaunch &P, double b2) {
  if (P.em_pe == 1.) return sqrt(b2);
  if (b2 == 0.) return P.em_pe < 1. ? nan("") : 0.;
  return exp64<true>(0.5 * P.em_pe * log(b2));
}

// |B_perp|^2 in G^2 up to which the sums of squares lose their last bits or all of
// them (a thin disk far from the plane): the angle then comes from fields scaled
// by kTinyScale.
constexpr double kTinyB2 = 1e-290;
constexpr double kTinyScale = 0x1p500;

// cos 2ipa and sin 2ipa of sky components (xv, yv) below that; ipa of a zero B_perp
// is 0 (atan2(0, 0)), and so is that of one below 1e-295 G.
__device__ __forceinline__ void angle64(double xv, double yv, double &c2, double &s2) {
  xv *= kTinyScale;
  yv *= kTinyScale;
  const double rr = fma(yv, yv, xv * xv);
  const double inv = rr > kTinyB2 ? rcp64(rr) : 0.;
  c2 = rr > kTinyB2 ? fma(-yv, yv, xv * xv) * inv : 1.;
  s2 = 2. * (xv * yv) * inv;
}

// Warp gw of shell launch P (32/C pixels, C lanes each) for the NF frequency
// passes of Fq.  All 32 lanes of the warp call it with the same gw.  kFast:
// the launch's models satisfy fast_models and fast_ok (the other models and the
// exponentials' range checks compiled out).
template <int NG, bool kExt, int NF, bool kFast>
__device__ __forceinline__ void fp64_tile(const ShellLaunch &P, const FreqSet<NF> &Fq,
                                          long long gw, int lane) {
  // the warp's 32/C pixels side by side, chunk after chunk: the lanes of a
  // load's quarter warp are neighbouring rays at the same distance, which
  // share cache lines
  const int S = 32 >> P.log2_chunks;
  const int seg = lane & (S - 1);
  const int c = lane >> (5 - P.log2_chunks);
  const Hpx h = hpx_make((uint64_t)P.nside);
  const unsigned long long nest =
      shard_nest(P, (unsigned long long)gw * S + seg);
  const bool valid = nest < h.npix;
  uint64_t ring = 0;
  bool live = false;
  if (valid) {
    ring = hpx_nest2ring(h, nest);
    live = (P.mask == nullptr) || (P.mask[ring] != 0);
  }
  double dm = 0., fd = 0., si[NF], sq[NF], su[NF];
#pragma unroll
  for (int f = 0; f < NF; ++f) si[f] = sq[f] = su[f] = 0.;
  if (live) {
    double th, ph;
    hpx_pix2ang(h, ring, th, ph);
    double inner = 0.;
    if (P.fdmap != nullptr) {
      const Hpx hf = hpx_make((uint64_t)P.nside_fdmap);
      inner = hpx_interpolate(hf, P.fdmap, th, ph);
    }
    if (NF == 1 && P.ck_inner != nullptr && c == 0) P.ck_inner[ring] = inner;
    const double st = sin(th), ct = cos(th), sp = sin(ph), cp = cos(ph);
    // los_versor (integrator.cc:268-272)
    const double u[3] = {cp * st, sp * st, ct};
    const DevModels &M = P.models;
    const FastModels &F = P.fast;
    const double oz = P.obs[2];
    const bool fast_b = M.breg == kBregSpiral;
    const bool fast_t = M.tereg == kTeregExpdisk;
    const bool slow_b = !kFast && M.breg != kBregNone && !fast_b;
    const bool slow_t = !kFast && M.tereg != kTeregNone && !fast_t;
    const bool cre_ana = kFast || M.cre == kCreAna;
    // Faraday phase in quarter turns: q0 + quarter_k * (FD sum), per pass
    double q0[NF];
#pragma unroll
    for (int f = 0; f < NF; ++f)
      q0[f] = Fq.inner[f] ? inner * Fq.quarter_i[f] : 0.;
    const bool pe2 = P.em_const && P.em_pe == 2.;
    double sdm = 0., sfd = 0., last_index = nan(""), gt = P.em_gt, gp = P.em_gp;
    int i0, i1;
    chunk_range64(P, u, c, i0, i1);
    int ga = i1, gb = i1;
    if (NG == 1) grid_range64(P, P.groups[0], u, i0, i1, ga, gb);
    double oX, YY, csY, ssY;
    turned_observer(P, st, cp, sp, i0, i1, oX, YY, csY, ssY);
    double x = (double)i0 + 0.5;
#pragma unroll 1
    for (int i = i0; i < i1; ++i, x += 1.) {
      const double d = fma(x, P.delta, P.d_start);
      const double z = fma(ct, d, oz);
      const double X = fma(st, d, oX);
      const double r2 = fma(X, X, YY);
      double p3[3] = {0., 0., 0.};
      if (!kFast || NG > 1) {
#pragma unroll
        for (int k = 0; k < 3; ++k) p3[k] = fma(u[k], d, P.obs[k]);
        // an inner radius can split a ray's passing samples in two runs
        if (!kFast && P.gc_r_min > 0. && sqrt(r2 + z * z) < P.gc_r_min) continue;
      }
      // the grid first: its loads return while the models are evaluated
      double g[4] = {0., 0., 0., 0.};
      if (NG == 1) {
        if ((unsigned)(i - ga) < (unsigned)(gb - ga)) {
          Cell64 W;
          cell_of64(P.groups[0], u, d, W);
          trilinear64(P.groups[0], W, g);
        }
      } else if (NG > 1) {
        double b3[3] = {0., 0., 0.};
        CellCache<double> cc;
#pragma unroll 1
        for (int k = 0; k < P.ngroups; ++k)
          sample_group<double, false>(P.groups[k], p3[0], p3[1], p3[2], cc, b3, g[3]);
        g[0] = b3[0];
        g[1] = b3[1];
        g[2] = b3[2];
      }
      double ir;
      const double r = sqrt64(r2, ir);
      const double az = fabs(z);
      double bX = 0., bY = 0., bz = 0., te = 0.;
      // positive doubles compare like integers, off the FP64 pipe
      if (fast_b && __double_as_longlong(r2) >= __double_as_longlong(F.rc2_lo) &&
          __double_as_longlong(r2) <= __double_as_longlong(F.rc2_hi)) {
        const double a = F.sp_b0 * (exp64<!kFast>(spiral_arg64(F, r, az)) * ir);
        bX = a * fma(F.sp_sin, X, -csY);
        bY = a * fma(F.sp_cos, X, ssY);
      }
      if (fast_t) te = F.ex_n0 * exp64<!kFast>(disk_arg64(F, r, az));
      if (slow_b) {
        const V3<double> B = breg_model_x<kExt, true>(M, P.ext, p3[0], p3[1], p3[2], p3);
        bX = fma(cp, B.x, sp * B.y);
        bY = fma(cp, B.y, -(sp * B.x));
        bz = B.z;
      }
      if (slow_t) te = tereg_model_x<kExt>(M, P.ext, p3[0], p3[1], p3[2], p3);
      if (NG > 0) {
        bX = fma(cp, g[0], fma(sp, g[1], bX));
        bY = fma(cp, g[1], fma(-sp, g[0], bY));
        bz += g[2];
        te += g[3];
      }
      // n_e clamped at 0 (integrator.cc:201); NaN stays NaN
      if (__double2hiint(te) < 0) te *= 0.;
      sdm += te;
      sfd = fma(te, fma(st, bX, ct * bz), sfd);
      if (P.do_sync) {
        // B_perp on the sky basis: |B_perp|^2 = xv^2 + yv^2, cos 2ipa =
        // (xv^2 - yv^2) / |B_perp|^2, sin 2ipa = 2 xv yv / |B_perp|^2
        // (integrator.cc:257-265); both signs of (xv, yv) give the same
        const double xv = bY, yv = fma(ct, bX, -(st * bz));
        const double x2 = xv * xv;
        const double rr = fma(yv, yv, x2), cc2 = fma(-yv, yv, x2), hs2 = xv * yv;
        double wt[NF], wpc[NF], wps[NF];
        constexpr int NW = kFast ? 1 : NF;
        bool shared_w = true;
        if (kExt && M.cre == kCreGrid) {
          // spectral integral over the CRE grid (integrator.cc:288-330,
          // 357-400); the host fuses no CRE-grid pass
          double jt, jp;
          cre_grid_j(P.ext->cre, p3[0], p3[1], p3[2], sqrt(rr), jt, jp);
          const double inv = rr > 0. ? 1. / rr : 0.;
          wt[0] = jt;
          wpc[0] = rr > 0. ? jp * cc2 * inv : jp;
          wps[0] = 2. * jp * hs2 * inv;
        } else {
          const double prof = cre_ana ? cre_ana_prof64<!kFast>(F, r, az)
                                      : cre_profile<double>(M, p3[0], p3[1], p3[2], p3);
          if (pe2) {
            wt[0] = prof * rr;
            wpc[0] = prof * cc2;
            wps[0] = (prof + prof) * hs2;
          } else {
            double wp[NF];
            if (kFast || P.em_const) {
              wt[0] = wp[0] = prof * bperp_pow64(P, rr * 0x1p40);
            } else {
              shared_w = false;
              const double index = cre_index<double>(M, p3[0], p3[1], p3[2]);
              if (index != last_index) {
                gt = tgamma(-0.25 * index + 19. / 12.) * tgamma(-0.25 * index - 1. / 12.);
                gp = tgamma(-0.25 * index + 7. / 12.) * tgamma(-0.25 * index - 1. / 12.);
                last_index = index;
              }
              const double bper = sqrt(rr);
#pragma unroll
              for (int f = 0; f < NW; ++f) {
                const double base = prof * bper * pow(Fq.a_s[f] / bper, 0.5 * (index + 1));
                wt[f] = base * gt / (1. - index);
                wp[f] = base * gp;
              }
            }
            const double inv = rcp64(rr);
            double c2 = cc2 * inv, s2 = 2. * hs2 * inv;
            if (rr < kTinyB2) angle64(xv, yv, c2, s2);
#pragma unroll
            for (int f = 0; f < NW; ++f) {
              if (f > 0 && shared_w) break;
              wpc[f] = wp[f] * c2;
              wps[f] = wp[f] * s2;
            }
          }
        }
        if (shared_w) {
#pragma unroll
          for (int f = 1; f < NF; ++f) {
            wt[f] = wt[0];
            wpc[f] = wpc[0];
            wps[f] = wps[0];
          }
        }
        si[0] += wt[0];
        if (!kFast) {
#pragma unroll
          for (int f = 1; f < NF; ++f) si[f] += wt[f];
        }
#pragma unroll
        for (int f = 0; f < NF; ++f) {
          double sf, cf;
          sincos_quarter(fma(Fq.quarter_k[f], sfd, q0[f]), sf, cf);
          sq[f] = fma(cf, wpc[f], fma(-sf, wps[f], sq[f]));
          su[f] = fma(sf, wpc[f], fma(cf, wps[f], su[f]));
        }
      }
    }
    dm = sdm * P.delta;
    fd = sfd * P.fd_fore * P.delta;
    // I is one sum for all passes of the constant-index models
    const double s0 = si[0];
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      si[f] = (kFast ? s0 : si[f]) * Fq.k_t[f];
      sq[f] *= Fq.k_p[f];
      su[f] *= Fq.k_p[f];
    }
  }
  if (NF == 1 && P.ck != nullptr) store_checkpoint(P, live, nest, c, S, fd, sq[0], su[0]);
  combine_chunks_nf<NF>(P, Fq, c, dm, fd, si, sq, su, S);
  if (live && c == 0) {
    if (P.do_dm) P.out[0][ring] = dm;
    if (P.do_fd || P.do_sync) P.out[1][ring] = fd;
    if (P.do_sync) {
#pragma unroll
      for (int f = 0; f < NF; ++f) {
        Fq.out[f][0][ring] = si[f] * Fq.tc_a[f] * Fq.tc_a[f] / Fq.tc_b[f];
        Fq.out[f][1][ring] = sq[f] * Fq.tc_a[f] * Fq.tc_a[f] / Fq.tc_b[f];
        Fq.out[f][2][ring] = su[f] * Fq.tc_a[f] * Fq.tc_a[f] / Fq.tc_b[f];
      }
    }
  } else if (valid && !live && c == 0) {
    // masked pixel: every observable is zero (integrator.cc:63-67, 98-115)
    if (P.do_dm) P.out[0][ring] = 0.;
    if (P.do_fd || P.do_sync) P.out[1][ring] = 0.;
    if (P.do_sync) {
#pragma unroll
      for (int f = 0; f < NF; ++f)
        Fq.out[f][0][ring] = Fq.out[f][1][ring] = Fq.out[f][2][ring] = 0.;
    }
  }
}

// One frequency pass: the pass's constants from its launch block.
template <int NG, bool kExt, bool kFast>
__device__ __forceinline__ void fp64_tile(const ShellLaunch &P, long long gw, int lane) {
  FreqSet<1> Fq;
  freq_of_launch(P, Fq);
  fp64_tile<NG, kExt, 1, kFast>(P, Fq, gw, lane);
}

template <int NG, bool kExt, bool kFast>
__global__ void __launch_bounds__(HXG_FP64_THREADS,
                                  kExt ? HXG_FP64_EXT_MIN_BLOCKS : HXG_FP64_MIN_BLOCKS)
shell_fp64_kernel(const ShellLaunch P) {
  fp64_tile<NG, kExt, kFast>(P, ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5,
                             threadIdx.x & 31);
}

// NF frequency passes in one traversal of the shell.
template <int NG, bool kExt, int NF, bool kFast>
__global__ void __launch_bounds__(HXG_FP64_THREADS,
                                  kExt ? HXG_FP64_EXT_MIN_BLOCKS : HXG_FP64_MULTI_MIN_BLOCKS)
shell_fp64_multi_kernel(const ShellLaunch P, const FreqSet<NF> Fq) {
  fp64_tile<NG, kExt, NF, kFast>(P, Fq, ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5,
                                 threadIdx.x & 31);
}

// The grid-group count of P's instantiation.
inline int shape64(const ShellLaunch &P) {
  const DevGridGroup &G = P.groups[0];
  return fp64_groups(P.ngroups, G.rec, G.nx, G.ny, G.nz);
}

// The plans of a batch level, kGroupPlans to a kernel.
template <int NG, bool kExt, int NF, bool kFast>
__global__ void __launch_bounds__(HXG_FP64_THREADS,
                                  kExt ? HXG_FP64_EXT_MIN_BLOCKS : HXG_FP64_MULTI_MIN_BLOCKS)
shell_fp64_group_kernel(const __grid_constant__ PlanGroup<NF> G) {
  unsigned block;
  const int k = group_plan(G, block);
  fp64_tile<NG, kExt, NF, kFast>(G.P[k], G.F[k],
                                 ((long long)block * blockDim.x + threadIdx.x) >> 5,
                                 threadIdx.x & 31);
}

}  // namespace hxg
