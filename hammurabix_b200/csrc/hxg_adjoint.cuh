// hxg_adjoint.cuh -- adjoint (reverse-mode) shell kernel of the FP64 form.
//
// Given dL/d(shell maps) of one shell, it accumulates dL/d(packed grid
// records), dL/d(model parameters) and dL/d(inner-shell Faraday-depth map).
// Per-shell checkpointing: the forward kernel stored, for every (pixel,
// chunk), the Faraday depth before the chunk and Q, U from the chunk on
// (store_checkpoint), plus the pixel's inner-shell Faraday depth, so a
// single forward-ordered sweep suffices: the reverse-accumulated phase
// sensitivity S_i = sum_{k >= i} dL/dchi_k equals
// 2 (gU (Q - Q_{<i}) - gQ (U - U_{<i})), one running sum since gQ, gU are
// constant along a ray.
//
// Per sample i (symbols of integrator.cc:173-226):
//   t_i   = n_e B_par K dl           (Faraday-depth term, K = fd_forefactor)
//   chi_i = (FD_inner + sum_{k<=i} t_k) lambda^2 + ipa_i
//   dL/dt_i   = gFD + lambda^2 S_i
//   dL/dJt_i  = gI,  dL/dJp_i = gQ cos 2chi_i + gU sin 2chi_i
//   J ~ |B_perp|^(1-e), e = (index+1)/2  ->  dJ/d|B_perp| = (1-e) J / |B_perp|
//   dipa/dB = (-x e_theta + y e_phi) / (x^2 + y^2),  y = -e_theta.B,
//   x = -e_phi.B
//
// The sample is fp64_tile's, in the frame turned by the ray's azimuth (there
// u = (st, 0, ct), e_theta = (ct, 0, -st), e_phi = (0, 1, 0)); its reverse
// adds about 90 FP64 instructions to the forward's 170.  The grid-record
// gradient of a cell is summed in registers while the ray stays in it and
// flushed with 32 atomic adds at record offsets (the cell index is the offset
// of its first corner: no divisions).
#pragma once

#include "hxg_fp64.cuh"

namespace hxg {

// Parameter-gradient slots: spiral B (b0, pitch, r_scale, h_scale),
// exponential n_e disk (n0, r_scale, h_scale), CRE normalisation j0.
constexpr int kNumParams = 8;

struct AdjointLaunch {
  ShellLaunch F;            // the forward launch of this shell
  const double *ck;         // [(nest * C + c) * 3]: store_checkpoint's values
  const double *ck_inner;   // [ring]: inner-shell FD of each pixel
  const double *g[5];       // dL/d(shell maps) (ring): dm, fd, I, Q, U (I,Q,U
                            // already times the temp_convert factor)
  double *grad_rec;         // [N * 4] dL/d(group-0 records), or null
  double *grad_par;         // [kNumParams], or null
  double *g_fdmap;          // [npix(nside_fdmap)] dL/d(accumulated FD map), or null
  int by_chunk;             // FP32C: a block's lanes take one chunk of 128 pixels
  int want_j0;              // 1 when the CRE normalisation gradient is wanted
};

constexpr unsigned kNoCell = 0xFFFFFFFFu;

// Adds the accumulators of the cell whose corner 000 is record `key` into the
// record gradient and clears them.
template <typename T>
__device__ __forceinline__ void flush_cell(double *grad_rec, unsigned key, unsigned ny,
                                           unsigned nz, T acc[8][4]) {
  if (key == kNoCell) return;
  const unsigned nyz = ny * nz;
#pragma unroll
  for (int dx = 0; dx < 2; ++dx)
#pragma unroll
    for (int dy = 0; dy < 2; ++dy) {
      double *p = grad_rec + 4 * (size_t)(key + dx * nyz + dy * nz);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        T &a = acc[dx * 4 + dy * 2 + (k >> 2)][k & 3];
        atomicAdd(p + k, (double)a);
        a = T(0);
      }
    }
}

// Launch shape of the adjoint shell kernel (threads per block, resident
// blocks per SM its register allocation must allow).  128 x 3 (168
// registers, 12 warps per SM; the per-cell gradient accumulators take 64)
// runs forward, loss and backward on 256^3 grids, Nside 64/128/256, in 23.0 ms
// against 25.4 ms at 128 x 4 (128 registers, spills) and 26.1 ms at 128 x 2;
// 44.7 ms with the kernel before, which evaluated the sample with the
// reference's operations, divided 64-bit indices in every flush and had
// 1670 warp instructions a sample (FP64 pipe 37 % busy).
#ifndef HXG_ADJ_THREADS
#define HXG_ADJ_THREADS 128
#endif
#ifndef HXG_ADJ_MIN_BLOCKS
#define HXG_ADJ_MIN_BLOCKS 3
#endif

// kFast: the forward launch's models satisfy fast_models (the other models
// compiled out).
template <int NG, bool kExt, bool kFast>
__global__ void __launch_bounds__(HXG_ADJ_THREADS, HXG_ADJ_MIN_BLOCKS)
shell_fp64_adjoint_kernel(const AdjointLaunch A) {
  const ShellLaunch &P = A.F;
  const int lane = threadIdx.x & 31;
  const long long gw =
      ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int C = P.chunks;
  // the forward's lanes (fp64_tile): chunks of a pixel S lanes apart
  const int S = 32 >> P.log2_chunks;
  const int seg = lane & (S - 1);
  const int c = lane >> (5 - P.log2_chunks);
  const Hpx h = hpx_make((uint64_t)P.nside);
  // shard `shard` of `nshards` of the shell (the forward's pixels)
  const unsigned long long nest =
      shard_nest(P, (unsigned long long)gw * S + seg);
  const bool valid = nest < h.npix;
  uint64_t ring = 0;
  bool live = false;
  if (valid) {
    ring = hpx_nest2ring(h, nest);
    live = (P.mask == nullptr) || (P.mask[ring] != 0);
  }
  // the Faraday depth before this chunk, Q and U from it on
  double Fc = 0., Qs = 0., Us = 0.;
  if (live) {
    const unsigned long long ci = nest * (unsigned long long)C + c;
    Fc = A.ck[3 * ci];
    Qs = A.ck[3 * ci + 1];
    Us = A.ck[3 * ci + 2];
  }
  const double l2 = P.lambda2;
  double gp[kNumParams];
#pragma unroll
  for (int k = 0; k < kNumParams; ++k) gp[k] = 0.;
  if (live) {
    const double gdm = P.do_dm ? A.g[0][ring] : 0.;
    const double gfd = (P.do_fd || P.do_sync) ? A.g[1][ring] : 0.;
    const double gI = P.do_sync ? A.g[2][ring] : 0.;
    const double gQ = P.do_sync ? A.g[3][ring] : 0.;
    const double gU = P.do_sync ? A.g[4][ring] : 0.;
    double th, ph;
    hpx_pix2ang(h, ring, th, ph);
    const double inner = A.ck_inner[ring];
    // dL/d(inner FD) = lambda^2 sum_i dL/dchi_i, scattered through the
    // transpose of the HEALPix interpolation that produced it
    if (c == 0 && A.g_fdmap != nullptr && P.fdmap != nullptr && P.do_sync) {
      const double g_inner = l2 * 2. * (gU * Qs - gQ * Us);
      const Hpx hf = hpx_make((uint64_t)P.nside_fdmap);
      uint64_t pix[4];
      double w[4];
      hpx_interp_weights(hf, th, ph, pix, w);
      const double wtot = w[0] + w[1] + w[2] + w[3];
      if (wtot != 0.)
        for (int k = 0; k < 4; ++k) atomicAdd(A.g_fdmap + pix[k], g_inner * w[k] / wtot);
    }
    const double st = sin(th), ct = cos(th), sp = sin(ph), cp = cos(ph);
    const double u[3] = {cp * st, sp * st, ct};
    const DevModels &M = P.models;
    const FastModels &F = P.fast;
    const double oz = P.obs[2];
    const bool fast_b = M.breg == kBregSpiral;
    const bool fast_t = M.tereg == kTeregExpdisk;
    const bool slow_b = !kFast && M.breg != kBregNone && !fast_b;
    const bool slow_t = !kFast && M.tereg != kTeregNone && !fast_t;
    const bool pe2 = P.em_const && P.em_pe == 2.;
    // dL/d(the sample's weights): the launch scales folded in
    const double gIk = gI * P.k_t, gQk = gQ * P.k_p, gUk = gU * P.k_p;
    const double K = P.fd_fore * P.delta, gdmd = gdm * P.delta;
    // gfd + lambda^2 S_i, running: S starts at the chunk's own
    double gtt = fma(2. * l2, gU * Qs - gQ * Us, gfd);
    if (!P.do_sync) gtt = gfd;
    const double l2x2 = 2. * l2;
    // Faraday phase in quarter turns: inner + Fc + the running chunk FD (the
    // sample's own term included)
    const double q0 = (inner + Fc) * P.quarter_i;
    double acc[8][4];
#pragma unroll
    for (int k = 0; k < 8; ++k)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[k][q] = 0.;
    unsigned acc_key = kNoCell;
    double gt = P.em_gt, gpp = P.em_gp, last_index = nan("");
    double sfd = 0.;  // running FD of this chunk (FD-sum units)
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
      if (!kFast) {
#pragma unroll
        for (int k = 0; k < 3; ++k) p3[k] = fma(u[k], d, P.obs[k]);
        if (P.gc_r_min > 0. && sqrt(r2 + z * z) < P.gc_r_min) continue;
      }
      double g[4] = {0., 0., 0., 0.};
      Cell64 W;
      W.key = kNoCell;
      if (NG == 1 && (unsigned)(i - ga) < (unsigned)(gb - ga)) {
        cell_of64(P.groups[0], u, d, W);
        trilinear64(P.groups[0], W, g);
      }
      double ir;
      const double r = sqrt64(r2, ir);
      const double az = fabs(z);
      double sX = 0., sY = 0., bX = 0., bY = 0., bz = 0., te_d = 0.;
      if (fast_b && __double_as_longlong(r2) >= __double_as_longlong(F.rc2_lo) &&
          __double_as_longlong(r2) <= __double_as_longlong(F.rc2_hi)) {
        const double a = F.sp_b0 * (exp64<!kFast>(spiral_arg64(F, r, az)) * ir);
        sX = a * fma(F.sp_sin, X, -csY);
        sY = a * fma(F.sp_cos, X, ssY);
      }
      bX = sX;
      bY = sY;
      if (fast_t) te_d = F.ex_n0 * exp64<!kFast>(disk_arg64(F, r, az));
      double te = te_d;
      if (slow_b) {
        const V3<double> B = breg_model_x<kExt>(M, P.ext, p3[0], p3[1], p3[2], p3);
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
      const bool te_on = te > 0.;
      if (!te_on) te *= 0.;
      const double bpar = fma(st, bX, ct * bz);
      sfd = fma(te, bpar, sfd);
      double g_te = gdmd, g_bpar = 0., g_th = 0., g_ph = 0.;
      if (P.do_fd || P.do_sync) {
        // phase sensitivity of the samples k >= i, the sample's own included
        const double gk = gtt * K;
        if (P.do_sync) {
          const double xv = bY, yv = fma(ct, bX, -(st * bz));
          const double x2 = xv * xv;
          const double rr = fma(yv, yv, x2), cc2 = fma(-yv, yv, x2), hs2 = xv * yv;
          const double irr = rcp64(rr);
          double wt, wpc, wps, pe = P.em_pe;
          const double prof = (kFast || M.cre == kCreAna)
                                  ? cre_ana_prof64<!kFast>(F, r, az)
                                  : cre_profile<double>(M, p3[0], p3[1], p3[2], p3);
          if (pe2) {
            wt = prof * rr;
            wpc = prof * cc2;
            wps = (prof + prof) * hs2;
          } else {
            double wp;
            if (kFast || P.em_const) {
              wt = wp = prof * bperp_pow64(P, rr * 0x1p40);
            } else {
              const double index = cre_index<double>(M, p3[0], p3[1], p3[2]);
              if (index != last_index) {
                gt = tgamma(-0.25 * index + 19. / 12.) * tgamma(-0.25 * index - 1. / 12.);
                gpp = tgamma(-0.25 * index + 7. / 12.) * tgamma(-0.25 * index - 1. / 12.);
                last_index = index;
              }
              const double bper = sqrt(rr), e = 0.5 * (index + 1);
              const double base = prof * bper * pow(P.a_s / bper, e);
              wt = base * gt / (1. - index);
              wp = base * gpp;
              pe = 1. - e;
            }
            double c2 = cc2 * irr, s2 = 2. * hs2 * irr;
            if (rr < kTinyB2) angle64(xv, yv, c2, s2);
            wpc = wp * c2;
            wps = wp * s2;
          }
          double sf, cf;
          sincos_quarter(fma(P.quarter_k, sfd, q0), sf, cf);
          const double qi = fma(cf, wpc, -(sf * wps)), ui = fma(sf, wpc, cf * wps);
          const double dG = fma(gUk, qi, -(gQk * ui));
          gtt = fma(-l2x2, dG, gtt);
          const double ej = fma(gIk, wt, fma(gQk, qi, gUk * ui));
          if (A.want_j0) gp[7] += ej;
          // |B_perp|^pe along B_perp, the angle across it
          const double ke = ej * pe * irr, ki = 2. * dG * irr;
          g_th = fma(ke, yv, ki * xv);
          g_ph = fma(ke, xv, -(ki * yv));
          if (rr < kTinyB2) {  // both fields scaled, as in angle64
            const double xs = xv * kTinyScale, ys = yv * kTinyScale;
            const double ra = fma(ys, ys, xs * xs);
            const double ira = ra > kTinyB2 ? rcp64(ra) : 0.;
            g_th = fma(ej * pe, ys, 2. * dG * xs) * ira * kTinyScale;
            g_ph = fma(ej * pe, xs, -(2. * dG * ys)) * ira * kTinyScale;
          }
        }
        g_te = fma(gk, bpar, g_te);
        g_bpar = gk * te;
      }
      if (!te_on) g_te = 0.;
      const double gX = fma(ct, g_th, st * g_bpar), gz = fma(ct, g_bpar, -(st * g_th));
      // analytic-model parameter gradients (the constants after the loop);
      // B = amp (sin(pitch - phi), cos(pitch - phi)), so dB/dpitch is B turned
      // by -90 degrees
      if (fast_b) {
        const double gdotb = fma(gX, sX, g_ph * sY);
        gp[0] += gdotb;
        gp[1] += fma(gX, sY, -(g_ph * sX));
        gp[2] = fma(gdotb, r - F.sp_rsun, gp[2]);
        gp[3] = fma(gdotb, az, gp[3]);
      }
      if (fast_t) {
        const double gd = g_te * te_d;
        gp[4] += gd;
        gp[5] = fma(gd, r, gp[5]);
        gp[6] = fma(gd, az, gp[6]);
      }
      // grid-record gradients, accumulated per cell
      if (NG > 0 && W.key != kNoCell && A.grad_rec != nullptr) {
        if (W.key != acc_key) {
          flush_cell(A.grad_rec, acc_key, (unsigned)P.groups[0].ny, (unsigned)P.groups[0].nz,
                     acc);
          acc_key = W.key;
        }
        const double gv[4] = {fma(cp, gX, -(sp * g_ph)), fma(sp, gX, cp * g_ph), gz, g_te};
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const double w = W.w4[k >> 1] * (k & 1 ? W.fz : W.ez);
#pragma unroll
          for (int q = 0; q < 4; ++q) acc[k][q] = fma(w, gv[q], acc[k][q]);
        }
      }
    }
    if (NG > 0 && A.grad_rec != nullptr)
      flush_cell(A.grad_rec, acc_key, (unsigned)P.groups[0].ny, (unsigned)P.groups[0].nz, acc);
    gp[0] = M.sp_b0 != 0. ? gp[0] / M.sp_b0 : 0.;
    gp[2] *= F.sp_irs * F.sp_irs;
    gp[3] *= F.sp_ihs * F.sp_ihs;
    gp[4] = M.tex_n0 != 0. ? gp[4] / M.tex_n0 : 0.;
    gp[5] *= F.ex_irn * F.ex_irn;
    gp[6] *= F.ex_ihn * F.ex_ihn;
    if (!fast_b) gp[0] = gp[1] = gp[2] = gp[3] = 0.;
    if (!fast_t) gp[4] = gp[5] = gp[6] = 0.;
  }
  // parameter gradients: warp reduction, one atomic per warp and slot
  if (A.grad_par != nullptr) {
#pragma unroll
    for (int k = 0; k < kNumParams; ++k) {
      double v = gp[k];
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0 && v != 0.) atomicAdd(A.grad_par + k, v);
    }
  }
}

}  // namespace hxg
