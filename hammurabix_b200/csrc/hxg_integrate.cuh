// hxg_integrate.cuh -- shell integration kernels (the per-pixel radial loop
// of Integrator::radial_integration, source/integrator/integrator.cc:136-228,
// run for every pixel of one shell, integrator.cc:60-116).
//
// Mapping: each warp owns 32/C pixels of a compact NESTED sky patch (so
// neighbouring rays share grid cache lines) and C lanes split each pixel's
// radial range into contiguous chunks.  Chunk c integrates with the phase of
// its own partial Faraday depth; once the chunk sums are known, its Stokes
// Q/U are rotated by 2*lambda^2*(Faraday depth of the chunks before it) --
// algebraically identical to the reference's running phase
// (integrator.cc:221-225) -- and the chunks are reduced with warp shuffles.
// With C = 1 (large shells) each lane is one pixel in the reference's order.
#pragma once

#include "hxg_common.cuh"
#include "hxg_fields.cuh"
#include "hxg_math64.cuh"

namespace hxg {

constexpr int kMaxGroups = 4;

// The spiral B, exponential n_e and CRE_ana models as the sample loops
// evaluate them: reciprocals and launch constants precomputed, in FP64 and the
// working units of the form (FP32C: kpc and 2^-20 G).
struct FastModels {
  double sp_b0, sp_irs, sp_crs, sp_ihs;  // amplitude, 1/r_s, r_sun/r_s, 1/h_s
  double sp_sin, sp_cos;                 // sin, cos of the pitch angle
  double ex_n0, ex_irn, ex_ihn;          // exp-disk n0, 1/r_s, 1/h_s
  // the kFast sample loop folds the amplitudes into the exponents:
  // r_sun/r_s + ln|b0| and ln n0, the sign of b0 into sp_*_s
  double sp_crs_l, ex_ln0;
  double sp_sin_s, sp_cos_s;             // sign(b0) sin, sign(b0) cos
  double sp_rsun;                        // r_sun
  // FP64 form: the rounding of sp_irs, sp_ihs, ex_irn, ex_ihn, which would
  // move every sample's exponent the same way
  double sp_irs_l, sp_ihs_l, ex_irn_l, ex_ihn_l;
  double cre64_R0, cre64_ir0, cre64_2iz0;  // CRE_ana: R0, 1/r0, 2/|z0|
  float sp_sinf_s, sp_cosf_s;            // the same in FP32
  // launch constants in the types the sample loop uses, so that the loop
  // reads them as operands instead of converting them
  double r2min, r2max;                   // gc_r_min^2, gc_r_max^2
  double rc2_hi, rc2_lo;                 // spiral cylinder: (20 kpc)^2, (3 kpc)^2
  float sp_sinf, sp_cosf;                // sp_sin, sp_cos
  float cre_ir0, cre_2iz0, cre_R0;       // CRE_ana: 1/r0, 2/z0, R0
  // the same for base-2 exponentials: log2(e)/r0, 2 log2(e)/z0 and
  // 2 + R0 log2(e)/r0 (the factor 4 of 4 e^x / (1 + t)^2 folded in)
  float cre_ir0_l2, cre_2iz0_l2, cre_R0_l2;
  float pe;                              // em_pe
};

// Everything one shell launch needs, in the working units of its form.
struct ShellLaunch {
  double obs[3];             // observer
  double d_start, delta;     // first-sample distance and radial step
  long long step;            // samples per ray (integrator.cc:237-240)
  double gc_r_min, gc_r_max, gc_z_min, gc_z_max;
  int nside, chunks, log2_chunks;
  // shard `shard` of `nshards` of the shell: the NESTED blocks of
  // 2^shard_log2 pixels b with b % nshards == shard (interleaved over the
  // sky, so that the shards see the same mix of ray lengths; a block is a
  // compact sky patch); 0 of 1 for the whole shell
  unsigned shard, nshards, shard_log2;
  int do_dm, do_fd, do_sync;
  const double *fdmap;       // accumulated FD map of inner shells (or null)
  int nside_fdmap;
  const unsigned char *mask; // 1 = integrate (integrator.cc:69-70), or null
  double *out[5];            // shell maps (RING): dm, fd, is, qs, us
  // FD and synchrotron constants
  double fd_fore;            // FP64: -qe^3/(2 pi mec2^2); FP32C: that * delta * 2^-20 G
  double lambda2;            // (c/nu)^2
  double i2bt;               // c^2 / (2 kB nu^2)
  double tc_a, tc_b;         // temp_convert(t) = t*a*a/b (integrator.cc:275-279)
  // analytic synchrotron emissivity (integrator.cc:332-346, 401-415)
  int em_const;              // spectral index constant over space
  double em_index;           // constant index
  double em_n0u;             // j0 * gamma0^-index(observer) * unit
  double em_qe3, em_den_t, em_den_p, em_anum, em_3qe;
  double em_gt, em_gp;       // Gamma products at the constant index
  // scales applied in FP64 after the sums
  double k_t, k_p, k_dm;     // I, Q/U and DM scale factors
  double phase_k;            // 2 lambda^2 * FD per unit of the FD sum
  double quarter_k;          // the same in quarter turns (FP64 form), and
  double quarter_i;          // quarter turns per unit of the inner-shell FD
  double a_s;                // A * |B_perp| in 2^-20 G (variable-index path)
  double em_pe;              // exponent of |B_perp| (constant index, FP32C)
  DevModels models;
  DevGridGroup groups[kMaxGroups];
  int ngroups;
  // adjoint checkpoint: per (pixel, chunk) what store_checkpoint writes, per
  // pixel the inner-shell FD; null = off
  double *ck;
  double *ck_inner;
  FastModels fast;
  // FP32C: per-lane sums instead of maps (shell_combine_kernel finishes them),
  // a block of the launch taking one chunk of its neighbouring pixels; null = off
  double *part;
  unsigned long long part_n;  // lanes of the launch (the sums' stride)
  // FP64 form: every exponent of the FastModels is below 680 in size; FP32C:
  // its constants are finite (the kFast instantiations need it)
  int fast_ok;
  const ExtModels *ext;  // Jaffe / JF12 / YMW16 blocks (device), or null
};

// The models of the grid workloads: B none, grid or spiral; n_e none, grid
// or exponential disk; CRE_ana with a constant index; no inner radius cut
// (gc_r_min = 0, so that the samples of a ray that pass the cuts are one
// contiguous run).  The shell kernels have an instantiation (kFast) for
// launches whose models are among these, with the other models' paths
// compiled out, so that its registers are allocated for this path alone.
__host__ __device__ inline bool fast_models(const ShellLaunch &P) {
  const DevModels &M = P.models;
  return P.ext == nullptr && !(P.gc_r_min > 0.) &&
         // amplitudes folded into the exponents as logarithms (FastModels)
         (M.breg != kBregSpiral || M.sp_b0 != 0.) &&
         (M.tereg != kTeregExpdisk || M.tex_n0 > 0.) &&
         (M.breg == kBregNone || M.breg == kBregGrid || M.breg == kBregSpiral) &&
         (M.tereg == kTeregNone || M.tereg == kTeregGrid || M.tereg == kTeregExpdisk) &&
         (!P.do_sync || (M.cre == kCreAna && P.em_const));
}

// The frequency-dependent constants of NF frequency passes that share one
// shell traversal (same observer, shells, limits and models): each pass's
// phase scale, emissivity scales, temp_convert and I/Q/U shell maps.  The
// positions, field samples, emissivity weights, DM and FD of a sample do not
// depend on the frequency and are computed once for all NF passes.
// Launch shape of the fused-frequency shell kernel: threads per block and
// the resident blocks per SM its register budget is cut for.  128 x 5
// (96 registers) keeps 20 warps per SM; for the general instantiation it ran
// config 3 in 91.3 ms against 92.8 ms at 256 x 2 (128 registers) and
// 97.2 ms at 128 x 6 (80 registers, more spills).  The kFast instantiation
// runs 128 x 7 (72 registers, 28 warps): config 3's fused step 59.1 ms
// against 59.5 ms at 128 x 5, 59.7 ms at 128 x 6, 61.3 ms at 128 x 8 and
// 68.5 ms at 128 x 9 (the spills grow with each step).
#ifndef HXG_FP32C_MULTI_THREADS
#define HXG_FP32C_MULTI_THREADS 128
#endif
#ifndef HXG_FP32C_MULTI_MIN_BLOCKS_FAST
#define HXG_FP32C_MULTI_MIN_BLOCKS_FAST 7
#endif
#ifndef HXG_FP32C_MULTI_MIN_BLOCKS
#define HXG_FP32C_MULTI_MIN_BLOCKS 5
#endif

template <int NF>
struct FreqSet {
  double lambda2[NF];   // (c/nu)^2
  double phase_k[NF];   // 2 lambda^2 * FD per unit of the FD sum
  double quarter_k[NF]; // the same in quarter turns (FP64 form)
  double quarter_i[NF]; // quarter turns per unit of the inner-shell FD
  double k_t[NF], k_p[NF];
  double tc_a[NF], tc_b[NF];
  double a_s[NF];       // A * |B_perp| scale of the variable-index emissivity
  int inner[NF];        // 1: the pass reads the inner-shell FD (its do_fd)
  double *out[NF][3];   // I, Q, U shell maps
};

// One pass's constants from its launch block.
__host__ __device__ __forceinline__ void freq_of_launch(const ShellLaunch &P, FreqSet<1> &Fq) {
  Fq.lambda2[0] = P.lambda2;
  Fq.phase_k[0] = P.phase_k;
  Fq.quarter_k[0] = P.quarter_k;
  Fq.quarter_i[0] = P.quarter_i;
  Fq.k_t[0] = P.k_t;
  Fq.k_p[0] = P.k_p;
  Fq.tc_a[0] = P.tc_a;
  Fq.tc_b[0] = P.tc_b;
  Fq.a_s[0] = P.a_s;
  Fq.inner[0] = 1;
  Fq.out[0][0] = P.out[2];
  Fq.out[0][1] = P.out[3];
  Fq.out[0][2] = P.out[4];
}

// Shell launches of one instantiation in one kernel: plan k takes the blocks before
// end[k] that the plans before it leave.  A kernel parameter, so that the plans'
// values stay in constant memory.
constexpr int kGroupPlans = 16;
template <int NF>
struct PlanGroup {
  unsigned end[kGroupPlans];
  ShellLaunch P[kGroupPlans];
  FreqSet<NF> F[kGroupPlans];
};
static_assert(sizeof(PlanGroup<3>) <= 32764, "kernel parameters");

// The plan of this block and the block's place in it.
template <int NF>
__device__ __forceinline__ int group_plan(const PlanGroup<NF> &G, unsigned &block) {
  int k = 0;
  while (k < kGroupPlans - 1 && blockIdx.x >= G.end[k]) ++k;
  block = blockIdx.x - (k ? G.end[k - 1] : 0u);
  return k;
}

// NESTED index of the shard's local pixel `local`: local pixels run through
// the shard's blocks in order.
__device__ __forceinline__ unsigned long long shard_nest(const ShellLaunch &P,
                                                         unsigned long long local) {
  if (P.nshards == 1) return local;
  const unsigned L = P.shard_log2;
  return (((local >> L) * P.nshards + P.shard) << L) + (local & ((1ull << L) - 1));
}

// Sample window [lo, hi) of one ray: the samples that can pass the
// spherical |pos| <= r_max and vertical z_min <= z <= z_max cuts
// (integrator.cc:179-182), from the roots of |o + u d|^2 = r_max^2 and
// o_z + u_z d = z_min / z_max, widened by two samples on each side.  Samples
// outside the window fail the cuts; the callers test the others.
__device__ __forceinline__ void ray_window(const ShellLaunch &P, double ux,
                                           double uy, double uz, long long &lo,
                                           long long &hi) {
  const double ox = P.obs[0], oy = P.obs[1], oz = P.obs[2];
  const double b = ox * ux + oy * uy + oz * uz;  // o.u
  const double c = (ox * ox + oy * oy + oz * oz) - P.gc_r_max * P.gc_r_max;
  const double disc = b * b - c;
  lo = 0;
  hi = 0;
  if (!(disc >= 0.)) return;  // the ray misses the r_max sphere
  const double sq = sqrt(disc);
  double da = -b - sq, db = -b + sq;
  if (uz > 0.) {
    da = fmax(da, (P.gc_z_min - oz) / uz);
    db = fmin(db, (P.gc_z_max - oz) / uz);
  } else if (uz < 0.) {
    da = fmax(da, (P.gc_z_max - oz) / uz);
    db = fmin(db, (P.gc_z_min - oz) / uz);
  } else if (oz < P.gc_z_min || oz > P.gc_z_max) {
    return;
  }
  if (!(da <= db)) return;
  // d_i = d_start + (i + 1/2) delta
  const double n = (double)P.step;
  const double xa = (da - P.d_start) / P.delta - 0.5, xb = (db - P.d_start) / P.delta - 0.5;
  const double fa = fmin(fmax(floor(xa) - 2., 0.), n);
  const double fb = fmin(fmax(ceil(xb) + 3., 0.), n);
  lo = (long long)fa;
  hi = (long long)fb;
}

// Sample range [ga, gb) of [i0, i1) in which the ray can be inside the grid
// box 0 < g < n - 1 on every axis (from the slab intersections in FP64,
// widened by two samples; the caller's own test decides each sample).
__device__ __forceinline__ void grid_window(const ShellLaunch &P, const DevGridGroup &G,
                                            const double g0[3], const double gv[3],
                                            int i0, int i1, int &ga, int &gb) {
  double da = -1e300, db = 1e300;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (gv[k] != 0.) {
      const double t0 = -g0[k] / gv[k], t1 = (G.gmax[k] - g0[k]) / gv[k];
      da = fmax(da, fmin(t0, t1));
      db = fmin(db, fmax(t0, t1));
    } else if (!(g0[k] > 0. && g0[k] < G.gmax[k])) {
      db = -1e300;
    }
  }
  ga = i1;
  gb = i1;
  if (!(da <= db)) return;
  const double xa = (da - P.d_start) / P.delta - 0.5, xb = (db - P.d_start) / P.delta - 0.5;
  ga = (int)fmin(fmax(floor(xa) - 2., (double)i0), (double)i1);
  gb = (int)fmin(fmax(ceil(xb) + 3., (double)ga), (double)i1);
}

// Kahan-compensated FP32 accumulator.
struct KahanF {
  float s, c;
  __device__ __forceinline__ void add(float v) {
    const float y = v - c;
    const float t = s + y;
    c = (t - s) - y;
    s = t;
  }
  __device__ __forceinline__ double value() const {
    return double(s) - double(c);
  }
};

// Two-level FP32 sum: a plain running sum over a block of samples, folded
// into a Kahan-compensated total by flush() (the caller flushes every 16
// sample indices).  The block sums' rounding (a few ulp of at most 16
// terms) is random from block to block, and the total is compensated.
struct BlockKahanF {
  float acc;
  KahanF tot;
  __device__ __forceinline__ void add(float v) { acc += v; }
  __device__ __forceinline__ void flush() {
    tot.add(acc);
    acc = 0.f;
  }
  __device__ __forceinline__ double value() const {
    KahanF t = tot;
    t.add(acc);
    return t.value();
  }
};

__device__ __forceinline__ double shfl_xor_d(double v, int o) {
  return __shfl_xor_sync(0xffffffffu, v, o);
}

// Combine the C chunk partial sums of each pixel: exclusive FD prefix over
// the chunks, rotation of each chunk's Q/U by 2*lambda^2*prefix, butterfly
// reduction over the pixel's C lanes, `stride` lanes apart.  All 32 lanes
// participate.
template <int NF>
__device__ __forceinline__ void combine_chunks_nf(const ShellLaunch &P, const FreqSet<NF> &Fq,
                                                  int c, double &dm, double &fd, double si[NF],
                                                  double sq[NF], double su[NF],
                                                  int stride = 1) {
  const int C = P.chunks;
  if (C == 1) return;
  // inclusive scan of fd within the segment
  double incl = fd;
  for (int o = 1; o < C; o <<= 1) {
    const double v = __shfl_up_sync(0xffffffffu, incl, o * stride);
    if (c >= o) incl += v;
  }
  double excl = __shfl_up_sync(0xffffffffu, incl, stride);
  if (c == 0) excl = 0.;
#pragma unroll
  for (int f = 0; f < NF; ++f) {
    if (P.do_sync && c > 0) {
      double sr, cr;
      sincos(2. * Fq.lambda2[f] * excl, &sr, &cr);
      const double q = sq[f] * cr - su[f] * sr;
      const double u = sq[f] * sr + su[f] * cr;
      sq[f] = q;
      su[f] = u;
    }
  }
  for (int o = C >> 1; o > 0; o >>= 1) {
    dm += shfl_xor_d(dm, o * stride);
    fd += shfl_xor_d(fd, o * stride);
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      si[f] += shfl_xor_d(si[f], o * stride);
      sq[f] += shfl_xor_d(sq[f], o * stride);
      su[f] += shfl_xor_d(su[f], o * stride);
    }
  }
}

// The adjoint's checkpoint of one pass, per (pixel, chunk): the Faraday depth
// of the chunks before it, and Q, U of it and the chunks after it in the
// pixel's frame (the chunk sums sq, su are in the chunk's own, which starts
// without the earlier chunks' rotation).  All 32 lanes participate; lanes that
// are not live store nothing and hold zeros.
__device__ __forceinline__ void store_checkpoint(const ShellLaunch &P, bool live,
                                                 unsigned long long nest, int c, int stride,
                                                 double fd, double sq, double su) {
  const int C = P.chunks;
  double incl = fd;
  for (int o = 1; o < C; o <<= 1) {
    const double v = __shfl_up_sync(0xffffffffu, incl, o * stride);
    if (c >= o) incl += v;
  }
  double before = C > 1 ? __shfl_up_sync(0xffffffffu, incl, stride) : 0.;
  if (c == 0) before = 0.;
  if (P.do_sync && c > 0) {
    double sr, cr;
    sincos(2. * P.lambda2 * before, &sr, &cr);
    const double q = sq * cr - su * sr;
    su = sq * sr + su * cr;
    sq = q;
  }
  for (int o = 1; o < C; o <<= 1) {
    const double vq = __shfl_down_sync(0xffffffffu, sq, o * stride);
    const double vu = __shfl_down_sync(0xffffffffu, su, o * stride);
    if (c + o < C) {
      sq += vq;
      su += vu;
    }
  }
  if (!live) return;
  const unsigned long long ci = nest * (unsigned long long)C + c;
  P.ck[3 * ci] = before;
  P.ck[3 * ci + 1] = sq;
  P.ck[3 * ci + 2] = su;
}

// cos(2*ipa), sin(2*ipa) of the IAU polarisation angle
// ipa = atan2(-e_theta.B, -e_phi.B) (integrator.cc:257-265), from the
// double-angle identities (no atan2).
template <typename T>
__device__ __forceinline__ void ipa2(T xv, T yv, T &c2, T &s2) {
  const T r2 = xv * xv + yv * yv;
  if (r2 > T(0)) {
    const T inv = T(1) / r2;
    c2 = (xv * xv - yv * yv) * inv;
    s2 = T(2) * xv * yv * inv;
  } else {
    c2 = T(1);
    s2 = T(0);
  }
}

}  // namespace hxg
