// AFAR stage kernels for sm_103a: reconstruct, BVD switch, adaptive flux, fused residual gather +
// SSP-RK3 update + boundary ghosts, plus the setup kernels that build the device operators.
//
// Device layout (one mesh):
//   per cell      W[Nc+Nb] (ghosts after the cells), U/U0[Nc], grad[2Nc], lim[Nc], si[Nc+Nb]
//   per slot      slot-major "[slot][ldc]" arrays, slot i of every cell contiguous so that a warp
//                 of consecutive cells reads one coalesced row per slot:
//                   sten[maxS]            global stencil cell ids
//                   cf[maxM]              signed face ids (+f+1 owner side, -(f+1) neighbour side)
//                   lsm[maxM]             least-squares gradient rows (M1, M2)
//                   sg[maxM], sr[maxM]    face offset from the cell centre; (delta r, fraction)
//                   wts[maxM*(maxS+1)]    O3 weights of the cell's side of each face
//   per face      on[Nf], fd[Nf] (face offsets from owner and neighbour), fs[Nf+Nb] (Sf, |Sf|),
//                 dtg[Nf] (CFL geometry), fv[2Nf] face values, flux[Nf+Nb]
// Every kernel here is one thread per cell or per face; every output element has one writer, so
// the stage is deterministic (no atomics except the min of the time step, which is exact).
#pragma once

#include "afar_policy.cuh"
#include "afar_tail_layout.h"

namespace afar {

struct StepCtl {
  unsigned long long dt_bits;  // running min of the CFL time step (bits of a non-negative double)
  double t;                    // simulated time
  double t_end;                // > 0: clip the last step to land on t_end
  double dt_fixed;             // > 0: fixed step, else CFL step
  double cfl;
  double last_dt;
  long long steps;
  unsigned err;  // bit 0: a bounded device wait gave up (the stage's results are not valid)
  double write_interval;  // > 0: land on its multiples like OpenFOAM's adjustableRunTime
  long long write_index;  // write times passed
  unsigned tiles_done;    // tiles of the last stage that are through (fused tail)
};

// The step of the current RK step: fixed or CFL, spread over the steps left to the next write time
// when write times are set, clipped to t_end; <= 0 means "no step".  The write-time rule is
// OpenFOAM's Time::adjustDeltaT for writeControl adjustableRunTime (the reference application
// sets each step with runTime.setDeltaT, cudaEuler2DmixO3RK3solver.cpp:44-48): with r the time to
// the next write, n = floor(r/dt - small) + 1 steps of r/n, the change held within [dt/5, 2 dt].
__device__ __forceinline__ double step_dt(const StepCtl* c) {
  // (the tests as integers: thread 0 of every update block takes this way, and each FP64 comparison
  // would hold its SM's FP64 pipe 16 clocks)
  double dt = gt_zero(c->dt_fixed) ? c->dt_fixed : __longlong_as_double((long long)c->dt_bits);
  if (gt_zero(c->write_interval)) {
    const double r = (double)(c->write_index + 1) * c->write_interval - c->t;
    if (r > 0.0) {
      const double nd = r / (floor(r / dt - 1e-15) + 1.0);
      dt = nd >= dt ? fmin(nd, 2.0 * dt) : fmax(nd, 0.2 * dt);
    }
  }
  if (gt_zero(c->t_end)) dt = fmin(dt, c->t_end - c->t);
  return dt;
}

// The SSP-RK3 coefficients of one stage: U = b1 Un + b2 U + b3 dt R (truncated decimals, reference
// GPUevolve.cu:222-225), their float-pair splits for the mixed policy (computed on the host so no
// thread converts them), and the first/last-stage flags.
struct StageCoef {
  double b1, b2, b3;
  float b1h, b1l, b2h, b2l;
  int first, last;
};

template <class P>
struct StageArgs {
  using S = typename P::S;
  using G = typename P::G;
  int Nc, Nf, Nb, ldc, maxS, maxM;
  // operators (read-only)
  const V2<double>* cellC;    // Nc+Nb cell centres, ghosts = boundary face centres
  const int2* on;             // Nf (owner, neighbour)
  const V4<G>* fd;            // Nf (xf-x_own, yf-y_own, xf-x_nei, yf-y_nei)
  const V4<G>* fs;            // Nf+Nb (Sfx, Sfy, magSf, 1/magSf; ref: 0)
  const V2<double>* dtg;      // Nf (delta r, fraction) of the CFL estimate (mixed: with the multi-point flux)
  const V2<double>* bn;       // Nb unit normal of each boundary face
  const uint8_t* btype;       // Nb cudaEulerBCs label
  const double* vol;          // Nc
  const double* vinv;         // Nc 1/V (policies without the reference's divisions)
  const float* vinvf;         // Nc 1/V as float (mixed)
  const uint8_t* nS;          // Nc stencil size
  const uint8_t* nM;          // Nc faces per cell (compact stencil size)
  const uint8_t* tileS;       // ceil(Nc/128): the largest stencil size of each 128-cell tile
  const int* sten;            // [maxS][ldc]
  const int* cf;              // [maxM][ldc]
  const V2<S>* lsm;           // [maxM][ldc]
  const V2<G>* sg;            // [maxM][ldc]
  const V2<S>* sr;            // [maxM][ldc]
  const S* wts;               // [maxM*(maxS+1)][ldc]
  const struct TileMaps* tmaps;  // mixed: TMA tensor maps of the operator rows (tile-staged reconstruct)
  // state and stage intermediates
  V4<typename P::W>* W;       // Nc+Nb
  V4<double>* U;              // Nc conserved state (mixed: DF4 float pairs, same 32 bytes)
  V4<double>* U0;             // Nc state at the start of the step (mixed: DF4)
  V4<G>* grad;                // 2Nc
  V4<S>* lim;                 // Nc
  int8_t* si;                 // 2(Nc+Nb): [2c] troubled-cell flag, [2c+1] final switch type
  V4<G>* fv;                  // 2Nf
  V4<typename P::F>* flux;    // Nf+Nb
  StepCtl* ctl;
  V4<double>* res_dbg;        // optional residual dump (parity hook)
  double R, Cv, invR, gamma;
  double Cp, gm1, gR;  // Cv + R, gamma - 1, gamma R (fp64)
  float gm1f, invRf;  // gamma - 1 and 1/R as floats (mixed)
  float Rf, Cvf, gRf;  // R, Cv and gamma*R as floats (mixed)
  double px, py;       // periods of a periodic mesh (0: none); setup kernels only
  const V2<float>* dtgf;  // Nf (delta r, fraction) as floats (mixed Courant estimate)
  // mixed: the fused stage tail (tail_body)
  const struct TailTile* tail;   // its tiles of tailT cells
  const int* thalo;              // [tile][kTailHalo] the cells across each tile's border
  const int* thcode;             // [tile][4][kTailHalo] the faces of their slots (see tail_body)
  const V2<typename P::G>* thsg; // [tile][4][kTailHalo] and sg of each
  const int* textra;             // [tile][kTailExtra] the tile's faces past its own
  const uint16_t* tlf;           // [maxM][ldc] local face of a cell's slot; bit 15: its neighbour side
  const int* tlist;              // [tile][kTailList] the 128-cell tiles its stencils reach
  unsigned* wflag;               // a bit for each cell: troubled (written by the reconstruct)
  V4<typename P::W>* W3[3];      // the state's buffers: W, and the outputs of the first two stages
  int nTail, tailT;              // its tiles and the cells of one
  // the optional multi-point face flux (ng > 0 points per face; 0: the face-centre flux)
  int ng;
  const S* wg;       // [(maxM*ng)*(maxS+1)][ldc] O3 weights at the face Gauss points, per cell slot
  const V2<G>* sgk;  // [maxM*ng][ldc] point minus cell centre, per cell slot
  const V2<G>* fgk;  // [Nf*ng] point minus face centre
  V4<G>* fvg;        // [2Nf*ng] face values at the points ((2f + side)*ng + k)
  G gw[4];           // the points' weights, normalised to sum to one
};

// limiterProcess (reference cudaLimiter.h:35-50), ref policy
__device__ __forceinline__ void limiter_process(float& limiter, float& phif, const float phic, const float phiMax,
                                                const float phiMin, const double gx, const double gy, const double dx,
                                                const double dy) {
  using S = float;
  phif = to_float(to_double(phic) + (gx * dx + gy * dy));
  const S d2 = phif - phic;
  const S d1 = (phif < phic) * (phiMin - phic) + (phif >= phic) * (phiMax - phic);
  S yy = fmn(S(2), S(0.5) * d1 / (d2 + (d2 >= S(0)) * AFAR_LIT(S, 1e-10) - (d2 < S(0)) * AFAR_LIT(S, 1e-10)));
  const bool valid = (fab(d2) >= AFAR_LIT(S, 1e-5));
  yy = valid * yy + (1 - valid) * S(1);
  limiter = fmn(limiter, yy);
}

// limiterProcess for the mixed policy: the same ratio with selects and the fast float division
// (2 ulp, MUFU reciprocal); the ratio feeds a min() with 2 and 1, so a rounding apart is all it
// changes.
__device__ __forceinline__ void limiter_process_fast(float& limiter, float& phif, const float phic, const float phiMax,
                                                     const float phiMin, const float gx, const float gy,
                                                     const float dx, const float dy) {
  phif = phic;
  phif += gx * dx + gy * dy;
  const float d2 = phif - phic;
  const float d1 = phif < phic ? phiMin - phic : phiMax - phic;
  const float yy = fabsf(d2) >= 1e-5f ? fminf(2.f, __fdividef(0.5f * d1, d2 + (d2 >= 0.f ? 1e-10f : -1e-10f))) : 1.f;
  limiter = fminf(limiter, yy);
}

// limiterProcess for the fp64 policy: the face's ratio min(2, d1 / (2 (d2 +- 1e-10))) as a fraction
// num/den of positive numbers (d1 and d2 have one sign), 1/1 where |d2| < 1e-5; the smaller of it and
// the cell's smallest so far is kept, told apart by their FP32 quotients (20 bits of each operand), or
// by cross-multiplication where those agree to 1e-5.  So a cell divides once for all variables
// (limiter_ratios) instead of once per face and variable, and no comparison or selection takes the
// FP64 pipe.  d2: the jump from the cell to phif.
struct LimiterRatio {
  double num, den;
  float q;
};
__device__ __forceinline__ void limiter_process_ratio(LimiterRatio& r, double& phif, double& d2, const double phic,
                                                      const double phiMax, const double phiMin, const double gx,
                                                      const double gy, const double dx, const double dy) {
  phif = phic + (gx * dx + gy * dy);
  d2 = phif - phic;
  const bool valid = abs_ge(d2, 1e-5);
  const double num = valid ? dabs_((neg_(d2) ? phiMin : phiMax) - phic) : 1.0;
  const double den = valid ? __fma_rn(2.0, dabs_(d2), 2e-10) : 1.0;
  const float q = __fdividef(top_float(num), top_float(den));
  bool less = q < r.q * 0.99999f;
  if (!less && !(q > r.q * 1.00001f)) less = dbits(num * r.den) < dbits(r.num * den);
  if (less) r = LimiterRatio{num, den, q};
}
// The four ratios of a cell from one reciprocal (simultaneous inversion, a few ulps from four
// divisions).  Every den is 1, or 2 |d2| + 2e-10 >= 2e-5 with d2 a jump of the flow over a face: the
// product of four leaves the range of double only where one of them is not finite, or for jumps of 1e77: those
// divide each, so that what is wrong with one variable stays with it.
__device__ __forceinline__ V4<double> limiter_ratios(const LimiterRatio& a, const LimiterRatio& b,
                                                     const LimiterRatio& c, const LimiterRatio& d) {
  const double ab = a.den * b.den, cd = c.den * d.den, all = ab * cd;
  if (!pos_normal(all)) return V4<double>{a.num / a.den, b.num / b.den, c.num / c.den, d.num / d.den};
  const double inv = rcp64(all);
  const double iab = inv * cd, icd = inv * ab;
  return V4<double>{a.num * (iab * b.den), b.num * (iab * a.den), c.num * (icd * d.den), d.num * (icd * c.den)};
}

// Faces per cell: triangles and quadrilaterals, the only cells the reference's quadrature accepts
// (d2GaussQuadrature.C:65-148); the stencil upload rejects larger compact stencils.
constexpr int kMaxFaces = 4;

// The mixed policy's FP32 Courant estimate of one internal face (setDeltaT, reference
// cudaFieldOperation.h:140-157): dt = CFL deltaR |Sf| / ((1-w)|U_o.Sf| + w|U_n.Sf| + c |Sf|),
// c = sqrt(gamma R ((1-w) T_o + w T_n)).  Every rounding is written out, so the fused stage-1 flux
// and the separate pass (afar_adjustTimeStep) give the same bits wherever the compiler places them.
__device__ __forceinline__ float courant_den_f32(const float fraction, const float magSf, const float Sfx,
                                                 const float Sfy, const V4<float>& Wo, const V4<float>& Wn,
                                                 const float gRf) {
  const float w0 = __fadd_rn(1.f, -fraction);
  const float unL = fabsf(__fmaf_rn(Wo.y, Sfx, __fmul_rn(Wo.z, Sfy)));
  const float unR = fabsf(__fmaf_rn(Wn.y, Sfx, __fmul_rn(Wn.z, Sfy)));
  const float c = __fsqrt_rn(__fmul_rn(gRf, __fmaf_rn(w0, Wo.w, __fmul_rn(fraction, Wn.w))));
  return __fmaf_rn(c, magSf, __fmaf_rn(w0, unL, __fmul_rn(fraction, unR)));
}
__device__ __forceinline__ float courant_dt_f32(const float cfl, const float deltaR, const float magSf,
                                                const float den) {
  return __fdiv_rn(__fmul_rn(__fmul_rn(cfl, deltaR), magSf), den);
}

// What the mixed reconstructs add for the fused stage tail (tail_body).
// The lanes of a warp of consecutive cells that have one.
__device__ __forceinline__ unsigned cell_lanes(const int c, const int Nc) {
  const int n = Nc - (c & ~31);
  return n >= 32 ? 0xffffffffu : (1u << n) - 1u;
}
// Troubled-cell flags as bits, a word for each warp's cells.
template <class P>
__device__ __forceinline__ void put_troubled(const StageArgs<P>& a, const int c, const int8_t flag) {
  const unsigned b = __ballot_sync(cell_lanes(c, a.Nc), flag != 0);
  if ((threadIdx.x & 31) == 0 && a.wflag) a.wflag[c >> 5] = b;
}
// DT (first stage): the Courant step's minimum over the internal faces that the warp's cells own, from
// the states at the start of the step: the cell's and, across each face, the stencil member of that
// face's slot.  The same estimate, to the bit, as in the stage-1 flux.  The geometry is loaded ahead
// (courant_load); one atomic a warp, which nothing waits for.
template <int NF>
struct CourantFaces {
  V4<float> fs[NF];
  V2<float> g[NF];
  float cfl;  // < 0: a fixed step
};
template <int NF, class P>
__device__ __forceinline__ void courant_load(CourantFaces<NF>& q, const StageArgs<P>& a, const int* fid,
                                             const bool* inner) {
  q.cfl = gt_zero(a.ctl->dt_fixed) ? -1.f : (float)a.ctl->cfl;
#pragma unroll
  for (int fi = 0; fi < NF; ++fi)
    if (inner[fi] && fid[fi] > 0) {
      q.fs[fi] = a.fs[fid[fi] - 1];
      q.g[fi] = a.dtgf[fid[fi] - 1];
    }
}
template <int NF, class P>
__device__ __forceinline__ void courant_min(const CourantFaces<NF>& q, const StageArgs<P>& a, const int c,
                                            const int* fid, const bool* inner, const V4<float>& wc,
                                            const V4<float>* wj) {
  if (q.cfl < 0.f) return;
  unsigned m = 0x7F800000u;
#pragma unroll
  for (int fi = 0; fi < NF; ++fi) {
    if (inner[fi] && fid[fi] > 0) {
      const V4<float> fs = q.fs[fi];
      const float dt =
          courant_dt_f32(q.cfl, q.g[fi].x, fs.z, courant_den_f32(q.g[fi].y, fs.z, fs.x, fs.y, wc, wj[fi], a.gRf));
      if (dt >= 0.f) m = min(m, __float_as_uint(dt));
    }
  }
  m = __reduce_min_sync(cell_lanes(c, a.Nc), m);
  if ((threadIdx.x & 31) == 0 && m < 0x7F800000u)
    atomicMin(&a.ctl->dt_bits, (unsigned long long)__double_as_longlong((double)__uint_as_float(m)));
}

// reconstruct, register-pass variant for the mixed policy (the autotuner's alternative to the
// tile-staged kernel): LS gradient, stencil min/max, raw limiter, O3 RBF face values of this
// cell's side of each internal face, troubled-cell flag.
// One pass over the stencil: each member's state is gathered once and feeds the gradient and
// min/max (compact members) and the O3 sums of every face side at once, all in registers.  The
// loads of a batch of members (indices, gathers, weights) are issued together, so several are in
// flight per thread; no shared memory, so occupancy is set by registers alone.  Every sum is
// still accumulated in stencil order, as in the reference.
template <class P, bool DT>
__device__ __forceinline__ void recon_reg_body(const StageArgs<P>& a, const V4<typename P::W>* W, const int blk) {
  pdl_wait();
  using S = typename P::S;
  using G = typename P::G;
  using WT = typename P::W;
  const int c = blk * blockDim.x + threadIdx.x;
  if (c >= a.Nc) return;
  const int ldc = a.ldc;
  const int nS = a.nS[c], nM = a.nM[c];
  const int wrow = a.maxS + 1;
  int fid[kMaxFaces];
  bool inner[kMaxFaces];
  V2<S> lm[kMaxFaces];
#pragma unroll
  for (int fi = 0; fi < kMaxFaces; ++fi) {
    fid[fi] = fi < nM ? a.cf[fi * ldc + c] : 1;
    inner[fi] = fi < nM && abs(fid[fi]) - 1 < a.Nf;
    lm[fi] = fi < nM ? a.lsm[fi * ldc + c] : V2<S>{S(0), S(0)};
  }
  const V4<WT> wc = W[c];
  const S pc = (S)wc.x, uxc = (S)wc.y, uyc = (S)wc.z, tc = (S)wc.w;
  // O3 sums in difference form: sum_i w_i phi_i = phi_c + sum_{i>0} w_i (phi_i - phi_c), since the
  // weights of every face side sum to one.  In FP32 this drops the error phi_c * (sum of the float
  // weights' rounding), which is the same every step and grows like a change of scheme; what
  // remains is rounding relative to the neighbour differences.
  G acc[kMaxFaces][4];
#pragma unroll
  for (int fi = 0; fi < kMaxFaces; ++fi) acc[fi][0] = acc[fi][1] = acc[fi][2] = acc[fi][3] = G(0);
  G gPx = 0, gPy = 0, gUxx = 0, gUxy = 0, gUyx = 0, gUyy = 0, gTx = 0, gTy = 0;
  S pMax = pc, pMin = pc, uxMax = uxc, uxMin = uxc, uyMax = uyc, uyMin = uyc, tMax = tc, tMin = tc;
  S pn[kMaxFaces];  // pressure of the cell across each face
  {  // members 0..3: the face neighbours (compact stencil) come first
    int j[kMaxFaces];
#pragma unroll
    for (int u = 0; u < kMaxFaces; ++u) j[u] = u < nS ? a.sten[u * ldc + c] : c;
    V4<WT> wj[kMaxFaces];
#pragma unroll
    for (int u = 0; u < kMaxFaces; ++u) wj[u] = W[j[u]];
    if constexpr (DT) {
      CourantFaces<kMaxFaces> cour;
      courant_load<kMaxFaces>(cour, a, fid, inner);
      courant_min<kMaxFaces>(cour, a, c, fid, inner, wc, wj);
    }
    S wv[kMaxFaces][kMaxFaces];
#pragma unroll
    for (int u = 0; u < kMaxFaces; ++u)
#pragma unroll
      for (int fi = 0; fi < kMaxFaces; ++fi)
        wv[u][fi] = (u < nS && inner[fi]) ? a.wts[(size_t)(fi * wrow + u + 1) * ldc + c] : S(0);
#pragma unroll
    for (int u = 0; u < kMaxFaces; ++u) {
      if (u < nS) {
        const S vx = (S)wj[u].x, vy = (S)wj[u].y, vz = (S)wj[u].z, vw = (S)wj[u].w;
        const S dp = vx - pc, dux = vy - uxc, duy = vz - uyc, dt = vw - tc;
        if (u < nM) {  // reference :148-169 and :190-205
          const S M1 = lm[u].x, M2 = lm[u].y;
          gPx += M1 * dp;
          gPy += M2 * dp;
          gUxx += M1 * dux;
          gUyx += M2 * dux;
          gUxy += M1 * duy;
          gUyy += M2 * duy;
          gTx += M1 * dt;
          gTy += M2 * dt;
          pMax = fmx(vx, pMax);
          pMin = fmn(vx, pMin);
          uxMax = fmx(vy, uxMax);
          uxMin = fmn(vy, uxMin);
          uyMax = fmx(vz, uyMax);
          uyMin = fmn(vz, uyMin);
          tMax = fmx(vw, tMax);
          tMin = fmn(vw, tMin);
          pn[u] = vx;
        }
#pragma unroll
        for (int fi = 0; fi < kMaxFaces; ++fi) {
          acc[fi][0] += wv[u][fi] * dp;
          acc[fi][1] += wv[u][fi] * dux;
          acc[fi][2] += wv[u][fi] * duy;
          acc[fi][3] += wv[u][fi] * dt;
        }
      }
    }
  }
  constexpr int U = sizeof(WT) == 4 ? 4 : 2;
  for (int ci0 = kMaxFaces; ci0 < nS; ci0 += U) {  // the rest of the stencil: O3 sums only
    int j[U];
#pragma unroll
    for (int u = 0; u < U; ++u) j[u] = (ci0 + u < nS) ? a.sten[(ci0 + u) * ldc + c] : c;
    V4<WT> wj[U];
#pragma unroll
    for (int u = 0; u < U; ++u) wj[u] = W[j[u]];
    S wv[U][kMaxFaces];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int fi = 0; fi < kMaxFaces; ++fi)
        wv[u][fi] = (ci0 + u < nS && inner[fi]) ? a.wts[(size_t)(fi * wrow + ci0 + u + 1) * ldc + c] : S(0);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (ci0 + u < nS) {
        const S dp = (S)wj[u].x - pc, dux = (S)wj[u].y - uxc, duy = (S)wj[u].z - uyc, dt = (S)wj[u].w - tc;
#pragma unroll
        for (int fi = 0; fi < kMaxFaces; ++fi) {
          acc[fi][0] += wv[u][fi] * dp;
          acc[fi][1] += wv[u][fi] * dux;
          acc[fi][2] += wv[u][fi] * duy;
          acc[fi][3] += wv[u][fi] * dt;
        }
      }
    }
  }
  pdl_next();
  a.grad[2 * c] = V4<G>{gPx, gPy, gUxx, gUxy};
  a.grad[2 * c + 1] = V4<G>{gUyx, gUyy, gTx, gTy};

  const S SMALL = AFAR_LIT(S, 1e-5), VSMALL = AFAR_LIT(S, 1e-10);
  V4<S> L;
  int8_t flag0;
  if (fab(tMax - tMin) < VSMALL) {  // reference :208-233
    L = V4<S>{S(1), S(1), S(1), S(1)};
#pragma unroll
    for (int fi = 0; fi < kMaxFaces; ++fi) {
      if (!inner[fi]) continue;
      const bool isNei = fid[fi] < 0;
      const int f = abs(fid[fi]) - 1;
      const V2<G> d = a.sg[fi * ldc + c];
      const G dx = d.x, dy = d.y;
      V4<G> o;
      o.x = (G)(pc) + gPx * dx + gPy * dy;
      o.y = (G)(uxc) + gUxx * dx + gUyx * dy;
      o.z = (G)(uyc) + gUxy * dx + gUyy * dy;
      o.w = (G)(tc) + gTx * dx + gTy * dy;
      a.fv[2 * f + isNei] = o;
    }
    flag0 = 0;
  } else {  // reference :235-314
    S lp = S(2), lux = S(2), luy = S(2), lt = S(2);
    S smooth = S(0);
    bool notTrouble = true;
#pragma unroll
    for (int fi = 0; fi < kMaxFaces; ++fi) {
      if (!inner[fi]) continue;
      const bool isNei = fid[fi] < 0;
      const int f = abs(fid[fi]) - 1;
      const V2<G> d = a.sg[fi * ldc + c];
      const G dx = d.x, dy = d.y;
      const V2<S> rf = a.sr[fi * ldc + c];
      const S deltaR = rf.x, fraction = rf.y;
      const G pf = (G)pc + acc[fi][0], uxf = (G)uxc + acc[fi][1], uyf = (G)uyc + acc[fi][2], tf = (G)tc + acc[fi][3];
      S phif;
      V4<G> o;
      limiter_process_fast(lp, phif, pc, pMax, pMin, gPx, gPy, dx, dy);
      o.x = pick<P>(fab(pMax - pMin) >= SMALL, fab(pMax - pMin) < SMALL, pf, phif);
      notTrouble = phif > S(0);
      smooth = fmx(smooth, __fdividef(fab((S(1) - fraction) * pc + fraction * pn[fi] - phif), deltaR) +
                               (pf <= S(0)) * AFAR_LIT(S, 1e20) + (phif <= S(0)) * AFAR_LIT(S, 1e20));
      limiter_process_fast(lux, phif, uxc, uxMax, uxMin, gUxx, gUyx, dx, dy);
      o.y = pick<P>(fab(uxMax - uxMin) >= SMALL, fab(uxMax - uxMin) < SMALL, uxf, phif);
      limiter_process_fast(luy, phif, uyc, uyMax, uyMin, gUxy, gUyy, dx, dy);
      o.z = pick<P>(fab(uyMax - uyMin) >= SMALL, fab(uyMax - uyMin) < SMALL, uyf, phif);
      limiter_process_fast(lt, phif, tc, tMax, tMin, gTx, gTy, dx, dy);
      o.w = pick<P>(fab(tMax - tMin) >= SMALL, fab(tMax - tMin) < SMALL, tf, phif);
      notTrouble = phif > S(0);
      a.fv[2 * f + isNei] = o;
    }
    L.x = fmx(lp, S(0)) * notTrouble;
    L.y = fmx(lux, S(0)) * notTrouble;
    L.z = fmx(luy, S(0)) * notTrouble;
    L.w = fmx(lt, S(0)) * notTrouble;
    smooth = __fdividef(smooth, S(0.5) * (pMax + pMin) * notTrouble + VSMALL);
    flag0 = (smooth > S(1));
  }
  a.lim[c] = L;
  a.si[2 * c] = flag0;
  put_troubled(a, c, flag0);
}

// ---------------------------------------------------------------- mixed reconstruct, tile-staged
// One CTA per 128-cell tile.  The tile's slice of every per-cell operator row (face ids, LS rows,
// face offsets, (dr, fraction), stencil ids, O3 weights) and the cells' own states are contiguous
// 128-element runs of the slot-major arrays, so the CTA fetches them with the TMA unit (one tiled
// load per array from its tensor map, one bulk copy of the states, two mbarriers) instead of
// per-thread loads: ~50 KB per tile in flight from seven lanes, while registers stay free for the
// stencil gathers, which hit L2.  One load per array rather than one per row: the fetch was bound
// by the number of copies issued, not by their bytes.
constexpr int kTile = 128;
// Test hooks of the tiles' bounded waits (afar_debug_wait_injection_at): the wait limit in SM clocks,
// and bytes added to the transaction count that a barrier of every tile expects (never issued, so
// that barrier cannot complete and its wait runs out): x, y of the reconstruct's two, z, w of the
// stage tail's.  g_tail_late_tx: bytes that the tail counts as arrived once its first wait has run out,
// as a copy does that lands after it.  2^31 clocks and no bytes in normal operation.
static __device__ long long g_tile_wait_limit = 1ll << 31;
static __device__ uint4 g_tile_extra_tx = {0, 0, 0, 0};
static __device__ unsigned g_tail_late_tx = 0;
// Tensor maps of the mixed policy's slot-major operator rows, one tiled TMA load per array and
// tile: face ids [maxM][ldc] and the LS / face-geometry rows (float pairs, as 2 ldc floats), boxes
// of 128 cells x maxM rows; stencil ids, a box of 128 cells x S rows for each stencil size S; O3
// weights [maxM][maxS+1][ldc], a box of 128 cells x rows 1..S x maxM slots for each S (row 0, the
// cell's own weight, drops out of the difference-form sums).  A tile loads the boxes of its own
// largest stencil, so no row past it is fetched.
struct TileMaps {
  CUtensorMap cf, lsm, sg, sr;
  CUtensorMap sten[AFAR_MAX_VALID_STENCIL_SIZE];
  CUtensorMap wts[AFAR_MAX_VALID_STENCIL_SIZE];
};
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, unsigned long long* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n" ::
          "r"(smem_addr(dst)),
      "l"(map), "r"(x), "r"(y), "r"(smem_addr(bar))
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z,
                                            unsigned long long* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
      "[%5];\n" ::"r"(smem_addr(dst)),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_addr(bar))
      : "memory");
}

struct ReconTile {
  unsigned off_cf, off_lsm, off_sg, off_sr, off_sten, off_wts, off_w, off_bar, bytes;
};
__host__ __device__ inline ReconTile recon_tile_layout(const int maxM, const int maxS) {
  ReconTile L;
  unsigned o = 0;
  L.off_cf = o;
  o += maxM * kTile * 4;
  L.off_lsm = o;
  o += maxM * kTile * 8;
  L.off_sg = o;
  o += maxM * kTile * 8;
  L.off_sr = o;
  o += maxM * kTile * 8;
  L.off_sten = o;
  o += maxS * kTile * 4;
  L.off_wts = o;
  o += maxM * (maxS + 1) * kTile * 4;
  L.off_w = o;
  o += kTile * 16;
  L.off_bar = o;  // two mbarriers: the gather inputs, then the rest
  L.bytes = o + 16;
  return L;
}

// Issues the loads of tile `blk` (lanes 0-6 of warp 0): six tiled TMA loads of its operator rows
// (TileMaps) and one bulk copy of its own states.  The x coordinate of every box is the tile's
// first cell (a multiple of 128 elements: 512 or 1024 bytes, so 16-byte aligned); boxes reaching
// past the row ends of the last tile read zeros and count their full size.  Two barriers: bar[0]
// covers what the stencil gathers need (face ids, stencil ids, own states), bar[1] the LS rows,
// face geometry and O3 weights, so the first gathers are in flight while the weights still stream
// in.  Smem rows hold 128 cells: face ids [maxM][128], stencil ids [S][128], LS and geometry
// [maxM][128] pairs, weights [maxM][S][128] (S = the tile's largest stencil).
template <bool EARLY, class P>
__device__ __forceinline__ void recon_tile_fetch(const StageArgs<P>& a, const V4<typename P::W>* W, const int blk,
                                                 const ReconTile& L,
                                                 unsigned char* sm, unsigned long long* bar) {
  const int lane = threadIdx.x;
  const int c0 = blk * kTile;
  const int M = a.maxM, S = a.tileS[blk];
  const TileMaps* tm = a.tmaps;
  if (lane == 0) {
    const unsigned nw = (unsigned)min(kTile, a.Nc - c0);  // cells of the tile
    mbar_arrive_expect_tx(bar, kTile * 4 * (M + S) + nw * 16 + g_tile_extra_tx.x);
    mbar_arrive_expect_tx(bar + 1, kTile * 8 * 3 * M + kTile * 4 * S * M + g_tile_extra_tx.y);
  }
  __syncwarp();
  switch (lane) {
    case 0: tma_load_2d(sm + L.off_cf, &tm->cf, c0, 0, bar); break;
    case 1: tma_load_2d(sm + L.off_sten, &tm->sten[S - 1], c0, 0, bar); break;
    case 2:  // (the one copy of what the kernel before has written)
      pdl_wait<EARLY>();
      bulk_to_smem(sm + L.off_w, W + c0, (unsigned)min(kTile, a.Nc - c0) * 16u, bar);
      break;
    case 3: tma_load_2d(sm + L.off_lsm, &tm->lsm, 2 * c0, 0, bar + 1); break;
    case 4: tma_load_2d(sm + L.off_sg, &tm->sg, 2 * c0, 0, bar + 1); break;
    case 5: tma_load_2d(sm + L.off_sr, &tm->sr, 2 * c0, 0, bar + 1); break;
    case 6: tma_load_3d(sm + L.off_wts, &tm->wts[S - 1], c0, 1, 0, bar + 1); break;
    default: break;
  }
}

// reconstruct (reference cudaLimiter.h:53-316) for the mixed policy from the staged tile: LS
// gradient, stencil min/max, raw limiter, O3 RBF face values of this cell's side of each internal
// face, troubled-cell flag.  One pass over the stencil: each member's state is gathered once (in
// batches of 8, all in flight) and feeds the gradient and min/max (compact members) and the O3 sums
// of every face side; every sum is accumulated in stencil order, as in the reference.  NF: the
// largest number of faces of a cell (3 on all-triangle meshes, else 4).
template <class P, int NF, bool DT, bool EARLY = true>
__device__ __forceinline__ void recon_tile_body(const StageArgs<P>& a, const V4<typename P::W>* W, const int blk,
                                                unsigned char* sm) {
  using S = typename P::S;
  using G = typename P::G;
  using WT = typename P::W;
  const ReconTile L = recon_tile_layout(a.maxM, a.maxS);
  unsigned long long* bar = reinterpret_cast<unsigned long long*>(sm + L.off_bar);
  const int t = threadIdx.x;
  if (t == 0) {
    mbar_init(bar, 1);
    mbar_init(bar + 1, 1);
  }
  __syncthreads();
  if (t < 32) recon_tile_fetch<EARLY>(a, W, blk, L, sm, bar);
  const int c = blk * kTile + t;
  int nS = c < a.Nc ? a.nS[c] : 0, nM = c < a.Nc ? a.nM[c] : 0;
  pdl_wait<EARLY>();
  const long long limit = g_tile_wait_limit;
  // A lane whose wait runs out (each polls by its own clock) marks the step invalid, waits once more, since every
  // copy into the block's shared memory must have landed before the block ends, and goes on with the others of its
  // warp, whom it meets below (courant_min, put_troubled): without stencil and faces where the lists are still
  // missing, so that it follows no index that is not one.
  auto arrived = [&](unsigned long long* b) {
    if (mbar_wait_bounded(b, 0, limit)) return true;
    atomicOr(&a.ctl->err, 1u);
    return mbar_wait_bounded(b, 0, limit);
  };
  if (!arrived(bar)) nS = nM = 0;
  if (c >= a.Nc) {
    arrived(bar + 1);
    return;
  }
  const int* s_cf = reinterpret_cast<const int*>(sm + L.off_cf);
  const V2<S>* s_lsm = reinterpret_cast<const V2<S>*>(sm + L.off_lsm);
  const V2<G>* s_sg = reinterpret_cast<const V2<G>*>(sm + L.off_sg);
  const V2<S>* s_sr = reinterpret_cast<const V2<S>*>(sm + L.off_sr);
  const int* s_sten = reinterpret_cast<const int*>(sm + L.off_sten);
  const S* s_wts = reinterpret_cast<const S*>(sm + L.off_wts);
  const V4<WT>* s_w = reinterpret_cast<const V4<WT>*>(sm + L.off_w);
  const int wrow = a.tileS[blk];  // weight rows of a face slot in shared memory (members 1..S)

  int fid[NF];
  bool inner[NF];
#pragma unroll
  for (int fi = 0; fi < NF; ++fi) {
    fid[fi] = fi < nM ? s_cf[fi * kTile + t] : 1;
    inner[fi] = fi < nM && abs(fid[fi]) - 1 < a.Nf;
  }
  const V4<WT> wc = s_w[t];
  const S pc = (S)wc.x, uxc = (S)wc.y, uyc = (S)wc.z, tc = (S)wc.w;
  constexpr int U = 8;
  V4<WT> wj[U];  // the first batch of stencil states, gathered before the weights have landed
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (u < nS) wj[u] = W[s_sten[u * kTile + t]];
  CourantFaces<NF> cour;
  if constexpr (DT) courant_load<NF>(cour, a, fid, inner);
  arrived(bar + 1);
  if constexpr (DT) courant_min<NF>(cour, a, c, fid, inner, wc, wj);
  // O3 weights of boundary-face and missing slots are zero in the operator rows (setup), so only
  // slots past this mesh's largest cell (a batch may stage fewer rows than NF) are skipped
  const int nfm = a.maxM;
  G acc[NF][4];  // O3 sums in difference form, as in recon_reg_body
#pragma unroll
  for (int fi = 0; fi < NF; ++fi) acc[fi][0] = acc[fi][1] = acc[fi][2] = acc[fi][3] = G(0);
  G gPx = 0, gPy = 0, gUxx = 0, gUxy = 0, gUyx = 0, gUyy = 0, gTx = 0, gTy = 0;
  S pMax = pc, pMin = pc, uxMax = uxc, uxMin = uxc, uyMax = uyc, uyMin = uyc, tMax = tc, tMin = tc;
  S pn[NF];  // pressure of the cell across each face
#pragma unroll
  for (int fi = 0; fi < NF; ++fi) pn[fi] = S(0);
  for (int ci0 = 0; ci0 < nS; ci0 += U) {
    if (ci0 > 0) {
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (ci0 + u < nS) wj[u] = W[s_sten[(ci0 + u) * kTile + t]];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int ci = ci0 + u;
      if (ci < nS) {
        const S vx = (S)wj[u].x, vy = (S)wj[u].y, vz = (S)wj[u].z, vw = (S)wj[u].w;
        const S dp = vx - pc, dux = vy - uxc, duy = vz - uyc, dt = vw - tc;
        if (ci < nM) {  // the face neighbours (compact stencil) come first: reference :148-169, :190-205
          const V2<S> lm = s_lsm[ci * kTile + t];
          const S M1 = lm.x, M2 = lm.y;
          gPx += M1 * dp;
          gPy += M2 * dp;
          gUxx += M1 * dux;
          gUyx += M2 * dux;
          gUxy += M1 * duy;
          gUyy += M2 * duy;
          gTx += M1 * dt;
          gTy += M2 * dt;
          pMax = fmx(vx, pMax);
          pMin = fmn(vx, pMin);
          uxMax = fmx(vy, uxMax);
          uxMin = fmn(vy, uxMin);
          uyMax = fmx(vz, uyMax);
          uyMin = fmn(vz, uyMin);
          tMax = fmx(vw, tMax);
          tMin = fmn(vw, tMin);
#pragma unroll
          for (int fi = 0; fi < NF; ++fi)
            if (fi == ci) pn[fi] = vx;
        }
#pragma unroll
        for (int fi = 0; fi < NF; ++fi) {
          const S wv = fi < nfm ? s_wts[(fi * wrow + ci) * kTile + t] : S(0);
          acc[fi][0] += wv * dp;
          acc[fi][1] += wv * dux;
          acc[fi][2] += wv * duy;
          acc[fi][3] += wv * dt;
        }
      }
    }
  }
  pdl_next<EARLY>();
  a.grad[2 * c] = V4<G>{gPx, gPy, gUxx, gUxy};
  a.grad[2 * c + 1] = V4<G>{gUyx, gUyy, gTx, gTy};

  const S SMALL = AFAR_LIT(S, 1e-5), VSMALL = AFAR_LIT(S, 1e-10);
  V4<S> Lm;
  int8_t flag0;
  if (fab(tMax - tMin) < VSMALL) {  // reference :208-233
    Lm = V4<S>{S(1), S(1), S(1), S(1)};
#pragma unroll
    for (int fi = 0; fi < NF; ++fi) {
      if (!inner[fi]) continue;
      const bool isNei = fid[fi] < 0;
      const int f = abs(fid[fi]) - 1;
      const V2<G> d = s_sg[fi * kTile + t];
      const G dx = d.x, dy = d.y;
      V4<G> o;
      o.x = (G)(pc) + gPx * dx + gPy * dy;
      o.y = (G)(uxc) + gUxx * dx + gUyx * dy;
      o.z = (G)(uyc) + gUxy * dx + gUyy * dy;
      o.w = (G)(tc) + gTx * dx + gTy * dy;
      a.fv[2 * f + isNei] = o;
    }
    flag0 = 0;
  } else {  // reference :235-314
    S lp = S(2), lux = S(2), luy = S(2), lt = S(2);
    S smooth = S(0);
    bool notTrouble = true;
#pragma unroll
    for (int fi = 0; fi < NF; ++fi) {
      if (!inner[fi]) continue;
      const bool isNei = fid[fi] < 0;
      const int f = abs(fid[fi]) - 1;
      const V2<G> d = s_sg[fi * kTile + t];
      const G dx = d.x, dy = d.y;
      const V2<S> rf = s_sr[fi * kTile + t];
      const S deltaR = rf.x, fraction = rf.y;
      const G pf = (G)pc + acc[fi][0], uxf = (G)uxc + acc[fi][1], uyf = (G)uyc + acc[fi][2], tf = (G)tc + acc[fi][3];
      S phif;
      V4<G> o;
      limiter_process_fast(lp, phif, pc, pMax, pMin, gPx, gPy, dx, dy);
      o.x = pick<P>(fab(pMax - pMin) >= SMALL, fab(pMax - pMin) < SMALL, pf, phif);
      notTrouble = phif > S(0);
      smooth = fmx(smooth, __fdividef(fab((S(1) - fraction) * pc + fraction * pn[fi] - phif), deltaR) +
                               (pf <= S(0)) * AFAR_LIT(S, 1e20) + (phif <= S(0)) * AFAR_LIT(S, 1e20));
      limiter_process_fast(lux, phif, uxc, uxMax, uxMin, gUxx, gUyx, dx, dy);
      o.y = pick<P>(fab(uxMax - uxMin) >= SMALL, fab(uxMax - uxMin) < SMALL, uxf, phif);
      limiter_process_fast(luy, phif, uyc, uyMax, uyMin, gUxy, gUyy, dx, dy);
      o.z = pick<P>(fab(uyMax - uyMin) >= SMALL, fab(uyMax - uyMin) < SMALL, uyf, phif);
      limiter_process_fast(lt, phif, tc, tMax, tMin, gTx, gTy, dx, dy);
      o.w = pick<P>(fab(tMax - tMin) >= SMALL, fab(tMax - tMin) < SMALL, tf, phif);
      notTrouble = phif > S(0);
      a.fv[2 * f + isNei] = o;
    }
    Lm.x = fmx(lp, S(0)) * notTrouble;
    Lm.y = fmx(lux, S(0)) * notTrouble;
    Lm.z = fmx(luy, S(0)) * notTrouble;
    Lm.w = fmx(lt, S(0)) * notTrouble;
    smooth = __fdividef(smooth, S(0.5) * (pMax + pMin) * notTrouble + VSMALL);
    flag0 = (smooth > S(1));
  }
  a.lim[c] = Lm;
  a.si[2 * c] = flag0;
  put_troubled(a, c, flag0);
}

// reconstruct for the ref policy: the stencil values are staged in shared memory in batches (indices,
// then gathers), then each face side's O3 sum runs over the staged values with its weights loaded
// eight at a time.  The policy is bound by the FP64 pipe, so the kernel keeps the per-face loop (no
// work on missing face slots) and a small register set.
__device__ __forceinline__ void recon_ref_body(const StageArgs<PolicyRef>& a, const int blk) {
  using P = PolicyRef;
  using S = typename P::S;
  using G = typename P::G;
  using WT = typename P::W;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V4<S>* sv = reinterpret_cast<V4<S>*>(smem_raw);  // [maxS][blockDim] staged stencil values
  const int t = threadIdx.x, B = blockDim.x;
  const int c = blk * B + t;
  if (c >= a.Nc) return;
  const int ldc = a.ldc;
  const int nS = a.nS[c], nM = a.nM[c];
  const V4<WT> wc = a.W[c];
  const S pc = to_float(wc.x), uxc = to_float(wc.y), uyc = to_float(wc.z), tc = to_float(wc.w);
  constexpr int GB = 4;
  for (int i0 = 0; i0 < nS; i0 += GB) {
    int j[GB];
#pragma unroll
    for (int u = 0; u < GB; ++u) j[u] = (i0 + u < nS) ? a.sten[(i0 + u) * ldc + c] : c;
    V4<WT> wj[GB];
#pragma unroll
    for (int u = 0; u < GB; ++u) wj[u] = a.W[j[u]];
#pragma unroll
    for (int u = 0; u < GB; ++u)
      if (i0 + u < nS) sv[(i0 + u) * B + t] = V4<S>{to_float(wj[u].x), to_float(wj[u].y), to_float(wj[u].z), to_float(wj[u].w)};
  }

  G gPx = 0, gPy = 0, gUxx = 0, gUxy = 0, gUyx = 0, gUyy = 0, gTx = 0, gTy = 0;
  for (int i = 0; i < nM; ++i) {  // reference :148-169
    const V2<S> m = a.lsm[i * ldc + c];
    const S M1 = m.x, M2 = m.y;
    const V4<S> v = sv[i * B + t];
    S dphi = v.x - pc;
    gPx += to_double(M1 * dphi);
    gPy += to_double(M2 * dphi);
    dphi = v.y - uxc;
    gUxx += to_double(M1 * dphi);
    gUyx += to_double(M2 * dphi);
    dphi = v.z - uyc;
    gUxy += to_double(M1 * dphi);
    gUyy += to_double(M2 * dphi);
    dphi = v.w - tc;
    gTx += to_double(M1 * dphi);
    gTy += to_double(M2 * dphi);
  }
  a.grad[2 * c] = V4<G>{gPx, gPy, gUxx, gUxy};
  a.grad[2 * c + 1] = V4<G>{gUyx, gUyy, gTx, gTy};

  S pMax = pc, pMin = pc, uxMax = uxc, uxMin = uxc, uyMax = uyc, uyMin = uyc, tMax = tc, tMin = tc;
  for (int i = 0; i < nM; ++i) {  // reference :190-205
    const V4<S> v = sv[i * B + t];
    pMax = fmx(v.x, pMax);
    pMin = fmn(v.x, pMin);
    uxMax = fmx(v.y, uxMax);
    uxMin = fmn(v.y, uxMin);
    uyMax = fmx(v.z, uyMax);
    uyMin = fmn(v.z, uyMin);
    tMax = fmx(v.w, tMax);
    tMin = fmn(v.w, tMin);
  }

  const S SMALL = AFAR_LIT(S, 1e-5), VSMALL = AFAR_LIT(S, 1e-10);
  V4<S> L;
  int8_t flag0;
  if (fab(tMax - tMin) < VSMALL) {  // reference :208-233
    L = V4<S>{S(1), S(1), S(1), S(1)};
    for (int fi = 0; fi < nM; ++fi) {
      int f = a.cf[fi * ldc + c];
      const bool isNei = (f < 0);
      f = abs(f) - 1;
      if (f >= a.Nf) continue;
      const V2<G> d = a.sg[fi * ldc + c];
      const G dx = d.x, dy = d.y;
      V4<G> o;
      o.x = to_double(pc) + gPx * dx + gPy * dy;
      o.y = to_double(uxc) + gUxx * dx + gUyx * dy;
      o.z = to_double(uyc) + gUxy * dx + gUyy * dy;
      o.w = to_double(tc) + gTx * dx + gTy * dy;
      a.fv[2 * f + isNei] = o;
    }
    flag0 = 0;
  } else {  // reference :235-314
    S lp = S(2), lux = S(2), luy = S(2), lt = S(2);
    S smooth = S(0);
    bool notTrouble = true;
    for (int fi = 0; fi < nM; ++fi) {
      int f = a.cf[fi * ldc + c];
      const bool isNei = (f < 0);
      f = abs(f) - 1;
      if (f >= a.Nf) continue;
      const V2<G> d = a.sg[fi * ldc + c];
      const G dx = d.x, dy = d.y;
      const V2<S> rf = a.sr[fi * ldc + c];
      const S deltaR = rf.x, fraction = rf.y;
      const S* w = a.wts + (size_t)(fi * (a.maxS + 1)) * ldc + c;
      S wk = w[0];
      G pf = to_double(wk * pc);
      G uxf = to_double(wk * uxc);
      G uyf = to_double(wk * uyc);
      G tf = to_double(wk * tc);
      for (int ci0 = 0; ci0 < nS; ci0 += 8) {
        S wb[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) wb[u] = (ci0 + u < nS) ? w[(size_t)(ci0 + u + 1) * ldc] : S(0);
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          if (ci0 + u < nS) {
            const V4<S> v = sv[(ci0 + u) * B + t];
            pf += to_double(wb[u] * v.x);
            uxf += to_double(wb[u] * v.y);
            uyf += to_double(wb[u] * v.z);
            tf += to_double(wb[u] * v.w);
          }
        }
      }
      const S pnb = sv[fi * B + t].x;
      S phif;
      V4<G> o;
      limiter_process(lp, phif, pc, pMax, pMin, gPx, gPy, dx, dy);
      o.x = blend64(fab(pMax - pMin) >= SMALL, fab(pMax - pMin) < SMALL, pf, to_double(phif));
      notTrouble = phif > S(0);
      smooth = fmx(smooth, fab((S(1) - fraction) * pc + fraction * pnb - phif) / deltaR + le_zero(pf) * AFAR_LIT(S, 1e20) +
                               (phif <= S(0)) * AFAR_LIT(S, 1e20));
      limiter_process(lux, phif, uxc, uxMax, uxMin, gUxx, gUyx, dx, dy);
      o.y = blend64(fab(uxMax - uxMin) >= SMALL, fab(uxMax - uxMin) < SMALL, uxf, to_double(phif));
      limiter_process(luy, phif, uyc, uyMax, uyMin, gUxy, gUyy, dx, dy);
      o.z = blend64(fab(uyMax - uyMin) >= SMALL, fab(uyMax - uyMin) < SMALL, uyf, to_double(phif));
      limiter_process(lt, phif, tc, tMax, tMin, gTx, gTy, dx, dy);
      o.w = blend64(fab(tMax - tMin) >= SMALL, fab(tMax - tMin) < SMALL, tf, to_double(phif));
      notTrouble = phif > S(0);
      a.fv[2 * f + isNei] = o;
    }
    L.x = fmx(lp, S(0)) * notTrouble;
    L.y = fmx(lux, S(0)) * notTrouble;
    L.z = fmx(luy, S(0)) * notTrouble;
    L.w = fmx(lt, S(0)) * notTrouble;
    smooth = smooth / (S(0.5) * (pMax + pMin) * notTrouble + VSMALL);
    flag0 = (smooth > S(1));
  }
  a.lim[c] = L;
  a.si[2 * c] = flag0;
}

// reconstruct for the fp64 policy.  The FP64 pipe bounds it (one warp instruction in 16 clocks of the
// SM), so the kernel is laid out by its FP64 instructions: the O3 sums (4 products a member and face
// side) are most of them, every comparison, minimum and selection runs on integers, and the limiter
// divides once per cell (limiter_process_ratio).  Only the compact stencil (the face neighbours) is
// staged in shared memory: the gradient, the min/max and the uniform-cell test need nothing else, and
// the O3 loop of a cell that is not uniform reads the other members from memory.  500k triangles, no
// uniform cells: 628 us a launch with FP64 comparisons and a division per face and variable, 352 now
// (364 FP64 warp instructions, 180 of them the O3 sums; the pipe 86% busy).
__device__ __forceinline__ void recon_fp64_body(const StageArgs<PolicyFP64>& a, const int blk) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V4<double>* sv = reinterpret_cast<V4<double>*>(smem_raw);  // [maxM][blockDim] the face neighbours' states
  const int t = threadIdx.x, B = blockDim.x;
  const int c = blk * B + t;
  if (c >= a.Nc) return;
  const int ldc = a.ldc;
  const int nS = a.nS[c], nM = a.nM[c];
  const V4<double> wc = a.W[c];
  {
    int j[kMaxFaces];
#pragma unroll
    for (int u = 0; u < kMaxFaces; ++u) j[u] = u < nM ? a.sten[u * ldc + c] : c;
    V4<double> wj[kMaxFaces];
#pragma unroll
    for (int u = 0; u < kMaxFaces; ++u) wj[u] = a.W[j[u]];
#pragma unroll
    for (int u = 0; u < kMaxFaces; ++u)
      if (u < nM) sv[u * B + t] = wj[u];
  }
  // reference :148-169 (least-squares gradient) and :190-205 (min and max over the face neighbours)
  double gPx = 0, gPy = 0, gUxx = 0, gUxy = 0, gUyx = 0, gUyy = 0, gTx = 0, gTy = 0;
  V4<double> mx = wc, mn = wc;
  for (int i = 0; i < nM; ++i) {
    const V2<double> m = a.lsm[i * ldc + c];
    const V4<double> v = sv[i * B + t];
    double dphi = v.x - wc.x;
    gPx += m.x * dphi;
    gPy += m.y * dphi;
    dphi = v.y - wc.y;
    gUxx += m.x * dphi;
    gUyx += m.y * dphi;
    dphi = v.z - wc.z;
    gUxy += m.x * dphi;
    gUyy += m.y * dphi;
    dphi = v.w - wc.w;
    gTx += m.x * dphi;
    gTy += m.y * dphi;
    mx = V4<double>{dmax_(v.x, mx.x), dmax_(v.y, mx.y), dmax_(v.z, mx.z), dmax_(v.w, mx.w)};
    mn = V4<double>{dmin_(v.x, mn.x), dmin_(v.y, mn.y), dmin_(v.z, mn.z), dmin_(v.w, mn.w)};
  }
  a.grad[2 * c] = V4<double>{gPx, gPy, gUxx, gUxy};
  a.grad[2 * c + 1] = V4<double>{gUyx, gUyy, gTx, gTy};

  V4<double> L{1.0, 1.0, 1.0, 1.0};
  int8_t flag0 = 0;
  const double rangeT = mx.w - mn.w;
  const bool flat = abs_lt(rangeT, 1e-10);  // reference :208-233: linear face values, no limiting
  // which variables take the O3 value (the reference's threshold on their range)
  const bool o3x = abs_ge(mx.x - mn.x, 1e-5), o3y = abs_ge(mx.y - mn.y, 1e-5), o3z = abs_ge(mx.z - mn.z, 1e-5),
             o3w = abs_ge(rangeT, 1e-5);
  LimiterRatio lp{2.0, 1.0, 2.f}, lux = lp, luy = lp, lt = lp;
  double smooth = 0.0;
  bool notTrouble = true;
  for (int fi = 0; fi < nM; ++fi) {
    int f = a.cf[fi * ldc + c];
    const bool isNei = (f < 0);
    f = abs(f) - 1;
    if (f >= a.Nf) continue;
    const V2<double> d = a.sg[fi * ldc + c];
    V4<double> o;
    if (flat) {
      o.x = wc.x + gPx * d.x + gPy * d.y;
      o.y = wc.y + gUxx * d.x + gUyx * d.y;
      o.z = wc.z + gUxy * d.x + gUyy * d.y;
      o.w = wc.w + gTx * d.x + gTy * d.y;
    } else {  // reference :235-314
      const V2<double> rf = a.sr[fi * ldc + c];  // (1 / delta r, fraction)
      const double* w = a.wts + (size_t)(fi * (a.maxS + 1)) * ldc + c;
      const double w0 = w[0];
      double pf = w0 * wc.x, uxf = w0 * wc.y, uyf = w0 * wc.z, tf = w0 * wc.w;
      // weights, stencil ids and the members past the compact stencil in batches of four (those from
      // memory, the compact ones staged); sums in stencil order
      for (int ci0 = 0; ci0 < nS; ci0 += 4) {
        double wb[4];
        int jj[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int ci = ci0 + u;
          wb[u] = ci < nS ? w[(size_t)(ci + 1) * ldc] : 0.0;
          jj[u] = (ci < nS && ci >= nM) ? a.sten[ci * ldc + c] : c;
        }
        V4<double> wv[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) wv[u] = a.W[jj[u]];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int ci = ci0 + u;
          if (ci < nS) {
            const V4<double> v = ci < nM ? sv[ci * B + t] : wv[u];
            pf += wb[u] * v.x;
            uxf += wb[u] * v.y;
            uyf += wb[u] * v.z;
            tf += wb[u] * v.w;
          }
        }
      }
      const double pnb = sv[fi * B + t].x;
      double phif, d2;
      limiter_process_ratio(lp, phif, d2, wc.x, mx.x, mn.x, gPx, gPy, d.x, d.y);
      o.x = o3x ? pf : phif;
      // |(1 - w) p_c + w p_n - p_f| / delta r
      double jump = dabs_(rf.y * (pnb - wc.x) - d2) * rf.x;
      if (le_zero(pf) || le_zero(phif)) jump += le_zero(pf) && le_zero(phif) ? 2e20 : 1e20;
      smooth = dnan_(jump) ? smooth : dbits(jump) > dbits(smooth) ? jump : smooth;
      limiter_process_ratio(lux, phif, d2, wc.y, mx.y, mn.y, gUxx, gUyx, d.x, d.y);
      o.y = o3y ? uxf : phif;
      limiter_process_ratio(luy, phif, d2, wc.z, mx.z, mn.z, gUxy, gUyy, d.x, d.y);
      o.z = o3z ? uyf : phif;
      limiter_process_ratio(lt, phif, d2, wc.w, mx.w, mn.w, gTx, gTy, d.x, d.y);
      o.w = o3w ? tf : phif;
      notTrouble = gt_zero(phif);
    }
    a.fv[2 * f + isNei] = o;
  }
  if (!flat) {
    if (notTrouble)
      L = limiter_ratios(lp, lux, luy, lt);
    else
      L = V4<double>{0.0, 0.0, 0.0, 0.0};
    const double scale = notTrouble ? 0.5 * (mx.x + mn.x) + 1e-10 : 1e-10;
    flag0 = !neg_(scale) && dbits(smooth) > dbits(scale);  // smooth / scale > 1
  }
  a.lim[c] = L;
  a.si[2 * c] = flag0;
}

__device__ __forceinline__ double mul64(const double a, const double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add64(const double a, const double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub64(const double a, const double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double fma64(const double a, const double b, const double c) { return __fma_rn(a, b, c); }
// w + lim (ga dx + gb dy): the limited linear (TVD) value
__device__ __forceinline__ double tvd64(const double w, const double lim, const double ga, const double gb,
                                        const double dx, const double dy) {
  return fma64(lim, fma64(ga, dx, mul64(gb, dy)), w);
}

// Limiter maps (reference cudaLimiter.h:14-32)
template <class S>
__device__ __forceinline__ S to_bj(const S y) {
  return gmn(S(2) * y, S(1));
}
template <class S>
__device__ __forceinline__ S to_venkat(const S y) {
  const S num = y * y + y + AFAR_LIT(S, 1e-10), den = y * y + S(0.5) + S(0.5) * y + AFAR_LIT(S, 1e-10);
  if constexpr (std::is_same<S, double>::value)
    return dmin_(num * rcp64(den), 1.0);
  else
    return fmn(num / den, S(1));
}

// BVDindicator (reference cudaLimiter.h:319-464): stencil flag counts, BVD test on T, final
// switch type, limiter transform.
template <class P>
__device__ __forceinline__ void bvd_body(const StageArgs<P>& a, const int blk) {
  using S = typename P::S;
  using G = typename P::G;
  const int c = blk * blockDim.x + threadIdx.x;
  if (c >= a.Nc) return;
  const int ldc = a.ldc;
  const int nS = a.nS[c], nM = a.nM[c];
  int8_t shockType = a.si[2 * c];
  int8_t shockTypeExt = shockType;
  // troubled-cell flags of the stencil, eight index loads then eight flag loads at a time
  for (int i0 = 0; i0 < nS; i0 += 8) {
    int j[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) j[u] = (i0 + u < nS) ? a.sten[(i0 + u) * ldc + c] : c;
    int8_t fl[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) fl[u] = a.si[2 * j[u]];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int ci = i0 + u;
      if (ci < nM) {
        shockType += fl[u];
        shockTypeExt = shockType;
      } else if (ci < nS) {
        shockTypeExt += fl[u];
      }
    }
  }

  S tc;
  if constexpr (P::id == PolicyRef::id) tc = to_float(a.W[c].w);
  else tc = (S)a.W[c].w;
  const V4<G> g1 = a.grad[2 * c + 1];
  const G gTx = g1.z, gTy = g1.w;
  V4<S> L = a.lim[c];
  int bvdType = 0, bfaces = 0;
  for (int fi = 0; fi < nM; ++fi) {
    int f = a.cf[fi * ldc + c];
    const bool isNei = (f < 0);
    f = abs(f) - 1;
    if (f >= a.Nf) {
      bfaces += 1;
      if (bfaces >= 2) {  // corner cell: low order
        bvdType = 1;
        break;
      }
      continue;
    }
    const V2<G> d = a.sg[fi * ldc + c];
    const G tfOwn = a.fv[2 * f].w;
    const G tfNei = a.fv[2 * f + 1].w;
    int typeval, notFlat, limited;
    if constexpr (P::id == PolicyMixed::id) {
      const G tfCur = isNei ? tfNei : tfOwn, tfOther = isNei ? tfOwn : tfNei;
      const G lim = to_bj(L.w);
      const G tfTVD = tc + lim * (gTx * d.x + gTy * d.y);
      typeval = fab(tfTVD - tfOther) < 0.5f * fab(tfCur - tfOther);
      notFlat = fab(tfCur - tfOther) > 1e-10f;
      limited = (lim < 0.9f) + (shockTypeExt > 0);
    } else {  // the comparisons on integers
      double jump, tfTVD, tfOther;
      if constexpr (P::id == PolicyFP64::id) {
        tfOther = isNei ? tfOwn : tfNei;
        jump = dabs_((isNei ? tfNei : tfOwn) - tfOther);
        tfTVD = tvd64(tc, to_bj(L.w), gTx, gTy, d.x, d.y);
        limited = (dbits(L.w) < dbits(0.45)) + (shockTypeExt > 0);  // (L.w >= 0)
      } else {
        tfOther = blend64(!isNei, isNei, tfNei, tfOwn);
        jump = dabs_(blend64(isNei, !isNei, tfNei, tfOwn) - tfOther);
        const S lim = to_bj(L.w);
        tfTVD = to_double(tc) + to_double(lim) * (gTx * d.x + gTy * d.y);
        limited = (lim < 0.9f) + (shockTypeExt > 0);
      }
      const double flat = AFAR_LIT(S, 1e-10);
      typeval = dbits(dabs_(tfTVD - tfOther)) < dbits(0.5 * jump) && !dnan_(jump);
      notFlat = dbits(jump) > dbits(flat) && !dnan_(jump);
    }
    bvdType = max(bvdType, notFlat * limited * typeval);
  }
  const int finalType = (shockType > 0) * (shockTypeExt > 1) * (-2) + (bvdType > 0);
  a.si[2 * c + 1] = (int8_t)finalType;
  const bool isShock = finalType < 0;
  if constexpr (P::exact_blend) {  // the reference's blend evaluates both maps
    L.x = pick<P>(isShock, !isShock, to_venkat(L.x), to_bj(L.x));
    L.y = pick<P>(isShock, !isShock, to_venkat(L.y), to_bj(L.y));
    L.z = pick<P>(isShock, !isShock, to_venkat(L.z), to_bj(L.z));
    L.w = pick<P>(isShock, !isShock, to_venkat(L.w), to_bj(L.w));
  } else if (isShock) {  // only the map that applies: Venkatakrishnan's has a division
    L.x = to_venkat(L.x);
    L.y = to_venkat(L.y);
    L.z = to_venkat(L.z);
    L.w = to_venkat(L.w);
  } else {
    L.x = to_bj(L.x);
    L.y = to_bj(L.y);
    L.z = to_bj(L.z);
    L.w = to_bj(L.w);
  }
  a.lim[c] = L;
}

// minimizeDeltaValue (reference cudaRiemannSolver.h:7-14)
template <class D, class G>
__device__ __forceinline__ D min_delta(const G l, const G r, const G lT, const G rT) {
  D d = fab(r - l);
  d = fmn((G)(d), fab(r - lT));
  d = fmn((G)(d), fab(rT - l));
  d = fmn((G)(d), fab(rT - lT));
  d = (r >= l) * d - (r < l) * d;
  return d;
}

// KFVSFlux (reference cudaRiemannSolver.h:16-68): adds (kinetic flux - central) so the face
// carries the kinetic flux-vector-splitting flux.
template <class D, class RC, class G>
__device__ __forceinline__ void kfvs_flux(G& rhoFlux, G& rhoUxFlux, G& rhoUyFlux, G& rhoEFlux, const D& rhoL,
                                          const D& rhoR, const D& pL, const D& pR, const D& uxL, const D& uxR,
                                          const D& uyL, const D& uyR, const D& tL, const D& tR, const RC& R,
                                          const RC& Cv, const D magSf, const D Sfx, const D Sfy) {
  const D nfx = Sfx / magSf;
  const D nfy = Sfy / magSf;
  const D uLl = uxL * nfx + uyL * nfy;
  const D vLl = uyL * nfx - uxL * nfy;
  const D uRl = uxR * nfx + uyR * nfy;
  const D vRl = uyR * nfx - uxR * nfy;
  const D lamL = D(0.5) * rhoL / pL;
  const D lamR = D(0.5) * rhoR / pR;
  // the reference writes pi as the float literal 3.141593f; the FP64 policy uses pi itself
  const D PI = std::is_same<D, float>::value ? (D)3.141593f : (D)3.14159265358979323846;
  const D m0p = D(0.5) * erfc_(-sqr_(lamL) * uLl);
  const D m1p = uLl * m0p + D(0.5) * exp_(-lamL * uLl * uLl) / (sqr_(PI * lamL));
  const D m2p = uLl * m1p + D(0.5) * m0p / lamL;
  const D m3p = uLl * m2p + m1p / lamL;
  const D m0n = D(0.5) * erfc_(sqr_(lamR) * uRl);
  const D m1n = uRl * m0n - D(0.5) * exp_(-lamR * uRl * uRl) / (sqr_(PI * lamR));
  const D m2n = uRl * m1n + D(0.5) * m0n / lamR;
  const D m3n = uRl * m2n + m1n / lamR;
  const D& mvL = vLl;
  const D& mvR = vRl;
  const D K = D(2) * Cv / R - D(2);
  const D trho = rhoL * m1p + rhoR * m1n;
  const D trhoUx = rhoL * m2p + rhoR * m2n;
  const D trhoUy = rhoL * m1p * mvL + rhoR * m1n * mvR;
  const D trhoE = D(0.5) * rhoL * (m3p + m1p * (vLl * mvL + D(0.5) / lamL) + m1p * K * D(0.5) / lamL) +
                  D(0.5) * rhoR * (m3n + m1n * (vRl * mvR + D(0.5) / lamR) + m1n * K * D(0.5) / lamR);
  rhoUxFlux += trhoUx * Sfx - trhoUy * Sfy - D(0.5) * ((D)(rhoFlux)*uxL + pL * Sfx) - D(0.5) * ((D)(rhoFlux)*uxR + pR * Sfx);
  rhoUyFlux += trhoUx * Sfy + trhoUy * Sfx - D(0.5) * ((D)(rhoFlux)*uyL + pL * Sfy) - D(0.5) * ((D)(rhoFlux)*uyR + pR * Sfy);
  rhoEFlux += trhoE * magSf - D(0.5) * (D)(rhoFlux) * (Cv * tL + D(0.5) * (uxL * uxL + uyL * uyL) + pL / rhoL) -
              D(0.5) * (D)(rhoFlux) * (Cv * tR + D(0.5) * (uxR * uxR + uyR * uyR) + pR / rhoR);
  rhoFlux += trho * magSf - D(0.5) * rhoL * (uxL * Sfx + uyL * Sfy) - D(0.5) * rhoR * (uxR * Sfx + uyR * Sfy);
}

// RoeFlux (reference cudaRiemannSolver.h:71-136): Roe dissipation with a Harten-type entropy fix.
// R and Cv are double in it, the rest float; conversions and the division by Cv off the FP64 pipe.
__device__ __forceinline__ void roe_flux(double& rhoFlux, double& rhoUxFlux, double& rhoUyFlux, double& rhoEFlux,
                                         const float& rhoL, const float& rhoR, const float& pL, const float& pR,
                                         const float& uxL, const float& uxR, const float& uyL, const float& uyR,
                                         const float& tL, const float& tR, const float& deltaP, const float& deltaRho,
                                         const double& R, const double& Cv, const float magSf, const float Sfx,
                                         const float Sfy) {
  using D = float;
  const D gamma = to_float(div64(Cv + R, Cv));
  const D nfx = Sfx / magSf;
  const D nfy = Sfy / magSf;
  const D cvL = uxL * nfx + uyL * nfy;
  const D cvR = uxR * nfx + uyR * nfy;
  const D hL = to_float(Cv * to_double(tL) + to_double(D(0.5) * (uxL * uxL + uyL * uyL)) + to_double(pL / rhoL));
  const D hR = to_float(Cv * to_double(tR) + to_double(D(0.5) * (uxR * uxR + uyR * uyR)) + to_double(pR / rhoR));
  const D tiny = AFAR_LIT(D, 1e-20);
  const D rhoT = sqr_(fmx(rhoL * rhoR, tiny));
  const D wL = sqr_(fmx(rhoL, tiny)) / (sqr_(fmx(rhoL, tiny)) + sqr_(fmx(rhoR, tiny)));
  const D wR = D(1) - wL;
  const D uxT = uxL * wL + uxR * wR;
  const D uyT = uyL * wL + uyR * wR;
  const D hT = hL * wL + hR * wR;
  const D q2 = uxT * uxT + uyT * uyT;
  const D cT = sqr_(fmx((gamma - D(1)) * (hT - D(0.5) * q2), tiny));
  const D cvT = uxT * nfx + uyT * nfy;
  const D dUx = uxR - uxL;
  const D dUy = uyR - uyL;
  const D dCv = dUx * nfx + dUy * nfy;
  const D r1 = (deltaP - rhoT * cT * dCv) / (D(2) * cT * cT);
  const D r2 = deltaRho - deltaP / (cT * cT);
  const D r3 = (deltaP + rhoT * cT * dCv) / (D(2) * cT * cT);
  const D& UL = cvL;
  const D& UR = cvR;
  const D cL = sqr_(fmx((gamma - D(1)) * (hL - D(0.5) * (uxL * uxL + uyL * uyL)), tiny));
  const D cR = sqr_(fmx((gamma - D(1)) * (hR - D(0.5) * (uxR * uxR + uyR * uyR)), tiny));
  const D eps0 = AFAR_LIT(D, 1e-30);
  D eps = D(2) * fmx(D(0), (UR - cR) - (UL - cL));
  D l1 = fab(cvT - cT);
  l1 = (l1 >= eps) * l1 + (l1 < eps) * ((l1 * l1 + eps * eps) / (D(2) * eps + eps0));
  eps = D(2) * fmx(D(0), UR - UL);
  D l2 = fab(cvT);
  l2 = (l2 >= eps) * l2 + (l2 < eps) * ((l2 * l2 + eps * eps) / (D(2) * eps + eps0));
  eps = D(2) * fmx(D(0), (UR + cR) - (UL + cL));
  D l3 = fab(cvT + cT);
  l3 = (l3 >= eps) * l3 + (l3 < eps) * ((l3 * l3 + eps * eps) / (D(2) * eps + eps0));
  rhoFlux -= to_double(D(0.5) * (l1 * r1 + l2 * r2 + l3 * r3) * magSf);
  rhoUxFlux -= to_double(D(0.5) * (l1 * r1 * (uxT - cT * nfx) + l2 * (r2 * uxT + rhoT * (dUx - dCv * nfx)) + l3 * r3 * (uxT + cT * nfx)) * magSf);
  rhoUyFlux -= to_double(D(0.5) * (l1 * r1 * (uyT - cT * nfy) + l2 * (r2 * uyT + rhoT * (dUy - dCv * nfy)) + l3 * r3 * (uyT + cT * nfy)) * magSf);
  rhoEFlux -= to_double(D(0.5) *
              (l1 * r1 * (hT - cT * cvT) + l2 * (r2 * D(0.5) * q2 + rhoT * (uxT * dUx + uyT * dUy - cvT * dCv)) +
               l3 * r3 * (hT + cT * cvT)) *
              magSf);
}

// ---------------------------------------------------------------- dissipation, fp64 and mixed
// The same Roe and KFVS dissipation for the policies without bit parity, with their divisions
// folded: p/rho as R T (the state's own equation of state), one reciprocal of magSf (precomputed
// per face), of c^2 and of lambda, gamma and K computed once on the host, and the entropy fix's
// division only on the faces that need it.  Equal to the reference's expressions up to rounding.
__device__ __forceinline__ float fdiv(const float a, const float b) { return __fdividef(a, b); }
__device__ __forceinline__ float rsqrt_(const float a) { return rsqrtf(a); }

template <class D>
__device__ __forceinline__ void entropy_fix(D& l, const D eps) {
  if (l < eps) l = fdiv(l * l + eps * eps, D(2) * eps + AFAR_LIT(D, 1e-30));
}

template <class D>
__device__ __forceinline__ void roe_flux_fast(D& rhoFlux, D& rhoUxFlux, D& rhoUyFlux, D& rhoEFlux, const D rhoL,
                                              const D rhoR, const D uxL, const D uxR, const D uyL, const D uyR,
                                              const D tL, const D tR, const D deltaP, const D deltaRho, const D R,
                                              const D Cv, const D gamma, const D magSf, const D nfx, const D nfy) {
  const D cvL = uxL * nfx + uyL * nfy;
  const D cvR = uxR * nfx + uyR * nfy;
  const D kL = D(0.5) * (uxL * uxL + uyL * uyL), kR = D(0.5) * (uxR * uxR + uyR * uyR);
  const D hL = Cv * tL + kL + R * tL;
  const D hR = Cv * tR + kR + R * tR;
  const D tiny = AFAR_LIT(D, 1e-20);
  const D sL = sqr_(fmx(rhoL, tiny)), sR = sqr_(fmx(rhoR, tiny));
  const D rhoT = sL * sR;  // sqrt(rhoL rhoR) from the two roots the weights need anyway
  const D wL = fdiv(sL, sL + sR);
  const D wR = D(1) - wL;
  const D uxT = uxL * wL + uxR * wR;
  const D uyT = uyL * wL + uyR * wR;
  const D hT = hL * wL + hR * wR;
  const D q2 = uxT * uxT + uyT * uyT;
  const D cT2 = fmx((gamma - D(1)) * (hT - D(0.5) * q2), tiny);
  const D rcT = rsq_(cT2);  // 1/cT: the speed and 1/cT^2 from one reciprocal root
  const D cT = cT2 * rcT;
  const D ic2 = rcT * rcT;
  const D cvT = uxT * nfx + uyT * nfy;
  const D dUx = uxR - uxL;
  const D dUy = uyR - uyL;
  const D dCv = dUx * nfx + dUy * nfy;
  const D r1 = (deltaP - rhoT * cT * dCv) * (D(0.5) * ic2);
  const D r2 = deltaRho - deltaP * ic2;
  const D r3 = (deltaP + rhoT * cT * dCv) * (D(0.5) * ic2);
  const D cL = sqr_(fmx((gamma - D(1)) * (hL - kL), tiny));
  const D cR = sqr_(fmx((gamma - D(1)) * (hR - kR), tiny));
  D l1 = fab(cvT - cT), l2 = fab(cvT), l3 = fab(cvT + cT);
  entropy_fix(l1, D(2) * fmx(D(0), (cvR - cR) - (cvL - cL)));
  entropy_fix(l2, D(2) * fmx(D(0), cvR - cvL));
  entropy_fix(l3, D(2) * fmx(D(0), (cvR + cR) - (cvL + cL)));
  rhoFlux -= D(0.5) * (l1 * r1 + l2 * r2 + l3 * r3) * magSf;
  rhoUxFlux -= D(0.5) * (l1 * r1 * (uxT - cT * nfx) + l2 * (r2 * uxT + rhoT * (dUx - dCv * nfx)) + l3 * r3 * (uxT + cT * nfx)) * magSf;
  rhoUyFlux -= D(0.5) * (l1 * r1 * (uyT - cT * nfy) + l2 * (r2 * uyT + rhoT * (dUy - dCv * nfy)) + l3 * r3 * (uyT + cT * nfy)) * magSf;
  rhoEFlux -= D(0.5) *
              (l1 * r1 * (hT - cT * cvT) + l2 * (r2 * D(0.5) * q2 + rhoT * (uxT * dUx + uyT * dUy - cvT * dCv)) +
               l3 * r3 * (hT + cT * cvT)) *
              magSf;
}

template <class D>
__device__ __forceinline__ void kfvs_flux_fast(D& rhoFlux, D& rhoUxFlux, D& rhoUyFlux, D& rhoEFlux, const D rhoL,
                                               const D rhoR, const D pL, const D pR, const D uxL, const D uxR,
                                               const D uyL, const D uyR, const D tL, const D tR, const D R, const D Cv,
                                               const D K, const D magSf, const D nfx, const D nfy) {
  const D Sfx = nfx * magSf, Sfy = nfy * magSf;
  const D uLl = uxL * nfx + uyL * nfy;
  const D vLl = uyL * nfx - uxL * nfy;
  const D uRl = uxR * nfx + uyR * nfy;
  const D vRl = uyR * nfx - uxR * nfy;
  const D ilamL = D(2) * R * tL, ilamR = D(2) * R * tR;  // 1/lambda = 2 p / rho
  const D lamL = fdiv(D(1), ilamL), lamR = fdiv(D(1), ilamR);
  const D PI = std::is_same<D, float>::value ? (D)3.141593f : (D)3.14159265358979323846;
  const D m0p = D(0.5) * erfc_(-sqr_(lamL) * uLl);
  const D m1p = uLl * m0p + D(0.5) * exp_(-lamL * uLl * uLl) * rsqrt_(PI * lamL);
  const D m2p = uLl * m1p + D(0.5) * m0p * ilamL;
  const D m3p = uLl * m2p + m1p * ilamL;
  const D m0n = D(0.5) * erfc_(sqr_(lamR) * uRl);
  const D m1n = uRl * m0n - D(0.5) * exp_(-lamR * uRl * uRl) * rsqrt_(PI * lamR);
  const D m2n = uRl * m1n + D(0.5) * m0n * ilamR;
  const D m3n = uRl * m2n + m1n * ilamR;
  const D trho = rhoL * m1p + rhoR * m1n;
  const D trhoUx = rhoL * m2p + rhoR * m2n;
  const D trhoUy = rhoL * m1p * vLl + rhoR * m1n * vRl;
  const D trhoE = D(0.5) * rhoL * (m3p + m1p * (vLl * vLl + D(0.5) * ilamL) + m1p * K * D(0.5) * ilamL) +
                  D(0.5) * rhoR * (m3n + m1n * (vRl * vRl + D(0.5) * ilamR) + m1n * K * D(0.5) * ilamR);
  rhoUxFlux += trhoUx * Sfx - trhoUy * Sfy - D(0.5) * (rhoFlux * uxL + pL * Sfx) - D(0.5) * (rhoFlux * uxR + pR * Sfx);
  rhoUyFlux += trhoUx * Sfy + trhoUy * Sfx - D(0.5) * (rhoFlux * uyL + pL * Sfy) - D(0.5) * (rhoFlux * uyR + pR * Sfy);
  rhoEFlux += trhoE * magSf - D(0.5) * rhoFlux * (Cv * tL + D(0.5) * (uxL * uxL + uyL * uyL) + R * tL) -
              D(0.5) * rhoFlux * (Cv * tR + D(0.5) * (uxR * uxR + uyR * uyR) + R * tR);
  rhoFlux += trho * magSf - D(0.5) * rhoL * (uxL * Sfx + uyL * Sfy) - D(0.5) * rhoR * (uxR * Sfx + uyR * Sfy);
}

// One side of a face: the state that the flux uses, and p and T of its TVD state.
struct MixedSide {
  float p, ux, uy, T, pT, tT;
};
// The mixed policy's flux of an internal face (reference cudaRiemannSolver.h:16-251): central flux with the
// Roe dissipation, or the KFVS flux; the expressions of roe_flux_fast and kfvs_flux_fast.  Every rounding
// is written out, in the pattern in which the compiler fuses those expressions in the separate flux
// kernel (found by comparing results: each candidate rounding on 65k random faces, equal to the bit), so
// that the kernels that call it agree bit for bit whatever the code around the call.  E: the energy flux's
// sum of two products fused, as the compiler had it in the batched stage-1 flux (DT) and nowhere else when the
// roundings were written out; kept, so that a batch's results stay what they were.
__device__ __forceinline__ float fm_(const float a, const float b, const float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float ml_(const float a, const float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float ad_(const float a, const float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float dot_(const float a, const float b, const float c, const float d) {  // a b + c d
  return fm_(a, b, ml_(c, d));
}
// w + lim (ga dx + gb dy): the limited linear (TVD) value
__device__ __forceinline__ float tvd_mixed(const float w, const float lim, const float ga, const float gb,
                                           const V2<float> d) {
  return fm_(lim, dot_(ga, d.x, gb, d.y), w);
}
// __fdividef(a, b) is a times this, to the bit, for |b| up to 2^126 (checked on 2.7e9 pairs); it also spends
// four instructions on larger ones
__device__ __forceinline__ float rcp_(const float x) {
  float y;
  asm("rcp.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// The density p/(R T) as the product it is, for the differences that round the product away
struct MixedRho {
  float num, rcp, rho;
};
__device__ __forceinline__ MixedRho mixed_rho(const float p, const float iR, const float T) {
  MixedRho r;
  r.num = ml_(p, iR);
  r.rcp = rcp_(T);
  r.rho = ml_(r.num, r.rcp);
  return r;
}
// minimizeDeltaValue's last step: the smallest jump d >= 0 with the sign of r - l
__device__ __forceinline__ float signed_jump(const float d, const float l, const float r) { return r >= l ? d : -d; }
__device__ __forceinline__ void entropy_fix_mixed(float& l, const float jump) {
  const float eps = ml_(2.f, fmaxf(0.f, jump));
  if (l < eps) l = ml_(fm_(eps, eps, ml_(l, l)), rcp_(fm_(2.f, eps, 1e-30f)));
}
// One side's kinetic moments: the half-range fluxes of mass, normal momentum and energy moments.
struct MixedKinetic {
  float m1, m2, m3;
};
__device__ __forceinline__ MixedKinetic mixed_kinetic(const bool left, const float u, const float lam, const float il) {
  const float su = ml_(sqrtf(lam), u);
  const float m0 = ml_(0.5f, erfcf(left ? -su : su));
  const float ex = ml_(0.5f, expf(ml_(ml_(-lam, u), u))), rs = rsqrtf(ml_(3.141593f, lam));
  MixedKinetic q;
  q.m1 = left ? fm_(ex, rs, ml_(u, m0)) : fm_(u, m0, ml_(-ex, rs));
  q.m2 = fm_(ml_(0.5f, m0), il, ml_(u, q.m1));
  q.m3 = fm_(q.m1, il, ml_(u, q.m2));
  return q;
}
template <bool E>
__device__ __forceinline__ V4<float> mixed_flux(const MixedSide& l, const MixedSide& r, const bool isShock,
                                                const V4<float>& fs, const float R, const float Cv, const float iR,
                                                const float gam) {
  const float h = 0.5f, Sfx = fs.x, Sfy = fs.y, magSf = fs.z;
  const MixedRho dl = mixed_rho(l.p, iR, l.T), dr = mixed_rho(r.p, iR, r.T);
  const float rhoL = dl.rho, rhoR = dr.rho;
  // central flux
  const float unL = dot_(l.ux, Sfx, l.uy, Sfy), unR = dot_(r.ux, Sfx, r.uy, Sfy);
  const float F0 = dot_(ml_(h, rhoL), unL, ml_(h, rhoR), unR);
  const float F1 = dot_(h, dot_(l.p, Sfx, F0, l.ux), h, dot_(r.p, Sfx, F0, r.ux));
  const float F2 = dot_(h, dot_(l.p, Sfy, F0, l.uy), h, dot_(r.p, Sfy, F0, r.uy));
  const float kkL = dot_(l.ux, l.ux, l.uy, l.uy), kkR = dot_(r.ux, r.ux, r.uy, r.uy);
  const float hF = ml_(h, F0);
  const float htL = fm_(R, l.T, fm_(Cv, l.T, ml_(h, kkL))), htR = fm_(R, r.T, fm_(Cv, r.T, ml_(h, kkR)));
  const float F3 = E ? dot_(hF, htL, hF, htR) : ad_(ml_(hF, htL), ml_(hF, htR));
  const float nfx = ml_(Sfx, fs.w), nfy = ml_(Sfy, fs.w);  // fs.w = 1/|Sf| (setup)
  const float cvL = dot_(l.ux, nfx, l.uy, nfy), cvR = dot_(r.ux, nfx, r.uy, nfy);
  if (isShock) {
    const float K = fm_(ml_(2.f, Cv), iR, -2.f);
    const float Gx = ml_(nfx, magSf), Gy = ml_(nfy, magSf);
    const float vL = dot_(l.uy, nfx, -l.ux, nfy), vR = dot_(r.uy, nfx, -r.ux, nfy);
    const float ilL = ml_(ml_(2.f, R), l.T), ilR = ml_(ml_(2.f, R), r.T);  // 1/lambda = 2 p / rho
    const MixedKinetic a = mixed_kinetic(true, cvL, rcp_(ilL), ilL);
    const MixedKinetic b = mixed_kinetic(false, cvR, rcp_(ilR), ilR);
    const float rmL = ml_(rhoL, a.m1), rmR = ml_(rhoR, b.m1);
    const float t0 = ad_(rmL, rmR), tx = dot_(rhoL, a.m2, rhoR, b.m2), ty = dot_(rmL, vL, rmR, vR);
    const float hrL = ml_(h, rhoL), hrR = ml_(h, rhoR);
    const float enL = fm_(ml_(ml_(a.m1, K), h), ilL, fm_(a.m1, fm_(vL, vL, ml_(h, ilL)), a.m3));
    const float enR = fm_(ml_(ml_(b.m1, K), h), ilR, fm_(b.m1, fm_(vR, vR, ml_(h, ilR)), b.m3));
    const float t3 = dot_(hrL, enL, hrR, enR);
    const float x1 = fm_(-h, dot_(r.p, Gx, F0, r.ux), fm_(-h, dot_(l.p, Gx, F0, l.ux), dot_(tx, Gx, -ty, Gy)));
    const float x2 = fm_(-h, dot_(r.p, Gy, F0, r.uy), fm_(-h, dot_(l.p, Gy, F0, l.uy), dot_(ty, Gx, tx, Gy)));
    const float x3 = E ? fm_(-hF, htR, fm_(t3, magSf, -ml_(hF, htL))) : ad_(fm_(t3, magSf, -ml_(hF, htL)), -ml_(hF, htR));
    const float x0 = fm_(-hrR, dot_(r.ux, Gx, r.uy, Gy), fm_(t0, magSf, ml_(-hrL, dot_(l.ux, Gx, l.uy, Gy))));
    return V4<float>{ad_(F0, x0), ad_(F1, x1), ad_(F2, x2), ad_(F3, x3)};
  }
  const MixedRho dlT = mixed_rho(l.pT, iR, l.tT), drT = mixed_rho(r.pT, iR, r.tT);
  float dP = fabsf(ad_(r.p, -l.p));
  dP = fminf(dP, fabsf(ad_(r.p, -l.pT)));
  dP = fminf(dP, fabsf(ad_(r.pT, -l.p)));
  dP = fminf(dP, fabsf(ad_(r.pT, -l.pT)));
  dP = signed_jump(dP, l.p, r.p);
  float dRho = fabsf(ad_(rhoR, -rhoL));
  dRho = fminf(dRho, fabsf(fm_(-dlT.num, dlT.rcp, rhoR)));
  dRho = fminf(dRho, fabsf(fm_(drT.num, drT.rcp, -rhoL)));
  dRho = fminf(dRho, fabsf(fm_(drT.num, drT.rcp, -dlT.rho)));
  dRho = signed_jump(dRho, rhoL, rhoR);
  const float kL = ml_(h, kkL), kR = ml_(h, kkR);
  const float hL = fm_(R, l.T, fm_(Cv, l.T, kL)), hR = fm_(R, r.T, fm_(Cv, r.T, kR));
  const float tiny = 1e-20f;
  const float sL = sqrtf(fmaxf(rhoL, tiny)), sR = sqrtf(fmaxf(rhoR, tiny));
  const float rhoT = ml_(sL, sR);  // sqrt(rhoL rhoR) from the two roots the weights need anyway
  const float wL = ml_(sL, rcp_(ad_(sL, sR))), wR = ad_(1.f, -wL);
  const float uxT = dot_(l.ux, wL, r.ux, wR), uyT = dot_(l.uy, wL, r.uy, wR), hT = dot_(hL, wL, hR, wR);
  const float q2 = dot_(uxT, uxT, uyT, uyT), gm1 = ad_(gam, -1.f);
  const float cT2 = fmaxf(ml_(gm1, fm_(-h, q2, hT)), tiny);
  const float rcT = rsqrtf(cT2);  // 1/cT: the speed and 1/cT^2 from one reciprocal root
  const float cT = ml_(cT2, rcT), ic2 = ml_(rcT, rcT);
  const float cvT = dot_(uxT, nfx, uyT, nfy);
  const float dUx = ad_(r.ux, -l.ux), dUy = ad_(r.uy, -l.uy);
  const float dCv = dot_(dUx, nfx, dUy, nfy);
  const float rc = ml_(rhoT, cT), hic2 = ml_(h, ic2);
  const float r1 = ml_(fm_(-rc, dCv, dP), hic2), r2 = fm_(-dP, ic2, dRho), r3 = ml_(fm_(rc, dCv, dP), hic2);
  float l1 = fabsf(ad_(cvT, -cT)), l2 = fabsf(cvT), l3 = fabsf(ad_(cvT, cT));
  entropy_fix_mixed(l2, ad_(cvR, -cvL));
  {  // the acoustic waves: the sides' sound speeds exactly only where approximate ones do not rule the fix out
    const float xL = fmaxf(ml_(gm1, ad_(hL, -kL)), tiny), xR = fmaxf(ml_(gm1, ad_(hR, -kR)), tiny);
    float cL, cR;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(cL) : "f"(xL));
    asm("sqrt.approx.f32 %0, %1;" : "=f"(cR) : "f"(xR));
    const float margin = 1e-5f * (fabsf(cvL) + fabsf(cvR) + cL + cR + cT), dcv = cvR - cvL, dc = cR - cL;
    if (!(l1 > fmaxf(0.f, 2.f * (dcv - dc)) + margin && l3 > fmaxf(0.f, 2.f * (dcv + dc)) + margin)) {
      cL = sqrtf(xL);
      cR = sqrtf(xR);
      entropy_fix_mixed(l1, ad_(ad_(cvR, -cR), -ad_(cvL, -cL)));
      entropy_fix_mixed(l3, ad_(ad_(cvR, cR), -ad_(cvL, cL)));
    }
  }
  const float a1 = ml_(l1, r1), a3 = ml_(l3, r3);
  const float s0 = ad_(a3, fm_(l2, r2, a1));
  const float s1 = fm_(a3, fm_(cT, nfx, uxT),
                       dot_(a1, fm_(-cT, nfx, uxT), l2, dot_(rhoT, fm_(-dCv, nfx, dUx), r2, uxT)));
  const float s2 = fm_(a3, fm_(cT, nfy, uyT),
                       dot_(a1, fm_(-cT, nfy, uyT), l2, dot_(rhoT, fm_(-dCv, nfy, dUy), r2, uyT)));
  const float shear = fm_(-cvT, dCv, dot_(uxT, dUx, uyT, dUy));
  const float s3 = fm_(a3, fm_(cT, cvT, hT), dot_(a1, fm_(-cT, cvT, hT), l2, dot_(ml_(r2, h), q2, rhoT, shear)));
  return V4<float>{fm_(-ml_(h, s0), magSf, F0), fm_(-ml_(h, s1), magSf, F1), fm_(-ml_(h, s2), magSf, F2),
                   fm_(-ml_(h, s3), magSf, F3)};
}
// The Euler flux of a boundary face's ghost state, its roundings written out as the compiler fuses them in
// flux_body (the separate flux kernels), so that both forms of the stage give the same bits.
__device__ __forceinline__ V4<float> mixed_boundary_flux(const V4<float>& wb, const V4<float>& fs, const float R,
                                                         const float Cv) {
  const float rho = wb.x / __fmul_rn(R, wb.w);
  const float rhoFlux = __fmul_rn(rho, __fmaf_rn(wb.y, fs.x, __fmul_rn(wb.z, fs.y)));
  const float ke2 = __fmaf_rn(wb.y, wb.y, __fmul_rn(wb.z, wb.z));
  const float h = __fadd_rn(__fmaf_rn(0.5f, ke2, __fmul_rn(Cv, wb.w)), wb.x / rho);
  return V4<float>{rhoFlux, __fmaf_rn(wb.x, fs.x, __fmul_rn(rhoFlux, wb.y)),
                   __fmaf_rn(wb.x, fs.y, __fmul_rn(rhoFlux, wb.z)), __fmul_rn(rhoFlux, h)};
}

// minimizeDeltaValue (min_delta) of doubles with the minima and the sign on integers.
__device__ __forceinline__ double min_delta64(const double l, const double r, const double lT, const double rT) {
  const double d = __dsub_rn(r, l);
  double m = min_nonneg(dabs_(d), dabs_(__dsub_rn(r, lT)));
  m = min_nonneg(m, dabs_(__dsub_rn(rT, l)));
  m = min_nonneg(m, dabs_(__dsub_rn(rT, lT)));
  return flip_sign(m, __double2hiint(d) & (int)0x80000000);
}

// One side of a face under the fp64 policy: the state that the flux uses.
struct Side64 {
  double p, ux, uy, T, rho;
};

// The flux of a face under the fp64 policy: central flux with the Roe dissipation, or the KFVS flux,
// laid out by FP64 instructions: the two sides share their factors; the central flux takes Sf itself,
// so that the fluxes of a uniform stream close over a cell as its face vectors do; the Roe weights
// from one root and one reciprocal (sqrt(rhoL)/(sqrt(rhoL)+sqrt(rhoR)) = rhoL/(rhoL + sqrt(rhoL rhoR)));
// the wave strengths summed before they multiply the eigenvectors; and the acoustic entropy fix, which
// needs both sides' sound speeds, behind an FP32 look (20 bits of each operand, a margin of 1e-5 of
// all speeds) at whether its waves are surely outside it, as all but the near-sonic ones are.
// Every rounding is written out: the kernels of this policy (single and batched, of every block size,
// face-centre and multi-point) then agree bit for bit whatever multiply-adds the compiler would fuse.
// 750k faces: 426 us a launch before (244 FP64 instructions a face), 240 now (158 issued; the pipe 85%
// busy); the stage-1 form with the Courant step 280.
struct Gas64 {
  double R, Cv, Cp, gm1, iR;
  float gRf;
};
template <class A>
__device__ __forceinline__ Gas64 gas64(const A& a) {
  return Gas64{a.R, a.Cv, a.Cp, a.gm1, a.invR, a.gRf};
}
// The entropy fix of one wave: |lambda| below eps = 2 max(0, jump) becomes (lambda^2 + eps^2)/(2 eps).
__device__ __forceinline__ double entropy_fix64(const double l, const double jump) {
  const double eps = gt_zero(jump) ? add64(jump, jump) : 0.0;
  if (!(dbits(l) < dbits(eps))) return l;
  return mul64(fma64(l, l, mul64(eps, eps)), rcp64(fma64(2.0, eps, 1e-30)));
}
// One side's kinetic moments (reference cudaRiemannSolver.h:16-68): the half-range fluxes of mass,
// normal and tangential momentum and energy per unit area; sign +1 from the left, -1 from the right.
__device__ __forceinline__ V4<double> kinetic_side64(const Side64& q, const double sign, const double u, const double v,
                                                     const double R, const double K) {
  const double il = mul64(add64(R, R), q.T);  // 1/lambda = 2 p / rho
  const double lam = rcp64(il), rs = rsq64(lam);
  const double m0 = mul64(0.5, erfc(mul64(-sign, mul64(mul64(lam, rs), u))));
  const double ex = mul64(mul64(sign * 0.28209479177387814, rs), exp(mul64(mul64(-lam, u), u)));  // 1/(2 sqrt(pi))
  const double m1 = fma64(u, m0, ex);
  const double m2 = fma64(u, m1, mul64(mul64(0.5, m0), il));
  const double m3 = fma64(u, m2, mul64(m1, il));
  const double e = fma64(m1, fma64(v, v, mul64(mul64(0.5, il), add64(1.0, K))), m3);
  const double rm1 = mul64(q.rho, m1);
  return V4<double>{rm1, mul64(q.rho, m2), mul64(rm1, v), mul64(mul64(0.5, q.rho), e)};
}
__device__ __forceinline__ V4<double> face_flux64(const Side64& l, const Side64& r, const double pLT, const double pRT,
                                                  const double rhoLT, const double rhoRT, const bool isShock,
                                                  const Gas64& k, const V4<double>& fs) {
  const double Sfx = fs.x, Sfy = fs.y, nx = mul64(Sfx, fs.w), ny = mul64(Sfy, fs.w);
  const double unL = fma64(l.uy, Sfy, mul64(l.ux, Sfx)), unR = fma64(r.uy, Sfy, mul64(r.ux, Sfx));  // times |Sf|
  const double cvL = mul64(unL, fs.w), cvR = mul64(unR, fs.w);
  if (isShock) {
    const double K = fma64(mul64(2.0, k.Cv), k.iR, -2.0);
    const V4<double> a = kinetic_side64(l, 1.0, cvL, fma64(l.uy, nx, mul64(-l.ux, ny)), k.R, K);
    const V4<double> b = kinetic_side64(r, -1.0, cvR, fma64(r.uy, nx, mul64(-r.ux, ny)), k.R, K);
    const double tn = add64(a.y, b.y), tt = add64(a.z, b.z);
    return V4<double>{mul64(add64(a.x, b.x), fs.z), fma64(tn, Sfx, mul64(-tt, Sfy)), fma64(tn, Sfy, mul64(tt, Sfx)),
                      mul64(add64(a.w, b.w), fs.z)};
  }
  const double kL = fma64(l.uy, l.uy, mul64(l.ux, l.ux)), kR = fma64(r.uy, r.uy, mul64(r.ux, r.ux));
  const double hL = fma64(0.5, kL, mul64(k.Cp, l.T)), hR = fma64(0.5, kR, mul64(k.Cp, r.T));  // p/rho = R T
  const double M = fma64(r.rho, unR, mul64(l.rho, unL)), hF = mul64(0.25, M), hp = mul64(0.5, add64(l.p, r.p));
  const double dP = min_delta64(l.p, r.p, pLT, pRT), dRho = min_delta64(l.rho, r.rho, rhoLT, rhoRT);
  const double tiny = 1e-20;
  const double rl = dmax_(l.rho, tiny), rr = dmax_(r.rho, tiny);
  const double rho2 = mul64(rl, rr);
  const double rhoT = mul64(rho2, rsq64(rho2));
  const double wL = mul64(rl, rcp64(add64(rl, rhoT)));
  const double dUx = sub64(r.ux, l.ux), dUy = sub64(r.uy, l.uy);
  const double uxT = fma64(-wL, dUx, r.ux), uyT = fma64(-wL, dUy, r.uy);
  const double hT = fma64(-wL, sub64(hR, hL), hR);
  const double kT = mul64(0.5, fma64(uyT, uyT, mul64(uxT, uxT)));
  const double cT2 = dmax_(mul64(k.gm1, sub64(hT, kT)), tiny);
  const double rcT = rsq64(cT2);
  const double cT = mul64(cT2, rcT), ic2 = mul64(rcT, rcT);
  const double cvT = fma64(uyT, ny, mul64(uxT, nx));
  const double dCv = fma64(dUy, ny, mul64(dUx, nx));
  const double rc = mul64(mul64(rhoT, cT), dCv), hic2 = mul64(0.5, ic2);
  double l1 = dabs_(sub64(cvT, cT)), l3 = dabs_(add64(cvT, cT));
  const double l2 = entropy_fix64(dabs_(cvT), sub64(cvR, cvL));
  {
    const float uL = top_float(cvL), uR = top_float(cvR), c = top_float(cT);
    const float cL = sqrtf(k.gRf * top_float(l.T)), cR = sqrtf(k.gRf * top_float(r.T));
    const float margin = 1e-5f * (fabsf(uL) + fabsf(uR) + cL + cR + c);
    const bool clear1 = top_float(l1) > 2.f * fmaxf(0.f, (uR - cR) - (uL - cL)) + margin;
    const bool clear3 = top_float(l3) > 2.f * fmaxf(0.f, (uR + cR) - (uL + cL)) + margin;
    if (!(clear1 && clear3)) {
      const double xL = dmax_(mul64(k.gm1, mul64(k.Cp, l.T)), tiny), xR = dmax_(mul64(k.gm1, mul64(k.Cp, r.T)), tiny);
      const double sL = mul64(xL, rsq64(xL)), sR = mul64(xR, rsq64(xR));
      l1 = entropy_fix64(l1, sub64(sub64(cvR, sR), sub64(cvL, sL)));
      l3 = entropy_fix64(l3, sub64(add64(cvR, sR), add64(cvL, sL)));
    }
  }
  const double a1 = mul64(mul64(sub64(dP, rc), hic2), l1), a3 = mul64(mul64(add64(dP, rc), hic2), l3);
  const double a2 = mul64(fma64(-dP, ic2, dRho), l2);
  const double s13 = add64(a1, a3), s = add64(s13, a2), b = mul64(sub64(a3, a1), cT);
  const double gt = mul64(mul64(l2, rhoT), fma64(dUy, nx, mul64(-dUx, ny)));  // the shear wave
  const double h = mul64(-0.5, fs.z);
  const double d1 = fma64(-gt, ny, fma64(b, nx, mul64(s, uxT)));
  const double d2 = fma64(gt, nx, fma64(b, ny, mul64(s, uyT)));
  const double d3 = fma64(gt, fma64(uyT, nx, mul64(-uxT, ny)), fma64(a2, kT, fma64(b, cvT, mul64(s13, hT))));
  return V4<double>{fma64(h, s, mul64(0.5, M)), fma64(h, d1, fma64(hp, Sfx, mul64(hF, add64(l.ux, r.ux)))),
                    fma64(h, d2, fma64(hp, Sfy, mul64(hF, add64(l.uy, r.uy)))), fma64(h, d3, mul64(hF, add64(hL, hR)))};
}
// The densities of a face's two states and their two TVD states (p/(R T)) from one reciprocal
// (simultaneous inversion of the four temperatures, a few ulps from four divisions; their product
// neither overflows nor underflows).
__device__ __forceinline__ void densities64(double& rhoL, double& rhoR, double& rhoLT, double& rhoRT, const double pL,
                                            const double pR, const double pLT, const double pRT, const double tL,
                                            const double tR, const double tLT, const double tRT, const double iR) {
  const double tt = mul64(tL, tR), ttT = mul64(tLT, tRT);
  const double inv = mul64(iR, rcp64(mul64(tt, ttT)));
  const double itt = mul64(inv, ttT), ittT = mul64(inv, tt);  // 1/(R tL tR), 1/(R tLT tRT)
  rhoL = mul64(pL, mul64(itt, tR));
  rhoR = mul64(pR, mul64(itt, tL));
  rhoLT = mul64(pLT, mul64(ittT, tRT));
  rhoRT = mul64(pRT, mul64(ittT, tLT));
}
// The Courant step of one face in FP64 for the fp64 policy (setDeltaT, reference
// cudaFieldOperation.h:140-157).  Every rounding is written out, so the fused stage-1 flux and the
// separate pass give the same bits.
__device__ __forceinline__ double courant_dt64(const double CFL, const double gR, const V2<double> g,
                                               const V4<double>& fs, const V4<double>& Wo, const V4<double>& Wn) {
  const double w1 = g.y, w0 = __dadd_rn(1.0, -w1);
  const double unL = dabs_(__fma_rn(Wo.y, fs.x, __dmul_rn(Wo.z, fs.y)));
  const double unR = dabs_(__fma_rn(Wn.y, fs.x, __dmul_rn(Wn.z, fs.y)));
  const double c2 = __dmul_rn(gR, __fma_rn(w0, Wo.w, __dmul_rn(w1, Wn.w)));
  const double c = __dmul_rn(c2, rsq64(c2));
  const double den = __fma_rn(c, fs.z, __fma_rn(w0, unL, __dmul_rn(w1, unR)));
  return __dmul_rn(__dmul_rn(__dmul_rn(CFL, g.x), fs.z), rcp64(den));
}
// Bounds of a face's step over the Courant number in FP32, from 20 bits of each operand (i: 1/|Sf|):
// every operand's error counts against the largest term, so a velocity across the face that is the
// difference of large components, or a sound speed far below them, widens the bounds.  A bound that
// cannot be had is 0 below and infinite above.
struct CourantBounds {
  float lo, hi;
};
__device__ __forceinline__ CourantBounds courant_bounds(const float gR, const V2<double> g, const V4<double>& fs,
                                                        const float i, const V4<double>& Wo, const V4<double>& Wn) {
  const float inf = __int_as_float(0x7F800000);
  const float w1 = top_float(g.y), w0 = 1.f - w1, ws = fabsf(w0) + fabsf(w1);
  const float x = i * top_float(fs.x), y = i * top_float(fs.y), dr = top_float(g.x);
  const float ax = top_float(Wo.y) * x, ay = top_float(Wo.z) * y, bx = top_float(Wn.y) * x, by = top_float(Wn.z) * y;
  const float tL = top_float(Wo.w), tR = top_float(Wn.w);
  const float un = w0 * fabsf(ax + ay) + w1 * fabsf(bx + by);
  const float eu = 1e-5f * ws * fmaxf(fabsf(ax) + fabsf(ay), fabsf(bx) + fabsf(by));
  const float c2 = gR * (w0 * tL + w1 * tR), e2 = 1e-5f * gR * ws * fmaxf(fabsf(tL), fabsf(tR));
  const float most = un + eu + sqrtf(c2 + e2), least = un - eu + sqrtf(fmaxf(c2 - e2, 0.f));
  CourantBounds r;
  r.lo = most > 1e-18f ? 0.9999f * __fdividef(dr, most) : 0.f;  // (0 where it is not a number either)
  r.hi = least > 1e-18f && least < 1e37f ? 1.0001f * __fdividef(dr, least) : inf;
  return r;
}

// The smallest Courant step of a block's faces into *bits: only the smallest counts, so a face is
// evaluated in FP64 only where its lower bound is not above the smallest upper bound of the block and
// the smallest step of any block so far -- a few faces of a few blocks of a flow that varies instead of
// 25 to 45 FP64 instructions a face.  The minimum is that over all faces, exactly.  All threads of the
// block take part.
template <class Exact>
__device__ __forceinline__ void courant_block_min(const CourantBounds est, const double cfl, unsigned long long* bits,
                                                  const bool face, Exact exact) {
  __shared__ unsigned wmin[8];
  __shared__ float s_prior;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned v = __float_as_uint(est.hi);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
  if (lane == 0) wmin[warp] = v;
  if (threadIdx.x == 0)
    s_prior = 1.0001f *
              __fdividef((float)__longlong_as_double((long long)*(const volatile unsigned long long*)bits), (float)cfl);
  __syncthreads();
  unsigned b = wmin[0];
  for (int k = 1; k < (int)(blockDim.x >> 5); ++k) b = min(b, wmin[k]);
  const bool near = face && !(est.lo > fminf(__uint_as_float(b), s_prior));
  if (!__any_sync(0xffffffffu, near)) return;
  unsigned long long d = kInfBits;
  if (near) {
    d = dbits(exact());
    if (d > kInfBits) d = kInfBits;  // not a number, negative: no step from here
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long u = __shfl_xor_sync(0xffffffffu, d, o);
    d = u < d ? u : d;
  }
  if (lane == 0 && d < *(const volatile unsigned long long*)bits) atomicMin(bits, d);
}

// ---------------------------------------------------------------- ref policy: face flux
// The ref policy's face flux reproduces the reference kernel's results bit for bit.  Two things
// besides the arithmetic itself decide that, both established by comparing with the reference
// kernels' results on the parity meshes (never by reading compiled code):
//  * nvcc contracts plain a*b + c expressions into fused multiply-adds in ways that depend on the
//    surrounding code, so every double-precision rounding of the state selection and the central
//    flux is written out (__fma_rn / __dmul_rn / __dadd_rn) in the pattern the reference's build
//    produces (identified on 24,300 faces of a mixed quad/triangle Riemann mesh, every candidate
//    rounding evaluated exactly);
//  * the float Roe/KFVS dissipation rounds like the reference's only when it is compiled as a
//    function of its own that takes its inputs by reference and is called through a pointer: inlined,
//    called directly, or taking its inputs by value, its float expressions round differently on a
//    few hundred flux entries per mesh (a few ulp of float).
// A blend c1*a + c2*b with c in {0, 1} is exact either way; it keeps the reference's propagation of
// a non-finite unused operand.

// One side of an internal face: the limited linear (TVD) state at the face centre, and the state
// the flux uses (the O3 face value, or the TVD state where the cell's switch asks for it), with
// p/(R T) of both; reference cudaRiemannSolver.h:190-216.
struct RefSide {
  double p, ux, uy, T, rho;  // the state the flux uses
  double pT, rhoT;           // pressure and density of the TVD state
};
__device__ __forceinline__ double ref_tvd(const double w, const float lim, const double ga, const double gb,
                                          const double dx, const double dy) {
  return __fma_rn(to_double(lim), __fma_rn(ga, dx, __dmul_rn(gb, dy)), w);  // w + lim (ga dx + gb dy)
}
__device__ __forceinline__ double ref_blend(const bool tvd, const double o3, const double t) {
  return blend64(!tvd, tvd, o3, t);
}
__device__ __forceinline__ RefSide ref_face_side(const StageArgs<PolicyRef>& a, const int c, const int slot,
                                                 const double dx, const double dy, const bool tvd) {
  const V4<double> w = a.W[c];
  const V4<double> g0 = a.grad[2 * c], g1 = a.grad[2 * c + 1];  // (px py uxx uxy), (uyx uyy tx ty)
  const V4<float> lm = a.lim[c];
  const V4<double> o3 = a.fv[slot];
  const double R = a.R;
  const double pT = ref_tvd(w.x, lm.x, g0.x, g0.y, dx, dy);
  const double uxT = ref_tvd(w.y, lm.y, g0.z, g1.x, dx, dy);
  const double uyT = ref_tvd(w.z, lm.z, g0.w, g1.y, dx, dy);
  const double tT = ref_tvd(w.w, lm.w, g1.z, g1.w, dx, dy);
  RefSide s;
  s.pT = pT;
  s.rhoT = div64(pT, __dmul_rn(R, tT));
  s.p = ref_blend(tvd, o3.x, pT);
  s.ux = ref_blend(tvd, o3.y, uxT);
  s.uy = ref_blend(tvd, o3.z, uyT);
  s.T = ref_blend(tvd, o3.w, tT);
  s.rho = div64(s.p, __dmul_rn(R, s.T));
  return s;
}
// Cv T + |u|^2 / 2 + p / rho of a side (its total enthalpy per unit mass)
__device__ __forceinline__ double ref_enthalpy(const RefSide& s, const double Cv) {
  return __dadd_rn(__dadd_rn(__dmul_rn(Cv, s.T), half64(__fma_rn(s.ux, s.ux, __dmul_rn(s.uy, s.uy)))),
                   div64(s.p, s.rho));
}

// min_delta of doubles, kept in a float: rounding keeps the order, so the minima are taken after it
__device__ __forceinline__ float ref_min_delta(const double l, const double r, const double lT, const double rT) {
  const double j = r - l;
  float d = fabsf(to_float(j));
  d = fminf(d, fabsf(to_float(r - lT)));
  d = fminf(d, fabsf(to_float(rT - l)));
  d = fminf(d, fabsf(to_float(rT - lT)));
  bool lt = neg_(j) && (dbits(j) << 1) != 0ull, ge = !lt;
  if (dnan_(j)) ge = r >= l, lt = r < l;
  return ge * d - lt * d;
}

// The float dissipation of the ref policy: adds the Roe dissipation, or replaces the central flux
// by the KFVS flux, in the four double flux components (reference cudaRiemannSolver.h:16-136).
using RefDissipation = void (*)(double&, double&, double&, double&, const float&, const float&, const float&,
                                const float&, const float&, const float&, const float&, const float&, const float&,
                                const float&, const float&, const float&, const double&, const double&, const float,
                                const float, const float);
__device__ __noinline__ void ref_roe(double& rhoFlux, double& rhoUxFlux, double& rhoUyFlux, double& rhoEFlux,
                                     const float& rhoL, const float& rhoR, const float& pL, const float& pR,
                                     const float& uxL, const float& uxR, const float& uyL, const float& uyR,
                                     const float& tL, const float& tR, const float& dP, const float& dRho,
                                     const double& R, const double& Cv, const float magSf, const float Sfx,
                                     const float Sfy) {
  roe_flux(rhoFlux, rhoUxFlux, rhoUyFlux, rhoEFlux, rhoL, rhoR, pL, pR, uxL, uxR, uyL, uyR, tL,
                                  tR, dP, dRho, R, Cv, magSf, Sfx, Sfy);
}
__device__ __noinline__ void ref_kfvs(double& rhoFlux, double& rhoUxFlux, double& rhoUyFlux, double& rhoEFlux,
                                      const float& rhoL, const float& rhoR, const float& pL, const float& pR,
                                      const float& uxL, const float& uxR, const float& uyL, const float& uyR,
                                      const float& tL, const float& tR, const float&, const float&,
                                      const double& R, const double& Cv, const float magSf, const float Sfx,
                                      const float Sfy) {
  kfvs_flux<float, double, double>(rhoFlux, rhoUxFlux, rhoUyFlux, rhoEFlux, rhoL, rhoR, pL, pR, uxL, uxR, uyL, uyR, tL,
                                   tR, R, Cv, magSf, Sfx, Sfy);
}

// evaluateFlux of internal face f under the ref policy (reference cudaRiemannSolver.h:171-251):
// both sides' states, the minimised jumps of p and rho, the central flux in double, then the float
// Roe dissipation, or the KFVS flux where either cell is a shock cell.
// The FP64 pipe bounds it, so what need not run there does not: selections and conversions on integers,
// divisions by div64, minima of the jumps as floats, with the same bits.  129 FP64 instructions a face
// now; 121k triangles 108 -> 88 us a launch (the pipe 79% busy), the update 33 -> 26, the BVD 19 -> 14.
__device__ __forceinline__ void flux_ref_face(const StageArgs<PolicyRef>& a, const int f) {
  const int2 on = a.on[f];
  const V4<double> d = a.fd[f];   // face centre - owner centre, face centre - neighbour centre
  const V4<double> sf = a.fs[f];  // Sfx, Sfy, |Sf|
  const int8_t swL = a.si[2 * on.x + 1], swR = a.si[2 * on.y + 1];
  const RefSide L = ref_face_side(a, on.x, 2 * f, d.x, d.y, swL != 0);
  const RefSide Rs = ref_face_side(a, on.y, 2 * f + 1, d.z, d.w, swR != 0);
  const double Sfx = sf.x, Sfy = sf.y, magSf = sf.z, Cv = a.Cv, R = a.R;
  const float dP = ref_min_delta(L.p, Rs.p, L.pT, Rs.pT);
  const float dRho = ref_min_delta(L.rho, Rs.rho, L.rhoT, Rs.rhoT);
  // central flux: the mean of the two sides' Euler fluxes through Sf
  double F0, F1, F2, F3;
  const double unL = __fma_rn(L.ux, Sfx, __dmul_rn(L.uy, Sfy)), unR = __fma_rn(Rs.ux, Sfx, __dmul_rn(Rs.uy, Sfy));
  F0 = __fma_rn(half64(L.rho), unL, __dmul_rn(half64(Rs.rho), unR));
  F1 = __dadd_rn(half64(__fma_rn(L.p, Sfx, __dmul_rn(F0, L.ux))),
                 half64(__fma_rn(Rs.p, Sfx, __dmul_rn(F0, Rs.ux))));
  F2 = __dadd_rn(half64(__fma_rn(L.p, Sfy, __dmul_rn(F0, L.uy))),
                 half64(__fma_rn(Rs.p, Sfy, __dmul_rn(F0, Rs.uy))));
  const double half = half64(F0);
  F3 = __fma_rn(half, ref_enthalpy(L, Cv), __dmul_rn(half, ref_enthalpy(Rs, Cv)));
  // the dissipation sees the states, face vector and jumps as floats; R and Cv stay double
  const float rhoL = to_float(L.rho), rhoR = to_float(Rs.rho), pL = to_float(L.p), pR = to_float(Rs.p),
              uxL = to_float(L.ux), uxR = to_float(Rs.ux), uyL = to_float(L.uy), uyR = to_float(Rs.uy),
              tL = to_float(L.T), tR = to_float(Rs.T);
  const RefDissipation diss = (swL < 0 || swR < 0) ? ref_kfvs : ref_roe;
  diss(F0, F1, F2, F3, rhoL, rhoR, pL, pR, uxL, uxR, uyL, uyR, tL, tR, dP, dRho, R, Cv, to_float(magSf),
       to_float(Sfx), to_float(Sfy));
  a.flux[f] = V4<double>{F0, F1, F2, F3};
}

// evaluateFlux (reference cudaRiemannSolver.h:155-271): one thread per internal face, then one per
// boundary face (ids Nf..Nf+Nb-1; the reference's grid covers boundary faces b < 128*ceil(Nf/128)
// only, which holds on every mesh with Nf >= Nb).  DT: also reduce the CFL step of the reference's
// setDeltaT (cudaFieldOperation.h:124-180) from the state at the start of the step.
template <class P, bool DT, bool BATCH = false>
__device__ __forceinline__ void flux_body(const StageArgs<P>& a, const int blk) {
  using S = typename P::S;
  using G = typename P::G;
  using D = typename P::D;
  using RC = typename P::RC;
  constexpr bool kF32 = std::is_same<G, float>::value;  // mixed: no per-thread FP64 at all
  const int id = blk * blockDim.x + threadIdx.x;
  // the Courant step: mixed estimates it in FP32 from block constants read once by thread 0
  __shared__ float s_cfl;
  __shared__ int s_cfl_step;
  if constexpr (DT && kF32) {
    if (threadIdx.x == 0) {
      s_cfl_step = !(a.ctl->dt_fixed > 0.0);
      s_cfl = (float)a.ctl->cfl;
    }
    __syncthreads();
  }
  float dtf32 = 1e5f;
  CourantBounds est{__int_as_float(0x7F800000), __int_as_float(0x7F800000)};  // fp64: of the face's Courant step
  if (id < a.Nf) {
    if constexpr (P::id == PolicyRef::id) {
      static_assert(!DT, "under the ref policy the Courant step is a kernel of its own, as in the reference");
      flux_ref_face(a, id);
    } else if constexpr (P::id == PolicyFP64::id) {
      const int2 on = a.on[id];
      const V4<double> fd = a.fd[id], fs = a.fs[id];
      const int8_t sL = a.si[2 * on.x + 1], sR = a.si[2 * on.y + 1];
      const V4<double> Wo = a.W[on.x], Wn = a.W[on.y];
      const V4<double> go0 = a.grad[2 * on.x], go1 = a.grad[2 * on.x + 1];
      const V4<double> gn0 = a.grad[2 * on.y], gn1 = a.grad[2 * on.y + 1];
      const V4<double> lo = a.lim[on.x], ln = a.lim[on.y];
      const V4<double> fo = a.fv[2 * id], fn = a.fv[2 * id + 1];
      const double pLT = tvd64(Wo.x, lo.x, go0.x, go0.y, fd.x, fd.y), tLT = tvd64(Wo.w, lo.w, go1.z, go1.w, fd.x, fd.y);
      const double pRT = tvd64(Wn.x, ln.x, gn0.x, gn0.y, fd.z, fd.w), tRT = tvd64(Wn.w, ln.w, gn1.z, gn1.w, fd.z, fd.w);
      Side64 l{fo.x, fo.y, fo.z, fo.w, 0.0}, r{fn.x, fn.y, fn.z, fn.w, 0.0};
      if (sL != 0)  // the TVD velocities only where the switch asks for them
        l = Side64{pLT, tvd64(Wo.y, lo.y, go0.z, go1.x, fd.x, fd.y), tvd64(Wo.z, lo.z, go0.w, go1.y, fd.x, fd.y), tLT, 0.0};
      if (sR != 0)
        r = Side64{pRT, tvd64(Wn.y, ln.y, gn0.z, gn1.x, fd.z, fd.w), tvd64(Wn.z, ln.z, gn0.w, gn1.y, fd.z, fd.w), tRT, 0.0};
      double rhoLT, rhoRT;
      densities64(l.rho, r.rho, rhoLT, rhoRT, l.p, r.p, pLT, pRT, l.T, r.T, tLT, tRT, a.invR);
      a.flux[id] = face_flux64(l, r, pLT, pRT, rhoLT, rhoRT, sL < 0 || sR < 0, gas64(a), fs);
      if constexpr (DT) {
        est = courant_bounds(a.gRf, a.dtg[id], fs, top_float(fs.w), Wo, Wn);
      }
    } else {
      const int2 on = a.on[id];
      const int own = on.x, nei = on.y;
      const V4<G> fd = a.fd[id];
      const G dxL = fd.x, dyL = fd.y, dxR = fd.z, dyR = fd.w;
      const int8_t sL = a.si[2 * own + 1], sR = a.si[2 * nei + 1];
      const bool tvdL = sL != 0, tvdR = sR != 0;
      const V4<G> fs = a.fs[id];
      const V4<typename P::W> Wo = a.W[own], Wn = a.W[nei];
      const V4<G> go0 = a.grad[2 * own], go1 = a.grad[2 * own + 1];
      const V4<G> gn0 = a.grad[2 * nei], gn1 = a.grad[2 * nei + 1];
      const V4<S> lo = a.lim[own], ln = a.lim[nei];
      const V4<G> fo = a.fv[2 * id], fn = a.fv[2 * id + 1];
      const G pLT = Wo.x + lo.x * (go0.x * dxL + go0.y * dyL);
      const G uxLT = Wo.y + lo.y * (go0.z * dxL + go1.x * dyL);
      const G uyLT = Wo.z + lo.z * (go0.w * dxL + go1.y * dyL);
      const G tLT = Wo.w + lo.w * (go1.z * dxL + go1.w * dyL);
      const G pRT = Wn.x + ln.x * (gn0.x * dxR + gn0.y * dyR);
      const G uxRT = Wn.y + ln.y * (gn0.z * dxR + gn1.x * dyR);
      const G uyRT = Wn.z + ln.z * (gn0.w * dxR + gn1.y * dyR);
      const G tRT = Wn.w + ln.w * (gn1.z * dxR + gn1.w * dyR);
      const MixedSide l{tvdL ? pLT : fo.x, tvdL ? uxLT : fo.y, tvdL ? uyLT : fo.z, tvdL ? tLT : fo.w, pLT, tLT};
      const MixedSide r{tvdR ? pRT : fn.x, tvdR ? uxRT : fn.y, tvdR ? uyRT : fn.z, tvdR ? tRT : fn.w, pRT, tRT};
      const G Sfx = fs.x, Sfy = fs.y, magSf = fs.z;
      a.flux[id] = mixed_flux<BATCH && DT>(l, r, sL < 0 || sR < 0, fs, a.Rf, a.Cvf, a.invRf, a.gm1f + 1.f);
      if constexpr (DT) {
        if (s_cfl_step) {  // setDeltaT, cudaFieldOperation.h:140-157, as an FP32 estimate
          const V2<float> g = a.dtgf[id];
          dtf32 = courant_dt_f32(s_cfl, g.x, magSf, courant_den_f32(g.y, magSf, Sfx, Sfy, Wo, Wn, a.gRf));
        }
      }
    }
  } else if (id < a.Nf + a.Nb) {  // boundary faces, reference :254-270
    const int b = id - a.Nf;
    const V4<typename P::W> wb = a.W[a.Nc + b];
    const V4<G> fs = a.fs[id];
    const G Sfx = fs.x, Sfy = fs.y;
    G R, Cv;
    if constexpr (kF32) {
      R = a.Rf;
      Cv = a.Cvf;
    } else {
      R = (G)a.R;
      Cv = (G)a.Cv;
    }
    const G bp = wb.x, bUx = wb.y, bUy = wb.z, bT = wb.w;
    const G rho = bp / (R * bT);
    const G rhoFlux = rho * (bUx * Sfx + bUy * Sfy);
    a.flux[id] = V4<typename P::F>{(typename P::F)rhoFlux, (typename P::F)(rhoFlux * bUx + bp * Sfx),
                                   (typename P::F)(rhoFlux * bUy + bp * Sfy),
                                   (typename P::F)(rhoFlux * (Cv * bT + G(0.5) * (bUx * bUx + bUy * bUy) + bp / rho))};
  }
  if constexpr (DT && kF32) {
    // block min of the float estimates on their bit patterns (non-negative floats order like
    // them; NaN sorts above +inf), then one atomicMin per block on the double's bits
    unsigned v = (unsigned)__float_as_int(dtf32);
    if (!(dtf32 >= 0.f)) v = 0x7F800000u;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned u = __shfl_xor_sync(0xffffffffu, v, o);
      v = u < v ? u : v;
    }
    __shared__ unsigned wmin32[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) wmin32[warp] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned m = wmin32[0];
      for (int k = 1; k < (int)(blockDim.x >> 5); ++k) m = wmin32[k] < m ? wmin32[k] : m;
      const float mf = __int_as_float((int)m);
      const unsigned long long bits =
          m >= 0x7F800000u ? 0x7FF0000000000000ull : (unsigned long long)__double_as_longlong((double)mf);
      atomicMin(&a.ctl->dt_bits, bits);
    }
  } else if constexpr (DT) {
    if (gt_zero(a.ctl->dt_fixed)) return;  // (the same in every thread)
    courant_block_min(est, a.ctl->cfl, &a.ctl->dt_bits, id < a.Nf, [&] {
      const int2 on = a.on[id];
      return courant_dt64(a.ctl->cfl, a.gR, a.dtg[id], a.fs[id], a.W[on.x], a.W[on.y]);
    });
  }
}

// Ghost state of boundary face b from its owner's state (reference cudaEulerBCs.h:45-95 and
// BCs/2D/<label>.h:4-10).
__device__ __forceinline__ V4<double> boundary_value(const int type, const V4<double> w, const V2<double> n) {
  switch (type) {
    case 0:  // constantTemperatureWallBoundary
      return V4<double>{w.x, 0.0, 0.0, 1.0};
    case 1:  // adiabaticWallBoundary
      return V4<double>{w.x, 0.0, 0.0, w.w};
    case 2:  // symmetryBoundary
      return V4<double>{w.x, w.y - (w.y * n.x + w.z * n.y) * n.x, w.z - (w.y * n.x + w.z * n.y) * n.y, w.w};
    case 3:  // fixedValueBoundary
      return V4<double>{1.0, 3.0, 0.0, 1.0};
    case 4:  // outletBoundary
      return w;
    case 5:  // fixedValue2Boundary
      return V4<double>{30.05945, 4.07795, 0.0, 5.97677};
    default:
      return w;
  }
}

// Error-free float addition (Knuth two-sum): s + e == a + b exactly.
__device__ __forceinline__ void two_sum(float& s, float& e, const float a, const float b) {
  s = a + b;
  const float bp = s - a;
  e = (a - (s - bp)) + (b - bp);
}

// The RK combine of one cell of the mixed policy from its residual (hi + lo) and its Un and U (from0, from):
// U (and Un after the last stage) are stored, the new primitive state returned.
__device__ __forceinline__ V4<float> advance_mixed(const StageArgs<PolicyMixed>& a, const int c, const StageCoef& k,
                                                   const float bdt, const float* hi, const float* lo,
                                                   const DF4* from0, const DF4* from) {
  const float s3 = -bdt * a.vinvf[c];
  DF4* const U = reinterpret_cast<DF4*>(a.U);
  DF4* const U0 = reinterpret_cast<DF4*>(a.U0);
  const DF4 o = *from0;
  DF base[4] = {{o.hi.x, o.lo.x}, {o.hi.y, o.lo.y}, {o.hi.z, o.lo.z}, {o.hi.w, o.lo.w}};
  if (!k.first) {  // stages 2, 3: beta1 Un + beta2 U (stage 1 is Un + increment, U not read)
    const DF4 u = *from;
    const DF b1{k.b1h, k.b1l}, b2{k.b2h, k.b2l};
    const DF uu[4] = {{u.hi.x, u.lo.x}, {u.hi.y, u.lo.y}, {u.hi.z, u.lo.z}, {u.hi.w, u.lo.w}};
#pragma unroll
    for (int q = 0; q < 4; ++q) base[q] = df_add(df_mul(b1, base[q]), df_mul(b2, uu[q]));
  }
  DF un[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) un[q] = df_add(base[q], __fmul_rn(s3, __fadd_rn(hi[q], lo[q])));
  const DF4 st{{un[0].hi, un[1].hi, un[2].hi, un[3].hi}, {un[0].lo, un[1].lo, un[2].lo, un[3].lo}};
  U[c] = st;
  if (k.last) U0[c] = st;
  float irf = __fdividef(1.f, un[0].hi);  // 1/rho: fast reciprocal + one Newton step (~1 ulp)
  irf = __fmaf_rn(irf, __fmaf_rn(-un[0].hi, irf, 1.f), irf);
  const DF ke2 = df_div(df_add(df_sqr(un[1]), df_sqr(un[2])), un[0], irf);  // |rhoU|^2 / rho
  const DF e = df_add(un[3], DF{-0.5f * ke2.hi, -0.5f * ke2.lo});
  const float pf = a.gm1f * __fadd_rn(e.hi, e.lo);
  return V4<float>{pf, un[1].hi * irf, un[2].hi * irf, pf * irf * a.invRf};
}
// The ghost of boundary face b from its cell's new state.
__device__ __forceinline__ void ghost_mixed(const StageArgs<PolicyMixed>& a, const int b, const V4<float>& wn,
                                            V4<float>* W) {
  if (a.btype[b] == AFAR_BC_FIXED_INITIAL) return;  // the ghost keeps its uploaded state
  const V4<double> g =
      boundary_value(a.btype[b], V4<double>{(double)wn.x, (double)wn.y, (double)wn.z, (double)wn.w}, a.bn[b]);
  W[a.Nc + b] = V4<float>{(float)g.x, (float)g.y, (float)g.z, (float)g.w};
}

// The mixed policy's gather + update, with no FP64 arithmetic on the path (GB300's FP64 pipe is
// 1/53 of FP32): the residual of the float fluxes is summed error-free as a float pair, the
// conserved state U, Un is stored and combined as float pairs (DF4, ~48 bits), and the pressure is
// the float-pair difference rhoE - |rhoU|^2/(2 rho) (the cancellation at high Mach costs no
// precision), rounded once to float.  k = {beta3*dt, beta1 (hi, lo), beta2 (hi, lo)} of the stage.
__device__ __forceinline__ void update_mixed(const StageArgs<PolicyMixed>& a, const int c, const StageCoef& k,
                                             const int* s_go, const float* s_bdt) {
  const int ldc = a.ldc;
  const bool live = c < a.Nc;
  const int nM = live ? a.nM[c] : 0;
  float hi[4] = {0.f, 0.f, 0.f, 0.f}, lo[4] = {0.f, 0.f, 0.f, 0.f};
  constexpr int MB = 4;
  for (int f0 = 0; f0 < nM; f0 += MB) {  // the gather needs no step size: it overlaps thread 0's work
    int fid[MB];
#pragma unroll
    for (int u = 0; u < MB; ++u) fid[u] = (f0 + u < nM) ? a.cf[(f0 + u) * ldc + c] : 1;
    V4<float> fl[MB];
#pragma unroll
    for (int u = 0; u < MB; ++u) fl[u] = a.flux[abs(fid[u]) - 1];
#pragma unroll
    for (int u = 0; u < MB; ++u) {
      if (f0 + u < nM) {
        const float sgn = fid[u] > 0 ? 1.f : -1.f;
        const float x[4] = {sgn * fl[u].x, sgn * fl[u].y, sgn * fl[u].z, sgn * fl[u].w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const DF t = df_two_sum(hi[q], x[q]);
          hi[q] = t.hi;
          lo[q] = __fadd_rn(lo[q], t.lo);
        }
      }
    }
  }
  __syncthreads();  // the block's step size (thread 0)
  if (!live || !*s_go) return;
  if (a.res_dbg) a.res_dbg[c] = V4<double>{(double)hi[0] + lo[0], (double)hi[1] + lo[1], (double)hi[2] + lo[2],
                                          (double)hi[3] + lo[3]};
  const V4<float> wn = advance_mixed(a, c, k, *s_bdt, hi, lo, reinterpret_cast<const DF4*>(a.U0) + c,
                                     reinterpret_cast<const DF4*>(a.U) + c);
  a.W[c] = wn;
  for (int fi = 0; fi < nM; ++fi) {
    const int f = abs(a.cf[fi * ldc + c]) - 1;
    if (f >= a.Nf) ghost_mixed(a, f - a.Nf, wn, a.W);
  }
}

// evaluateResidual + updateFieldData + updateBoundaryFieldData (+ storeConservedFieldData on the
// last stage), reference cudaFieldOperation.h:183-268, cudaEulerBCs.h:64-95: signed gather of the
// face fluxes in the cell's face order (no atomics), SSP-RK3 combine, conserved -> primitive, and
// the ghost state of this cell's boundary faces from the new state.
template <class P>
__device__ __forceinline__ void update_body(const StageArgs<P>& a, const int blk, const StageCoef& k) {
  // Block constants, computed once by thread 0 (a block never spans two solves): the step size,
  // whether the step is live, and for mixed beta3*dt as a float.  Per-thread code then makes no
  // FP64 operation in the mixed policy (on GB300 even an FP64 comparison costs FP64-pipe time).
  __shared__ double s_dt, s_nb3dt;  // the step; -beta3 times the step
  __shared__ int s_go;
  __shared__ float s_bdt;
  if (threadIdx.x == 0) {
    s_dt = step_dt(a.ctl);
    s_nb3dt = -k.b3 * s_dt;
    s_go = gt_zero(s_dt);  // past t_end: the step is a no-op
    if constexpr (P::id == PolicyMixed::id) s_bdt = (float)(k.b3 * s_dt);
  }
  const int c = blk * blockDim.x + threadIdx.x;
  if constexpr (P::id == PolicyMixed::id) {
    update_mixed(a, c, k, &s_go, &s_bdt);  // synchronises the block after its flux gather
  } else {
  __syncthreads();
  if (c >= a.Nc || !s_go) return;
  const double beta1 = k.b1, beta2 = k.b2, beta3 = k.b3;
  const int last_stage = k.last;
  const double deltaT = s_dt, nb3dt = s_nb3dt;
  const int ldc = a.ldc;
  const int nM = a.nM[c];
  double Rrho = 0.0, RrhoUx = 0.0, RrhoUy = 0.0, RrhoE = 0.0;
  constexpr int MB = 4;  // face ids, then fluxes, four loads in flight; sums keep the face order
  for (int f0 = 0; f0 < nM; f0 += MB) {
    int fid[MB];
#pragma unroll
    for (int u = 0; u < MB; ++u) fid[u] = (f0 + u < nM) ? a.cf[(f0 + u) * ldc + c] : 1;
    V4<typename P::F> fl[MB];
#pragma unroll
    for (int u = 0; u < MB; ++u) fl[u] = a.flux[abs(fid[u]) - 1];
#pragma unroll
    for (int u = 0; u < MB; ++u) {
      if (f0 + u < nM) {
        // the neighbour's sign as a flip of the sign bit: no conversion or product on the FP64 pipe
        const int flip = fid[u] & (int)0x80000000;
        Rrho += flip_sign(fl[u].x, flip);
        RrhoUx += flip_sign(fl[u].y, flip);
        RrhoUy += flip_sign(fl[u].z, flip);
        RrhoE += flip_sign(fl[u].w, flip);
      }
    }
  }
  if (a.res_dbg) a.res_dbg[c] = V4<double>{Rrho, RrhoUx, RrhoUy, RrhoE};
  const V4<double> o = a.U0[c];
  using WT = typename P::W;
  V4<double> un;
  V4<WT> wn;
  if constexpr (P::exact_blend) {  // the reference's eight divisions (cudaFieldOperation.h:229-242)
    const V4<double> u = a.U[c];
    const double R = a.R;
    const double gamma = a.gamma;  // R/Cv + 1, computed once on the host like GPUevolve.cu:222
    const double V = a.vol[c];
    constexpr int kSign = (int)0x80000000;
    const double rV = rcp64(V);
    const double rho = beta1 * o.x + beta2 * u.x + beta3 * deltaT * flip_sign(div64(Rrho, V, rV), kSign);
    const double rhoUx = beta1 * o.y + beta2 * u.y + beta3 * deltaT * flip_sign(div64(RrhoUx, V, rV), kSign);
    const double rhoUy = beta1 * o.z + beta2 * u.z + beta3 * deltaT * flip_sign(div64(RrhoUy, V, rV), kSign);
    const double rhoE = beta1 * o.w + beta2 * u.w + beta3 * deltaT * flip_sign(div64(RrhoE, V, rV), kSign);
    un = V4<double>{rho, rhoUx, rhoUy, rhoE};
    const double rr = rcp64(rho);
    const double p = (gamma - 1.0) * (rhoE - div64(half64(rhoUx * rhoUx + rhoUy * rhoUy), rho, rr));
    wn = V4<WT>{(WT)p, (WT)div64(rhoUx, rho, rr), (WT)div64(rhoUy, rho, rr), (WT)div64(p, R * rho)};
  } else {  // FP64 is scarce on GB300: 1/V precomputed, one reciprocal for 1/rho
    const double s3 = nb3dt * a.vinv[c];
    if (k.first) {  // beta1 = 1, beta2 = 0: U is not read
      un = V4<double>{o.x + s3 * Rrho, o.y + s3 * RrhoUx, o.z + s3 * RrhoUy, o.w + s3 * RrhoE};
    } else {
      const V4<double> u = a.U[c];
      un = V4<double>{beta1 * o.x + beta2 * u.x + s3 * Rrho, beta1 * o.y + beta2 * u.y + s3 * RrhoUx,
                      beta1 * o.z + beta2 * u.z + s3 * RrhoUy, beta1 * o.w + beta2 * u.w + s3 * RrhoE};
    }
    const double ir = rcp64(un.x);
    const double ux = un.y * ir, uy = un.z * ir;
    const double p = a.gm1 * (un.w - 0.5 * (un.y * ux + un.z * uy));
    wn = V4<WT>{(WT)p, (WT)ux, (WT)uy, (WT)(p * ir * a.invR)};
  }
  a.U[c] = un;
  if (last_stage) a.U0[c] = un;
  a.W[c] = wn;
  for (int fi = 0; fi < nM; ++fi) {
    const int f = abs(a.cf[fi * ldc + c]) - 1;
    if (f < a.Nf) continue;
    const int b = f - a.Nf;
    if (a.btype[b] == AFAR_BC_FIXED_INITIAL) continue;  // the ghost keeps its uploaded state
    const V4<double> g =
        boundary_value(a.btype[b], V4<double>{(double)wn.x, (double)wn.y, (double)wn.z, (double)wn.w}, a.bn[b]);
    a.W[a.Nc + b] = V4<WT>{(WT)g.x, (WT)g.y, (WT)g.z, (WT)g.w};
  }
  }
}

// Closes a step: advance time, record the step, re-arm the CFL minimum for the next step.
__device__ __forceinline__ void finish_one(StepCtl* ctl) {
  const double dt = step_dt(ctl);
  if (dt > 0.0) {
    ctl->t += dt;
    ctl->steps += 1;
    ctl->last_dt = dt;
    if (ctl->write_interval > 0.0)  // passed a write time (within rounding): aim at the next one
      for (int k = 0; k < 4 && ctl->t >= (double)(ctl->write_index + 1) * ctl->write_interval * (1.0 - 1e-12); ++k)
        ctl->write_index += 1;
  }
  ctl->dt_bits = (unsigned long long)__double_as_longlong(1e5);
}
// ---------------------------------------------------------------- mixed: the stage after the reconstruct
// BVD switch, face flux, residual and RK update of a tile of consecutive cells in one kernel.  As three
// kernels these pass limiters, switches and fluxes through memory and gather the cells' states and
// gradients at random (504 of the 903 B a cell and stage of the four kernels).  Here the two O3 states of
// the tile's faces come into shared memory; a cell's thread decides its switch from them and adds its
// side's TVD state; a face's thread makes the flux; the cell's thread sums its fluxes and advances.  Cells
// across the tile's border (the tiles are compact patches of the Hilbert order: about 50 for 192
// triangles) have their switch decided in every tile that needs it and a border face its flux in both its
// tiles, by the same instructions on the same inputs: the same bits.  The new states go to another buffer
// than the one read (three in turn, so a step of three stages ends where it began).
//
// What bounds it is the chain of waits of a tile, so its loads start at once: the tile's own faces (first
// cell in the tile: a contiguous range) and conserved states by bulk copies, its own cells' operands into
// registers, border and boundary faces by the threads.  The stencils' troubled-cell flags are read only
// where a 128-cell tile that they reach holds one (words of 32 flags, written by the reconstruct).
// 256 threads: with its halo a tile of 192 triangles or 152 quads is mostly one pass of the block.  Four
// blocks a SM (64 registers); five spilled and lost 8%.  us a step, separate kernels in the caller's order / fused,
// with early starts: 2.5k quads 51 / 33, 65k 68 / 60, 4.0M 2276 / 2183; 2k triangles 53 / 35, 200k 147 / 120, 2.0M 1178 / 942
// (the tail itself 443 us a step at 2.0M triangles: 1.5 TB/s; its blocks wait, on the halo's gathers and at
// their two barriers).
struct TailTile {
  int fstart;  // the tile's own faces are fstart .. fstart + nOwn - 1
  int nOwn;
  int nFace;  // with the extra ones: faces of earlier tiles' cells, boundary faces
  int nHalo;  // cells across the border; in the upper half the number of 128-cell tiles in tlist (0xFFFF: too many)
};
// Shared memory of a tile of nf faces: O3 and TVD states of both sides, face vectors, Un and U of the
// cells, the sides' switches, two mbarriers.
struct TailSmem {
  unsigned tv, tu, fs, u0, u, sw, bar, bytes;
};
__host__ __device__ inline TailSmem tail_smem(const int nf, const int cells) {
  TailSmem L;
  L.tv = nf * 32;
  L.tu = L.tv + nf * 16;
  L.fs = L.tu + nf * 16;
  L.u0 = L.fs + nf * 16;
  L.u = L.u0 + cells * 32;
  L.sw = L.u + cells * 32;
  L.bar = L.sw + (nf * 2 + 15) / 16 * 16;
  L.bytes = L.bar + 16;
  return L;
}

// A halo cell's slot: its local face with the neighbour side in bit 15 where the face is one of the tile's,
// kNoFace, kWall for a boundary face, else 2 f + side of the face, from kElsewhere on.
constexpr int kNoFace = -1, kWall = -2, kElsewhere = 0x10000;

template <int NF, bool E, bool EARLY = true>
__device__ __forceinline__ void tail_body(const StageArgs<PolicyMixed>& a, const V4<float>* Win, V4<float>* Wout,
                                          const int blk, const StageCoef& k, unsigned char* sm) {
  __shared__ int s_go, s_extra[kTailExtra];
  __shared__ float s_bdt;
  const int tid = threadIdx.x, ldc = a.ldc;
  const int T = a.tailT;  // cells a tile
  const int c0 = blk * T, nc = min(T, a.Nc - c0);
  const bool own0 = tid < T;  // this thread has an own cell first, else a halo cell
  // Loads that need no other's result, all issued before the first wait: the tile's header and lists, an
  // own cell's operands, a halo cell's id and slots; first those that no kernel writes.
  const int4 hdr = reinterpret_cast<const int4*>(a.tail)[blk];
  const int xid = tid < kTailExtra ? a.textra[(size_t)blk * kTailExtra + tid] : 0;
  const int reach = tid < kTailList ? a.tlist[(size_t)blk * kTailList + tid] : 0;
  uint2 extra_tx{0, 0};  // a test's (see g_tile_extra_tx)
  if (tid == 0) extra_tx = reinterpret_cast<const uint2*>(&g_tile_extra_tx)[1];
  int c = c0 + (own0 && tid < nc ? tid : 0), nM = 0, nS = 0;
  int lf[NF];
  V2<float> d[NF];
  float wp, wT, Lp, LT;
  V2<float> gp, gT;
  // what the switch and the TVD p and T need of a cell; the velocities' part is read where it is used
  auto load_cell = [&]() {
    wp = Win[c].x;
    wT = Win[c].w;
    gp = reinterpret_cast<const V2<float>*>(a.grad)[4 * (size_t)c];
    gT = reinterpret_cast<const V2<float>*>(a.grad)[4 * (size_t)c + 3];
    Lp = a.lim[c].x;
    LT = a.lim[c].w;
  };
  auto load_slots = [&](const int h) {  // of halo cell h
#pragma unroll
    for (int fi = 0; fi < NF; ++fi) {
      lf[fi] = a.thcode[((size_t)blk * 4 + fi) * kTailHalo + h];
      d[fi] = a.thsg[((size_t)blk * 4 + fi) * kTailHalo + h];
    }
  };
  if (own0) {
#pragma unroll
    for (int fi = 0; fi < NF; ++fi) {
      if (fi >= 3 && a.maxM < 4) continue;  // (a member of triangles in a batch with quads)
      lf[fi] = a.tlf[(size_t)fi * ldc + c];
      d[fi] = a.sg[(size_t)fi * ldc + c];  // (rows past a cell's faces hold something)
    }
    nM = a.nM[c];
    nS = a.nS[c];
  } else {
    const int h = tail_first_halo(tid, T);
    c = a.thalo[(size_t)blk * kTailHalo + h];
    load_slots(h);
  }
  pdl_wait<EARLY>();
  if (own0) load_cell();
  const int fstart = hdr.x, nOwn = hdr.y, nF = hdr.z, nX = nF - nOwn, nHalo = hdr.w & 0xFFFF, nReach = (int)((unsigned)hdr.w >> 16);
  const TailSmem S = tail_smem(nF, T);
  V4<float>* const st = reinterpret_cast<V4<float>*>(sm);          // [2 nF] O3 state of each side; then the flux
  V2<float>* const tv = reinterpret_cast<V2<float>*>(sm + S.tv);   // [2 nF] TVD p and T
  V2<float>* const tu = reinterpret_cast<V2<float>*>(sm + S.tu);   // [2 nF] TVD velocity, where the switch asks
  V4<float>* const sfs = reinterpret_cast<V4<float>*>(sm + S.fs);  // [nF] face vectors
  const DF4* const su0 = reinterpret_cast<const DF4*>(sm + S.u0);
  const DF4* const su = reinterpret_cast<const DF4*>(sm + S.u);
  int8_t* const sw = reinterpret_cast<int8_t*>(sm + S.sw);         // [2 nF] switch of each side's cell
  unsigned long long* const bar = reinterpret_cast<unsigned long long*>(sm + S.bar);
  const long long limit = g_tile_wait_limit;
  if (tid == 0) {
    mbar_init(bar, 1);
    mbar_init(bar + 1, 1);
    mbar_arrive_expect_tx(bar, (unsigned)nOwn * 48u + extra_tx.x);
    if (nOwn) {
      bulk_to_smem(st, a.fv + 2 * (size_t)fstart, (unsigned)nOwn * 32u, bar);
      bulk_to_smem(sfs, a.fs + fstart, (unsigned)nOwn * 16u, bar);
    }
    mbar_arrive_expect_tx(bar + 1, (unsigned)nc * (k.first ? 32u : 64u) + extra_tx.y);
    bulk_to_smem(sm + S.u0, a.U0 + c0, (unsigned)nc * 32u, bar + 1);
    if (!k.first) bulk_to_smem(sm + S.u, a.U + c0, (unsigned)nc * 32u, bar + 1);
  }
  // the last tile of the last stage to finish closes the step: every tile has read the step control by then
  auto done = [&]() {
    if (!k.last || tid != kTailThreads - 1) return;
    __threadfence();
    if (atomicAdd(&a.ctl->tiles_done, 1u) == (unsigned)a.nTail - 1u) {
      a.ctl->tiles_done = 0;
      finish_one(a.ctl);
    }
  };
  // Loads that needed those: border and boundary faces, the flags of the 128-cell tiles that the stencils
  // reach, a halo cell's operands, the T values of its faces elsewhere.
  V4<float> xfs, xl, xr;
  if (tid < nX) {
    xfs = a.fs[xid];
    xl = xid < a.Nf ? a.fv[2 * xid] : Win[a.Nc + (xid - a.Nf)];
    if (xid < a.Nf) xr = a.fv[2 * xid + 1];
  }
  int near = nReach == 0xFFFF;  // does any stencil of the tile reach a troubled cell?
  if (!near && tid < nReach) {
    const uint4 w = reinterpret_cast<const uint4*>(a.wflag)[reach];
    near = (w.x | w.y | w.z | w.w) != 0;
  }
  float tCur[NF], tOther[NF];
  auto load_elsewhere = [&]() {
#pragma unroll
    for (int fi = 0; fi < NF; ++fi)
      if (lf[fi] >= kElsewhere) {
        tCur[fi] = a.fv[lf[fi] - kElsewhere].w;
        tOther[fi] = a.fv[(lf[fi] - kElsewhere) ^ 1].w;
      }
  };
  bool live = own0 ? tid < nc : tid - T < nHalo;
  if (!own0 && live) {
    load_cell();
    load_elsewhere();
  }
#pragma unroll
  for (int fi = 0; fi < NF; ++fi)
    if (!live || (own0 && fi >= nM)) lf[fi] = kNoFace;
  if (tid < nX) {
    const int j = nOwn + tid;
    s_extra[tid] = xid;
    sfs[j] = xfs;
    st[2 * j] = xl;
    if (xid < a.Nf) st[2 * j + 1] = xr;
  }
  if (tid == kTailThreads - 1) {  // the block's step, as in update_body
    const double dt = step_dt(a.ctl);
    s_go = gt_zero(dt);
    s_bdt = (float)(k.b3 * dt);
  }
  // One thread polls, the block's barriers tell.  A wait that runs out marks the step invalid at once, since the
  // copy may land before the next barrier; where it has not by then, the block leaves there.
  if (tid == 0 && !mbar_wait_bounded(bar, 0, limit)) {
    near = 1;
    atomicOr(&a.ctl->err, 1u);
    if (g_tail_late_tx) mbar_complete_tx(bar, g_tail_late_tx);
  }
  near = __syncthreads_or(near);
  int lfs[NF];  // of this thread's own cell: local face of each slot, bit 15: the neighbour side; -1: none
#pragma unroll
  for (int fi = 0; fi < NF; ++fi) lfs[fi] = kNoFace;
  // first the own cells and the halo's first, then the rest of the halo
  for (int h0 = -T; h0 < nHalo; h0 += kTailThreads) {
    const int h = h0 + tid;
    const bool own = h < 0;
    if (h0 >= 0) {
      live = h < nHalo;
      if (live) {
        c = a.thalo[(size_t)blk * kTailHalo + h];
        load_slots(h);
        load_cell();
        load_elsewhere();
      } else {
#pragma unroll
        for (int fi = 0; fi < NF; ++fi) lf[fi] = kNoFace;
      }
    }
    // the switch (bvd_body)
    int shockType = 0, shockTypeExt = 0;
    if (near && live) {
      if (!own) {
        nS = a.nS[c];
        nM = a.nM[c];
      }
      shockType = (a.wflag[c >> 5] >> (c & 31)) & 1;
      shockTypeExt = shockType;
      for (int q0 = 0; q0 < nS; q0 += 10) {
        int j[10];
#pragma unroll
        for (int u = 0; u < 10; ++u) j[u] = (q0 + u < nS) ? a.sten[(size_t)(q0 + u) * ldc + c] : a.Nc;
#pragma unroll
        for (int u = 0; u < 10; ++u) {
          const int fl = j[u] < a.Nc ? (a.wflag[j[u] >> 5] >> (j[u] & 31)) & 1 : 0;  // ghosts carry no flags
          if (q0 + u < nM) shockType += fl;
          shockTypeExt += fl;
        }
      }
    }
    int bvdType = 0, walls = 0;
    const float lim = to_bj(LT);
#pragma unroll
    for (int fi = 0; fi < NF; ++fi) {
      if (lf[fi] == kNoFace) continue;
      const int l = lf[fi] & 0x7FFF;
      if (own && l >= nOwn && s_extra[l - nOwn] >= a.Nf) lf[fi] |= 0x40000;  // a boundary face of its own
      if (lf[fi] == kWall || (own && lf[fi] >= 0x40000)) {
        walls += 1;
        if (walls >= 2) bvdType = 1;  // corner cell: low order
        continue;
      }
      if (lf[fi] < kElsewhere) {
        const int side = (lf[fi] >> 15) & 1;
        tCur[fi] = st[2 * l + side].w;
        tOther[fi] = st[2 * l + (side ^ 1)].w;
      }
      const float tfTVD = tvd_mixed(wT, lim, gT.x, gT.y, d[fi]);
      const int typeval = fab(ad_(tfTVD, -tOther[fi])) < ml_(0.5f, fab(ad_(tCur[fi], -tOther[fi])));
      const int notFlat = fab(ad_(tCur[fi], -tOther[fi])) > 1e-10f;
      const int limited = (lim < 0.9f) + (shockTypeExt > 0);
      bvdType = max(bvdType, notFlat * limited * typeval);
    }
    const int type = (shockType > 0) * (shockTypeExt > 1) * (-2) + (bvdType > 0);
    if (own && live) a.si[2 * c + 1] = (int8_t)type;
    Lp = type < 0 ? to_venkat(Lp) : to_bj(Lp);
    LT = type < 0 ? to_venkat(LT) : to_bj(LT);
    V2<float> wu, gx, gy, Lu;  // Ux, Uy: state, gradients (d/dx, d/dy of each), limiters
    if (type != 0 && live) {
      wu = V2<float>{Win[c].y, Win[c].z};
      const V4<float> g0 = a.grad[2 * c], g1 = a.grad[2 * c + 1];
      gx = V2<float>{g0.z, g0.w};
      gy = V2<float>{g1.x, g1.y};
      const V4<float> L = a.lim[c];
      Lu = type < 0 ? V2<float>{to_venkat(L.y), to_venkat(L.z)} : V2<float>{to_bj(L.y), to_bj(L.z)};
    }
    // the TVD states of its faces
#pragma unroll
    for (int fi = 0; fi < NF; ++fi) {
      if (lf[fi] >= 0 && lf[fi] < kElsewhere) {
        const int at = 2 * (lf[fi] & 0x7FFF) + ((lf[fi] >> 15) & 1);
        tv[at] = V2<float>{tvd_mixed(wp, Lp, gp.x, gp.y, d[fi]), tvd_mixed(wT, LT, gT.x, gT.y, d[fi])};
        if (type != 0)
          tu[at] = V2<float>{tvd_mixed(wu.x, Lu.x, gx.x, gy.x, d[fi]), tvd_mixed(wu.y, Lu.y, gx.y, gy.y, d[fi])};
        sw[at] = (int8_t)type;
      }
    }
    if (own) {
#pragma unroll
      for (int fi = 0; fi < NF; ++fi) lfs[fi] = lf[fi];
    }
  }
  bool ok = true;
  if (tid == 0) ok = mbar_wait_bounded(bar, 0, 1) && mbar_wait_bounded(bar + 1, 0, limit);
  if (!__syncthreads_and(ok)) {  // a bulk copy did not arrive: wait (bounded) once more for both, leave
    if (tid == 0) atomicOr(&a.ctl->err, 1u);
    mbar_wait_bounded(bar, 0, limit);
    mbar_wait_bounded(bar + 1, 0, limit);
    return done();
  }
  pdl_next<EARLY>();
  // the faces' fluxes, each in the place of its first side's state
  for (int j = tid; j < nF; j += kTailThreads) {
    const V4<float> fs = sfs[j];
    V4<float> sl = st[2 * j], F;
    if (j < nOwn || s_extra[j - nOwn] < a.Nf) {
      V4<float> sr = st[2 * j + 1];
      const V4<float> t = reinterpret_cast<const V4<float>*>(tv)[j];  // both sides' p and T
      const char2 w = reinterpret_cast<const char2*>(sw)[j];
      if (w.x) sl = V4<float>{t.x, tu[2 * j].x, tu[2 * j].y, t.y};
      if (w.y) sr = V4<float>{t.z, tu[2 * j + 1].x, tu[2 * j + 1].y, t.w};
      const MixedSide l{sl.x, sl.y, sl.z, sl.w, t.x, t.y}, r{sr.x, sr.y, sr.z, sr.w, t.z, t.w};
      F = mixed_flux<E>(l, r, (signed char)w.x < 0 || (signed char)w.y < 0, fs, a.Rf, a.Cvf, a.invRf, a.gm1f + 1.f);
    } else {
      F = mixed_boundary_flux(sl, fs, a.Rf, a.Cvf);
    }
    st[2 * j] = F;
  }
  __syncthreads();
  if (tid < nc) {
    const int c = c0 + tid;
    if (s_go) {
      float hi[4] = {0.f, 0.f, 0.f, 0.f}, lo[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int fi = 0; fi < NF; ++fi) {
        if (lfs[fi] >= 0) {
          const V4<float> F = st[2 * (lfs[fi] & 0x7FFF)];
          const float sgn = (lfs[fi] & 0x8000) ? -1.f : 1.f;
          const float x[4] = {sgn * F.x, sgn * F.y, sgn * F.z, sgn * F.w};
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            if (fi == 0) {  // (every cell has a first face)
              hi[q] = x[q];
            } else {
              const DF t = df_two_sum(hi[q], x[q]);
              hi[q] = t.hi;
              lo[q] = __fadd_rn(lo[q], t.lo);
            }
          }
        }
      }
      const V4<float> wn = advance_mixed(a, c, k, s_bdt, hi, lo, su0 + tid, su + tid);
      Wout[c] = wn;
#pragma unroll
      for (int fi = 0; fi < NF; ++fi)
        if (lfs[fi] >= 0x40000) ghost_mixed(a, s_extra[(lfs[fi] & 0x7FFF) - nOwn] - a.Nf, wn, Wout);
    } else {  // past t_end: the step is a no-op, the state moves on to the next buffer
      Wout[c] = Win[c];
#pragma unroll
      for (int fi = 0; fi < NF; ++fi) {
        if (lfs[fi] < 0x40000) continue;
        const int g = a.Nc + s_extra[(lfs[fi] & 0x7FFF) - nOwn] - a.Nf;
        Wout[g] = Win[g];
      }
    }
  }
  done();
}

// ---- the tiles' lists (set-up; one block of 128 threads a tile)
constexpr int kTailHash = 512;  // halo cells of a tile in shared memory: open addressing
__device__ __forceinline__ int tail_hash_find(int* key, const int c, const bool insert) {
  for (int i = 0; i < kTailHash; ++i) {
    const int at = (int)(((unsigned)c * 2654435761u >> 7) + i) & (kTailHash - 1);
    const int was = insert ? atomicCAS(&key[at], -1, c) : key[at];
    if (was == c || (insert && was == -1)) return at;
    if (was == -1) return -1;
  }
  return -1;
}
// limits[0]: the most faces of a tile; limits[1]: set when a tile has more cells or faces than it may
__global__ void __launch_bounds__(128) k_tail_tiles(StageArgs<PolicyMixed> a, const int* start, TailTile* tiles,
                                                    int* halo, int* hcode, V2<float>* hsg, int* extra, uint16_t* lfo,
                                                    int* limits) {
  __shared__ int key[kTailHash], idx[kTailHash], nH, nX, bad;
  const int blk = blockIdx.x, tid = threadIdx.x, ldc = a.ldc;
  const int c0 = blk * a.tailT, c1 = min(c0 + a.tailT, a.Nc);
  const int f0 = start[c0], f1 = c1 < a.Nc ? start[c1] : a.Nf, nOwn = f1 - f0;
  for (int i = tid; i < kTailHash; i += 128) key[i] = -1;
  if (tid == 0) nH = nX = bad = 0;
  __syncthreads();
  for (int c = c0 + tid; c < c1; c += 128)
    for (int fi = 0; fi < a.nM[c]; ++fi) {
      const int fid = a.cf[(size_t)fi * ldc + c], f = abs(fid) - 1;
      int l = f - f0;
      if (f >= a.Nf || f < f0 || f >= f1) {
        const int x = atomicAdd(&nX, 1);
        if (x < kTailExtra)
          extra[(size_t)blk * kTailExtra + x] = f;
        else
          bad = 1;
        l = nOwn + x;
      }
      lfo[(size_t)fi * ldc + c] = (uint16_t)(min(l, 0x7FFE) | (fid < 0 ? 0x8000 : 0));
      if (f < a.Nf) {
        const int o = fid > 0 ? a.on[f].y : a.on[f].x;
        if ((o < c0 || o >= c1) && tail_hash_find(key, o, true) < 0) bad = 1;
      }
    }
  __syncthreads();
  for (int i = tid; i < kTailHash; i += 128)
    if (key[i] >= 0) {
      idx[i] = atomicAdd(&nH, 1);
      if (idx[i] < kTailHalo) halo[(size_t)blk * kTailHalo + idx[i]] = key[i];
    }
  __syncthreads();
  if (nH <= kTailHalo && nX <= kTailExtra && !bad) {
    for (int i = tid; i < 4 * nH; i += 128) {  // the halo's slots as faces elsewhere
      const int h = i >> 2, q = i & 3, o = halo[(size_t)blk * kTailHalo + h];
      const size_t at = ((size_t)blk * 4 + q) * kTailHalo + h;
      int code = kNoFace;
      if (q < a.nM[o]) {
        const int fid = a.cf[(size_t)q * ldc + o], f = abs(fid) - 1;
        code = f < a.Nf ? kElsewhere + 2 * f + (fid < 0) : kWall;
        hsg[at] = a.sg[(size_t)q * ldc + o];
      }
      hcode[at] = code;
    }
    __syncthreads();  // (the condition is the block's)
    for (int c = c0 + tid; c < c1; c += 128)  // those that are the tile's
      for (int fi = 0; fi < a.nM[c]; ++fi) {
        const int fid = a.cf[(size_t)fi * ldc + c], f = abs(fid) - 1;
        if (f >= a.Nf) continue;
        const int o = fid > 0 ? a.on[f].y : a.on[f].x;
        if (o >= c0 && o < c1) continue;
        const int h = idx[tail_hash_find(key, o, false)];
        for (int q = 0; q < a.nM[o]; ++q)
          if (a.cf[(size_t)q * ldc + o] == -fid)
            hcode[((size_t)blk * 4 + q) * kTailHalo + h] =
                (lfo[(size_t)fi * ldc + c] & 0x7FFF) | (fid > 0 ? 0x8000 : 0);
      }
  }
  if (tid == 0) {
    if (nH > kTailHalo || nX > kTailExtra || bad || nOwn + nX > 0x7FF0) atomicExch(limits + 1, 1);
    atomicMax(limits, nOwn + nX);
    tiles[blk] = TailTile{f0, nOwn, nOwn + min(nX, kTailExtra), min(nH, kTailHalo)};
  }
}
// The 128-cell tiles that the stencils of a tile's cells and halo reach.
__global__ void __launch_bounds__(128) k_tail_lists(StageArgs<PolicyMixed> a, TailTile* tiles, const int* halo,
                                                    int* list) {
  __shared__ int set[128], n, many;
  const int blk = blockIdx.x, tid = threadIdx.x;
  const int c0 = blk * a.tailT, nc = min(a.tailT, a.Nc - c0), nLoc = nc + tiles[blk].nHalo;
  set[tid] = -1;
  if (tid == 0) n = many = 0;
  __syncthreads();
  for (int i = tid; i < nLoc; i += 128) {
    const int c = i < nc ? c0 + i : halo[(size_t)blk * kTailHalo + (i - nc)];
    for (int q = -1; q < a.nS[c]; ++q) {  // the cell itself and its stencil
      const int j = q < 0 ? c : a.sten[(size_t)q * a.ldc + c];
      if (j >= a.Nc) continue;  // ghosts carry no flags
      const int t = j >> 7;
      int p = 0;
      for (; p < 128; ++p) {
        const int at = (t + p) & 127;
        const int was = atomicCAS(&set[at], -1, t);
        if (was == -1 || was == t) break;
      }
      if (p == 128) many = 1;
    }
  }
  __syncthreads();
  if (set[tid] >= 0) {
    const int at = atomicAdd(&n, 1);
    if (at < kTailList) list[(size_t)blk * kTailList + at] = set[tid];
  }
  __syncthreads();
  if (tid == 0) tiles[blk].nHalo |= (n > kTailList || many ? 0xFFFF : n) << 16;
}


// ------------------------------------------------------------------------- single-solve kernels
// One solve per launch, arguments by value (read from the parameter bank).
template <class P, bool DT>
__global__ void __launch_bounds__(128, 5) k_reconstruct_reg(StageArgs<P> a) {
  recon_reg_body<P, DT>(a, a.W, blockIdx.x);
}
template <class P, int NF, bool DT>
__global__ void __launch_bounds__(kTile, 4) k_reconstruct_tile(StageArgs<P> a) {
  extern __shared__ __align__(128) unsigned char sm[];
  recon_tile_body<P, NF, DT>(a, a.W, blockIdx.x, sm);
}
template <int NF>
__global__ void __launch_bounds__(kTailThreads, kTailBlocks) k_tail(StageArgs<PolicyMixed> a, V4<float>* Wout, const StageCoef k) {
  extern __shared__ __align__(128) unsigned char sm[];
  tail_body<NF, false>(a, a.W, Wout, blockIdx.x, k, sm);
}
template <class P>
__global__ void __launch_bounds__(128) k_reconstruct_staged(StageArgs<P> a) {
  recon_ref_body(a, blockIdx.x);
}
// fp64: its compact staging leaves room for 4 blocks an SM, which 128 registers a thread allow
template <>
__global__ void __launch_bounds__(128, 4) k_reconstruct_staged<PolicyFP64>(StageArgs<PolicyFP64> a) {
  recon_fp64_body(a, blockIdx.x);
}
template <class P>
__global__ void __launch_bounds__(128) k_bvd(StageArgs<P> a) {
  bvd_body<P>(a, blockIdx.x);
}
template <class P, bool DT>
__global__ void __launch_bounds__(256) k_flux(StageArgs<P> a) {
  flux_body<P, DT>(a, blockIdx.x);
}
// mixed: 48 registers, 5 blocks an SM (the stage-1 form takes 54 unbounded, and 4 blocks).  The
// bound is for this policy only: a minimum-blocks bound of 1 on the FP64 policies lets ptxas take
// up to 162 registers (one block an SM) where the plain bound keeps 80-120.
template <>
__global__ void __launch_bounds__(256, 5) k_flux<PolicyMixed, false>(StageArgs<PolicyMixed> a) {
  flux_body<PolicyMixed, false>(a, blockIdx.x);
}
template <>
__global__ void __launch_bounds__(256, 5) k_flux<PolicyMixed, true>(StageArgs<PolicyMixed> a) {
  flux_body<PolicyMixed, true>(a, blockIdx.x);
}
template <class P>
__global__ void __launch_bounds__(128) k_update(StageArgs<P> a, const StageCoef k) {
  update_body<P>(a, blockIdx.x, k);
}

// ---------------------------------------------------------------- the multi-point face flux
// An option of the fp64 and mixed policies (no counterpart in the reference, whose flux uses the
// face centre): the face flux as the weighted sum of the fluxes at the face's Gauss points.  The
// switch decisions (troubled cells, BVD) stay those of the face-centre values; at each point the
// state is the O3 value there, or the TVD state extrapolated there with the cell's limited
// gradient, as the cell's switch asks.

// The face values of a cell's side of each internal face at the Gauss points, with the selection
// rules of the face-centre values (recon_*_body): the O3 value where the variable varies over the
// compact stencil by at least 1e-5, else its unlimited linear value; every variable linear in a
// cell of flat temperature.  Runs after the reconstruct, whose gradient it reads.
template <class P>
__global__ void __launch_bounds__(128) k_reconstruct_gauss(StageArgs<P> a) {
  using S = typename P::S;
  using G = typename P::G;
  using WT = typename P::W;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= a.Nc) return;
  const int ldc = a.ldc, nS = a.nS[c], nM = a.nM[c], ng = a.ng, wrow = a.maxS + 1;
  const V4<WT> wc = a.W[c];
  const S pc = (S)wc.x, uxc = (S)wc.y, uyc = (S)wc.z, tc = (S)wc.w;
  S pMax = pc, pMin = pc, uxMax = uxc, uxMin = uxc, uyMax = uyc, uyMin = uyc, tMax = tc, tMin = tc;
  for (int i = 0; i < nM; ++i) {
    const V4<WT> v = a.W[a.sten[i * ldc + c]];
    pMax = gmx((S)v.x, pMax);
    pMin = gmn((S)v.x, pMin);
    uxMax = gmx((S)v.y, uxMax);
    uxMin = gmn((S)v.y, uxMin);
    uyMax = gmx((S)v.z, uyMax);
    uyMin = gmn((S)v.z, uyMin);
    tMax = gmx((S)v.w, tMax);
    tMin = gmn((S)v.w, tMin);
  }
  const V4<G> g0 = a.grad[2 * c], g1 = a.grad[2 * c + 1];  // (px py uxx uxy), (uyx uyy tx ty)
  const S SMALL = AFAR_LIT(S, 1e-5), VSMALL = AFAR_LIT(S, 1e-10);
  const bool flat = abs_lt(tMax - tMin, VSMALL);
  const bool o3p = !flat && abs_ge(pMax - pMin, SMALL), o3ux = !flat && abs_ge(uxMax - uxMin, SMALL);
  const bool o3uy = !flat && abs_ge(uyMax - uyMin, SMALL), o3t = !flat && abs_ge(tMax - tMin, SMALL);
  for (int fi = 0; fi < nM; ++fi) {
    const int fid = a.cf[fi * ldc + c];
    const int f = abs(fid) - 1;
    if (f >= a.Nf) continue;
    const int side = fid < 0;
    V4<G>* const out = a.fvg + (size_t)(2 * f + side) * ng;
    const bool all3 = o3p && o3ux && o3uy && o3t, any3 = o3p || o3ux || o3uy || o3t;
    if constexpr (std::is_same<G, double>::value) {
      // two points at a time: each member's state is read once for both, and the linear values are
      // formed only in a cell with a variable that takes them
      for (int k0 = 0; k0 < ng; k0 += 2) {
        const int n2 = min(2, ng - k0);
        V4<double> o[2];
        if (any3) {
          const double* w = a.wg + (size_t)((fi * ng + k0) * wrow) * ldc + c;
          const size_t next = n2 > 1 ? (size_t)wrow * ldc : 0;  // a single point twice
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const double w0 = w[q * next];
            o[q] = V4<double>{w0 * pc, w0 * uxc, w0 * uyc, w0 * tc};
          }
          for (int j = 0; j < nS; ++j) {
            const V4<double> v = a.W[a.sten[j * ldc + c]];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              if (q < n2) {
                const double wj = w[q * next + (size_t)(j + 1) * ldc];
                o[q].x += wj * v.x;
                o[q].y += wj * v.y;
                o[q].z += wj * v.z;
                o[q].w += wj * v.w;
              }
            }
          }
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          if (q >= n2) break;
          if (!all3) {
            const V2<double> d = a.sgk[(fi * ng + k0 + q) * ldc + c];
            if (!o3p) o[q].x = pc + g0.x * d.x + g0.y * d.y;
            if (!o3ux) o[q].y = uxc + g0.z * d.x + g1.x * d.y;
            if (!o3uy) o[q].z = uyc + g0.w * d.x + g1.y * d.y;
            if (!o3t) o[q].w = tc + g1.z * d.x + g1.w * d.y;
          }
          out[k0 + q] = o[q];
        }
      }
    } else {
      for (int k = 0; k < ng; ++k) {
        const V2<G> d = a.sgk[(fi * ng + k) * ldc + c];
        V4<G> o;
        o.x = (G)pc + g0.x * d.x + g0.y * d.y;
        o.y = (G)uxc + g0.z * d.x + g1.x * d.y;
        o.z = (G)uyc + g0.w * d.x + g1.y * d.y;
        o.w = (G)tc + g1.z * d.x + g1.w * d.y;
        if (any3) {  // the difference form of recon_tile_body
          const S* w = a.wg + (size_t)((fi * ng + k) * wrow) * ldc + c;
          G sp, sux, suy, st;
          sp = sux = suy = st = G(0);
          for (int j = 0; j < nS; ++j) {
            const S wj = w[(size_t)(j + 1) * ldc];
            const V4<WT> v = a.W[a.sten[j * ldc + c]];
            sp += wj * ((S)v.x - pc);
            sux += wj * ((S)v.y - uxc);
            suy += wj * ((S)v.z - uyc);
            st += wj * ((S)v.w - tc);
          }
          sp += (G)pc;
          sux += (G)uxc;
          suy += (G)uyc;
          st += (G)tc;
          if (o3p) o.x = sp;
          if (o3ux) o.y = sux;
          if (o3uy) o.z = suy;
          if (o3t) o.w = st;
        }
        out[k] = o;
      }
    }
  }
}

// The multi-point face flux: for each internal face, the flux at every Gauss point (state
// selection, minimised jumps, central flux and Roe/KFVS dissipation as in flux_body) times the
// point's weight, summed; boundary faces as flux_body (the ghost state is constant along the face,
// so its flux is the same at every point).  The Courant step of the first stage runs as k_delta_t.
template <class P>
__global__ void __launch_bounds__(256) k_flux_gauss(StageArgs<P> a) {
  using S = typename P::S;
  using G = typename P::G;
  const int id = blockIdx.x * blockDim.x + threadIdx.x;
  G R, Cv, iR;
  if constexpr (std::is_same<G, float>::value) {
    R = a.Rf;
    Cv = a.Cvf;
    iR = a.invRf;
  } else {
    R = (G)a.R;
    Cv = (G)a.Cv;
    iR = (G)a.invR;
  }
  if (id < a.Nf) {
    const int2 on = a.on[id];
    const int cell[2] = {on.x, on.y};
    const V4<G> fd = a.fd[id];
    const int8_t sw[2] = {a.si[2 * on.x + 1], a.si[2 * on.y + 1]};
    const bool isShock = sw[0] < 0 || sw[1] < 0;
    const V4<G> fs = a.fs[id];
    const G Sfx = fs.x, Sfy = fs.y, magSf = fs.z, nfx = Sfx * fs.w, nfy = Sfy * fs.w;
    const G gam = std::is_same<G, float>::value ? (G)(a.gm1f + 1.f) : (G)a.gamma;
    const G K = G(2) * Cv * iR - G(2);
    G acc[4] = {G(0), G(0), G(0), G(0)};
    if constexpr (std::is_same<G, double>::value) {
      for (int k = 0; k < a.ng; ++k) {
        const V2<double> off = a.fgk[(size_t)id * a.ng + k];
        Side64 st[2];
        double pT[2], tT[2];
#pragma unroll
        for (int sd = 0; sd < 2; ++sd) {
          const int c = cell[sd];
          const double dx = (sd ? fd.z : fd.x) + off.x, dy = (sd ? fd.w : fd.y) + off.y;
          const V4<double> w = a.W[c], g0 = a.grad[2 * c], g1 = a.grad[2 * c + 1], l = a.lim[c];
          pT[sd] = tvd64(w.x, l.x, g0.x, g0.y, dx, dy);
          tT[sd] = tvd64(w.w, l.w, g1.z, g1.w, dx, dy);
          if (sw[sd] != 0) {
            st[sd] = Side64{pT[sd], tvd64(w.y, l.y, g0.z, g1.x, dx, dy), tvd64(w.z, l.z, g0.w, g1.y, dx, dy), tT[sd], 0.0};
          } else {
            const V4<double> o3 = a.fvg[(size_t)(2 * id + sd) * a.ng + k];
            st[sd] = Side64{o3.x, o3.y, o3.z, o3.w, 0.0};
          }
        }
        double rhoLT, rhoRT;
        densities64(st[0].rho, st[1].rho, rhoLT, rhoRT, st[0].p, st[1].p, pT[0], pT[1], st[0].T, st[1].T, tT[0], tT[1], iR);
        const V4<double> F = face_flux64(st[0], st[1], pT[0], pT[1], rhoLT, rhoRT, isShock, gas64(a), fs);
        const double wk = a.gw[k];
        acc[0] += wk * F.x;
        acc[1] += wk * F.y;
        acc[2] += wk * F.z;
        acc[3] += wk * F.w;
      }
    } else {
      for (int k = 0; k < a.ng; ++k) {
        const V2<G> off = a.fgk[id * a.ng + k];
        G st[2][4], T[2][4], rho[2], rhoT[2];
  #pragma unroll
        for (int sd = 0; sd < 2; ++sd) {
          const int c = cell[sd];
          const G dx = (sd ? fd.z : fd.x) + off.x, dy = (sd ? fd.w : fd.y) + off.y;
          const V4<typename P::W> w = a.W[c];
          const V4<G> g0 = a.grad[2 * c], g1 = a.grad[2 * c + 1];
          const V4<S> l = a.lim[c];
          T[sd][0] = (G)w.x + l.x * (g0.x * dx + g0.y * dy);
          T[sd][1] = (G)w.y + l.y * (g0.z * dx + g1.x * dy);
          T[sd][2] = (G)w.z + l.z * (g0.w * dx + g1.y * dy);
          T[sd][3] = (G)w.w + l.w * (g1.z * dx + g1.w * dy);
          const V4<G> o3 = a.fvg[(2 * id + sd) * a.ng + k];
          const bool tvd = sw[sd] != 0;
          st[sd][0] = tvd ? T[sd][0] : o3.x;
          st[sd][1] = tvd ? T[sd][1] : o3.y;
          st[sd][2] = tvd ? T[sd][2] : o3.z;
          st[sd][3] = tvd ? T[sd][3] : o3.w;
          rho[sd] = fdiv(st[sd][0] * iR, st[sd][3]);
          rhoT[sd] = fdiv(T[sd][0] * iR, T[sd][3]);
        }
        const G dP = min_delta<G, G>(st[0][0], st[1][0], T[0][0], T[1][0]);
        const G dRho = min_delta<G, G>(rho[0], rho[1], rhoT[0], rhoT[1]);
        const G h = G(0.5);
        G F0 = h * rho[0] * (st[0][1] * Sfx + st[0][2] * Sfy) + h * rho[1] * (st[1][1] * Sfx + st[1][2] * Sfy);
        G F1 = h * (F0 * st[0][1] + st[0][0] * Sfx) + h * (F0 * st[1][1] + st[1][0] * Sfx);
        G F2 = h * (F0 * st[0][2] + st[0][0] * Sfy) + h * (F0 * st[1][2] + st[1][0] * Sfy);
        G F3 = h * F0 * (Cv * st[0][3] + h * (st[0][1] * st[0][1] + st[0][2] * st[0][2]) + R * st[0][3]) +
               h * F0 * (Cv * st[1][3] + h * (st[1][1] * st[1][1] + st[1][2] * st[1][2]) + R * st[1][3]);
        if (isShock)
          kfvs_flux_fast<G>(F0, F1, F2, F3, rho[0], rho[1], st[0][0], st[1][0], st[0][1], st[1][1], st[0][2], st[1][2],
                            st[0][3], st[1][3], R, Cv, K, magSf, nfx, nfy);
        else
          roe_flux_fast<G>(F0, F1, F2, F3, rho[0], rho[1], st[0][1], st[1][1], st[0][2], st[1][2], st[0][3], st[1][3],
                           dP, dRho, R, Cv, gam, magSf, nfx, nfy);
        const G wk = a.gw[k];
        acc[0] += wk * F0;
        acc[1] += wk * F1;
        acc[2] += wk * F2;
        acc[3] += wk * F3;
      }
    }
    a.flux[id] = V4<typename P::F>{(typename P::F)acc[0], (typename P::F)acc[1], (typename P::F)acc[2],
                                   (typename P::F)acc[3]};
  } else if (id < a.Nf + a.Nb) {  // boundary faces: the Euler flux of the ghost state
    const int b = id - a.Nf;
    const V4<typename P::W> wb = a.W[a.Nc + b];
    const V4<G> fs = a.fs[id];
    const G Sfx = fs.x, Sfy = fs.y;
    const G bp = wb.x, bUx = wb.y, bUy = wb.z, bT = wb.w;
    const G rho = bp / (R * bT);
    const G rhoFlux = rho * (bUx * Sfx + bUy * Sfy);
    a.flux[id] = V4<typename P::F>{(typename P::F)rhoFlux, (typename P::F)(rhoFlux * bUx + bp * Sfx),
                                   (typename P::F)(rhoFlux * bUy + bp * Sfy),
                                   (typename P::F)(rhoFlux * (Cv * bT + G(0.5) * (bUx * bUx + bUy * bUy) + bp / rho))};
  }
}

// ------------------------------------------------------------------------- batch kernels
// Many independent solves in one launch: block b works on solve map[b].x (its arguments are
// tab[map[b].x]), as that solve's block map[b].y.  A block never spans two solves, so block-level
// reductions (the CFL minimum, the step size) stay within one solve, and a solve's result does not
// depend on which other solves share the batch.
//
// A block first copies its member's arguments from the table into shared memory (one coalesced
// read of the entry), so the body reads every pointer and constant at shared-memory latency instead
// of one dependent load through L1 per field (the single-solve kernels have them in the parameter
// bank).  Every thread of the block takes part: call it before any thread can leave.
template <class P>
__device__ __forceinline__ const StageArgs<P>& member_args(const StageArgs<P>* __restrict__ tab, const int i) {
  static_assert(sizeof(StageArgs<P>) % 4 == 0, "the argument block is copied as 32-bit words");
  __shared__ __align__(16) unsigned raw[sizeof(StageArgs<P>) / 4];
  const unsigned* src = reinterpret_cast<const unsigned*>(tab + i);
  for (int w = threadIdx.x; w < (int)(sizeof(StageArgs<P>) / 4); w += blockDim.x) raw[w] = __ldg(src + w);
  __syncthreads();
  return *reinterpret_cast<const StageArgs<P>*>(raw);
}
template <class P, int NF>
__global__ void __launch_bounds__(kTile, 4) kb_reconstruct_tile(const StageArgs<P>* __restrict__ tab,
                                                                const int2* __restrict__ map) {
  extern __shared__ __align__(128) unsigned char sm[];
  const int2 m = map[blockIdx.x];
  const StageArgs<P>& a = member_args(tab, m.x);
  recon_tile_body<P, NF, false, false>(a, a.W, m.y, sm);
}
// The two kernels of the fused stage over up to kMembers solves, whose arguments are the launch's own
// parameters: the block finds its member from its index alone, so every pointer and constant of the
// body is an operand in the parameter bank, as in the single solve.  With the arguments staged in
// shared memory (member_args) the body keeps them in registers: the tail spilled 132 bytes a thread
// (64 registers) and took 260 us a stage at 2.0M quads, and the whole step was no faster than the separate
// kernels.  us a step, separate kernels (64-cell BVD blocks, 128-face flux blocks) / shared memory /
// parameters: 10 members of 160k quads 1110 / 1105 / 974, 8 of 90k 572 / 550 / 488, 4 of 40k
// 146 / 154 / 136, 4 of 4k 63 / 52 / 48; 12 members of 121k triangles 963 / 863 / 760, 4 of 6k 64 / 49 / 47.
template <class P>
struct MemberTable {
  static constexpr int kMembers = 48;  // what fits the 32 KB of a launch's parameters
  int n;                      // members
  int first[kMembers + 1];    // member i has blocks [first[i], first[i + 1]) of the launch
  StageArgs<P> m[kMembers];
};
template <class P>
__device__ __forceinline__ int member_of(const MemberTable<P>& t) {
  int lo = 0, hi = t.n;  // first[lo] <= block < first[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if ((int)blockIdx.x >= t.first[mid]) lo = mid;
    else hi = mid;
  }
  return lo;
}
static_assert(sizeof(MemberTable<PolicyMixed>) + sizeof(StageCoef) + 16 <= 32764, "a launch's parameters");
// (EARLY: launched as programmatic dependents; the two instructions alone cost ten members of 160k quads 1%)
template <int NF, bool DT, bool EARLY>
__global__ void __launch_bounds__(kTile, 4)
    kp_reconstruct_tile(const __grid_constant__ MemberTable<PolicyMixed> t, const int buf) {
  extern __shared__ __align__(128) unsigned char sm[];
  const int i = member_of(t);
  recon_tile_body<PolicyMixed, NF, DT, EARLY>(t.m[i], t.m[i].W3[buf], blockIdx.x - t.first[i], sm);
}
template <int NF, bool FIRST, bool EARLY>
__global__ void __launch_bounds__(kTailThreads, kTailBlocks)
    kp_tail(const __grid_constant__ MemberTable<PolicyMixed> t, const int buf, const StageCoef k) {
  extern __shared__ __align__(128) unsigned char sm[];
  const int i = member_of(t);
  tail_body<NF, FIRST, EARLY>(t.m[i], t.m[i].W3[buf], t.m[i].W3[buf == 2 ? 0 : buf + 1], blockIdx.x - t.first[i], k, sm);
}
__global__ void __launch_bounds__(128, 4) kb_reconstruct_fp64(const StageArgs<PolicyFP64>* __restrict__ tab,
                                                              const int2* __restrict__ map) {
  const int2 m = map[blockIdx.x];
  recon_fp64_body(member_args(tab, m.x), m.y);
}
// the register-pass reconstruct of the mixed policy over the members that ask for it
template <class P>
__global__ void __launch_bounds__(128, 5) kb_reconstruct_reg(const StageArgs<P>* __restrict__ tab,
                                                            const int2* __restrict__ map) {
  const int2 m = map[blockIdx.x];
  const StageArgs<P>& a = member_args(tab, m.x);
  recon_reg_body<P, false>(a, a.W, m.y);
}
// BVD and flux in blocks of B threads (the batch autotuner's choice; the map's blocks are B cells
// or faces of one member).  mixed BVD: 32 registers, the full 64 warps per SM; fp64: 40 warps.
template <class P, int B>
__global__ void __launch_bounds__(B, (P::id == PolicyMixed::id ? 2048 : 1280) / B) kb_bvd(
    const StageArgs<P>* __restrict__ tab, const int2* __restrict__ map) {
  const int2 m = map[blockIdx.x];
  bvd_body<P>(tab[m.x], m.y);  // staging its arguments cost more than it saved (32 registers)
}
template <class P, bool DT, int B>
__global__ void __launch_bounds__(B) kb_flux(const StageArgs<P>* __restrict__ tab, const int2* __restrict__ map) {
  const int2 m = map[blockIdx.x];
  flux_body<P, DT, true>(member_args(tab, m.x), m.y);
}
template <class P>
__global__ void __launch_bounds__(128) kb_update(const StageArgs<P>* __restrict__ tab, const int2* __restrict__ map,
                                                 const StageCoef k) {
  const int2 m = map[blockIdx.x];
  update_body<P>(member_args(tab, m.x), m.y, k);
}

template <class P>
__global__ void kb_finish_step(const StageArgs<P>* __restrict__ tab, const int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) finish_one(tab[i].ctl);
}

__global__ void k_finish_step(StepCtl* ctl) {
  if (threadIdx.x == 0 && blockIdx.x == 0) finish_one(ctl);
}

// The CFL step alone (adjustTimeStep of the drop-in API): min over internal faces into *bits.
// With ctl != nullptr (the step graph) it reduces into ctl->dt_bits with ctl->cfl, and does nothing
// when the step size is fixed.
template <class P>
__global__ void __launch_bounds__(256) k_delta_t(StageArgs<P> a, double CFL, unsigned long long* bits,
                                                 const StepCtl* ctl) {
  if (ctl) {
    if (ctl->dt_fixed > 0.0) return;
    CFL = ctl->cfl;
  }
  const int id = blockIdx.x * blockDim.x + threadIdx.x;
  if constexpr (P::id == PolicyMixed::id) {  // (the mixed policy's multi-point flux: in FP64 all the same)
    double dtf = 1e5;
    if (id < a.Nf) {
      const int2 on = a.on[id];
      const V4<float> Wo = a.W[on.x], Wn = a.W[on.y], fs = a.fs[id];
      const double sfx = (double)fs.x, sfy = (double)fs.y, msf = (double)fs.z;
      const V2<double> g = a.dtg[id];
      const double deltaR = g.x, fraction = g.y, Rd = a.R, Cvd = a.Cv;
      dtf = CFL * deltaR * msf /
            ((1.0 - fraction) * fabs((double)Wo.y * sfx + (double)Wo.z * sfy) +
             fraction * fabs((double)Wn.y * sfx + (double)Wn.z * sfy) +
             sqrt((Rd / Cvd + 1.0) * Rd * ((1.0 - fraction) * (double)Wo.w + fraction * (double)Wn.w)) * msf);
    }
    unsigned long long v = (unsigned long long)__double_as_longlong(dtf);
    if (!(dtf >= 0.0)) v = 0x7FF0000000000000ull;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long u = __shfl_xor_sync(0xffffffffu, v, o);
      v = u < v ? u : v;
    }
    if ((threadIdx.x & 31) == 0) atomicMin(bits, v);
  } else {
    CourantBounds est{__int_as_float(0x7F800000), __int_as_float(0x7F800000)};
    if (id < a.Nf) {
      const int2 on = a.on[id];
      const V4<double> fs = a.fs[id];
      const float i = P::id == PolicyFP64::id ? top_float(fs.w) : __fdividef(1.f, top_float(fs.z));
      est = courant_bounds((float)a.gR, a.dtg[id], fs, i, a.W[on.x], a.W[on.y]);
    }
    courant_block_min(est, CFL, bits, id < a.Nf, [&] {
      const int2 on = a.on[id];
      const V4<double> fs = a.fs[id], Wo = a.W[on.x], Wn = a.W[on.y];
      const V2<double> g = a.dtg[id];
      if constexpr (P::id == PolicyFP64::id) {
        return courant_dt64(CFL, a.gR, g, fs, Wo, Wn);
      } else {
        const double deltaR = g.x, fraction = g.y, Rd = a.R, Cvd = a.Cv;
        return CFL * deltaR * fs.z /
               ((1.0 - fraction) * fabs(Wo.y * fs.x + Wo.z * fs.y) + fraction * fabs(Wn.y * fs.x + Wn.z * fs.y) +
                sqrt((Rd / Cvd + 1.0) * Rd * ((1.0 - fraction) * Wo.w + fraction * Wn.w)) * fs.z);
      }
    });
  }
}

// The Courant step of the mixed policy for afar_adjustTimeStep: the FP32 estimate of its fused
// stage-1 flux (same expression), warp minimum on the float bits, one atomicMin per warp on the
// double's bits.  No FP64 arithmetic per face.
__global__ void __launch_bounds__(256) k_delta_t_mixed(StageArgs<PolicyMixed> a, const float cfl,
                                                       unsigned long long* bits) {
  const int id = blockIdx.x * blockDim.x + threadIdx.x;
  float dtf = 1e5f;
  if (id < a.Nf) {
    const int2 on = a.on[id];
    const V4<float> Wo = a.W[on.x], Wn = a.W[on.y];
    const V4<float> fs = a.fs[id];
    const float Sfx = fs.x, Sfy = fs.y, magSf = fs.z;
    const V2<float> g = a.dtgf[id];
    dtf = courant_dt_f32(cfl, g.x, magSf, courant_den_f32(g.y, magSf, Sfx, Sfy, Wo, Wn, a.gRf));
  }
  unsigned v = (unsigned)__float_as_int(dtf);
  if (!(dtf >= 0.f)) v = 0x7F800000u;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned u = __shfl_xor_sync(0xffffffffu, v, o);
    v = u < v ? u : v;
  }
  if ((threadIdx.x & 31) == 0) {
    const unsigned long long b = v >= 0x7F800000u
                                     ? 0x7FF0000000000000ull
                                     : (unsigned long long)__double_as_longlong((double)__int_as_float((int)v));
    atomicMin(bits, b);
  }
}

// ---------------------------------------------------------------------------------- setup kernels

// A coordinate difference taken to the nearest periodic image (L > 0), else unchanged.
__device__ __forceinline__ double wrapd(const double d, const double L) { return L > 0.0 ? d - L * rint(d / L) : d; }

// calcLeastSquareMatrix (reference cudaFieldOperation.h:91-120) into the slot-major matrix, in
// FP64 math, stored in the policy's operator type.
template <class P>
__global__ void k_setup_lsm(StageArgs<P> a, V2<typename P::S>* lsm, float* lsm_ref_layout, int maxM_ref,
                            const int* perm) {
  using S = typename P::S;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= a.Nc) return;
  const int m = a.nM[c];
  double Sxx = 0.0, Sxy = 0.0, Syy = 0.0;
  const double x0 = a.cellC[c].x, y0 = a.cellC[c].y;
  for (int i = 0; i < m; ++i) {
    const int j = a.sten[i * a.ldc + c];
    const double dx = wrapd(a.cellC[j].x - x0, a.px), dy = wrapd(a.cellC[j].y - y0, a.py);
    Sxx += dx * dx;
    Sxy += dx * dy;
    Syy += dy * dy;
  }
  for (int i = 0; i < m; ++i) {
    const int j = a.sten[i * a.ldc + c];
    const double dx = wrapd(a.cellC[j].x - x0, a.px), dy = wrapd(a.cellC[j].y - y0, a.py);
    const S m1 = (Syy * dx - Sxy * dy) / (Sxx * Syy - Sxy * Sxy);
    const S m2 = (-Sxy * dx + Sxx * dy) / (Sxx * Syy - Sxy * Sxy);
    lsm[i * a.ldc + c] = V2<S>{m1, m2};
    if (lsm_ref_layout) {
      const size_t row = perm ? perm[c] : c;  // the caller's cell
      lsm_ref_layout[2 * (size_t)maxM_ref * row + 2 * i] = (float)m1;
      lsm_ref_layout[2 * (size_t)maxM_ref * row + 2 * i + 1] = (float)m2;
    }
  }
}

// Geometry constants of each (cell, face slot): the face offset from the cell centre and the
// (delta r, fraction) pair reconstruct uses, with the reference's expressions
// (cudaLimiter.h:258-262), so the values are bit-identical to what its kernel computes per stage.
template <class P>
__global__ void k_setup_slot_geom(StageArgs<P> a, const V4<double>* faceXY) {
  using S = typename P::S;
  using G = typename P::G;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= a.Nc) return;
  const int m = a.nM[c];
  const double x0 = a.cellC[c].x, y0 = a.cellC[c].y;
  V2<G>* sg = const_cast<V2<G>*>(a.sg);
  V2<S>* sr = const_cast<V2<S>*>(a.sr);
  for (int fi = 0; fi < m; ++fi) {
    const int f = abs(a.cf[fi * a.ldc + c]) - 1;
    const double dx = wrapd(faceXY[f].x - x0, a.px);
    const double dy = wrapd(faceXY[f].y - y0, a.py);
    sg[fi * a.ldc + c] = V2<G>{(G)dx, (G)dy};
    S dR = S(1), fr = S(0);
    if (f < a.Nf) {
      const int nb = a.sten[fi * a.ldc + c];
      const double nx = wrapd(a.cellC[nb].x - x0, a.px), ny = wrapd(a.cellC[nb].y - y0, a.py);
      const float deltaR = hypot(nx, ny);
      const float fraction = sqrt(dx * dx + dy * dy) / deltaR;
      if (P::id == PolicyFP64::id) {
        const double dRd = hypot(nx, ny);
        dR = (S)(1.0 / dRd);  // its kernel multiplies by the reciprocal
        fr = (S)(sqrt(dx * dx + dy * dy) / dRd);
      } else {
        dR = (S)deltaR;
        fr = (S)fraction;
      }
    }
    sr[fi * a.ldc + c] = V2<S>{dR, fr};
  }
}

// Per-face constants: offsets of the face centre from owner and neighbour (evaluateFlux :178-182),
// the CFL geometry (setDeltaT :145-146), face vectors, boundary unit normals (symmetryBoundary.h).
template <class P>
__global__ void k_setup_face_geom(StageArgs<P> a, const V4<double>* faceXY, const V4<double>* faceS) {
  using G = typename P::G;
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= a.Nf + a.Nb) return;
  const V4<double> xy = faceXY[f];  // x, y
  const V4<double> s = faceS[f];    // Sfx, Sfy, magSf
  // fs.w: 1/|Sf| for the dissipation of the policies without bit parity (the ref policy's flux
  // divides like the reference)
  const_cast<V4<G>*>(a.fs)[f] = V4<G>{(G)s.x, (G)s.y, (G)s.z, P::id == PolicyRef::id ? G(0) : (G)(1.0 / s.z)};
  if (f < a.Nf) {
    const int2 on = a.on[f];
    const V2<double> co = a.cellC[on.x], cn = a.cellC[on.y];
    const double oxd = wrapd(xy.x - co.x, a.px), oyd = wrapd(xy.y - co.y, a.py);
    const double nxd = wrapd(xy.x - cn.x, a.px), nyd = wrapd(xy.y - cn.y, a.py);
    const_cast<V4<G>*>(a.fd)[f] = V4<G>{(G)oxd, (G)oyd, (G)nxd, (G)nyd};
    const double deltaR = hypot(wrapd(cn.x - co.x, a.px), wrapd(cn.y - co.y, a.py));
    const double fraction = hypot(oxd, oyd) / deltaR;
    if (a.dtg) const_cast<V2<double>*>(a.dtg)[f] = V2<double>{deltaR, fraction};
    if constexpr (P::id == PolicyMixed::id)
      const_cast<V2<float>*>(a.dtgf)[f] = V2<float>{(float)deltaR, (float)fraction};
  } else {
    const int b = f - a.Nf;
    const_cast<V2<double>*>(a.bn)[b] = V2<double>{s.x / s.z, s.y / s.z};
  }
}

// The multi-point face flux's per-cell arrays from the face-ordered inputs: each cell slot's O3
// weights at the points (its side's row of rbfg [face][side][point][maxS+1]; zeros past the stencil
// and for boundary faces) and the points minus the cell centre (nearest periodic image).
template <class P>
__global__ void k_setup_gauss(StageArgs<P> a, const double* rbfg, const double* pts, const int* fperm) {
  using S = typename P::S;
  using G = typename P::G;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= a.Nc) return;
  const int ng = a.ng, nmax = a.maxS + 1, ldc = a.ldc;
  S* wg = const_cast<S*>(a.wg);
  V2<G>* sgk = const_cast<V2<G>*>(a.sgk);
  const double x0 = a.cellC[c].x, y0 = a.cellC[c].y;
  for (int fi = 0; fi < a.nM[c]; ++fi) {
    const int fid = a.cf[fi * ldc + c];
    const int f = abs(fid) - 1;
    if (f >= a.Nf) continue;
    const int side = fid < 0;
    for (int k = 0; k < ng; ++k) {
      const size_t hf = fperm ? fperm[f] : f;  // the caller's face
      const double px = pts[2 * (hf * ng + k)], py = pts[2 * (hf * ng + k) + 1];
      sgk[(fi * ng + k) * ldc + c] = V2<G>{(G)wrapd(px - x0, a.px), (G)wrapd(py - y0, a.py)};
      const double* src = rbfg + ((hf * 2 + side) * ng + k) * nmax;
      for (int j = 0; j <= a.nS[c]; ++j) wg[(size_t)((fi * ng + k) * nmax + j) * ldc + c] = (S)src[j];
    }
  }
}
template <class P>
__global__ void k_setup_gauss_faces(StageArgs<P> a, const double* pts, const V4<double>* faceXY, const int* fperm) {
  using G = typename P::G;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.Nf * a.ng) return;
  const int f = i / a.ng;
  const V4<double> xy = faceXY[f];
  const size_t h = (size_t)(fperm ? fperm[f] : f) * a.ng + i % a.ng;  // the caller's face and point
  const_cast<V2<G>*>(a.fgk)[i] = V2<G>{(G)wrapd(pts[2 * h] - xy.x, a.px), (G)wrapd(pts[2 * h + 1] - xy.y, a.py)};
}

}  // namespace afar
