// pfwi acoustic path on sm_100a: forward modelling, FWI gradients (the
// reference's gradient_av imaging and the exact discrete adjoint with
// checkpointing), residual / FP64 misfit and gradient post-processing.
//
// Scheme (pywave/src/wave_fwimodeling.c:72-104, wave_fwigradient.c:132-241):
//   term = Lap8(a) (zero outside [4,pad-4)) + rr*w[it]
//   a_new = S((2a - S(b)) + (v*v*dt^2)*term),   S = sponge, b = previous a
// on the padded grid (nz+2nb) x (nx+2nb).  Field layout and two-buffer scheme
// of the afd kernels, with an 8th-order stencil; a thread updates one float4
// of z cells of one x plane.  All shots of a batch advance together in one
// launch per step, sharing V = v^2 dt^2.
#include "pw_common.cuh"

#include <algorithm>
#include <cfloat>
#include <map>
#include <mutex>
#include <cmath>

namespace pw {
namespace pf {

constexpr int HZ = 4;        // z halo (cells) in front of iz = 0
constexpr int HX = 4;        // x halo (planes) in front of ix = 0
constexpr int PF_XW = 4;     // x planes (warps) per CTA of the step kernel
constexpr int MAXS = 64;     // shots per launch
constexpr int MAXSRCW = 16;  // source-map cells per shot

// Shot geometry resolved on the host (preparation, wave_fwiutil.c:44-71).
struct ShotGeo {
  int r0v, r02, nr2;          // receivers rx = r0v + ir*drv, ir < nr2, stored at trace r02 + ir
  int nsrc;                   // non-zero source-map cells
  int sx0, sx1, sz0, sz1;     // bounding box of those cells
  int scell[MAXSRCW];         // (ix << 16) | iz of each cell
  float sw[MAXSRCW];          // source-map weight rr
};

enum Mode { FWD = 0, ADJ_REF = 1, ADJ_EXACT = 2 };

// Division by a constant d > 0 with the method of Brisebarre, Muller and
// Raina ("Accelerating correctly rounded floating-point division when the
// divisor is known in advance", IEEE Trans. Computers 53(8), 2004):
//   zh = RN(1/d), zl = RN(1/d - zh),  q = RN(x*zh + RN(x*zl))  (one FMA).
// It returns the correctly rounded x/d for every x only for some d, so each
// divisor is checked on the GPU against __fdiv_rn for all 2^23 significands
// of x in one binade; scaling x by 2^k scales every step exactly while the
// intermediate values stay normal, which |x| in [xmin, xmax] ensures.
// Below xmin (the tiny values at the edge of a wavefield) and above xmax, or
// when the check fails: div_f64; for NaN or infinity, or a divisor that is not
// finite and positive (the square of a spacing over- or underflows): __fdiv_rn,
// in step kernels of their own.
// div_f64 is checked against __fdiv_rn as well (div_f64_check_kernel); a
// divisor that failed would take __fdiv_rn there.
struct DivC {
  float d, zh, zl, xmin, xmax;  // xmin > xmax: no numerator takes the method
  int f64;                      // 1: d is finite and positive and passed the check of div_f64
  double dd, rd;                // d and RN(1/d)
};

struct PfArgs {
  int pnz, pnx;               // padded grid
  int lz;                     // leading dimension of the field layout
  int nb, nz, nx;             // sponge width, interior
  float c0, c1, c2, c3, c4;   // 8th-order coefficients (wave_fwiutil.c:17)
  float one;                  // 1.0f at run time: keeps packed products unfused (pk2 helpers)
  DivC divx, divz;            // fast exact division by dx2 / dz2
  float xlo, xhi;             // numerators that both divide as they are
  FastDiv nz4;                // float4 per padded column
  int src_z0, src_z1;         // rows of the shots' source cells
  const float *cur;           // the shots' current fields, fstep floats apart
  float *nxt;                 // the shots' previous fields, overwritten with the next
  long long fstep;
  const float *V;             // v*v*dt^2 (field layout)
  const float *bz, *bx;       // sponge factor per z / x cell (1 off the faces)
  int it, nt;
  int zig;                    // 1: odd steps run their blocks backwards
  const ShotGeo *geo;         // [nshots] (device)
  int rz, drv, nr;
  const float *wav;           // forward: wavelet [nt]
  const float *dsrc;          // forward, passive sources: field [shot][nt][nx][nz] added to the
                              // term of every interior cell (replaces the wavelet), or null
  long long dsrc_stride;      // floats between the shots' source fields
  float *rec;                 // forward: traces [shot][nt][nr] or null
  float *snap;                // forward: interior snapshot for this step [shot][nx][nz] or null
  long long snap_stride;      // floats between shots' snapshots
  float *tout;                // forward: term output [shot] (field layout) or null
  long long tout_stride;
  const float *res;           // adjoint: residual [shot][nt][nr]
  // ADJ_REF imaging: grad[ix][iz] += (w1-2w0+wm1)/wdt2 * phi * (-2/v^3) in double
  const float *wprev, *wcur, *wnext;  // snapshots wit-1, wit, wit+1 [shot][nx][nz]
  long long wstride;
  float wdt2;
  const float *m2v3;          // (float)(-2/(double)v^3) per interior cell [nx][nz]
  float *grad;                // [nx][nz] (ADJ_REF) or field layout (ADJ_EXACT: sum phi*term)
  long long gstride;          // floats between the shots' gradient slices (0: one accumulator)
  const float *tin;           // ADJ_EXACT: term of the forward step [shot] (field layout)
  long long tin_stride;
  int imaging;                // ADJ_REF: this step images
  int prev;                   // host: the mode last launched with these arguments.  A step that
                              // follows one of its own mode overlaps it (its arguments of that
                              // mode are read ahead); any other waits for all that came before
};

__device__ __forceinline__ float el(const float4 &v, int e) {
  return e == 0 ? v.x : (e == 1 ? v.y : (e == 2 ? v.z : v.w));
}
__device__ __forceinline__ void set_el(float4 &v, int e, float x) {
  if (e == 0) v.x = x; else if (e == 1) v.y = x; else if (e == 2) v.z = x; else v.w = x;
}
__device__ __forceinline__ long long pfoff(int lz, int iz, int ix) {
  return (long long)(iz + HZ) + (long long)lz * (ix + HX);
}

// largest / smallest |x| of three (a NaN wins the maximum)
__device__ __forceinline__ float max3abs(float a, float b, float c) {
  float r;
  asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float min3abs(float a, float b, float c) {
  float r;
  asm("min.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// v / d rounded once, through FP64, for finite d > 0: q = v * RN(1/d) corrected by its exact
// remainder is v / d to within a rounding of 53 bits, and equals it where
// v / d has at most 53 bits; a quotient of two floats that is no tie of the
// float grid (subnormal or not) lies at least 2^-48 of itself from every
// tie, so rounding q to float gives the correctly rounded quotient.
__device__ __forceinline__ float div_f64(float v, double d, double rd) {
  const double x = (double)v, q = __dmul_rn(x, rd);
  return __double2float_rn(__fma_rn(__fma_rn(-q, d, x), rd, q));
}

// tx / cx.d + tz / cz.d for the two pairs of cells of a float4, each quotient
// correctly rounded.  Every |numerator| in [xlo, xhi], the common part of the
// divisors' [xmin, xmax], or no result used (`unused`): the constant-divisor
// method, two values per op.  All zero (ahead of the numerical wavefront):
// zero.  Otherwise (the shell of tiny values around that zone, which crosses
// most columns while a wave expands) through FP64, or by __fdiv_rn where a
// numerator is infinite or NaN.  The first test is 8 three-operand minima and
// maxima for the 8 numerators.  IEEE: __fdiv_rn for every numerator, where a
// divisor is not finite and positive (x / inf is 0 and 0 / 0 NaN, which the
// other forms do not give); as a test in the common kernel it cost the exact
// gradient 0.6% (16 shots of 420 x 720, 20.44 -> 20.56 us per step).
// The sign of a zero quotient is not kept (these forms can give +0 for -0):
// no output depends on it.  The sum of the quotients is then +0 where it
// should be -0 only if both numerators are -0, for which the centre value c
// must be +0 (c0 c is +0 for c = -0, and a sum that starts at +0 never
// becomes -0); the update (2c - b) + V t has 2c - b = +0 - b, which is not
// -0, so adding +0 or -0 gives the same bits, and the gradient sums start at
// +0, which adding either zero leaves unchanged.
template <bool IEEE>
__device__ __forceinline__ void div4_sum(const f2 (&tx)[2], const f2 (&tz)[2], const DivC &cx,
                                         const DivC &cz, float xlo, float xhi, bool unused,
                                         f2 (&t)[2]) {
  const float4 x = join2(tx[0], tx[1]), z = join2(tz[0], tz[1]);
  float4 r;
  if (IEEE) {
#pragma unroll 1
    for (int e = 0; e < 4; e++) set_el(r, e, fadd(__fdiv_rn(el(x, e), cx.d), __fdiv_rn(el(z, e), cz.d)));
    t[0] = lo2(r);
    t[1] = hi2(r);
    return;
  }
  const float mx = max3abs(max3abs(max3abs(x.x, x.y, x.z), x.w, z.x), z.y, max3abs(z.z, z.w, 0.f));
  const float mn = min3abs(min3abs(min3abs(x.x, x.y, x.z), x.w, z.x), z.y, min3abs(z.z, z.w, z.w));
  const f2 xh = pk2(cx.zh, cx.zh), xl = pk2(cx.zl, cx.zl);
  const f2 zh = pk2(cz.zh, cz.zh), zl = pk2(cz.zl, cz.zl);
  if (unused || (mn >= xlo && mx <= xhi)) {
#pragma unroll
    for (int h = 0; h < 2; h++)
      t[h] = add2(fma2(tx[h], xh, mul2(tx[h], xl)), fma2(tz[h], zh, mul2(tz[h], zl)));
    return;
  }
  t[0] = t[1] = 0ull;
  if (mx == 0.f) return;
  if (mx <= FLT_MAX) {
#pragma unroll
    for (int e = 0; e < 4; e++)
      set_el(r, e, fadd(div_f64(el(x, e), cx.dd, cx.rd), div_f64(el(z, e), cz.dd, cz.rd)));
  } else {
#pragma unroll 1
    for (int e = 0; e < 4; e++) set_el(r, e, fadd(__fdiv_rn(el(x, e), cx.d), __fdiv_rn(el(z, e), cz.d)));
  }
  t[0] = lo2(r);
  t[1] = hi2(r);
}

__device__ __forceinline__ void pdl_sync() {
  pdl_wait();
  pdl_launch();
}
__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }

// One pfwi step: a thread updates one float4 of z cells (z4) of one x plane of
// one shot, straight from global memory (9 loads of its own column, the two z
// neighbours, the previous field and V; for the adjoint the forward term and
// the gradient).  No march, no shared memory, no barrier: the registers of
// one plane (80) leave 24 warps per SM to hide the load latency.  Lanes are
// numbered z4 + nz4 * (group of PF_XW planes) without regard to columns, so
// none is idle whatever the padded depth; the PF_XW warps of a CTA take the
// planes of the group, whose 9-plane columns overlap in L1.
// Bound: instruction issue and L1 / L2 latency (a 16-shot field pair of 420 x
// 720 sits in L2).  Measured, one launch: 16 shots of 420 x 720, forward and
// exact adjoint together 20.3 us on average (39.5 with the former x march of
// 8 planes over a shared-memory ring: 626 instructions per float4, now 290);
// 8 shots of 271 x 421 forward 6.4 us (16.1).  Marching 4 to 16 planes with
// the 9-deep queue in registers ran 23 to 28 us, two planes per thread 20.7,
// 8 planes per CTA 21.9, CTAs of consecutive lanes only 21.4.  A small survey
// (4 shots of 140 x 201) is bound by the latency of dependent launches: with
// all that no step of the mode writes read (and the imaging's division done)
// before the previous step has ended, forward and reference adjoint take 3.4
// us on average, 3.9 with all reads after it.
template <int MODE, bool PAS, bool IEEE>
__global__ void __launch_bounds__(32 * PF_XW, MODE == ADJ_REF || PAS ? 5 : 6)
    pf_step_kernel(const __grid_constant__ PfArgs a) {
  const int s = zigzag(a.it & a.zig, blockIdx.y, gridDim.y);
  const unsigned item = zigzag(a.it & a.zig, blockIdx.x, gridDim.x) * 32 + (threadIdx.x & 31);
  const int chunk = fast_div(item, a.nz4);
  const int z4 = (int)item - chunk * a.nz4.d;
  const int x = chunk * PF_XW + (threadIdx.x >> 5);
  const int iz0 = 4 * z4;
  const bool live = x < a.pnx;
  const long long lz = a.lz;
  const long long o0 = pfoff(a.lz, iz0, x);  // own float4
  const float *pc = a.cur + s * a.fstep + o0;
  float *pn = a.nxt + s * a.fstep + o0;
  float *pg = MODE == ADJ_EXACT ? a.grad + s * a.gstride + o0 : nullptr;
  float *po = (MODE == FWD && a.tout) ? a.tout + s * a.tout_stride + o0 : nullptr;
  float *const gs = MODE == ADJ_REF ? a.grad + s * a.gstride : nullptr;
  const ShotGeo &sg = a.geo[s];
  const bool rec_row = a.rz >= iz0 && a.rz < iz0 + 4;
  const bool xin = x >= a.nb && x < a.nb + a.nx;
  const bool img = MODE == ADJ_REF && a.imaging && xin;

  // what no step of this mode writes, read before the previous step has ended
  float4 V4 = make_float4(0.f, 0.f, 0.f, 0.f), bz4 = V4, tf = V4, g4 = V4;
  float bxf = 0.f, resid = 0.f;
  int rir = -1;
  double rw[4];  // ADJ_REF imaging operands
  float rt[4], rg[4];
  if (live) {
    V4 = ld4(a.V + o0);
    bz4 = ld4(a.bz + iz0);
    bxf = a.bx[x];
    if (MODE == ADJ_EXACT)
      tf = __ldcs(reinterpret_cast<const float4 *>(a.tin + s * a.tin_stride + o0));
    if (rec_row) {
      const int d = x - sg.r0v;
      if (d >= 0) {
        const int ir = a.drv == 1 ? d : (d % a.drv == 0 ? d / a.drv : -1);
        if (ir >= 0 && ir < sg.nr2) rir = sg.r02 + ir;
      }
      if (MODE != FWD && rir >= 0) resid = a.res[((size_t)s * a.nt + a.it) * a.nr + rir];
    }
  }
  if (MODE == ADJ_REF) {
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const int iz = iz0 + e;
      rw[e] = 0.;
      rt[e] = 0.f;
      if (img && iz >= a.nb && iz < a.nb + a.nz) {
        const size_t k = (size_t)(x - a.nb) * a.nz + (iz - a.nb);
        const size_t ks = s * a.wstride + k;
        // (wave[wit+1] - 2.*wave[wit] + wave[wit-1]) / wdt2 in double, left to right
        rw[e] = __dadd_rn(__dsub_rn((double)a.wnext[ks], __dmul_rn(2., (double)a.wcur[ks])),
                          (double)a.wprev[ks]);
        rw[e] = __ddiv_rn(rw[e], (double)a.wdt2);
        rt[e] = a.m2v3[k];
      }
    }
  }
  pdl_sync();
  if (!live) return;

  float4 q[9];  // own column, planes x-4 .. x+4
#pragma unroll
  for (int d = 0; d < 9; d++) q[d] = ld4(pc + (d - 4) * lz);
  const float4 c = q[4], L = ld4(pc - 4), R = ld4(pc + 4), p4 = ld4(pn);
  if (MODE == ADJ_EXACT) g4 = ld4(pg);
  if (MODE == ADJ_REF) {
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const int iz = iz0 + e;
      rg[e] = img && iz >= a.nb && iz < a.nb + a.nz ? gs[(size_t)(x - a.nb) * a.nz + (iz - a.nb)] : 0.f;
    }
  }
  // the stencil's rows [4, pnz - 4): the first and the last float4 of a column
  // hold none, at most one float4 holds some of both
  const bool lz_any = z4 >= 1 && iz0 < a.pnz - 4;
  const bool lz_full = lz_any && iz0 + 3 < a.pnz - 4;
  const bool src_z = MODE == FWD && !PAS && iz0 <= a.src_z1 && iz0 + 3 >= a.src_z0;
  const f2 k1 = pk2(a.one, a.one);
  const f2 kc[5] = {pk2(a.c0, a.c0), pk2(a.c1, a.c1), pk2(a.c2, a.c2), pk2(a.c3, a.c3),
                    pk2(a.c4, a.c4)};
  float dv[4] = {0.f, 0.f, 0.f, 0.f};
  if (MODE == FWD && PAS) {
    // the interior cells' source samples
    const float *row = a.dsrc + s * a.dsrc_stride +
                       ((long long)a.it * a.nx + (xin ? x - a.nb : 0)) * a.nz;
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const int iz = iz0 + e;
      if (xin && iz >= a.nb && iz < a.nb + a.nz) dv[e] = __ldcs(row + (iz - a.nb));
    }
  }
  // receivers read the field before the update (wave_fwimodeling.c:76-79)
  if (MODE == FWD && rir >= 0 && a.rec)
    a.rec[((size_t)s * a.nt + a.it) * a.nr + rir] = el(c, a.rz - iz0);
  if (MODE == FWD && a.snap && xin) {
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const int iz = iz0 + e;
      if (iz >= a.nb && iz < a.nb + a.nz)
        a.snap[s * a.snap_stride + (size_t)(x - a.nb) * a.nz + (iz - a.nb)] = el(c, e);
    }
  }
  // the x and z sums of the 8th-order Laplacian in the reference's order,
  // cells (0, 1) and (2, 3) of the float4 per f32x2 op; the z neighbours
  // at odd distances are the float4s shifted by one cell
  const f2 cl = lo2(c), ch = hi2(c);
  const bool lx_ok = x >= 4 && x < a.pnx - 4;
  f2 t2[2];
  {
    const f2 s_wx = pk2(L.w, c.x), s_yz = pk2(c.y, c.z), s_wR = pk2(c.w, R.x);
    const f2 s_Lyz = pk2(L.y, L.z), s_Ryz = pk2(R.y, R.z);
    // z partners (+d, -d) of each pair, d = 1 .. 4
    const f2 zp[2][4] = {{s_yz, ch, s_wR, lo2(R)}, {s_wR, lo2(R), s_Ryz, hi2(R)}};
    const f2 zm[2][4] = {{s_wx, hi2(L), s_Lyz, lo2(L)}, {s_yz, cl, s_wx, hi2(L)}};
    f2 tx2[2], tz2[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      f2 tx = mul2(mul2(kc[0], h ? ch : cl), k1);
      f2 tz = tx;
#pragma unroll
      for (int d = 1; d <= 4; d++) {
        const float4 &xp = q[4 + d], &xm = q[4 - d];
        const f2 xs = h ? add2(hi2(xp), hi2(xm)) : add2(lo2(xp), lo2(xm));
        tx = add2(tx, mul2(mul2(kc[d], xs), k1));
      }
#pragma unroll
      for (int d = 1; d <= 4; d++)
        tz = add2(tz, mul2(mul2(kc[d], add2(zp[h][d - 1], zm[h][d - 1])), k1));
      tx2[h] = tx;
      tz2[h] = tz;
    }
    div4_sum<IEEE>(tx2, tz2, a.divx, a.divz, a.xlo, a.xhi, !(lz_any && lx_ok), t2);
  }
  float4 term4 = join2(t2[0], t2[1]);
  if (!(lz_full && lx_ok)) {
#pragma unroll
    for (int e = 0; e < 4; e++)
      if (!(lz_any && lx_ok && iz0 + e < a.pnz - 4)) set_el(term4, e, 0.f);
  }
  if (MODE == FWD && PAS) {
    // gradient_pas_av (wave_fwigradient.c:732-737): the interior's source
    // sample; its update covers the stencil's cells only, so none is
    // added on the 4-cell rim
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const int iz = iz0 + e;
      if (iz >= 4 && iz < a.pnz - 4 && lx_ok && xin && iz >= a.nb && iz < a.nb + a.nz)
        set_el(term4, e, fadd(el(term4, e), dv[e]));
    }
  } else if (MODE == FWD) {
    if (src_z && x >= sg.sx0 && x <= sg.sx1) {
      const float w = a.wav[a.it];
#pragma unroll
      for (int e = 0; e < 4; e++)
        for (int k = 0; k < sg.nsrc; k++)
          if (sg.scell[k] == ((x << 16) | (iz0 + e)))
            set_el(term4, e, fadd(el(term4, e), fmul(sg.sw[k], w)));
    }
  } else if (rir >= 0) {
#pragma unroll
    for (int e = 0; e < 4; e++)
      if (iz0 + e == a.rz) set_el(term4, e, fadd(el(term4, e), resid));
  }
  {
    // b = S(a_{k-1} as stored): z faces then x faces (apply_sponge);
    // 2 c as c + c (the same bits, and no product to fuse into the
    // subtraction).  Cells beyond pnz and pnx stay zero: every operand
    // is zero there
    const f2 bx2 = pk2(bxf, bxf);
    f2 r2[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const f2 bz2 = h ? hi2(bz4) : lo2(bz4);
      const f2 cv2 = h ? ch : cl;
      const f2 p = mul2(mul2(bx2, mul2(bz2, h ? hi2(p4) : lo2(p4))), k1);
      const f2 vt = mul2(mul2(h ? hi2(V4) : lo2(V4), h ? hi2(term4) : lo2(term4)), k1);
      const f2 v = add2(sub2(add2(cv2, cv2), p), vt);
      r2[h] = mul2(bx2, mul2(bz2, v));
    }
    *reinterpret_cast<float4 *>(pn) = join2(r2[0], r2[1]);
  }
  if (MODE == FWD && a.tout) __stcs(reinterpret_cast<float4 *>(po), term4);
  if (MODE == ADJ_EXACT) {
    // dJ/dV accumulates phi_n * term_n (divided by V at the end)
    *reinterpret_cast<float4 *>(pg) =
        join2(add2(lo2(g4), mul2(mul2(cl, lo2(tf)), k1)),
              add2(hi2(g4), mul2(mul2(ch, hi2(tf)), k1)));
  }
  if (MODE == ADJ_REF && img) {
    // gradient_av (wave_fwigradient.c:221-230): the C expression in
    // double, unfused, added to the float gradient
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const int iz = iz0 + e;
      if (iz >= a.nb && iz < a.nb + a.nz) {
        const size_t k = (size_t)(x - a.nb) * a.nz + (iz - a.nb);
        const double gsum = __dmul_rn(__dmul_rn(rw[e], (double)el(c, e)), (double)rt[e]);
        gs[k] = __double2float_rn(__dadd_rn((double)rg[e], gsum));
      }
    }
  }
}


// FP64 misfit and residual, one thread per (shot, it, ir):
//   REFERENCE: r = dobs - d, J += 0.5 r^2 (unweighted), adjoint source r*w
//   EXACT:     r = d - dobs, J += 0.5 w r^2, adjoint source w*r
// d, dobs, res: [shot][nt][nr]; w: [nr][nt] (residual_weighting layout) or
// null (every weight 1).
__global__ void residual_kernel(const float *d, const float *dobs, const float *w, float *res,
                                int ns, int nt, int nr, int exact, double *misfit) {
  const long long n = (long long)ns * nt * nr;
  double acc = 0.0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int ir = int(i % nr);
    const int it = int((i / nr) % nt);
    const float wt = w ? w[(size_t)ir * nt + it] : 1.f;
    if (exact) {
      const float r = fsub(d[i], dobs[i]);
      acc += 0.5 * (double)wt * (double)r * (double)r;
      res[i] = fmul(wt, r);
    } else {
      const float r = fsub(dobs[i], d[i]);
      acc += 0.5 * (double)r * (double)r;
      res[i] = fmul(r, wt);
    }
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  __shared__ double part[32];
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x < 32) {
    double v = threadIdx.x < (blockDim.x >> 5) ? part[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (threadIdx.x == 0) misfit[1 + blockIdx.x] = v;  // block sums, added in order below
  }
}

// misfit[0] += the block sums misfit[1 .. nblocks] in block order (the same
// bits on every run, whatever order the blocks ran in)
__global__ void misfit_sum_kernel(double *misfit, int nblocks) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    double s = misfit[0];
    for (int b = 0; b < nblocks; b++) s += misfit[1 + b];
    misfit[0] = s;
  }
}
constexpr int RESID_BLOCKS = 592;

// A Butterworth filter as np_butter_init builds it (wave_butter.c:18-62):
// for odd nn one first-order section (den[nn/2]), and nn/2 second-order
// sections sharing the middle coefficient `mid`.
constexpr int BUTTER_MAXP = 16;
struct ButterCoef {
  int nn, low;
  float den[BUTTER_MAXP / 2 + 1][2];
  float mid;
};

// One causal sweep of np_butter_apply (wave_butter.c:64-102) over the n
// samples x[0], x[st], ..., in index order or (bwd) from the last sample to
// the first -- reverse, apply, reverse in one pass.  Sections run one after
// the other over the whole trace, each product and sum in the reference's
// order.
__device__ __forceinline__ void butter_sweep(const ButterCoef &b, float *x, long long st, int n,
                                             bool bwd) {
  const float d1 = b.mid;
  if (b.nn % 2) {
    const float d0 = b.den[b.nn / 2][0], d2 = b.den[b.nn / 2][1];
    float x0 = 0.f, x1, y1 = 0.f;
    for (int k = 0; k < n; k++) {
      const long long i = (long long)(bwd ? n - 1 - k : k) * st;
      x1 = x0;
      x0 = x[i];
      const float u = b.low ? fadd(x0, x1) : fsub(x0, x1);
      y1 = fmul(fsub(u, fmul(d2, y1)), d0);
      x[i] = y1;
    }
  }
  for (int j = 0; j < b.nn / 2; j++) {
    const float d0 = b.den[j][0], d2 = b.den[j][1];
    float x0 = 0.f, x1 = 0.f, x2, y1 = 0.f, y2 = 0.f;
    for (int k = 0; k < n; k++) {
      const long long i = (long long)(bwd ? n - 1 - k : k) * st;
      x2 = x1;
      x1 = x0;
      x0 = x[i];
      const float t = fmul(2.f, x1);
      const float u = b.low ? fadd(fadd(x0, t), x2) : fadd(fsub(x0, t), x2);
      const float y0 = fmul(fsub(fsub(u, fmul(d1, y1)), fmul(d2, y2)), d0);
      y2 = y1;
      y1 = y0;
      x[i] = y0;
    }
  }
}

// pw_butter_apply: one causal sweep per trace, traces x [ntr][n]
__global__ void butter_traces_kernel(const ButterCoef b, float *x, int n, int ntr) {
  const int tr = blockIdx.x * blockDim.x + threadIdx.x;
  if (tr < ntr) butter_sweep(b, x + (size_t)tr * n, 1, n, false);
}

// The multiscale residual filter of gradient_pas_av (wave_fwigradient.c:
// 767-784) on res [shot][nt][nr]: per trace the zero-phase high-pass (apply,
// reverse, apply, reverse), then the low-pass, then the residual weight
// w [nr][nt] (or 1).
__global__ void butter_residual_kernel(const ButterCoef lo, const ButterCoef hi, int use_lo,
                                       int use_hi, float *res, int ns, int nt, int nr,
                                       const float *w) {
  const int tr = blockIdx.x * blockDim.x + threadIdx.x;
  if (tr >= ns * nr) return;
  const int s = tr / nr, ir = tr - s * nr;
  float *x = res + (size_t)s * nt * nr + ir;
  if (use_lo) {
    butter_sweep(lo, x, nr, nt, false);
    butter_sweep(lo, x, nr, nt, true);
  }
  if (use_hi) {
    butter_sweep(hi, x, nr, nt, false);
    butter_sweep(hi, x, nr, nt, true);
  }
  if (w)
    for (int it = 0; it < nt; it++) x[(size_t)it * nr] = fmul(x[(size_t)it * nr], w[(size_t)ir * nt + it]);
}

// np_butter_init on the host, its float/double mix kept
static ButterCoef butter_coef(bool low, float cutoff, int nn) {
  const double pi = 3.14159265358979323846264338328;
  ButterCoef b{};
  b.nn = nn;
  b.low = low ? 1 : 0;
  const float arg = 2. * pi * cutoff;
  const float sinw = ::sinf(arg), cosw = ::cosf(arg);
  float fact;
  if (nn % 2) {
    if (low) {
      fact = (1. + cosw) / sinw;
      b.den[nn / 2][0] = 1. / (1. + fact);
      b.den[nn / 2][1] = 1. - fact;
    } else {
      fact = sinw / (1. + cosw);
      b.den[nn / 2][0] = 1. / (fact + 1.);
      b.den[nn / 2][1] = fact - 1.;
    }
  }
  fact = low ? ::sinf(0.5 * arg) : ::cosf(0.5 * arg);
  fact *= fact;
  for (int j = 0; j < nn / 2; j++) {
    const float ss = ::sinf(pi * (2 * j + 1) / (2 * nn)) * sinw;
    b.den[j][0] = fact / (1. + ss);
    b.den[j][1] = (1. - ss) / fact;
  }
  b.mid = -2. * cosw / fact;
  return b;
}

// total[i] += slice_0[i] + slice_1[i] + ... in shot order (deterministic)
__global__ void sum_slices_kernel(const float *slices, int nb, long long n, float *total) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    float v = total[i];
    for (int s = 0; s < nb; s++) v = fadd(v, slices[s * n + i]);
    total[i] = v;
  }
}

// V = (v*v)*dt2 on the padded grid (pad2d edge replication, wave_fwiutil.c:123-147)
__global__ void pad_V_kernel(const float *vel, int nz, int nx, int nb, int pnz, int pnx, int lz,
                             float dt2, float *V) {
  const long long n = (long long)pnz * pnx;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int iz = int(i % pnz), ix = int(i / pnz);
    const int jz = min(max(iz - nb, 0), nz - 1), jx = min(max(ix - nb, 0), nx - 1);
    const float v = vel[(size_t)jx * nz + jz];
    V[pfoff(lz, iz, ix)] = fmul(fmul(v, v), dt2);
  }
}

// [rows][cols] -> [cols][rows]
__global__ void transpose_kernel(const float *in, float *out, long long rows, long long cols) {
  __shared__ float t[32][33];
  const long long c0 = (long long)blockIdx.x * 32, r0 = (long long)blockIdx.y * 32;
  for (int j = threadIdx.y; j < 32; j += blockDim.y) {
    const long long r = r0 + j, c = c0 + threadIdx.x;
    if (r < rows && c < cols) t[j][threadIdx.x] = in[r * cols + c];
  }
  __syncthreads();
  for (int j = threadIdx.y; j < 32; j += blockDim.y) {
    const long long c = c0 + j, r = r0 + threadIdx.x;
    if (r < rows && c < cols) out[c * rows + r] = t[threadIdx.x][j];
  }
}

// (float)(-2./temp) with temp = v*v*v in float (wave_fwigradient.c:224-226),
// once per call instead of per cell and step
__global__ void m2v3_kernel(const float *vel, size_t n, float *out) {
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n;
       k += (size_t)gridDim.x * blockDim.x) {
    const float v = vel[k];
    out[k] = __double2float_rn(__ddiv_rn(-2., (double)__fmul_rn(__fmul_rn(v, v), v)));
  }
}

// Sum of a value per thread over a block of 256, in a fixed tree (thread 0's result).
__device__ __forceinline__ double block_sum(double v) {
  __shared__ double part[8];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0)
    for (int k = 0; k < 8; k++) s += part[k];
  return s;
}

// Exact gradient: dJ/dv_pad = 2 * sum(phi*term) / v_pad, folded back through
// pad2d's edge replication onto the interior (the padded cells that copy an
// interior cell, summed in FP64 in a fixed order).
// Blocks 0 .. 3 sum the corner cells ((nb + 1)^2 padded cells each, 160 us
// for one thread at nb 60), the others every other cell, one per thread.
__global__ void __launch_bounds__(256) fold_grad_kernel(const float *gacc, const float *vel, int nz,
                                                        int nx, int nb, int pnz, int pnx, int lz,
                                                        float *grad) {
  if (blockIdx.x < 4) {
    const int jz = (blockIdx.x & 1) ? nz - 1 : 0, jx = (blockIdx.x & 2) ? nx - 1 : 0;
    const int z_lo = jz == 0 ? 0 : jz + nb, z_hi = jz == nz - 1 ? pnz - 1 : jz + nb;
    const int x_lo = jx == 0 ? 0 : jx + nb, x_hi = jx == nx - 1 ? pnx - 1 : jx + nb;
    const int cz = z_hi - z_lo + 1, n = cz * (x_hi - x_lo + 1);
    double s = 0.0;
    for (int k = threadIdx.x; k < n; k += 256)
      s += (double)gacc[pfoff(lz, z_lo + k % cz, x_lo + k / cz)];
    s = block_sum(s);
    const long long i = (long long)jx * nz + jz;
    if (threadIdx.x == 0) grad[i] = (float)(2.0 * s / (double)vel[i]);
    return;
  }
  const long long n = (long long)nz * nx;
  for (long long i = (blockIdx.x - 4) * 256LL + threadIdx.x; i < n; i += (gridDim.x - 4) * 256LL) {
    const int jz = int(i % nz), jx = int(i / nz);
    if ((jz == 0 || jz == nz - 1) && (jx == 0 || jx == nx - 1)) continue;
    const int z_lo = jz == 0 ? 0 : jz + nb, z_hi = jz == nz - 1 ? pnz - 1 : jz + nb;
    const int x_lo = jx == 0 ? 0 : jx + nb, x_hi = jx == nx - 1 ? pnx - 1 : jx + nb;
    double s = 0.0;
    for (int ix = x_lo; ix <= x_hi; ix++)
      for (int iz = z_lo; iz <= z_hi; iz++) s += (double)gacc[pfoff(lz, iz, ix)];
    grad[i] = (float)(2.0 * s / (double)vel[i]);
  }
}

// ---------------------------------------------- post-processing kernels --
// One line of np_smooth2 (wave_triangle.c:177-238) per thread, in the
// reference's float order; tmp: per-thread scratch of n + 2*rect floats.
__device__ void smooth2_line(int nb, int n, float *x, long long o, long long d, float *tmp) {
  const int np = n + 2 * nb;
  const float wt = (float)(1.0 / (nb * nb));
  float t;
  for (int i = 0; i < np; i++) tmp[i] = 0.f;
  for (int i = 0; i < n; i++) tmp[i] = fadd(tmp[i], fmul(-wt, x[o + i * d]));
  const float w2 = (float)(2. * wt);
  for (int i = 0; i < n; i++) tmp[i + nb] = fadd(tmp[i + nb], fmul(w2, x[o + i * d]));
  for (int i = 0; i < n; i++) tmp[i + 2 * nb] = fadd(tmp[i + 2 * nb], fmul(-wt, x[o + i * d]));
  t = 0.f;
  for (int i = 0; i < np; i++) { t = fadd(t, tmp[i]); tmp[i] = t; }
  t = 0.f;
  for (int i = np - 1; i >= 0; i--) { t = fadd(t, tmp[i]); tmp[i] = t; }
  for (int i = 0; i < n; i++) x[o + i * d] = tmp[i + nb];
  for (int m = 0; m < nb; m++) {  // right extension: mirrored, then direct, ...
    const int b = m / n, i = m % n;
    const int dst = (b % 2 == 0) ? (n - 1 - i) : i;
    x[o + dst * d] = fadd(x[o + dst * d], tmp[nb + n + m]);
  }
  for (int m = 0; m < nb; m++) {  // left extension: direct, then mirrored, ...
    const int b = m / n, i = m % n;
    const int dst = (b % 2 == 0) ? i : (n - 1 - i);
    x[o + dst * d] = fadd(x[o + dst * d], tmp[nb - 1 - m]);
  }
}

__global__ void smooth_lines_kernel(float *x, int nlines, int n, long long line_step,
                                    long long elem_step, int rect, float *scratch) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= nlines) return;
  smooth2_line(rect, n, x, (long long)l * line_step, elem_step, scratch + (size_t)l * (n + 2 * rect));
}

__global__ void absmax_kernel(const float *x, long long n, unsigned int *out) {
  float m = 0.f;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    m = fmaxf(m, fabsf(x[i]));
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out, __float_as_uint(m));
}

__global__ void vel_check_kernel(const float *x, long long n, unsigned int *out) {
  float m = 0.f;
  unsigned bad = 0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const float v = x[i];
    if (!(v > 0.f) || !isfinite(v)) bad = 1;
    else m = fmaxf(m, v);
  }
  for (int o = 16; o > 0; o >>= 1) {
    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    bad |= __shfl_xor_sync(0xffffffffu, bad, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMax(out, __float_as_uint(m));
    if (bad) atomicOr(out + 1, 1u);
  }
}

// waterz rows to zero and the scale factor (gradient_smooth2 tail,
// wave_fwiutil.c:323-334); scaling <= 0 means "derive 0.1/max|g| here"
__global__ void finish_kernel(float *g, int nz, int nx, int waterz, const unsigned int *mx,
                              float *scaling) {
  float sc = *scaling;
  if (sc <= 0.f) sc = (float)(0.1 / (double)__uint_as_float(*mx));
  const long long n = (long long)nz * nx;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int iz = int(i % nz);
    float v = g[i];
    if (waterz >= 0 ? iz < waterz : iz >= nz + waterz) v = 0.f;
    g[i] = fmul(v, sc);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0 && *scaling <= 0.f) *scaling = sc;
}

// ------------------------------------------------------------------ host --

// Restated source map: a unit spike at (sx, sz) smoothed with rect 2 along
// z then x (source_map, wave_fwiutil.c:149-177), on the host in float.
static void smooth_line_host(int nb, int n, float *x, long long o, long long d, std::vector<float> &tmp) {
  const int np = n + 2 * nb;
  tmp.assign(np, 0.f);
  const float wt = (float)(1.0 / (nb * nb));
  for (int i = 0; i < n; i++) tmp[i] += (-wt) * x[o + i * d];
  for (int i = 0; i < n; i++) tmp[i + nb] += ((float)(2. * wt)) * x[o + i * d];
  for (int i = 0; i < n; i++) tmp[i + 2 * nb] += (-wt) * x[o + i * d];
  float t = 0.f;
  for (int i = 0; i < np; i++) { t += tmp[i]; tmp[i] = t; }
  t = 0.f;
  for (int i = np - 1; i >= 0; i--) { t += tmp[i]; tmp[i] = t; }
  for (int i = 0; i < n; i++) x[o + i * d] = tmp[i + nb];
  for (int m = 0; m < nb; m++) {
    const int b = m / n, i = m % n;
    const int dst = (b % 2 == 0) ? (n - 1 - i) : i;
    x[o + dst * d] += tmp[nb + n + m];
  }
  for (int m = 0; m < nb; m++) {
    const int b = m / n, i = m % n;
    const int dst = (b % 2 == 0) ? i : (n - 1 - i);
    x[o + dst * d] += tmp[nb - 1 - m];
  }
}

static int source_map(int sx, int sz, int pnz, int pnx, ShotGeo &sg) {
  // the map is separable and local: smooth a small window around the spike
  const int r = 6;
  const int x_lo = std::max(0, sx - r), x_hi = std::min(pnx - 1, sx + r);
  const int z_lo = std::max(0, sz - r), z_hi = std::min(pnz - 1, sz + r);
  // the fold reflections need the full line when the spike is near an edge
  const bool full = x_lo == 0 || z_lo == 0 || x_hi == pnx - 1 || z_hi == pnz - 1;
  std::vector<float> m, tmp;
  int zs, xs, nzw, nxw;
  if (full) { zs = 0; xs = 0; nzw = pnz; nxw = pnx; }
  else { zs = z_lo; xs = x_lo; nzw = z_hi - z_lo + 1; nxw = x_hi - x_lo + 1; }
  // smoothing a window equals smoothing the full line when the window
  // holds the whole support (rect 2 spreads one cell each way)
  m.assign((size_t)nzw * nxw, 0.f);
  m[(size_t)(sx - xs) * nzw + (sz - zs)] = 1.f;
  for (int j = 0; j < nxw; j++) smooth_line_host(2, nzw, m.data(), (long long)j * nzw, 1, tmp);
  for (int j = 0; j < nzw; j++) smooth_line_host(2, nxw, m.data(), j, nzw, tmp);
  sg.nsrc = 0;
  sg.sx0 = sg.sz0 = 1 << 30;
  sg.sx1 = sg.sz1 = -1;
  for (int ix = 0; ix < nxw; ix++)
    for (int iz = 0; iz < nzw; iz++) {
      const float w = m[(size_t)ix * nzw + iz];
      if (w != 0.f) {
        PW_CHECK(sg.nsrc < MAXSRCW, PW_ERR_SHAPE, "source map has too many cells");
        const int gz = iz + zs, gx = ix + xs;
        PW_CHECK(gz >= 4 && gz < pnz - 4 && gx >= 4 && gx < pnx - 4, PW_ERR_SHAPE,
                 "source map reaches the zero border of the padded grid");
        sg.scell[sg.nsrc] = (gx << 16) | gz;
        sg.sw[sg.nsrc] = w;
        sg.nsrc++;
        sg.sx0 = std::min(sg.sx0, gx);
        sg.sx1 = std::max(sg.sx1, gx);
        sg.sz0 = std::min(sg.sz0, gz);
        sg.sz1 = std::max(sg.sz1, gz);
      }
    }
  return PW_OK;
}

// Exhaustive check of DivC against __fdiv_rn over the 2^23 significands of
// x in [scale, 2*scale) (a binade where every intermediate value is normal).
__device__ unsigned int fastdiv_bad;
__global__ void fastdiv_check_kernel(float d, float zh, float zl, float scale) {
  const unsigned int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= (1u << 23)) return;
  const float x = __fmul_rn(scale, __uint_as_float(0x3f800000u | m));  // exact (power of 2)
  const float q = __fmaf_rn(x, zh, __fmul_rn(x, zl));
  if (__float_as_uint(q) != __float_as_uint(__fdiv_rn(x, d))) atomicAdd(&fastdiv_bad, 1u);
}

// div_f64 against __fdiv_rn, both signs: for the 2^23 significands of x in
// [scale, 2 scale), where the quotient is a normal float (so for every x of
// such a quotient: no intermediate value of div_f64 leaves double's normal
// range, and scaling x by 2^k scales each step exactly), and for every x with
// bits up to `tiny`, which include all whose quotient is subnormal.
__global__ void __launch_bounds__(256) div_f64_check_kernel(DivC c, float scale, unsigned int tiny) {
  const unsigned int n = (1u << 23) + tiny, stride = gridDim.x * 256;
  unsigned int bad = 0;
  for (unsigned int i = blockIdx.x * 256 + threadIdx.x; i < n; i += stride) {
    const float x = i < (1u << 23) ? __fmul_rn(scale, __uint_as_float(0x3f800000u | i))
                                   : __uint_as_float(i - (1u << 23) + 1u);
    bad += __float_as_uint(div_f64(x, c.dd, c.rd)) != __float_as_uint(__fdiv_rn(x, c.d));
    bad += __float_as_uint(div_f64(-x, c.dd, c.rd)) != __float_as_uint(__fdiv_rn(-x, c.d));
  }
  if (bad) atomicAdd(&fastdiv_bad, bad);
}

// DivC for d (cached per process: the result depends on d only).
static int prepare_div(float d, DivC &c) {
  static std::mutex mu;
  static std::map<unsigned int, DivC> cache;
  unsigned int key;
  memcpy(&key, &d, 4);
  std::lock_guard<std::mutex> lock(mu);
  auto hit = cache.find(key);
  if (hit != cache.end()) {
    c = hit->second;
    return PW_OK;
  }
  c.d = d;
  c.dd = d;
  c.rd = 1.0 / (double)d;
  c.zh = c.zl = 0.f;
  c.xmin = 1.f;
  c.xmax = 0.f;
  c.f64 = d > 0.f && std::isfinite(d);
  if (c.f64) {
    // zh: the float nearest 1/d (float x float products are exact in double,
    // and 1 - zh*d is exact by Sterbenz's lemma)
    const float z0 = (float)(1.0 / (double)d);
    float zh = z0;
    double err = std::fabs(1.0 - (double)z0 * d);
    for (float cand : {std::nextafter(z0, 0.f), std::nextafter(z0, INFINITY)}) {
      const double e = std::fabs(1.0 - (double)cand * d);
      unsigned int cb;
      memcpy(&cb, &cand, 4);
      if (e < err || (e == err && (cb & 1u) == 0)) {
        zh = cand;
        err = e;
      }
    }
    const float zl = (float)((1.0 - (double)zh * d) / (double)d);
    // keep x*zh, x*zl and x/d normal and finite with a factor-4 margin
    const double fmin = (double)FLT_MIN, fmax = (double)FLT_MAX;
    double lo = std::max(fmin / zh, fmin * d);
    if (zl != 0.f) lo = std::max(lo, fmin / std::fabs((double)zl));
    lo *= 4;
    const double hi = std::min({fmax / 4 / zh, fmax / 4 * d, fmax});  // finite numerators only
    if (lo * 4 < hi) {
      const double scale = std::ldexp(1.0, (int)std::ceil(std::log2(lo)));
      unsigned int bad = 0;
      PW_CUDA(cudaMemcpyToSymbol(fastdiv_bad, &bad, sizeof bad));
      fastdiv_check_kernel<<<(1u << 23) / 256, 256>>>(d, zh, zl, (float)scale);
      PW_CUDA(cudaGetLastError());
      PW_CUDA(cudaMemcpyFromSymbol(&bad, fastdiv_bad, sizeof bad));
      if (bad == 0) {
        c.zh = zh;
        c.zl = zl;
        c.xmin = (float)lo;
        c.xmax = (float)hi;
      }
    }
    // quotients below FLT_MIN have numerators below FLT_MIN d (a margin of two)
    const float top = (float)std::min(2. * FLT_MIN * d + 2. * FLT_TRUE_MIN, (double)FLT_MAX);
    unsigned int tiny, bad = 0;
    memcpy(&tiny, &top, 4);
    const float scale = std::max(std::ldexp(1.f, (int)std::floor(std::log2((double)d))), FLT_MIN);
    PW_CUDA(cudaMemcpyToSymbol(fastdiv_bad, &bad, sizeof bad));
    div_f64_check_kernel<<<8 * 148, 256>>>(c, scale, tiny);
    PW_CUDA(cudaGetLastError());
    PW_CUDA(cudaMemcpyFromSymbol(&bad, fastdiv_bad, sizeof bad));
    c.f64 = bad == 0;
  }
  if (getenv("PW_PFWI_VERBOSE"))
    fprintf(stderr, "pfwi: division by %.9g: zh %.9g zl %.9g range [%.3g, %.3g], FP64 %d\n", d,
            c.zh, c.zl, c.xmin, c.xmax, c.f64);
  cache[key] = c;
  return PW_OK;
}

struct Setup {
  pw_fwi_args a;
  DivC divx, divz;
  int pnz, pnx, lz;
  long long fstride;  // floats per field (incl. halo)
  int nr, rz, drv, sz;
  std::vector<ShotGeo> geo;
  std::vector<float> bz, bx;
};

// passive: distributed sources (pfwi mode 4) -- no point source per shot
static int setup(const pw_fwi_args *a, Setup &S, bool passive = false) {
  PW_CHECK(a != nullptr, PW_ERR_VALUE, "null args");
  S.a = *a;
  PW_CHECK(a->nz >= 1 && a->nx >= 1 && a->nt >= 1 && a->ns >= 1 && a->nb >= 1, PW_ERR_SHAPE,
           "sizes must be positive (nz=%d nx=%d nt=%d ns=%d nb=%d)", a->nz, a->nx, a->nt, a->ns,
           a->nb);
  PW_CHECK(a->dx > 0 && a->dz > 0 && a->dt > 0, PW_ERR_VALUE, "spacings must be positive");
  const int nb = a->nb;
  S.pnz = a->nz + 2 * nb;
  S.pnx = a->nx + 2 * nb;
  PW_CHECK(S.pnx < 65536 && S.pnz < 65536, PW_ERR_SHAPE, "grid too large");
  S.lz = (int)round_up(HZ + round_up(S.pnz, 4) + 4, 32);
  PW_TRY(prepare_div(a->dx * a->dx, S.divx));
  PW_TRY(prepare_div(a->dz * a->dz, S.divz));
  S.fstride = (long long)S.lz * (S.pnx + 2 * HX) + 64;
  // preparation (wave_fwiutil.c:31-71) with pfwi.c's fixed acquisition
  std::vector<float> bc(nb);
  for (int i = 0; i < nb; i++) {
    float tmp = a->coef * (nb - i);
    bc[i] = expf(-tmp * tmp);
  }
  auto axis = [&](int n, std::vector<float> &f) {
    f.assign(n, 1.f);
    for (int i = 0; i < nb; i++) f[i] = bc[i];
    for (int i = n - nb; i < n; i++) f[i] = bc[n - i - 1];
  };
  axis(S.pnz, S.bz);
  axis(S.pnx, S.bx);
  S.bz.resize(round_up(S.pnz, 4), 1.f);  // read four at a time
  const float dx = a->dx;
  const int ds_v = (int)(a->ds / dx + 0.5);
  const int s0_v = (int)(a->os / dx + 0.5 + nb);
  S.sz = a->sz + nb;
  S.rz = a->rz + nb;
  S.nr = a->nx;
  const float dr = dx, r0 = a->ox, x0 = a->ox;
  S.drv = (int)(dr / dx + 0.5);
  PW_CHECK(S.drv >= 1, PW_ERR_SHAPE, "receiver interval below one cell");
  const float xend = x0 + (a->nx - 1) * dx;
  S.geo.assign(a->ns, ShotGeo{});
  for (int is = 0; is < a->ns; is++) {
    ShotGeo &g = S.geo[is];
    if (a->acqui_type == 1) {
      g.r0v = (int)((r0 - x0) / dx + 0.5 + nb);
      g.r02 = 0;
      g.nr2 = S.nr;
    } else {
      const float sx = a->os + a->ds * is;
      const float rbegin = (sx + r0 < x0) ? x0 : sx + r0;
      float rend = sx + r0 + (S.nr - 1) * dr;
      rend = (rend < xend) ? rend : xend;
      g.r0v = (int)(rbegin / dx + 0.5 + nb);
      g.r02 = (int)((rbegin - sx - r0) / dx + 0.5);
      g.nr2 = (int)((rend - rbegin) / dx + 1.5);
    }
    PW_CHECK(g.r02 >= 0 && g.r02 + g.nr2 <= S.nr && g.r0v >= 0 &&
                 g.r0v + (g.nr2 - 1) * S.drv < S.pnx,
             PW_ERR_SHAPE, "shot %d: receivers outside the grid", is);
    if (passive) {  // an empty source map
      g.nsrc = 0;
      g.sx0 = g.sz0 = 1;
      g.sx1 = g.sz1 = 0;
      continue;
    }
    const int sx = s0_v + is * ds_v;
    PW_CHECK(sx >= 0 && sx < S.pnx && S.sz >= 0 && S.sz < S.pnz, PW_ERR_SHAPE,
             "shot %d: source (x=%d, z=%d) outside the padded grid", is, sx, S.sz);
    PW_TRY(source_map(sx, S.sz, S.pnz, S.pnx, g));
  }
  PW_CHECK(S.rz >= 4 && S.rz < S.pnz - 4, PW_ERR_SHAPE, "receiver depth in the zero border");
  if (getenv("PW_PFWI_VERBOSE")) {
    // depth class of the padded grid: columns of up to 64 or 128 float4, and
    // how many such segments a column has.  The step kernel's lanes cross
    // columns and use neither; launch_one prints what it launches
    const int nz4 = ceil_div(S.pnz, 4), zw = nz4 <= 64 ? 64 : 128;
    fprintf(stderr, "pfwi plan: padded %d x %d, ZW=%d ztiles=%d\n", S.pnz, S.pnx, zw,
            ceil_div(nz4, zw));
  }
  return PW_OK;
}

template <int MODE, bool PAS = false>
static int launch_one(const Setup &S, PfArgs &p, int nshots, cudaStream_t st) {
  const long long lanes = (long long)p.nz4.d * ceil_div(S.pnx, PF_XW);
  const dim3 grid((unsigned)ceil_div(lanes, 32), (unsigned)nshots);
  auto fn = S.divx.f64 && S.divz.f64 ? pf_step_kernel<MODE, PAS, false>
                                     : pf_step_kernel<MODE, PAS, true>;
  if (p.prev == MODE) {
    PW_CUDA(launch_pdl(fn, grid, dim3(32 * PF_XW), 0, st, p));
  } else {
    if (getenv("PW_PFWI_VERBOSE"))
      fprintf(stderr, "pfwi step: mode=%d nz4=%d shots=%d grid=%ux%u threads=%d zig=%d\n", MODE,
              p.nz4.d, nshots, grid.x, grid.y, 32 * PF_XW, p.zig);
    fn<<<grid, 32 * PF_XW, 0, st>>>(p);
    PW_CUDA(cudaGetLastError());
  }
  p.prev = MODE;
  return PW_OK;
}

static int launch(const Setup &S, PfArgs &p, int mode, int nshots, cudaStream_t st) {
  p.zig = zigzag_pays((size_t)(2 * nshots + 1) * S.fstride * 4);
  if (mode == FWD)
    return p.dsrc ? launch_one<FWD, true>(S, p, nshots, st) : launch_one<FWD>(S, p, nshots, st);
  if (mode == ADJ_REF) return launch_one<ADJ_REF>(S, p, nshots, st);
  return launch_one<ADJ_EXACT>(S, p, nshots, st);
}

static void base_args(const Setup &S, PfArgs &p) {
  memset(&p, 0, sizeof p);
  p.prev = -1;
  p.pnz = S.pnz;
  p.pnx = S.pnx;
  p.lz = S.lz;
  p.nb = S.a.nb;
  p.nz = S.a.nz;
  p.nx = S.a.nx;
  const float c0 = -205. / 72, c1 = 8. / 5, c2 = -1. / 5, c3 = 8. / 315, c4 = -1. / 560;
  p.c0 = c0; p.c1 = c1; p.c2 = c2; p.c3 = c3; p.c4 = c4;
  p.one = 1.f;
  p.divx = S.divx;
  p.divz = S.divz;
  p.xlo = std::max(S.divx.xmin, S.divz.xmin);
  p.xhi = std::min(S.divx.xmax, S.divz.xmax);
  p.nt = S.a.nt;
  p.rz = S.rz;
  p.drv = S.drv;
  p.nr = S.nr;
  p.fstep = S.fstride;
  p.nz4 = make_fast_div(ceil_div(S.pnz, 4));
  p.src_z0 = 1 << 30;
  p.src_z1 = -1;
  for (const ShotGeo &g : S.geo) {
    p.src_z0 = std::min(p.src_z0, g.sz0);
    p.src_z1 = std::max(p.src_z1, g.sz1);
  }
}

}  // namespace pf
}  // namespace pw

using namespace pw;
using namespace pw::pf;

extern "C" int pw_fwi_args_from_pararray(const float *p, int n, pw_fwi_args *o) {
  PW_CHECK(p && o && n >= 20, PW_ERR_VALUE, "pararray needs 20 values");
  memset(o, 0, sizeof *o);
  o->nz = (int)p[0]; o->nx = (int)p[1]; o->dz = p[2]; o->dx = p[3]; o->oz = p[4]; o->ox = p[5];
  o->nt = (int)p[6]; o->dt = p[7]; o->ot = p[8]; o->ns = (int)p[10]; o->ds = p[11];
  o->os = p[12]; o->nb = (int)p[14]; o->coef = p[15]; o->f0 = p[16];
  o->acqui_type = (int)p[17]; o->interval = (int)p[18]; o->niter = (int)p[19];
  o->sz = 5; o->rz = 1;  // pfwi.c:796-800
  return PW_OK;
}

// --------------------------------------------------------------- drivers --
namespace pw {
namespace pf {

// residual_weighting with oreo=false as fwic sets it up (wave_fwiutil.c:225-296,
// pfwi.c:849-855): 1 inside, 10-sample sine tapers on both axes.  [nr][nt].
// residual_weighting (wave_fwiutil.c:225-296), both branches; w [nr][nt].
// Taper samples that would fall outside the array (a window closer than 10
// samples to its edge, where the reference writes out of bounds) are skipped.
static void weights_window(int nt, int nr, int wtn1, int wtn2, int woffn1, int woffn2, bool oreo,
                           float *w) {
  float sn[10];
  for (int i = 0; i < 10; i++) sn[i] = sinf(0.5 * M_PI * (i + 1) / 11.);
  float sink = 0.f;
  auto W = [&](int ir, int it) -> float & {
    return (ir >= 0 && ir < nr && it >= 0 && it < nt) ? w[(size_t)ir * nt + it] : sink;
  };
  if (oreo) {
    for (size_t i = 0; i < (size_t)nr * nt; i++) w[i] = 1.f;
    for (int ir = woffn1; ir <= woffn2; ir++)
      for (int it = wtn1; it <= wtn2; it++) W(ir, it) = 0.f;
    for (int ir = 0; ir < 10; ir++)
      for (int it = wtn1; it <= wtn2; it++) {
        if (woffn1 - ir > 0) W(woffn1 - ir, it) *= sn[ir];
        if (woffn2 + ir < nr) W(woffn2 + ir, it) *= sn[ir];
      }
    for (int it = 0; it < 10; it++) {
      for (int ir = 0; ir < woffn1; ir++) {
        W(ir, wtn1 + it) *= sn[it];
        W(ir, wtn2 - it) *= sn[it];
      }
      for (int ir = woffn2 + 1; ir < nr; ir++) {
        W(ir, wtn1 + it) *= sn[it];
        W(ir, wtn2 - it) *= sn[it];
      }
    }
    return;
  }
  for (size_t i = 0; i < (size_t)nr * nt; i++) w[i] = 0.f;
  for (int ir = woffn1; ir <= woffn2; ir++)
    for (int it = wtn1; it <= wtn2; it++) W(ir, it) = 1.f;
  for (int ir = 0; ir < 10; ir++)
    for (int it = wtn1; it <= wtn2; it++) {
      W(woffn1 + ir, it) *= sn[ir];
      W(woffn2 - ir, it) *= sn[ir];
    }
  for (int it = 0; it < 10; it++)
    for (int ir = woffn1; ir <= woffn2; ir++) {
      W(ir, wtn1 + it) *= sn[it];
      W(ir, wtn2 - it) *= sn[it];
    }
}

static void residual_weights(const pw_fwi_args &a, int nr, std::vector<float> &w) {
  const int nt = a.nt;
  const float t0 = a.ot, dt = a.dt, r0 = a.ox, dr = a.dx;
  const float wt1 = t0, wt2 = t0 + (nt - 1) * dt;
  const float woff1 = r0, woff2 = r0 + (nr - 1) * dr;
  const int wtn1 = (int)((wt1 - t0) / dt + 0.5), wtn2 = (int)((wt2 - t0) / dt + 0.5);
  const int woffn1 = (int)((woff1 - r0) / dr + 0.5), woffn2 = (int)((woff2 - r0) / dr + 0.5);
  w.assign((size_t)nr * nt, 0.f);
  weights_window(nt, nr, wtn1, wtn2, woffn1, woffn2, false, w.data());
}

struct Fields {
  float *V = nullptr;
  float *A = nullptr, *B = nullptr;  // [nshots][fstride] each
  ShotGeo *geo = nullptr;
  float *bz = nullptr, *bx = nullptr, *wav = nullptr;
};

// Common device state of a call: V, the two wavefield sets, geometry.
static int bind_common(const Setup &S, int nsb, Carve &cv, size_t &o_V, size_t &o_A, size_t &o_B,
                       size_t &o_geo, size_t &o_bz, size_t &o_bx, size_t &o_wav) {
  o_V = cv.add(S.fstride * 4);
  o_A = cv.add((size_t)nsb * S.fstride * 4);
  o_B = cv.add((size_t)nsb * S.fstride * 4);
  o_geo = cv.add(sizeof(ShotGeo) * S.a.ns);
  o_bz = cv.add(S.bz.size() * 4);
  o_bx = cv.add(S.bx.size() * 4);
  o_wav = cv.add((size_t)S.a.nt * 4);
  return PW_OK;
}

static int upload_common(const Setup &S, char *base, size_t o_geo, size_t o_bz, size_t o_bx,
                         size_t o_wav, const float *wav, bool host, cudaStream_t st) {
  PW_CUDA(cudaMemcpyAsync(base + o_geo, S.geo.data(), sizeof(ShotGeo) * S.a.ns,
                          cudaMemcpyHostToDevice, st));
  PW_CUDA(cudaMemcpyAsync(base + o_bz, S.bz.data(), S.bz.size() * 4, cudaMemcpyHostToDevice, st));
  PW_CUDA(cudaMemcpyAsync(base + o_bx, S.bx.data(), S.bx.size() * 4, cudaMemcpyHostToDevice, st));
  if (wav) PW_TRY(to_device(base + o_wav, wav, (size_t)S.a.nt * 4, host, st));
  return PW_OK;
}

static int check_vel_cfl(const Setup &S, const float *vel_dev, size_t n, cudaStream_t st,
                         unsigned *scratch) {
  // largest velocity (CFL) and a flag for non-finite / non-positive values
  PW_CUDA(cudaMemsetAsync(scratch, 0, 8, st));
  vel_check_kernel<<<296, 256, 0, st>>>(vel_dev, (long long)n, scratch);
  PW_CUDA(cudaGetLastError());
  unsigned hv[2] = {0, 0};
  PW_CUDA(cudaMemcpyAsync(hv, scratch, 8, cudaMemcpyDeviceToHost, st));
  PW_CUDA(cudaStreamSynchronize(st));
  float vmax;
  memcpy(&vmax, &hv[0], 4);
  PW_CHECK(hv[1] == 0 && vmax > 0.f, PW_ERR_VALUE, "velocity has non-finite or non-positive values");
  if (S.a.flags & PW_NO_CFL_CHECK) return PW_OK;
  // 8th-order leapfrog in 2-D: v dt / h <= 0.555 (measured limit)
  const float hmin = std::min(S.a.dx, S.a.dz);
  const float cfl = vmax * S.a.dt / hmin;
  PW_CHECK(cfl <= 0.555f, PW_ERR_CFL, "unstable: vmax*dt/h = %g exceeds 0.555", cfl);
  return PW_OK;
}

}  // namespace pf
}  // namespace pw

extern "C" int pw_pfwi_forward(const pw_fwi_args *a, const float *vel, const float *wav,
                               float *data, void *stream) {
  cudaStream_t st = (cudaStream_t)stream;
  Setup S;
  PW_TRY(setup(a, S));
  const bool host = (a->flags & PW_HOST_PTRS) != 0;
  const int ns = a->ns, nt = a->nt, nr = S.nr;
  const int nsb = std::min(ns, MAXS);
  const size_t nvel = (size_t)a->nz * a->nx;
  Carve cv;
  size_t o_V, o_A, o_B, o_geo, o_bz, o_bx, o_wav;
  bind_common(S, nsb, cv, o_V, o_A, o_B, o_geo, o_bz, o_bx, o_wav);
  const size_t o_vel = cv.add(host ? nvel * 4 : 0);
  const size_t o_rec = cv.add((size_t)ns * nt * nr * 4);
  const size_t o_out = cv.add(host ? (size_t)ns * nt * nr * 4 : 0);
  const size_t o_mx = cv.add(16);
  Workspace &ws = Workspace::for_current_device();
  std::lock_guard<std::mutex> lock(ws.mutex());
  PW_TRY(ws.reserve(cv.total()));
  char *base = ws.base();
  PW_CUDA(cudaMemsetAsync(base, 0, cv.total(), st));
  const float *d_vel = vel;
  if (host) {
    PW_TRY(to_device(base + o_vel, vel, nvel * 4, true, st));
    d_vel = at<float>(base, o_vel);
  }
  PW_TRY(check_vel_cfl(S, d_vel, nvel, st, at<unsigned>(base, o_mx)));
  PW_TRY(upload_common(S, base, o_geo, o_bz, o_bx, o_wav, wav, host, st));
  float *V = at<float>(base, o_V);
  pad_V_kernel<<<1184, 256, 0, st>>>(d_vel, a->nz, a->nx, a->nb, S.pnz, S.pnx, S.lz, a->dt * a->dt, V);
  PW_CUDA(cudaGetLastError());
  float *rec = at<float>(base, o_rec);
  PfArgs p;
  base_args(S, p);
  p.V = V;
  p.bz = at<float>(base, o_bz);
  p.bx = at<float>(base, o_bx);
  p.wav = at<float>(base, o_wav);
  LoopTimer timer(st);
  timer.start();
  long long launches = 0;
  for (int s0 = 0; s0 < ns; s0 += nsb) {
    const int nb_ = std::min(nsb, ns - s0);
    float *A = at<float>(base, o_A), *B = at<float>(base, o_B);
    PW_CUDA(cudaMemsetAsync(A, 0, (size_t)nsb * S.fstride * 4, st));
    PW_CUDA(cudaMemsetAsync(B, 0, (size_t)nsb * S.fstride * 4, st));
    p.geo = at<ShotGeo>(base, o_geo) + s0;
    p.rec = rec + (size_t)s0 * nt * nr;
    for (int it = 0; it < nt; it++) {
      p.it = it;
      p.cur = A;
      p.nxt = B;
      PW_TRY(launch(S, p, FWD, nb_, st));
      launches++;
      std::swap(A, B);
    }
  }
  timer.stop();
  // [shot][nt][nr] -> [shot][nr][nt]
  float *dst = host ? at<float>(base, o_out) : data;
  for (int s = 0; s < ns; s++) {
    dim3 tb(32, 8), tg(ceil_div(nr, 32), ceil_div(nt, 32));
    transpose_kernel<<<tg, tb, 0, st>>>(rec + (size_t)s * nt * nr, dst + (size_t)s * nt * nr, nt, nr);
  }
  PW_CUDA(cudaGetLastError());
  if (host) PW_TRY(to_host(data, dst, (size_t)ns * nt * nr * 4, true, st));
  PW_CUDA(cudaStreamSynchronize(st));
  timer.finish(launches, launches + 3 + ns);
  return PW_OK;
}

// Checkpoint plan of the exact gradient under an HBM budget.  The working
// set of a batch of nsb shots is, in field-sized buffers per shot: the two
// wavefield pairs, the gradient slice and traces (about 5), the checkpoints
// (two fields every k steps) and the segment buffer of k forward terms.  The
// forward pass keeps the terms of the last segment, so the backward pass
// recomputes the (nck - 1) k steps before it: the recompute factor (forward
// steps run / nt) is 1 + (nck - 1) k / nt.  Once the shots of a batch fill
// the GPU a step costs in proportion to its shots, so the planner picks,
// over batch sizes nsb = ns, ns/2, ..., 1 (every batch sums its shots' slices
// into the gradient in shot order, so the result does not depend on nsb),
// the largest k that fits the budget, and among those the plan with the
// least recompute, then the largest batch.  k = nt stores every term and
// recomputes nothing; a fixed ckpt_k > 0 keeps k and only shrinks the batch
// if needed.
struct ExactPlan {
  int k = 0, nsb = 0;
  double recompute = 1.0;
  size_t bytes = 0;
};

static ExactPlan plan_exact(const Setup &S, int ckpt_k, size_t held) {
  const int nt = S.a.nt;
  size_t freeb = 0, totb = 0;
  if (cudaMemGetInfo(&freeb, &totb) != cudaSuccess) {
    cudaGetLastError();
    freeb = totb = (size_t)32 << 30;
  }
  // budget: the caller's, or a quarter of the device; never more than 80% of
  // what is free plus the workspace this call reuses
  double budget = S.a.hbm_budget > 0 ? (double)S.a.hbm_budget : 0.25 * (double)totb;
  budget = std::min(budget, 0.8 * (double)(freeb + held));
  const double fb = (double)S.fstride * 4;
  auto need = [&](int kk, int nb) {
    const int nck = (nt + kk - 1) / kk;
    return fb * nb * (5.0 + 2.0 * nck + kk) + fb * 2;
  };
  auto recompute = [&](int kk) {
    const int nck = (nt + kk - 1) / kk;
    return 1.0 + (double)(nck - 1) * kk / nt;
  };
  const int kmin = std::min(nt, std::max(1, (int)std::lround(std::sqrt(2.0 * nt))));
  const int nsb_max = std::min(S.a.ns, MAXS);
  ExactPlan best;
  for (int nb = nsb_max; nb >= 1; nb = (nb + 1) / 2) {
    int k;
    if (ckpt_k > 0) {
      k = std::min(ckpt_k, nt);
      if (need(k, nb) > budget && nb > 1) continue;
    } else if (need(nt, nb) <= budget) {
      k = nt;
    } else if (need(kmin, nb) <= budget) {
      // need() rises with k above kmin: the largest k in [kmin, nt) that fits
      int lo = kmin, hi = nt;
      while (hi - lo > 1) {
        const int mid = lo + (hi - lo) / 2;
        if (need(mid, nb) <= budget) lo = mid;
        else hi = mid;
      }
      k = lo;
    } else {
      k = 0;
    }
    if (k > 0) {
      const double rc = recompute(k);
      if (best.k == 0 || rc < best.recompute - 1e-12) {
        best.k = k;
        best.nsb = nb;
        best.recompute = rc;
        best.bytes = (size_t)need(k, nb);
      }
      if (ckpt_k > 0 || rc == 1.0) break;  // nothing better below
    }
    if (nb == 1) break;
  }
  if (best.k == 0) {
    // nothing fits the budget: the smallest working set (one shot, k =
    // sqrt(2 nt)); the allocation reports if even that fails
    best.nsb = 1;
    best.k = ckpt_k > 0 ? std::min(ckpt_k, nt) : kmin;
    best.recompute = recompute(best.k);
    best.bytes = (size_t)need(best.k, best.nsb);
  }
  return best;
}

// Per-thread record of the last exact gradient's checkpoint plan.
struct PlanRecord {
  int k = 0, nsb = 0;
  long long bytes = 0;
  double recompute = 0.0;
};
static PlanRecord &plan_record() {
  static thread_local PlanRecord r;
  return r;
}

namespace pw {
namespace pf {
// The gradient of pw_pfwi_gradient (wav: point sources) and of
// pw_pfwi_gradient_passive (dsrc: a source field per shot, [ns][nt][nx][nz]).
static int gradient_impl(const pw_fwi_args *a, int mode, const float *vel, const float *wav,
                         const float *dsrc, const float *dobs, const float *weight, float *grad,
                         double *misfit, int ckpt_k, void *stream) {
  cudaStream_t st = (cudaStream_t)stream;
  PW_CHECK(mode == PW_GRAD_REFERENCE || mode == PW_GRAD_EXACT, PW_ERR_VALUE, "bad gradient mode");
  PW_CHECK(vel && dobs && grad && (wav || dsrc), PW_ERR_VALUE, "null array");
  Setup S;
  PW_TRY(setup(a, S, dsrc != nullptr));
  const bool host = (a->flags & PW_HOST_PTRS) != 0;
  const bool per_shot = (a->flags & PW_PER_SHOT) != 0;
  const int ns = a->ns, nt = a->nt, nr = S.nr, nz = a->nz, nx = a->nx;
  const size_t nvel = (size_t)nz * nx;
  const bool exact = mode == PW_GRAD_EXACT;
  const int interval = std::max(1, a->interval);
  const int wnt = (nt - 1) / interval + 1;
  Workspace &ws = Workspace::for_current_device();
  std::lock_guard<std::mutex> lock(ws.mutex());
  int k = 0, nsb = per_shot ? 1 : std::min(ns, MAXS);
  if (exact) {
    const ExactPlan ep = plan_exact(S, ckpt_k, ws.capacity());
    k = ep.k;
    nsb = per_shot ? 1 : ep.nsb;
    plan_record().k = k;
    plan_record().nsb = nsb;
    plan_record().recompute = ep.recompute;
  }
  const int nck = exact ? (nt + k - 1) / k : 0;
  std::vector<float> wts;
  if (weight == nullptr) residual_weights(*a, nr, wts);
  // multiscale residual filter (gradient_pas_init, wave_fwigradient.c:657-658:
  // soupar's cutoffs times dt, compared in double)
  const float flo_dt = a->flo * a->dt, fhi_dt = a->fhi * a->dt;
  const bool use_lo = flo_dt > 0.0001, use_hi = a->fhi > 0.f && fhi_dt < 0.5 - 0.0001;
  PW_CHECK(!(exact && (use_lo || use_hi)), PW_ERR_VALUE,
           "the multiscale residual filter applies to the reference-mode gradient only");
  const ButterCoef blo = use_lo ? butter_coef(false, flo_dt, 3) : ButterCoef{};
  const ButterCoef bhi = use_hi ? butter_coef(true, fhi_dt, 3) : ButterCoef{};

  Carve cv;
  size_t o_V, o_A, o_B, o_geo, o_bz, o_bx, o_wav;
  bind_common(S, nsb, cv, o_V, o_A, o_B, o_geo, o_bz, o_bx, o_wav);
  const size_t o_vel = cv.add(host ? nvel * 4 : 0);
  const size_t o_w = cv.add((size_t)nr * nt * 4);
  const size_t o_dobs = cv.add((size_t)ns * nt * nr * 4);    // [shot][nt][nr]
  const size_t o_dobs_in = cv.add(host ? (size_t)ns * nt * nr * 4 : 0);
  const size_t o_d = cv.add((size_t)nsb * nt * nr * 4);      // recorded [shot][nt][nr]
  const size_t o_res = cv.add((size_t)nsb * nt * nr * 4);
  const size_t o_snap = cv.add(exact ? 0 : (size_t)nsb * wnt * nvel * 4);
  const size_t o_ck = cv.add(exact ? (size_t)nsb * nck * 2 * S.fstride * 4 : 0);
  const size_t o_tb = cv.add(exact ? (size_t)nsb * k * S.fstride * 4 : 0);
  const size_t o_ga = cv.add(exact ? (size_t)S.fstride * 4 : 0);
  // shots of one launch run in different CTAs: each accumulates its gradient
  // in its own slice, summed into the total in shot order after the batch
  const size_t gslice = exact ? (size_t)S.fstride : nvel;
  // exact mode: always through the slices (one shot per batch too), so the
  // shots are summed in the same order whatever the batch size
  const bool sliced = exact || nsb > 1;
  const size_t o_gs = cv.add(sliced ? (size_t)nsb * gslice * 4 : 0);
  const size_t o_grad = cv.add(nvel * 4);
  const size_t o_m2v3 = cv.add(exact ? 0 : nvel * 4);
  const size_t o_mis = cv.add(8 * (1 + RESID_BLOCKS));
  const size_t o_mx = cv.add(16);
  const size_t nsrcf = (size_t)nvel * nt;  // one shot's source field
  const size_t o_dsrc = cv.add(dsrc && host ? (size_t)ns * nsrcf * 4 : 0);
  PW_TRY(ws.reserve(cv.total()));
  if (exact) plan_record().bytes = (long long)cv.total();
  char *base = ws.base();
  // snapshots, checkpoints and segment terms are written before they are
  // read: zero the rest only (the term buffer alone is tens of GB)
  PW_CUDA(cudaMemsetAsync(base, 0, o_snap, st));
  PW_CUDA(cudaMemsetAsync(base + o_ga, 0, cv.total() - o_ga, st));
  const float *d_vel = vel;
  if (host) {
    PW_TRY(to_device(base + o_vel, vel, nvel * 4, true, st));
    d_vel = at<float>(base, o_vel);
  }
  PW_TRY(check_vel_cfl(S, d_vel, nvel, st, at<unsigned>(base, o_mx)));
  PW_TRY(upload_common(S, base, o_geo, o_bz, o_bx, o_wav, wav, host, st));
  const float *d_dsrc = dsrc;
  if (dsrc && host) {
    PW_TRY(to_device(base + o_dsrc, dsrc, (size_t)ns * nsrcf * 4, true, st));
    d_dsrc = at<float>(base, o_dsrc);
  }
  if (weight) PW_TRY(to_device(base + o_w, weight, (size_t)nr * nt * 4, host, st));
  else PW_CUDA(cudaMemcpyAsync(base + o_w, wts.data(), wts.size() * 4, cudaMemcpyHostToDevice, st));
  {
    // dobs [shot][nr][nt] -> [shot][nt][nr]
    const float *src = dobs;
    if (host) {
      PW_TRY(to_device(base + o_dobs_in, dobs, (size_t)ns * nt * nr * 4, true, st));
      src = at<float>(base, o_dobs_in);
    }
    for (int s = 0; s < ns; s++) {
      dim3 tb(32, 8), tg(ceil_div(nt, 32), ceil_div(nr, 32));
      transpose_kernel<<<tg, tb, 0, st>>>(src + (size_t)s * nr * nt,
                                          at<float>(base, o_dobs) + (size_t)s * nt * nr, nr, nt);
    }
    PW_CUDA(cudaGetLastError());
  }
  float *V = at<float>(base, o_V);
  pad_V_kernel<<<1184, 256, 0, st>>>(d_vel, nz, nx, a->nb, S.pnz, S.pnx, S.lz, a->dt * a->dt, V);
  PW_CUDA(cudaGetLastError());
  float *gdev = at<float>(base, o_grad);
  float *gacc = at<float>(base, o_ga);
  double *dmis = at<double>(base, o_mis);
  PfArgs p;
  base_args(S, p);
  p.V = V;
  p.bz = at<float>(base, o_bz);
  p.bx = at<float>(base, o_bx);
  p.wav = at<float>(base, o_wav);
  if (!exact) {
    m2v3_kernel<<<592, 256, 0, st>>>(d_vel, nvel, at<float>(base, o_m2v3));
    PW_CUDA(cudaGetLastError());
    p.m2v3 = at<float>(base, o_m2v3);
  }
  p.wdt2 = (a->dt * interval) * (a->dt * interval);
  float *gtotal = exact ? gacc : gdev;
  float *gslices = at<float>(base, o_gs);
  p.grad = sliced ? gslices : gtotal;
  p.gstride = sliced ? (long long)gslice : 0;
  const size_t fs = (size_t)S.fstride;
  long long launches = 0;
  LoopTimer timer(st);
  timer.start();
  for (int s0 = 0; s0 < ns; s0 += nsb) {
    const int nb_ = std::min(nsb, ns - s0);
    // the shots' wavefield pairs, `stride` floats apart; a step swaps the pair
    float *A, *B;
    auto reset = [&]() -> int {
      A = at<float>(base, o_A);
      B = at<float>(base, o_B);
      PW_CUDA(cudaMemsetAsync(A, 0, (size_t)nsb * fs * 4, st));
      PW_CUDA(cudaMemsetAsync(B, 0, (size_t)nsb * fs * 4, st));
      return PW_OK;
    };
    auto step = [&](int mode_, int it, float *&cur, float *&nxt, size_t stride) -> int {
      p.it = it;
      p.cur = cur;
      p.nxt = nxt;
      p.fstep = (long long)stride;
      PW_TRY(launch(S, p, mode_, nb_, st));
      launches++;
      std::swap(cur, nxt);
      return PW_OK;
    };
    p.geo = at<ShotGeo>(base, o_geo) + s0;
    p.dsrc = d_dsrc ? d_dsrc + (size_t)s0 * nsrcf : nullptr;
    p.dsrc_stride = (long long)nsrcf;
    float *dd = at<float>(base, o_d);
    float *res = at<float>(base, o_res);
    float *ck = at<float>(base, o_ck);
    float *tb = at<float>(base, o_tb);
    float *snap = at<float>(base, o_snap);
    // ---- forward: traces, and snapshots (reference) or checkpoints (exact)
    PW_TRY(reset());
    p.rec = dd;
    p.tout = nullptr;
    p.snap_stride = (long long)wnt * nvel;
    const int n_last = exact ? (nck - 1) * k : nt;  // first step of the last segment
    p.tout_stride = (long long)k * fs;
    for (int it = 0; it < nt; it++) {
      if (exact && it % k == 0 && it < n_last) {
        const int m = it / k;
        for (int s = 0; s < nb_; s++) {
          float *c = ck + ((size_t)s * nck + m) * 2 * fs;
          PW_CUDA(cudaMemcpyAsync(c, A + s * fs, fs * 4, cudaMemcpyDeviceToDevice, st));
          PW_CUDA(cudaMemcpyAsync(c + fs, B + s * fs, fs * 4, cudaMemcpyDeviceToDevice, st));
        }
      }
      p.snap = (!exact && it % interval == 0) ? snap + (size_t)(it / interval) * nvel : nullptr;
      // the last segment's terms, which the backward pass reads first
      p.tout = it >= n_last ? tb + (size_t)(it - n_last) * fs : nullptr;
      PW_TRY(step(FWD, it, A, B, fs));
    }
    p.rec = nullptr;
    p.snap = nullptr;
    p.tout = nullptr;
    // ---- residual and FP64 misfit
    const bool filt = use_lo || use_hi;  // weights applied after the filter
    residual_kernel<<<RESID_BLOCKS, 256, 0, st>>>(dd, at<float>(base, o_dobs) + (size_t)s0 * nt * nr,
                                                  filt ? nullptr : at<float>(base, o_w), res, nb_,
                                                  nt, nr, exact ? 1 : 0, dmis);
    misfit_sum_kernel<<<1, 32, 0, st>>>(dmis, RESID_BLOCKS);
    PW_CUDA(cudaGetLastError());
    if (filt) {
      butter_residual_kernel<<<ceil_div((long long)nb_ * nr, 128), 128, 0, st>>>(
          blo, bhi, use_lo, use_hi, res, nb_, nt, nr, at<float>(base, o_w));
      PW_CUDA(cudaGetLastError());
    }
    p.res = res;
    if (!exact) {
      // ---- backward with gradient_av's imaging (wave_fwigradient.c:201-241)
      PW_TRY(reset());
      p.wstride = (long long)wnt * nvel;
      for (int it = nt - 1; it >= 0; it--) {
        const int wit = it / interval;
        p.imaging = (it % interval == 0) && wit != wnt - 1 && wit != 0;
        if (p.imaging) {
          p.wprev = snap + (size_t)(wit - 1) * nvel;
          p.wcur = snap + (size_t)wit * nvel;
          p.wnext = snap + (size_t)(wit + 1) * nvel;
        }
        PW_TRY(step(ADJ_REF, it, A, B, fs));
      }
    } else {
      // ---- backward by segments: recompute the forward terms of the segment
      // from its checkpoint, run the exact adjoint over it
      PW_TRY(reset());  // the adjoint reuses the forward pair
      p.tout_stride = (long long)k * fs;
      p.tin_stride = (long long)k * fs;
      for (int m = nck - 1; m >= 0; m--) {
        const int n0 = m * k, n1 = std::min(nt, n0 + k);
        // the forward pair lives in checkpoint m (overwritten, no longer needed)
        float *FA = ck + (size_t)m * 2 * fs, *FB = FA + fs;
        for (int n = n0; n < n1 && m < nck - 1; n++) {  // the last segment is kept
          p.tout = tb + (size_t)(n - n0) * fs;
          PW_TRY(step(FWD, n, FA, FB, (size_t)nck * 2 * fs));
        }
        p.tout = nullptr;
        for (int n = n1 - 1; n >= n0; n--) {
          p.tin = tb + (size_t)(n - n0) * fs;
          PW_TRY(step(ADJ_EXACT, n, A, B, fs));
        }
      }
      p.tin = nullptr;
    }
    if (sliced) {
      sum_slices_kernel<<<592, 256, 0, st>>>(gslices, nb_, (long long)gslice, gtotal);
      PW_CUDA(cudaGetLastError());
      PW_CUDA(cudaMemsetAsync(gslices, 0, (size_t)nb_ * gslice * 4, st));
      launches++;
    }
  }
  timer.stop();
  if (exact) {
    fold_grad_kernel<<<4 + 592, 256, 0, st>>>(gacc, d_vel, nz, nx, a->nb, S.pnz, S.pnx, S.lz, gdev);
    PW_CUDA(cudaGetLastError());
  }
  PW_TRY(to_host(grad, gdev, nvel * 4, host, st));
  if (misfit) PW_CUDA(cudaMemcpyAsync(misfit, dmis, 8, cudaMemcpyDeviceToHost, st));
  PW_CUDA(cudaStreamSynchronize(st));
  timer.finish(launches, launches + 8);
  return PW_OK;
}
}  // namespace pf
}  // namespace pw

extern "C" int pw_butter_apply(int n, int ntr, int low, float cutoff, int npoles, float *x,
                               int flags, void *stream) {
  PW_CHECK(x && n >= 0 && ntr >= 0, PW_ERR_VALUE, "bad arguments");
  PW_CHECK(npoles >= 1 && npoles <= BUTTER_MAXP, PW_ERR_VALUE, "npoles must be 1..%d", BUTTER_MAXP);
  if (n == 0 || ntr == 0) return PW_OK;
  cudaStream_t st = (cudaStream_t)stream;
  const bool host = (flags & PW_HOST_PTRS) != 0;
  const ButterCoef b = butter_coef(low != 0, cutoff, npoles);
  const size_t bytes = (size_t)n * ntr * 4;
  Workspace &ws = Workspace::for_current_device();
  std::lock_guard<std::mutex> lock(ws.mutex());
  float *d = x;
  if (host) {
    PW_TRY(ws.reserve(bytes));
    d = reinterpret_cast<float *>(ws.base());
    PW_TRY(to_device(d, x, bytes, true, st));
  }
  butter_traces_kernel<<<ceil_div(ntr, 128), 128, 0, st>>>(b, d, n, ntr);
  PW_CUDA(cudaGetLastError());
  if (host) PW_TRY(to_host(x, d, bytes, true, st));
  PW_CUDA(cudaStreamSynchronize(st));
  return PW_OK;
}

extern "C" int pw_residual_weights(int nt, int nr, int wtn1, int wtn2, int woffn1, int woffn2,
                                   int oreo, float *w) {
  PW_CHECK(w && nt >= 1 && nr >= 1, PW_ERR_VALUE, "bad arguments");
  PW_CHECK(0 <= wtn1 && wtn1 <= wtn2 && wtn2 < nt && 0 <= woffn1 && woffn1 <= woffn2 &&
               woffn2 < nr,
           PW_ERR_SHAPE, "window [%d,%d] x [%d,%d] must lie in %d x %d", woffn1, woffn2, wtn1,
           wtn2, nr, nt);
  weights_window(nt, nr, wtn1, wtn2, woffn1, woffn2, oreo != 0, w);
  return PW_OK;
}

extern "C" int pw_pfwi_gradient(const pw_fwi_args *a, int mode, const float *vel, const float *wav,
                                const float *dobs, const float *weight, float *grad,
                                double *misfit, int ckpt_k, void *stream) {
  PW_CHECK(wav != nullptr, PW_ERR_VALUE, "null wavelet");
  return gradient_impl(a, mode, vel, wav, nullptr, dobs, weight, grad, misfit, ckpt_k, stream);
}

extern "C" int pw_pfwi_gradient_passive(const pw_fwi_args *a, int mode, const float *vel,
                                        const float *src, const float *dobs, const float *weight,
                                        float *grad, double *misfit, int ckpt_k, void *stream) {
  PW_CHECK(src != nullptr, PW_ERR_VALUE, "null source field");
  return gradient_impl(a, mode, vel, nullptr, src, dobs, weight, grad, misfit, ckpt_k, stream);
}

// ------------------------------------------------------- visco-acoustic --
// forward_modeling (wave_fwimodeling.c:116-220) and gradient_v
// (wave_fwigradient.c:264-452): the pfwi scheme with a memory variable r,
//   r2 = (tau/taus*L + (idt - 0.5/taus)*r1) / (idt + 0.5/taus),
//   term = L*(1 + tau) - (r2 + r1)*0.5 + rr*w,  p2 = 2 p1 - p0 + V term,
// sponge on p0, p1 and r1; the adjoint pass forms r2 and tmp = p1*(1 + tau)
// - 0.5*(r2 + r1) from p1, r1 and takes the Laplacian of tmp.  The
// reference mixes float and double in these expressions; each operation is
// written with the matching explicitly rounded intrinsic.  Fields use a plain
// [pnx][pnz] layout; one thread per padded cell, Laplacian loads through L2.
// Only the cells [4, pad-4) change: the reference's forward_modeling also
// updates the 4-cell rim, where everything stays zero as long as no source
// cell lies there (the drivers check that).  As in the acoustic scheme, a
// field whose sponged value the step reads is stored before its last sponge
// (B for p0, R for r1), so p and r need no third buffer.
namespace pw {
namespace pf {

struct ViscoArgs {
  int pnz, pnx, nb, nz, nx;
  float c0, c1, c2, c3, c4, dx2, dz2, idt;
  const float *V, *tau, *taus, *bz, *bx;
  const float *A;        // p1 (sponged)
  float *B;              // in: p0 before its second sponge; out: the new p1
  float *R;              // in: r1 before its sponge; out: r2
  const float *rr;       // forward: dense source maps [shot][pnx][pnz]
  const float *wav;
  int it, nt;
  const ShotGeo *geo;
  int rz, drv, nr;
  float *rec;            // forward: traces [shot][nt][nr] or null
  float *snap;           // forward: interior snapshot of this step [nx][nz] or null
  long long fstride;     // floats per field (per shot)
  // adjoint
  const float *T;        // tmp field
  const float *res;      // residual [nt][nr] of the shot
  int imaging;
  const float *wprev, *wcur, *wnext, *m2v3;
  float wdt2;
  float *grad;
};

__device__ __forceinline__ float visco_lap(const ViscoArgs &a, const float *p, long long j) {
  const long long s = a.pnz;
  float tx = fmul(a.c0, p[j]);
  tx = fadd(tx, fmul(a.c1, fadd(p[j + s], p[j - s])));
  tx = fadd(tx, fmul(a.c2, fadd(p[j + 2 * s], p[j - 2 * s])));
  tx = fadd(tx, fmul(a.c3, fadd(p[j + 3 * s], p[j - 3 * s])));
  tx = fadd(tx, fmul(a.c4, fadd(p[j + 4 * s], p[j - 4 * s])));
  float tz = fmul(a.c0, p[j]);
  tz = fadd(tz, fmul(a.c1, fadd(p[j + 1], p[j - 1])));
  tz = fadd(tz, fmul(a.c2, fadd(p[j + 2], p[j - 2])));
  tz = fadd(tz, fmul(a.c3, fadd(p[j + 3], p[j - 3])));
  tz = fadd(tz, fmul(a.c4, fadd(p[j + 4], p[j - 4])));
  return fadd(fdiv(tx, a.dx2), fdiv(tz, a.dz2));
}

__device__ __forceinline__ float visco_sponge(const ViscoArgs &a, float v, int ix, int iz) {
  return fmul(a.bx[ix], fmul(a.bz[iz], v));  // z faces, then x faces (apply_sponge)
}

// one forward step of every shot of the batch (blockIdx.y = shot)
__global__ void visco_fwd_kernel(const ViscoArgs a) {
  const int s = blockIdx.y;
  const long long n = (long long)a.pnz * a.pnx;
  const float *A = a.A + s * a.fstride;
  float *B = a.B + s * a.fstride, *R = a.R + s * a.fstride;
  const float *rr = a.rr + s * n;
  const ShotGeo &g = a.geo[s];
  const float wv = a.wav[a.it];
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < n;
       j += (long long)gridDim.x * blockDim.x) {
    const int ix = (int)(j / a.pnz), iz = (int)(j - (long long)ix * a.pnz);
    const float p1 = A[j];
    if (a.rec && iz == a.rz) {  // traces read p1 before the step (wave_fwimodeling.c:181-185)
      const int d = ix - g.r0v;
      if (d >= 0 && d % a.drv == 0 && d / a.drv < g.nr2)
        a.rec[((size_t)s * a.nt + a.it) * a.nr + g.r02 + d / a.drv] = p1;
    }
    if (a.snap && ix >= a.nb && ix < a.nb + a.nx && iz >= a.nb && iz < a.nb + a.nz)
      a.snap[s * (long long)a.nx * a.nz + (long long)(ix - a.nb) * a.nz + (iz - a.nb)] = p1;
    if (ix < 4 || ix >= a.pnx - 4 || iz < 4 || iz >= a.pnz - 4) continue;
    const float L = visco_lap(a, A, j);
    const float tau = a.tau[j], taus = a.taus[j];
    const float r1 = visco_sponge(a, R[j], ix, iz);
    const double hts = __ddiv_rn(0.5, (double)taus);
    const double num = __dadd_rn((double)fmul(fdiv(tau, taus), L),
                                 __dmul_rn(__dsub_rn((double)a.idt, hts), (double)r1));
    const float r2 = __double2float_rn(__ddiv_rn(num, __dadd_rn((double)a.idt, hts)));
    const double tt = __dadd_rn(__dsub_rn(__dmul_rn((double)L, __dadd_rn(1.0, (double)tau)),
                                          __dmul_rn((double)fadd(r2, r1), 0.5)),
                                (double)fmul(rr[j], wv));
    const float t = __double2float_rn(tt);
    const float p0 = visco_sponge(a, B[j], ix, iz);
    const float p2 = fadd(fsub(fmul(2.f, p1), p0), fmul(a.V[j], t));
    B[j] = visco_sponge(a, p2, ix, iz);
    R[j] = r2;
  }
}

// adjoint, first half of a step: r2 and tmp from p1 and r1 (wave_fwigradient.c:393-403)
__global__ void visco_adj_pre_kernel(const ViscoArgs a) {
  const long long n = (long long)a.pnz * a.pnx;
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < n;
       j += (long long)gridDim.x * blockDim.x) {
    const int ix = (int)(j / a.pnz), iz = (int)(j - (long long)ix * a.pnz);
    if (ix < 4 || ix >= a.pnx - 4 || iz < 4 || iz >= a.pnz - 4) continue;
    const float p1 = a.A[j], tau = a.tau[j], taus = a.taus[j];
    const float r1 = visco_sponge(a, a.R[j], ix, iz);
    const double hts = __ddiv_rn(0.5, (double)taus);
    const double nidt = -(double)a.idt;
    const double num = __dadd_rn((double)fmul(fdiv(-tau, taus), p1),
                                 __dmul_rn(__dadd_rn(nidt, hts), (double)r1));
    const float r2 = __double2float_rn(__ddiv_rn(num, __dsub_rn(nidt, hts)));
    const double tm = __dsub_rn(__dmul_rn((double)p1, __dadd_rn(1.0, (double)tau)),
                                __dmul_rn(0.5, (double)fadd(r2, r1)));
    const_cast<float *>(a.T)[j] = __double2float_rn(tm);
    a.R[j] = r2;
  }
}

// adjoint, second half: Laplacian of tmp plus the residual, the update, and
// gradient_av's imaging with p1 (wave_fwigradient.c:405-438)
__global__ void visco_adj_kernel(const ViscoArgs a) {
  const long long n = (long long)a.pnz * a.pnx;
  const ShotGeo &g = a.geo[0];
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < n;
       j += (long long)gridDim.x * blockDim.x) {
    const int ix = (int)(j / a.pnz), iz = (int)(j - (long long)ix * a.pnz);
    if (ix < 4 || ix >= a.pnx - 4 || iz < 4 || iz >= a.pnz - 4) continue;
    float L = visco_lap(a, a.T, j);
    if (iz == a.rz) {
      const int d = ix - g.r0v;
      if (d >= 0 && d % a.drv == 0 && d / a.drv < g.nr2)
        L = fadd(L, a.res[(size_t)a.it * a.nr + g.r02 + d / a.drv]);
    }
    const float p1 = a.A[j];
    const float p0 = visco_sponge(a, a.B[j], ix, iz);
    const float p2 = fadd(fsub(fmul(2.f, p1), p0), fmul(a.V[j], L));
    if (a.imaging && ix >= a.nb && ix < a.nb + a.nx && iz >= a.nb && iz < a.nb + a.nz) {
      const size_t k = (size_t)(ix - a.nb) * a.nz + (iz - a.nb);
      const double w = __dadd_rn(__dsub_rn((double)a.wnext[k], __dmul_rn(2., (double)a.wcur[k])),
                                 (double)a.wprev[k]);
      const double gsum = __dmul_rn(__dmul_rn(__ddiv_rn(w, (double)a.wdt2), (double)p1),
                                    (double)a.m2v3[k]);
      a.grad[k] = __double2float_rn(__dadd_rn((double)a.grad[k], gsum));
    }
    a.B[j] = visco_sponge(a, p2, ix, iz);
  }
}

// preparation's tau, taus (wave_fwiutil.c:90-96) and the pad2d copies
static void visco_tables(const Setup &S, const float *q_host, std::vector<float> &tp,
                         std::vector<float> &tsp, std::vector<float> &Vp, const float *vel_host) {
  const pw_fwi_args &a = S.a;
  const double pi = 3.14159265358979323846264338328;
  const size_t nzx = (size_t)a.nz * a.nx, np = (size_t)S.pnz * S.pnx;
  std::vector<float> t1(nzx), ts1(nzx);
  for (size_t i = 0; i < nzx; i++) {
    const float qq = q_host[i];
    const float tmp = sqrtf(qq * qq + 1);
    const float taue = (tmp + 1) / (2. * pi * a.f0 * qq);
    ts1[i] = (tmp - 1) / (2. * pi * a.f0 * qq);
    t1[i] = taue / ts1[i] - 1;
  }
  const float dt2 = a.dt * a.dt;
  tp.resize(np);
  tsp.resize(np);
  Vp.resize(np);
  for (int ix = 0; ix < S.pnx; ix++)
    for (int iz = 0; iz < S.pnz; iz++) {
      const int jx = std::min(std::max(ix - a.nb, 0), a.nx - 1);
      const int jz = std::min(std::max(iz - a.nb, 0), a.nz - 1);
      const size_t j = (size_t)ix * S.pnz + iz, k = (size_t)jx * a.nz + jz;
      tp[j] = t1[k];
      tsp[j] = ts1[k];
      const float v = vel_host[k];
      Vp[j] = (v * v) * dt2;
    }
}

// the shots' source maps as dense fields, checked clear of the 4-cell rim
static int visco_sources(const Setup &S, int ns, std::vector<float> &rr) {
  const size_t np = (size_t)S.pnz * S.pnx;
  rr.assign(np * ns, 0.f);
  for (int is = 0; is < ns; is++) {
    const ShotGeo &g = S.geo[is];
    for (int k = 0; k < g.nsrc; k++) {
      const int x = g.scell[k] >> 16, z = g.scell[k] & 0xffff;
      PW_CHECK(x >= 4 && x < S.pnx - 4 && z >= 4 && z < S.pnz - 4, PW_ERR_SHAPE,
               "visco-acoustic path: shot %d's source map reaches the 4-cell rim", is);
      rr[np * is + (size_t)x * S.pnz + z] = g.sw[k];
    }
  }
  return PW_OK;
}

static void visco_base(const Setup &S, ViscoArgs &v) {
  v = ViscoArgs{};
  v.pnz = S.pnz;
  v.pnx = S.pnx;
  v.nb = S.a.nb;
  v.nz = S.a.nz;
  v.nx = S.a.nx;
  const float c0 = -205. / 72, c1 = 8. / 5, c2 = -1. / 5, c3 = 8. / 315, c4 = -1. / 560;
  v.c0 = c0; v.c1 = c1; v.c2 = c2; v.c3 = c3; v.c4 = c4;
  v.dx2 = S.a.dx * S.a.dx;
  v.dz2 = S.a.dz * S.a.dz;
  v.idt = 1. / S.a.dt;
  v.nt = S.a.nt;
  v.rz = S.rz;
  v.drv = S.drv;
  v.nr = S.nr;
  v.fstride = (long long)S.pnz * S.pnx;
}

// the acoustic path's stability limit on the host copy of the velocity
static int check_cfl_host(const Setup &S, const std::vector<float> &vh) {
  if (S.a.flags & PW_NO_CFL_CHECK) return PW_OK;
  float vmax = 0.f;
  for (float v : vh) vmax = std::max(vmax, v);
  const float cfl = vmax * S.a.dt / std::min(S.a.dx, S.a.dz);
  PW_CHECK(cfl <= 0.555f, PW_ERR_CFL, "unstable: vmax*dt/h = %g exceeds 0.555", cfl);
  return PW_OK;
}

// the host copies a visco call needs: velocity and quality factor
static int visco_host_inputs(const pw_fwi_args *a, const float *vel, const float *q,
                             std::vector<float> &vh, std::vector<float> &qh, cudaStream_t st) {
  const size_t nzx = (size_t)a->nz * a->nx;
  vh.resize(nzx);
  qh.resize(nzx);
  const bool host = (a->flags & PW_HOST_PTRS) != 0;
  if (host) {
    memcpy(vh.data(), vel, nzx * 4);
    memcpy(qh.data(), q, nzx * 4);
  } else {
    PW_CUDA(cudaMemcpyAsync(vh.data(), vel, nzx * 4, cudaMemcpyDeviceToHost, st));
    PW_CUDA(cudaMemcpyAsync(qh.data(), q, nzx * 4, cudaMemcpyDeviceToHost, st));
    PW_CUDA(cudaStreamSynchronize(st));
  }
  for (size_t i = 0; i < nzx; i++)
    PW_CHECK(vh[i] > 0.f && std::isfinite(vh[i]) && qh[i] > 0.f && std::isfinite(qh[i]),
             PW_ERR_VALUE, "velocity and quality factor must be finite and positive");
  return PW_OK;
}

}  // namespace pf
}  // namespace pw

extern "C" int pw_pfwi_forward_visco(const pw_fwi_args *a, const float *vel, const float *q,
                                     const float *wav, float *data, void *stream) {
  PW_CHECK(a && vel && q && wav && data, PW_ERR_VALUE, "null argument");
  cudaStream_t st = (cudaStream_t)stream;
  Setup S;
  PW_TRY(setup(a, S));
  const bool host = (a->flags & PW_HOST_PTRS) != 0;
  const int ns = a->ns, nt = a->nt, nr = S.nr;
  std::vector<float> vh, qh, tp, tsp, Vp, rr;
  PW_TRY(visco_host_inputs(a, vel, q, vh, qh, st));
  PW_TRY(check_cfl_host(S, vh));
  visco_tables(S, qh.data(), tp, tsp, Vp, vh.data());
  PW_TRY(visco_sources(S, ns, rr));
  const size_t np = (size_t)S.pnz * S.pnx;
  Carve cv;
  const size_t o_V = cv.add(np * 4), o_t = cv.add(np * 4), o_ts = cv.add(np * 4);
  const size_t o_A = cv.add((size_t)ns * np * 4), o_B = cv.add((size_t)ns * np * 4);
  const size_t o_R = cv.add((size_t)ns * np * 4), o_rr = cv.add((size_t)ns * np * 4);
  const size_t o_bz = cv.add(S.bz.size() * 4), o_bx = cv.add(S.bx.size() * 4);
  const size_t o_w = cv.add((size_t)nt * 4), o_geo = cv.add(sizeof(ShotGeo) * ns);
  const size_t o_rec = cv.add((size_t)ns * nt * nr * 4), o_out = cv.add((size_t)ns * nt * nr * 4);
  Workspace &ws = Workspace::for_current_device();
  std::lock_guard<std::mutex> lock(ws.mutex());
  struct Drain {
    cudaStream_t st;
    ~Drain() { cudaStreamSynchronize(st); }
  } drain{st};
  PW_TRY(ws.reserve(cv.total()));
  char *base = ws.base();
  PW_CUDA(cudaMemsetAsync(base, 0, cv.total(), st));
  PW_CUDA(cudaMemcpyAsync(base + o_V, Vp.data(), np * 4, cudaMemcpyHostToDevice, st));
  PW_CUDA(cudaMemcpyAsync(base + o_t, tp.data(), np * 4, cudaMemcpyHostToDevice, st));
  PW_CUDA(cudaMemcpyAsync(base + o_ts, tsp.data(), np * 4, cudaMemcpyHostToDevice, st));
  PW_CUDA(cudaMemcpyAsync(base + o_rr, rr.data(), rr.size() * 4, cudaMemcpyHostToDevice, st));
  PW_CUDA(cudaMemcpyAsync(base + o_bz, S.bz.data(), S.bz.size() * 4, cudaMemcpyHostToDevice, st));
  PW_CUDA(cudaMemcpyAsync(base + o_bx, S.bx.data(), S.bx.size() * 4, cudaMemcpyHostToDevice, st));
  PW_CUDA(cudaMemcpyAsync(base + o_geo, S.geo.data(), sizeof(ShotGeo) * ns,
                          cudaMemcpyHostToDevice, st));
  PW_TRY(to_device(base + o_w, wav, (size_t)nt * 4, host, st));
  ViscoArgs v;
  visco_base(S, v);
  v.V = at<float>(base, o_V);
  v.tau = at<float>(base, o_t);
  v.taus = at<float>(base, o_ts);
  v.bz = at<float>(base, o_bz);
  v.bx = at<float>(base, o_bx);
  v.rr = at<float>(base, o_rr);
  v.wav = at<float>(base, o_w);
  v.geo = at<ShotGeo>(base, o_geo);
  v.rec = at<float>(base, o_rec);
  v.R = at<float>(base, o_R);
  float *A = at<float>(base, o_A), *B = at<float>(base, o_B);
  const dim3 grid((unsigned)std::min<long long>(ceil_div((long long)np, 256), 1184), (unsigned)ns);
  LoopTimer timer(st);
  timer.start();
  for (int it = 0; it < nt; it++) {
    v.it = it;
    v.A = A;
    v.B = B;
    visco_fwd_kernel<<<grid, 256, 0, st>>>(v);
    PW_CUDA(cudaGetLastError());
    std::swap(A, B);
  }
  timer.stop();
  // traces [shot][nt][nr] -> data [shot][nr][nt]
  float *out = at<float>(base, o_out);
  for (int s = 0; s < ns; s++) {
    dim3 tb(32, 8), tg(ceil_div(nr, 32), ceil_div(nt, 32));
    transpose_kernel<<<tg, tb, 0, st>>>(v.rec + (size_t)s * nt * nr, out + (size_t)s * nr * nt,
                                        nt, nr);
  }
  PW_CUDA(cudaGetLastError());
  PW_TRY(to_host(data, out, (size_t)ns * nr * nt * 4, host, st));
  timer.finish(nt, nt + ns);
  PW_CUDA(cudaStreamSynchronize(st));
  return PW_OK;
}

extern "C" int pw_pfwi_gradient_visco(const pw_fwi_args *a, const float *vel, const float *q,
                                      const float *wav, const float *dobs, const float *weight,
                                      float *grad, double *misfit, void *stream) {
  PW_CHECK(a && vel && q && wav && dobs && grad, PW_ERR_VALUE, "null argument");
  cudaStream_t st = (cudaStream_t)stream;
  Setup S;
  PW_TRY(setup(a, S));
  const bool host = (a->flags & PW_HOST_PTRS) != 0;
  const int ns = a->ns, nt = a->nt, nr = S.nr, nz = a->nz, nx = a->nx;
  const size_t nzx = (size_t)nz * nx, np = (size_t)S.pnz * S.pnx;
  const int interval = std::max(1, a->interval);
  const int wnt = (nt - 1) / interval + 1;
  std::vector<float> vh, qh, tp, tsp, Vp, rr, wts;
  PW_TRY(visco_host_inputs(a, vel, q, vh, qh, st));
  PW_TRY(check_cfl_host(S, vh));
  visco_tables(S, qh.data(), tp, tsp, Vp, vh.data());
  PW_TRY(visco_sources(S, ns, rr));
  if (weight == nullptr) residual_weights(*a, nr, wts);
  Carve cv;
  const size_t o_V = cv.add(np * 4), o_t = cv.add(np * 4), o_ts = cv.add(np * 4);
  const size_t o_A = cv.add(np * 4), o_B = cv.add(np * 4), o_R = cv.add(np * 4);
  const size_t o_T = cv.add(np * 4), o_rr = cv.add((size_t)ns * np * 4);
  const size_t o_bz = cv.add(S.bz.size() * 4), o_bx = cv.add(S.bx.size() * 4);
  const size_t o_w = cv.add((size_t)nt * 4), o_geo = cv.add(sizeof(ShotGeo) * ns);
  const size_t o_wt = cv.add((size_t)nr * nt * 4);
  const size_t o_dobs = cv.add((size_t)ns * nt * nr * 4), o_din = cv.add((size_t)ns * nt * nr * 4);
  const size_t o_rec = cv.add((size_t)nt * nr * 4), o_res = cv.add((size_t)nt * nr * 4);
  const size_t o_snap = cv.add((size_t)wnt * nzx * 4);
  const size_t o_m2v3 = cv.add(nzx * 4), o_vel = cv.add(nzx * 4), o_grad = cv.add(nzx * 4);
  const size_t o_mis = cv.add(8 * (1 + RESID_BLOCKS));
  Workspace &ws = Workspace::for_current_device();
  std::lock_guard<std::mutex> lock(ws.mutex());
  struct Drain {
    cudaStream_t st;
    ~Drain() { cudaStreamSynchronize(st); }
  } drain{st};
  PW_TRY(ws.reserve(cv.total()));
  char *base = ws.base();
  PW_CUDA(cudaMemsetAsync(base, 0, cv.total(), st));
  PW_CUDA(cudaMemcpyAsync(base + o_V, Vp.data(), np * 4, cudaMemcpyHostToDevice, st));
  PW_CUDA(cudaMemcpyAsync(base + o_t, tp.data(), np * 4, cudaMemcpyHostToDevice, st));
  PW_CUDA(cudaMemcpyAsync(base + o_ts, tsp.data(), np * 4, cudaMemcpyHostToDevice, st));
  PW_CUDA(cudaMemcpyAsync(base + o_rr, rr.data(), rr.size() * 4, cudaMemcpyHostToDevice, st));
  PW_CUDA(cudaMemcpyAsync(base + o_bz, S.bz.data(), S.bz.size() * 4, cudaMemcpyHostToDevice, st));
  PW_CUDA(cudaMemcpyAsync(base + o_bx, S.bx.data(), S.bx.size() * 4, cudaMemcpyHostToDevice, st));
  PW_CUDA(cudaMemcpyAsync(base + o_geo, S.geo.data(), sizeof(ShotGeo) * ns,
                          cudaMemcpyHostToDevice, st));
  PW_CUDA(cudaMemcpyAsync(base + o_vel, vh.data(), nzx * 4, cudaMemcpyHostToDevice, st));
  PW_TRY(to_device(base + o_w, wav, (size_t)nt * 4, host, st));
  if (weight) PW_TRY(to_device(base + o_wt, weight, (size_t)nr * nt * 4, host, st));
  else PW_CUDA(cudaMemcpyAsync(base + o_wt, wts.data(), wts.size() * 4, cudaMemcpyHostToDevice, st));
  {
    PW_TRY(to_device(base + o_din, dobs, (size_t)ns * nt * nr * 4, host, st));
    for (int s = 0; s < ns; s++) {  // dobs [shot][nr][nt] -> [shot][nt][nr]
      dim3 tb(32, 8), tg(ceil_div(nt, 32), ceil_div(nr, 32));
      transpose_kernel<<<tg, tb, 0, st>>>(at<float>(base, o_din) + (size_t)s * nr * nt,
                                          at<float>(base, o_dobs) + (size_t)s * nt * nr, nr, nt);
    }
    PW_CUDA(cudaGetLastError());
  }
  m2v3_kernel<<<592, 256, 0, st>>>(at<float>(base, o_vel), nzx, at<float>(base, o_m2v3));
  PW_CUDA(cudaGetLastError());
  ViscoArgs v;
  visco_base(S, v);
  v.V = at<float>(base, o_V);
  v.tau = at<float>(base, o_t);
  v.taus = at<float>(base, o_ts);
  v.bz = at<float>(base, o_bz);
  v.bx = at<float>(base, o_bx);
  v.wav = at<float>(base, o_w);
  v.R = at<float>(base, o_R);
  v.T = at<float>(base, o_T);
  v.m2v3 = at<float>(base, o_m2v3);
  v.grad = at<float>(base, o_grad);
  v.wdt2 = (a->dt * interval) * (a->dt * interval);
  float *snap = at<float>(base, o_snap);
  double *dmis = at<double>(base, o_mis);
  const dim3 g1((unsigned)std::min<long long>(ceil_div((long long)np, 256), 1184), 1);
  LoopTimer timer(st);
  timer.start();
  long long launches = 0;
  // one shot at a time: the gradient sums the shots in the reference's order
  for (int is = 0; is < ns; is++) {
    float *A = at<float>(base, o_A), *B = at<float>(base, o_B);
    PW_CUDA(cudaMemsetAsync(A, 0, np * 4, st));
    PW_CUDA(cudaMemsetAsync(B, 0, np * 4, st));
    PW_CUDA(cudaMemsetAsync(v.R, 0, np * 4, st));
    v.geo = at<ShotGeo>(base, o_geo) + is;
    v.rr = at<float>(base, o_rr) + (size_t)is * np;
    v.rec = at<float>(base, o_rec);
    for (int it = 0; it < nt; it++) {
      v.it = it;
      v.A = A;
      v.B = B;
      v.snap = it % interval == 0 ? snap + (size_t)(it / interval) * nzx : nullptr;
      visco_fwd_kernel<<<g1, 256, 0, st>>>(v);
      PW_CUDA(cudaGetLastError());
      launches++;
      std::swap(A, B);
    }
    v.snap = nullptr;
    v.rec = nullptr;
    residual_kernel<<<RESID_BLOCKS, 256, 0, st>>>(at<float>(base, o_rec),
                                                  at<float>(base, o_dobs) + (size_t)is * nt * nr,
                                                  at<float>(base, o_wt), at<float>(base, o_res), 1,
                                                  nt, nr, 0, dmis);
    misfit_sum_kernel<<<1, 32, 0, st>>>(dmis, RESID_BLOCKS);
    PW_CUDA(cudaGetLastError());
    v.res = at<float>(base, o_res);
    PW_CUDA(cudaMemsetAsync(A, 0, np * 4, st));
    PW_CUDA(cudaMemsetAsync(B, 0, np * 4, st));
    PW_CUDA(cudaMemsetAsync(v.R, 0, np * 4, st));
    for (int it = nt - 1; it >= 0; it--) {
      const int wit = it / interval;
      v.it = it;
      v.A = A;
      v.B = B;
      v.imaging = (it % interval == 0) && wit != wnt - 1 && wit != 0;
      if (v.imaging) {
        v.wprev = snap + (size_t)(wit - 1) * nzx;
        v.wcur = snap + (size_t)wit * nzx;
        v.wnext = snap + (size_t)(wit + 1) * nzx;
      }
      visco_adj_pre_kernel<<<g1, 256, 0, st>>>(v);
      visco_adj_kernel<<<g1, 256, 0, st>>>(v);
      PW_CUDA(cudaGetLastError());
      launches += 2;
      std::swap(A, B);
    }
  }
  timer.stop();
  PW_TRY(to_host(grad, at<float>(base, o_grad), nzx * 4, host, st));
  if (misfit) PW_CUDA(cudaMemcpyAsync(misfit, dmis, 8, cudaMemcpyDeviceToHost, st));
  timer.finish(launches, launches + 4 * ns + 2);
  PW_CUDA(cudaStreamSynchronize(st));
  return PW_OK;
}

extern "C" int pw_last_fwi_plan(int *ckpt_k, int *shots_per_batch, long long *bytes,
                                double *recompute) {
  const PlanRecord &r = plan_record();
  if (ckpt_k) *ckpt_k = r.k;
  if (shots_per_batch) *shots_per_batch = r.nsb;
  if (bytes) *bytes = r.bytes;
  if (recompute) *recompute = r.recompute;
  return PW_OK;
}

extern "C" int pw_gradient_postprocess(int nz, int nx, int rect, int waterz, float *grad,
                                       float *scaling, int flags, void *stream) {
  cudaStream_t st = (cudaStream_t)stream;
  PW_CHECK(nz >= 1 && nx >= 1 && grad && scaling, PW_ERR_VALUE, "bad arguments");
  const bool host = (flags & PW_HOST_PTRS) != 0;
  const size_t n = (size_t)nz * nx;
  Carve cv;
  const size_t o_g = cv.add(host ? n * 4 : 0);
  const size_t o_tmp = cv.add(rect > 1 ? (size_t)std::max(nz, nx) * (std::max(nz, nx) + 2 * rect) * 4 : 0);
  const size_t o_mx = cv.add(16);
  const size_t o_sc = cv.add(16);
  Workspace &ws = Workspace::for_current_device();
  std::lock_guard<std::mutex> lock(ws.mutex());
  PW_TRY(ws.reserve(cv.total()));
  char *base = ws.base();
  float *g = host ? at<float>(base, o_g) : grad;
  if (host) PW_TRY(to_device(g, grad, n * 4, true, st));
  unsigned *mx = at<unsigned>(base, o_mx);
  float *sc = at<float>(base, o_sc);
  PW_CUDA(cudaMemsetAsync(mx, 0, 4, st));
  PW_CUDA(cudaMemcpyAsync(sc, scaling, 4, host ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice, st));
  // the first-call scale comes from the raw gradient (wave_fwigradient.c:245-251)
  absmax_kernel<<<296, 256, 0, st>>>(g, (long long)n, mx);
  if (rect > 1) {
    float *tmp = at<float>(base, o_tmp);
    smooth_lines_kernel<<<ceil_div(nx, 128), 128, 0, st>>>(g, nx, nz, nz, 1, rect, tmp);
    smooth_lines_kernel<<<ceil_div(nz, 128), 128, 0, st>>>(g, nz, nx, 1, nz, rect, tmp);
  }
  finish_kernel<<<296, 256, 0, st>>>(g, nz, nx, waterz, mx, sc);
  PW_CUDA(cudaGetLastError());
  if (host) PW_TRY(to_host(grad, g, n * 4, true, st));
  PW_CUDA(cudaMemcpyAsync(scaling, sc, 4, host ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice, st));
  PW_CUDA(cudaStreamSynchronize(st));
  return PW_OK;
}

// =========================================================================
// 3-D extension of the pfwi scheme (config: 400 x 400 x 200 batched FWI
// gradient).  The reference has no 3-D FWI; the scheme restates its 2-D
// acoustic step (wave_fwimodeling.c:21-114, wave_fwiutil.c:19-223) on three
// axes, exactly as the FP64 / FP32 oracle of oracle/pw_oracle3d_body.h does:
//   term = ((Tx / dx^2 + Tz / dz^2) + Ty / dy^2) + r w_n   (each T the
//          8th-order sum, zero outside [4, pad-4) on every axis; the
//          divisions as products with 1/h^2 rounded to float),
//   next = S(2 a - S b + V term),  S = Sy(Sx(Sz u)),  V = (v v) dt^2.
// Field layout: z contiguous with a 4-cell halo in front, 4 halo columns and
// 4 halo planes on each side:  off(iz, ix, iy) = (iz + 4) + sx (ix + 4) +
// sy (iy + 4), sx = lz (a multiple of 32 floats), sy = lz (pnx + 8).
// =========================================================================
namespace pw {
namespace pf3 {

using pf::FWD;
using pf::ADJ_EXACT;
constexpr int MAXS3 = 16;    // shots per launch
constexpr int MAXSRC = 64;   // source-map cells per shot
constexpr int XW3 = 4;       // columns (warps) per CTA, of one plane

struct Shot {
  int nsrc;
  int sz0, sz1, sx0, sx1, sy0, sy1;  // bounding box of the source cells
  int scell[MAXSRC];                 // iz | ix << 11 | iy << 22
  float sw[MAXSRC];
};

struct Args {
  int pnz, pnx, pny, lz;
  long long sx, sy, fstride;
  FastDiv nz4;          // float4 per padded column
  int zig;              // 1: odd steps run their blocks backwards
  int src_z0, src_z1;   // rows of the shots' source cells
  float c0, c1, c2, c3, c4, rdx2, rdz2, rdy2;
  float one;  // 1.0f at run time: keeps packed products unfused (pk2 helpers)
  int nshots;
  const float *cur;          // the shots' current fields, fstep floats apart
  float *nxt;                // the shots' previous fields, overwritten with the next
  long long fstep;
  const float *V;
  const float *bz, *bx, *by;
  int it, nt;
  const Shot *shots;
  int rz, nrx, nr;
  const int *rxmap, *rymap;  // receiver index along x / y, or -1
  const float *wav;
  float *rec;                // FWD: traces [shot][nt][nr] or null
  float *tout;               // FWD: term of this step [shot] (field layout) or null
  long long tout_stride;
  const float *res;          // ADJ: residual [shot][nt][nr]
  const float *tin;          // ADJ: forward term of this step [shot]
  long long tin_stride;
  float *grad;               // ADJ: phi * term accumulators (field layout) [shot]
  long long gstride;
};

__host__ __device__ inline long long off3(const Args &a, int iz, int ix, int iy) {
  return (long long)(iz + 4) + a.sx * (ix + 4) + a.sy * (iy + 4);
}

// One 3-D step: a thread updates one float4 of z cells of one column and plane
// of one shot, straight from global memory (8 x and 8 y neighbour float4s, the
// two z neighbours, the previous field and V; for the adjoint the forward term
// and the gradient), as the 2-D step does.  Shots are the fastest block index,
// so the shots of a cell share V through L2.
// Bound: load latency and L1's data pipe (21 float4 loads per float4; L1's load
// pipe is 75% busy, issue 55%, the return from L2 31%; DRAM
// would allow 57 us forward and 80 us adjoint).  Measured, one launch, 2 shots
// of 160 x 240 x 240, average of forward and adjoint: 95.6 us (157 with the
// former 3-plane shared-memory ring and a barrier per plane); 1 shot of 200 x
// 340 x 340 124 us (190), of 100 x 120 x 120 9.9 us (33).  72 registers (28
// warps per SM): 64 (spills) 102, 80 100, 96 104, 114 112; CTAs of 8 columns
// 107, of 4 columns x 2 planes 106, x 4 planes 143.
template <int MODE>
__global__ void __launch_bounds__(32 * XW3, 7) pf3_step_kernel(const __grid_constant__ Args a) {
  const int tile = blockIdx.x / a.nshots, s = blockIdx.x - tile * a.nshots;
  const unsigned item = tile * 32 + (threadIdx.x & 31);
  const int chunk = fast_div(item, a.nz4);
  const int z4 = (int)item - chunk * a.nz4.d;
  const int x = chunk * XW3 + (threadIdx.x >> 5), y = zigzag(a.it & a.zig, blockIdx.y, gridDim.y);
  const int iz0 = 4 * z4;
  pf::pdl_sync();
  if (x >= a.pnx) return;
  const long long sx = a.sx, sy = a.sy;
  const long long o = (iz0 + 4) + (long long)((unsigned long long)(unsigned)sx * (unsigned)(x + 4)) +
                      (long long)((unsigned long long)(unsigned)sy * (unsigned)(y + 4));
  const float *pc = a.cur + s * a.fstep + o;
  float *pn = a.nxt + s * a.fstep + o;
  const float4 c = pf::ld4(pc), L = pf::ld4(pc - 4), R = pf::ld4(pc + 4);
  float4 xp[4], xm[4], yp[4], ym[4];
#pragma unroll
  for (int d = 0; d < 4; d++) {
    xp[d] = pf::ld4(pc + (d + 1) * sx);
    xm[d] = pf::ld4(pc - (d + 1) * sx);
  }
#pragma unroll
  for (int d = 0; d < 4; d++) {
    yp[d] = pf::ld4(pc + (d + 1) * sy);
    ym[d] = pf::ld4(pc - (d + 1) * sy);
  }
  const float4 pv = pf::ld4(pn), V4 = pf::ld4(a.V + o);
  float4 tf = make_float4(0.f, 0.f, 0.f, 0.f), g0 = tf;
  float *pg = nullptr;
  if (MODE == ADJ_EXACT) {
    tf = __ldcs(reinterpret_cast<const float4 *>(a.tin + s * a.tin_stride + o));
    pg = a.grad + s * a.gstride + o;
    g0 = pf::ld4(pg);
  }
  const float bxf = a.bx[x], byf = a.by[y];
  const float4 bz4 = pf::ld4(a.bz + iz0);
  const bool lxy = x >= 4 && x < a.pnx - 4 && y >= 4 && y < a.pny - 4;
  // the stencil's rows [4, pnz - 4): see the 2-D step
  const bool lz_any = z4 >= 1 && iz0 < a.pnz - 4;
  const bool full = lxy && lz_any && iz0 + 3 < a.pnz - 4;
  const f2 k1 = pk2(a.one, a.one);
  float4 term4;
  {
    // the 8th-order sums along x, z and y in the reference's order, and
    // (tx / dx^2 + tz / dz^2) + ty / dy^2, for cells (0, 1) and (2, 3)
    // of the float4 per f32x2 op; the z neighbours at odd distances are
    // the float4s shifted by one cell
    const f2 kc[5] = {pk2(a.c0, a.c0), pk2(a.c1, a.c1), pk2(a.c2, a.c2), pk2(a.c3, a.c3),
                      pk2(a.c4, a.c4)};
    const f2 rx2 = pk2(a.rdx2, a.rdx2), rz2 = pk2(a.rdz2, a.rdz2), ry2 = pk2(a.rdy2, a.rdy2);
    const f2 cl = lo2(c), ch = hi2(c);
    const f2 s_wx = pk2(L.w, c.x), s_yz = pk2(c.y, c.z), s_wR = pk2(c.w, R.x);
    const f2 s_Lyz = pk2(L.y, L.z), s_Ryz = pk2(R.y, R.z);
    const f2 zp[2][4] = {{s_yz, ch, s_wR, lo2(R)}, {s_wR, lo2(R), s_Ryz, hi2(R)}};
    const f2 zm[2][4] = {{s_wx, hi2(L), s_Lyz, lo2(L)}, {s_yz, cl, s_wx, hi2(L)}};
    f2 t2[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      auto P = [h](const float4 &v) { return h ? hi2(v) : lo2(v); };
      f2 tx = mul2(mul2(kc[0], P(c)), k1), tz = tx, ty = tx;
#pragma unroll
      for (int d = 1; d <= 4; d++)
        tx = add2(tx, mul2(mul2(kc[d], add2(P(xp[d - 1]), P(xm[d - 1]))), k1));
#pragma unroll
      for (int d = 1; d <= 4; d++)
        tz = add2(tz, mul2(mul2(kc[d], add2(zp[h][d - 1], zm[h][d - 1])), k1));
#pragma unroll
      for (int d = 1; d <= 4; d++)
        ty = add2(ty, mul2(mul2(kc[d], add2(P(yp[d - 1]), P(ym[d - 1]))), k1));
      const f2 sxz = add2(mul2(mul2(tx, rx2), k1), mul2(mul2(tz, rz2), k1));
      t2[h] = add2(sxz, mul2(mul2(ty, ry2), k1));
    }
    term4 = join2(t2[0], t2[1]);
  }
  if (!full) {
#pragma unroll
    for (int e = 0; e < 4; e++)
      if (!(lxy && lz_any && iz0 + e < a.pnz - 4)) pf::set_el(term4, e, 0.f);
  }
  if (a.rz >= iz0 && a.rz < iz0 + 4) {
    // receivers: traces read the field before the step, residuals enter the adjoint
    const int rx_i = a.rxmap[x], ry_j = a.rymap[y];
    if (rx_i >= 0 && ry_j >= 0) {
      const size_t k = ((size_t)s * a.nt + a.it) * a.nr + (ry_j * a.nrx + rx_i);
      if (MODE == FWD) {
        if (a.rec) a.rec[k] = pf::el(c, a.rz - iz0);
      } else {
        const float r = a.res[k];
#pragma unroll
        for (int e = 0; e < 4; e++)
          if (iz0 + e == a.rz) pf::set_el(term4, e, fadd(pf::el(term4, e), r));
      }
    }
  }
  if (MODE == FWD && iz0 <= a.src_z1 && iz0 + 3 >= a.src_z0) {
    const Shot &sh = a.shots[s];
    if (x >= sh.sx0 && x <= sh.sx1 && y >= sh.sy0 && y <= sh.sy1) {
      const float wv = a.wav[a.it];
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const int key = (iz0 + e) | (x << 11) | (y << 22);
        for (int k = 0; k < sh.nsrc; k++)
          if (sh.scell[k] == key)
            pf::set_el(term4, e, fadd(pf::el(term4, e), fmul(sh.sw[k], wv)));
      }
    }
  }
  {
    // taper of the stored u_{k-1} (z, then x, then y faces), the update
    // with 2 c as c + c (the same bits, no product to fuse), the taper;
    // cells beyond pnz stay zero: every operand is zero there
    const f2 bx2 = pk2(bxf, bxf), by2 = pk2(byf, byf);
    f2 r2[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const f2 bz2 = h ? hi2(bz4) : lo2(bz4);
      const f2 cv2 = h ? hi2(c) : lo2(c);
      const f2 p = mul2(mul2(by2, mul2(bx2, mul2(bz2, h ? hi2(pv) : lo2(pv)))), k1);
      const f2 vt = mul2(mul2(h ? hi2(V4) : lo2(V4), h ? hi2(term4) : lo2(term4)), k1);
      const f2 v = add2(sub2(add2(cv2, cv2), p), vt);
      r2[h] = mul2(by2, mul2(bx2, mul2(bz2, v)));
    }
    *reinterpret_cast<float4 *>(pn) = join2(r2[0], r2[1]);
  }
  if (MODE == FWD && a.tout)
    __stcs(reinterpret_cast<float4 *>(a.tout + s * a.tout_stride + o), term4);
  if (MODE == ADJ_EXACT)
    *reinterpret_cast<float4 *>(pg) = join2(add2(lo2(g0), mul2(mul2(lo2(c), lo2(tf)), k1)),
                                            add2(hi2(g0), mul2(mul2(hi2(c), hi2(tf)), k1)));
}

// V = (v v) dt^2 on the padded grid (edge replication on every face)
__global__ void pad_V3_kernel(const float *vel, int nz, int nx, int ny, int nb, Args g, float dt2,
                              float *V) {
  const long long n = (long long)g.pnz * g.pnx * g.pny;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int iz = int(i % g.pnz), ix = int((i / g.pnz) % g.pnx), iy = int(i / ((long long)g.pnz * g.pnx));
    const int jz = min(max(iz - nb, 0), nz - 1), jx = min(max(ix - nb, 0), nx - 1);
    const int jy = min(max(iy - nb, 0), ny - 1);
    const float v = vel[((size_t)jy * nx + jx) * nz + jz];
    V[off3(g, iz, ix, iy)] = fmul(fmul(v, v), dt2);
  }
}

// dJ/dv = 2 / v * sum of the accumulators of the padded cells that pad3d
// copies from the interior cell (edge replication adjoint).  The first
// `edges` blocks take one edge or corner cell each ((nb + 1)^2 or (nb + 1)^3
// padded cells; one thread per cell took 1.1 ms at nb 20), the others every
// other cell, one per thread.
__device__ __forceinline__ void fold_range(int j, int n, int pn, int nb, int &lo, int &hi) {
  lo = j == 0 ? 0 : j + nb;
  hi = j == n - 1 ? pn - 1 : j + nb;
}
__global__ void __launch_bounds__(256) fold_grad3_kernel(const float *gacc, const float *vel, int nz,
                                                         int nx, int ny, int nb, Args g,
                                                         float *grad, int edges) {
  int z0, z1, x0, x1, y0, y1;
  if ((int)blockIdx.x < edges) {
    // block 4 k + corner: along y (k < ny), then x, then z
    const int corner = blockIdx.x & 3;
    int k = blockIdx.x >> 2, jz, jx, jy;
    if (k < ny) {
      jy = k;
      jz = (corner & 1) ? nz - 1 : 0;
      jx = (corner & 2) ? nx - 1 : 0;
    } else if (k < ny + nx) {
      jx = k - ny;
      jz = (corner & 1) ? nz - 1 : 0;
      jy = (corner & 2) ? ny - 1 : 0;
    } else {
      jz = k - ny - nx;
      jx = (corner & 1) ? nx - 1 : 0;
      jy = (corner & 2) ? ny - 1 : 0;
    }
    fold_range(jz, nz, g.pnz, nb, z0, z1);
    fold_range(jx, nx, g.pnx, nb, x0, x1);
    fold_range(jy, ny, g.pny, nb, y0, y1);
    const int cz = z1 - z0 + 1, cx = x1 - x0 + 1;
    const long long n = (long long)cz * cx * (y1 - y0 + 1);
    double s = 0.0;
    for (long long q = threadIdx.x; q < n; q += 256)
      s += (double)gacc[off3(g, z0 + (int)(q % cz), x0 + (int)(q / cz % cx), y0 + (int)(q / cz / cx))];
    s = pf::block_sum(s);
    const size_t i = ((size_t)jy * nx + jx) * nz + jz;
    if (threadIdx.x == 0) grad[i] = (float)(2.0 * s / (double)vel[i]);
    return;
  }
  const long long n = (long long)nz * nx * ny;
  for (long long i = (blockIdx.x - edges) * 256LL + threadIdx.x; i < n;
       i += (gridDim.x - edges) * 256LL) {
    const int jz = int(i % nz), jx = int((i / nz) % nx), jy = int(i / ((long long)nz * nx));
    const int faces = (jz == 0 || jz == nz - 1) + (jx == 0 || jx == nx - 1) + (jy == 0 || jy == ny - 1);
    if (faces >= 2) continue;
    fold_range(jz, nz, g.pnz, nb, z0, z1);
    fold_range(jx, nx, g.pnx, nb, x0, x1);
    fold_range(jy, ny, g.pny, nb, y0, y1);
    double s = 0.0;
    for (int iy = y0; iy <= y1; iy++)
      for (int ix = x0; ix <= x1; ix++)
        for (int iz = z0; iz <= z1; iz++) s += (double)gacc[off3(g, iz, ix, iy)];
    grad[i] = (float)(2.0 * s / (double)vel[i]);
  }
}

struct Setup3 {
  pw_fwi3d_args a;
  Args g;  // geometry part of the step arguments
  std::vector<float> bz, bx, by;
  std::vector<Shot> shots;
  std::vector<int> rxmap, rymap;
  int nr;
};

// Source map of one shot: the spike at padded (sz, sx, sy) smoothed by the
// rect-2 triangle along z and x (pf::source_map) and along y.
static int source_map3(int sz, int sx, int sy, const Setup3 &S, Shot &sh) {
  pf::ShotGeo g2;
  PW_TRY(pf::source_map(sx, sz, S.g.pnz, S.g.pnx, g2));
  const int pny = S.g.pny, r = 6;
  const int y_lo = std::max(0, sy - r), y_hi = std::min(pny - 1, sy + r);
  const bool full = y_lo == 0 || y_hi == pny - 1;
  const int ys = full ? 0 : y_lo, nyw = full ? pny : y_hi - y_lo + 1;
  std::vector<float> fy(nyw, 0.f), tmp;
  fy[sy - ys] = 1.f;
  pf::smooth_line_host(2, nyw, fy.data(), 0, 1, tmp);
  sh.nsrc = 0;
  sh.sz0 = sh.sx0 = sh.sy0 = 1 << 30;
  sh.sz1 = sh.sx1 = sh.sy1 = -1;
  for (int j = 0; j < nyw; j++) {
    if (fy[j] == 0.f) continue;
    const int gy = j + ys;
    PW_CHECK(gy >= 4 && gy < pny - 4, PW_ERR_SHAPE,
             "source map reaches the zero border of the padded grid");
    for (int k = 0; k < g2.nsrc; k++) {
      PW_CHECK(sh.nsrc < MAXSRC, PW_ERR_SHAPE, "source map has too many cells");
      const int gx = g2.scell[k] >> 16, gz = g2.scell[k] & 0xffff;
      sh.scell[sh.nsrc] = gz | (gx << 11) | (gy << 22);
      sh.sw[sh.nsrc] = g2.sw[k] * fy[j];
      sh.nsrc++;
      sh.sz0 = std::min(sh.sz0, gz); sh.sz1 = std::max(sh.sz1, gz);
      sh.sx0 = std::min(sh.sx0, gx); sh.sx1 = std::max(sh.sx1, gx);
      sh.sy0 = std::min(sh.sy0, gy); sh.sy1 = std::max(sh.sy1, gy);
    }
  }
  return PW_OK;
}

static int setup3(const pw_fwi3d_args *a, Setup3 &S) {
  PW_CHECK(a != nullptr, PW_ERR_VALUE, "null args");
  S.a = *a;
  PW_CHECK(a->nz >= 1 && a->nx >= 1 && a->ny >= 1 && a->nt >= 1 && a->ns >= 1 && a->nb >= 5,
           PW_ERR_SHAPE, "sizes must be positive and nb >= 5 (nz=%d nx=%d ny=%d nt=%d ns=%d nb=%d)",
           a->nz, a->nx, a->ny, a->nt, a->ns, a->nb);
  PW_CHECK(a->dx > 0 && a->dy > 0 && a->dz > 0 && a->dt > 0, PW_ERR_VALUE,
           "spacings must be positive");
  PW_CHECK(a->src && a->rx && a->ry && a->nrx >= 1 && a->nry >= 1, PW_ERR_VALUE,
           "sources and receivers are required");
  Args &g = S.g;
  memset(&g, 0, sizeof g);
  const int nb = a->nb;
  g.pnz = a->nz + 2 * nb;
  g.pnx = a->nx + 2 * nb;
  g.pny = a->ny + 2 * nb;
  PW_CHECK(g.pnz < 2048 && g.pnx < 2048 && g.pny < 512, PW_ERR_SHAPE,
           "padded grid beyond 2047 x 2047 x 511");
  g.lz = (int)round_up(4 + round_up(g.pnz, 4) + 4, 32);
  g.sx = g.lz;
  g.sy = (long long)g.lz * (g.pnx + 8);
  g.fstride = g.sy * (g.pny + 8) + 64;
  g.nz4 = make_fast_div(ceil_div(g.pnz, 4));
  g.fstep = g.fstride;
  const float c0 = -205. / 72, c1 = 8. / 5, c2 = -1. / 5, c3 = 8. / 315, c4 = -1. / 560;
  g.c0 = c0; g.c1 = c1; g.c2 = c2; g.c3 = c3; g.c4 = c4;
  g.rdz2 = 1.f / (a->dz * a->dz);
  g.rdx2 = 1.f / (a->dx * a->dx);
  g.rdy2 = 1.f / (a->dy * a->dy);
  g.one = 1.f;
  g.nt = a->nt;
  std::vector<float> bc(nb);
  for (int i = 0; i < nb; i++) {
    const float tmp = a->coef * (nb - i);
    bc[i] = expf(-tmp * tmp);
  }
  auto axis = [&](int n, std::vector<float> &f) {
    f.assign(n, 1.f);
    for (int i = 0; i < nb; i++) f[i] = bc[i];
    for (int i = n - nb; i < n; i++) f[i] = bc[n - i - 1];
  };
  axis(g.pnz, S.bz);
  S.bz.resize(round_up(g.pnz, 4), 1.f);  // read four at a time
  axis(g.pnx, S.bx);
  axis(g.pny, S.by);
  // receivers: the nrx x nry grid (rx[i], ry[j]) at depth rz, trace j nrx + i
  PW_CHECK(a->rz >= 0 && a->rz < a->nz, PW_ERR_SHAPE, "receiver depth outside the model");
  g.rz = a->rz + nb;
  g.nrx = a->nrx;
  S.nr = a->nrx * a->nry;
  g.nr = S.nr;
  S.rxmap.assign(g.pnx, -1);
  S.rymap.assign(g.pny, -1);
  for (int i = 0; i < a->nrx; i++) {
    PW_CHECK(a->rx[i] >= 0 && a->rx[i] < a->nx, PW_ERR_SHAPE, "receiver x index %d outside", i);
    PW_CHECK(S.rxmap[a->rx[i] + nb] < 0, PW_ERR_SHAPE, "receiver x index %d repeated", i);
    S.rxmap[a->rx[i] + nb] = i;
  }
  for (int j = 0; j < a->nry; j++) {
    PW_CHECK(a->ry[j] >= 0 && a->ry[j] < a->ny, PW_ERR_SHAPE, "receiver y index %d outside", j);
    PW_CHECK(S.rymap[a->ry[j] + nb] < 0, PW_ERR_SHAPE, "receiver y index %d repeated", j);
    S.rymap[a->ry[j] + nb] = j;
  }
  S.shots.assign(a->ns, Shot{});
  for (int is = 0; is < a->ns; is++) {
    const int z = a->src[3 * is], x = a->src[3 * is + 1], y = a->src[3 * is + 2];
    PW_CHECK(z >= 0 && z < a->nz && x >= 0 && x < a->nx && y >= 0 && y < a->ny, PW_ERR_SHAPE,
             "shot %d: source (z=%d, x=%d, y=%d) outside the model", is, z, x, y);
    PW_TRY(source_map3(z + nb, x + nb, y + nb, S, S.shots[is]));
  }
  g.src_z0 = 1 << 30;
  g.src_z1 = -1;
  for (const Shot &sh : S.shots) {
    g.src_z0 = std::min(g.src_z0, sh.sz0);
    g.src_z1 = std::max(g.src_z1, sh.sz1);
  }
  return PW_OK;
}

static int launch3(Args &p, int mode, cudaStream_t st) {
  p.zig = zigzag_pays((size_t)(2 * p.nshots + 1) * p.fstride * 4);
  const long long lanes = (long long)p.nz4.d * ceil_div(p.pnx, XW3);
  const dim3 grid((unsigned)(ceil_div(lanes, 32) * p.nshots), (unsigned)p.pny);
  PW_CUDA(launch_pdl(mode == FWD ? pf3_step_kernel<FWD> : pf3_step_kernel<ADJ_EXACT>, grid,
                     dim3(32 * XW3), 0, st, p));
  return PW_OK;
}

}  // namespace pf3
}  // namespace pw

using namespace pw::pf3;

// common device state of a 3-D call
namespace pw {
namespace pf3 {
struct Bound3 {
  size_t o_V, o_A, o_B, o_bz, o_bx, o_by, o_shots, o_rxm, o_rym, o_wav;
};
static void carve3(const Setup3 &S, int nsb, Carve &cv, Bound3 &b) {
  const size_t fb = (size_t)S.g.fstride * 4;
  b.o_V = cv.add(fb);
  b.o_A = cv.add((size_t)nsb * fb);
  b.o_B = cv.add((size_t)nsb * fb);
  b.o_bz = cv.add(S.bz.size() * 4);
  b.o_bx = cv.add(S.bx.size() * 4);
  b.o_by = cv.add(S.by.size() * 4);
  b.o_shots = cv.add(sizeof(Shot) * S.shots.size());
  b.o_rxm = cv.add(S.rxmap.size() * 4);
  b.o_rym = cv.add(S.rymap.size() * 4);
  b.o_wav = cv.add((size_t)S.a.nt * 4);
}
static int upload3(const Setup3 &S, char *base, const Bound3 &b, const float *wav, bool host,
                   cudaStream_t st) {
  PW_CUDA(cudaMemcpyAsync(base + b.o_bz, S.bz.data(), S.bz.size() * 4, cudaMemcpyHostToDevice, st));
  PW_CUDA(cudaMemcpyAsync(base + b.o_bx, S.bx.data(), S.bx.size() * 4, cudaMemcpyHostToDevice, st));
  PW_CUDA(cudaMemcpyAsync(base + b.o_by, S.by.data(), S.by.size() * 4, cudaMemcpyHostToDevice, st));
  PW_CUDA(cudaMemcpyAsync(base + b.o_shots, S.shots.data(), sizeof(Shot) * S.shots.size(),
                          cudaMemcpyHostToDevice, st));
  PW_CUDA(cudaMemcpyAsync(base + b.o_rxm, S.rxmap.data(), S.rxmap.size() * 4,
                          cudaMemcpyHostToDevice, st));
  PW_CUDA(cudaMemcpyAsync(base + b.o_rym, S.rymap.data(), S.rymap.size() * 4,
                          cudaMemcpyHostToDevice, st));
  PW_TRY(to_device(base + b.o_wav, wav, (size_t)S.a.nt * 4, host, st));
  return PW_OK;
}
static void bind3(const Setup3 &S, char *base, const Bound3 &b, Args &p) {
  p = S.g;
  p.V = at<float>(base, b.o_V);
  p.bz = at<float>(base, b.o_bz);
  p.bx = at<float>(base, b.o_bx);
  p.by = at<float>(base, b.o_by);
  p.shots = at<Shot>(base, b.o_shots);
  p.rxmap = at<int>(base, b.o_rxm);
  p.rymap = at<int>(base, b.o_rym);
  p.wav = at<float>(base, b.o_wav);
}
static int prep_vel3(const Setup3 &S, const float *vel, bool host, char *base, size_t o_vel,
                     size_t o_mx, const Bound3 &b, const float **d_vel, cudaStream_t st) {
  const size_t nvel = (size_t)S.a.nz * S.a.nx * S.a.ny;
  *d_vel = vel;
  if (host) {
    PW_TRY(to_device(base + o_vel, vel, nvel * 4, true, st));
    *d_vel = at<float>(base, o_vel);
  }
  unsigned *mx = at<unsigned>(base, o_mx);
  PW_CUDA(cudaMemsetAsync(mx, 0, 8, st));
  pf::vel_check_kernel<<<296, 256, 0, st>>>(*d_vel, (long long)nvel, mx);
  PW_CUDA(cudaGetLastError());
  unsigned hv[2] = {0, 0};
  PW_CUDA(cudaMemcpyAsync(hv, mx, 8, cudaMemcpyDeviceToHost, st));
  PW_CUDA(cudaStreamSynchronize(st));
  float vmax;
  memcpy(&vmax, &hv[0], 4);
  PW_CHECK(hv[1] == 0 && vmax > 0.f, PW_ERR_VALUE, "velocity has non-finite or non-positive values");
  if (!(S.a.flags & PW_NO_CFL_CHECK)) {
    // 8th-order leapfrog in 3-D: v dt / h <= 0.453 (measured limit)
    const float h = std::min(S.a.dx, std::min(S.a.dy, S.a.dz));
    const float cfl = vmax * S.a.dt / h;
    PW_CHECK(cfl <= 0.453f, PW_ERR_CFL, "unstable: vmax*dt/h = %g exceeds 0.453", cfl);
  }
  pad_V3_kernel<<<1184, 256, 0, st>>>(*d_vel, S.a.nz, S.a.nx, S.a.ny, S.a.nb, S.g,
                                      S.a.dt * S.a.dt, at<float>(base, b.o_V));
  PW_CUDA(cudaGetLastError());
  return PW_OK;
}
}  // namespace pf3
}  // namespace pw

extern "C" int pw_pfwi3d_forward(const pw_fwi3d_args *a, const float *vel, const float *wav,
                                 float *data, void *stream) {
  cudaStream_t st = (cudaStream_t)stream;
  Setup3 S;
  PW_TRY(setup3(a, S));
  const bool host = (a->flags & PW_HOST_PTRS) != 0;
  const int ns = a->ns, nt = a->nt, nr = S.nr;
  const int nsb = std::min(ns, MAXS3);
  const size_t nvel = (size_t)a->nz * a->nx * a->ny;
  const size_t fs = (size_t)S.g.fstride;
  Carve cv;
  Bound3 b;
  carve3(S, nsb, cv, b);
  const size_t o_vel = cv.add(host ? nvel * 4 : 0);
  const size_t o_rec = cv.add((size_t)ns * nt * nr * 4);
  const size_t o_out = cv.add(host ? (size_t)ns * nt * nr * 4 : 0);
  const size_t o_mx = cv.add(16);
  Workspace &ws = Workspace::for_current_device();
  std::lock_guard<std::mutex> lock(ws.mutex());
  PW_TRY(ws.reserve(cv.total()));
  char *base = ws.base();
  PW_CUDA(cudaMemsetAsync(base, 0, cv.total(), st));
  const float *d_vel;
  PW_TRY(upload3(S, base, b, wav, host, st));
  PW_TRY(prep_vel3(S, vel, host, base, o_vel, o_mx, b, &d_vel, st));
  Args p;
  bind3(S, base, b, p);
  float *rec = at<float>(base, o_rec);
  LoopTimer timer(st);
  timer.start();
  long long launches = 0;
  for (int s0 = 0; s0 < ns; s0 += nsb) {
    const int nb_ = std::min(nsb, ns - s0);
    float *A = at<float>(base, b.o_A), *B = at<float>(base, b.o_B);
    PW_CUDA(cudaMemsetAsync(A, 0, (size_t)nsb * fs * 4, st));
    PW_CUDA(cudaMemsetAsync(B, 0, (size_t)nsb * fs * 4, st));
    p.nshots = nb_;
    p.shots = at<Shot>(base, b.o_shots) + s0;
    p.rec = rec + (size_t)s0 * nt * nr;
    for (int it = 0; it < nt; it++) {
      p.it = it;
      p.cur = A;
      p.nxt = B;
      PW_TRY(launch3(p, FWD, st));
      launches++;
      std::swap(A, B);
    }
  }
  timer.stop();
  // [shot][nt][nr] -> [shot][nr][nt]
  float *dst = host ? at<float>(base, o_out) : data;
  for (int s = 0; s < ns; s++) {
    dim3 tb(32, 8), tg(ceil_div(nr, 32), ceil_div(nt, 32));
    pf::transpose_kernel<<<tg, tb, 0, st>>>(rec + (size_t)s * nt * nr, dst + (size_t)s * nt * nr,
                                            nt, nr);
  }
  PW_CUDA(cudaGetLastError());
  if (host) PW_TRY(to_host(data, dst, (size_t)ns * nt * nr * 4, true, st));
  PW_CUDA(cudaStreamSynchronize(st));
  timer.finish(launches, launches + 3 + ns);
  return PW_OK;
}

extern "C" int pw_pfwi3d_gradient(const pw_fwi3d_args *a, const float *vel, const float *wav,
                                  const float *dobs, const float *weight, float *grad,
                                  double *misfit, int ckpt_k, void *stream) {
  cudaStream_t st = (cudaStream_t)stream;
  Setup3 S;
  PW_TRY(setup3(a, S));
  const bool host = (a->flags & PW_HOST_PTRS) != 0;
  const int ns = a->ns, nt = a->nt, nr = S.nr;
  const size_t nvel = (size_t)a->nz * a->nx * a->ny;
  const size_t fs = (size_t)S.g.fstride;
  Workspace &ws = Workspace::for_current_device();
  std::lock_guard<std::mutex> lock(ws.mutex());
  // checkpoint plan: the 2-D planner's rule on 3-D fields
  pf::Setup P{};
  P.a.nt = nt;
  P.a.ns = std::min(ns, MAXS3);
  P.a.hbm_budget = a->hbm_budget;
  P.fstride = S.g.fstride;
  const ExactPlan ep = plan_exact(P, ckpt_k, ws.capacity());
  const int k = ep.k, nsb = ep.nsb, nck = (nt + k - 1) / k;
  plan_record().k = k;
  plan_record().nsb = nsb;
  plan_record().recompute = ep.recompute;
  Carve cv;
  Bound3 b;
  carve3(S, nsb, cv, b);
  const size_t o_vel = cv.add(host ? nvel * 4 : 0);
  const size_t o_w = cv.add(weight ? (size_t)nr * nt * 4 : 0);
  const size_t o_dobs = cv.add((size_t)ns * nt * nr * 4);  // [shot][nt][nr]
  const size_t o_dobs_in = cv.add(host ? (size_t)ns * nt * nr * 4 : 0);
  const size_t o_d = cv.add((size_t)nsb * nt * nr * 4);
  const size_t o_res = cv.add((size_t)nsb * nt * nr * 4);
  const size_t o_ck = cv.add((size_t)nsb * nck * 2 * fs * 4);
  const size_t o_tb = cv.add((size_t)nsb * k * fs * 4);
  const size_t o_ga = cv.add(fs * 4);
  const size_t o_gs = cv.add((size_t)nsb * fs * 4);  // shot slices, summed in shot order
  const size_t o_grad = cv.add(nvel * 4);
  const size_t o_mis = cv.add(8 * (1 + RESID_BLOCKS));
  const size_t o_mx = cv.add(16);
  PW_TRY(ws.reserve(cv.total()));
  plan_record().bytes = (long long)cv.total();
  char *base = ws.base();
  // checkpoints and segment terms are written before they are read
  PW_CUDA(cudaMemsetAsync(base, 0, o_ck, st));
  PW_CUDA(cudaMemsetAsync(base + o_ga, 0, cv.total() - o_ga, st));
  const float *d_vel;
  PW_TRY(upload3(S, base, b, wav, host, st));
  PW_TRY(prep_vel3(S, vel, host, base, o_vel, o_mx, b, &d_vel, st));
  float *d_w = nullptr;
  if (weight) {
    PW_TRY(to_device(base + o_w, weight, (size_t)nr * nt * 4, host, st));
    d_w = at<float>(base, o_w);
  }
  {
    const float *src = dobs;
    if (host) {
      PW_TRY(to_device(base + o_dobs_in, dobs, (size_t)ns * nt * nr * 4, true, st));
      src = at<float>(base, o_dobs_in);
    }
    for (int s = 0; s < ns; s++) {
      dim3 tb(32, 8), tg(ceil_div(nt, 32), ceil_div(nr, 32));
      pf::transpose_kernel<<<tg, tb, 0, st>>>(src + (size_t)s * nr * nt,
                                              at<float>(base, o_dobs) + (size_t)s * nt * nr, nr,
                                              nt);
    }
    PW_CUDA(cudaGetLastError());
  }
  Args p;
  bind3(S, base, b, p);
  float *gacc = at<float>(base, o_ga), *gslices = at<float>(base, o_gs);
  double *dmis = at<double>(base, o_mis);
  p.grad = gslices;
  p.gstride = (long long)fs;
  LoopTimer timer(st);
  timer.start();
  long long launches = 0;
  for (int s0 = 0; s0 < ns; s0 += nsb) {
    const int nb_ = std::min(nsb, ns - s0);
    float *A = at<float>(base, b.o_A), *B = at<float>(base, b.o_B);
    PW_CUDA(cudaMemsetAsync(A, 0, (size_t)nsb * fs * 4, st));
    PW_CUDA(cudaMemsetAsync(B, 0, (size_t)nsb * fs * 4, st));
    p.nshots = nb_;
    p.shots = at<Shot>(base, b.o_shots) + s0;
    auto step = [&](int mode, int it, float *&cur, float *&nxt, size_t stride) -> int {
      p.it = it;
      p.cur = cur;
      p.nxt = nxt;
      p.fstep = (long long)stride;
      PW_TRY(launch3(p, mode, st));
      launches++;
      std::swap(cur, nxt);
      return PW_OK;
    };
    float *dd = at<float>(base, o_d), *res = at<float>(base, o_res);
    float *ck = at<float>(base, o_ck), *tb = at<float>(base, o_tb);
    // ---- forward: traces, checkpoints, the last segment's terms
    p.rec = dd;
    p.tout_stride = (long long)k * fs;
    const int n_last = (nck - 1) * k;
    for (int it = 0; it < nt; it++) {
      if (it % k == 0 && it < n_last) {
        const int m = it / k;
        for (int s = 0; s < nb_; s++) {
          float *c = ck + ((size_t)s * nck + m) * 2 * fs;
          PW_CUDA(cudaMemcpyAsync(c, A + s * fs, fs * 4, cudaMemcpyDeviceToDevice, st));
          PW_CUDA(cudaMemcpyAsync(c + fs, B + s * fs, fs * 4, cudaMemcpyDeviceToDevice, st));
        }
      }
      p.tout = it >= n_last ? tb + (size_t)(it - n_last) * fs : nullptr;
      PW_TRY(step(FWD, it, A, B, fs));
    }
    p.rec = nullptr;
    p.tout = nullptr;
    // ---- FP64 misfit and the weighted residual
    pf::residual_kernel<<<pf::RESID_BLOCKS, 256, 0, st>>>(
        dd, at<float>(base, o_dobs) + (size_t)s0 * nt * nr, d_w, res, nb_, nt, nr, 1, dmis);
    pf::misfit_sum_kernel<<<1, 32, 0, st>>>(dmis, pf::RESID_BLOCKS);
    PW_CUDA(cudaGetLastError());
    p.res = res;
    // ---- backward by segments (the adjoint pair reuses the forward pair)
    A = at<float>(base, b.o_A);
    B = at<float>(base, b.o_B);
    PW_CUDA(cudaMemsetAsync(A, 0, (size_t)nsb * fs * 4, st));
    PW_CUDA(cudaMemsetAsync(B, 0, (size_t)nsb * fs * 4, st));
    p.tin_stride = (long long)k * fs;
    for (int m = nck - 1; m >= 0; m--) {
      const int n0 = m * k, n1 = std::min(nt, n0 + k);
      float *FA = ck + (size_t)m * 2 * fs, *FB = FA + fs;
      for (int n = n0; n < n1 && m < nck - 1; n++) {  // the last segment is kept
        p.tout = tb + (size_t)(n - n0) * fs;
        PW_TRY(step(FWD, n, FA, FB, (size_t)nck * 2 * fs));
      }
      p.tout = nullptr;
      for (int n = n1 - 1; n >= n0; n--) {
        p.tin = tb + (size_t)(n - n0) * fs;
        PW_TRY(step(ADJ_EXACT, n, A, B, fs));
      }
    }
    p.tin = nullptr;
    {
      pf::sum_slices_kernel<<<592, 256, 0, st>>>(gslices, nb_, (long long)fs, gacc);
      PW_CUDA(cudaGetLastError());
      PW_CUDA(cudaMemsetAsync(gslices, 0, (size_t)nb_ * fs * 4, st));
      launches++;
    }
  }
  timer.stop();
  float *gdev = at<float>(base, o_grad);
  const int edges = 4 * (a->nz + a->nx + a->ny);
  fold_grad3_kernel<<<edges + 592, 256, 0, st>>>(gacc, d_vel, a->nz, a->nx, a->ny, a->nb, S.g, gdev,
                                                 edges);
  PW_CUDA(cudaGetLastError());
  PW_TRY(to_host(grad, gdev, nvel * 4, host, st));
  if (misfit) PW_CUDA(cudaMemcpyAsync(misfit, dmis, 8, cudaMemcpyDeviceToHost, st));
  PW_CUDA(cudaStreamSynchronize(st));
  timer.finish(launches, launches + 8);
  return PW_OK;
}
