// shoc_tr_tile64.cuh -- the plain FP64 transport kernels, bitwise equal to the
// reference: model/hd/tracers/tracers.c's arithmetic operation by operation
// (compiled without FMA contraction; quotients correctly rounded).  They step
// every scheme and every wet column but those whose thin-surface cursor
// couples tracers or whose implicit solve is degenerate (k_general).
//
//  k_adv64  a warp per segment of columns and chunk of layers: the face
//           values of the scheme with ULTIMATE and horizontal diffusion of the
//           cell's west, south, north and top faces (quickest :1819-1931,
//           ulimate_filter :3501-3557, van_leer_do :2087-2119, hor_diffuse
//           :3595-3668), the flux divergence and the interior update
//           (advect_diffuse :888-925).  The Courant numbers are formed in the
//           kernel exactly as :730-736 form them.
//  k_vd64   one thread per (column, tracer): tr_bounds (:3217-3324),
//           surf_conc (:3047-3207), the copy above the surface, and the
//           implicit vertical diffusion (implicit_vdiff_tr :4067-4214) with
//           the LU factors k_set_dz builds.
//
// A face two cells share is computed from the same operands in the same order
// wherever it is computed, so the results are those of column_pass.
#pragma once
#include <type_traits>

#include "shoc_tr_tile.cuh"

namespace shoc {

// ---------------------------------------------------------------------------
// k_adv64
//
// A warp owns a segment of the column order (Tile::seg: up to 32 neighbouring
// columns; where the 32nd is the east neighbour of the 31st it only lends its
// west flux, the halo lane) and a chunk of layers, and climbs the chunk: the
// east flux is the next lane's west flux (a shuffle) and the bottom flux the
// top flux of the layer below (kept per tracer in shared memory), so a cell
// costs four face values where one thread per cell and no climbing cost six
// executed ones (the east one for a warp's last lane alone).  The warps are
// independent of one another.
//
// What bounds it: FP64 instructions and the latency of their chains.  The
// reference divides by 6, by the cell area and thickness and up to four times
// in ULTIMATE for every face; nothing but its own operation order gives its
// bits.  So
//  - quotients by divisors no tracer changes (6, area, dz, |cr|) come from the
//    correctly rounded reciprocal and two residual corrections (quot), and
//    ULTIMATE's by td - tu from one reciprocal that Van Leer's slope shares;
//  - all of it is computed for every face and selected, so a cell's faces are
//    one straight line of code the compiler interleaves; one check of the
//    exponents of the cell's stencil values decides whether quotients may be
//    formed this way, and a cell that fails it (values below 2^-400 or above
//    2^490, NaN), or has a divisor recip does not round, computes its faces by
//    the reference's divisions;
//  - the faces' factors live in shared memory, written when a layer is set up
//    (in registers they left 12 warps on an SM), and a tracer's stencil values
//    are loaded while the one before it is computed, of the two values beyond a
//    face only the upwind one.
// 384 x 320 x 40, 10 tracers (B200), a sub-step: 1.75 ms with one thread per
// cell and the reference's divisions; climbing, 2.35 ms with the limiter's
// cases as branches, 1.15 ms as selections, 1.08 ms with upwind loads alone,
// 1.00 ms with loads a tracer ahead and one-warp blocks (four-warp blocks wait
// for their deepest column: 1.04), 0.81 with chunks of the layers the columns have
// (build_tile_tables).  A warp per face with the fluxes meeting in
// shared memory took 1.25 ms: more warps, but a quarter more instructions.

// Correctly rounded a / b from y = RN(1 / b) (P. Markstein, IBM J. Res. Dev.
// 34, 1990: with y the correctly rounded reciprocal, q within an ulp of a / b
// and r = a - b q exact, RN(q + r y) is RN(a / b); the first correction brings
// RN(a y) within an ulp) where neither a, b nor a / b are near the ends of the
// range, or a is 0.  A zero quotient may have the other sign (a = -0 over b > 0);
// with a residual of the opposite sign, which costs the same, it has a's.
__device__ __forceinline__ double quot(double a, double b, double y) {
  double q = __dmul_rn(a, y);
  q = __fma_rn(__fma_rn(-b, q, a), y, q);
  return __fma_rn(__fma_rn(-b, q, a), y, q);
}
// the same for b > 0, of a zero too
__device__ __forceinline__ double quot_pos(double a, double b, double y) {
  double q = __dmul_rn(a, y);
  q = __fma_rn(-__fma_rn(b, q, -a), y, q);
  return __fma_rn(-__fma_rn(b, q, -a), y, q);
}
// |x| outside 2^-lim .. 2^lim (a zero too)
template <unsigned LIM>
__device__ __forceinline__ bool far_out(double x) {
  return ((unsigned)__double2hiint(x) & 0x7fffffffu) - ((1023u - LIM) << 20) >= ((2 * LIM) << 20);
}
// Whether quot may form a / b for a b the caller keeps 1 / b of.  lo: kDivLo
// where b lies in 2^-200 .. 2^200, so that nothing under- or overflows for |a|
// in 2^-700 .. 2^700; kDivNever where it does not.
constexpr unsigned kDivLo = (1023u - 700u) << 20, kDivSpan = 1400u << 20;
constexpr unsigned kDivNever = 0x80000000u;
__device__ __forceinline__ unsigned div_range(double b) {
  return far_out<200>(b) ? kDivNever : kDivLo;
}
__device__ __forceinline__ bool div_fast(double a, unsigned lo) {
  return ((unsigned)__double2hiint(a) & 0x7fffffffu) - lo < kDivSpan;
}
// RN(1 / d) for |d| in 2^-500 .. 2^500: Newton steps from the hardware's
// approximation (20 bits); the last one starts within an ulp, so it rounds
// correctly (Markstein) unless d's significand is all ones: there it meets a
// tie (2 - 2^-52: 0.5, not 0.5 + 2^-53) that quot does not make good.  unsafe:
// d may be such a divisor (its low word decides, one comparison)
__device__ __forceinline__ double recip(double d) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  y = __fma_rn(__fma_rn(-d, y, 1.0), y, y);
  y = __fma_rn(__fma_rn(-d, y, 1.0), y, y);
  return __fma_rn(__fma_rn(-d, y, 1.0), y, y);
}
__device__ __forceinline__ bool recip_unsafe(double d) { return __double2loint(d) == -1; }

// One face, set up once per cell for every tracer, in the warp's shared memory
// (a row of 32 doubles each): the Courant number, the scheme's factors for its
// sign (the curvature is D (P td + Q tu) - 2 tc; e: 1 - cr^2, Van Leer
// (1 -+ cr) / 2), 1 / |cr| for the limiter and the volume flux
enum { FC_CR, FC_U, FC_E, FC_Y, FC_D, FC_DB, FC_P, FC_Q, FC_N };
constexpr int F64_POS = 1, F64_MOVE = 2, F64_VNZ = 4, F64_LIM = 8, F64_VAL = 16, F64_REF = 32;

// hm, h0, hp: the metric at the cell behind, at and ahead of the face; val:
// the scheme fills this face; lim: the limiter acts on it.  Returns its flags.
template <int SCH>
__device__ __forceinline__ int set_face_64(double *f, double cr, double vel, double d, double db,
                                           double df, double hm, double h0, double hp, double U,
                                           bool val, bool lim) {
  constexpr bool byvel = SCH == SHOC_TR_VANLEER || SCH == SHOC_TR_ORDER2_UW;
  const bool pos = byvel ? vel > 0.0 : cr > 0.0;
  if (byvel) val = val && vel != 0.0;
  int bits = (pos ? F64_POS : 0) | (cr != 0.0 ? F64_MOVE : 0) | (val ? F64_VAL : 0);
  bool ref = false;
  f[FC_U * 32] = U;
  f[FC_CR * 32] = cr;
  if (SCH == SHOC_TR_QUICKEST || SCH == SHOC_TR_QUICKEST_CO) f[FC_E * 32] = 1.0 - cr * cr;
  if (SCH == SHOC_TR_VANLEER) f[FC_E * 32] = pos ? 0.5 * (1.0 - cr) : 0.5 * (1.0 + cr);
  if (SCH == SHOC_TR_QUICKEST) {
    const double D = pos ? db : df, P = pos ? hm : hp;
    f[FC_D * 32] = d;
    f[FC_DB * 32] = D;
    f[FC_P * 32] = P;
    f[FC_Q * 32] = h0;
    ref = far_out<60>(D) || far_out<60>(P) || far_out<60>(h0);
  }
  if (SCH == SHOC_TR_ORDER2) f[FC_D * 32] = d;
  if (lim && cr != 0.0) {
    const double acr = fabs(cr);
    f[FC_Y * 32] = 1.0 / acr;
    bits |= F64_LIM;
    // by velocity's sign the limiter's upwind side is the scheme's
    ref = ref || far_out<200>(acr) || acr > 0x1p20 || (byvel && pos != (cr > 0.0));
  } else {
    f[FC_Y * 32] = 1.0;
  }
  return bits | (ref ? F64_REF : 0);
}

// The flux by the reference's operations and divisions; of tm2 and tp1 (the
// values at i-2 and i+1) only the upwind one, tu, is needed but by ORDER4
template <int SCH, bool ULT>
__device__ __noinline__ double face_ref64(const double *f, int bits, double tu, double tm1,
                                          double t0, double tm2, double tp1) {
  const double cr = f[FC_CR * 32];
  const bool pos = (bits & F64_POS) != 0;
  const double vel = (bits & F64_VAL) ? (pos ? 1.0 : -1.0) : 0.0;
  double v = 0.0;
  if (SCH == SHOC_TR_QUICKEST) {
    const double grad = t0 - tm1, tc = pos ? tm1 : t0, td = pos ? t0 : tm1;
    v = f[FC_D * 32] * grad + tm1;
    double curv = 0.0;
    if (bits & F64_MOVE)
      curv = f[FC_DB * 32] * (f[FC_P * 32] * td + f[FC_Q * 32] * tu) - 2.0 * tc;
    v = v - 0.5 * cr * grad - f[FC_E * 32] * curv / 6.0;
  } else if (SCH == SHOC_TR_QUICKEST_CO) {
    v = quickest_co_face(cr, tu, tm1, t0, tu);
  } else if (SCH == SHOC_TR_VANLEER) {
    v = vanleer_face(vel, cr, tu, tm1, t0, tu);
  } else if (SCH == SHOC_TR_ORDER2 && (bits & F64_VAL)) {
    v = order2_face(f[FC_D * 32], tm1, t0);
  } else if (SCH == SHOC_TR_ORDER4 && (bits & F64_VAL)) {
    v = order4_face(tm2, tm1, t0, tp1);
  } else if (SCH == SHOC_TR_ORDER2_UW) {
    v = order2_uw_face(vel, cr, tu, tm1, t0, tu);
  }
  if (ULT && (bits & F64_LIM))  // (its unused side's value is not read)
    v = cr > 0.0 ? ultimate_face(cr, v, SCH == SHOC_TR_ORDER4 ? tm2 : tu, tm1, t0, t0)
                 : ultimate_face(cr, v, t0, tm1, t0, SCH == SHOC_TR_ORDER4 ? tp1 : tu);
  return v * f[FC_U * 32];
}

// The face's flux from the values tm1, t0 beside it and the upwind one beyond
// them, tu (i-2 for a positive Courant number, i+1 for a negative one; tm2 and
// tp1, both of them, for ORDER4) (advect: quickest :1870-1884, van_leer_do
// :2102-2117, the other schemes, then ulimate_filter), without horizontal
// diffusion, for values in the checked range; redo is set where a divisor is not
// recip's and face_ref64 has to be asked
template <int SCH, bool ULT>
__device__ __forceinline__ double face_flux64(const double *f, int bits, double tu, double tm1,
                                              double t0, double tm2, double tp1, bool &redo) {
  if (SCH == SHOC_TR_ORDER1) return order1_flux(f[FC_U * 32], tm1, t0);
  const bool pos = (bits & F64_POS) != 0, val = (bits & F64_VAL) != 0;
  const double tc = pos ? tm1 : t0, td = pos ? t0 : tm1;
  const double diff = td - tu, c = tc - tu, cr = f[FC_CR * 32];
  double y = 0.0;
  if (ULT || SCH == SHOC_TR_VANLEER) {
    y = recip(diff);
    redo = redo || recip_unsafe(diff);
  }
  double v;
  if (SCH == SHOC_TR_QUICKEST) {
    const double grad = t0 - tm1;
    v = f[FC_D * 32] * grad + tm1;
    // (2 tc is exact, so its fused subtraction rounds as the separate one)
    const double curv =
        __fma_rn(-2.0, tc, f[FC_DB * 32] * (f[FC_P * 32] * td + f[FC_Q * 32] * tu));
    const double q = v - 0.5 * cr * grad - quot_pos(f[FC_E * 32] * curv, 6.0, 1.0 / 6.0);
    v = (bits & F64_MOVE) ? q : v;
  } else if (SCH == SHOC_TR_QUICKEST_CO) {
    const double curv = pos ? t0 - 2.0 * tm1 + tu : tu - 2.0 * t0 + tm1;
    const double w = (bits & F64_MOVE) ? f[FC_E * 32] * curv : 0.0;
    v = 0.5 * (t0 + tm1) - 0.5 * cr * (t0 - tm1) - quot_pos(w, 6.0, 1.0 / 6.0);
  } else if (SCH == SHOC_TR_VANLEER) {
    // with the flow negative the reference's differences, and their quotient,
    // have the opposite signs (a zero too), and the value is t0 minus the term
    const double p = c * (td - tc);
    const double s = p > 0.0 ? quot(2.0 * p, diff, y) : pos ? 0.0 : -0.0;
    v = val ? tc + f[FC_E * 32] * s : 0.0;
  } else if (SCH == SHOC_TR_ORDER2) {
    v = val ? order2_face(f[FC_D * 32], tm1, t0) : 0.0;
  } else if (SCH == SHOC_TR_ORDER4) {
    v = val ? quot_pos(7.0 * (tm1 + t0) - (tp1 + tm2), 12.0, 1.0 / 12.0) : 0.0;
  } else {  // ORDER2_UW
    v = val ? 0.5 * (3.0 - cr) * tc - 0.5 * (1.0 - cr) * tu : 0.0;
  }
  if (ULT) {
    const double nc = quot(c, diff, y), nu = quot(v - tu, diff, y), acr = fabs(cr);
    const double ya = f[FC_Y * 32], p = nc * diff;
    const bool in = nc >= 0.0 && nc <= 1.0;
    const bool cap = nu > quot_pos(nc, acr, ya);
    const double up = tu + p, upc = tu + quot_pos(p, acr, ya);
    double l = cap ? upc : v;
    l = nu < nc ? up : l;
    l = nu > 1.0 ? td : l;
    l = in ? l : up;
    v = (diff != 0.0 && (bits & F64_LIM)) ? l : v;
  }
  return v * f[FC_U * 32];
}

// What the reference has for a floor that lets nothing through (w = 0): 0 times the
// face value between the ghost below, which holds t0, t0 and tp1 above.  It
// matters where t0 is a zero whose sign it may decide (the schemes of
// kFloorZero64: the others' is +0 then), or not finite.
template <int SCH>
constexpr bool kFloorZero64 = SCH == SHOC_TR_ORDER1 || SCH == SHOC_TR_ORDER4 ||
                              SCH == SHOC_TR_QUICKEST_CO;
template <int SCH>
__device__ __forceinline__ double floor_flux64(double t0, double tp1) {
  if (SCH == SHOC_TR_VANLEER || SCH == SHOC_TR_ORDER2_UW) return 0.0;
  if (SCH == SHOC_TR_ORDER4) return 0.0 * order4_face(t0, t0, t0, tp1);
  return 0.0 * (kFloorZero64<SCH> ? t0 : 0.0 + t0);
}

// Whether every value of a list lies in 2^-400 .. 2^490 or is 0: differences
// of such values are 0 or above 2^-453, and the faces' quotients stay inside
// the range quot takes.  (h - 1 orders a zero high word last; a subnormal
// below 2^-1042 counts as 0 only where its low word is 0 too.)
struct ExpCheck {
  unsigned hi = 0, lo = 0xffffffffu;
  __device__ __forceinline__ void add(double x) {
    const unsigned h = (unsigned)__double2hiint(x) & 0x7fffffffu;
    hi = max(hi, h);
    lo = min(lo, (h | min((unsigned)__double2loint(x), 1u)) - 1u);
  }
  __device__ __forceinline__ bool bad() const {
    return hi >= ((1023u + 490u) << 20) || lo < ((1023u - 400u) << 20) - 1u;
  }
};

constexpr int kAdv64Warps = 1;   // warps of a block (they share nothing)
constexpr int kAdv64Group = 32;  // tracers whose bottom fluxes a launch row keeps
constexpr int kAdv64Faces = 4;   // west, south, north, top
inline size_t adv64_smem(int ng) {
  return (size_t)kAdv64Warps * (kAdv64Faces * FC_N + ng) * 32 * sizeof(double);
}

// PLAIN: every advected tracer is advected without horizontal diffusion.
// A warp's work is item kAdv64Warps blockIdx.x + its number of the list: a segment
// (x) and layers k0 to below k1 of it (y: k0 | k1 << 16); blockIdx.y: groups of ng
// tracers.
template <int SCH, bool ULT, bool PLAIN>
__global__ void __launch_bounds__(kAdv64Warps * 32, 16)
    k_adv64(Geo G, Flow F, Work W, TrSet T, SubStep ss, Tile Tl,
            const double *__restrict__ tri, double *__restrict__ tro, double *__restrict__ fzs,
            const int2 *__restrict__ items, int nitem, int ng) {
  extern __shared__ double sAdv[];  // per warp: [kAdv64Faces][FC_N][32], [ng][32]
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, wy = threadIdx.x >> 5;
  const int item = blockIdx.x * kAdv64Warps + wy;
  if (item >= nitem) return;
  const int2 it = __ldg(&items[item]);
  const int seg = it.x, k0 = it.y & 0xffff, k1 = it.y >> 16;
  const int sl0 = blockIdx.y * ng, sl1 = min(T.ntb, sl0 + ng);
  double *const fw = sAdv + (size_t)wy * (kAdv64Faces * FC_N + ng) * 32 + lane;
  double *const fs = fw + FC_N * 32, *const fn = fs + FC_N * 32, *const ft = fn + FC_N * 32;
  double *const sF = ft + FC_N * 32;  // the flux through the layer's bottom, per tracer

  const int sc = Tl.seg[seg * 32 + lane];
  const bool own = sc >= 0 && !(sc & kSegHalo);
  const int col = sc >= 0 ? (sc & ~kSegHalo) : -1;
  int kb = G.nz, ks = -1, c2 = 0, ntc = 0;
  bool staged = false, open = false;  // open: water goes through the floor, in this chunk
  if (col >= 0) {
    const int4 r = __ldg(&Tl.colrec[col]);
    kb = r.z;
    c2 = r.y;
    const ColInfo ci = W.col[col];
    staged = own && (ci.flags & COL_STAGED);
    ks = ci.ks;
    ntc = __ldg(&G.colntr[col]);
    if (staged && kb >= k0 && kb < k1) open = __double_as_longlong(__ldg(&F.w[r.x])) != 0;
  }
  if (!__any_sync(FULL, staged)) return;
  const double dtu = ss.dtu;
  const double area = col >= 0 ? __ldg(&G.cellarea[c2]) : 1.0;
  const double yarea = 1.0 / area;
  // the bottom face of cell cc (below it zm, above it zp)
  auto zset = [&](double *f, int cc, int zm, int zp) {
    const double w9c = W.w9[cc], w = __ldg(&F.w[cc]);
    return set_face_64<SCH>(f, w * dtu / (w9c * 1.0), w,
                            (SCH == SHOC_TR_QUICKEST || SCH == SHOC_TR_ORDER2) ? W.w5[cc] : 0.0,
                            W.dbz[cc], W.dfz[cc], W.w9[zm], w9c, W.w9[zp],
                            SCH == SHOC_TR_ORDER1 ? w : w * dtu, true, ULT);
  };
  // the tracers of this row (at most 32), a lane each
  const int my_tr = sl0 + lane < sl1 ? __ldg(&T.slot_tr[sl0 + lane]) : 0;
  // order1's vertical flux (:1611-1616)
  auto order1_z = [&](double w, double tm1, double t0) {
    return dtu * (0.5 * (w + fabs(w)) * tm1 + 0.5 * (w - fabs(w)) * t0);
  };

  // the flux through the bottom of the chunk's first layer, or through an open
  // floor in the chunk, for every tracer (a closed floor's is 0)
  {
    const int kk = open ? kb : k0;
    const int c = (staged && (open || k0 > kb) && kk <= ks)
                      ? __ldg(&Tl.cellk[(size_t)kk * Tl.ncolp + col]) : 0;
    int4 nzv = make_int4(0, 0, 0, 0);
    int bits = 0;
    const bool flow = c != 0;
    if (flow) {
      nzv = __ldg(&Tl.nbz[c]);
      bits = zset(ft, c, nzv.x, nzv.z);
    }
    const int vm1 = (kk - 1 >= kb) ? nzv.x : c, vm2 = (kk - 2 >= kb) ? nzv.y : vm1;
    for (int s = sl0; s < sl1; ++s) {
      double Fz = 0.0;
      const int n = __ldg(&T.slot_tr[s]);
      if (flow && n < ntc && (PLAIN || (__ldg(&T.trf[n]) & TR_ADV))) {
        const double *__restrict__ tr = tri + (size_t)n * G.S;
        const double tm2 = tr[vm2], tm1 = tr[vm1], t0 = tr[c], tp1 = tr[nzv.z];
        const double tu = (bits & F64_POS) ? tm2 : tp1;
        ExpCheck ec;
        ec.add(tu);
        ec.add(tm1);
        ec.add(t0);
        if (SCH == SHOC_TR_ORDER1) {
          Fz = order1_z(ft[FC_U * 32], tm1, t0);
        } else {
          bool redo = ec.bad() || (bits & F64_REF);
          Fz = face_flux64<SCH, ULT>(ft, bits, tu, tm1, t0, tm2, tp1, redo);
          if (redo) Fz = face_ref64<SCH, ULT>(ft, bits, tu, tm1, t0, tm2, tp1);
        }
      }
      sF[(s - sl0) * 32] = Fz;
    }
  }

  for (int k = k0; k < k1; ++k) {
    const int c = (col >= 0 && k >= kb) ? __ldg(&Tl.cellk[(size_t)k * Tl.ncolp + col]) : 0;
    const bool on = c != 0, st = on && staged;
    if (!__any_sync(FULL, st)) continue;
    int4 n1 = make_int4(0, 0, 0, 0), n2 = n1, nzv = n1;
    int2 me = make_int2(0, 0);
    int fl = 0;
    if (on) {
      n1 = __ldg(&Tl.nb1[c]);
      n2 = __ldg(&Tl.nb2[c]);
      nzv = __ldg(&Tl.nbz[c]);
      me = __ldg(&Tl.m2e[c]);
      fl = __ldg(&Tl.fl[c]);
    }
    // a wet east neighbour is the next lane's cell (the segments see to it; where
    // it is not, k_adv64_apart does the cell again)
    const bool ewet = (fl & FL_XP_WET) != 0;
    const bool nwet = (fl & FL_YP_WET) != 0;
    const bool below = k < ks;  // interior cell: its top face is in the water

    int bw = 0, bs = 0, bn = 0, bt = 0;
    double ydz = 0.0, dzc = 1.0;
    unsigned rng = kDivNever;
    if (on) {
      const Face2D mx = G.fx[c2];
      const double h = __ldg(&G.h1au1[c2]), u = __ldg(&F.u1[c]);
      const bool e1 = fl & CF_E1;
      bw = set_face_64<SCH>(fw, u * dtu / h, u, mx.d, mx.db, mx.df, mx.hm, mx.h0, mx.hp,
                            __ldg(&F.u1flux3d[c]), e1, ULT && e1);
    }
    if (st) {
      const Face2D my = G.fy[c2];
      const double h = __ldg(&G.h2au2[c2]), u = __ldg(&F.u2[c]);
      const bool e2 = fl & CF_E2;
      bs = set_face_64<SCH>(fs, u * dtu / h, u, my.d, my.db, my.df, my.hm, my.h0, my.hp,
                            __ldg(&F.u2flux3d[c]), e2, ULT && e2);
      if (nwet || SCH == SHOC_TR_ORDER1) {  // order1 fills the ghost cells' faces too
        const int yp = n1.w;
        const Face2D mn = G.fy[me.y];
        const double hn = nwet ? __ldg(&G.h2au2[me.y]) : 1.0, un = __ldg(&F.u2[yp]);
        const bool e2n = fl & FL_YP_E2;
        bn = set_face_64<SCH>(fn, un * dtu / hn, un, mn.d, mn.db, mn.df, mn.hm, mn.h0, mn.hp,
                              __ldg(&F.u2flux3d[yp]), e2n, ULT && e2n);
      } else {
        fn[FC_U * 32] = 0.0;
      }
      if (below)
        bt = zset(ft, nzv.z, c, nzv.w);  // the bottom face of the cell above
      else
        ft[FC_U * 32] = 0.0;
      dzc = W.dz[c];
      ydz = 1.0 / dzc;
      rng = div_range(dzc) == kDivLo && div_range(area) == kDivLo ? kDivLo : kDivNever;
    }
    const int refs = (bw | bs | bn | bt) & F64_REF;
    // vertical neighbour (bottom: the sediment ghost holds the bottom value,
    // tracers.c:827-830)
    const int vm1 = (k - 1 >= kb) ? nzv.x : c;
    // the upwind value beyond each face: one load instead of two and a choice
    const int uw = (bw & F64_POS) ? n2.x : n1.y, us = (bs & F64_POS) ? n2.z : n1.w;
    const int un = (bn & F64_POS) ? n1.z : n2.w, ut = (bt & F64_POS) ? vm1 : nzv.w;
    // the next tracer's stencil values are loaded while this one is computed
    constexpr int NV = 9;
    const int idx[NV] = {c, n1.x, n1.z, n1.w, nzv.z, uw, us, un, ut};
    double nv[NV];
    int nn = __shfl_sync(FULL, my_tr, 0), nn2 = __shfl_sync(FULL, my_tr, 1);
    auto fetch = [&](int n) {
      const double *__restrict__ p = tri + (size_t)n * G.S;
#pragma unroll
      for (int q = 0; q < NV; ++q) nv[q] = p[idx[q]];
    };
    fetch(nn);
    for (int s = sl0; s < sl1; ++s) {
      const int n = nn;
      const double t0 = nv[0], txm1 = nv[1], tym1 = nv[2], typ1 = nv[3], tp1 = nv[4];
      const double tuw = nv[5], tus = nv[6], tun = nv[7], tut = nv[8];
      if (s + 1 < sl1) {
        nn = nn2;
        nn2 = __shfl_sync(FULL, my_tr, (s + 2 - sl0) & 31);
        fetch(nn);
      }
      if (!__any_sync(FULL, st && n < ntc)) continue;  // no lane carries it
      const int tf = PLAIN ? TR_ADV : __ldg(&T.trf[n]);
      const bool adv = PLAIN || (tf & TR_ADV), hd = !PLAIN && (tf & TR_HDIFF);
      const double *__restrict__ tr = tri + (size_t)n * G.S;
      double txm2 = 0.0, txp1 = 0.0, tym2 = 0.0, typ2 = 0.0, tm1 = 0.0, tp2 = 0.0;
      if (SCH == SHOC_TR_ORDER4) {  // both values beyond each face
        txm2 = tr[n2.x];
        txp1 = tr[n1.y];
        tym2 = tr[n2.z];
        typ2 = tr[n2.w];
        tm1 = tr[vm1];
        tp2 = tr[nzv.w];
      }
      double Fxw = 0.0, Fys = 0.0, Fyn = 0.0, Fzt = 0.0;
      if (adv) {
        // (faces a lane does not have hold whatever their factors give: they
        // are not used)
        bool redo = refs != 0;
        Fxw = face_flux64<SCH, ULT>(fw, bw, tuw, txm1, t0, txm2, txp1, redo);
        Fys = face_flux64<SCH, ULT>(fs, bs, tus, tym1, t0, tym2, typ1, redo);
        Fyn = face_flux64<SCH, ULT>(fn, bn, tun, t0, typ1, tym1, typ2, redo);
        Fzt = SCH == SHOC_TR_ORDER1 ? order1_z(ft[FC_U * 32], t0, tp1)
                                    : face_flux64<SCH, ULT>(ft, bt, tut, t0, tp1, tm1, tp2, redo);
        if (SCH != SHOC_TR_ORDER1) {
          ExpCheck ec;
          ec.add(t0);
          ec.add(txm1);
          ec.add(tym1);
          ec.add(typ1);
          ec.add(tp1);
          ec.add(tuw);
          ec.add(tus);
          ec.add(tun);
          ec.add(tut);
          if (SCH == SHOC_TR_ORDER4) {
            ec.add(txm2);
            ec.add(txp1);
            ec.add(tym2);
            ec.add(typ2);
            ec.add(tm1);
            ec.add(tp2);
          }
          if (ec.bad() || redo) {
            if (k == kb && !open) sF[(s - sl0) * 32] = floor_flux64<SCH>(t0, tp1);
#pragma unroll 1
            for (int q = 0; q < 4; ++q) {  // (one call: four would cost registers)
              const bool w = q == 0, y = q == 1, z = q == 3;
              const double v = face_ref64<SCH, ULT>(
                  fw + q * FC_N * 32, w ? bw : y ? bs : z ? bt : bn,
                  w ? tuw : y ? tus : z ? tut : tun, w ? txm1 : y ? tym1 : t0,
                  (w || y) ? t0 : z ? tp1 : typ1, w ? txm2 : y ? tym2 : z ? tm1 : tym1,
                  w ? txp1 : y ? typ1 : z ? tp2 : typ2);
              if (w) Fxw = v;
              else if (y) Fys = v;
              else if (z) Fzt = v;
              else Fyn = v;
            }
          }
        }
      }
      if (hd && on) {
        // hor_diffuse (tracers.c:3654-3667): csx = dzu1 h2au1 mdx, then
        // csx u1kh (t0 - tm1) / h1au1 (the e2 analogue for y)
        Fxw -= F.dzu1[c] * G.h2au1[c2] * 1.0 * F.u1kh[c] * (t0 - txm1) / G.h1au1[c2];
        if (st) {
          Fys -= F.dzu2[c] * G.h1au2[c2] * 1.0 * F.u2kh[c] * (t0 - tym1) / G.h2au2[c2];
          if (nwet) {
            const int yp = n1.w;
            Fyn -= F.dzu2[yp] * G.h1au2[me.y] * 1.0 * F.u2kh[yp] * (typ1 - t0) / G.h2au2[me.y];
          }
        }
      }
      double Fxe = __shfl_down_sync(FULL, Fxw, 1);
      if (!st || n >= ntc) continue;
      if (!ewet)  // order1 fills the ghost cells' faces too
        Fxe = (SCH == SHOC_TR_ORDER1 && adv) ? order1_flux(F.u1flux3d[n1.y], t0, tr[n1.y]) : 0.0;
      if (SCH != SHOC_TR_ORDER1 && !nwet) Fyn = 0.0;
      // dtracer (tracers.c:888-892)
      const double dtr = (Fxe - Fxw + Fyn - Fys) * dtu;
      double val = dtr;
      if (k <= ks) {
        const double Fzb = kFloorZero64<SCH> && k == kb && !open ? floor_flux64<SCH>(t0, tp1)
                                                          : sF[(s - sl0) * 32];
        if (below) {
          sF[(s - sl0) * 32] = Fzt;
          // interior cell (tracers.c:912-925); Ds = Hn1 = 1 in z coordinates
          const double net = quot_pos(dtr, area, yarea) + (Fzt - Fzb);
          val = t0 - quot_pos(net, dzc, ydz);
          if (!((div_fast(dtr, rng) || dtr == 0.0) && (div_fast(net, rng) || net == 0.0)))
            val = t0 - (dtr / area + (Fzt - Fzb)) / dzc;
        } else {
          fzs[(size_t)n * G.ncol + col] = Fzb;
        }
      }
      tro[(size_t)n * G.S + c] = val;
    }
  }
}

// The cells of maps that do not stack: k_adv64 gave them another cell's flux for
// their east one.  A thread per (cell, tracer) forms their value again from the
// same operands.  (An east face of its own in k_adv64's loop cost every window:
// 384 x 320 x 40, 10 tracers 5.45 -> 6.25 ms for 4 steps.  Their columns on the
// general path cost 0.33 ms a step at 200 x 180 x 30, however few they were.)
__global__ void __launch_bounds__(128)
    k_adv64_apart(Geo G, Flow F, Work W, Opt O, TrSet T, SubStep ss, Tile Tl,
                  const double *__restrict__ tri, double *__restrict__ tro) {
  const double dtu = ss.dtu;
  const long long tot = (long long)Tl.napart * T.ntb;
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < tot;
       q += (long long)gridDim.x * blockDim.x) {
    const int c = Tl.apart[q % Tl.napart], n = T.slot_tr[q / Tl.napart];
    const TileCol tc = tile_column(G, W, Tl, Tl.colof[c]);
    if (!tc.act || n >= G.colntr[Tl.colof[c]]) continue;
    const int tf = T.trf[n], k = Tl.kof[c], fl = Tl.fl[c];
    const bool adv = (tf & TR_ADV) != 0, hd = (tf & TR_HDIFF) != 0;
    const int4 n1 = Tl.nb1[c], n2 = Tl.nb2[c], nzv = Tl.nbz[c];
    const int2 me = Tl.m2e[c];
    const double *tr = tri + (size_t)n * G.S;
    const double t0 = tr[c], txm1 = tr[n1.x], txp1 = tr[n1.y], tym1 = tr[n1.z], typ1 = tr[n1.w];
    double Fxw = 0.0, Fys = 0.0, Fxe = 0.0, Fyn = 0.0;
    if (adv || hd) {
      Fxw = flux_x(G, F, W, O, fl, adv, hd, c, tc.c2, tr[n2.x], txm1, t0, txp1, dtu);
      Fys = flux_y(G, F, W, O, fl, adv, hd, c, tc.c2, tr[n2.z], tym1, t0, typ1, dtu);
      Fxe = flux_x(G, F, W, O, (fl & FL_XP_E1) ? CF_E1 : 0, adv, hd, n1.y, me.x, txm1, t0, txp1,
                   tr[n2.y], dtu);
      if (fl & FL_YP_WET)
        Fyn = flux_y(G, F, W, O, (fl & FL_YP_E2) ? CF_E2 : 0, adv, hd, n1.w, me.y, tym1, t0,
                     typ1, tr[n2.w], dtu);
      else if (adv && O.trasc == SHOC_TR_ORDER1)
        Fyn = order1_flux(F.u2flux3d[n1.w], t0, typ1);
    }
    const double dtr = (Fxe - Fxw + Fyn - Fys) * dtu;
    double val = dtr;
    if (k < tc.ks) {
      double Fzb = 0.0, Fzt = 0.0;
      if (adv) {
        const double tm1 = k > tc.kb ? tr[nzv.x] : t0, tm2 = k - 1 > tc.kb ? tr[nzv.y] : tm1;
        const double tp1 = tr[nzv.z], w9c = W.w9[c], w9p = W.w9[nzv.z];
        Fzb = flux_z(F, W, O, c, W.w9[nzv.x], w9c, w9p, tm2, tm1, t0, tp1, dtu);
        Fzt = flux_z(F, W, O, nzv.z, w9c, w9p, W.w9[nzv.w], tm1, t0, tp1, tr[nzv.w], dtu);
      }
      val = t0 - (dtr / G.cellarea[tc.c2] + (Fzt - Fzb)) / W.dz[c];
    }
    tro[(size_t)n * G.S + c] = val;
  }
}

// ---------------------------------------------------------------------------
// k_vd64
//
// A block is one tile of 32 columns, deepest tiles first, the tile's
// tracer-independent arrays (cells, the LU factors and the reciprocal of the
// divisor) staged once; each warp steps its share of the tracers, a thread per
// column.  Every block of a launch has the same shared memory, of which a warp
// takes as much as the tile is deep, so one launch serves every depth unless there
// are too few tracers for that (col_launches).
//
// What bounds it: the serial chain of the Thomas sweeps (memory is 16 bytes a
// value).  The forward sweep's IEEE division was most of the chain: the
// divisor does not depend on the tracer, so k_set_dz stores its reciprocal and
// quot takes five dependent operations; and a row waited for its factors from
// L2, which a row's branch keeps the compiler from fetching ahead.  The advected
// values are copied to shared memory in one batch of asynchronous copies and
// replaced by the forward sweep's row by row; the back substitution reads them
// again (from L2), so a warp keeps one array instead of two.
// A sub-step (B200): 384 x 320 x 40, 10 tracers 0.51 ms with divisions and the
// factors read from L2, 0.37 with reciprocals, 0.23 with the factors in shared
// memory, a row without branches (a row whose quotient is not quot's to form
// marks its column, which is swept again) and the tile's cells read eight layers
// at a time; 64 x 64 x 20, 1 tracer 25 and 18 us.
// Columns whose surface crosses layer faces during the step run here too: the
// cells from the lower of the old and new surface cells up to the old one add
// to the surface balance, and the solve runs up to the new one.

constexpr int kVd64MaxWarps = 16;
// shared memory (bytes) for columns of at most nd layers: factors dzdt, cm1,
// div, 1 / div, ud double[5][nd][32], S double[nd][nw][32], cells int[nd][32]
inline size_t vd64_smem(int nd, int nw) {
  return (size_t)nd * 32 * (5 * 8 + 4) + (size_t)nd * nw * 32 * 8;
}
// what a setting of nw warps is held to (a launch takes the warps that do fit)
inline size_t vd64_tuned(int nz, int nw) { return (size_t)nz * 32 * (4 + 2 * 8 * nw); }
// Warps per block at full depth where the caller sets none: two blocks per SM
// within 160 KB of its memory, balanced rounds.  The rest is left to the L1,
// which the back substitution's values come from.  Where four blocks of four
// warps fit (22 layers), col_warps as in k_vd32; deeper, 192 x 160 x 24 (6 tracers)
// 6 warps 42.6 us, 3 45.1: 384 x 320 x 40 (10 tracers)
// 2 warps 0.23 ms, 4 (194 KB) 0.27; 200 x 180 x 30 (6 tracers) 3 warps 0.051, 6
// 0.049.  Deeper columns, where that is a single warp, take two, while two such
// blocks fit (512 x 256 x 50, 24 tracers: 1 warp 1.32 ms, 2 0.94, 3 0.88, 4 1.13);
// still deeper ones what a block has within 200 KB (448 x 300 x 60, 16 tracers: 1
// warp 1.21 ms, 2 0.91, 3 1.15, 6 0.89; 400 x 300 x 80, 12 tracers: 1 warp 1.69, 2
// 1.24, 4 0.95, 5 1.05).
inline int vd64_default_warps(int nz, int nslot, int ntile) {
  int nw = 1;
  const int b0 = col_blocks(ntile);  // (few tiles: as many warps as a block may have)
  const bool shallow = b0 > 2 && 4 * (vd64_smem(nz, 4) + 1024) <= 227 * 1024;
  const int most = shallow ? col_warps(nslot) : kVd64MaxWarps / 2;
  if (b0 > 1)
    while (nw < most && 2 * (vd64_smem(nz, nw + 1) + 1024) <= 160 * 1024) nw++;
  else
    while (nw < most && vd64_smem(nz, nw + 1) <= 200 * 1024 &&
           vd64_tuned(nz, nw + 1) <= 227 * 1024)
      nw++;
  if (nw == 1) {
    nw = 2;
    if (2 * (vd64_smem(nz, nw) + 1024) > 227 * 1024)
      while (nw < kVd64MaxWarps / 2 && vd64_smem(nz, nw + 1) <= 200 * 1024 &&
             vd64_tuned(nz, nw + 1) <= 227 * 1024)
        nw++;
  }
  const int rounds = nslot > 0 ? (nslot + nw - 1) / nw : 1;
  return nslot > 0 ? (nslot + rounds - 1) / rounds : 1;
}

// What the tracers of one column share: rows nk, nc, no of the cells s (the lower
// of the old and new surface cells), cs (new) and co (old), nl of the column;
// surf_conc's elevations and thicknesses (tracers.c:3097-3112)
struct Col64 {
  ColInfo ci;
  int nk, nc, no, nl, cbot, sed;
  double area, botz, wbot, wb, sub, osub, dz_s, dz_cs;
};

// One (column, tracer) pair: S0 (row stride sa) the column's shared memory, F0
// its factors (n1 doubles apart: dzdt, cm1, div, 1 / div, ud), C0 its cells; Fzb:
// the flux through the bottom of s.
template <bool LAST>
__device__ __forceinline__ void vd64_column(const Geo &G, const Flow &F, const Work &W,
                                            const Opt &O, const TrSet &T, const SubStep &ss,
                                            const Col64 &L, int n, const double *tr, double *to,
                                            double Fzb, double *S0, int sa, const double *F0,
                                            int n1, const int *C0, unsigned long long &nwarn,
                                            int &stat) {
  const ColInfo &ci = L.ci;
  const int nk = L.nk, nc = L.nc, no = L.no, nl = L.nl;
  const int tf = T.trf[n];
  const bool tbdy = (tf & TR_TBDY) != 0;
  const bool adv = tbdy && (tf & TR_ADV);
  const bool vdf = LAST && (tf & TR_VDIFF);
  const bool single = (ci.flags & COL_SINGLE) != 0;
  const bool solve = vdf && !single;
  // the column: advection results (advected tracers) or the old values
  const double *src = tbdy ? to : tr;
  for (int j = 0; j < nl; ++j) cp_async8(&S0[j * sa], src + C0[j * 32]);
  cp_async_commit();
  const double mn = T.mintr[n], mx = T.maxtr[n];
  to[L.sed] = tbdy ? tr[L.cbot] : tr[L.sed];  // sediment ghost (tracers.c:827-830)
  const int cell_s = ci.s, cs = ci.cs;
  const double ts_old = tr[cell_s];
  cp_async_wait<0>();

  double solp = 0.0;
  const bool clip = mn <= kClipEps;
  // row j of the forward sweep (:4185-4196) for the value a.  Without a branch,
  // so that the rows' factors are fetched ahead; bad: a row's quotient is not
  // quot's to form, and the sweep is run again with the reference's division
  bool bad = false;
  auto row_rhs = [&](int j, double a) {
    const double *f = F0 + j * 32;
    double rhs = f[0] * a;
    if (j == 0) return rhs + 0.0;
    if (j == nc) rhs = rhs - 0.0;
    return rhs - f[n1] * solp;
  };
  auto forward = [&](int j, double a) {
    const double *f = F0 + j * 32;
    const double rhs = row_rhs(j, a), y = f[3 * n1];
    bad = bad || !(div_fast(rhs, kDivLo) || rhs == 0.0) || __double2hiint(y) == 0;
    solp = quot(rhs, f[2 * n1], y);
    S0[j * sa] = solp;
  };
  double vs = ts_old;
  if (!tbdy) {
    // tracers without advection / diffusion keep their values, then diffuse
    for (int j = 0; j < nl; ++j) {
      const double a = S0[j * sa];
      to[C0[j * 32]] = a;
      if (isnan(a)) stat |= ST_NAN;
    }
    if (vdf && single) {
      const double h = L.dz_cs > O.hmin ? L.dz_cs : O.hmin;
      const double v = S0[nc * sa];
      to[cs] = v + F.dt * (0.0 - 0.0) / h;
    } else if (solve) {
#pragma unroll 4
      for (int j = 0; j <= nc; ++j) forward(j, S0[j * sa]);
    }
  } else {
    // surf_conc's balance (tracers.c:3097-3206), before the sweep replaces
    // the divergences at and above s
    double sv = 0.0;
    if (adv) {
      const double area = L.area;
      const double fcbot = -Fzb * area;
      double surftr = -fcbot;
      double wbot = L.wbot;
      const double dzs = L.sub - wbot;
      const double svol = dzs * area;
      double t0 = ts_old;
      int j = nk;
      for (; j < no; ++j) {  // cells the old surface was above
        const double wtop = G.gridz[C0[(j + 1) * 32]];
        surftr += (t0 * area * (wtop - wbot) - S0[j * sa]);
        wbot = wtop;
        t0 = tr[C0[(j + 1) * 32]];
      }
      surftr += (t0 * area * (L.osub - L.wb) - S0[j * sa]);
      for (++j; j < nl; ++j) surftr -= (S0[j * sa]);
      if (svol == 0.0 || (surftr < 0.0 && dzs <= O.hmin))
        sv = 0.0;
      else
        sv = surftr / svol;
      vs = (L.botz > 0.0 && L.dz_s < O.hmin) ? ts_old : sv;
    }
    double a_below = nk > 0 ? S0[(nk - 1) * sa] : 0.0;
#pragma unroll 4
    for (int j = 0; j < nk; ++j) {
      double a = S0[j * sa];
      // tr_bounds clip and range check (:3278-3293)
      if (clip && a < mn) a = mn;
      if (a < mn || a > mx) nwarn++;
      if (isnan(a)) stat |= ST_NAN;
      if (solve)
        forward(j, a);
      else
        to[C0[j * 32]] = a;
    }
    // tr_bounds thin-surface fix (:3250-3272); the cursor cannot move here
    if ((ci.flags & COL_THIN) && (vs < mn || vs > mx)) vs = a_below;
    if (clip && vs < mn) vs = mn;
    if (vs < mn || vs > mx) nwarn++;
    if (isnan(vs)) stat |= ST_NAN;
    for (int j = nk; j < nl; ++j) to[C0[j * 32]] = vs;
    if (vdf && single) {
      const double h = L.dz_cs > O.hmin ? L.dz_cs : O.hmin;
      to[cs] = vs + F.dt * (0.0 - 0.0) / h;
    } else if (solve) {
      for (int j = nk; j <= nc; ++j) forward(j, vs);
    }
  }
  if (solve) {
    // the value before the solve
    auto before = [&](int j) {
      if (tbdy && j >= nk) return vs;
      double a = src[C0[j * 32]];
      if (tbdy && clip && a < mn) a = mn;
      return a;
    };
    if (bad)
      for (int j = 0; j <= nc; ++j) {
        solp = row_rhs(j, before(j)) / F0[j * 32 + 2 * n1];
        S0[j * sa] = solp;
      }
    // back substitution and update (:4197-4205)
    double x = S0[nc * sa];
    double a = before(nc);
    double fin = a + (x - a) * 1.0;
    if (isnan(fin)) stat |= ST_NAN;
    double udp = F0[nc * 32 + 4 * n1];
    // the values are read kBack rows ahead of the rows they replace
    constexpr int kBack = 8;
    to[cs] = fin;
    double nx[kBack];
#pragma unroll
    for (int q = 0; q < kBack; ++q) nx[q] = before(max(nc - 1 - q, 0));
    for (int j0 = nc - 1; j0 >= 0; j0 -= kBack) {
      double av[kBack];
#pragma unroll
      for (int q = 0; q < kBack; ++q) av[q] = nx[q];
#pragma unroll
      for (int q = 0; q < kBack; ++q) nx[q] = before(max(j0 - kBack - q, 0));
#pragma unroll
      for (int q = 0; q < kBack; ++q) {
        if (j0 - q < 0) break;
        x = S0[(j0 - q) * sa] - udp * x;
        const double f = av[q] + (x - av[q]) * 1.0;
        to[C0[(j0 - q) * 32]] = f;
        if (isnan(f)) stat |= ST_NAN;
        udp = F0[(j0 - q) * 32 + 4 * n1];
      }
    }
  }
}

template <bool LAST>
__global__ void __launch_bounds__(kVd64MaxWarps * 32)
    k_vd64(Geo G, Flow F, Work W, Opt O, TrSet T, SubStep ss, Tile Tl,
           const double *__restrict__ tri, double *__restrict__ tro,
           const double *__restrict__ fzs, int smem_bytes, int tile0) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x, wy = threadIdx.y;
  const int tile = tile0 + gridDim.x - 1 - blockIdx.x;  // (the tiles are sorted by depth)
  const int col = Tl.vdcol[tile * 32 + lane];
  const TileCol tc = tile_column(G, W, Tl, col);
  const bool act = tc.act;
  const int kb = tc.kb, ks = tc.ks, cbot = tc.cbot, c2 = tc.c2;
  const ColInfo ci = tc.ci;
  // the arrays hold layers kbase .. nz-1, row r = layer - kbase
  const int nz = G.nz, kbase = __reduce_min_sync(FULL, act ? kb : nz), nd = nz - kbase;
  if (nd == 0) return;
  // warps that step tracers: what the shared memory holds at this depth
  const int nw = min((int)blockDim.y, (smem_bytes / (nd * 32) - (5 * 8 + 4)) / 8);
  const int n1 = nd * 32;  // doubles per factor
  double *const Fc = reinterpret_cast<double *>(smem);  // [5][nd][32]
  double *const Sv = Fc + 5 * n1;                        // [nd][nw][32]
  int *const colC = reinterpret_cast<int *>(Sv + nw * n1);  // [nd][32]
  const int sa = nw * 32;
  const bool single = (ci.flags & COL_SINGLE) != 0;
  Col64 L{ci, ks - kb, 0, 0, 0, cbot, 0, 1.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  int ntc = 0;
  if (act) {
    L.nc = (ci.cs == ci.s) ? L.nk : G.kof[ci.cs] - kb;
    L.no = (ci.co == ci.s) ? L.nk : G.kof[ci.co] - kb;
    L.nl = nz - kb;
    L.sed = G.zm1[cbot];
    L.area = G.cellarea[c2];
    L.botz = G.botz[c2];
    L.wbot = (ci.s == cbot) ? L.botz : G.gridz[ci.s];
    L.wb = (ci.co == cbot) ? L.botz : G.gridz[ci.co];
    L.dz_s = W.dz[ci.s];
    L.dz_cs = W.dz[ci.cs];
    const double eta = F.eta[c2], oe = F.oldeta[c2];
    L.sub = oe + ss.subeta_f * (eta - oe);
    L.osub = ss.first ? oe : oe + ss.osub_f * (eta - oe);
    ntc = G.colntr[col];
  }
  for (int kq = kbase + wy; kq < nz; kq += kStage * blockDim.y) {
    int cq[kStage];  // the cells first: one latency for all of them
#pragma unroll
    for (int i = 0; i < kStage; ++i) {
      const int k = kq + i * blockDim.y;
      cq[i] = (act && k >= kb && k < nz) ? Tl.cellk[(size_t)k * Tl.ncolp + col] : 0;
    }
#pragma unroll
    for (int i = 0; i < kStage; ++i) {
      const int k = kq + i * blockDim.y, c = cq[i], q = (k - kbase) * 32 + lane;
      if (k >= nz) break;
      colC[q] = c;
      if (LAST && c && !single && k - kb <= L.nc) {
        cp_async8(&Fc[q], &W.vd_dzdt[c]);
        cp_async8(&Fc[n1 + q], &W.vd_cm1[c]);
        cp_async8(&Fc[2 * n1 + q], &W.vd_div[c]);
        cp_async8(&Fc[3 * n1 + q], &W.vd_rdiv[c]);
        cp_async8(&Fc[4 * n1 + q], &W.vd_ud[c]);
      }
    }
  }
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  if (wy >= nw) return;

  const int row0 = act ? kb - kbase : 0;
  double *const S0 = Sv + row0 * sa + wy * 32 + lane;
  const double *const F0 = Fc + row0 * 32 + lane;
  const int *const C0 = colC + row0 * 32 + lane;
  const int ntmax = __reduce_max_sync(FULL, ntc);
  unsigned long long nwarn = 0;
  int stat = 0;
  for (int slot = wy; slot < T.nslot; slot += nw) {
    const int n = T.slot_tr[slot];
    if (n >= ntmax) continue;  // not carried in this tile
    if (n < ntc)
      vd64_column<LAST>(G, F, W, O, T, ss, L, n, tri + (size_t)n * G.S, tro + (size_t)n * G.S,
                        fzs[(size_t)n * G.ncol + col], S0, sa, F0, n1, C0, nwarn, stat);
    __syncwarp();
  }
  if (nwarn) atomicAdd(W.nwarn, nwarn);
  if (stat) atomicOr(W.status, stat);
}

}  // namespace shoc
