// shoc_tr_tile.cuh -- the FP32-mixed transport kernels of the columns whose
// surface cell stays in its layer during the step (staged columns).
//
// One sub-step is two launches:
//
//  k_adv32  advection and horizontal diffusion (advect_diffuse, tracers.c:
//           849-925): one thread per wet cell, tile by tile (columns side by
//           side), layer by layer, so a warp's cells are adjacent cells of one
//           layer and its loads coalesce.  The thread folds its cell's
//           tracer-independent face coefficients once (QUICKEST weights,
//           ULTIMATE 1/|cr|, volume flux, horizontal-diffusion factor) and
//           then loops over the advected tracers: the stencil values are
//           independent loads, the west-face flux of the next lane's cell is
//           this cell's east-face flux (shuffle), and every face a cell
//           computes for itself is rounded as its neighbour rounds it.  The
//           flux divergence and the new value are FP64.  Output, in the
//           destination tracer array (FP32): the new value of cells below
//           the surface, the horizontal flux divergence of the surface cell
//           and the cells above it; beside it, the FP32 rounding residual of
//           each of those values (value - stored, so stored + residual is the
//           FP64 value to 2^-48); the surface cell's bottom-face flux goes to
//           a per-(tracer, column) array.
//
//  k_vd32   one thread per (column, tracer): tr_bounds (tracers.c:3217-3324),
//           surf_conc's column-mass balance (:3097-3206, FP64 Neumaier), the
//           copy above the surface and, on the last sub-step, the implicit
//           vertical diffusion (implicit_vdiff_tr, :4067-4214) as an FP32
//           Thomas sweep, an FP64 residual and one FP32 correction solve,
//           with the column's FP64 mass carry (column_finish).  A block owns
//           32 neighbouring columns, the blocks in order of depth; the
//           columns' values, residuals, LU factors and FP64 thicknesses are
//           staged into shared memory by asynchronous copies.
//
// Mass carry.  Storing FP32 values loses mass at every rounding (and the
// FP32 solve conserves the column mass only to its residual).  Per (tracer,
// column) the kernels keep, in FP64, the mass the stored values owe the
// column: carry' = carry + M_exact - M_stored, where M_exact is the FP64 mass
// the sub-step computed (the FP64 advected values, the surf_conc surface
// value, tr_bounds' clipping) and M_stored the mass of what was stored.  The
// carry goes back into the column at the next sub-step as a uniform shift of
// its values (carry / (area x depth)), inside the solve's FP64 residual when
// there is a solve, so the stored values plus the carry conserve mass to
// FP64 round-off and the carry stays within a few FP32 ulps of the column
// mass.  The mass diagnostic adds it.  Columns whose surface moves during the
// step (eta != oldeta) keep their carry as it is.
//
// The cells of a column at every layer come from a static layer-by-column
// table, so no thread walks a column to find them.
#pragma once
#include "shoc_tr_stage.cuh"

namespace shoc {

// asynchronous global -> shared copies; a thread waits for its own copies
__device__ __forceinline__ void cp_async4(void *dst, const void *src) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(void *dst, const void *src) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// The column `col` of a tile kernel: whether the tile kernels handle it this
// step (k_set_dz decides, COL_STAGED), its bottom and surface layers, 2D cell
// and bottom cell.  (The layer-by-column cell table agrees with the maps:
// handle creation checks every column's layers.)
struct TileCol {
  ColInfo ci;
  int cbot, c2, kb, ks;
  bool act;
};
__device__ __forceinline__ TileCol tile_column(const Geo &G, const Work &W, const Tile &Tl,
                                               int col) {
  TileCol t;
  t.ci = {0, 0, 0, 0, 0, 0};
  t.cbot = t.c2 = t.ks = 0;
  t.kb = G.nz;
  t.act = false;
  if (col >= 0 && col < G.ncol) {
    t.ci = W.col[col];
    const int4 r = Tl.colrec[col];
    if (t.ci.flags & COL_STAGED) {
      t.act = true;
      t.cbot = r.x;
      t.c2 = r.y;
      t.kb = r.z;
      t.ks = t.ci.ks;
    }
  }
  return t;
}

namespace f32 {

// Face coefficients of one horizontal face at a cell with the given flags
// (cr = u dt / h, rounded by the caller as __fmul_rn(__fmul_rn(u, dt), 1/h)).
__device__ __forceinline__ void hface(Face &f, bool wet, bool eb, bool quick, bool ult,
                                      float cr, double U, float K, const Face2 &m) {
  if (!wet) {  // a ghost: the face carries nothing
    face_zero(f);
    return;
  }
  if (!quick && !eb) {  // Van Leer advects interior faces only
    face_zero(f);
    f.K = K;
    return;
  }
  set_face(f, quick, cr, m.d, m.Ap, m.Bp, m.Am, m.Bm, U, ult && eb, K);
}

// Vertical face at the bottom of a cell from the thicknesses of the two cells
// below it (dzm2, dzm1), the cell (dz0) and the one above (dzp1; the
// surface-layer cell maps onto itself, top != 0), and w * dtu (wv in FP32
// for the Courant number, U in FP64 for the flux); IEEE divisions, so the
// cell below folds its top face to the same bits.
__device__ __forceinline__ void zface(Face &f, bool quick, bool ult, float dzm2, float dzm1,
                                      float dz0, float dzp1, bool top, float wv, double U) {
  const float w9m = __fmul_rn(0.5f, __fadd_rn(dzm1, dzm2));
  const float w90 = __fmul_rn(0.5f, __fadd_rn(dz0, dzm1));
  const float w9p = top ? w90 : __fmul_rn(0.5f, __fadd_rn(dzp1, dz0));
  const float cz = __fdiv_rn(wv, w90);
  const float db = __fdiv_rn(2.f, __fadd_rn(w9m, w90)), df = __fdiv_rn(2.f, __fadd_rn(w90, w9p));
  set_face(f, quick, cz, __fdiv_rn(dzm1, __fadd_rn(dzm1, dz0)), __fmul_rn(db, w9m),
           __fmul_rn(db, w90), __fmul_rn(df, w90), __fmul_rn(df, w9p), U, ult, 0.f);
}

}  // namespace f32

// ---------------------------------------------------------------------------
// k_adv32
//
// What bounds it: instructions issued, compares and selections above all (ALU
// pipe), DRAM runs far below its peak.  So a cell evaluates five faces, its
// east flux always being the next lane's west flux: the cell list (Tile::wet)
// gives a run of cells that goes on beyond a warp's last lane or its tile a
// halo lane, whose west flux is used and which the next warp updates.  Of the
// two values beyond a face only the upwind one is fetched.  The vertical
// neighbours are read from warps of the same block (four layers of a tile):
// climbing a chunk of layers with the bottom flux kept, as k_adv64 does,
// needs four faces and nine values but lost that reuse (4.6 ms on the case
// below at first, 3.4 at best).  A third stage of the values' ring, and four or six
// blocks an SM, were no faster.  No function is called from the loop: one that
// took the kernel's parameters by reference put them in local memory (4.3 ms).
// 1024 x 512 x 50, 24 tracers (B200), a sub-step: 3.45 ms with six faces and
// thirteen values, 3.02 ms so; with compensations (448 x 300 x 50, 16 tracers)
// 1.17 and 1.04 ms.

// 128 threads, 5 blocks per SM (at most 102 registers a thread: 20 warps per SM
// where 256-thread blocks fit 16; measured 13.0 ms against 14.3 on stiff2048)
constexpr int kAdv32Block = 128, kAdv32MinBlocks = 5;
constexpr int kAdvValues = 11;     // stencil values of a cell and tracer
// dynamic shared memory of k_adv32: the double-buffered stencil values
constexpr size_t kAdvSmem = (size_t)2 * kAdvValues * kAdv32Block * sizeof(float);
constexpr int kMaxTracers = 256;   // tracers a launch of k_adv32 lists (a handle without
                                   // the compensated store may carry)

namespace f32 {

// The faces of k_adv32's cells.  COMP (FP32_COMP): set up in FP64 (set_face64)
template <bool QUICK, bool ULT, bool COMP>
struct Faces {
  const Geo &G;
  const Flow32 &F3;
  const Work &W;
  const Face2 *__restrict__ fx2, *__restrict__ fy2;
  double dtu;
  float fdtu;
  bool hdf;  // horizontal diffusion factors exist

  // the backward face of cell c with 2D cell c2 along x (or y): wet: c is wet
  // (else the face carries nothing), eb: an interior face
  __device__ __forceinline__ void h(Face &f, bool x, int c, int c2, bool wet, bool eb) const {
    const float K = hdf ? (x ? F3.khx[c] : F3.khy[c]) : 0.f;
    const double U = x ? F3.u1flux3d[c] : F3.u2flux3d[c];
    if constexpr (COMP) {
      // FP64 Courant number (tracers.c:730-736) and metric factors
      if (!wet) {
        face_zero(f);
      } else if (!QUICK && !eb) {  // Van Leer advects interior faces only
        face_zero(f);
        f.K = K;
      } else {
        const Face2D m = x ? G.fx[c2] : G.fy[c2];
        const double u = x ? F3.u1_64[c] : F3.u2_64[c], hh = x ? G.h1au1[c2] : G.h2au2[c2];
        set_face64(f, QUICK, u * dtu / hh, m.d, m.db * m.hm, m.db * m.h0, m.df * m.h0,
                   m.df * m.hp, U, ULT && eb, K);
      }
    } else {
      const Face2 m = x ? fx2[c2] : fy2[c2];
      const float u = x ? F3.u1[c] : F3.u2[c];
      hface(f, wet, eb, QUICK, ULT, __fmul_rn(__fmul_rn(u, fdtu), m.ih), U, K, m);
    }
  }
  // the bottom face of cell c: below it zm and zmm, above it zp
  __device__ __forceinline__ void z(Face &f, int c, int zm, int zmm, int zp) const {
    const double U = __dmul_rn(F3.w64[c], dtu);
    if constexpr (COMP) {
      const double w90 = W.w9[c];
      set_face64(f, QUICK, F3.w64[c] * dtu / (w90 * 1.0), W.w5[c], W.dbz[c] * W.w9[zm],
                 W.dbz[c] * w90, W.dfz[c] * w90, W.dfz[c] * W.w9[zp], U, ULT, 0.f);
    } else {
      // (the sediment has no thickness, the surface-layer cell maps onto itself)
      zface(f, QUICK, ULT, W.dz32[zmm], W.dz32[zm], W.dz32[c], W.dz32[zp], zp == c,
            __fmul_rn(F3.w[c], fdtu), U);
    }
  }
};

}  // namespace f32

// PLAIN: every advected tracer is advected without horizontal diffusion.
// COMP (FP32_COMP): every stencil value is read with its compensation from loi
// (face_cu); 4 blocks per SM.
template <bool QUICK, bool ULT, bool PLAIN, bool COMP>
__global__ void __launch_bounds__(kAdv32Block, COMP ? 4 : kAdv32MinBlocks)
    k_adv32(Geo G, Flow32 F3, Work W, TrSet T, SubStep ss, Tile Tl,
            const f32::Face2 *__restrict__ fx2, const f32::Face2 *__restrict__ fy2,
            const float *__restrict__ tri, float *__restrict__ tro, float *__restrict__ rso,
            double *__restrict__ fzs, int any_hd, const int16_t *__restrict__ loi) {
  using namespace f32;
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ int sTr[kMaxTracers], sTf[kMaxTracers];
  const int i = blockIdx.x * kAdv32Block + threadIdx.x;
  for (int s = threadIdx.x; s < T.ntb; s += kAdv32Block) {
    const int n = T.slot_tr[s];
    sTr[s] = n;
    sTf[s] = T.trf[n];
  }
  __syncthreads();

  // this thread's cell and its column (ntc: tracers carried by the column); st:
  // its to update (not a halo lane, not a column of the general path)
  int c = 0, col = 0, kb = G.nz, ks = 0, k = 0, c2 = 0, ntc = 0;
  bool st = false;
  if (i < Tl.nwet) {
    const int e = Tl.wet[i];
    if (e >= 0) {
      c = e & ~kSegHalo;
      col = Tl.colof[c];
      k = Tl.kof[c];
      const int4 r = Tl.colrec[col];
      const ColInfo ci = W.col[col];
      kb = r.z;
      c2 = r.y;
      ks = ci.ks;
      st = !(e & kSegHalo) && (ci.flags & COL_STAGED);
      ntc = G.colntr[col];
    }
  }
  const bool on = c != 0;
  if (!__any_sync(FULL, st)) return;
  int4 n1 = make_int4(0, 0, 0, 0), n2 = n1, nzv = n1;
  int fl = 0;
  if (on) {
    n1 = Tl.nb1[c];
    n2 = Tl.nb2[c];
    nzv = Tl.nbz[c];
    fl = Tl.fl[c];
  }
  // a wet east neighbour is the next lane's cell (the cell list sees to it)
  const bool ewet = (fl & FL_XP_WET) != 0;
  const bool zf = k <= ks, zt = k < ks;

  // tracer-independent face coefficients
  const double dtu = ss.dtu;
  const Faces<QUICK, ULT, COMP> set{G, F3, W, fx2, fy2, dtu, (float)dtu, any_hd != 0};
  Face fw, fs, fn, fzb, fzt;
  face_zero(fw);
  face_zero(fs);
  face_zero(fn);
  face_zero(fzb);
  face_zero(fzt);
  double idz = 0.0, ia = 0.0;
  if (on) set.h(fw, true, c, c2, fl & CF_WET, fl & CF_E1);
  if (st) {
    set.h(fs, false, c, c2, fl & CF_WET, fl & CF_E2);
    if (fl & FL_YP_WET) set.h(fn, false, n1.w, Tl.m2e[c].y, true, fl & FL_YP_E2);
    if (zf) set.z(fzb, c, nzv.x, nzv.y, nzv.z);
    if (zt) set.z(fzt, nzv.z, c, nzv.x, nzv.w);  // the bottom face of the cell above
    idz = 1.0 / W.dz[c];  // the FP64 thickness: the update conserves mass to FP64 round-off
    ia = 1.0 / G.cellarea[c2];
  }
  // vertical neighbours (bottom: the sediment ghost holds the bottom value,
  // tracers.c:827-830)
  const int vm1 = (k - 1 >= kb) ? nzv.x : c;
  const int vm2 = (k - 2 >= kb) ? nzv.y : vm1;
  const int ntb = T.ntb;

  // The stencil values of the next tracer are copied into this thread's slots of
  // a double buffer while the current one is computed: the cell, its west,
  // south, north, bottom and top neighbours, and the upwind value beyond each
  // face (threads without a cell, and neighbours a cell does not use, read
  // valid cells).
  constexpr int NQ = kAdvValues, B = kAdv32Block;
  const int idx[NQ] = {c,
                       n1.x,
                       n1.z,
                       n1.w,
                       vm1,
                       nzv.z,
                       (fw.bits & FB_POS) ? n2.x : n1.y,
                       (fs.bits & FB_POS) ? n2.z : n1.w,
                       (fn.bits & FB_POS) ? n1.z : n2.w,
                       (fzb.bits & FB_POS) ? vm2 : nzv.z,
                       (fzt.bits & FB_POS) ? vm1 : nzv.w};
  extern __shared__ float pf[];  // [2][NQ][kAdv32Block]
  auto issue = [&](int s, int buf) {
    const float *tr = tri + (size_t)sTr[s] * G.S;
    float *d = pf + buf * NQ * B + threadIdx.x;
#pragma unroll
    for (int q = 0; q < NQ; ++q) cp_async4(d + q * B, tr + idx[q]);
    cp_async_commit();
  };
  issue(0, 0);
  for (int s = 0; s < ntb; ++s) {
    const int n = sTr[s];
    // COMP: the stencil's compensations, in flight while the stencil values'
    // copies complete
    int16_t lq[NQ];
    if constexpr (COMP) {
      const int16_t *Lp = loi + (size_t)n * G.S;
#pragma unroll
      for (int q = 0; q < NQ; ++q) lq[q] = Lp[idx[q]];
    }
    if (s + 1 < ntb) {
      issue(s + 1, (s + 1) & 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    // tracers are ascending when columns carry different numbers of them
    if (!__any_sync(FULL, st && n < ntc)) continue;
    const int tf = PLAIN ? TR_ADV : sTf[s];
    const bool adv = PLAIN || (tf & TR_ADV), hd = !PLAIN && (tf & TR_HDIFF);
    const float *v = pf + (s & 1) * NQ * B + threadIdx.x;
    const float t0 = v[0], txm1 = v[B], tym1 = v[2 * B], typ1 = v[3 * B], tm1 = v[4 * B];
    const float tp1 = v[5 * B], tuw = v[6 * B], tus = v[7 * B], tun = v[8 * B];
    const float tub = v[9 * B], tut = v[10 * B];
    double Fxw, Fys, Fyn, Fzb = 0.0, Fzt = 0.0;
    float l0 = 0.f;
    if constexpr (COMP) {
      l0 = lo_val(lq[0]);
      const float lxm1 = lo_val(lq[1]), lym1 = lo_val(lq[2]), lyp1 = lo_val(lq[3]);
      const float lm1 = lo_val(lq[4]), lp1 = lo_val(lq[5]), luw = lo_val(lq[6]);
      const float lus = lo_val(lq[7]), lun = lo_val(lq[8]), lub = lo_val(lq[9]);
      const float lut = lo_val(lq[10]);
      Fxw = face_cu<QUICK, ULT>(fw, adv, hd, tuw, txm1, t0, luw, lxm1, l0);
      Fys = face_cu<QUICK, ULT>(fs, adv, hd, tus, tym1, t0, lus, lym1, l0);
      Fyn = face_cu<QUICK, ULT>(fn, adv, hd, tun, t0, typ1, lun, l0, lyp1);
      if (zf) Fzb = face_cu<QUICK, ULT>(fzb, adv, false, tub, tm1, t0, lub, lm1, l0);
      if (zt) Fzt = face_cu<QUICK, ULT>(fzt, adv, false, tut, t0, tp1, lut, l0, lp1);
    } else {
      Fxw = face_u<QUICK, ULT>(fw, adv, hd, tuw, txm1, t0);
      Fys = face_u<QUICK, ULT>(fs, adv, hd, tus, tym1, t0);
      Fyn = face_u<QUICK, ULT>(fn, adv, hd, tun, t0, typ1);
      if (zf) Fzb = face_u<QUICK, ULT>(fzb, adv, false, tub, tm1, t0);
      if (zt) Fzt = face_u<QUICK, ULT>(fzt, adv, false, tut, t0, tp1);
    }
    double Fxe = __shfl_down_sync(FULL, Fxw, 1);
    if (!st || n >= ntc) continue;
    if (!ewet) Fxe = 0.0;
    // FP64 flux divergence (tracers.c:888-892)
    const double dtr = ((Fxe - Fxw) + (Fyn - Fys)) * dtu;
    double a = dtr;
    if (zt) {
      const double t0d = COMP ? (double)t0 + (double)l0 : (double)t0;
      a = t0d - (dtr * ia + (Fzt - Fzb)) * idz;
    } else if (zf) {
      fzs[(size_t)n * G.ncol + col] = Fzb;
    }
    const float val = (float)a;
    const size_t o = (size_t)n * G.S + c;
    tro[o] = val;
    rso[o] = (float)(a - (double)val);
  }
}

// ---------------------------------------------------------------------------
// column_finish: the end of an FP32-mixed sub-step for one (column, tracer),
// shared by k_vd32 and the fused k_step32.

// Advected tracers' column sums from the advection: the FP64 mass of the
// advected values below the surface (sum of a dz), the FP64 horizontal
// divergence of the surface cell and the cells above it, and the surface
// cell's bottom-face flux.
struct ColSums {
  double m, dv, fzb;
};

// A0, S0: the column's values and Thomas storage from its bottom layer up, row
// stride sa; an advected tracer (tbdy) holds its advected values below the
// surface, any other tracer every layer's old value (A0 is overwritten, so is
// S0).  fac: the tridiagonal factors of row j: cm1, the reciprocal diagonals rdiv
// (eliminated from the bottom: LU) and re (from the top: UL), and dzdt or, with UD,
// the elimination factor ud of LU (0 in the bottom row).  C0, D0: cells and
// FP64 thicknesses, row stride 32; H: the water depth the carry is spread over,
// the thicknesses from the surface cell's and then the bottom up.
// RES: an advected tracer's A0 holds every layer's stored advection result
// and S0 its rounding residual (k_vd32), and the column sums cs.m and cs.dv
// are taken from them; else they come in cs (k_step32).
// carry: [ntr][ncol] (null: none).  Adds the values it flags to nwarn and
// sets bad for a NaN among what it stores.  The mass bookkeeping sums are
// FP64 sums of at most nz terms: their rounding (a few 1e-16 of the column mass, of
// either sign) is what the carry may miss per step.  The stored mass is summed from
// the bottom up, thick layers first, and keeps its rounding errors: without them
// the 24-bit values of the thin layers on top end on ties, which lean one way
// (512 x 256 x 50 stiff layers, 1000 steps: a drift of -7e-16 of the mass against 5e-17).
template <bool LAST, bool RES, bool UD, class Fac>
__device__ __forceinline__ void column_finish(const Geo &G, const Flow &F, const Work &W,
                                              const Opt &O, const TrSet &T, const SubStep &ss,
                                              const TileCol &tc, int col, int n, bool tbdy,
                                              bool adv, bool vdf, float *A0, float *S0, int sa,
                                              const Fac &fac, const int *C0, const double *D0,
                                              double H, const float *tr, float *to, double area, double ia,
                                              double idt, ColSums cs,
                                              double *carry, bool steady, long long &nwarn,
                                              bool &bad, int16_t *R0 = nullptr,
                                              const int16_t *li = nullptr,
                                              int16_t *lout = nullptr) {
  // FP32_COMP (R0, li, lout non-null): R0 keeps each row's value - stored
  // (the advection's rounding residual, or the old value's compensation) in
  // the compensation's format for the solve's residual and the final value;
  // li is the tracer's compensation on the way in, lout on the way out
  const ColInfo &ci = tc.ci;
  const int kb = tc.kb, nz = G.nz, c2 = tc.c2;
  const int nk = tc.ks - kb;  // cells below the surface cell
  const bool single = (ci.flags & COL_SINGLE) != 0;
  const bool solve = vdf && !single;
  const double mn = T.mintr[n], mx = T.maxtr[n];
  const double dzs_old = (double)W.dz32[ci.s];
  // surface value before the sub-step
  const double ts_old = (double)tr[ci.s] + (li ? lo_dec(li[ci.s], tr[ci.s]) : 0.0);
  const double dzs = D0[nk * 32];
  // FP64 mass bookkeeping per unit area: what the step computed (mxs) and
  // what is stored (mss + msc)
  double mxs = 0.0, mss = 0.0, msc = 0.0;
  long long nw = 0;
  double vs = ts_old;  // the surface value
  // tr_bounds clip and range check (:3278-3293) of the cells below the
  // surface (advected tracers); a < mn and a > mx of a float a, exactly, as
  // float compares
  const float mnf = (float)mn, mn_up = __double2float_ru(mn), mx_dn = __double2float_rd(mx);
  const bool clip = tbdy && mn <= kClipEps;
  if (RES && tbdy) {  // the divergence at and above the surface: stored + residual
    double dv = 0.0;
    for (int j = nk; j < nz - kb; ++j) dv += (double)A0[j * sa] + (double)S0[j * sa];
    cs.dv = dv;
  }
  if (!tbdy) {
    vs = (double)A0[nk * sa];
    if (li) vs += lo_dec(li[C0[nk * 32]], A0[nk * sa]);
    for (int j = nk + 1; j < nz - kb; ++j) {
      to[C0[j * 32]] = A0[j * sa];
      if (lout) lout[C0[j * 32]] = li[C0[j * 32]];
      bad |= isnan(A0[j * sa]);
    }
  }
  // one pass up the column below the surface: the computed mass (an
  // advected tracer's FP64 values are stored + residual, or come in cs.m),
  // the clip and, with a solve, the FP32 forward sweep
  float z = 0.f;  // UD: the sweep's right side, else that over the diagonal
  auto sweep = [&](int j, double dzdt, float a) {
    if constexpr (UD) {
      z = (float)dzdt * a - fac.x(j) * z;
      return z * fac.rdiv(j);
    }
    z = (fac.x(j) * a - fac.cm1(j) * z) * fac.rdiv(j);
    return z;
  };
  double m = 0.0;
  for (int j = 0; j < nk; ++j) {
    float a = A0[j * sa];
    const double dz = D0[j * 32];
    // the row's value - stored: the advection's rounding residual, or the
    // old value's compensation
    double r = 0.0;
    if (tbdy && RES) r = (double)S0[j * sa];
    else if (!tbdy && li) r = lo_dec(li[C0[j * 32]], a);
    if (!tbdy || RES) m += ((double)a + r) * dz;
    if (clip && a < mn_up) {
      mxs += ((double)mnf - ((double)a + r)) * dz;
      a = mnf;
      r = 0.0;
      A0[j * sa] = a;
    }
    if (R0) R0[j * sa] = lo_bits((float)r);
    if (tbdy) nw += (a < mn_up || a > mx_dn);
    if (solve) {
      S0[j * sa] = sweep(j, dz * idt, a);
    }
  }
  mxs += (tbdy && !RES) ? cs.m : m;
  if (tbdy) {
    const double a_below =
        nk > 0 ? (double)A0[(nk - 1) * sa] + (R0 ? (double)lo_val(R0[(nk - 1) * sa]) : 0.0)
               : 0.0;
    // surf_conc with s == co (tracers.c:3097-3206): column mass in FP64
    if (adv) {
      const double wb = (ci.s == tc.cbot) ? G.botz[c2] : G.gridz[ci.s];
      const double eta = F.eta[c2], oe = F.oldeta[c2];
      const double osub = ss.first ? oe : oe + ss.osub_f * (eta - oe);
      const double sub = oe + ss.subeta_f * (eta - oe);
      double ssum = 0.0, scomp = 0.0;
      f32::neumaier_add(ssum, scomp, __dmul_rn(cs.fzb, area));
      f32::neumaier_add(ssum, scomp, __dmul_rn(__dmul_rn(ts_old, area), osub - wb));
      f32::neumaier_add(ssum, scomp, -cs.dv);
      const double dzn = sub - wb;
      const double svol = dzn * area;
      const double st = ssum + scomp;
      const double sv = (svol == 0.0 || (st < 0.0 && dzn <= O.hmin)) ? 0.0 : st / svol;
      vs = (G.botz[c2] > 0.0 && dzs_old < O.hmin) ? ts_old : sv;
    }
    if ((ci.flags & COL_THIN) && (vs < mn || vs > mx)) vs = a_below;
    if (mn <= kClipEps && vs < mn) vs = mn;
    if (vs < mn || vs > mx) ++nw;
    bad |= isnan(vs);
    const float vs32 = (float)vs;
    const int16_t qs = lout ? lo_enc(vs, vs32) : (int16_t)0;
    for (int j = nk + 1; j < nz - kb; ++j) {
      to[C0[j * 32]] = vs32;
      if (lout) lout[C0[j * 32]] = qs;
    }
  }
  mxs += vs * dzs;
  const double carry_in = (carry && steady) ? carry[(size_t)n * G.ncol + col] : 0.0;
  // the carry goes back as a uniform shift of the column's values
  const double dl = H > 0.0 ? carry_in * ia / H : 0.0;
  if (H > 0.0) mxs += carry_in * ia;
  // stores one final value: FP32 (and, FP32_COMP, its compensation); adds
  // what is stored to the stored mass
  auto store = [&](int c, double v, double dz) {
    const float fin = (float)v;
    to[c] = fin;
    bad |= isnan(fin);
    double st = (double)fin;
    if (lout) {
      double dec;
      lout[c] = lo_round(v, fin, dec);
      st += dec;
    }
    const double t = __fma_rn(st, dz, mss);
    msc += __fma_rn(st, dz, mss - t);  // what the sum's rounding left out
    mss = t;
  };
  if (!solve) {
    // the values as they are, plus the carry's shift (tr_bounds has run)
    for (int j = 0; j < nk; ++j)
      store(C0[j * 32], (double)A0[j * sa] + (R0 ? (double)lo_val(R0[j * sa]) : 0.0) + dl,
            D0[j * 32]);
    const double h = dzs_old > O.hmin ? dzs_old : O.hmin;
    store(ci.s, (vdf && single) ? vs + dl + F.dt * (0.0 - 0.0) / h : vs + dl, dzs);
  } else {
    // the surface row of the forward sweep
    double dzdt1 = dzs * idt;
    // one pass down: the back substitution (FP32), x(j) replacing s(j), and one
    // row behind it the FP64 residual of b - A x for A = dz/dt I + the diffusion
    // operator,
    //   r(j) = dz/dt (a + dl - x) - cm1 (x(j-1) - x) - cp1 (x(j+1) - x)
    // (cp1(j) = cm1(j+1); the bottom row has no cm1 term, the top row no cp1
    // term), whose correction solve's elimination, from the top (UL), follows in
    // the same pass, its right side h(j) (UD) or h(j) / e(j) replacing a(j).
    // With UD, which FP32_COMP takes, the FP32 solves' operands are FP64 values rounded
    // once.  Else the elimination factors are FP32 products, cm1 / div and cm1 / e of
    // rounded cm1, 1 / div and 1 / e: the first solve is up to 1.2 times as far off in
    // stiff columns (RMS), the corrected one the same to three digits, as what is left is
    // cm1's own rounding; plain FP32 storage shows neither.  The residual's diagonal is the FP64
    // dz / dt, so the refined solve keeps the column mass the mass diagnostic
    // measures; cm1 is the FP32 factor's (the FP64 one, staged as well, changed
    // neither the maximum nor the RMS error over 1000 stiff2048 steps, and its
    // shared memory cost warps).  The FP64 copies of x and of the factors are
    // carried from row to row.
    float x1 = sweep(nk, dzdt1, (float)vs);  // x of row j + 1
    S0[nk * sa] = x1;
    float l1 = fac.cm1(nk), u1 = fac.x(nk);  // factors of row j + 1
    float g = 0.f, l2 = 0.f;  // of row j + 2: the elimination's right side over e, cm1
    double xd1 = (double)x1, xd2 = 0.0;
    double a1 = vs;  // the value before the solve of row j + 1
    for (int j = nk - 1; j >= 0; --j) {
      const float x = S0[j * sa] - (UD ? u1 : l1 * fac.rdiv(j)) * x1;
      S0[j * sa] = x;
      const double xd = (double)x;
      double r = dzdt1 * ((a1 + dl) - xd1) - (double)l1 * (xd - xd1);
      if (j + 1 < nk) r = r - (double)l2 * (xd2 - xd1);
      a1 = (double)A0[j * sa] + (R0 ? (double)lo_val(R0[j * sa]) : 0.0);
      const float h1 = (float)r - l2 * g;
      g = h1 * fac.re(j + 1);
      A0[(j + 1) * sa] = UD ? h1 : g;
      x1 = x;
      xd2 = xd1;
      xd1 = xd;
      l2 = l1;
      l1 = fac.cm1(j);
      u1 = fac.x(j);
      dzdt1 = D0[j * 32] * idt;
    }
    double r = dzdt1 * ((a1 + dl) - xd1);
    if (nk > 0) r = r - (double)l2 * (xd2 - xd1);
    // up again: the correction's back substitution and the update in FP64
    float d = ((float)r - l2 * g) * fac.re(0);
    store(C0[0], (double)S0[0] + (double)d, D0[0]);
    for (int j = 1; j <= nk; ++j) {
      d = UD ? (A0[j * sa] - fac.cm1(j) * d) * fac.re(j)
             : A0[j * sa] - fac.cm1(j) * fac.re(j) * d;
      store(C0[j * 32], (double)S0[j * sa] + (double)d, D0[j * 32]);
    }
  }
  if (carry && steady) carry[(size_t)n * G.ncol + col] = ((mxs - mss) - msc) * area;
  nwarn += nw;
}

// ---------------------------------------------------------------------------
// k_vd32

// k_vd32: a block is one tile of 32 columns, deepest tiles first; the tile's
// tracer-independent column arrays are staged once and each warp steps its
// share of the tracers through them.  Every block of a launch has the same shared
// memory, of which a warp takes as much as the tile is deep: the deepest tile runs
// the handle's warps per block, a shallow one more, and one launch serves every
// depth, unless there are too few tracers for that (col_launches).
//
// What bounds it: latency (shared memory and conversions in each thread's
// chains along the column) at the 8 to 16 warps an SM holds (128 registers a
// thread, and the shared memory; vd32_default_warps).  So
// - the correction solve is eliminated from the top, in the pass that forms the
//   residual: a tracer takes three passes along the column instead of four;
// - the factors are arrays of one float a lane, of which a pass reads those it
//   needs (a float4 a row made 35 shared-memory wavefronts a row of what are now
//   24), and the water depth is summed once per column;
// - the warp's lanes stay together: tracers are taken in step, those a column
//   does not carry being left out.
// Fetching the next tracer's rows into the current one's as its last pass frees
// them cost more than it hid (2.90 against 2.57 ms on the first case below).
// A sub-step (B200) with four passes, and now: 1024 x 512 x 50, 24 tracers 2.86 and
// 2.41 ms; 448 x 300 x 50, 16 tracers, FP32_COMP 0.91 and 0.70; 333 x 217 x 37, 5
// tracers 0.128 and 0.076; a batch of 56 447 columns, 60 layers, 4 to 32 tracers 0.93
// and 0.68.

constexpr int kStage = 8;  // layers a warp of a column kernel stages together
constexpr int kVd32MaxWarps = 16;
// shared memory of k_vd32 (bytes) for columns of at most nd layers:
// thicknesses double[nd][32], four factors float[nd][32], cells int[nd][32], A,
// S float[nd][nw][32] (twice with pf: the next tracer's column is staged
// while the current one is solved), with comp (FP32_COMP) R, compensations
// int16[nd][nw][32]
constexpr int kVd32Row = 8 + 4 * 4 + 4;
inline size_t vd32_smem(int nd, int nw, bool pf = false, bool comp = false) {
  return (size_t)nd * 32 * kVd32Row + (size_t)(pf ? 4 : 2) * nd * nw * 32 * 4 +
         (comp ? (size_t)nd * nw * 32 * 2 : 0);
}
// Warps per k_vd32 block at full depth where the caller sets none: the most
// blocks per SM (up to four) that leave a block three warps, else two blocks,
// within 196 KB of an SM's memory.  Filling the 227 KB takes the L1 the column's
// loads go through: 1024 x 512 x 50 (24 tracers) 4 warps 2.4 ms, 5 warps 2.6;
// 333 x 217 x 37 (5 tracers) three blocks of 3 warps 0.074 ms, of 4 0.085, two of
// 5 0.098; a batch of 60 layers (32 tracers) two of 2 warps 0.67, of 4 0.84.
// Shallow columns leave memory for any number; blocks of four warps, or of the
// tracers where they are five at most, still let one block copy its column arrays
// while others solve, and fill the 16 warps the registers allow (col_warps; the
// column kernel, FP32-mixed and FP64: 500 x 400 x 4, 16 tracers 0.186 and 0.170 ms,
// 16 and 8 warps 0.325 and 0.212; 400 x 300 x 8, 16 tracers 0.142 and 0.131, 0.223
// and 0.152; 300 x 300 x 20, 24 tracers 0.235 and 0.221, 6 and 8 warps 0.291 and 0.232).
inline int col_warps(int nslot) { return nslot <= 5 ? 5 : 4; }
// A window with few tiles has no more blocks for an SM (148 of them), and those take
// as many warps as there are tracers, up to 16 an SM: 46 x 139 x 9 (140 tiles, 24
// tracers, FP32_COMP) 12 warps 25 us, 4 45; 152 x 20 x 35 (5 tracers) 5 warps 24, 3 34.
inline int col_blocks(int ntile) {
  return ntile > 3 * 148 ? 4 : ntile > 0 ? (ntile + 147) / 148 : 1;
}
inline int vd32_default_warps(int nz, int nslot, bool comp, int ntile) {
  int nw = 1;
  const int b0 = col_blocks(ntile);
  for (int b = b0; b >= (b0 < 2 ? b0 : 2); b--) {
    nw = 1;
    const int most = b == 4 ? col_warps(nslot) : kVd32MaxWarps / b;
    while (nw < most && b * (vd32_smem(nz, nw + 1, false, comp) + 1024) <= 196 * 1024)
      nw++;
    if (nw >= 3) break;
  }
  // balanced rounds over the tracers
  const int rounds = nslot > 0 ? (nslot + nw - 1) / nw : 1;
  return nslot > 0 ? (nslot + rounds - 1) / rounds : 1;
}
// row j of a column's factors in k_vd32's shared memory (p: the column's dz/dt
// or ud at its bottom row, n: floats per factor)
struct FacSmem {
  const float *p;
  int n;
  __device__ __forceinline__ float x(int j) const { return p[j * 32]; }
  __device__ __forceinline__ float cm1(int j) const { return p[n + j * 32]; }
  __device__ __forceinline__ float rdiv(int j) const { return p[2 * n + j * 32]; }
  __device__ __forceinline__ float re(int j) const { return p[3 * n + j * 32]; }
};

// COMP: FP32_COMP, each value's 16-bit compensation read from loi and
// written to loo ([ntr][S] like the values)
template <bool LAST, bool PF, bool COMP>
__global__ void __launch_bounds__(kVd32MaxWarps * 32)
    k_vd32(Geo G, Flow F, Work W, Opt O, TrSet T, SubStep ss, Tile Tl,
           const float4 *__restrict__ lu32, const float *__restrict__ tri,
           float *__restrict__ tro, const float *__restrict__ rsi, double *__restrict__ carry,
           const double *__restrict__ fzs, const int16_t *__restrict__ loi,
           int16_t *__restrict__ loo, int smem_bytes, int tile0) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x, wy = threadIdx.y;
  const int tile = tile0 + gridDim.x - 1 - blockIdx.x;  // (the tiles are sorted by depth)
  const int col = Tl.vdcol[tile * 32 + lane];
  const TileCol tc = tile_column(G, W, Tl, col);
  const bool act = tc.act;
  const int kb = tc.kb, ks = tc.ks, cbot = tc.cbot, c2 = tc.c2;
  // the arrays hold layers kbase .. nz-1, row r = layer - kbase
  const int nz = G.nz, kbase = __reduce_min_sync(FULL, act ? kb : nz), nd = nz - kbase;
  if (nd == 0) return;
  // warps that step tracers: what the shared memory holds at this depth
  constexpr int per_row = (PF ? 4 : 2) * 4 + (COMP ? 2 : 0);
  const int nw = min((int)blockDim.y, (smem_bytes / (nd * 32) - kVd32Row) / per_row);
  double *DZ = reinterpret_cast<double *>(smem);      // [nd][32]
  float *LU = reinterpret_cast<float *>(DZ + nd * 32);  // [4][nd][32]
  int *colC = reinterpret_cast<int *>(LU + 4 * nd * 32);  // [nd][32]
  // per buffer (two with PF): A, S float [nd][nw][32]; then R (COMP)
  float *const bufs = reinterpret_cast<float *>(colC + nd * 32);
  const int sa = nw * 32;

  // the tile's tracer-independent column arrays, once for every tracer
  for (int kq = kbase + wy; kq < nz; kq += kStage * blockDim.y) {
    int cq[kStage];  // the cells first: one latency for all of them
#pragma unroll
    for (int i = 0; i < kStage; ++i) {
      const int k = kq + i * blockDim.y;
      cq[i] = (act && k >= kb && k < nz) ? Tl.cellk[(size_t)k * Tl.ncolp + col] : 0;
    }
#pragma unroll
    for (int i = 0; i < kStage; ++i) {
      const int k = kq + i * blockDim.y, c = cq[i], r = k - kbase;
      if (k >= nz) break;
      colC[r * 32 + lane] = c;
      if (LAST && c && k <= ks) {
        const float *lu = reinterpret_cast<const float *>(&lu32[c]);
#pragma unroll
        for (int q = 0; q < 4; ++q) cp_async4(&LU[(q * nd + r) * 32 + lane], lu + q);
      }
      if (c && k <= ks) cp_async8(&DZ[r * 32 + lane], &W.dz[c]);
    }
  }
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  if (wy >= nw) return;

  const int row0 = act ? kb - kbase : 0;
  const size_t off = (size_t)wy * 32 + lane + (size_t)row0 * sa;
  auto A0of = [&](int b) { return bufs + (size_t)b * 2 * nd * sa + off; };
  auto S0of = [&](int b) { return bufs + (size_t)b * 2 * nd * sa + (size_t)nd * sa + off; };
  int16_t *const R0 =
      COMP ? reinterpret_cast<int16_t *>(bufs + (size_t)(PF ? 4 : 2) * nd * sa) + off : nullptr;
  const FacSmem fac{LU + row0 * 32 + lane, nd * 32};
  const int *const C0 = colC + row0 * 32 + lane;
  const double *const D0 = DZ + row0 * 32 + lane;
  double area = 1.0, ia = 1.0, H = 0.0;
  bool steady = false;
  int ntc = 0, sed = 0;
  if (act) {
    area = G.cellarea[c2];
    ia = 1.0 / area;
    steady = F.eta[c2] == F.oldeta[c2];
    ntc = G.colntr[col];
    sed = G.zm1[cbot];
    H = D0[(ks - kb) * 32];  // the water depth
    for (int j = 0; j < ks - kb; ++j) H += D0[j * 32];
  }
  const int nl = act ? nz - kb : 0;
  // the column's values of slot s into buffer b, one batch of asynchronous
  // copies: advection results and their rounding residuals (advected tracers;
  // the residuals go to the Thomas storage until the sweep) or the old values
  // (the rest)
  auto stage = [&](int s, int b) {
    if (s < T.nslot) {
      const int n = T.slot_tr[s];
      const bool tb = (T.trf[n] & TR_TBDY) != 0;
      const float *src = (tb ? tro : tri) + (size_t)n * G.S;
      const float *rs = rsi + (size_t)n * G.S;
      float *const A0 = A0of(b), *const S0 = S0of(b);
      const int rows = n < ntc ? nl : 0;
      for (int j = 0; j < rows; ++j) {
        const int c = C0[j * 32];
        cp_async4(&A0[j * sa], src + c);
        if (tb) cp_async4(&S0[j * sa], rs + c);
      }
    }
    cp_async_commit();
  };
  // warp wy takes the tracers wy, wy + nw, ... that a column of the tile carries
  const int ntmax = __reduce_max_sync(FULL, ntc);
  auto next = [&](int s) {
    for (; s < T.nslot; s += nw)
      if (T.slot_tr[s] < ntmax) return s;
    return T.nslot;
  };
  long long nwarn = 0;
  bool bad = false;  // a NaN among the values this thread stores
  int slot = next(wy), b = 0;
  if (slot < T.nslot) stage(slot, 0);
  while (slot < T.nslot) {
    const int nxt = next(slot + nw);
    if (PF) {  // the next tracer's column is copied while this one is solved
      stage(nxt, b ^ 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    const int n = T.slot_tr[slot];
    if (n < ntc) {
      const int tf = T.trf[n];
      const bool tbdy = (tf & TR_TBDY) != 0;
      const bool adv = tbdy && (tf & TR_ADV);
      const bool vdf = LAST && (tf & TR_VDIFF);
      const float *tr = tri + (size_t)n * G.S;
      float *to = tro + (size_t)n * G.S;
      to[sed] = tbdy ? tr[cbot] : tr[sed];  // sediment ghost (tracers.c:827-830)
      const int16_t *li = COMP ? loi + (size_t)n * G.S : nullptr;
      int16_t *lo = COMP ? loo + (size_t)n * G.S : nullptr;
      if (COMP) lo[sed] = tbdy ? li[cbot] : li[sed];
      const ColSums cs{0.0, 0.0, adv ? fzs[(size_t)n * G.ncol + col] : 0.0};
      column_finish<LAST, true, COMP>(G, F, W, O, T, ss, tc, col, n, tbdy, adv, vdf, A0of(b), S0of(b),
                                sa, fac, C0, D0, H, tr, to, area, ia, 1.0 / F.dt, cs, carry,
                                steady, nwarn, bad, R0, li, lo);
    }
    __syncwarp();
    slot = nxt;
    if (PF)
      b ^= 1;
    else if (slot < T.nslot)
      stage(slot, 0);
  }
  if (bad) atomicOr(W.status, ST_NAN);
  if (nwarn) atomicAdd(W.nwarn, (unsigned long long)nwarn);
}

}  // namespace shoc
