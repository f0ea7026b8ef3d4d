// shoc_tr_gpu.cu -- host side and per-step kernels of the B200 SHOC tracer
// step (C-ABI in include/shoc_tr_gpu.h).
//
// Per step, on the handle's stream:
//   k_lateral   set_lateral_BC_tr (tracers.c:5574) into both tracer buffers,
//               and the per-step reductions cleared (k_reset where it is not run)
//   k_set_dz    one block per tile of 32 columns: set_dz (tracers.c:5731-5848), the
//               scheme work arrays w5/w9 (:561-567) and their 2/(w9+w9)
//               factors, the sub-step search (:591-668) as a min-reduction,
//               and the tracer-independent tridiagonal LU factors of
//               vert_diffuse_3d / implicit_vdiff_tr (:3841-3889, :4185-4195)
//   per sub-step:
//     k_adv32 + k_vd32 (FP32-mixed, shoc_tr_tile.cuh; or the one fused
//                 k_step32 of shoc_tr_fused.cuh, SHOC_TR_GPU_KERNELS=fused)
//                 or k_adv64 + k_vd64 (FP64, shoc_tr_tile64.cuh): advection,
//                 one thread per cell (k_adv32) or a warp per segment of
//                 columns and chunk of layers (k_adv64), then one thread per
//                 (column, tracer).  FP32-mixed: QUICKEST and Van Leer, columns
//                 whose surface cell stays in its layer
//     k_general   the other columns (thin-surface fix coupling tracers,
//                 degenerate solve range; FP32-mixed: surface crossing a layer
//                 face, other schemes), one thread per (column, tracer):
//                 column_pass
// Tracers ping-pong between two buffers; a step is captured in a CUDA graph
// once its sub-step schedule is known.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstddef>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include <sys/stat.h>
#include <unistd.h>

#include "shoc_tr_gpu.h"
#include "shoc_tr_kernels.cuh"
#include "shoc_tr_launch.h"
#include "shoc_tr_tile64.cuh"

using namespace shoc;

namespace {

constexpr int kItermax = 20;  // tracers.c:430
constexpr int kGeneralBlocks = 148 * 8;  // general-path kernel: most blocks of one launch

struct Sched {
  double dtm = 0.0;
  std::vector<SubStep> sub;
};

}  // namespace

struct shoc_tr_gpu {
  int device = 0;
  int precision = SHOC_TR_FP64;
  cudaStream_t stream = nullptr;
  int ntr = 0, S = 0, S2 = 0, nz = 0, ncol = 0, nbpt = 0;
  Geo G{};
  Flow F{};
  Work W{};
  Opt O{};
  TrSet T{};
  int nslot = 0;
  bool any_vdiff = false, any_hdiff = false;
  double dt = 0.0;
  // device allocations
  std::vector<void *> allocs;
  void *tr[2] = {nullptr, nullptr};   // double (FP64) or float (FP32-mixed)
  size_t esize = sizeof(double);
  bool comp = false;                  // SHOC_TR_FP32_COMP: 16-bit compensation beside each value
  int16_t *lo[2] = {nullptr, nullptr};  // [ntr][S] compensation of tr[0] / tr[1]
  double *xfer = nullptr;             // one tracer of FP64, for FP32 upload / download
  Flow32 F3{};
  f32::Face2 *fx2 = nullptr, *fy2 = nullptr;
  Tile tl{};                          // static tables of the column-tile kernels
  float *rnd = nullptr;               // [ntr][S] FP32 rounding residual of k_adv32's values
  double *fzs64 = nullptr;            // [ntr][ncol] surface-cell bottom-face flux
  int adv_flags = 0;                  // 1 / 2: every advected tracer without / with hdiff
  double *cols = nullptr;             // column-solve entry points: their device arrays
  int *halo_send = nullptr, *halo_recv = nullptr;  // halo exchange plan (device cell lists)
  int *colown = nullptr;              // columns counted in the sub-step minimum (null: all)
  double dmin_set = 0.0;              // sub-step minimum imposed by the caller (0: own)
  int nhalo_send = 0, nhalo_recv = 0;
  struct Preamble {                   // transport-mode flow preamble (k_faces, k_wvel)
    bool on = false, ok = false;      // enabled; the window's face lists support it
    int n1 = 0, n2 = 0;               // e1 and e2 face columns
    int2 *fc = nullptr;               // [n1 + n2] {2D cell, bottom face cell}
    double *bz = nullptr;             // [n1 + n2] the faces' floors (botzu1 / botzu2)
    double *detadt = nullptr;         // [S2] surface velocity (wtop)
  } pre;
  Fused fu{};                         // FP32-mixed: the columns' mass carry; k_step32's tiles
  bool fused = false;                 // FP32-mixed sub-steps run k_step32
  size_t fused_bytes = 0;             // its dynamic shared memory
  struct FusedTiles {                 // k_step32 tiles of width 8, 16, 32
    const int *tcol = nullptr, *tkmin = nullptr;
    int ntile = 0;
  } ftile[3];
  int fnwb_max = 0;                   // phase-B warps k_step32 may have (0: no k_step32)
  struct AdvItems {                   // k_adv64's list for a number of tracer groups
    int lmax = 0, n = 0;
    int2 *d = nullptr;
  };
  std::vector<AdvItems> adv_items;
  std::vector<int> vd_depth;          // layers of the column kernels' tiles, ascending
  std::vector<long long> vd_layers;   // of the first i of them together
  bool staged = false;                // column-tile fast path
  int cur = 0;
  int *bpt = nullptr, *bin = nullptr;
  // host mirror of the per-tracer flags
  std::vector<uint8_t> trf;
  // schedule / graph
  int probe_left = 2;
  bool have_sched = false;
  Sched sched;
  cudaGraphExec_t graph[2] = {nullptr, nullptr};
  long long graph_launches[2] = {0, 0};
  int graph_nsub = -1;
  // tiling
  int tw = 8, tw_default = 8;
  bool vd_pf = false;  // k_vd32 stages the next tracer's column during the solve
  // profiling
  bool profile = false;
  struct ProfEv {
    int part;  // 0 transport of the last sub-step, 1 advection kernel, 2 column kernel
    cudaEvent_t a, b;
  };
  std::vector<ProfEv> ev;
  double prof_ms[3] = {0.0, 0.0, 0.0};
  int prof_n[3] = {0, 0, 0};
  long long launches = 0;
  // pinned readback
  // (W.dtm_bits, W.nwarn, W.status and d_counts are one device block, so one
  // copy reads them)
  struct Readback {
    unsigned long long dtm, nwarn;
    int status, pad, counts[2];
  };
  Readback *h_rb = nullptr, *d_rb = nullptr;
  int *d_counts = nullptr;  // [0] vcs, [1] vc
  int last_status = 0;
  long long warn_total = 0;
  // pipeline of the drop-in step on host arrays (made on its first use)
  std::vector<int> slot_host;       // slot -> tracer, as T.slot_tr
  cudaStream_t s_up = nullptr, s_dn = nullptr;  // host -> device, device -> host
  cudaStream_t s_cv = nullptr;      // what an arrived tracer needs on the device
  double *xup[2] = {nullptr, nullptr};  // FP32-mixed: arriving tracers (FP64)
  cudaEvent_t ev_in[2] = {nullptr, nullptr}, ev_cv[2] = {nullptr, nullptr};
  int *h_surf = nullptr;            // page-locked surface vectors, 2 x (ncol + 1)
  std::vector<cudaEvent_t> pev;     // [0] flow sent, then per chunk: sent, stepped
  double *xout = nullptr;           // FP32-mixed: one tracer of FP64 for the way back
  bool pipe_ready = false;
  uint8_t *c3s = nullptr;           // [kItermax + 2][ncol] k_general cursors between chunks
};

namespace {

#define CK(x)                                       \
  do {                                              \
    cudaError_t e_ = (x);                           \
    if (e_ != cudaSuccess) {                        \
      fprintf(stderr, "shoc_tr_gpu: %s:%d %s\n", __FILE__, __LINE__, cudaGetErrorString(e_)); \
      return SHOC_TR_ECUDA;                         \
    }                                               \
  } while (0)

// Makes a device current for the scope of one entry point and gives the
// caller's current device back on the way out, so a host model that drives
// several devices from one thread keeps its own choice.
struct DeviceScope {
  int prev = -1;
  bool ok = false;
  explicit DeviceScope(int dev) {
    if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
    ok = cudaSetDevice(dev) == cudaSuccess;
  }
  ~DeviceScope() {
    if (prev >= 0) cudaSetDevice(prev);
  }
};

template <class T>
int dalloc(shoc_tr_gpu *h, T **p, size_t n) {
  void *q = nullptr;
  cudaError_t e = cudaMalloc(&q, (n ? n : 1) * sizeof(T));
  if (e != cudaSuccess) return SHOC_TR_ENOMEM;
  h->allocs.push_back(q);
  *p = (T *)q;
  return 0;
}

// Waits for the default stream: cudaMemset, and cudaMemcpy from pageable
// memory, may still be under way when they return, and the handle's stream
// is non-blocking.  Called after every use of them, before the handle's
// stream may read what they write.
int default_stream_done() {
  CK(cudaStreamSynchronize(cudaStreamLegacy));
  return 0;
}

template <class T>
int dupload(shoc_tr_gpu *h, T **p, const T *src, size_t n) {
  int rc = dalloc(h, p, n);
  if (rc) return rc;
  if (src && n) CK(cudaMemcpy(*p, src, n * sizeof(T), cudaMemcpyHostToDevice));
  else CK(cudaMemset(*p, 0, (n ? n : 1) * sizeof(T)));
  return 0;
}

// ---------------------------------------------------------------------------
// kernels

__device__ __forceinline__ void reset_reductions(const Work &W, int *counts) {
  *W.dtm_bits = 0x7ff0000000000000ull;  // +inf
  *W.serial_count = 0;
  counts[0] = 0;
  counts[1] = 0;
}
__global__ void k_reset(Work W, int *counts) {
  if (threadIdx.x == 0 && blockIdx.x == 0) reset_reductions(W, counts);
}

// Lateral ghosts take their interior value (set_lateral_BC_tr): written into
// both tracer buffers so the value read during every sub-step, and the value
// left in the returned array, is the start-of-step one.  la / lb (FP32_COMP):
// the buffers' compensations, copied alike.  counts (or null): also clears
// the step's reductions, which saves a launch.
template <class TR>
__global__ void k_lateral(int nbpt, const int *bpt, const int *bin, const int *slot_tr,
                          int nslot, int S, TR *tra, TR *trb, int16_t *la, int16_t *lb, Work W,
                          int *counts) {
  if (counts && threadIdx.x == 0 && blockIdx.x == 0) reset_reductions(W, counts);
  long long tot = (long long)nbpt * nslot;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < tot;
       i += (long long)gridDim.x * blockDim.x) {
    int n = slot_tr[i / nbpt], b = (int)(i % nbpt);
    size_t off = (size_t)n * S;
    TR v = tra[off + bin[b]];
    tra[off + bpt[b]] = v;
    trb[off + bpt[b]] = v;
    if (la) {
      const int16_t q = la[off + bin[b]];
      la[off + bpt[b]] = q;
      lb[off + bpt[b]] = q;
    }
  }
}

__device__ __forceinline__ void atomic_min_pos(unsigned long long *p, double v) {
  atomicMin(p, (unsigned long long)__double_as_longlong(v));
}

// The step's set-up, a block of up to kSetDzWarps warps per tile of 32 columns (lane =
// column): set_dz (tracers.c:5731-5848), the scheme work arrays w5/w9 (:561-567)
// and their 2/(w9+w9) factors, the sub-step search (:591-668) as a
// min-reduction, the column flags and the tracer-independent LU factors of
// vert_diffuse_3d / implicit_vdiff_tr (:3841-3889, :4185-4195).
//
// What bounds it: one thread per column walked its column twice through
// dependent loads (cell, face, thickness, divisions): 31 us at 64 x 64 x 20,
// 0.60 ms at 1024 x 512 x 50, however few columns there were.  Here
// only the LU recurrence is serial.  Layer j of a column (j = 0 the sediment
// cell, j = 1..nk the wet layers from the bottom up) is a function of the
// surface cells and of the layer faces around it, so the warps of the block
// share the layers: (0) cells and bottom faces into shared memory; (1) per
// layer the thicknesses, the work arrays, the sub-step search and the rows of
// the tridiagonal matrix (their divisions included); (2) one warp runs the
// recurrence div(j) = C(j) - cm1(j) cp1(j-1) / div(j-1) from shared memory;
// (3) all warps write the factors.  (In shared memory a row is 28 bytes: four
// blocks an SM at 50 layers, where a column for each value made three.)  Every
// value is the reference's expression
// on the reference's operands; the sub-step minimum does not depend on the
// order the cells are visited in.
//
// list_all: put every column the tile kernels do not handle on the
// general-path list (else only the tracer-coupled thin-surface columns).
// what: SD_* flags.  own (or null): 1 for the columns whose cells count in the
// sub-step minimum (a strip of a decomposed basin counts its own columns, not
// its halo).  Without SD_SEARCH there is no sub-step search: a step whose
// schedule is known does not read its result.
constexpr int SD_PROBE = 1;   // leave the surface vectors as they are
constexpr int SD_SEARCH = 2;  // the sub-step minimum into W.dtm_bits
constexpr int SD_F32 = 4;     // also the FP32 thickness and LU factors
constexpr int SD_WORK = 8;    // w5, w9, dbz, dfz of the tile kernels' columns
constexpr int SD_UD = 32;     // FP32_COMP: ud in place of dz / dt
constexpr int SD_LU64 = 16;   // FP64 LU factors of the tile kernels' columns
                              // (the general path's columns get all of them)
// Warps of a block: one per layer up to eight (a window of few layers has nothing
// for more: 1000 x 800 x 2, 3 tracers, FP32-mixed 0.58 ms a step with eight, 0.43
// so), and two at least, of which the second eliminates from the top.
constexpr int kSetDzWarps = 8;
inline int set_dz_warps(int nz) { return std::max(2, std::min(nz, kSetDzWarps)); }
// bytes: FP64 faces (then the diagonal eliminated from the top with SD_F32, else
// the elimination factors), rows cm1 and dz/dt (then div) and the cells of nz
// layers of 32 columns: those of the window's deepest column (300 x 200, 128 layers
// of which the columns have 20 at most, 1 tracer, FP32-mixed: 61 us a step beside the transport
// with rows for 128 layers, 27 so)
inline size_t set_dz_smem(int nd) { return (size_t)nd * 32 * (3 * 8 + 4); }

__global__ void __launch_bounds__(kSetDzWarps * 32, 4)
    k_set_dz(Geo G, Flow F, Work W, Opt O, Tile Tl, int any_vdiff, int *counts, int list_all,
             int what, const int *own, int nd) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr unsigned FULL = 0xffffffffu;
  const int nz = G.nz, lane = threadIdx.x, wy = threadIdx.y, nwarp = blockDim.y;
  // row k of each array is layer k, of which no column has one below k0
  const int k0 = nz - nd, r0 = lane - k0 * 32;
  double *const sZ = reinterpret_cast<double *>(smem) + r0;  // bottom face z, then sE
  double *const sCm = sZ + nd * 32;                          // cm1
  double *const sDv = sCm + nd * 32;                         // dz / dt, then div
  double *const sE = sZ;                                     // dz / dt, then e (SD_F32)
  int *const sC = reinterpret_cast<int *>(reinterpret_cast<double *>(smem) + 3 * nd * 32) + r0;
  __shared__ int sJa[32];        // highest layer <= jn of zero thickness
  __shared__ double sMin[kSetDzWarps];
  const int col = blockIdx.x * 32 + lane;
  const bool on = col < G.ncol;
  const int4 rec = Tl.colrec[col];  // {bottom cell, top cell, bottom layer}
  const int bot = rec.x, top = rec.y, kb = rec.z, nk = on ? nz - kb : 0;

  // (0) cells and faces; the surface before the step
  if (wy == 0) sJa[lane] = 0;
  const int sur = on ? W.nsur_t[col] : 0;
  const int sed = on ? __ldg(&G.zm1[bot]) : 0;
  for (int k = k0 + wy; k < nz; k += nwarp)
    if (on && k >= kb) {
      const int c = __ldg(&Tl.cellk[(size_t)k * Tl.ncolp + col]);
      sC[k * 32] = c;
      sZ[k * 32] = __ldg(&G.gridz[c]);
    }
  __syncthreads();

  // the column: new and old surface cells (tracers.c:5739-5755), down from the
  // top while the cell's bottom is at or above eta, at most to the sediment;
  // membership (:5778-5800): s is the lower of the two
  int jn = nk, nsur = 0, js0 = 0, js = 0, s = 0, c2 = 0;
  bool wet = false, pre_staged = false;
  double oet = 0.0, bott = 0.0, dzsed = 0.0;
  if (on) {
    const double etat = F.eta[top];
    while (jn > 0 && sZ[(kb + jn - 1) * 32] >= etat) --jn;
    nsur = jn ? sC[(kb + jn - 1) * 32] : sed;
    js0 = sur == sed ? 0 : max(0, __ldg(&G.kof[sur]) - kb + 1);
    js = js0 < jn ? js0 : jn;
    s = sur > nsur ? sur : nsur;
    c2 = __ldg(&G.m2d[s]);
    const int t2 = __ldg(&G.m2d[sur]);
    oet = F.oldeta[t2];
    bott = __ldg(&G.botz[t2]);
    dzsed = W.dz[sed];
    const double tz = F.eta[c2] < F.oldeta[c2] ? F.eta[c2] : F.oldeta[c2];
    const double bz = SHOC_TR_DRY_FRAC * O.hmin + __ldg(&G.botz[c2]);
    wet = (tz > bz && js > 0);
    pre_staged = O.tiled && wet && (O.cross || (s == sur && s == nsur));
  }
  // thickness of layer j (:5824-5846): from the old surface down to the
  // bottom, the layers above the old surface copy the old surface cell's
  // (with the old surface in the sediment, every layer copies the sediment's)
  auto dzof = [&](int j) -> double {
    const int jj = j < js0 ? j : js0;
    if (jj == 0) return dzsed;
    const double tp = (jj == js0) ? oet : sZ[(kb + jj) * 32];
    return tp - ((jj > 1) ? sZ[(kb + jj - 1) * 32] : bott);
  };
  const bool quick = O.trasc == SHOC_TR_QUICKEST;
  const double dt = F.dt;
  // w5, w9 and their factors of layer j (:530-567)
  auto work_arrays = [&](int j, int cc) {
    const double dzc = dzof(j), dzm = dzof(j - 1);
    const double w9c = 0.5 * (dzc + dzm);
    const double w9m = j >= 2 ? 0.5 * (dzm + dzof(j - 2)) : 0.0;
    const double w9p = j < nk ? 0.5 * (dzof(j + 1) + dzc) : w9c;
    if (quick || O.trasc == SHOC_TR_ORDER2) W.w5[cc] = dzm / (dzm + dzc);
    W.w9[cc] = w9c;
    W.dbz[cc] = 2.0 / (w9m + w9c);
    W.dfz[cc] = 2.0 / (w9c + w9p);
  };

  // (1) every layer
  double dtmin = __longlong_as_double(0x7ff0000000000000ll);
  const bool search = (what & SD_SEARCH) && O.substep != 0 && wet && (!own || own[col]);
  const bool all_work = (what & SD_WORK) || !pre_staged;
  for (int k = nz - 1 - wy; k >= k0; k -= nwarp) {
    if (!on || k < kb) continue;
    const int j = k - kb + 1, cc = sC[k * 32];
    const double dzc = dzof(j), dzm = dzof(j - 1);
    W.dz[cc] = dzc;
    if (what & SD_F32) W.dz32[cc] = (float)dzc;
    if (all_work) work_arrays(j, cc);
    if (j <= jn && !dzc) atomicMax(&sJa[lane], j);
    if (any_vdiff) {  // rows of the implicit solve (:3841-3889)
      sDv[k * 32] = dzc / dt;
      sCm[k * 32] = -__ldg(&F.Kz[cc]) / (0.5 * (dzm + dzc));
    }
    if (search && j <= js) {
      const int xp = __ldg(&G.xp1[cc]), yp = __ldg(&G.yp1[cc]);
      double d4 = 0.5 * (__ldg(&F.u1[cc]) + __ldg(&F.u1[xp]));
      if (fabs(d4) < kMinVal) d4 = kMinVal;
      const double d1 = kSF * fabs(__ldg(&G.h1acell[c2]) / d4);
      if (d1 < dtmin) dtmin = d1;
      d4 = 0.5 * (__ldg(&F.u2[cc]) + __ldg(&F.u2[yp]));
      if (fabs(d4) < kMinVal) d4 = kMinVal;
      const double d2 = kSF * fabs(__ldg(&G.h2acell[c2]) / d4);
      if (d2 < dtmin) dtmin = d2;
      if (j != js) {
        d4 = 0.5 * (__ldg(&F.w[cc]) + __ldg(&F.w[j < nk ? sC[(k + 1) * 32] : cc]));
        if (fabs(d4) < kMinVal) d4 = kMinVal;
        const double d3 = kSF * fabs(dzc * 1.0 / d4);
        if (d3 > 0.0 && d3 < dtmin) dtmin = d3;
      }
    }
  }
  // what the flags need, before the faces' shared memory is used again
  const double dz_js0 = on ? dzof(js0) : 0.0;
  const double dz_jn = on ? dzof(jn) : 0.0, dz_jn1 = (on && jn > 0) ? dzof(jn - 1) : 0.0;
  for (int o = 16; o > 0; o >>= 1) dtmin = fmin(dtmin, __shfl_xor_sync(FULL, dtmin, o));
  if (lane == 0) sMin[wy] = dtmin;
  __syncthreads();

  // the faces are done with: the second elimination's rows take their place
  if ((what & SD_F32) && any_vdiff) {
    for (int k = k0 + wy; k < nz; k += nwarp)
      if (on && k >= kb) sE[k * 32] = sDv[k * 32];
    __syncthreads();
  }

  // (2) flags and the solve's range, in every warp alike; warp 0 runs the LU
  int flags = 0, cbs = 0, jb = 0, stat = 0;
  bool solve = false;
  if (on && wet) {
    flags |= COL_WET;
    // tr_bounds thin-surface test (:3250-3252)
    if (js > 1 && dz_js0 < O.hmin) {
      flags |= COL_THIN;
      if (s != top) flags |= COL_SERIAL;
    }
    if (jn <= 1 || !dz_jn1) {
      flags |= COL_SINGLE;
    } else if (any_vdiff && !dz_jn) {
      // zero-thickness surface cell: the reference solves over an empty
      // range and reads stale work memory; report instead of guessing
      flags |= COL_NOSOLVE;
      stat |= ST_GEOM;
    } else if (any_vdiff) {
      jb = sJa[lane] + 1;  // bottom of the solve
      cbs = sC[(kb + jb - 1) * 32];
      solve = true;
    }
  } else if (on && col == G.v2col) {
    stat |= ST_LASTDRY;
  }
  ColInfo ci;
  ci.s = wet ? s : 0;
  ci.co = sur;
  ci.cs = nsur;
  ci.cbs = cbs;
  ci.flags = flags;
  ci.ks = kb + js - 1;
  const bool staged = on && O.tiled && staged_column(ci, bot, O.cross != 0);
  if (staged) ci.flags |= COL_STAGED;
  if (wy == 0) {
    if (solve) {
      // LU (:4185-4195), bottom up from the lowest layer of the solve; the
      // upper diagonal of a row is the lower one of the row above it
      int k = kb + jb - 1;
      double bp1 = sCm[(k + 1) * 32];
      double div = sDv[k * 32] - bp1;
      sCm[k * 32] = 0.0;
      sDv[k * 32] = div;
      const int kt = kb + jn - 1;
#pragma unroll 2
      for (++k; k <= kt; ++k) {
        const double cm1 = sCm[k * 32], cp1 = k < kt ? sCm[(k + 1) * 32] : 0.0;
        double C = sDv[k * 32] - cm1;
        if (k < kt) C = C - cp1;
        const double ud = bp1 / div;
        div = C - cm1 * ud;
        if (div == 0.0) stat |= ST_PIVOT;
        sDv[k * 32] = div;
        if (!(what & SD_F32)) sZ[k * 32] = ud;
        bp1 = cp1;
      }
    }
    if (stat) atomicOr(W.status, stat);
  }
  if (wy == 1 && solve && (what & SD_F32)) {
    // the same matrix eliminated from the top (the FP32-mixed correction
    // solve): e(j) = C(j) - cm1(j+1) cm1(j+1) / e(j+1)
    const int kt = kb + jn - 1, kl = kb + jb - 1;
    double up = sCm[kt * 32], e = sE[kt * 32] - up;
    sE[kt * 32] = e;
    for (int k = kt - 1; k >= kl; --k) {
      const double cm1 = k > kl ? sCm[k * 32] : 0.0;
      e = (sE[k * 32] - cm1 - up) - up * (up / e);
      sE[k * 32] = e;
      up = cm1;
    }
  }
  if (wy == 0) {
    if (on) {
      if (!(what & SD_PROBE)) {
        W.sur_t[col] = sur;
        W.nsur_t[col] = nsur;
      }
      W.col[col] = ci;
      if ((flags & COL_SERIAL) || (list_all && !staged)) {
        const int i = atomicAdd(W.serial_count, 1);
        W.serial_list[i] = col;
      }
    }
    const int wc = __reduce_add_sync(FULL, (on && wet) ? 1 : 0);
    const int wn = __reduce_add_sync(FULL, (on && wet) ? js : 0);
    if (lane == 0) {
      if (wc) atomicAdd(&counts[0], wc);
      if (wn) atomicAdd(&counts[1], wn);
      double v = sMin[0];
      for (int i = 1; i < nwarp; ++i) v = fmin(v, sMin[i]);
      if (v < __longlong_as_double(0x7ff0000000000000ll)) atomic_min_pos(W.dtm_bits, v);
    }
  }
  __syncthreads();

  // (3) the factors (and the work arrays of a column the tile kernels turned
  // out not to handle, whose faces may be overwritten: from W.dz)
  const bool lu64 = (what & SD_LU64) || !staged;
  const bool late = on && pre_staged && !staged && !(what & SD_WORK);
  if (!solve && !late) return;
  for (int k = k0 + wy; k < nz; k += nwarp) {
    if (k < kb) continue;
    const int j = k - kb + 1, cc = sC[k * 32];
    const double dzc = W.dz[cc];
    if (solve && j >= jb && j <= jn) {
      const double cm1 = sCm[k * 32], div = sDv[k * 32];
      // the elimination factor, as the recurrence formed it (cm1 is the upper
      // diagonal of the row below); where the second elimination has the faces'
      // place it is formed again
      double ud = 0.0;
      if (j > jb && (lu64 || (what & SD_UD)))
        ud = (what & SD_F32) ? cm1 / sDv[(k - 1) * 32] : sZ[k * 32];
      const double dzdt = dzc / dt;
      if (lu64) {
        W.vd_cm1[cc] = cm1;
        W.vd_div[cc] = div;
        W.vd_ud[cc] = ud;
        W.vd_dzdt[cc] = dzdt;
        if (what & SD_LU64) W.vd_rdiv[cc] = div_range(div) == kDivLo ? 1.0 / div : 0.0;
      }
      if (what & SD_F32)
        W.lu32[cc] = make_float4((float)((what & SD_UD) ? ud : dzdt), (float)cm1,
                                 (float)(1.0 / div), (float)(1.0 / sE[k * 32]));
    }
    if (late) {
      const double dzm = j > 1 ? W.dz[sC[(k - 1) * 32]] : dzsed;
      const double w9c = 0.5 * (dzc + dzm);
      const double dzmm = j > 2 ? W.dz[sC[(k - 2) * 32]] : dzsed;
      const double w9m = j >= 2 ? 0.5 * (dzm + dzmm) : 0.0;
      const double w9p = j < nk ? 0.5 * (W.dz[sC[(k + 1) * 32]] + dzc) : w9c;
      if (quick || O.trasc == SHOC_TR_ORDER2) W.w5[cc] = dzm / (dzm + dzc);
      W.w9[cc] = w9c;
      W.dbz[cc] = 2.0 / (w9m + w9c);
      W.dfz[cc] = 2.0 / (w9c + w9p);
    }
  }
}

// The general path: the columns the tile kernels do not handle, one thread per
// (listed column, tracer), a warp holding 32 listed columns of one tracer (the
// list keeps neighbouring columns together, so most of a warp's loads
// coalesce).  Only where tr_bounds' thin-surface cursor can move between
// tracers (COL_SERIAL) one thread steps a column's tracers in tbdy order, as
// the reference loops.  One thread per column for every column left the chip
// idle: at 200 x 180 x 30 with 6 tracers (every column listed) a sub-step took
// 2.52 ms, at 192 x 160 x 24 with 800 listed columns 0.69 ms.
// When the tracers go through in chunks of slots (the drop-in step's
// pipeline), c3s holds each listed column's cursor state between the chunks
// of one sub-step: read when c3_load, written back always.  lo_out
// (FP32_COMP): these columns step their FP32 values as stored, and their
// compensations, from the sediment ghost to the top cell, are set to 0.
constexpr int kGeneralThreads = 128;
template <bool LAST, class TR>
__global__ void __launch_bounds__(kGeneralThreads)
    k_general(Geo G, Flow F, Work W, Opt O, TrSet T, SubStep ss, Tile Tl,
              const TR *__restrict__ tr_in, TR *__restrict__ tr_out, uint8_t *__restrict__ c3s,
              int c3_load, int16_t *__restrict__ lo_out = nullptr) {
  const int cnt = *W.serial_count;
  const int cntp = (cnt + 31) & ~31;
  const long long tot = (long long)cntp * T.nslot;
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < tot;
       q += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(q % cntp);
    int sl = (int)(q / cntp);
    if (i >= cnt) continue;
    const int col = W.serial_list[i];
    const bool coupled = (W.col[col].flags & COL_SERIAL) != 0;
    if (coupled && sl > 0) continue;
    const int sl1 = coupled ? T.nslot : sl + 1;
    LocalSol sol;
    bool c3 = (coupled && c3s && c3_load) ? c3s[i] != 0 : false;
    unsigned long long warn = 0;
    int stat = 0;
    for (; sl < sl1; ++sl) {
      const int n = T.slot_tr[sl];
      if (n >= G.colntr[col]) continue;  // not carried in this column
      column_pass<LAST>(G, F, W, O, T, ss, Tl, tr_in + (size_t)n * G.S,
                        tr_out + (size_t)n * G.S, col, n, sol, c3, warn, stat);
      if (lo_out) {
        int16_t *lo = lo_out + (size_t)n * G.S;
        int c = G.zm1[G.col_bot[col]];
        lo[c] = 0;
        do {
          c = G.zp1[c];
          lo[c] = 0;
        } while (c != G.col_top[col]);
      }
    }
    if (coupled && c3s) c3s[i] = c3 ? 1 : 0;
    if (warn) atomicAdd(W.nwarn, warn);
    if (stat) atomicOr(W.status, stat);
  }
}

// Compensated (Neumaier) FP64 mass sum per tracer: sum of tr * dz * area
// over each column from its current surface cell (nsur_t, top at eta) down
// to the bottom (botz), the water the column holds now.  One thread per
// (column, tracer); block partials are summed on the host.
__device__ __forceinline__ void neumaier(double &s, double &comp, double v) {
  double u = s + v;
  comp += (fabs(s) >= fabs(v)) ? (s - u) + v : (v - u) + s;
  s = u;
}

// ---------------------------------------------------------------------------
// Transport-mode flow preamble (transport_step, model/hd/tracers/
// transport.c:436-462): what SHOC's transport mode computes from the
// velocities and the surface before the tracer step, on the device.  A z-level
// window, linear free surface (wtop = detadt), no point sources (waterss = 0),
// conserve = CONS_W, mdx = mdy = 1 and no one-cell-deep face list (the
// momentum step builds that list; transport mode does not run it).

// set_dz_at_u1 / set_dz_at_u2 (model/hd/momentum/vel3d.c:720-853, :2718-2850,
// z coordinates) and set_flux_3d (vel3d.c:4041-4175, VEL3D) of one face
// column per thread, e1 faces first: the face's surface is the higher of the
// two elevations beside it (at least the face's floor botzu), its surface cell
// the first cell down from the surface layer whose bottom is at or below it,
// its thicknesses from there to the bottom face cell (the layers above copy
// the surface cell's), the volume flux u dzu h2au1 (h1au2) at and below the
// surface and zero above.  The arrays start zeroed (the reference's memsets).
// fc: {2D cell, bottom face cell} per face column, bz: its floor.
//
// What bounds both kernels of the preamble: the loads' latency down a column.
// kPreBatch cells at a time are found, their values loaded together and then
// worked through in order.  200 x 180 x 30: k_faces 24.1 us, k_wvel 17.8 us; a
// layer at a time, with stores no load may pass, 31.0 and 23.7.
constexpr int kPreBatch = 8;
__global__ void k_faces(Geo G, Flow F, int n1, int n, const int2 *fc, const double *bz,
                        double *dzu1, double *dzu2, double *f1, double *f2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const bool e1 = i < n1;
  const int2 col = __ldg(&fc[i]);
  const int c2 = col.x, cb = col.y;
  const int nb = __ldg(e1 ? &G.xm1[c2] : &G.ym1[c2]);
  const double *u = e1 ? F.u1 : F.u2;
  const double hf = __ldg(e1 ? &G.h2au1[c2] : &G.h1au2[c2]);
  double *dzu = e1 ? dzu1 : dzu2, *flux = e1 ? f1 : f2;
  const double floor = __ldg(&bz[i]), ec = __ldg(&F.eta[c2]), en = __ldg(&F.eta[nb]);
  double top = ec > en ? ec : en;
  top = top > floor ? top : floor;
  int c = c2, zm = __ldg(&G.zm1[c]);
  while (c != zm && __ldg(&G.gridz[c]) > top) {
    c = zm;
    zm = __ldg(&G.zm1[c]);
  }
  const int sur = c;
  double t = top, ds = 0.0;
  while (c != cb) {
    int q[kPreBatch];
    double g[kPreBatch], v[kPreBatch];
#pragma unroll
    for (int b = 0; b < kPreBatch; b++) {
      q[b] = c;
      if (c != cb) c = __ldg(&G.zm1[c]);
    }
#pragma unroll
    for (int b = 0; b < kPreBatch; b++) {
      g[b] = __ldg(&G.gridz[q[b]]);
      v[b] = __ldg(&u[q[b]]);
    }
#pragma unroll
    for (int b = 0; b < kPreBatch; b++) {
      if (q[b] == cb) break;
      const double d = t - g[b];
      if (q[b] == sur) ds = d;
      dzu[q[b]] = d;
      flux[q[b]] = v[b] * d * hf;
      t = g[b];
    }
  }
  {
    const double d = t - floor;
    if (cb == sur) ds = d;
    dzu[cb] = d;
    flux[cb] = __ldg(&u[cb]) * d * hf;
  }
  c = sur;
  while (c != c2) {
    c = __ldg(&G.zp1[c]);
    dzu[c] = ds;
  }
}

// vel_w_update (vel3d.c:4609-4760, z coordinates, CONS_W) of one water column
// per thread, before k_set_dz: the column's old surface cell (the previous
// step's new one) and new surface cell, and whether the column is processed,
// as set_dz decides them (tracers.c:5739-5800); then w from continuity from
// the bottom (wbot = 0) up to the old surface, wtop = detadt in the cells the
// surface moved through, and set_w_dry (vel3d.c:5116-5135): wtop in every
// cell above the new surface cell, in every column.  w starts zeroed (the
// reference's memset).
__global__ void k_wvel(Geo G, Flow F, Work W, Opt O, Tile Tl, const double *detadt, double *w) {
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= G.ncol) return;
  const int4 rec = __ldg(&Tl.colrec[col]);  // {bottom cell, top cell, bottom layer}
  const int bot = rec.x, top = rec.y;
  const int sur = __ldg(&W.nsur_t[col]);
  int nsur = top, zm = __ldg(&G.zm1[nsur]);
  const double etat = __ldg(&F.eta[top]);
  while (nsur != zm && __ldg(&G.gridz[nsur]) >= etat) {
    nsur = zm;
    zm = __ldg(&G.zm1[nsur]);
  }
  const int s = sur > nsur ? sur : nsur;
  const int c2 = __ldg(&G.m2d[s]);
  const double en = __ldg(&F.eta[c2]), eo = __ldg(&F.oldeta[c2]);
  const double tz = en < eo ? en : eo;
  const double bz = SHOC_TR_DRY_FRAC * O.hmin + __ldg(&G.botz[c2]);
  if (tz > bz && s != __ldg(&G.zm1[s])) {
    const int cs = __ldg(&G.m2d[bot]);
    const double area = __ldg(&G.cellarea[cs]);
    int c = bot;
    const double wb = 0.0;  // wbot (vel_w_bounds, z coordinates)
    w[c] = wb;
    double fcbot = wb * area;
    for (int k = rec.z; c > sur; k += kPreBatch) {
      int q[kPreBatch + 1];
      double a[kPreBatch], ax[kPreBatch], b[kPreBatch], by[kPreBatch];
#pragma unroll
      for (int j = 0; j <= kPreBatch; j++)
        q[j] = k + j < G.nz ? __ldg(&Tl.cellk[(size_t)(k + j) * Tl.ncolp + col]) : top;
#pragma unroll
      for (int j = 0; j < kPreBatch; j++) {
        const int xp = __ldg(&G.xp1[q[j]]), yp = __ldg(&G.yp1[q[j]]);
        a[j] = __ldg(&F.u1flux3d[q[j]]);
        ax[j] = __ldg(&F.u1flux3d[xp]);
        b[j] = __ldg(&F.u2flux3d[q[j]]);
        by[j] = __ldg(&F.u2flux3d[yp]);
      }
#pragma unroll
      for (int j = 0; j < kPreBatch; j++) {
        if (!(c > sur)) break;
        const double fctop = fcbot + a[j] - ax[j] + b[j] - by[j] + 0.0;  // + waterss
        w[q[j + 1]] = fctop / area;
        fcbot = fctop;
        c = q[j + 1];
      }
    }
    while (c > nsur) {
      const int zp = __ldg(&G.zp1[c]);
      w[zp] = __ldg(&detadt[cs]);  // wtop (vel_w_bounds, linear surface)
      c = zp;
    }
  }
  // set_w_dry
  const int cs = __ldg(&G.m2d[nsur]);
  int c = nsur, zp = __ldg(&G.zp1[c]);
  while (c != zp) {
    w[zp] = __ldg(&detadt[cs]);
    c = zp;
    zp = __ldg(&G.zp1[c]);
  }
}
// the preamble's arrays start zeroed (the reference's memsets)
__global__ void k_zero5(double *a, double *b, double *c, double *d, double *e, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    a[i] = b[i] = c[i] = d[i] = e[i] = 0.0;
}

__global__ void k_to_f32(const double *a, float *b, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    b[i] = (float)a[i];
}
// one uploaded tracer into both ping-pong buffers (and, SHOC_TR_FP32_COMP,
// the compensation of both: lb / lc non-null)
__global__ void k_to_f32x2(const double *a, float *b, float *c, size_t n, int16_t *lb = nullptr,
                           int16_t *lc = nullptr) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const float v = (float)a[i];
    b[i] = v;
    c[i] = v;
    if (lb) {
      const int16_t q = lo_enc(a[i], v);
      lb[i] = q;
      lc[i] = q;
    }
  }
}
// a tracer back to FP64 (with its compensation where l is non-null)
__global__ void k_to_f64(const float *a, double *b, size_t n, const int16_t *l = nullptr) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    b[i] = l ? (double)a[i] + lo_dec(l[i], a[i]) : (double)a[i];
}
// K = dzu h2au1 u1kh / h1au1 (e1) or dzu2 h1au2 u2kh / h2au2 (e2): the
// tracer-independent factor of hor_diffuse (tracers.c:3660-3666)
__global__ void k_khfac(Geo G, Flow F, float *khx, float *khy) {
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < G.S; c += gridDim.x * blockDim.x) {
    if (!(G.cflag[c] & CF_WET)) continue;
    int c2 = G.m2d[c];
    khx[c] = (float)(F.dzu1[c] * G.h2au1[c2] * F.u1kh[c] / G.h1au1[c2]);
    khy[c] = (float)(F.dzu2[c] * G.h1au2[c2] * F.u2kh[c] / G.h2au2[c2]);
  }
}

// carry (FP32-mixed path, else null): [ntr][ncol] mass the stored
// values owe each column, part of the state's mass.
// colreg (or null): the region of each column; only region `reg` is summed.
template <class TR>
__global__ void k_mass(Geo G, Flow F, Work W, const TR *tr, const double *carry, double *out,
                       const int *colreg = nullptr, int reg = 0, const int16_t *lo = nullptr) {
  const int n = blockIdx.y;
  const TR *t = tr + (size_t)n * G.S;
  const int16_t *l = lo ? lo + (size_t)n * G.S : nullptr;  // compensation (FP32_COMP)
  double s = 0.0, comp = 0.0;
  for (int col = blockIdx.x * blockDim.x + threadIdx.x; col < G.ncol;
       col += gridDim.x * blockDim.x) {
    if (colreg && colreg[col] != reg) continue;
    const int top = G.col_top[col], bot = G.col_bot[col];
    int c = W.nsur_t[col];
    if (n >= G.colntr[col]) continue;  // tracer not carried in this column
    if (carry) neumaier(s, comp, carry[(size_t)n * G.ncol + col]);
    if (c == G.zm1[c]) continue;  // surface below the bottom: dry
    const double area = G.cellarea[top];
    double tz = F.eta[top];
    for (int it = 0; it <= G.nz; ++it) {
      double bz = (c == bot) ? G.botz[top] : G.gridz[c];
      double h = tz - bz;
      if (h > 0.0) {
        const double v = l ? (double)t[c] + lo_dec(l[c], (float)t[c]) : (double)t[c];
        neumaier(s, comp, v * h * area);
      }
      if (c == bot) break;
      tz = bz;
      c = G.zm1[c];
    }
  }
  s += comp;
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  __shared__ double part[32];
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double b = 0.0, bc = 0.0;
    for (int i = 0; i < (int)(blockDim.x >> 5); i++) neumaier(b, bc, part[i]);
    out[(size_t)n * gridDim.x + blockIdx.x] = b + bc;
  }
}

// Differences between the tracers of two handles of one window: one thread
// per (column, tracer) over the column's wet cells (bottom to top layer), for
// the tracers both handles carry in the column.  Per (region, tracer): the
// largest |a - b| and |b| (atomicMax on the bits of a non-negative double,
// which order as unsigned integers) and the sums of (a - b)^2 and b^2.
template <class TA, class TB>
__global__ void k_compare(Geo G, Tile Tl, const int *colntr_b, const TA *ta, const TB *tb,
                          const int *region, int nreg, unsigned long long *maxabs,
                          unsigned long long *maxref, double *ssd, double *ssr,
                          const int16_t *la, const int16_t *lb) {
  const int n = blockIdx.y;
  for (int col = blockIdx.x * blockDim.x + threadIdx.x; col < G.ncol;
       col += gridDim.x * blockDim.x) {
    if (n >= G.colntr[col] || n >= colntr_b[col]) continue;
    const int r = region ? region[col] : 0;
    if (r < 0 || r >= nreg) continue;
    double ma = 0.0, mr = 0.0, sd = 0.0, sr = 0.0;
    for (int k = G.col_kb[col]; k < G.nz; ++k) {
      const int c = Tl.cellk[(size_t)k * Tl.ncolp + col];
      if (!c) continue;
      const size_t i = (size_t)n * G.S + c;
      double a = (double)ta[i], b = (double)tb[i];
      if (la) a += lo_dec(la[i], (float)ta[i]);  // FP32_COMP: value + compensation
      if (lb) b += lo_dec(lb[i], (float)tb[i]);
      const double d = a - b;
      ma = fmax(ma, fabs(d));
      mr = fmax(mr, fabs(b));
      sd += d * d;
      sr += b * b;
    }
    const size_t o = (size_t)r * gridDim.y + n;
    atomicMax(&maxabs[o], (unsigned long long)__double_as_longlong(ma));
    atomicMax(&maxref[o], (unsigned long long)__double_as_longlong(mr));
    atomicAdd(&ssd[o], sd);
    atomicAdd(&ssr[o], sr);
  }
}

// ---------------------------------------------------------------------------
// The other per-column tridiagonal solves, one thread per water column (from
// its bottom cell up to its surface cell, the handle's current nsur_t; a
// column whose surface is its sediment cell is dry).  The arithmetic is the
// reference's, operation by operation (this file is compiled without FMA
// contraction, with IEEE division), so the results are bitwise its own.  The
// reference keeps the rows in layer-indexed work vectors; here every array is
// indexed by SHOC cell (a cell carries the row of its layer).

// tridiagonal (model/hd/closure/MY2-5.c:499-536): the closures' solve
__global__ void k_tridiag(Geo G, Work W, const double *C, const double *Cm1, const double *Cp1,
                          const double *rhs, double *var, double *sol, double *ud,
                          double minvar) {
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= G.ncol) return;
  const int cs = W.nsur_t[col], cb = G.col_bot[col];
  if (cs == G.zm1[cs]) return;
  int stat = 0;
  double div = C[cb];
  sol[cb] = rhs[cb] / div;
  int c = cb;
  for (int it = 0; c != cs && it < G.nz; ++it) {
    const int cn = G.zp1[c];
    ud[cn] = Cp1[c] / div;
    div = C[cn] - Cm1[cn] * ud[cn];
    if (div == 0.0) stat |= ST_PIVOT;
    sol[cn] = (rhs[cn] - Cm1[cn] * sol[c]) / div;
    c = cn;
  }
  if (c != cs) stat |= ST_GEOM;
  for (int it = 0; c != cb && it < G.nz; ++it) {
    const int cd = G.zm1[c];
    sol[cd] -= ud[c] * sol[c];
    c = cd;
  }
  for (int it = 0; it <= G.nz; ++it) {
    var[c] = sol[c] > minvar ? sol[c] : minvar;
    if (c == cs) break;
    c = G.zp1[c];
  }
  if (stat) atomicOr(W.status, stat);
}

// implicit_vdiff_at_cc (model/hd/tracers/tracers.c:7407-7545): implicit
// vertical diffusion of var with bottom / top fluxes fb, ft, sources Splus,
// Sminus (may be null) and the scale factor, with no thin layers
__global__ void k_vdiff_cols(Geo G, Work W, double *var, const double *dzcell, const double *C,
                             const double *Cm1, const double *Cp1, const double *fb,
                             const double *ft, const double *Splus, const double *Sminus,
                             const double *scale, double *sol, double *ud, double dt,
                             double dt_win, double hmin) {
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= G.ncol) return;
  const int cs = W.nsur_t[col], cb = G.col_bot[col];
  if (cs == G.zm1[cs]) return;
  const int c2 = G.m2d[cs];
  const int zm1 = G.zm1[cs];
  int stat = 0;
  // single layer (the surface in the bottom layer, :7459-7467)
  if (zm1 == G.zm1[zm1] || !dzcell[zm1]) {
    const double h = dzcell[cs] > hmin ? dzcell[cs] : hmin;
    var[cs] += dt_win * (fb[c2] - ft[c2]) / h;
    return;
  }
  // right-hand side (:7479-7508) into sol, the main diagonal with the
  // negative sources into ud (both are rewritten by the sweep below)
  int c = cb;
  for (int it = 0; it <= G.nz; ++it) {
    const double dzdt = dzcell[c] / dt;
    double r = dzdt * var[c];
    if (c == cb) r = r + fb[c2];
    if (c == cs) r = r - ft[c2];
    sol[c] = r;
    ud[c] = C[c];
    if (c == cs) break;
    c = G.zp1[c];
  }
  if (c != cs) stat |= ST_GEOM;
  if (Splus) {
    for (int cc = cb, it = 0; it <= G.nz; cc = G.zp1[cc], ++it) {
      sol[cc] += dzcell[cc] * Splus[cc];
      if (cc == cs) break;
    }
  }
  if (Sminus) {
    for (int cc = cb, it = 0; it <= G.nz; cc = G.zp1[cc], ++it) {
      ud[cc] += dzcell[cc] * Sminus[cc] / var[cc];
      if (cc == cs) break;
    }
  }
  // Thomas sweep (:7517-7526): the main diagonal B sits in ud until the row
  // is eliminated, then ud holds the elimination factor
  double div = ud[cb];
  sol[cb] = sol[cb] / div;
  c = cb;
  for (int it = 0; c != cs && it < G.nz; ++it) {
    const int cn = G.zp1[c];
    const double B = ud[cn];
    ud[cn] = Cp1[c] / div;
    div = B - Cm1[cn] * ud[cn];
    if (div == 0.0) stat |= ST_PIVOT;
    sol[cn] = (sol[cn] - Cm1[cn] * sol[c]) / div;
    c = cn;
  }
  // update (:7530-7536)
  const double sc = scale[c2];
  var[cs] += (sol[cs] - var[cs]) * sc;
  for (int it = 0; c != cb && it < G.nz; ++it) {
    const int cd = G.zm1[c];
    sol[cd] -= ud[c] * sol[c];
    var[cd] += (sol[cd] - var[cd]) * sc;
    c = cd;
  }
  if (stat) atomicOr(W.status, stat);
}

// Halo exchange of a strip of a decomposed basin: gather the send cells of
// every tracer into a contiguous buffer, or scatter a buffer into the
// receive cells of both tracer buffers.
template <class TR>
__global__ void k_halo_pack(const TR *tr, int S, int ntr, const int *cells, int n, TR *buf) {
  const long long tot = (long long)ntr * n;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < tot;
       i += (long long)gridDim.x * blockDim.x) {
    const int t = (int)(i / n), j = (int)(i % n);
    buf[i] = tr[(size_t)t * S + cells[j]];
  }
}
template <class TR>
__global__ void k_halo_unpack(TR *tra, TR *trb, int S, int ntr, const int *cells, int n,
                              const TR *buf) {
  const long long tot = (long long)ntr * n;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < tot;
       i += (long long)gridDim.x * blockDim.x) {
    const int t = (int)(i / n), j = (int)(i % n);
    const size_t o = (size_t)t * S + cells[j];
    tra[o] = buf[i];
    trb[o] = buf[i];
  }
}

cudaError_t tile64_set_smem_attr();

// Static tables of the column-tile kernel: the cell of every column at every
// layer (cells are numbered layer by layer, so a column's cells are found by
// walking zp1 up from its bottom cell), the first and second horizontal
// neighbours of every cell, the 2D cells of its east and north neighbours and
// their flags.
int build_tile_tables(shoc_tr_gpu *h, const shoc_tr_geom *g, const std::vector<uint8_t> &cflag,
                      const std::vector<int> &col_bot, const std::vector<int> &col_kb) {
  const int S = h->S, nz = h->nz, ncol = h->ncol;
  const int ncolp = (ncol + 31) / 32 * 32;
  std::vector<int> cellk((size_t)nz * ncolp, 0);
  for (int col = 0; col < ncol; col++) {
    int c = col_bot[col];
    for (int k = col_kb[col]; k < nz; k++) {
      if (c <= 0 || c >= S) break;
      cellk[(size_t)k * ncolp + col] = c;
      c = g->zp1[c];
    }
  }
  auto in = [S](int c) { return c >= 0 && c < S ? c : 0; };
  const int S2 = h->S2;
  auto in2 = [S2](int c) { return c >= 0 && c < S2 ? c : 0; };
  std::vector<int4> nb1(S), nb2(S);
  std::vector<int2> m2e(S);
  std::vector<uint8_t> fl(S);
  for (int c = 0; c < S; c++) {
    const int xm = in(g->xm1[c]), xp = in(g->xp1[c]), ym = in(g->ym1[c]), yp = in(g->yp1[c]);
    nb1[c] = make_int4(xm, xp, ym, yp);
    nb2[c] = make_int4(in(g->xm1[xm]), in(g->xp1[xp]), in(g->ym1[ym]), in(g->yp1[yp]));
    m2e[c] = make_int2(in2(g->m2d[xp]), in2(g->m2d[yp]));
    uint8_t f = cflag[c] & (CF_WET | CF_E1 | CF_E2);
    if (cflag[xp] & CF_WET) f |= FL_XP_WET;
    if (cflag[xp] & CF_E1) f |= FL_XP_E1;
    if (cflag[yp] & CF_WET) f |= FL_YP_WET;
    if (cflag[yp] & CF_E2) f |= FL_YP_E2;
    fl[c] = f;
  }
  // vertical neighbours and the column of each wet cell
  std::vector<int4> nbz(S);
  for (int c = 0; c < S; c++) {
    const int zm = in(g->zm1[c]), zp = in(g->zp1[c]);
    nbz[c] = make_int4(zm, in(g->zm1[zm]), zp, in(g->zp1[zp]));
  }
  std::vector<int> colof(S, 0);
  for (int col = 0; col < ncol; col++)
    for (int k = col_kb[col]; k < nz; k++) {
      const int c = cellk[(size_t)k * ncolp + col];
      if (c) colof[c] = col;
    }
  // k_adv32 cell order: segment by segment (up to 31 adjacent columns), layer by
  // layer within one, so the vertical and y-neighbours a block reads were read
  // by blocks shortly before it (cache reuse) and a warp's cells are mostly
  // adjacent cells of one layer.  A cell's east neighbour, where it is wet, is
  // the next lane's: a run that goes on beyond the segment, or beyond a warp's
  // last lane, is given a halo lane there.
  std::vector<int> wet;
  wet.reserve((size_t)g->a3_t + g->a3_t / 16);
  for (int col0 = 0; col0 < ncol; col0 += 31) {
    const int col1 = std::min(ncol, col0 + 31);
    for (int k = nz - 1; k >= 0; k--) {
      const int *row = &cellk[(size_t)k * ncolp];
      for (int col = col0; col < col1; col++) {
        const int c = row[col];
        if (!c || !(fl[c] & CF_WET)) continue;
        const int e = (fl[c] & FL_XP_WET) ? nb1[c].y : 0;  // its wet east neighbour
        if ((wet.size() & 31) == 31 && e) {
          // a warp's last lane: the cell lends its west flux to the lane before
          // it, or the lane stays empty
          const int w = wet.back() & ~kSegHalo;
          wet.push_back((wet.back() >= 0 && (fl[w] & FL_XP_WET) && nb1[w].y == c)
                            ? c | kSegHalo : -1);
        }
        wet.push_back(c);
        // the run's end in this segment with a wet east neighbour beyond it
        if (e && (col + 1 >= col1 || row[col + 1] != e)) wet.push_back(e | kSegHalo);
      }
    }
  }
  // k_vd32 column order: tiles of 32 adjacent columns (a warp's lanes at one
  // layer are adjacent cells: coalesced loads and stores), the tiles sorted
  // by depth so that blocks running at the same time are alike
  const int ntile = ncolp / 32;
  std::vector<int> tdepth(ntile, 0), tord(ntile);
  for (int t = 0; t < ntile; t++) {
    int kmin = nz;
    for (int l = 0; l < 32 && t * 32 + l < ncol; l++) kmin = std::min(kmin, col_kb[t * 32 + l]);
    tdepth[t] = nz - kmin;
    tord[t] = t;
  }
  std::stable_sort(tord.begin(), tord.end(), [&](int a, int b) { return tdepth[a] < tdepth[b]; });
  std::vector<int> vdcol(ncolp, -1);
  h->vd_depth.resize(ntile);
  h->vd_layers.assign(ntile + 1, 0);
  for (int i = 0; i < ntile; i++) {
    const int t = tord[i];
    h->vd_depth[i] = tdepth[t];
    h->vd_layers[i + 1] = h->vd_layers[i] + tdepth[t];
    for (int l = 0; l < 32; l++) vdcol[i * 32 + l] = (t * 32 + l < ncol) ? t * 32 + l : -1;
  }
  // k_adv64's segments: columns in order, 32 to a warp.  A column's wet east
  // neighbours are the next lane's cells: where the next column is not its east
  // neighbour, or the warp is full, that one is added as a halo lane.
  std::vector<int> col_of_top(h->S2, -1);
  for (int col = 0; col < ncol; col++) col_of_top[g->w2_t[col + 1]] = col;
  std::vector<int> east_of(ncol, -1);
  for (int col = 0; col < ncol; col++) {
    const int e = in(g->xp1[g->w2_t[col + 1]]);
    if (e < h->S2) east_of[col] = col_of_top[e];
  }
  std::vector<int> seg;
  for (int col = 0; col < ncol; col++) {
    const int e = east_of[col];
    if ((seg.size() & 31) == 31 && e >= 0) {  // the last lane: a halo lane, or none
      const int b = seg.back();
      seg.push_back(b >= 0 && !(b & kSegHalo) && east_of[b] == col ? col | kSegHalo : -1);
    }
    seg.push_back(col);
    if (e >= 0 && e != col + 1) seg.push_back(e | kSegHalo);
  }
  while (seg.size() & 31) seg.push_back(-1);
  // cells whose wet east neighbour is not in their column's east column (maps that
  // do not stack): k_adv64_apart's
  std::vector<int> apart;
  if (h->O.cross)
    for (int c = 1; c < S; c++) {
      if ((fl[c] & (CF_WET | FL_XP_WET)) != (CF_WET | FL_XP_WET)) continue;
      const int e = nb1[c].y;
      if (east_of[colof[c]] != colof[e] || g->s2k[c] != g->s2k[e]) apart.push_back(c);
    }
  std::vector<int4> colrec(ncolp, make_int4(0, 0, nz, 0));
  for (int col = 0; col < ncol; col++)
    colrec[col] = make_int4(col_bot[col], g->w2_t[col + 1], col_kb[col], 0);
  Tile &T = h->tl;
  T.ncolp = ncolp;
  T.nwet = (int)wet.size();
  int *ip;
  int rc;
  if ((rc = dupload(h, &ip, cellk.data(), cellk.size()))) return rc;
  T.cellk = ip;
  int4 *i4;
  if ((rc = dupload(h, &i4, nb1.data(), S))) return rc;
  T.nb1 = i4;
  if ((rc = dupload(h, &i4, nb2.data(), S))) return rc;
  T.nb2 = i4;
  int2 *i2;
  if ((rc = dupload(h, &i2, m2e.data(), S))) return rc;
  T.m2e = i2;
  uint8_t *u8;
  if ((rc = dupload(h, &u8, fl.data(), S))) return rc;
  T.fl = u8;
  T.kof = h->G.kof;
  if ((rc = dupload(h, &i4, nbz.data(), S))) return rc;
  T.nbz = i4;
  if ((rc = dupload(h, &i4, colrec.data(), colrec.size()))) return rc;
  T.colrec = i4;
  if ((rc = dupload(h, &ip, colof.data(), S))) return rc;
  T.colof = ip;
  if ((rc = dupload(h, &ip, wet.data(), wet.size()))) return rc;
  T.wet = ip;
  if ((rc = dupload(h, &ip, vdcol.data(), vdcol.size()))) return rc;
  T.vdcol = ip;
  if ((rc = dupload(h, &ip, seg.data(), seg.size()))) return rc;
  T.seg = ip;
  // k_adv64's work: the layers of each segment in chunks, a warp each.  A longer
  // climb computes fewer bottom faces twice (one per chunk), a shorter one gives more
  // warps: the chunks are the longest that still make about six rounds of the warps
  // the chip holds.  The layers are those the segments' columns have: counted and
  // cut over the window's layers, chunks were too long and many of them empty (384 x
  // 320 x 40, 2 to 40 layers deep, 10 tracers, 4 steps 5.44 ms, 4.69 so; 400 x 300, 60
  // layers of which the columns have 8 at most, 1 tracer, k_adv64 0.155 and 0.093).
  if (h->O.cross) {
    const int nseg = (int)(seg.size() / 32);
    std::vector<int> kmin(nseg, nz);
    long long layers = 0;
    for (int i = 0; i < nseg; i++) {
      for (int l = 0; l < 32; l++) {
        const int e = seg[i * 32 + l];
        if (e >= 0 && !(e & kSegHalo)) kmin[i] = std::min(kmin[i], col_kb[e]);
      }
      layers += nz - kmin[i];
    }
    const int groups = (h->T.ntb + kAdv64Group - 1) / kAdv64Group;
    const long long resident = 148LL * std::min<long long>(
        16, 233472 / (adv64_smem(std::min(std::max(h->T.ntb, 1), kAdv64Group)) + 1024));
    for (int q = 1; q <= groups; q++) {
      shoc_tr_gpu::AdvItems it;
      it.lmax = (int)std::max<long long>(1, layers * q / (resident * 6));
      if (q > 1 && h->adv_items.back().lmax == it.lmax) {
        h->adv_items.push_back(h->adv_items.back());
        continue;
      }
      std::vector<int2> list;
      for (int i = 0; i < nseg; i++) {
        const int d = nz - kmin[i], n = (d + it.lmax - 1) / it.lmax;
        for (int j = 0; j < n; j++) {
          const int k0 = kmin[i] + j * ((d + n - 1) / n), k1 = std::min(nz, k0 + (d + n - 1) / n);
          if (k0 < k1) list.push_back(make_int2(i, k0 | k1 << 16));
        }
      }
      it.n = (int)list.size();
      if ((rc = dupload(h, &it.d, list.data(), list.size()))) return rc;
      h->adv_items.push_back(it);
    }
  }
  T.nseg = (int)(seg.size() / 32);
  if (!apart.empty()) {
    if ((rc = dupload(h, &ip, apart.data(), apart.size()))) return rc;
    T.apart = ip;
    T.napart = (int)apart.size();
  }
  return 0;
}

// Tiles of the fused FP32-mixed kernel: tx x ty water columns, ty = 32 / tx
// (lane = tx * iy + ix for the column at (tx * ti + ix, ty * tj + iy)), in
// row-major tile order so that blocks running at the same time hold
// neighbouring tiles; a tile's lowest layer bounds its layer loop.
int build_fused_tiles(shoc_tr_gpu *h, const shoc_tr_geom *g, const std::vector<int> &col_kb,
                      int tx, shoc_tr_gpu::FusedTiles &out) {
  const int ty = 32 / tx;
  const int ncol = h->ncol;
  int imax = 0, jmax = 0;
  for (int col = 0; col < ncol; col++) {
    const int top = g->w2_t[col + 1];
    if (g->s2i[top] < 0 || g->s2j[top] < 0) return SHOC_TR_EGEOM;
    imax = std::max(imax, g->s2i[top]);
    jmax = std::max(jmax, g->s2j[top]);
  }
  const long long nti = imax / tx + 1, ntj = jmax / ty + 1;
  std::vector<int> tid((size_t)(nti * ntj), -1);
  std::vector<int> tcol, tkmin;
  std::vector<int> order(ncol);
  for (int col = 0; col < ncol; col++) order[col] = col;
  auto key = [&](int col) {
    const int top = g->w2_t[col + 1];
    return (long long)(g->s2j[top] / ty) * nti + g->s2i[top] / tx;
  };
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return key(a) < key(b); });
  for (int col : order) {
    const int top = g->w2_t[col + 1];
    const int i = g->s2i[top], j = g->s2j[top];
    int &t = tid[(size_t)key(col)];
    if (t < 0) {
      t = (int)tkmin.size();
      tkmin.push_back(h->nz);
      tcol.insert(tcol.end(), 32, -1);
    }
    const int lane = (j % ty) * tx + i % tx;
    if (tcol[(size_t)t * 32 + lane] >= 0) return SHOC_TR_EGEOM;  // two columns at one (i, j)
    tcol[(size_t)t * 32 + lane] = col;
    tkmin[t] = std::min(tkmin[t], col_kb[col]);
  }
  out.ntile = (int)tkmin.size();
  int *ip;
  int rc;
  if ((rc = dupload(h, &ip, tcol.data(), tcol.size()))) return rc;
  out.tcol = ip;
  if ((rc = dupload(h, &ip, tkmin.data(), tkmin.size()))) return rc;
  out.tkmin = ip;
  return 0;
}

// k_step32's shared memory with nwb phase-B warps, and its reduction group:
// as many advected tracers per phase-A reduction pass as fit the space the
// phase-B arrays leave.
size_t fused_config(const shoc_tr_gpu *h, int nwb, int *ngrp) {
  const int ntb = h->T.ntb;
  const size_t room = (size_t)2 * nwb * h->nz * 32 * 4;
  const size_t buf = (size_t)2 * kStencil * kFusedThreads * 4;
  const int gmax = room > buf ? (int)((room - buf) / fused_red(1)) : 1;
  *ngrp = std::max(1, std::min(std::max(ntb, 1), gmax));
  return fused_smem(h->nz, nwb, ntb, *ngrp);
}

int tile_index(int tx) { return tx == 8 ? 0 : tx == 16 ? 1 : tx == 32 ? 2 : -1; }

void drop_graphs(shoc_tr_gpu *h) {
  for (int i = 0; i < 2; i++)
    if (h->graph[i]) {
      cudaGraphExecDestroy(h->graph[i]);
      h->graph[i] = nullptr;
    }
}

// The launch configuration of the transport kernels (validated; takes
// effect at the next step).
int apply_tuning(shoc_tr_gpu *h, const shoc_tr_tuning &t) {
  const bool f32 = h->esize == sizeof(float);
  if (t.tracers_per_block < 1 || t.tracers_per_block > (f32 ? kVd32MaxWarps : 8))
    return SHOC_TR_EUNSUPPORTED;
  if (t.prefetch && !f32) return SHOC_TR_EUNSUPPORTED;
  // the window's layers decide, but for what the default needs in columns that do
  // not have them all
  auto fits = [&](int nd) {
    return (f32 ? vd32_smem(nd, t.tracers_per_block, t.prefetch != 0, h->comp)
                : vd64_tuned(nd, t.tracers_per_block)) <= 227 * 1024;
  };
  if (!fits(t.tracers_per_block > h->tw_default ? h->nz : std::max(1, h->vd_depth.back())))
    return SHOC_TR_EUNSUPPORTED;
  if (t.fused) {
    const int ti = tile_index(t.tile_x);
    if (!f32 || h->comp || !h->fnwb_max || ti < 0 || !h->ftile[ti].tcol) return SHOC_TR_EUNSUPPORTED;
    if (t.phase_b_warps < 1 || t.phase_b_warps > h->fnwb_max) return SHOC_TR_EUNSUPPORTED;
  } else if (f32 && !h->rnd) {
    const int rc = dalloc(h, &h->rnd, (size_t)h->ntr * h->S);
    if (rc) return rc;
  }
  h->tw = t.tracers_per_block;
  h->vd_pf = t.prefetch != 0;
  h->fused = t.fused != 0;
  if (h->fused) {
    const auto &ft = h->ftile[tile_index(t.tile_x)];
    h->fu.tcol = ft.tcol;
    h->fu.tkmin = ft.tkmin;
    h->fu.ntile = ft.ntile;
    h->fu.tx = t.tile_x;
    h->fu.nwb = t.phase_b_warps;
    h->fused_bytes = fused_config(h, t.phase_b_warps, &h->fu.ngrp);
  }
  drop_graphs(h);
  return SHOC_TR_OK;
}

shoc_tr_tuning current_tuning(const shoc_tr_gpu *h) {
  shoc_tr_tuning t;
  t.fused = h->fused ? 1 : 0;
  t.tracers_per_block = h->tw;
  t.tile_x = h->fused ? h->fu.tx : 8;
  t.phase_b_warps = h->fused ? h->fu.nwb : h->fnwb_max;
  t.prefetch = h->vd_pf ? 1 : 0;
  return t;
}

int map_status(int st) {
  if (st & ST_GEOM) return SHOC_TR_EGEOM;
  if (st & ST_PIVOT) return SHOC_TR_EPIVOT;
  if (st & ST_NAN) return SHOC_TR_ENAN;
  if (st & ST_LASTDRY) return SHOC_TR_EUNSUPPORTED;
  if (st & ST_SCRATCH) return SHOC_TR_ESCRATCH;
  return SHOC_TR_OK;
}

int check_geom(const shoc_tr_geom *g, const shoc_tr_opts *o, int ntr) {
  if (!g || !o || ntr < 0) return SHOC_TR_EARG;
  switch (o->trasc) {  // FFSL and LAGRANGE are not built
    case SHOC_TR_QUICKEST: case SHOC_TR_VANLEER: case SHOC_TR_ORDER1: case SHOC_TR_ORDER2:
    case SHOC_TR_ORDER4: case SHOC_TR_QUICKEST_CO: case SHOC_TR_ORDER2_UW: break;
    default: return SHOC_TR_EUNSUPPORTED;
  }
  if (g->v3_t != g->b3_t || g->b3_t != g->a3_t) return SHOC_TR_EUNSUPPORTED;  // OBC / aux cells
  if (g->v2_t != g->b2_t || g->b2_t != g->a2_t) return SHOC_TR_EUNSUPPORTED;
  if (g->nz < 1 || g->nz > kMaxLayers) return SHOC_TR_EUNSUPPORTED;
  if (o->ntr2d) {  // per-column tracer counts: the advected tracers in ascending order
    for (int i = 1; i < o->ntbdy; i++)
      if (o->tbdy[i] <= o->tbdy[i - 1]) return SHOC_TR_EARG;
  }
  if (g->sgsiz < 2 || g->sgsizS < 2 || g->b2_t < 1) return SHOC_TR_EGEOM;
  const int S = g->sgsiz;
  std::vector<uint8_t> wet(S, 0);
  for (int i = 1; i <= g->a3_t; i++) {
    int c = g->w3_t[i];
    if (c < 1 || c >= S) return SHOC_TR_EGEOM;
    wet[c] = 1;
  }
  for (int c = 1; c < S; c++) {
    const int *mp[6] = {g->xp1, g->xm1, g->yp1, g->ym1, g->zp1, g->zm1};
    for (int q = 0; q < 6; q++)
      if (mp[q][c] < 0 || mp[q][c] >= S) return SHOC_TR_EGEOM;
    if (!wet[c]) continue;
    if (g->m2d[c] < 1 || g->m2d[c] >= g->sgsizS) return SHOC_TR_EGEOM;
    // the stencil of the neighbouring face reuses this cell's values
    if (wet[g->xp1[c]] && g->xm1[g->xp1[c]] != c) return SHOC_TR_EGEOM;
    if (wet[g->yp1[c]] && g->ym1[g->yp1[c]] != c) return SHOC_TR_EGEOM;
    if (g->zp1[c] != c && g->zm1[g->zp1[c]] != c) return SHOC_TR_EGEOM;
  }
  for (int cc = 1; cc <= g->b2_t; cc++) {
    int top = g->w2_t[cc], bot = g->bot_t[cc];
    if (top < 1 || top >= g->sgsizS || !wet[top] || bot < 1 || bot >= S || !wet[bot])
      return SHOC_TR_EGEOM;
    if (g->zp1[top] != top || g->s2k[top] != g->nz - 1) return SHOC_TR_EGEOM;
    // bottom reaches the top through zp1 and sits on a self-mapping sediment
    int sed = g->zm1[bot];
    if (sed == bot || wet[sed] || g->zm1[sed] != sed || g->zp1[sed] != bot) return SHOC_TR_EGEOM;
    // and every cell on the way sits one layer above the previous one
    int c = bot, steps = 0;
    const int kb = g->s2k[bot];
    if (kb < 0 || kb >= g->nz) return SHOC_TR_EGEOM;
    while (c != top && steps <= g->nz) {
      if (g->s2k[c] != kb + steps) return SHOC_TR_EGEOM;
      c = g->zp1[c];
      steps++;
    }
    if (c != top || kb + steps != g->nz - 1) return SHOC_TR_EGEOM;
  }
  for (int i = 1; i <= g->nbpt; i++)
    if (g->bpt[i] < 1 || g->bpt[i] >= S || g->bin[i] < 1 || g->bin[i] >= S) return SHOC_TR_EGEOM;
  return SHOC_TR_OK;
}

}  // namespace

// ---------------------------------------------------------------------------
// C-ABI

// The e1 (e2) face columns of a window as SHOC lists them in w2_e1, bot_e1
// and botzu1 (w2_e2, bot_e2, botzu2): the surface-layer cells of w3_e1, each
// column's deepest w3_e1 cell (the faces are wet from the surface layer
// down to it) and the higher of the floors on the two sides of the face
// (hd_init.c:1443).  bm: the backward map (xm1 or ym1).  False where w3_e1 is
// not one run from the surface layer down in every face column.
bool face_columns(const shoc_tr_geom *g, int ne, const int *w3, const int *bm,
                  std::vector<int2> &fc, std::vector<double> &bz) {
  const int S = g->sgsiz;
  if (ne > 0 && !w3) return false;
  std::vector<uint8_t> in(S, 0);
  for (int i = 1; i <= ne; i++) {
    const int c = w3[i];
    if (c <= 0 || c >= S || in[c]) return false;
    in[c] = 1;
  }
  long long covered = 0;
  for (int i = 1; i <= ne; i++) {
    const int c2 = w3[i];
    if (g->zp1[c2] != c2) continue;  // below the surface layer
    int c = c2, cb = c2;
    while (g->zm1[c] != c && in[c]) {
      cb = c;
      covered++;
      c = g->zm1[c];
    }
    fc.push_back(make_int2(c2, cb));
    const double a = g->botz[bm[c2]], b = g->botz[c2];
    bz.push_back(a > b ? a : b);
  }
  return covered == ne;
}

extern "C" {

const char *shoc_tr_gpu_strerror(int st) {
  switch (st) {
    case SHOC_TR_OK: return "ok";
    case SHOC_TR_ESUBSTEP: return "maximum number of tracer sub-steps exceeded";
    case SHOC_TR_EPIVOT: return "zero pivot in the implicit vertical diffusion solve";
    case SHOC_TR_ENAN: return "NaN in a tracer after the step";
    case SHOC_TR_EGEOM: return "geometry fails the layout checks";
    case SHOC_TR_EUNSUPPORTED: return "unsupported option";
    case SHOC_TR_ECUDA: return "CUDA runtime error";
    case SHOC_TR_EARG: return "bad argument";
    case SHOC_TR_ENOMEM: return "allocation failed";
    case SHOC_TR_ESCRATCH: return "problem larger than the fixed scratch area";
  }
  return "unknown status";
}

void shoc_tr_gpu_destroy(shoc_tr_gpu *h) {
  if (!h) return;
  DeviceScope dev_(h->device);
  if (h->stream) cudaStreamSynchronize(h->stream);
  for (int i = 0; i < 2; i++)
    if (h->graph[i]) cudaGraphExecDestroy(h->graph[i]);
  {
    std::vector<cudaEvent_t> done;  // pairs may share events
    for (auto &e : h->ev)
      for (cudaEvent_t x : {e.a, e.b})
        if (std::find(done.begin(), done.end(), x) == done.end()) done.push_back(x);
    for (cudaEvent_t x : done) cudaEventDestroy(x);
  }
  for (cudaStream_t x : {h->s_up, h->s_cv, h->s_dn})
    if (x) cudaStreamSynchronize(x);
  for (cudaEvent_t x : h->pev)
    if (x) cudaEventDestroy(x);
  for (cudaEvent_t x : {h->ev_in[0], h->ev_in[1], h->ev_cv[0], h->ev_cv[1]})
    if (x) cudaEventDestroy(x);
  for (void *p : h->allocs) cudaFree(p);
  if (h->h_rb) cudaFreeHost(h->h_rb);
  if (h->h_surf) cudaFreeHost(h->h_surf);
  for (cudaStream_t x : {h->s_up, h->s_cv, h->s_dn})
    if (x) cudaStreamDestroy(x);
  if (h->stream) cudaStreamDestroy(h->stream);
  delete h;
}

int shoc_tr_gpu_create(const shoc_tr_geom *g, const shoc_tr_opts *o, int ntr, int precision,
                       int device, shoc_tr_gpu **out) {
  if (!out) return SHOC_TR_EARG;
  *out = nullptr;
  int rc = check_geom(g, o, ntr);
  if (rc) return rc;
  if (precision != SHOC_TR_FP64 && precision != SHOC_TR_FP32_MIXED &&
      precision != SHOC_TR_FP32_COMP)
    return SHOC_TR_EUNSUPPORTED;
  if (precision == SHOC_TR_FP32_MIXED && ntr > kMaxTracers) return SHOC_TR_EUNSUPPORTED;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0 || device < 0 || device >= ndev)
    return SHOC_TR_ECUDA;
  shoc_tr_gpu *h = new shoc_tr_gpu();
  h->device = device;
  h->precision = precision;
  h->ntr = ntr;
  h->S = g->sgsiz;
  h->S2 = g->sgsizS;
  h->nz = g->nz;
  h->ncol = g->b2_t;
  h->nbpt = g->nbpt;
#define TRY(x)                \
  do {                        \
    int r_ = (x);             \
    if (r_) {                 \
      shoc_tr_gpu_destroy(h); \
      return r_;              \
    }                         \
  } while (0)
  DeviceScope dev_(device);
  if (!dev_.ok) TRY(SHOC_TR_ECUDA);
  if (cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) != cudaSuccess)
    TRY(SHOC_TR_ECUDA);
  const int S = h->S, S2 = h->S2, ncol = h->ncol;

  // ---- host precomputation ----
  std::vector<uint8_t> cflag(S, 0);
  for (int i = 1; i <= g->a3_t; i++) cflag[g->w3_t[i]] |= CF_WET;
  for (int i = 1; i <= g->v3_e1; i++) cflag[g->w3_e1[i]] |= CF_E1;
  for (int i = 1; i <= g->v3_e2; i++) cflag[g->w3_e2[i]] |= CF_E2;
  std::vector<Face2D> fx(S2), fy(S2);
  for (int c2 = 1; c2 < S2; c2++) {
    int xm = g->xm1[c2], xp = g->xp1[c2], ym = g->ym1[c2], yp = g->yp1[c2];
    if (xm >= S2 || xp >= S2 || ym >= S2 || yp >= S2) continue;  // not a 2D cell
    Face2D a, b;
    // d3 / d4 (tracers.c:568-577) and the QUICKEST metric factors (:1862-1864)
    a.d = g->h1acell[xm] / (g->h1acell[xm] + g->h1acell[c2]);
    a.db = 2.0 / (g->h1au1[xm] + g->h1au1[c2]);
    a.df = 2.0 / (g->h1au1[c2] + g->h1au1[xp]);
    a.hm = g->h1au1[xm];
    a.h0 = g->h1au1[c2];
    a.hp = g->h1au1[xp];
    b.d = g->h2acell[ym] / (g->h2acell[ym] + g->h2acell[c2]);
    b.db = 2.0 / (g->h2au2[ym] + g->h2au2[c2]);
    b.df = 2.0 / (g->h2au2[c2] + g->h2au2[yp]);
    b.hm = g->h2au2[ym];
    b.h0 = g->h2au2[c2];
    b.hp = g->h2au2[yp];
    fx[c2] = a;
    fy[c2] = b;
  }
  std::vector<int> col_top(ncol), col_bot(ncol), col_kb(ncol), sur0(ncol, 0);
  for (int cc = 1; cc <= ncol; cc++) {
    col_top[cc - 1] = g->w2_t[cc];
    col_bot[cc - 1] = g->bot_t[cc];
    col_kb[cc - 1] = g->s2k[g->bot_t[cc]];
  }

  // ---- device geometry ----
  Geo &G = h->G;
  G.S = S;
  G.S2 = S2;
  G.nz = g->nz;
  G.ncol = ncol;
  G.v2col = g->v2_t - 1;
  int *ip;
  TRY(dupload(h, &ip, g->xp1, S)); G.xp1 = ip;
  TRY(dupload(h, &ip, g->xm1, S)); G.xm1 = ip;
  TRY(dupload(h, &ip, g->yp1, S)); G.yp1 = ip;
  TRY(dupload(h, &ip, g->ym1, S)); G.ym1 = ip;
  TRY(dupload(h, &ip, g->zp1, S)); G.zp1 = ip;
  TRY(dupload(h, &ip, g->zm1, S)); G.zm1 = ip;
  TRY(dupload(h, &ip, g->m2d, S)); G.m2d = ip;
  uint8_t *u8;
  TRY(dupload(h, &u8, cflag.data(), S)); G.cflag = u8;
  TRY(dupload(h, &ip, col_top.data(), ncol)); G.col_top = ip;
  TRY(dupload(h, &ip, col_bot.data(), ncol)); G.col_bot = ip;
  TRY(dupload(h, &ip, col_kb.data(), ncol)); G.col_kb = ip;
  TRY(dupload(h, &ip, g->s2k, S)); G.kof = ip;
  {
    std::vector<int> colntr(ncol, ntr);
    if (o->ntr2d)
      for (int col = 0; col < ncol; col++)
        colntr[col] = std::max(0, std::min(ntr, o->ntr2d[col_top[col]]));
    TRY(dupload(h, &ip, colntr.data(), ncol)); G.colntr = ip;
  }
  double *dp;
  TRY(dupload(h, &dp, g->h1au1, S2)); G.h1au1 = dp;
  TRY(dupload(h, &dp, g->h2au2, S2)); G.h2au2 = dp;
  TRY(dupload(h, &dp, g->h1au2, S2)); G.h1au2 = dp;
  TRY(dupload(h, &dp, g->h2au1, S2)); G.h2au1 = dp;
  TRY(dupload(h, &dp, g->h1acell, S2)); G.h1acell = dp;
  TRY(dupload(h, &dp, g->h2acell, S2)); G.h2acell = dp;
  TRY(dupload(h, &dp, g->cellarea, S2)); G.cellarea = dp;
  TRY(dupload(h, &dp, g->botz, S2)); G.botz = dp;
  TRY(dupload(h, &dp, g->gridz, S)); G.gridz = dp;
  Face2D *fp;
  TRY(dupload(h, &fp, fx.data(), S2)); G.fx = fp;
  TRY(dupload(h, &fp, fy.data(), S2)); G.fy = fp;
  if (g->nbpt > 0) {
    TRY(dupload(h, &h->bpt, g->bpt + 1, g->nbpt));
    TRY(dupload(h, &h->bin, g->bin + 1, g->nbpt));
  }

  // ---- options and tracers ----
  h->O.trasc = o->trasc;
  // order1 is monotonic and switches the limiter off (tracers.c:497-503)
  h->O.ultimate = o->trasc == SHOC_TR_ORDER1 ? 0 : o->ultimate;
  h->O.cross = precision == SHOC_TR_FP64 ? 1 : 0;
  h->O.tiled = (o->trasc == SHOC_TR_QUICKEST || o->trasc == SHOC_TR_VANLEER || h->O.cross) ? 1 : 0;
  h->O.substep =
      (o->stab & (SHOC_TR_SUB_STEP | SHOC_TR_SUB_STEP_NOSURF | SHOC_TR_SUB_STEP_TRACER)) ? 1 : 0;
  h->O.hmin = o->hmin;
  h->trf.assign(ntr, 0);
  std::vector<int> slot;
  for (int i = 0; i < o->ntbdy; i++) {
    int n = o->tbdy[i];
    if (n < 0 || n >= ntr) TRY(SHOC_TR_EARG);
    h->trf[n] |= TR_TBDY;
    if (o->advect[n]) h->trf[n] |= TR_ADV;
    if (o->diffuse[n]) {
      h->trf[n] |= TR_HDIFF;
      h->any_hdiff = true;
    }
    slot.push_back(n);
  }
  for (int i = 0; i < o->ntdif_v; i++) {
    int n = o->tdif_v[i];
    if (n < 0 || n >= ntr) TRY(SHOC_TR_EARG);
    h->trf[n] |= TR_VDIFF;
    h->any_vdiff = true;
  }
  for (int n = 0; n < ntr; n++)
    if (!(h->trf[n] & TR_TBDY)) slot.push_back(n);
  {
    bool all_a = true, all_h = true, no_h = true;
    for (int i = 0; i < o->ntbdy; i++) {
      const uint8_t f = h->trf[o->tbdy[i]];
      all_a = all_a && (f & TR_ADV);
      all_h = all_h && (f & TR_HDIFF);
      no_h = no_h && !(f & TR_HDIFF);
    }
    h->adv_flags = !all_a ? 0 : (no_h ? 1 : (all_h ? 2 : 0));
  }
  h->nslot = (int)slot.size();
  h->slot_host = slot;
  TrSet &T = h->T;
  T.ntr = ntr;
  T.nslot = h->nslot;
  T.ntb = o->ntbdy;
  TRY(dupload(h, &ip, slot.data(), slot.size())); T.slot_tr = ip;
  TRY(dupload(h, &u8, h->trf.data(), ntr)); T.trf = u8;
  TRY(dupload(h, &dp, o->mintr, ntr)); T.mintr = dp;
  TRY(dupload(h, &dp, o->maxtr, ntr)); T.maxtr = dp;

  // ---- work arrays ----
  Work &W = h->W;
  TRY(dupload<double>(h, &W.dz, nullptr, S));
  TRY(dupload<double>(h, &W.w5, nullptr, S));
  TRY(dupload<double>(h, &W.w9, nullptr, S));
  TRY(dupload<double>(h, &W.dbz, nullptr, S));
  TRY(dupload<double>(h, &W.dfz, nullptr, S));
  TRY(dupload<double>(h, &W.vd_cm1, nullptr, S));
  TRY(dupload<double>(h, &W.vd_div, nullptr, S));
  TRY(dupload<double>(h, &W.vd_ud, nullptr, S));
  TRY(dupload<double>(h, &W.vd_dzdt, nullptr, S));
  if (precision == SHOC_TR_FP64) TRY(dupload<double>(h, &W.vd_rdiv, nullptr, S));
  TRY(dupload<int>(h, &W.sur_t, nullptr, ncol));
  TRY(dupload<int>(h, &W.nsur_t, nullptr, ncol));
  TRY(dupload<ColInfo>(h, &W.col, nullptr, ncol));
  TRY(dupload<shoc_tr_gpu::Readback>(h, &h->d_rb, nullptr, 1));
  W.status = &h->d_rb->status;
  W.dtm_bits = &h->d_rb->dtm;
  W.nwarn = &h->d_rb->nwarn;
  h->d_counts = h->d_rb->counts;
  TRY(dupload<int>(h, &W.serial_list, nullptr, ncol));
  TRY(dupload<int>(h, &W.serial_count, nullptr, 1));
  const bool f32p = precision != SHOC_TR_FP64;
  h->esize = f32p ? sizeof(float) : sizeof(double);
  h->comp = precision == SHOC_TR_FP32_COMP;
  h->staged = true;
  for (int b = 0; b < 2; b++) {
    if (f32p) {
      float *fp = nullptr;
      TRY(dupload<float>(h, &fp, nullptr, (size_t)ntr * S));
      h->tr[b] = fp;
      if (h->comp) TRY(dupload<int16_t>(h, &h->lo[b], nullptr, (size_t)ntr * S));
    } else {
      double *dp2 = nullptr;
      TRY(dupload<double>(h, &dp2, nullptr, (size_t)ntr * S));
      h->tr[b] = dp2;
    }
  }
  if (f32p) {
    TRY(dupload<double>(h, &h->xfer, nullptr, S));
    TRY(dupload<float>(h, &W.dz32, nullptr, S));
    TRY(dupload<float4>(h, &W.lu32, nullptr, S));
    float *fp;
    TRY(dupload<float>(h, &fp, nullptr, S)); h->F3.u1 = fp;
    TRY(dupload<float>(h, &fp, nullptr, S)); h->F3.u2 = fp;
    TRY(dupload<float>(h, &fp, nullptr, S)); h->F3.w = fp;
    if (h->any_hdiff) {
      TRY(dupload<float>(h, &fp, nullptr, S)); h->F3.khx = fp;
      TRY(dupload<float>(h, &fp, nullptr, S)); h->F3.khy = fp;
    }
    // per-column metric factors of the FP32 face values
    std::vector<f32::Face2> ax(S2), ay(S2);
    for (int c2 = 1; c2 < S2; c2++) {
      const Face2D &a = fx[c2], &b = fy[c2];
      ax[c2] = {(float)a.d, (float)(a.db * a.hm), (float)(a.db * a.h0), (float)(a.df * a.h0),
                (float)(a.df * a.hp), a.h0 != 0.0 ? (float)(1.0 / a.h0) : 0.f};
      ay[c2] = {(float)b.d, (float)(b.db * b.hm), (float)(b.db * b.h0), (float)(b.df * b.h0),
                (float)(b.df * b.hp), b.h0 != 0.0 ? (float)(1.0 / b.h0) : 0.f};
    }
    TRY(dupload(h, &h->fx2, ax.data(), S2));
    TRY(dupload(h, &h->fy2, ay.data(), S2));
    // the FP64 mass each column's stored values owe it
    TRY(dupload<double>(h, &h->fu.carry, nullptr, (size_t)ntr * ncol));
  }
  TRY(dupload<double>(h, &h->fzs64, nullptr, (size_t)ntr * ncol));
  TRY(build_tile_tables(h, g, cflag, col_bot, col_kb));
  // tiling: warps per column-kernel block
  const int nd = std::max(1, h->vd_depth.back());
  const int ntile = h->tl.ncolp / 32;
  h->tw = f32p ? vd32_default_warps(nd, h->nslot, h->comp, ntile)
               : vd64_default_warps(nd, h->nslot, ntile);
  h->tw_default = h->tw;
  {  // face columns of the transport-mode preamble
    std::vector<int2> fc;
    std::vector<double> bz;
    bool ok = face_columns(g, g->v3_e1, g->w3_e1, g->xm1, fc, bz);
    const int n1 = (int)fc.size();
    ok = ok && face_columns(g, g->v3_e2, g->w3_e2, g->ym1, fc, bz);
    h->pre.ok = ok;
    if (ok && !fc.empty()) {
      h->pre.n1 = n1;
      h->pre.n2 = (int)fc.size() - n1;
      TRY(dupload(h, &h->pre.fc, fc.data(), fc.size()));
      TRY(dupload(h, &h->pre.bz, bz.data(), bz.size()));
    }
  }
  if (f32p) {
    // the fused sub-step kernel k_step32: every advected tracer's
    // accumulators and the column arrays of up to as many phase-B warps as
    // keep two blocks per SM; tiles of every width the autotuner may choose
    // (not with FP32_COMP: k_step32 keeps no compensation)
    if (o->ntbdy <= kFusedMaxTracers && !h->comp) {
      for (int c = kFusedWarps; c >= 1 && !h->fnwb_max; c--) {
        int gq;
        if (fused_config(h, c, &gq) <= 113 * 1024) h->fnwb_max = c;
      }
    }
    if (h->fnwb_max) {
      int gq;
      if (fused32_set_smem_attr((int)fused_config(h, h->fnwb_max, &gq)) != cudaSuccess)
        TRY(SHOC_TR_ECUDA);
      for (int tx : {8, 16, 32}) TRY(build_fused_tiles(h, g, col_kb, tx, h->ftile[tile_index(tx)]));
    }
    // the two-kernel sub-step is the default (measured faster);
    // SHOC_TR_GPU_KERNELS=fused starts with k_step32 (8 x 4 tiles)
    const char *env = getenv("SHOC_TR_GPU_KERNELS");
    shoc_tr_tuning t0 = current_tuning(h);
    if (env && strcmp(env, "fused") == 0 && h->fnwb_max && !h->comp) {
      t0.fused = 1;
      t0.tile_x = 8;
      t0.phase_b_warps = h->fnwb_max;
    }
    TRY(apply_tuning(h, t0));
  }
  // flow fields
  Flow &F = h->F;
  TRY(dupload<double>(h, (double **)&F.u1, nullptr, S));
  TRY(dupload<double>(h, (double **)&F.u2, nullptr, S));
  TRY(dupload<double>(h, (double **)&F.w, nullptr, S));
  TRY(dupload<double>(h, (double **)&F.u1flux3d, nullptr, S));
  TRY(dupload<double>(h, (double **)&F.u2flux3d, nullptr, S));
  TRY(dupload<double>(h, (double **)&F.Kz, nullptr, S));
  if (f32p) {  // the FP32-mixed kernels take the FP64 volume fluxes
    h->F3.u1flux3d = F.u1flux3d;
    h->F3.u1_64 = F.u1;
    h->F3.u2_64 = F.u2;
    h->F3.u2flux3d = F.u2flux3d;
    h->F3.w64 = F.w;
  }
  if (h->any_hdiff) {
    TRY(dupload<double>(h, (double **)&F.dzu1, nullptr, S));
    TRY(dupload<double>(h, (double **)&F.dzu2, nullptr, S));
    TRY(dupload<double>(h, (double **)&F.u1kh, nullptr, S));
    TRY(dupload<double>(h, (double **)&F.u2kh, nullptr, S));
  }
  TRY(dupload<double>(h, (double **)&F.eta, nullptr, S2));
  TRY(dupload<double>(h, (double **)&F.oldeta, nullptr, S2));
  // pinned readback words
  void *pin = nullptr;
  if (cudaHostAlloc(&pin, 64, cudaHostAllocDefault) != cudaSuccess) TRY(SHOC_TR_ENOMEM);
  h->h_rb = (shoc_tr_gpu::Readback *)pin;
  if (cudaFuncSetAttribute(k_set_dz, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)set_dz_smem(kMaxLayers)) != cudaSuccess ||
      tile64_set_smem_attr() != cudaSuccess ||
      tile32_set_smem_attr() != cudaSuccess)
    TRY(SHOC_TR_ECUDA);
  // the uploads and fills above went to the default stream, which the
  // handle's non-blocking stream does not wait for
  if (default_stream_done() != 0) TRY(SHOC_TR_ECUDA);
#undef TRY
  *out = h;
  return SHOC_TR_OK;
}

}  // extern "C"

namespace {

// Sub-step schedule from the device minimum (tracers.c:591-668, :715-720).
int make_schedule(shoc_tr_gpu *h, double dmin, Sched &s) {
  double dt = h->dt, dtm = dt;
  if (h->O.substep) {
    if (dmin < dtm) dtm = dmin;
    if (dtm != dt) dtm = floor(dtm);
  }
  s.dtm = dtm;
  s.sub.clear();
  if (dtm == 0.0 || (int)(dt / dtm) > kItermax) return SHOC_TR_ESUBSTEP;
  double trem = dt, prev_f = 0.0;
  bool first = true;
  while (trem > 0) {
    double dtu = dtm;
    if (trem < dtu) dtu = trem;
    if (dtu > 0.0) {
      SubStep ss;
      ss.dtu = dtu;
      ss.trem = trem;
      ss.subeta_f = 1.0 + (dtu - trem) / dt;
      ss.osub_f = prev_f;
      ss.first = first ? 1 : 0;
      prev_f = ss.subeta_f;
      first = false;
      s.sub.push_back(ss);
    }
    trem -= dtu;
  }
  return SHOC_TR_OK;
}

// set_lateral_BC_tr for the tracers of T (every tracer, or one chunk of the
// drop-in step's pipeline) into both buffers; reset: clear the step's
// reductions too
void launch_lateral(shoc_tr_gpu *h, int cur, const TrSet &T, bool reset) {
  cudaStream_t st = h->stream;
  if (h->nbpt <= 0 || T.nslot <= 0) {
    if (reset) {
      k_reset<<<1, 32, 0, st>>>(h->W, h->d_counts);
      h->launches++;
    }
    return;
  }
  int *counts = reset ? h->d_counts : nullptr;
  long long tot = (long long)h->nbpt * T.nslot;
  int blocks = (int)std::min<long long>((tot + 255) / 256, 148 * 16);
  if (h->esize == sizeof(float))
    k_lateral<float><<<blocks, 256, 0, st>>>(h->nbpt, h->bpt, h->bin, T.slot_tr, T.nslot, h->S,
                                             (float *)h->tr[cur], (float *)h->tr[cur ^ 1],
                                             h->comp ? h->lo[cur] : nullptr,
                                             h->comp ? h->lo[cur ^ 1] : nullptr, h->W, counts);
  else
    k_lateral<double><<<blocks, 256, 0, st>>>(h->nbpt, h->bpt, h->bin, T.slot_tr, T.nslot,
                                              h->S, (double *)h->tr[cur],
                                              (double *)h->tr[cur ^ 1], nullptr, nullptr, h->W,
                                              counts);
  h->launches++;
}

// k_set_dz over every column; what: SD_PROBE / SD_SEARCH (the arrays to write
// follow from the precision)
void launch_set_dz(shoc_tr_gpu *h, int what) {
  if (h->esize == sizeof(float))
    what |= SD_F32 | (h->comp ? SD_WORK | SD_UD : 0);
  else
    what |= SD_WORK | SD_LU64;
  const int nd = std::max(1, h->vd_depth.back());
  k_set_dz<<<h->tl.ncolp / 32, dim3(32, set_dz_warps(nd)), set_dz_smem(nd), h->stream>>>(
      h->G, h->F, h->W, h->O, h->tl, h->any_vdiff ? 1 : 0, h->d_counts, h->staged ? 1 : 0, what,
      h->colown, nd);
  h->launches++;
}

// The transport-mode flow preamble: dzu1, dzu2, u1flux3d, u2flux3d and w
// from the velocities, the surface and detadt (k_faces, k_wvel), and the
// FP32-mixed path's copies of what changed.
int launch_preamble(shoc_tr_gpu *h) {
  cudaStream_t st = h->stream;
  const size_t S = (size_t)h->S;
  double *f1 = (double *)h->F.u1flux3d, *f2 = (double *)h->F.u2flux3d, *w = (double *)h->F.w;
  double *d1 = (double *)h->F.dzu1, *d2 = (double *)h->F.dzu2;
  k_zero5<<<592, 256, 0, st>>>(f1, f2, w, d1, d2, S);
  h->launches++;
  const int n = h->pre.n1 + h->pre.n2;
  if (n > 0) {
    k_faces<<<(n + 127) / 128, 128, 0, st>>>(h->G, h->F, h->pre.n1, n, h->pre.fc, h->pre.bz, d1,
                                             d2, f1, f2);
    h->launches++;
  }
  k_wvel<<<(h->ncol + 127) / 128, 128, 0, st>>>(h->G, h->F, h->W, h->O, h->tl, h->pre.detadt, w);
  h->launches++;
  if (h->esize == sizeof(float)) {
    k_to_f32<<<592, 256, 0, st>>>(h->F.w, (float *)h->F3.w, S);
    h->launches++;
    if (h->any_hdiff) {
      k_khfac<<<592, 256, 0, st>>>(h->G, h->F, (float *)h->F3.khx, (float *)h->F3.khy);
      h->launches++;
    }
  }
  CK(cudaGetLastError());
  return 0;
}

// Step set-up: counters, lateral boundaries (when `lateral`), the flow
// preamble (when on) and k_set_dz (with the sub-step search when `search`:
// a step whose schedule is known does not need it).  k_set_dz reads no tracer,
// so the lateral copies may follow it instead.
int launch_part_a(shoc_tr_gpu *h, int cur, bool lateral, bool search) {
  cudaStream_t st = h->stream;
  if (lateral) {
    launch_lateral(h, cur, h->T, true);
  } else {
    k_reset<<<1, 32, 0, st>>>(h->W, h->d_counts);
    h->launches++;
  }
  if (h->pre.on) {
    const int rc = launch_preamble(h);
    if (rc) return rc;
  }
  launch_set_dz(h, search ? SD_SEARCH : 0);
  CK(cudaGetLastError());
  return 0;
}

// One sub-step of the general-path columns for the tracers of T
template <class TR>
void launch_general(shoc_tr_gpu *h, bool last, const TrSet &T, const SubStep &ss, const TR *tin,
                    TR *tout, uint8_t *c3row, bool c3_load, int16_t *lo_out) {
  // as many threads as the longest list has (column, tracer) pairs, at most
  // eight blocks per SM
  const long long tot = (long long)(h->ncol + 31) / 32 * 32 * T.nslot;
  const int blocks = (int)std::min<long long>((tot + kGeneralThreads - 1) / kGeneralThreads,
                                              kGeneralBlocks);
  if (last)
    k_general<true, TR><<<blocks, kGeneralThreads, 0, h->stream>>>(
        h->G, h->F, h->W, h->O, T, ss, h->tl, tin, tout, c3row, c3_load, lo_out);
  else
    k_general<false, TR><<<blocks, kGeneralThreads, 0, h->stream>>>(
        h->G, h->F, h->W, h->O, T, ss, h->tl, tin, tout, c3row, c3_load, lo_out);
  h->launches++;
}

// The launches of the column kernel for nslot tracers and nw warps a block: one,
// with the shared memory the window's deepest tile needs, whose shallower tiles use
// theirs up with more warps.  Where the tracers are too few for that and an SM
// would hold four warps or less of its 16, the shallower tiles may be launched by
// themselves, with twice the warps an SM.  That gains the time they take off the
// deep launch, and loses what they filled beside its last deep tiles, about half a
// deep tile's time: in units of a layer's time, the tiles' layers over 148 SMs times
// the rounds of tracers per resident block, before less after, against half the
// deepest tile's layers and rounds.  (150 x 120 x 128 of any depth, 3 tracers
// FP32-mixed: 326 us a step in one launch, 405 in three.  From six warps an SM on the
// shallow launch gained nothing: 400 x 300 x 60, half of it 18 layers at most, 3
// tracers 432 and 460.)
// 400 x 300, 60 layers of which the columns have 8 at most, 1 tracer: the kernel
// takes 25 us FP32-mixed and 27 FP64, 70 and 93 with memory for 60 layers; 300 x
// 200, 128 layers on 3 % of the columns and 18 at most on the others 167 and 168 us,
// 279 and 275 in one launch.
constexpr int kColLaunches = 4;
int col_launches(const shoc_tr_gpu *h, int nslot, int nw, ColLaunch *out) {
  const bool f32 = h->esize == sizeof(float);
  const int full = kVd32MaxWarps;
  static_assert(kVd32MaxWarps == kVd64MaxWarps, "one rule for both column kernels");
  auto config = [&](int depth, int &blocks) {
    ColLaunch l{};
    const size_t need = f32 ? vd32_smem(depth, nw, h->vd_pf, h->comp) : vd64_smem(depth, nw);
    l.bytes = (int)std::min<size_t>(need, 227 * 1024);
    blocks = std::max(1, 233472 / (l.bytes + 1024));
    l.warps = std::max(1, std::min(nslot, std::max(nw, full / blocks)));
    return l;
  };
  const std::vector<int> &depth = h->vd_depth;
  int n = 0, hi = (int)depth.size();
  while (hi > 0) {
    int blocks, b;
    ColLaunch l = config(std::max(1, depth[hi - 1]), blocks);
    int lo = 0;
    if (n + 1 < kColLaunches)
      for (int d = depth[hi - 1] - 1; d >= 1 && !lo; d--) {
        if (blocks * l.warps > 4) break;
        const ColLaunch s = config(d, b);
        if (std::min(full, b * s.warps) < 2 * std::min(full, blocks * l.warps)) continue;
        lo = (int)(std::upper_bound(depth.begin(), depth.begin() + hi, d) - depth.begin());
        if (lo == 0) break;
        const ColLaunch t = config(std::max(1, depth[lo - 1]), b);
        auto rounds = [&](int w) { return (nslot + w - 1) / w; };
        const double gain = h->vd_layers[lo] / 148.0 * ((double)rounds(l.warps) / blocks -
                                            (double)rounds(t.warps) / b);
        if (gain <= 0.5 * depth[hi - 1] * rounds(std::max(nw, 1))) lo = 0;
        break;
      }
    l.tile0 = lo;
    l.ntile = hi - lo;
    out[n++] = l;
    hi = lo;
  }
  return n;
}

// One FP64 transport sub-step over the staged columns: k_adv64, then k_vd64.
// Returns the kernels launched.
//
template <int SCH, bool U>
void adv64(const shoc_tr_gpu *h, const SubStep &ss, const Tile &tl, const TrSet &T,
           const double *tin, double *tout) {
  const int ng = std::min(T.ntb, kAdv64Group), groups = (T.ntb + ng - 1) / ng;
  const shoc_tr_gpu::AdvItems &it = h->adv_items[groups - 1];
  const dim3 grid((it.n + kAdv64Warps - 1) / kAdv64Warps, groups);
  const size_t smem = adv64_smem(ng);
  if (h->adv_flags == 1)
    k_adv64<SCH, U, true><<<grid, kAdv64Warps * 32, smem, h->stream>>>(
        h->G, h->F, h->W, T, ss, tl, tin, tout, h->fzs64, it.d, it.n, ng);
  else
    k_adv64<SCH, U, false><<<grid, kAdv64Warps * 32, smem, h->stream>>>(
        h->G, h->F, h->W, T, ss, tl, tin, tout, h->fzs64, it.d, it.n, ng);
}
template <int SCH>
void adv64_ult(const shoc_tr_gpu *h, const SubStep &ss, const Tile &tl, const TrSet &T,
               const double *tin, double *tout) {
  if (h->O.ultimate)
    adv64<SCH, true>(h, ss, tl, T, tin, tout);
  else
    adv64<SCH, false>(h, ss, tl, T, tin, tout);
}
static_assert(kAdv64Warps * (kAdv64Faces * FC_N + kAdv64Group) * 32 * 8 <= 48 * 1024,
              "k_adv64 stays below the opt-in shared memory size");
cudaError_t tile64_set_smem_attr() {
  const cudaError_t r[] = {
      cudaFuncSetAttribute(k_vd64<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024),
      cudaFuncSetAttribute(k_vd64<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           227 * 1024)};
  for (auto x : r)
    if (x != cudaSuccess) return x;
  return cudaSuccess;
}
int tile64_substep(const shoc_tr_gpu *h, bool last, const SubStep &ss, const Tile &tl,
                   const TrSet &T, const double *tin, double *tout, int nw, cudaEvent_t *ev) {
  cudaStream_t st = h->stream;
  int nl = 0;
  if (ev) cudaEventRecord(ev[0], st);
  if (T.ntb > 0 && tl.nwet > 0) {
    switch (h->O.trasc) {
      case SHOC_TR_QUICKEST: adv64_ult<SHOC_TR_QUICKEST>(h, ss, tl, T, tin, tout); break;
      case SHOC_TR_VANLEER: adv64_ult<SHOC_TR_VANLEER>(h, ss, tl, T, tin, tout); break;
      case SHOC_TR_ORDER1: adv64_ult<SHOC_TR_ORDER1>(h, ss, tl, T, tin, tout); break;
      case SHOC_TR_ORDER2: adv64_ult<SHOC_TR_ORDER2>(h, ss, tl, T, tin, tout); break;
      case SHOC_TR_ORDER4: adv64_ult<SHOC_TR_ORDER4>(h, ss, tl, T, tin, tout); break;
      case SHOC_TR_QUICKEST_CO: adv64_ult<SHOC_TR_QUICKEST_CO>(h, ss, tl, T, tin, tout); break;
      case SHOC_TR_ORDER2_UW: adv64_ult<SHOC_TR_ORDER2_UW>(h, ss, tl, T, tin, tout); break;
    }
    nl++;
    if (tl.napart > 0) {
      const int blocks = (int)std::min<long long>(((long long)tl.napart * T.ntb + 127) / 128,
                                                  kGeneralBlocks);
      k_adv64_apart<<<blocks, 128, 0, st>>>(h->G, h->F, h->W, h->O, T, ss, tl, tin, tout);
      nl++;
    }
  }
  if (ev) cudaEventRecord(ev[1], st);
  ColLaunch cl[kColLaunches];
  const int ncl = col_launches(h, T.nslot, nw, cl);
  for (int i = 0; i < ncl; i++) {
    auto kern = last ? k_vd64<true> : k_vd64<false>;
    kern<<<cl[i].ntile, dim3(32, cl[i].warps), cl[i].bytes, st>>>(
        h->G, h->F, h->W, h->O, T, ss, tl, tin, tout, h->fzs64, cl[i].bytes, cl[i].tile0);
  }
  nl += ncl;
  if (ev) cudaEventRecord(ev[2], st);
  return nl;
}

// The transport sub-steps of one step for the tracers of T (every tracer, or
// one chunk of the drop-in step's pipeline; c3s/c3_load as k_general takes
// them, one row of ncol bytes per sub-step).
int launch_part_b(shoc_tr_gpu *h, const Sched &s, int cur0, const TrSet &T,
                  uint8_t *c3s = nullptr, bool c3_load = false) {
  cudaStream_t st = h->stream;
  int cur = cur0;
  const int nsub = (int)s.sub.size();
  const int tw = std::max(1, std::min(h->tw, T.nslot));  // no idle tracer rows
  for (int i = 0; i < nsub; i++) {
    const SubStep &ss = s.sub[i];
    bool last = (i == nsub - 1);
    uint8_t *c3row = c3s ? c3s + (size_t)i * h->ncol : nullptr;
    if (h->esize == sizeof(float) && T.nslot > 0) {  // FP32-mixed
      const float *tin = (const float *)h->tr[cur];
      float *tout = (float *)h->tr[cur ^ 1];
      bool prof = h->profile && last;
      cudaEvent_t ev[3] = {nullptr, nullptr, nullptr};
      if (prof)
        for (auto &e : ev) cudaEventCreate(&e);
      if (h->fused) {
        if (prof) cudaEventRecord(ev[0], st);
        fused32_substep(last, h->O.trasc == SHOC_TR_QUICKEST, h->O.ultimate != 0, st, h->G, h->F,
                        h->F3, h->W, h->O, T, ss, h->tl, h->fu, h->fx2, h->fy2, tin, tout,
                        h->any_hdiff ? 1 : 0, h->fused_bytes);
        if (prof) {
          cudaEventRecord(ev[1], st);
          h->ev.push_back({0, ev[0], ev[1]});
          h->ev.push_back({1, ev[0], ev[1]});
          cudaEventDestroy(ev[2]);
        }
        h->launches += h->fu.ntile > 0 ? 1 : 0;
      } else {
        ColLaunch cl[kColLaunches];
        const int ncl = col_launches(h, T.nslot, tw, cl);
        tile32_substep(last, h->O.trasc == SHOC_TR_QUICKEST, h->O.ultimate != 0, st, h->G, h->F,
                       h->F3, h->W, h->O, T, ss, h->tl, h->fx2, h->fy2, tin, tout, h->rnd,
                       h->fu.carry, h->fzs64, h->comp ? h->lo[cur] : nullptr,
                       h->comp ? h->lo[cur ^ 1] : nullptr, cl, ncl, h->vd_pf ? 1 : 0,
                       h->any_hdiff ? 1 : 0, h->adv_flags, prof ? ev : nullptr);
        if (prof) {  // pairs share events; sync destroys each event once
          h->ev.push_back({0, ev[0], ev[2]});
          h->ev.push_back({1, ev[0], ev[1]});
          h->ev.push_back({2, ev[1], ev[2]});
        }
        h->launches += (h->tl.nwet > 0 ? (T.ntb + kMaxTracers - 1) / kMaxTracers : 0) + ncl;
      }
      int16_t *lo_out = h->comp ? h->lo[cur ^ 1] : nullptr;
      launch_general<float>(h, last, T, ss, tin, tout, c3row, c3_load, lo_out);
      cur ^= 1;
      continue;
    }
    const double *tin = (const double *)h->tr[cur];
    double *tout = (double *)h->tr[cur ^ 1];
    if (T.nslot > 0) {
      bool prof = h->profile && last;
      cudaEvent_t ev[3] = {nullptr, nullptr, nullptr};
      if (prof)
        for (auto &e : ev) cudaEventCreate(&e);
      const int nl = tile64_substep(h, last, ss, h->tl, T, tin, tout, tw, prof ? ev : nullptr);
      if (prof) {
        h->ev.push_back({0, ev[0], ev[2]});
        h->ev.push_back({1, ev[0], ev[1]});
        h->ev.push_back({2, ev[1], ev[2]});
      }
      h->launches += nl;
      launch_general<double>(h, last, T, ss, tin, tout, c3row, c3_load, nullptr);
    }
    cur ^= 1;
  }
  CK(cudaGetLastError());
  return 0;
}

int read_status(shoc_tr_gpu *h) {
  CK(cudaMemcpyAsync(h->h_rb, h->d_rb, sizeof(*h->h_rb), cudaMemcpyDeviceToHost, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  return 0;
}

// Part A of a step whose sub-step schedule is not known yet, then the
// sub-step minimum read back and the schedule built from it (tracers.c:
// 591-720).  lateral: whether part A fills every tracer's lateral boundary.
int probe_schedule(shoc_tr_gpu *h, bool lateral, Sched &s) {
  int rc = launch_part_a(h, h->cur, lateral, true);
  if (rc) return rc;
  rc = read_status(h);
  if (rc) return rc;
  int st = h->h_rb->status;
  if (st & (ST_LASTDRY | ST_GEOM)) {
    h->last_status = map_status(st);
    return h->last_status;
  }
  double dmin;
  unsigned long long b = h->h_rb->dtm;
  memcpy(&dmin, &b, 8);
  if (h->dmin_set > 0.0) dmin = h->dmin_set;  // the basin-wide minimum, given
  rc = make_schedule(h, dmin, s);
  if (rc) h->last_status = rc;
  return rc;
}

// Keep a probed schedule for the graph-replayed steps; graphs made for
// another schedule are dropped.
void adopt_schedule(shoc_tr_gpu *h, const Sched &s) {
  bool same = h->have_sched && s.sub.size() == h->sched.sub.size();
  if (same)
    for (size_t i = 0; i < s.sub.size(); i++)
      if (memcmp(&s.sub[i], &h->sched.sub[i], sizeof(SubStep)) != 0) same = false;
  if (!same) {
    for (int i = 0; i < 2; i++)
      if (h->graph[i]) {
        cudaGraphExecDestroy(h->graph[i]);
        h->graph[i] = nullptr;
      }
  }
  h->sched = s;
  h->have_sched = true;
  if (h->probe_left > 0) h->probe_left--;
}

// One step.  When the schedule is not yet known the step synchronises after
// k_set_dz to read the sub-step minimum; afterwards steps replay a graph.
int step_async(shoc_tr_gpu *h) {
  if (h->probe_left > 0 || !h->have_sched) {
    Sched s;
    int rc = probe_schedule(h, true, s);
    if (rc) return rc;
    rc = launch_part_b(h, s, h->cur, h->T);
    if (rc) return rc;
    if (s.sub.size() & 1) h->cur ^= 1;
    adopt_schedule(h, s);
    return 0;
  }
  if (h->profile) {
    // profiling launches directly so each transport launch is timed
    int rc = launch_part_a(h, h->cur, true, false);
    if (rc) return rc;
    rc = launch_part_b(h, h->sched, h->cur, h->T);
    if (rc) return rc;
    if (h->sched.sub.size() & 1) h->cur ^= 1;
    return 0;
  }
  int gi = h->cur;
  if (!h->graph[gi]) {
    // An odd number of sub-steps alternates the buffers from step to step:
    // both graphs are captured and uploaded together, so no later step pays
    // for a capture or a first upload.
    const int ng = (h->sched.sub.size() & 1) ? 2 : 1;
    for (int k = 0; k < ng; ++k) {
      const int g = gi ^ k;
      if (h->graph[g]) continue;
      cudaGraph_t graph;
      long long l0 = h->launches;
      CK(cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal));
      int rc = launch_part_a(h, g, true, false);
      if (!rc) rc = launch_part_b(h, h->sched, g, h->T);
      cudaError_t e = cudaStreamEndCapture(h->stream, &graph);
      if (rc) return rc;
      CK(e);
      CK(cudaGraphInstantiate(&h->graph[g], graph, 0));
      cudaGraphDestroy(graph);
      CK(cudaGraphUpload(h->graph[g], h->stream));
      h->graph_launches[g] = h->launches - l0;  // kernels in the graph
      h->launches = l0;
    }
  }
  CK(cudaGraphLaunch(h->graph[gi], h->stream));
  h->launches += h->graph_launches[gi];
  if (h->sched.sub.size() & 1) h->cur ^= 1;
  return 0;
}

// ---------------------------------------------------------------------------
// The drop-in step on host arrays, pipelined.  The tracers cross the host
// link in chunks of slots: chunk j goes up on one copy stream, is stepped on
// the main stream and comes back on a second copy stream, so the way back of
// chunk j overlaps the way up of the chunks after it (the link is full
// duplex) and every chunk's transport overlaps both.  Per tracer the kernels
// and their order are those of a whole step: the tracers of a step are
// independent apart from the general path's thin-surface cursor, which
// k_general carries from chunk to chunk (c3s); set_dz reads no tracer, so the
// lateral boundaries of a chunk may follow it.

// Slots of each chunk.  The first chunk should be back on its way early and the
// last one's step and copy back, which nothing overlaps, should be short: a 24th
// of the tracers.  In between, a chunk's step costs the faces and factors of
// every cell once more, whatever the number of its tracers, which the link hides
// from two tracers on; a chunk larger than that, or than a twelfth, only keeps
// the way back waiting.  But launching a chunk costs the host as much as some MB
// on the link, so where the tracers are small it takes more of them, up to a
// third.  The chunks double from the first size to that one, and shrink again.
// A call (B200), by the middle chunks: 256 x 256 x 40, 10 tracers, FP64 one
// tracer 5.55 ms, two 4.69, four 5.00; 400 x 400 x 40, 12, FP64 one 13.6, two 11.8;
// 1024 x 512 x 50, 24, FP32-mixed two 76.4, twelve 92.2 (first chunk two 76.8);
// 160 x 150 x 30, 24, FP64 (3 MB each) two 2.88, six 3.30; 100 x 90 x 30, 24, FP64
// (1.3 MB) two 1.47, four 1.42, eight 1.58.
// Twelfths throughout, with the arrived tracers' copies on the link's stream,
// took 6.13, 14.0, 76.8, 3.55 and 1.92 ms.  A window whose tracers cross the link
// in tens of microseconds goes as one chunk: the launches of each cost as much
// (20 x 14 x 6, 3 tracers: 258 us as three, 220 as one).
constexpr size_t kChunkGrow = (size_t)4 << 20;
std::vector<int> pipe_chunks(const shoc_tr_gpu *h) {
  const int n = h->nslot;
  if (n == 0) return {};
  const size_t bytes = (size_t)h->S * sizeof(double);
  if (n * bytes <= (size_t)2 << 20) return {n};
  std::vector<int> left, right;
  const int most = std::max({2, (n + 11) / 12,
                             std::min(n / 3, (int)((kChunkGrow + bytes - 1) / bytes))});
  for (int c = (n + 23) / 24, rest = n; rest > 0; c = std::min(2 * c, most)) {
    if (rest < 2 * c) {  // the middle
      left.push_back(rest);
      break;
    }
    left.push_back(c);
    right.push_back(c);
    rest -= 2 * c;
  }
  left.insert(left.end(), right.rbegin(), right.rend());
  return left;
}

int pipe_init(shoc_tr_gpu *h) {
  if (h->pipe_ready) return 0;
  for (cudaStream_t *x : {&h->s_up, &h->s_cv, &h->s_dn})
    if (!*x) CK(cudaStreamCreateWithFlags(x, cudaStreamNonBlocking));
  int rc = 0;
  if (h->esize == sizeof(float)) {
    if (!h->xout && (rc = dalloc(h, &h->xout, (size_t)h->S))) return rc;
    h->xup[0] = h->xfer;
    if (!h->xup[1] && (rc = dalloc(h, &h->xup[1], (size_t)h->S))) return rc;
  }
  if (!h->c3s && (rc = dalloc(h, &h->c3s, (size_t)(kItermax + 2) * h->ncol))) return rc;
  if (!h->h_surf &&
      cudaHostAlloc((void **)&h->h_surf, 2 * ((size_t)h->ncol + 1) * sizeof(int),
                    cudaHostAllocDefault) != cudaSuccess) {
    cudaGetLastError();
    h->h_surf = nullptr;
    return SHOC_TR_ENOMEM;
  }
  h->pev.resize(1 + 2 * (size_t)h->nslot, nullptr);
  for (auto &e : h->pev)
    if (!e) CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  for (cudaEvent_t *e : {&h->ev_in[0], &h->ev_in[1], &h->ev_cv[0], &h->ev_cv[1]})
    if (!*e) CK(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
  h->pipe_ready = true;
  return 0;
}

// wait for every copy that may still touch the caller's host arrays
void pipe_drain(shoc_tr_gpu *h) {
  cudaStreamSynchronize(h->s_up);
  cudaStreamSynchronize(h->s_cv);
  cudaStreamSynchronize(h->s_dn);
  cudaStreamSynchronize(h->stream);
}

// Tracer n, the i-th of the call, up the link on s_up; what it needs on the
// device then (the copy into the other ping-pong buffer, the conversion) runs on
// s_cv, so that the link does not wait for it (FP32-mixed: two buffers for the
// arriving FP64 values).
int up_tracer(shoc_tr_gpu *h, int cur, int i, int n, const double *src) {
  const size_t S = (size_t)h->S;
  const int b = i & 1;
  if (h->esize == sizeof(double)) {
    double *p = (double *)h->tr[cur] + n * S, *q = (double *)h->tr[cur ^ 1] + n * S;
    CK(cudaMemcpyAsync(p, src, S * sizeof(double), cudaMemcpyHostToDevice, h->s_up));
    CK(cudaEventRecord(h->ev_in[b], h->s_up));
    CK(cudaStreamWaitEvent(h->s_cv, h->ev_in[b], 0));
    CK(cudaMemcpyAsync(q, p, S * sizeof(double), cudaMemcpyDeviceToDevice, h->s_cv));
  } else {
    float *p = (float *)h->tr[cur] + n * S, *q = (float *)h->tr[cur ^ 1] + n * S;
    if (i >= 2) CK(cudaStreamWaitEvent(h->s_up, h->ev_cv[b], 0));
    CK(cudaMemcpyAsync(h->xup[b], src, S * sizeof(double), cudaMemcpyHostToDevice, h->s_up));
    CK(cudaEventRecord(h->ev_in[b], h->s_up));
    CK(cudaStreamWaitEvent(h->s_cv, h->ev_in[b], 0));
    k_to_f32x2<<<592, 256, 0, h->s_cv>>>(h->xup[b], p, q, S,
                                         h->comp ? h->lo[cur] + n * S : nullptr,
                                         h->comp ? h->lo[cur ^ 1] + n * S : nullptr);
    h->launches++;
    CK(cudaEventRecord(h->ev_cv[b], h->s_cv));
  }
  return 0;
}

int down_tracer(shoc_tr_gpu *h, int buf, int n, double *dst) {
  cudaStream_t s = h->s_dn;
  const size_t S = (size_t)h->S;
  if (h->esize == sizeof(double)) {
    CK(cudaMemcpyAsync(dst, (double *)h->tr[buf] + n * S, S * sizeof(double),
                       cudaMemcpyDeviceToHost, s));
  } else {
    k_to_f64<<<592, 256, 0, s>>>((float *)h->tr[buf] + n * S, h->xout, S,
                                 h->comp ? h->lo[buf] + n * S : nullptr);
    h->launches++;
    CK(cudaMemcpyAsync(dst, h->xout, S * sizeof(double), cudaMemcpyDeviceToHost, s));
  }
  return 0;
}

int step_pipelined(shoc_tr_gpu *h, shoc_tr_state *st) {
  int rc = pipe_init(h);
  if (rc) return rc;
  // the surface vectors go through page-locked memory (the caller's copies of
  // them are rarely registered)
  shoc_tr_state fl = *st;
  if (st->sur_t && st->nsur_t) {
    const size_t nb = (size_t)h->ncol * sizeof(int);  // elements 1 to ncol
    memcpy(h->h_surf + 1, st->sur_t + 1, nb);
    memcpy(h->h_surf + 1 + h->ncol + 1, st->nsur_t + 1, nb);
    fl.sur_t = h->h_surf;
    fl.nsur_t = h->h_surf + h->ncol + 1;
  }
  rc = shoc_tr_gpu_set_flow(h, &fl);
  if (rc) return rc;
  const int cur = h->cur;
  const std::vector<int> chunk = pipe_chunks(h);
  const int nch = (int)chunk.size();
  cudaEvent_t *ev = h->pev.data();  // [0] flow sent, [1 + 2j] chunk j sent, [2 + 2j] stepped
  // the tracers follow the flow fields up the link
  CK(cudaEventRecord(ev[0], h->stream));
  CK(cudaStreamWaitEvent(h->s_up, ev[0], 0));
  int up = 0;
  for (int j = 0, sl = 0; j < nch; j++) {
    for (const int end = sl + chunk[j]; sl < end; sl++) {
      const int n = h->slot_host[sl];
      rc = up_tracer(h, cur, up++, n, st->tr_wc[n]);
      if (rc) {
        pipe_drain(h);
        return rc;
      }
    }
    CK(cudaEventRecord(ev[1 + 2 * j], h->s_cv));
  }
  // the schedule from this step's flow, while the tracers travel
  Sched s;
  rc = probe_schedule(h, false, s);
  if (!rc && s.sub.size() > (size_t)kItermax + 2) rc = SHOC_TR_ESUBSTEP;
  if (rc) {
    pipe_drain(h);
    return rc;
  }
  const int fin = cur ^ (int)(s.sub.size() & 1);  // the buffer the step ends in
  for (int j = 0, s0 = 0; j < nch; s0 += chunk[j++]) {
    const int ns = chunk[j];
    TrSet Tc = h->T;
    Tc.slot_tr = h->T.slot_tr + s0;
    Tc.nslot = ns;
    Tc.ntb = std::max(0, std::min(h->T.ntb - s0, ns));
    CK(cudaStreamWaitEvent(h->stream, ev[1 + 2 * j], 0));
    launch_lateral(h, cur, Tc, false);
    rc = launch_part_b(h, s, cur, Tc, h->c3s, j > 0);
    if (rc) {
      pipe_drain(h);
      return rc;
    }
    CK(cudaEventRecord(ev[2 + 2 * j], h->stream));
    CK(cudaStreamWaitEvent(h->s_dn, ev[2 + 2 * j], 0));
    for (int sl = s0; sl < s0 + ns; sl++) {
      const int n = h->slot_host[sl];
      rc = down_tracer(h, fin, n, st->tr_wc[n]);
      if (rc) {
        pipe_drain(h);
        return rc;
      }
    }
  }
  // the main stream (and so the status read after it) waits for the way back
  CK(cudaEventRecord(ev[0], h->s_dn));
  CK(cudaStreamWaitEvent(h->stream, ev[0], 0));
  h->cur = fin;
  adopt_schedule(h, s);
  return 0;
}

}  // namespace

extern "C" {

int shoc_tr_gpu_upload_tracers(shoc_tr_gpu *h, double *const *tr_wc) {
  if (!h || !tr_wc) return SHOC_TR_EARG;
  DeviceScope dev_(h->device);
  const size_t S = (size_t)h->S;
  // new values: nothing is owed to any column
  if (h->fu.carry)
    CK(cudaMemsetAsync(h->fu.carry, 0, (size_t)h->ntr * h->ncol * sizeof(double), h->stream));
  for (int n = 0; n < h->ntr; n++) {
    if (h->esize == sizeof(double)) {
      double *a = (double *)h->tr[h->cur] + n * S, *b = (double *)h->tr[h->cur ^ 1] + n * S;
      CK(cudaMemcpyAsync(a, tr_wc[n], S * sizeof(double), cudaMemcpyHostToDevice, h->stream));
      CK(cudaMemcpyAsync(b, a, S * sizeof(double), cudaMemcpyDeviceToDevice, h->stream));
    } else {
      float *a = (float *)h->tr[h->cur] + n * S, *b = (float *)h->tr[h->cur ^ 1] + n * S;
      CK(cudaMemcpyAsync(h->xfer, tr_wc[n], S * sizeof(double), cudaMemcpyHostToDevice,
                         h->stream));
      k_to_f32x2<<<592, 256, 0, h->stream>>>(h->xfer, a, b, S,
                                             h->comp ? h->lo[h->cur] + n * S : nullptr,
                                             h->comp ? h->lo[h->cur ^ 1] + n * S : nullptr);
      h->launches++;
    }
  }
  return 0;
}

int shoc_tr_gpu_download_tracers(shoc_tr_gpu *h, double **tr_wc) {
  if (!h || !tr_wc) return SHOC_TR_EARG;
  DeviceScope dev_(h->device);
  const size_t S = (size_t)h->S;
  for (int n = 0; n < h->ntr; n++) {
    if (h->esize == sizeof(double)) {
      CK(cudaMemcpyAsync(tr_wc[n], (double *)h->tr[h->cur] + n * S, S * sizeof(double),
                         cudaMemcpyDeviceToHost, h->stream));
    } else {
      k_to_f64<<<592, 256, 0, h->stream>>>((float *)h->tr[h->cur] + n * S, h->xfer, S,
                                           h->comp ? h->lo[h->cur] + n * S : nullptr);
      h->launches++;
      CK(cudaMemcpyAsync(tr_wc[n], h->xfer, S * sizeof(double), cudaMemcpyDeviceToHost,
                         h->stream));
    }
  }
  CK(cudaStreamSynchronize(h->stream));
  return 0;
}

int shoc_tr_gpu_set_flow(shoc_tr_gpu *h, const shoc_tr_state *st) {
  if (!h || !st) return SHOC_TR_EARG;
  DeviceScope dev_(h->device);
  const size_t S = (size_t)h->S * sizeof(double), S2 = (size_t)h->S2 * sizeof(double);
  cudaStream_t s = h->stream;
  // with the flow preamble on, w, u1flux3d, u2flux3d, dzu1 and dzu2 are
  // computed by every step and not read from the state (they may be null)
  const bool pre = h->pre.on;
  const struct {
    const double *dst;
    const double *src;
    size_t n;
    bool need;
  } cp[] = {{h->F.u1, st->u1, S, true},
            {h->F.u2, st->u2, S, true},
            {h->F.w, st->w, S, !pre},
            {h->F.u1flux3d, st->u1flux3d, S, !pre},
            {h->F.u2flux3d, st->u2flux3d, S, !pre},
            {h->F.Kz, st->Kz, S, true},
            {h->F.eta, st->eta, S2, true},
            {h->F.oldeta, st->oldeta, S2, true}};
  for (auto &x : cp) {
    if (!x.need) continue;
    if (!x.src) return SHOC_TR_EARG;
    CK(cudaMemcpyAsync((void *)x.dst, x.src, x.n, cudaMemcpyHostToDevice, s));
  }
  if (h->any_hdiff) {
    if ((!pre && (!st->dzu1 || !st->dzu2)) || !st->u1kh || !st->u2kh) return SHOC_TR_EARG;
    if (!pre) {
      CK(cudaMemcpyAsync((void *)h->F.dzu1, st->dzu1, S, cudaMemcpyHostToDevice, s));
      CK(cudaMemcpyAsync((void *)h->F.dzu2, st->dzu2, S, cudaMemcpyHostToDevice, s));
    }
    CK(cudaMemcpyAsync((void *)h->F.u1kh, st->u1kh, S, cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync((void *)h->F.u2kh, st->u2kh, S, cudaMemcpyHostToDevice, s));
  }
  if (h->esize == sizeof(float)) {
    const size_t n = (size_t)h->S;
    k_to_f32<<<592, 256, 0, s>>>(h->F.u1, (float *)h->F3.u1, n);
    k_to_f32<<<592, 256, 0, s>>>(h->F.u2, (float *)h->F3.u2, n);
    h->launches += 2;
    if (!pre) {
      k_to_f32<<<592, 256, 0, s>>>(h->F.w, (float *)h->F3.w, n);
      h->launches++;
    }
    if (h->any_hdiff && !pre) {
      k_khfac<<<592, 256, 0, s>>>(h->G, h->F, (float *)h->F3.khx, (float *)h->F3.khy);
      h->launches++;
    }
    CK(cudaGetLastError());
  }
  if (st->sur_t && st->nsur_t) {
    CK(cudaMemcpyAsync(h->W.sur_t, st->sur_t + 1, (size_t)h->ncol * sizeof(int),
                       cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(h->W.nsur_t, st->nsur_t + 1, (size_t)h->ncol * sizeof(int),
                       cudaMemcpyHostToDevice, s));
  }
  if (st->dt != h->dt) {
    h->dt = st->dt;
    h->F.dt = st->dt;
    for (int i = 0; i < 2; i++)
      if (h->graph[i]) {
        cudaGraphExecDestroy(h->graph[i]);
        h->graph[i] = nullptr;
      }
    h->have_sched = false;
  }
  h->probe_left = 2;
  return 0;
}

int shoc_tr_gpu_get_surface(shoc_tr_gpu *h, int *sur_t, int *nsur_t) {
  if (!h) return SHOC_TR_EARG;
  DeviceScope dev_(h->device);
  if (sur_t)
    CK(cudaMemcpyAsync(sur_t + 1, h->W.sur_t, (size_t)h->ncol * sizeof(int),
                       cudaMemcpyDeviceToHost, h->stream));
  if (nsur_t)
    CK(cudaMemcpyAsync(nsur_t + 1, h->W.nsur_t, (size_t)h->ncol * sizeof(int),
                       cudaMemcpyDeviceToHost, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  return 0;
}

int shoc_tr_gpu_set_preamble(shoc_tr_gpu *h, int on) {
  if (!h) return SHOC_TR_EARG;
  if (on && !h->pre.ok) return SHOC_TR_EUNSUPPORTED;
  DeviceScope dev_(h->device);
  if (on) {
    // only what is made here is filled on the default stream and waited for: the
    // call must not wait for the caller's own work there every step
    const bool made = !h->F.dzu1 || !h->F.dzu2 || !h->pre.detadt;
    int rc = 0;
    if (!rc && !h->F.dzu1) rc = dupload<double>(h, (double **)&h->F.dzu1, nullptr, (size_t)h->S);
    if (!rc && !h->F.dzu2) rc = dupload<double>(h, (double **)&h->F.dzu2, nullptr, (size_t)h->S);
    if (!rc && !h->pre.detadt) rc = dupload<double>(h, &h->pre.detadt, nullptr, (size_t)h->S2);
    if (!rc && made) rc = default_stream_done();
    if (rc) return rc;
  }
  if (h->pre.on != (on != 0)) {
    h->pre.on = on != 0;
    for (int i = 0; i < 2; i++)  // the captured steps hold the old part A
      if (h->graph[i]) {
        cudaGraphExecDestroy(h->graph[i]);
        h->graph[i] = nullptr;
      }
    h->probe_left = std::max(h->probe_left, 1);  // w, and so the sub-steps, change
  }
  return SHOC_TR_OK;
}

int shoc_tr_gpu_set_detadt(shoc_tr_gpu *h, const double *detadt) {
  if (!h || !detadt) return SHOC_TR_EARG;
  if (!h->pre.detadt) return SHOC_TR_EARG;  // the preamble was never enabled
  DeviceScope dev_(h->device);
  CK(cudaMemcpyAsync(h->pre.detadt, detadt, (size_t)h->S2 * sizeof(double),
                     cudaMemcpyHostToDevice, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  return SHOC_TR_OK;
}

int shoc_tr_gpu_get_flow(shoc_tr_gpu *h, double *u1flux3d, double *u2flux3d, double *w,
                         double *dzu1, double *dzu2) {
  if (!h) return SHOC_TR_EARG;
  DeviceScope dev_(h->device);
  const size_t S = (size_t)h->S * sizeof(double);
  const struct {
    double *dst;
    const double *src;
  } cp[] = {{u1flux3d, h->F.u1flux3d}, {u2flux3d, h->F.u2flux3d}, {w, h->F.w},
            {dzu1, h->F.dzu1}, {dzu2, h->F.dzu2}};
  for (auto &x : cp) {
    if (!x.dst) continue;
    if (!x.src) return SHOC_TR_EARG;  // dzu1 / dzu2: neither uploaded nor computed
    CK(cudaMemcpyAsync(x.dst, x.src, S, cudaMemcpyDeviceToHost, h->stream));
  }
  CK(cudaStreamSynchronize(h->stream));
  return SHOC_TR_OK;
}

// ---- checkpoint / resume: a versioned raw image of the resident state ----
// [header 8 x int64][tracers: ntr x S values of the handle's precision]
// [compensations: ntr x S int16, FP32_COMP only]
// [carry: ntr x ncol doubles, FP32-mixed path only][sur_t, nsur_t: ncol ints each]
namespace {
constexpr long long kStateMagic = 0x53484f4354524731ll;  // "SHOCTRG1"
void state_layout(const shoc_tr_gpu *h, long long hd[8]) {
  hd[0] = kStateMagic;
  hd[1] = 1;  // version
  hd[2] = h->precision;
  hd[3] = h->ntr;
  hd[4] = h->S;
  hd[5] = h->ncol;
  hd[6] = h->fu.carry ? 1 : 0;
  hd[7] = 0;
}
size_t state_bytes(const shoc_tr_gpu *h) {
  return 8 * sizeof(long long) + (size_t)h->ntr * h->S * h->esize +
         (h->comp ? (size_t)h->ntr * h->S * sizeof(int16_t) : 0) +
         (h->fu.carry ? (size_t)h->ntr * h->ncol * sizeof(double) : 0) +
         2 * (size_t)h->ncol * sizeof(int);
}
}  // namespace

int shoc_tr_gpu_state_size(shoc_tr_gpu *h, size_t *bytes) {
  if (!h || !bytes) return SHOC_TR_EARG;
  *bytes = state_bytes(h);
  return SHOC_TR_OK;
}

int shoc_tr_gpu_save_state(shoc_tr_gpu *h, void *buf, size_t bytes) {
  if (!h || !buf || bytes < state_bytes(h)) return SHOC_TR_EARG;
  DeviceScope dev_(h->device);
  char *p = (char *)buf;
  long long hd[8];
  state_layout(h, hd);
  memcpy(p, hd, sizeof(hd));
  p += sizeof(hd);
  const size_t tb = (size_t)h->ntr * h->S * h->esize;
  CK(cudaMemcpyAsync(p, h->tr[h->cur], tb, cudaMemcpyDeviceToHost, h->stream));
  p += tb;
  if (h->comp) {
    const size_t lb = (size_t)h->ntr * h->S * sizeof(int16_t);
    CK(cudaMemcpyAsync(p, h->lo[h->cur], lb, cudaMemcpyDeviceToHost, h->stream));
    p += lb;
  }
  if (h->fu.carry) {
    const size_t cb = (size_t)h->ntr * h->ncol * sizeof(double);
    CK(cudaMemcpyAsync(p, h->fu.carry, cb, cudaMemcpyDeviceToHost, h->stream));
    p += cb;
  }
  CK(cudaMemcpyAsync(p, h->W.sur_t, (size_t)h->ncol * sizeof(int), cudaMemcpyDeviceToHost,
                     h->stream));
  p += (size_t)h->ncol * sizeof(int);
  CK(cudaMemcpyAsync(p, h->W.nsur_t, (size_t)h->ncol * sizeof(int), cudaMemcpyDeviceToHost,
                     h->stream));
  CK(cudaStreamSynchronize(h->stream));
  return SHOC_TR_OK;
}

int shoc_tr_gpu_load_state(shoc_tr_gpu *h, const void *buf, size_t bytes) {
  if (!h || !buf || bytes < state_bytes(h)) return SHOC_TR_EARG;
  long long hd[8], want[8];
  memcpy(hd, buf, sizeof(hd));
  state_layout(h, want);
  if (memcmp(hd, want, sizeof(hd)) != 0) return SHOC_TR_EARG;  // another window or precision
  DeviceScope dev_(h->device);
  const char *p = (const char *)buf + sizeof(hd);
  const size_t tb = (size_t)h->ntr * h->S * h->esize;
  // both ping-pong buffers hold the state (the values a step does not write
  // are read back from either)
  CK(cudaMemcpyAsync(h->tr[h->cur], p, tb, cudaMemcpyHostToDevice, h->stream));
  CK(cudaMemcpyAsync(h->tr[h->cur ^ 1], h->tr[h->cur], tb, cudaMemcpyDeviceToDevice, h->stream));
  p += tb;
  if (h->comp) {
    const size_t lb = (size_t)h->ntr * h->S * sizeof(int16_t);
    CK(cudaMemcpyAsync(h->lo[h->cur], p, lb, cudaMemcpyHostToDevice, h->stream));
    CK(cudaMemcpyAsync(h->lo[h->cur ^ 1], h->lo[h->cur], lb, cudaMemcpyDeviceToDevice,
                       h->stream));
    p += lb;
  }
  if (h->fu.carry) {
    const size_t cb = (size_t)h->ntr * h->ncol * sizeof(double);
    CK(cudaMemcpyAsync(h->fu.carry, p, cb, cudaMemcpyHostToDevice, h->stream));
    p += cb;
  }
  CK(cudaMemcpyAsync(h->W.sur_t, p, (size_t)h->ncol * sizeof(int), cudaMemcpyHostToDevice,
                     h->stream));
  p += (size_t)h->ncol * sizeof(int);
  CK(cudaMemcpyAsync(h->W.nsur_t, p, (size_t)h->ncol * sizeof(int), cudaMemcpyHostToDevice,
                     h->stream));
  CK(cudaStreamSynchronize(h->stream));
  return SHOC_TR_OK;
}

int shoc_tr_gpu_run(shoc_tr_gpu *h, int nsteps) {
  if (!h || nsteps < 0) return SHOC_TR_EARG;
  if (h->dt <= 0.0) return SHOC_TR_EARG;
  DeviceScope dev_(h->device);
  for (int i = 0; i < nsteps; i++) {
    int rc = step_async(h);
    if (rc) return rc;
  }
  return 0;
}

int shoc_tr_gpu_sync(shoc_tr_gpu *h, shoc_tr_diag *diag) {
  if (!h) return SHOC_TR_EARG;
  DeviceScope dev_(h->device);
  CK(cudaMemcpyAsync(h->h_rb, h->d_rb, sizeof(*h->h_rb), cudaMemcpyDeviceToHost, h->stream));
  // nwarn and, beside it, the status
  CK(cudaMemsetAsync(&h->d_rb->nwarn, 0, offsetof(shoc_tr_gpu::Readback, pad) -
                     offsetof(shoc_tr_gpu::Readback, nwarn), h->stream));
  CK(cudaStreamSynchronize(h->stream));
  int rc = map_status(h->h_rb->status);
  if (!rc) rc = h->last_status;
  h->last_status = 0;
  if (diag) {
    diag->nsub = (int)h->sched.sub.size();
    diag->dtm = h->sched.dtm;
    diag->nwarn = (long long)h->h_rb->nwarn;
    diag->vcs = h->h_rb->counts[0];
    diag->vc = h->h_rb->counts[1];
  }
  if (h->profile) {
    std::vector<cudaEvent_t> done;
    for (auto &e : h->ev) {
      float ms = 0.f;
      cudaEventElapsedTime(&ms, e.a, e.b);
      h->prof_ms[e.part] += ms;
      h->prof_n[e.part]++;
      for (cudaEvent_t x : {e.a, e.b})
        if (std::find(done.begin(), done.end(), x) == done.end()) done.push_back(x);
    }
    for (cudaEvent_t x : done) cudaEventDestroy(x);
    h->ev.clear();
  }
  return rc;
}

int shoc_tr_gpu_step(shoc_tr_gpu *h, shoc_tr_state *st, shoc_tr_diag *diag) {
  if (!h || !st || !st->tr_wc || st->ntr != h->ntr) return SHOC_TR_EARG;
  for (int n = 0; n < h->ntr; n++)
    if (!st->tr_wc[n]) return SHOC_TR_EARG;
  DeviceScope dev_(h->device);
  int rc = step_pipelined(h, st);
  if (rc) {
    shoc_tr_gpu_sync(h, nullptr);
    return rc;
  }
  // the surface vectors come back with the status
  const size_t nb = (size_t)h->ncol * sizeof(int);
  int *const sur = h->h_surf + 1, *const nsur = sur + h->ncol + 1;
  if (st->sur_t) CK(cudaMemcpyAsync(sur, h->W.sur_t, nb, cudaMemcpyDeviceToHost, h->stream));
  if (st->nsur_t) CK(cudaMemcpyAsync(nsur, h->W.nsur_t, nb, cudaMemcpyDeviceToHost, h->stream));
  rc = shoc_tr_gpu_sync(h, diag);
  if (st->sur_t) memcpy(st->sur_t + 1, sur, nb);
  if (st->nsur_t) memcpy(st->nsur_t + 1, nsur, nb);
  return rc;
}

int shoc_tr_gpu_host_register(void *ptr, size_t bytes) {
  if (!ptr || !bytes) return SHOC_TR_EARG;
  CK(cudaHostRegister(ptr, bytes, cudaHostRegisterDefault));
  return 0;
}

int shoc_tr_gpu_host_unregister(void *ptr) {
  if (!ptr) return SHOC_TR_EARG;
  CK(cudaHostUnregister(ptr));
  return 0;
}

int shoc_tr_gpu_mass(shoc_tr_gpu *h, double *mass) {
  if (!h || !mass) return SHOC_TR_EARG;
  DeviceScope dev_(h->device);
  const int nb = 148 * 2;
  double *part = nullptr;
  CK(cudaMallocAsync(&part, (size_t)nb * std::max(h->ntr, 1) * sizeof(double), h->stream));
  if (h->ntr > 0) {
    if (h->esize == sizeof(float))
      k_mass<float><<<dim3(nb, h->ntr), 256, 0, h->stream>>>(
          h->G, h->F, h->W, (const float *)h->tr[h->cur], h->fu.carry, part, nullptr, 0,
          h->lo[h->cur]);
    else
      k_mass<double><<<dim3(nb, h->ntr), 256, 0, h->stream>>>(
          h->G, h->F, h->W, (const double *)h->tr[h->cur], nullptr, part);
    h->launches++;
  }
  std::vector<double> hp((size_t)nb * h->ntr);
  CK(cudaMemcpyAsync(hp.data(), part, hp.size() * sizeof(double), cudaMemcpyDeviceToHost,
                     h->stream));
  CK(cudaFreeAsync(part, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  for (int n = 0; n < h->ntr; n++) {
    double s = 0.0, comp = 0.0;
    for (int b = 0; b < nb; b++) {
      double v = hp[(size_t)n * nb + b], u = s + v;
      comp += (fabs(s) >= fabs(v)) ? (s - u) + v : (v - u) + s;
      s = u;
    }
    mass[n] = s + comp;
  }
  return 0;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Mass reduction that allocates nothing.
//
// For host frameworks that hand all device memory out of a pool reserved at
// start-up and forbid any other allocation once the run is going (a coupled
// model sharing the GPU with other components): shoc_tr_gpu_mass allocates a
// stream-ordered buffer per call, this one does not.  The block partials live
// in the fixed device array below; the caller passes the (already allocated)
// handle and a host array for the result.
namespace {

constexpr int kNoAllocBlocks = 148 * 2;     // partial sums per tracer
constexpr int kNoAllocMaxTracers = 64;      // largest tracer count it serves
// [kNoAllocMaxTracers][kNoAllocBlocks] partials, then kNoAllocMaxTracers sums;
// about 152 KB that every device loading the library holds until exit
__device__ __align__(256) double g_noalloc_scratch[kNoAllocMaxTracers * kNoAllocBlocks +
                                                   kNoAllocMaxTracers];

// Per-tracer compensated sum of the block partials, in the order the
// allocating entry point sums them on the host (same result bit for bit).
__global__ void k_mass_finish(const double *part, int nb, int ntr, double *sums) {
  int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= ntr) return;
  double s = 0.0, comp = 0.0;
  for (int b = 0; b < nb; b++) {
    double v = part[(size_t)n * nb + b], u = s + v;
    comp += (fabs(s) >= fabs(v)) ? (s - u) + v : (v - u) + s;
    s = u;
  }
  sums[n] = s + comp;
}

std::mutex g_noalloc_mu;
double *g_noalloc_ptr[64] = {nullptr};

// Device address of the scratch array for the current device, looked up once
// per device and kept (the symbol's host-side name is not a device address).
// A reset of the device (cudaDeviceReset) invalidates the kept address, as it
// invalidates every handle's device memory.
int noalloc_scratch(int device, double **out) {
  if (device < 0 || device >= 64) return SHOC_TR_EARG;
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  if (!g_noalloc_ptr[device]) {
    void *p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) {
      fprintf(stderr, "shoc_tr_gpu: cudaGetSymbolAddress: %s\n", cudaGetErrorString(e));
      return SHOC_TR_ECUDA;
    }
    g_noalloc_ptr[device] = (double *)p;
  }
  *out = g_noalloc_ptr[device];
  return SHOC_TR_OK;
}

}  // namespace

extern "C" {

int shoc_tr_gpu_mass_noalloc(shoc_tr_gpu *h, double *mass) {
  if (!h || !mass) return SHOC_TR_EARG;
  if (h->ntr > kNoAllocMaxTracers) return SHOC_TR_ESCRATCH;
  DeviceScope dev_(h->device);
  if (!dev_.ok) return SHOC_TR_ECUDA;
  double *scr = nullptr;
  int rc = noalloc_scratch(h->device, &scr);
  if (rc) return rc;
  if (h->ntr == 0) return SHOC_TR_OK;
  // every partial and sum slot used below is written before it is read, so
  // nothing left over from an earlier call needs clearing
  double *part = scr, *sums = scr + (size_t)kNoAllocMaxTracers * kNoAllocBlocks;
  if (h->esize == sizeof(float))
    k_mass<float><<<dim3(kNoAllocBlocks, h->ntr), 256, 0, h->stream>>>(
        h->G, h->F, h->W, (const float *)h->tr[h->cur], h->fu.carry, part, nullptr, 0,
        h->lo[h->cur]);
  else
    k_mass<double><<<dim3(kNoAllocBlocks, h->ntr), 256, 0, h->stream>>>(
        h->G, h->F, h->W, (const double *)h->tr[h->cur], nullptr, part);
  k_mass_finish<<<(h->ntr + 63) / 64, 64, 0, h->stream>>>(part, kNoAllocBlocks, h->ntr, sums);
  h->launches += 2;
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(mass, sums, (size_t)h->ntr * sizeof(double), cudaMemcpyDeviceToHost,
                     h->stream));
  CK(cudaStreamSynchronize(h->stream));
  return SHOC_TR_OK;
}

int shoc_tr_gpu_compare(shoc_tr_gpu *a, shoc_tr_gpu *b, const int *region, int nregion,
                        double *maxabs, double *maxref, double *sumsq_diff, double *sumsq_ref) {
  if (!a || !b || !maxabs || !maxref || !sumsq_diff || !sumsq_ref) return SHOC_TR_EARG;
  if (nregion < 1 || (!region && nregion != 1)) return SHOC_TR_EARG;
  if (a->device != b->device || a->S != b->S || a->S2 != b->S2 || a->ncol != b->ncol ||
      a->ntr != b->ntr || a->nz != b->nz)
    return SHOC_TR_EARG;
  DeviceScope dev_(a->device);
  const int ntr = a->ntr;
  const size_t nout = (size_t)nregion * ntr;
  if (nout == 0) return SHOC_TR_OK;
  // both handles' work so far, then the comparison on a's stream
  cudaEvent_t ev;
  CK(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
  CK(cudaEventRecord(ev, b->stream));
  CK(cudaStreamWaitEvent(a->stream, ev, 0));
  cudaEventDestroy(ev);
  cudaStream_t st = a->stream;
  // per column region ids (region is indexed by 2D cell, as SHOC's 2D arrays)
  char *buf = nullptr;
  const size_t bytes = nout * 4 * sizeof(double) + (region ? (size_t)a->ncol * sizeof(int) : 0);
  CK(cudaMallocAsync((void **)&buf, bytes, st));
  unsigned long long *dmax = (unsigned long long *)buf, *dref = dmax + nout;
  double *dsd = (double *)(dref + nout), *dsr = dsd + nout;
  int *dreg = nullptr;
  CK(cudaMemsetAsync(buf, 0, nout * 4 * sizeof(double), st));
  std::vector<int> hcol;
  if (region) {
    std::vector<int> top(a->ncol);
    CK(cudaMemcpyAsync(top.data(), a->G.col_top, (size_t)a->ncol * sizeof(int),
                       cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    hcol.resize(a->ncol);
    for (int c = 0; c < a->ncol; c++) hcol[c] = region[top[c]];
    dreg = (int *)(dsr + nout);
    CK(cudaMemcpyAsync(dreg, hcol.data(), (size_t)a->ncol * sizeof(int),
                       cudaMemcpyHostToDevice, st));
  }
  const dim3 grid(148 * 2, ntr);
  const bool fa = a->esize == sizeof(float), fb = b->esize == sizeof(float);
  const void *ta = a->tr[a->cur], *tb = b->tr[b->cur];
  if (fa && fb)
    k_compare<float, float><<<grid, 256, 0, st>>>(a->G, a->tl, b->G.colntr, (const float *)ta,
                                                 (const float *)tb, dreg, nregion, dmax, dref,
                                                 dsd, dsr, a->lo[a->cur], b->lo[b->cur]);
  else if (fa)
    k_compare<float, double><<<grid, 256, 0, st>>>(a->G, a->tl, b->G.colntr, (const float *)ta,
                                                  (const double *)tb, dreg, nregion, dmax,
                                                  dref, dsd, dsr, a->lo[a->cur], b->lo[b->cur]);
  else if (fb)
    k_compare<double, float><<<grid, 256, 0, st>>>(a->G, a->tl, b->G.colntr, (const double *)ta,
                                                  (const float *)tb, dreg, nregion, dmax, dref,
                                                  dsd, dsr, a->lo[a->cur], b->lo[b->cur]);
  else
    k_compare<double, double><<<grid, 256, 0, st>>>(a->G, a->tl, b->G.colntr,
                                                   (const double *)ta, (const double *)tb, dreg,
                                                   nregion, dmax, dref, dsd, dsr, a->lo[a->cur], b->lo[b->cur]);
  a->launches++;
  CK(cudaGetLastError());
  std::vector<double> out(nout * 4);
  CK(cudaMemcpyAsync(out.data(), buf, nout * 4 * sizeof(double), cudaMemcpyDeviceToHost, st));
  CK(cudaFreeAsync(buf, st));
  CK(cudaStreamSynchronize(st));
  memcpy(maxabs, out.data(), nout * sizeof(double));
  memcpy(maxref, out.data() + nout, nout * sizeof(double));
  memcpy(sumsq_diff, out.data() + 2 * nout, nout * sizeof(double));
  memcpy(sumsq_ref, out.data() + 3 * nout, nout * sizeof(double));
  return SHOC_TR_OK;
}

// device arrays of the column-solve entry points: nine [S] fields and three
// [S2] fields, allocated on the first call
static int cols_buffer(shoc_tr_gpu *h) {
  if (h->cols) return 0;
  return dalloc(h, &h->cols, (size_t)9 * h->S + (size_t)3 * h->S2);
}

static int cols_status(shoc_tr_gpu *h) {
  CK(cudaMemcpyAsync(&h->h_rb->status, h->W.status, 4, cudaMemcpyDeviceToHost, h->stream));
  CK(cudaMemsetAsync(h->W.status, 0, 4, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  return map_status(h->h_rb->status);
}

int shoc_tr_gpu_tridiag(shoc_tr_gpu *h, const double *C, const double *Cm1, const double *Cp1,
                        const double *rhs, double *var, double minvar) {
  if (!h || !C || !Cm1 || !Cp1 || !rhs || !var) return SHOC_TR_EARG;
  DeviceScope dev_(h->device);
  int rc = cols_buffer(h);
  if (rc) return rc;
  const size_t S = (size_t)h->S, b = S * sizeof(double);
  double *dC = h->cols, *dCm1 = dC + S, *dCp1 = dCm1 + S, *dr = dCp1 + S, *dv = dr + S;
  double *dsol = dv + S, *dud = dsol + S;
  cudaStream_t st = h->stream;
  CK(cudaMemcpyAsync(dC, C, b, cudaMemcpyHostToDevice, st));
  CK(cudaMemcpyAsync(dCm1, Cm1, b, cudaMemcpyHostToDevice, st));
  CK(cudaMemcpyAsync(dCp1, Cp1, b, cudaMemcpyHostToDevice, st));
  CK(cudaMemcpyAsync(dr, rhs, b, cudaMemcpyHostToDevice, st));
  CK(cudaMemcpyAsync(dv, var, b, cudaMemcpyHostToDevice, st));
  k_tridiag<<<(h->ncol + 127) / 128, 128, 0, st>>>(h->G, h->W, dC, dCm1, dCp1, dr, dv, dsol, dud,
                                                   minvar);
  h->launches++;
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(var, dv, b, cudaMemcpyDeviceToHost, st));
  return cols_status(h);
}

int shoc_tr_gpu_vdiff_cols(shoc_tr_gpu *h, double *var, const double *dzcell, const double *C,
                           const double *Cm1, const double *Cp1, const double *fb,
                           const double *ft, const double *Splus, const double *Sminus,
                           const double *scale, double dt) {
  if (!h || !var || !dzcell || !C || !Cm1 || !Cp1 || !fb || !ft || !scale || !(dt > 0.0))
    return SHOC_TR_EARG;
  if (h->dt <= 0.0) return SHOC_TR_EARG;  // the window's dt (set_flow) is read too
  DeviceScope dev_(h->device);
  int rc = cols_buffer(h);
  if (rc) return rc;
  const size_t S = (size_t)h->S, b = S * sizeof(double), b2 = (size_t)h->S2 * sizeof(double);
  double *dC = h->cols, *dCm1 = dC + S, *dCp1 = dCm1 + S, *ddz = dCp1 + S, *dv = ddz + S;
  double *dsol = dv + S, *dud = dsol + S, *dsp = dud + S, *dsm = dsp + S;
  double *dfb = dsm + S, *dft = dfb + h->S2, *dsc = dft + h->S2;
  cudaStream_t st = h->stream;
  CK(cudaMemcpyAsync(dC, C, b, cudaMemcpyHostToDevice, st));
  CK(cudaMemcpyAsync(dCm1, Cm1, b, cudaMemcpyHostToDevice, st));
  CK(cudaMemcpyAsync(dCp1, Cp1, b, cudaMemcpyHostToDevice, st));
  CK(cudaMemcpyAsync(ddz, dzcell, b, cudaMemcpyHostToDevice, st));
  CK(cudaMemcpyAsync(dv, var, b, cudaMemcpyHostToDevice, st));
  if (Splus) CK(cudaMemcpyAsync(dsp, Splus, b, cudaMemcpyHostToDevice, st));
  if (Sminus) CK(cudaMemcpyAsync(dsm, Sminus, b, cudaMemcpyHostToDevice, st));
  CK(cudaMemcpyAsync(dfb, fb, b2, cudaMemcpyHostToDevice, st));
  CK(cudaMemcpyAsync(dft, ft, b2, cudaMemcpyHostToDevice, st));
  CK(cudaMemcpyAsync(dsc, scale, b2, cudaMemcpyHostToDevice, st));
  k_vdiff_cols<<<(h->ncol + 127) / 128, 128, 0, st>>>(
      h->G, h->W, dv, ddz, dC, dCm1, dCp1, dfb, dft, Splus ? dsp : nullptr,
      Sminus ? dsm : nullptr, dsc, dsol, dud, dt, h->dt, h->O.hmin);
  h->launches++;
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(var, dv, b, cudaMemcpyDeviceToHost, st));
  return cols_status(h);
}

int shoc_tr_gpu_halo_plan(shoc_tr_gpu *h, int nsend, const int *send_cells, int nrecv,
                          const int *recv_cells) {
  if (!h || nsend < 0 || nrecv < 0 || (nsend && !send_cells) || (nrecv && !recv_cells))
    return SHOC_TR_EARG;
  for (int i = 0; i < nsend; i++)
    if (send_cells[i] < 1 || send_cells[i] >= h->S) return SHOC_TR_EARG;
  for (int i = 0; i < nrecv; i++)
    if (recv_cells[i] < 1 || recv_cells[i] >= h->S) return SHOC_TR_EARG;
  DeviceScope dev_(h->device);
  int rc;
  if (nsend > h->nhalo_send && (rc = dalloc(h, &h->halo_send, (size_t)nsend))) return rc;
  if (nrecv > h->nhalo_recv && (rc = dalloc(h, &h->halo_recv, (size_t)nrecv))) return rc;
  if (nsend)
    CK(cudaMemcpy(h->halo_send, send_cells, (size_t)nsend * sizeof(int), cudaMemcpyHostToDevice));
  if (nrecv)
    CK(cudaMemcpy(h->halo_recv, recv_cells, (size_t)nrecv * sizeof(int), cudaMemcpyHostToDevice));
  h->nhalo_send = nsend;
  h->nhalo_recv = nrecv;
  return default_stream_done();
}

int shoc_tr_gpu_halo_pack(shoc_tr_gpu *h, void *buf) {
  if (!h || (h->nhalo_send && !buf)) return SHOC_TR_EARG;
  if (h->comp) return SHOC_TR_EUNSUPPORTED;  // the halo carries no compensation
  DeviceScope dev_(h->device);
  const int n = h->nhalo_send;
  if (n && h->ntr) {
    const long long tot = (long long)n * h->ntr;
    const int blocks = (int)std::min<long long>((tot + 255) / 256, 148 * 8);
    if (h->esize == sizeof(float))
      k_halo_pack<float><<<blocks, 256, 0, h->stream>>>((const float *)h->tr[h->cur], h->S,
                                                        h->ntr, h->halo_send, n, (float *)buf);
    else
      k_halo_pack<double><<<blocks, 256, 0, h->stream>>>((const double *)h->tr[h->cur], h->S,
                                                         h->ntr, h->halo_send, n, (double *)buf);
    h->launches++;
    CK(cudaGetLastError());
  }
  CK(cudaStreamSynchronize(h->stream));
  return SHOC_TR_OK;
}

int shoc_tr_gpu_halo_unpack(shoc_tr_gpu *h, const void *buf) {
  if (!h || (h->nhalo_recv && !buf)) return SHOC_TR_EARG;
  if (h->comp) return SHOC_TR_EUNSUPPORTED;
  DeviceScope dev_(h->device);
  const int n = h->nhalo_recv;
  if (n && h->ntr) {
    const long long tot = (long long)n * h->ntr;
    const int blocks = (int)std::min<long long>((tot + 255) / 256, 148 * 8);
    if (h->esize == sizeof(float))
      k_halo_unpack<float><<<blocks, 256, 0, h->stream>>>(
          (float *)h->tr[h->cur], (float *)h->tr[h->cur ^ 1], h->S, h->ntr, h->halo_recv, n,
          (const float *)buf);
    else
      k_halo_unpack<double><<<blocks, 256, 0, h->stream>>>(
          (double *)h->tr[h->cur], (double *)h->tr[h->cur ^ 1], h->S, h->ntr, h->halo_recv, n,
          (const double *)buf);
    h->launches++;
    CK(cudaGetLastError());
  }
  return SHOC_TR_OK;
}

int shoc_tr_gpu_mass_region(shoc_tr_gpu *h, const int *region, int reg, double *mass) {
  if (!h || !region || !mass) return SHOC_TR_EARG;
  DeviceScope dev_(h->device);
  const int nb = 148 * 2;
  std::vector<int> top(h->ncol), cr(h->ncol);
  CK(cudaMemcpyAsync(top.data(), h->G.col_top, (size_t)h->ncol * sizeof(int),
                     cudaMemcpyDeviceToHost, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  for (int c = 0; c < h->ncol; c++) cr[c] = region[top[c]];
  char *buf = nullptr;
  const size_t pb = (size_t)nb * std::max(h->ntr, 1) * sizeof(double);
  CK(cudaMallocAsync((void **)&buf, pb + (size_t)h->ncol * sizeof(int), h->stream));
  double *part = (double *)buf;
  int *dreg = (int *)(buf + pb);
  CK(cudaMemcpyAsync(dreg, cr.data(), (size_t)h->ncol * sizeof(int), cudaMemcpyHostToDevice,
                     h->stream));
  if (h->ntr > 0) {
    if (h->esize == sizeof(float))
      k_mass<float><<<dim3(nb, h->ntr), 256, 0, h->stream>>>(
          h->G, h->F, h->W, (const float *)h->tr[h->cur], h->fu.carry, part, dreg, reg,
          h->lo[h->cur]);
    else
      k_mass<double><<<dim3(nb, h->ntr), 256, 0, h->stream>>>(
          h->G, h->F, h->W, (const double *)h->tr[h->cur], nullptr, part, dreg, reg);
    h->launches++;
  }
  std::vector<double> hp((size_t)nb * h->ntr);
  CK(cudaMemcpyAsync(hp.data(), part, hp.size() * sizeof(double), cudaMemcpyDeviceToHost,
                     h->stream));
  CK(cudaFreeAsync(buf, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  for (int n = 0; n < h->ntr; n++) {
    double s = 0.0, comp = 0.0;
    for (int b = 0; b < nb; b++) {
      double v = hp[(size_t)n * nb + b], u = s + v;
      comp += (fabs(s) >= fabs(v)) ? (s - u) + v : (v - u) + s;
      s = u;
    }
    mass[n] = s + comp;
  }
  return SHOC_TR_OK;
}

int shoc_tr_gpu_set_owned(shoc_tr_gpu *h, const int *owned2d) {
  if (!h) return SHOC_TR_EARG;
  DeviceScope dev_(h->device);
  if (!owned2d) {
    h->colown = nullptr;  // every column counts again (the array stays allocated)
    return SHOC_TR_OK;
  }
  std::vector<int> top(h->ncol), own(h->ncol);
  CK(cudaMemcpy(top.data(), h->G.col_top, (size_t)h->ncol * sizeof(int), cudaMemcpyDeviceToHost));
  for (int c = 0; c < h->ncol; c++) own[c] = owned2d[top[c]] ? 1 : 0;
  int *d = nullptr;
  int rc = dupload(h, &d, own.data(), (size_t)h->ncol);
  if (!rc) rc = default_stream_done();
  if (rc) return rc;
  h->colown = d;
  return SHOC_TR_OK;
}

int shoc_tr_gpu_substep_min(shoc_tr_gpu *h, double *dmin) {
  if (!h || !dmin || h->dt <= 0.0) return SHOC_TR_EARG;
  DeviceScope dev_(h->device);
  cudaStream_t st = h->stream;
  k_reset<<<1, 32, 0, st>>>(h->W, h->d_counts);
  h->launches++;
  launch_set_dz(h, SD_PROBE | SD_SEARCH);
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(&h->h_rb->dtm, h->W.dtm_bits, 8, cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  unsigned long long b = h->h_rb->dtm;
  memcpy(dmin, &b, 8);
  return SHOC_TR_OK;
}

int shoc_tr_gpu_set_substep_min(shoc_tr_gpu *h, double dmin) {
  if (!h || dmin < 0.0) return SHOC_TR_EARG;
  if (dmin != h->dmin_set) {
    DeviceScope dev_(h->device);
    h->dmin_set = dmin;
    for (int i = 0; i < 2; i++)
      if (h->graph[i]) {
        cudaGraphExecDestroy(h->graph[i]);
        h->graph[i] = nullptr;
      }
    h->have_sched = false;
    h->probe_left = 2;
  }
  return SHOC_TR_OK;
}

void *shoc_tr_gpu_stream(shoc_tr_gpu *h) { return h ? (void *)h->stream : nullptr; }

int shoc_tr_gpu_set_tiling(shoc_tr_gpu *h, int cols_per_block, int tracers_per_block) {
  if (!h) return SHOC_TR_EARG;
  DeviceScope dev_(h->device);
  if (cols_per_block != 0 && cols_per_block != 32) return SHOC_TR_EUNSUPPORTED;
  if (tracers_per_block <= 0) return SHOC_TR_OK;
  shoc_tr_tuning t = current_tuning(h);
  t.tracers_per_block = tracers_per_block;
  return apply_tuning(h, t);
}

int shoc_tr_gpu_get_tuning(shoc_tr_gpu *h, shoc_tr_tuning *t) {
  if (!h || !t) return SHOC_TR_EARG;
  *t = current_tuning(h);
  return SHOC_TR_OK;
}

int shoc_tr_gpu_set_tuning(shoc_tr_gpu *h, const shoc_tr_tuning *t) {
  if (!h || !t) return SHOC_TR_EARG;
  DeviceScope dev_(h->device);
  return apply_tuning(h, *t);
}

}  // extern "C"

// ---- autotuner ----
namespace {

// The autotuner's cache: one line per GPU model and window configuration,
//   <key> <fused> <tracers_per_block> <tile_x> <phase_b_warps> <prefetch> <ms>
// in the file SHOC_TR_TUNE_CACHE names (default
// $HOME/.cache/shoc_tr_gpu/tuning.txt; "off": none).
std::string tune_cache_path() {
  const char *e = getenv("SHOC_TR_TUNE_CACHE");
  if (e) return strcmp(e, "off") == 0 ? std::string() : std::string(e);
  const char *home = getenv("HOME");
  if (!home || !*home) return std::string();
  return std::string(home) + "/.cache/shoc_tr_gpu/tuning.txt";
}

// The key names the build: a choice measured on other kernels, or under another
// meaning of a field, is not found.
#ifndef SHOC_TR_BUILD_ID  // the hash of the sources (ems_b200/_build.py)
#define SHOC_TR_BUILD_ID __DATE__ "_" __TIME__
#endif
std::string tune_key(const shoc_tr_gpu *h) {
  cudaDeviceProp p;
  if (cudaGetDeviceProperties(&p, h->device) != cudaSuccess) return std::string();
  std::string name = std::string(SHOC_TR_BUILD_ID "|") + p.name;
  for (char &c : name)
    if (c == ' ' || c == '\t') c = '_';
  char buf[512];
  snprintf(buf, sizeof buf, "v3|%s|sm%d%d|S%d|C%d|Z%d|N%d|B%d|P%d|A%d|U%d|F%d|H%d|V%d",
           name.c_str(), p.major, p.minor, h->S, h->ncol, h->nz, h->ntr, h->T.ntb, h->precision,
           h->O.trasc, h->O.ultimate, h->adv_flags, h->any_hdiff ? 1 : 0, h->any_vdiff ? 1 : 0);
  return std::string(buf);
}

bool tune_cache_get(const std::string &path, const std::string &key, shoc_tr_tuning *t) {
  if (path.empty() || key.empty()) return false;
  FILE *f = fopen(path.c_str(), "r");
  if (!f) return false;
  char line[1024];
  bool found = false;
  while (fgets(line, sizeof line, f)) {
    char k[600];
    shoc_tr_tuning v;
    double ms;
    if (sscanf(line, "%599s %d %d %d %d %d %lf", k, &v.fused, &v.tracers_per_block, &v.tile_x,
               &v.phase_b_warps, &v.prefetch, &ms) == 7 &&
        key == k) {
      *t = v;
      found = true;  // the last line for a key wins
    }
  }
  fclose(f);
  return found;
}

void tune_cache_put(const std::string &path, const std::string &key, const shoc_tr_tuning &t,
                    double ms) {
  if (path.empty() || key.empty()) return;
  // the directory, one level at a time
  for (size_t i = 1; i < path.size(); i++)
    if (path[i] == '/') mkdir(path.substr(0, i).c_str(), 0755);
  std::vector<std::string> keep;
  if (FILE *f = fopen(path.c_str(), "r")) {
    char line[1024];
    while (fgets(line, sizeof line, f)) {
      char k[600];
      if (sscanf(line, "%599s", k) == 1 && key != k) keep.push_back(line);
    }
    fclose(f);
  }
  const std::string tmp = path + ".tmp" + std::to_string((long long)getpid());
  FILE *f = fopen(tmp.c_str(), "w");
  if (!f) return;
  for (auto &l : keep) fputs(l.c_str(), f);
  fprintf(f, "%s %d %d %d %d %d %.6f\n", key.c_str(), t.fused, t.tracers_per_block, t.tile_x,
          t.phase_b_warps, t.prefetch, ms);
  fclose(f);
  rename(tmp.c_str(), path.c_str());
}

// Device copy of the resident state (both tracer buffers, mass carry,
// surface vectors) the trial steps start from.
// The resident state the autotuner's trial steps start from: the current
// tracer buffer (and compensation), put back into both ping-pong buffers as
// shoc_tr_gpu_load_state does.
struct Snapshot {
  void *tr = nullptr;
  int16_t *lo = nullptr;  // FP32_COMP: the current buffer's compensations
  double *carry = nullptr;
  int *sur = nullptr, *nsur = nullptr;
  int cur = 0;
};

int snap_take(shoc_tr_gpu *h, Snapshot &s) {
  const size_t tb = (size_t)h->ntr * h->S * h->esize;
  const size_t cb = (size_t)h->ntr * h->ncol * sizeof(double);
  const size_t ib = (size_t)h->ncol * sizeof(int);
  CK(cudaMallocAsync(&s.tr, tb ? tb : 1, h->stream));
  if (h->fu.carry) CK(cudaMallocAsync((void **)&s.carry, cb ? cb : 1, h->stream));
  CK(cudaMallocAsync((void **)&s.sur, 2 * ib, h->stream));
  s.nsur = s.sur + h->ncol;
  s.cur = h->cur;
  CK(cudaMemcpyAsync(s.tr, h->tr[h->cur], tb, cudaMemcpyDeviceToDevice, h->stream));
  if (h->comp) {
    const size_t lb = (size_t)h->ntr * h->S * sizeof(int16_t);
    CK(cudaMallocAsync((void **)&s.lo, lb ? lb : 1, h->stream));
    CK(cudaMemcpyAsync(s.lo, h->lo[h->cur], lb, cudaMemcpyDeviceToDevice, h->stream));
  }
  if (s.carry) CK(cudaMemcpyAsync(s.carry, h->fu.carry, cb, cudaMemcpyDeviceToDevice, h->stream));
  CK(cudaMemcpyAsync(s.sur, h->W.sur_t, ib, cudaMemcpyDeviceToDevice, h->stream));
  CK(cudaMemcpyAsync(s.nsur, h->W.nsur_t, ib, cudaMemcpyDeviceToDevice, h->stream));
  return 0;
}

int snap_restore(shoc_tr_gpu *h, const Snapshot &s) {
  const size_t tb = (size_t)h->ntr * h->S * h->esize;
  const size_t cb = (size_t)h->ntr * h->ncol * sizeof(double);
  const size_t ib = (size_t)h->ncol * sizeof(int);
  h->cur = s.cur;
  for (int b = 0; b < 2; b++)
    CK(cudaMemcpyAsync(h->tr[b], s.tr, tb, cudaMemcpyDeviceToDevice, h->stream));
  if (s.lo) {
    const size_t lb = (size_t)h->ntr * h->S * sizeof(int16_t);
    for (int b = 0; b < 2; b++)
      CK(cudaMemcpyAsync(h->lo[b], s.lo, lb, cudaMemcpyDeviceToDevice, h->stream));
  }
  if (s.carry) CK(cudaMemcpyAsync(h->fu.carry, s.carry, cb, cudaMemcpyDeviceToDevice, h->stream));
  CK(cudaMemcpyAsync(h->W.sur_t, s.sur, ib, cudaMemcpyDeviceToDevice, h->stream));
  CK(cudaMemcpyAsync(h->W.nsur_t, s.nsur, ib, cudaMemcpyDeviceToDevice, h->stream));
  return 0;
}

void snap_free(shoc_tr_gpu *h, Snapshot &s) {
  if (s.tr) cudaFreeAsync(s.tr, h->stream);
  if (s.lo) cudaFreeAsync(s.lo, h->stream);
  if (s.carry) cudaFreeAsync(s.carry, h->stream);
  if (s.sur) cudaFreeAsync(s.sur, h->stream);
  cudaStreamSynchronize(h->stream);
  s = Snapshot();
}

}  // namespace

extern "C" {

int shoc_tr_gpu_autotune_ex(shoc_tr_gpu *h, int steps, int use_cache, shoc_tr_tuning *best,
                            int *from_cache) {
  if (!h || steps < 1) return SHOC_TR_EARG;
  DeviceScope dev_(h->device);
  if (from_cache) *from_cache = 0;
  const std::string path = use_cache ? tune_cache_path() : std::string();
  const std::string key = use_cache ? tune_key(h) : std::string();
  shoc_tr_tuning t;
  if (use_cache && tune_cache_get(path, key, &t) && apply_tuning(h, t) == SHOC_TR_OK) {
    if (best) *best = t;
    if (from_cache) *from_cache = 1;
    return SHOC_TR_OK;
  }
  // candidates: warps per column-kernel block for the two-kernel sub-step;
  // tile widths and phase-B warps for the fused one (FP32-mixed, where it fits)
  std::vector<shoc_tr_tuning> cand;
  shoc_tr_tuning base = current_tuning(h);
  const std::vector<int> tws = h->esize == sizeof(float)
                                   ? std::vector<int>{2, 3, 4, 5, 6, 8, 12, 16}
                                   : std::vector<int>{2, 3, 4, 5, 6, 8};
  for (int pf : {0, 1}) {
    if (pf && h->esize != sizeof(float)) continue;
    for (int tw : tws) {
      shoc_tr_tuning c = base;
      c.fused = 0;
      c.tracers_per_block = tw;
      c.prefetch = pf;
      cand.push_back(c);
    }
  }
  if (h->esize == sizeof(float) && h->fnwb_max) {
    std::vector<int> nwbs = {h->fnwb_max};
    if (h->fnwb_max / 2 >= 1 && h->fnwb_max / 2 != h->fnwb_max) nwbs.push_back(h->fnwb_max / 2);
    for (int tx : {8, 16, 32})
      for (int nwb : nwbs) {
        shoc_tr_tuning c = base;
        c.fused = 1;
        c.prefetch = 0;
        c.tile_x = tx;
        c.phase_b_warps = nwb;
        cand.push_back(c);
      }
  }
  Snapshot snap;
  int rc = snap_take(h, snap);
  if (rc) {  // no room for the copy: nothing has run, the handle is unchanged
    cudaGetLastError();
    snap_free(h, snap);
    return SHOC_TR_ENOMEM;
  }
  const bool prof0 = h->profile;
  shoc_tr_tuning win = base;
  double best_ms = 1e300;
  // numbers of warps that make the same launches (more than the tracers, or than the
  // shared memory holds) are tried once
  std::vector<std::vector<int>> tried;
  for (const auto &c : cand) {
    if (apply_tuning(h, c) != SHOC_TR_OK) continue;
    if (!c.fused) {
      ColLaunch cl[kColLaunches];
      const int n = col_launches(h, h->nslot, std::max(1, std::min(h->tw, h->nslot)), cl);
      std::vector<int> key = {c.prefetch};
      for (int i = 0; i < n; i++) key.insert(key.end(), {cl[i].tile0, cl[i].bytes, cl[i].warps});
      if (std::find(tried.begin(), tried.end(), key) != tried.end()) continue;
      tried.push_back(key);
    }
    shoc_tr_gpu_profile(h, 1);
    rc = shoc_tr_gpu_run(h, steps);
    if (!rc) rc = shoc_tr_gpu_sync(h, nullptr);
    double ms = 0.0;
    int n = 0;
    shoc_tr_gpu_kernel_time(h, &ms, &n);
    if (!rc) rc = snap_restore(h, snap);
    if (rc) break;
    if (n > 0 && ms < best_ms) {
      best_ms = ms;
      win = c;
    }
  }
  if (!rc) rc = snap_restore(h, snap);
  snap_free(h, snap);
  h->profile = prof0;
  shoc_tr_gpu_profile(h, prof0 ? 1 : 0);
  const int rc2 = apply_tuning(h, win);
  if (rc) return rc;
  if (rc2) return rc2;
  if (use_cache && best_ms < 1e300) tune_cache_put(path, key, win, best_ms);
  if (best) *best = win;
  return SHOC_TR_OK;
}

int shoc_tr_gpu_autotune(shoc_tr_gpu *h, int steps, int *tracers_per_block) {
  shoc_tr_tuning t;
  const int rc = shoc_tr_gpu_autotune_ex(h, steps, 0, &t, nullptr);
  if (!rc && tracers_per_block) *tracers_per_block = t.tracers_per_block;
  return rc;
}

int shoc_tr_gpu_profile(shoc_tr_gpu *h, int enable) {
  if (!h) return SHOC_TR_EARG;
  h->profile = enable != 0;
  for (int i = 0; i < 3; i++) {
    h->prof_ms[i] = 0.0;
    h->prof_n[i] = 0;
  }
  return 0;
}

int shoc_tr_gpu_kernel_time_part(shoc_tr_gpu *h, int part, double *ms, int *n) {
  if (!h || part < 0 || part > 2) return SHOC_TR_EARG;
  if (ms) *ms = h->prof_n[part] ? h->prof_ms[part] / h->prof_n[part] : 0.0;
  if (n) *n = h->prof_n[part];
  h->prof_ms[part] = 0.0;
  h->prof_n[part] = 0;
  return 0;
}

int shoc_tr_gpu_kernel_time(shoc_tr_gpu *h, double *ms, int *n) {
  return shoc_tr_gpu_kernel_time_part(h, 0, ms, n);
}

long long shoc_tr_gpu_launch_count(shoc_tr_gpu *h) { return h ? h->launches : 0; }

}  // extern "C"
