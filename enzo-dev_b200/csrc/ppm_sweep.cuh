// ppm_sweep.cuh -- launch arguments shared by the sweep kernels and the host driver.
#pragma once

#include <cuda.h>  // CUtensorMap

#include <cstdint>
#include <cstring>
#include <vector>

namespace ppm {

// Per-cell coefficients along one sweep axis, precomputed by the host from the
// cell widths exactly as inteuler.F:140-158 computes them (same expressions, FP64).
struct Coef {
  double c1, c2, c3, c4, c5, c6, dx2i, dx;
};

// Subgrid-flux capture request for one pencil: flux of face `face` goes to
// `dst_offset` of capture slot `slot` (a contiguous range of the capture buffer).
struct FluxCapture {
  int64_t pencil;     // linear pencil id
  int32_t face;       // face index along the pencil (left face of cell `face`)
  int32_t pad;
  int64_t dst;        // base offset (in doubles) of this request in the capture buffer
};

enum { kMaxCounters = 32 };
// device counters (unsigned long long), see ppm_b200_stats
enum {
  kCntInterfaces = 0,
  kCntNewton = 1,
  kCntHist0 = 2,  // 2..9 : newton_hist[0..7]
  kCntFallbacks = 10,
  kCntFatal = 11,
  kCntGuessRejected = 12,
  kCntNonFinite = 13,
  kCntFlagged = 14,  // pencils handed to the fallback pass (index into BatchArgs::flagged)
  kCntTimeout = 15,  // bounded waits on asynchronous copies that gave up
  kCntWarpNewton = 16,  // sum over Riemann warps of the most Newton updates any lane took
  kCntWarps = 17,       // Riemann warps with at least one face
};

// The Riemann stages add their statistics (nine values a block) to one of kCounterCopies
// copies of the counters, chosen by the block's index; the host sums them.  On one copy
// the 137,000 blocks of a 256^3 sweep queue at one L2 line, about one addition a clock:
// 0.65 ms, more than the tolerance build's kernel takes without them (a 256^3 sweep: 1.08
// ms on one copy, 0.58 on 64).
enum { kCounterCopies = 64 };
constexpr size_t kCounterBytes = (size_t)kCounterCopies * kMaxCounters * sizeof(unsigned long long);

inline void sum_counters(const unsigned long long* copies, unsigned long long* c) {
  for (int k = 0; k < kMaxCounters; ++k) {
    c[k] = 0;
    for (int m = 0; m < kCounterCopies; ++m) c[k] += copies[m * kMaxCounters + k];
  }
}

struct SweepArgs {
  // geometry: pencils are indexed p = t2 * n1 + t1; cell a of pencil (t1, t2)
  // sits at element t1 * s1 + t2 * s2 + a * sa of every field array.
  int n;                 // pencil length (GridDimension[dim])
  int is, ie;            // active range along the pencil, 0-based inclusive
  int n1, n2;            // pencils along the two transverse axes
  int64_t s1, s2, sa;    // element strides
  int64_t npencils;
  // fields: d, e, u(sweep velocity), v, w, ge -- input and output sets (distinct)
  const double* __restrict__ in_d;
  const double* __restrict__ in_e;
  const double* __restrict__ in_u;
  const double* __restrict__ in_v;   // may be null (rank < 3): read as 0, not written
  const double* __restrict__ in_w;
  const double* __restrict__ in_ge;  // may be null unless dual
  const double* __restrict__ pres;   // pressure of this SolvePPM_DE call (stale across sweeps)
  const double* __restrict__ grav;   // acceleration along the sweep axis (GRAV only)
  double* __restrict__ out_d;
  double* __restrict__ out_e;
  double* __restrict__ out_u;
  double* __restrict__ out_v;
  double* __restrict__ out_w;
  double* __restrict__ out_ge;
  const Coef* __restrict__ coef;     // n entries
  // physics
  double gamma, dt, eta1, eta2, small_rho, pmin;
  const double* dt_device;           // if non-null, *dt_device replaces dt
  int fallback;                      // RiemannSolverFallback
  // subgrid flux capture (optional)
  const FluxCapture* captures;       // sorted by pencil
  int64_t ncaptures;
  double* capture_buf;               // 6 doubles per request: df, ef, uf, vf, wf, gef
  // face scratch of the three-stage sweep: plane v holds one value per (face, pencil),
  // element fi * npencils + pencil with fi = face - is in [0, ie - is + 1]
  double* fstate;                    // kFaceVars planes: dl dr pl pr ul ur vl vr wl wr gel ger
  double* fflux;                     // kFluxVars planes: df ef uf vf wf gef ub
  int64_t plane;                     // elements per plane = (ie - is + 2) * npencils
  // learned Newton start (ppm_guess.cuh): packed BF16 weights, used by the LEARNED kernels
  const uint32_t* guess;
  // optional log of sampled faces of the plain solver: 8 doubles per record
  // (dl dr pl pr ul ur p* +-iterations, negative when Newton did not converge)
  double* log;
  unsigned long long* log_count;     // records claimed (may exceed log_cap)
  int64_t log_cap;
  int log_stride;                    // about one face in log_stride is logged; 0 = off
  // Courant time step of the updated fields (calc_dt.F), computed in the update kernel of
  // a solve's last sweep when cfl_min_bits is set: the minimum over the batch of dt1
  // goes to *cfl_min_bits (positive doubles order as integers)
  unsigned long long* cfl_min_bits;
  const double* cw1;                 // cell widths along the t1 and t2 axes (device)
  const double* cw2;
  int dim, rank;                     // the sweep axis and GridRank
  int ts1, te1, ts2, te2;            // active ranges along the t1 and t2 axes
  double aye, vg[3], min_support;    // calc_dt's a, grid velocity, ComputePressure's floor
  // slope corrections: calcdiss's flattening (type 1 or 3) of every variable and
  // inteuler's steepening of the density, as per-cell coefficients of cells is-1 .. ie+1
  // in planes [cell - (is-1)][pencil], written by the corrections kernel; null when off
  double* flat;
  double* steep;
  int flatten, steepen;              // PPMFlatteningParameter, PPMSteepeningParameter
  // colour fields (NumberOfColours > 0): advected in place by the colour kernel after the
  // sweep's update.  col: device array of ncolour field pointers; fcol: kColVars face
  // planes that the density reconstruction and the Riemann stage leave for it; fhll: one
  // byte per face, set where the HLL fallback replaced the face's fluxes;
  // col_capture: ncolour doubles per subgrid-flux capture request (request r = dst / 6)
  int ncolour;
  double* const* col;
  double* fcol;
  unsigned char* fhll;
  double* col_capture;
  // Riemann solver (Grid_xEulerSweep.C:223-283): 0 two-shock, 1 HLL, 2 HLLC.  For HLL and
  // HLLC the flux plane XUB holds the gas-energy source ges of the face's right cell
  // instead of the Godunov velocity.
  int solver;
  // PressureFree: sound speed tiny in the characteristics (inteuler.F:199) and the time
  // step (calc_dt.F:78-137), the face densities the uncorrected ones (inteuler.F:556-561),
  // the two-shock solve replaced by p* = pmin, u* = (ul + ur)/2 (twoshock.F:124-130)
  int presfree;
  // EOSType 3 (isothermal): the folded time step's pressure is rho * eos_cs^2
  int eos_type;
  double eos_cs;
  // split of the marching stages (set_segments): a block of kMarchThreads threads takes
  // 2^pw_log2 pencils, each cut into kMarchThreads >> pw_log2 segments of seg_faces faces
  // (reconstruction); uw_log2 and seg_cells the same for the update and transport kernels,
  // whose segments are of cells
  int pw_log2, seg_faces, uw_log2, seg_cells;
  // one cell width along the sweep (uniform): the coefficients every cell shares
  int uniform;
  Coef uc;
};

enum { kFaceVars = 12, kFluxVars = 7 };
// colour face planes: dla dl0 dra dr0 (the density's characteristic averages), the
// corrected densities before the dual-energy override, the override flags (1 left,
// 2 right), the Godunov density db, and on faces the HLL fallback replaced its weights
// sl, bm0, sr, bp0 (written by the fallback pass only there)
enum { CDLA = 0, CDL0, CDRA, CDR0, CDLC, CDRC, COVR, CDB, CHSL, CHBM, CHSR, CHBP, kColVars };
enum { kMaxColours = 45 };  // MAX_COLOR (fortran.def:2)

// Threads per block of the marching stages and of the face-parallel Riemann stage.
// (Riemann blocks of 128 faces leave fewer idle lanes at the end of each face plane of
// the small grids of a level than 256: -18 % Riemann time on a 600-patch level, and
// slightly faster on 256^3.)
#ifndef PPM_RIEMANN_THREADS
#define PPM_RIEMANN_THREADS 128
#endif
#ifndef PPM_MARCH_THREADS
#define PPM_MARCH_THREADS 128
#endif
enum { kMarchThreads = PPM_MARCH_THREADS, kRiemannThreads = PPM_RIEMANN_THREADS };

// One launch over a batch of grids (an AMR level, or a single grid).  Every block
// belongs to one grid: grid g owns blocks [prefix[g], prefix[g+1]) of a stage; a
// block finds its grid by binary search over the prefix table.
//   reconstruction, corrections, colours (times the colour chunks): ceil(npencils /
//                   2^pw_log2) blocks per grid
//   update, transport: ceil(npencils / 2^uw_log2) blocks per grid
//   Riemann stage:   (ie - is + 2) * ceil(npencils / kRiemannThreads) blocks per grid
struct BatchArgs {
  SweepArgs one;                     // the record itself when ngrids == 1 (read from the
                                     // kernel parameter space, like a plain launch)
  const SweepArgs* grids;            // device array, ngrids records
  int ngrids;
  const int64_t* seg_prefix;         // ngrids + 1 (reconstruction)
  int64_t seg_blocks = 0;
  const int64_t* upd_prefix;         // ngrids + 1 (update, transport)
  int64_t upd_blocks = 0;
  int transport = 0;                 // the transport path (see transport_kernel)
  int both_roles = 0;                // both reconstructions in one launch
  int chained = 1;                   // the sweep's first kernel is a link of the launch chain
  unsigned long long* clear_bits = nullptr;  // folded time step to reset before this sweep
  const int64_t* riemann_prefix;     // ngrids + 1
  unsigned long long* counters;      // kCounterCopies x kMaxCounters, shared by the batch
  int64_t* flagged;                  // pencils needing the fallback pass: (grid << 40) | pencil
  int corrections = 0;               // the batch's grids carry flattening / steepening
  int uneven = 0;                    // a grid's cell widths differ along the sweep
  // x sweep of a single grid: the update kernel reads its input cells as TMA tiles of
  // kXTileRows pencils x kXTileCells cells, through 2-D tensor maps (cells x pencils) of
  // d, e, u, v, w, ge (absent fields: unused).  x_tma = 0: plain loads.
  int x_tma = 0;
  // test hook (ppm_b200_debug_tma_stall): bytes every TMA chunk expects beyond its
  // copies, so that its barrier never completes and the bounded waits run out; 0
  unsigned x_tma_extra_tx = 0;
  // colours: the batch's NumberOfColours (every grid the same) and the fallback-face
  // flags of all its grids (one region, cleared at the start of each sweep)
  int ncolour = 0;
  unsigned char* hll_flags = nullptr;
  int64_t hll_bytes = 0;
  int solver = 0;                    // the batch's Riemann solver (SweepArgs::solver)
  int presfree = 0;                  // PressureFree (SweepArgs::presfree)
  // two-shock Riemann stage (plain start, no colours): faces per block (64, 128 or 256;
  // the Riemann prefix table counts blocks of this size) and a persistent launch that
  // walks riemann_total blocks with a grid of the resident blocks
  int riemann_threads = kRiemannThreads;
  int persistent = 0;
  int64_t riemann_total = 0;
  // fused sweep (two-shock with the plain start, no colours or slope corrections): one
  // kernel reconstructs the interface states and solves the Riemann problems of a
  // (group of kFaceWarps pencils, segment of kFaceSeg faces) per block; face_prefix is
  // its block prefix table
  int fused = 0;
  const int64_t* face_prefix = nullptr;
  int64_t face_blocks = 0;
  // learned start from a tensor-core guess pass (tcgen05, ppm_guess_tc.cu) over the
  // interface states before the Riemann kernel, instead of inside it
  int learned_pass = 0;
  int sms = 148;
  CUtensorMap xin[7];                // d, e, u, v, w, ge, pressure
};

// The fused face kernel: a warp takes one pencil and kFaceSeg consecutive faces, lane
// l >= 1 the face of cell f0 - 1 + l (lane 0 the cell left of the first face); a block
// takes kFaceWarps consecutive pencils.
#ifndef PPM_FACE_WARPS
#define PPM_FACE_WARPS 8
#endif
enum { kFaceWarps = PPM_FACE_WARPS, kFaceThreads = 32 * PPM_FACE_WARPS, kFaceSeg = 31 };
__host__ __device__ inline int64_t face_segments(int is, int ie) {
  return (ie - is + 2 + kFaceSeg - 1) / kFaceSeg;
}
__host__ __device__ inline int64_t face_blocks(int64_t npencils, int is, int ie) {
  return ((npencils + kFaceWarps - 1) / kFaceWarps) * face_segments(is, ie);
}

// TMA tiles of the x sweep's update kernel: a warp's 32 pencils x 4 cells (32 bytes a
// pencil), double-buffered per warp
#ifndef PPM_X_BUFFERS
#define PPM_X_BUFFERS 2
#endif
#ifndef PPM_X_TILE_CELLS
#define PPM_X_TILE_CELLS 4
#endif
enum { kXTileRows = 32, kXTileCells = PPM_X_TILE_CELLS, kXBuffers = PPM_X_BUFFERS };

// inteuler.F:140-158 on the host (same expressions; 1-based i mapped to entry i-1): the
// coefficient table of one sweep axis.  Every entry point builds its table here, so the
// library's paths cannot drift apart; host code is compiled with -ffp-contract=off.
inline void build_coef(const double* dxi_in, int n, int is0, int ie0, std::vector<Coef>& out) {
  out.assign(n, Coef{0, 0, 0, 0, 0, 0, 0, 0});
  auto dxi = [&](int i) { return dxi_in[i - 1]; };
  const int i1 = is0 + 1, i2 = ie0 + 1;
  for (int i = 1; i <= n; ++i) out[i - 1].dx = dxi(i);
  for (int i = i1 - 2; i <= i2 + 2; i++) {
    double qa = dxi(i) / (dxi(i - 1) + dxi(i) + dxi(i + 1));
    out[i - 1].c1 = qa * (2.0 * dxi(i - 1) + dxi(i)) / (dxi(i + 1) + dxi(i));
    out[i - 1].c2 = qa * (2.0 * dxi(i + 1) + dxi(i)) / (dxi(i - 1) + dxi(i));
  }
  for (int i = i1 - 1; i <= i2 + 2; i++) {
    double qa = dxi(i - 2) + dxi(i - 1) + dxi(i) + dxi(i + 1);
    double qb = dxi(i - 1) / (dxi(i - 1) + dxi(i));
    double qc = (dxi(i - 2) + dxi(i - 1)) / (2.0 * dxi(i - 1) + dxi(i));
    double qd = (dxi(i + 1) + dxi(i)) / (2.0 * dxi(i) + dxi(i - 1));
    qb = qb + 2.0 * dxi(i) * qb / qa * (qc - qd);
    out[i - 1].c3 = 1.0 - qb;
    out[i - 1].c4 = qb;
    out[i - 1].c5 = dxi(i) / qa * qd;
    out[i - 1].c6 = -(dxi(i - 1) / qa * qc);
    out[i - 1].dx2i = 0.5 / dxi(i);
  }
}

// Segments of the marching stages.  A march along a whole pencil is a serial chain of n
// steps, so a batch with few pencils leaves the chip idle and waits for the chain: the
// pencils are cut (powers of two) until the batch has march_fill threads or a segment is
// down to kSegMin faces, each segment repeating the few cells of its neighbours that its
// first face and its first and last cells depend on.  Whole step, whole pencils -> cut
// (exact build unless stated): 100 cells in one dimension 501 -> 101 us, 256x192 1608 ->
// 161, 37x24x53 with HLLC 692 -> 240, 128^3 2703 -> 1879, 189x131x157 (tolerance) 3101 ->
// 2404.  march_fill is the chip's resident march threads (4 blocks of 128 an SM): with
// 2, 4 and 8 times that 128^3 measured 1865, 2168 and 2170 us in its sweeps against 1835,
// and 189x131x157 2711, 2525 and 2980 against 2339 (below 32 pencils a block the x sweep
// loses its staged stores); batches with more pencils than that (256^3 nearly, 512^3,
// levels) gain nothing from more threads and pay the repeated cells.
// Resident blocks per SM of the reconstruction (four keep a 256^3 sweep's pencils in a single
// wave) and of the transport kernel.
#ifndef PPM_RECON_MINBLOCKS
#define PPM_RECON_MINBLOCKS (4 * 128 / PPM_MARCH_THREADS)
#endif
#ifndef PPM_TRANS_MINBLOCKS
#define PPM_TRANS_MINBLOCKS (2 * 128 / PPM_MARCH_THREADS)
#endif
inline int64_t march_fill(int sms) { return (int64_t)sms * PPM_RECON_MINBLOCKS * kMarchThreads; }
inline int64_t transport_fill(int sms) {
  return (int64_t)sms * PPM_TRANS_MINBLOCKS * kMarchThreads;
}
#ifndef PPM_SEG_MIN
#define PPM_SEG_MIN 4
#endif
// The transport path (transport_kernel) holds half the resident threads of the kernels it
// replaces, so it pays where a batch fills the chip all the same.  Whole step, the two
// kernels -> transport (us): exact 80^3 622 -> 700, 96^3 979 -> 949, 128^3 1879 -> 1650,
// 900x900 690 -> 680, levels of 0.53 M cells 604 -> 657, of 1.5 M 1295 -> 1240; tolerance
// 64^3 283 -> 328, 80^3 403 -> 430, 900x900 (0.82 M cells) 573 -> 451, 96^3 673 -> 540.
#ifndef PPM_TRANSPORT_CELLS
#define PPM_TRANSPORT_CELLS 750000
#endif
inline bool use_transport(int64_t batch_cells) { return batch_cells >= PPM_TRANSPORT_CELLS; }
// Both reconstructions in one launch, where their blocks are resident together.
inline bool use_both_roles(int64_t seg_blocks, bool transport, int sms) {
  return !transport && 2 * seg_blocks <= (int64_t)sms * PPM_RECON_MINBLOCKS;
}
inline int64_t segment_blocks(const SweepArgs& a, int log_w) {
  return (a.npencils + (int64_t(1) << log_w) - 1) >> log_w;
}
// pgas2d_dual's energy of a cell may be formed without its left neighbour (see
// pgas2d_de_local, which needs 0 <= eta2: then a neighbour's energy can only keep the test
// from passing); otherwise the update needs whole pencils.
inline bool select_is_local(bool dual, double eta1, double eta2) {
  return !dual || (eta2 >= 0.0 && eta1 <= 0.25 * eta2);
}
// a: a record with its geometry; batch_pencils: pencils of all grids of the launch;
// local_select: select_is_local.
inline void set_segments(SweepArgs& a, int64_t batch_pencils, bool local_select, bool transport,
                         int sms) {
  int whole = 0;
  while ((1 << whole) < kMarchThreads) ++whole;
  const int faces = a.ie - a.is + 2;
  auto split = [&](int64_t fill, int& log_w) {
    int segs = 1;
    log_w = whole;
    while (segs < kMarchThreads && batch_pencils * segs < fill &&
           faces / (2 * segs) >= PPM_SEG_MIN) {
      segs *= 2;
      --log_w;
    }
    return segs;
  };
  int segs = split(march_fill(sms), a.pw_log2);
  a.seg_faces = (faces + segs - 1) / segs;
  if (local_select) {
    segs = split(transport ? transport_fill(sms) : march_fill(sms), a.uw_log2);
  } else {
    segs = 1;
    a.uw_log2 = whole;
  }
  // whole output chunks of the x sweep's staged stores
  const int cells = (a.n + segs - 1) / segs;
  a.seg_cells = (cells + 3) / 4 * 4;
}

// The record's shared coefficients, from its coefficient table on the host.
inline void set_uniform(SweepArgs& a, const double* width, const Coef* table) {
  // every width equal to the next: one comparison (a level prepares hundreds of grids)
  a.uniform = a.n < 2 || std::memcmp(width, width + 1, (size_t)(a.n - 1) * sizeof(double)) == 0;
  a.uc = table[a.is];
}

// Grid that owns block b of a stage, and the block's index inside that grid.
__device__ __forceinline__ int batch_locate(const int64_t* prefix, int ngrids, int64_t b,
                                            int64_t& local) {
  int lo = 0, hi = ngrids - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (prefix[mid] <= b) lo = mid; else hi = mid - 1;
  }
  local = b - prefix[lo];
  return lo;
}

}  // namespace ppm
