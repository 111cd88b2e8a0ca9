// gw_kernels.h -- host-side launch wrappers of the GWR kernels.
#pragma once

#include <cstddef>
#include <cuda_runtime.h>

#include "fx_geo.cuh"
#include "gw_common.cuh"

namespace gwgpu {

// Raises (never lowers) the dynamic shared memory limit of kernel fn on the
// current device to `bytes`; safe to call from concurrent host threads.
cudaError_t raise_smem_limit(const void* fn, size_t bytes);

// Dataset preparation on the device (k_prep.cu).  kPrepMin: points from which on it is
// faster than the host's.
constexpr int kPrepMin = 4096;
size_t hilbert_scratch_bytes(int n);
// perm: the points (2 x n, column-major) in Hilbert order over the grid
// ((u - umin) su, (v - vmin) sv), ties in index order.
cudaError_t launch_hilbert_order(int n, const double* coords, double umin, double su, double vmin, double sv, void* scratch,
                                 int* perm, cudaStream_t stream);
cudaError_t launch_gather_points(int n, const double* coords, const int* perm, bool radians, double* u, double* v,
                                 double* uR, double* vR, cudaStream_t stream);
// xs (n x p row-major) and ys from column-major x and y.
cudaError_t launch_gather_xy(int n, int p, const double* x, const double* y, const int* perm, double* xs, double* ys,
                             cudaStream_t stream);
// Planar tile boxes (null: not wanted), FP32 bounds and records.
cudaError_t launch_planar_proxy(int n, const double* u, const double* v, double uc, double vc, double slack, TileBox* box16,
                                TileBox* box32, float4* tb16, float4* tb32, float4* tb1024, float4* pts,
                                cudaStream_t stream);
// Statistics and scaled copies of the mixed form.  stat: p means, p scales, mean and
// scale of y, the intercept's column or -1 (2 p + 3 values); xs, ys: the centred and scaled
// X and y; tinv, tvec: the map of coefficients back.
size_t column_stats_bytes(int n, int p);
cudaError_t launch_column_stats(int n, int p, const double* x, const double* y, void* scratch, double* stat,
                                double* tinv, double* tvec, double* xs, double* ys, cudaStream_t stream);
// Integer coordinates; flags (two ints): a point does not fit, a bit was lost.
cudaError_t launch_int_coords(int n, const double* u, const double* v, double u0, double v0, int scale, longlong2* out,
                              int* flags, cudaStream_t stream);

// Solve modes of launch_solve.
enum SolveMode { kSolveAIC = 0, kSolveCV = 1, kSolveFit = 2, kSolveRefine = 3, kSolvePredict = 4 };

// Per-row k-th smallest distance (1-based rank), k_select.cu.
struct SelectArgs {
    int n, ntiles;                 // points, 32-point tiles
    DevPoints P;                   // FP64 coordinates (exact formula)
    const float4* pts;             // FP32 hi/lo proxy data (as the mixed path)
    const float4* tb;              // per tile: planar box (ulo, uhi, vlo, vhi) or cap (cx, cy, cz, rho)
    const float4* stb;             // per super-tile of 32 tiles (1024 points): the same bound, or null
    unsigned* hist_cache;          // n x 4096 proxy histograms of whole rows, or null
    int cache_valid;               // 1: hist_cache holds every row's histogram
    // n x 64: cumulative counts of hist_cache at the end of each 64-bin segment
    // (written by the histogram pass; used with cache_valid), or null
    unsigned* hist_coarse;
    unsigned rank;
    double dlo, dhi;               // expected range of positive distances (first histogram only)
    double eps, delta;             // proxy band: d in [p (1 - eps) - delta, p (1 + eps) + delta]
    double* out;
    int* err;                      // 2: a row's select failed (value left NaN)
    // Focus rows when they are not the data points (prediction): FP64
    // coordinates and FP32 records of F.n focus points.  Null F.u: the data.
    DevPoints F;
    const float4* fpts;
    // Geographic data rows only, or null: the distance cache that histogram pass
    // filled; the selects read their proxy values from it instead of recomputing them.
    const float* d2c;
    int* defer;                    // scratch of one int per focus row for exact geographic selects, or null
};
// exact: FP64 order statistics (bit-exact); otherwise the FP32 proxy's.
cudaError_t launch_select(const SelectArgs& a, bool geographic, bool exact, int num_sms, cudaStream_t stream);
size_t select_smem_bytes();
// Fills hist_cache with every row's whole-row proxy histogram (the cache a
// first select pass would store); the selects after it run with cache_valid.
cudaError_t launch_select_hist(const SelectArgs& a, bool geographic, int num_sms, cudaStream_t stream);
// The same histograms of geographic data rows read back from the filled
// distance cache a.d2c instead of recomputing the distances.
cudaError_t launch_select_hist_cached(const SelectArgs& a, int num_sms, cudaStream_t stream);
// Batched forms over many datasets and ranks in one launch each (device
// arrays of per-segment arguments; segment s owns the flattened items
// [start[s], start[s + 1])): whole-row histograms (items are groups of 8
// rows), selects (items are rows) and the FP32 copy of the thresholds.
cudaError_t launch_select_hist_batch(const SelectArgs* segs, const long long* start, int nseg, bool geographic,
                                     int num_sms, cudaStream_t stream);
cudaError_t launch_select_batch(const SelectArgs* segs, const long long* start, int nseg, bool geographic, bool exact,
                                int num_sms, cudaStream_t stream);
cudaError_t launch_to_float_batch(const double* const* in, float* const* out, const long long* start, int nseg,
                                  int num_sms, cudaStream_t stream);
constexpr int kSelHistRows = 8;  // rows per histogram item

// thr = fixbw of BandwidthWeight.cpp:40-53 from order statistics d0 (rank
// floor(bw), or the row maximum when bw >= n) and d1 (rank floor(bw)+1, may
// be null when bw is integral).
cudaError_t launch_threshold_combine(int n, double bw, const double* d0, const double* d1, double* thr,
                                     cudaStream_t stream);
// The same for `rows` focus rows over n data points (dn = bw / n).
cudaError_t launch_threshold_combine_rows(int rows, int n, double bw, const double* d0, const double* d1, double* thr,
                                          cudaStream_t stream);

// out[i] = (float)in[i].
cudaError_t launch_to_float(int n, const double* in, float* out, cudaStream_t stream);

// Z[j, :] = (upper triangle of x_j x_j^T packed by rows, x_j * y_j); X row-major n x p.
cudaError_t launch_build_z(int n, int p, const double* X, const double* y, double* Z, cudaStream_t stream);

// G[i, c] = sum_j w_ij^wpow Z[j, c] for c < mcols, with w_ij = K(d_ij, r_i)
// (r_i = thr[i], or bw when thr is null); exclude_self zeroes w_ii (CV).
// FP64 SIMT, the weight matrix is produced tile by tile and never stored.
// tb16: FP32 bounds of the 16-point tiles (planar box or geographic cap).
// blocks (optional): only some of the 64-row blocks.
struct RowBlocks {
    const int *flags, *all;  // those with a nonzero flag, or every one when *all is nonzero
    // or an ordered list of them, whose tiles are split nsplit ways where that many blocks
    // leave SMs idle (part: nsplit x count x 64 x mcols doubles of scratch)
    const int* list;
    int count, nsplit;
    double* part;
};
cudaError_t launch_contract64(const DevPoints& P, bool geographic, const float4* tb16, const double* Z, int ldz,
                              int mcols, double* G, int ldg, const double* thr, double bw, int kernel,
                              bool exclude_self, int wpow, bool skip_tiles, cudaStream_t stream,
                              const RowBlocks& blocks = RowBlocks{});
// The same with focus rows F (their 16-point tile bounds ftb16) that are not
// the data points: G[i, :] for every focus row i over the data P (predict).
cudaError_t launch_contract64_focus(const DevPoints& P, const float4* tb16, const DevPoints& F, const float4* ftb16,
                                    bool geographic, const double* Z, int ldz, int mcols, double* G, int ldg,
                                    const double* thr, double bw, int kernel, bool exclude_self, int wpow,
                                    bool skip_tiles, cudaStream_t stream, const RowBlocks& blocks = RowBlocks{});
// Splits of the tiles for `count` row blocks.
int contract64_splits(int count, int ntiles, int num_sms);

// Which rows of fixed-point sums are less exact than FP64 ones because a column of X
// rests on small weights there (a covariate that is zero near the row's location): the
// sums' errors are absolute, so the diagonals G_kk tell.  A row is low when G_kk of a
// column is below
//     lim_k = max(2^-17 T_k, 2^-14 V_k),  V_k = sqrt(sum_j 4^e_jk),
// T_k = sum_j x_jk^2 (truncated weights: 2^-60 T_k at most) and e_jk the exponent of the
// scale of each nonzero x_jk^2 (dropped digits: 2^-62 V_k, root mean square); 2^-14 T_k for
// squared weights.  Off-diagonal errors follow by Cauchy's inequality.  Measured against
// long double sums (2,000 and 10,000 points, an indicator or a lognormal column, gaussian
// and bisquare): above these lines coefficients are at most 1.1e-15 off and squared sums
// 1.2e-15, FP64 weights 2.3e-15 and 2.6e-15; at 2^-20 to 2^-25 they are 3e-14 and 3e-12 off.
// T_k and V_k count at most `points` points of the largest value (a compact kernel's
// neighbours).  The limits come with the sums (launch_contract_fx); the solve, which
// reads every G_kk anyway, tests them: flags[row / 64] and *any are set.
struct FxLimits {
    int p;               // columns of X
    double points, root; // and its square root
    const double* zsum;  // launch_build_zfx's
    const int* off;      // nonzero: FP64 sums follow, every limit is 0
    double* lim;         // p limits; null: none wanted
};
struct FxGuard {
    const double *lim, *lim2;  // limits of G and, optional, of G2 (fit mode); null: no test
    const int* done;           // optional: 64-row blocks that hold FP64 sums already
    int *flags, *any;          // *any: 1, and 2 for a row that is not one of a single variable of value 0
};

// The same sums on the tensor cores, in 62-bit fixed point (k_contract_fx.cu):
// bisquare and gaussian weights; geographic points within one spherical cap of
// chord radius 1/2.
// The mixed modes take the mixed contraction's FP32 weights (any kernel).
enum FxMode { kFxBisquare, kFxGauss, kFxGeoBisquare, kFxGeoGauss, kFxMixed, kFxMixedGeo };
struct FxArgs {
    int n, nf, ntiles;          // data points, focus rows, 16-point tiles
    const longlong2* pxy;       // integer coordinates of the data (u - u0, v - v0) 2^scale
    const longlong2* fxy;       // and of the focus rows
    int scale, exact;           // exact: no coordinate was rounded
    const fx::Vec3 *pe3, *fe3;  // geographic: unit vectors of the data and of the focus rows
    const fx::GeoCoef* geo;     // geographic: fx::geo_table
    const float4 *pts, *fpts;   // mixed modes: FP32 records, thresholds, kernel and, optional, the distance cache
    const float* thr32;
    int kernel;
    const float* d2c;
    const float4* tb16;         // FP32 bounds of the 16-point tiles of the data
    const float4* ftb16;        // and of the focus rows
    const double* thr;          // per-row threshold, or null for the fixed bandwidth bw
    double bw;
    int exclude_self, wpow;
    int ncols, N, zgroups;      // columns wanted, columns per group, groups of the Z image
    const unsigned char* zimg;  // launch_build_zfx
    const int* zexp;
    int zcols;                  // columns of zexp (N x groups of the image)
    double* out;                // split s: rows of ldo doubles at out + s split_stride
    size_t split_stride;
    int ldo;
    const double* rowscale;     // optional (one split only): row i's sums are multiplied by rowscale[i]
    unsigned* rowmax;           // splits x nf: high words of the largest weight
    int* err;                   // set to 1 if a bounded wait timed out
    unsigned wait_limit;        // polls of a pipeline wait before it times out (0: the default)
    int group0, groups;         // column groups of this launch (groups 0: all of ncols)
    // Weights kept for further passes over the same rows, points and thresholds: row block x
    // tile x 16 points x 128 rows (fx_weight_bytes); wstore writes them, wload reads them.
    unsigned long long* wstore;
    const unsigned long long* wload;
    FxLimits limits;
};
// Bytes of the kept weights of nf rows and n points.
size_t fx_weight_bytes(int nf, int n);
// Columns per group (a multiple of 16, at most 64) and groups for ncols columns of Z.
int fx_columns(int ncols, int* groups);
bool fx_fits(int N, int ntiles);  // whether a CTA's shared memory holds the tile mask too
int fx_splits(int blocks, int ntiles, int num_sms);
// Unit vectors times 2^61 of n points in radians.
cudaError_t launch_int_vectors(int n, const double* lon, const double* lat, fx::Vec3* out, cudaStream_t stream);
// img: (n / 16 tiles rounded up) x groups x N x 256 bytes; zexp: scale blocks of
// 1024 points x (N groups); *bad: whether Z needs FP64 sums instead.  With x the
// operand is x_j (Z[j, c] + [j = c]) (the multiscale hat update).  zsum (null with x): per
// entry of zexp the sum of |Z| and the number of nonzeros.
cudaError_t launch_build_zfx(int n, int ncols, int N, int groups, const double* Z, int ldz, const double* x,
                             unsigned char* img, int* zexp, double* zsum, int* bad, cudaStream_t stream);
// r = b - A beta of every row's packed normal equations (n x p), and for each kResidualRows
// rows in low[] whether a diagonal is below its limit (FxLimits::lim).
constexpr int kResidualRows = 8;
cudaError_t launch_normal_residual(int n, int p, const double* G, int ldg, const double* beta, const double* lim,
                                   double* r, int* low, cudaStream_t stream);
cudaError_t launch_contract_fx(const FxArgs& a, int mode, int nsplit, cudaStream_t stream);
// Sums the splits into G and, with flags, marks the 64-row blocks that need FP64 sums.
cudaError_t launch_fx_finish(const FxArgs& a, int nsplit, double* G, int ldg, int* flags, cudaStream_t stream);

// Warp-per-location Cholesky solve of A_i beta_i = b_i and the per-location
// criterion terms; partial sums per block in partials[block*4 + {0..3}] =
// (sum s_ii, sum residual^2, sum ||s_i||^2, failures).  Returns the number
// of partial blocks through nblocks.
//
// Where the sums go when the caller waits for them: pinned host memory, written by the
// kernel that forms them (host[0 .. 3] the sums, then as integers host[4] = *err,
// host[5] = *sel_err, host[6 .. 7] = fx_state[0 .. 2]; null sources are left out).  A copy per
// value cost about 2.5 us each on the stream.  ticket: a zeroed counter, zero again afterwards.
struct CriterionOut {
    double* host;
    const int *err, *sel_err, *fx_state;  // fx_state: three words
    unsigned* ticket;
};
struct SolveArgs {
    int n, p, mode, kernel;
    const double* G;   // n x m (A packed upper, then b)
    int ldg;
    const double* G2;  // n x p(p+1)/2 (X^T W^2 X packed upper), fit only
    int ldg2;
    const double* X;   // n x p row-major
    const double* y;
    const double* thr; // per-row threshold or null
    double bw;
    double* beta;      // n x p row-major
    double* sii;       // n
    double* resid;     // n
    double* v;         // n x p: A_i^{-1} x_i (fit)
    double* bse;       // n x p: diag(T A^-1 Q A^-1 T^T) (fit)
    double* partials;
    // Optional linear map T of the coefficients (fit): T = diag(tinv) except
    // row tcol = tvec (the intercept row after centring).  Null: identity.
    const double* tinv;
    const double* tvec;
    int tcol;
    // Refine mode: beta += A^-1 rvec (n x p), then the residuals are recomputed.
    const double* rvec;
    // Fit mode, optional: A_i^-1 (n x p x p, row-major per row).
    double* ainv;
    // launch_solve, optional: the partial blocks are summed too (as launch_reduce_partials)
    CriterionOut out;
    FxGuard guard;
};
// Largest grid launch_solve uses; callers size `partials` (4 doubles per block) for it.
constexpr int kSolveMaxBlocks = 4096;
cudaError_t launch_solve(const SolveArgs& a, int* nblocks, cudaStream_t stream);
// Criterion solves (kSolveAIC / kSolveCV) of many segments in one launch:
// block b solves rows [work[b].y, work[b].z) of segment work[b].x and writes
// partial slot work[b].w of that segment (device arrays; p <= max_p).
cudaError_t launch_solve_batch(const SolveArgs* segs, const int4* work, int nwork, int mode, int max_p,
                               cudaStream_t stream);
// out[4 s .. 4 s + 3] = fixed-order sums of partial blocks [first[s], first[s + 1]).
cudaError_t launch_reduce_batch(const double* partials, const int* first, int nseg, double* out, cudaStream_t stream);

// Sums nblocks x 4 partials into out[4] in a fixed order.
cudaError_t launch_reduce_partials(const double* partials, int nblocks, double* out, cudaStream_t stream);

// qdiag[j] = sum_i (delta_ij - s_ij)^2 with s_ij = w_ij v_i . x_j, w_ij =
// K(d_ij, r_i); also writes S when S != null and row row_target of S into
// s_row[perm[j]] when s_row != null.
enum HatMode { kHatPlanar, kHatGeo, kHatFxBisquare, kHatFxGauss, kHatFxGeoBisquare, kHatFxGeoGauss };
struct HatArgs {
    DevPoints P;
    const float4* tb16;
    const float* tile_thr;  // far-test threshold of each 16-point tile's largest r_i (launch_tile_far_thr)
    const double* X;        // n x p row-major
    int p;
    const double* v;        // n x p
    const double* thr;
    double bw;
    int kernel;
    const longlong2* xy;    // planar: integer coordinates for fixed-point weights, or null
    const fx::Vec3* e3;     // geographic: integer unit vectors for fixed-point weights, or null
    const fx::GeoCoef* geo; // (with e3)
    fx::Row* rows;          // scratch of n rows (with xy or e3)
    double* S;              // n x n zeros: s_ij goes to S[perm[i] + perm[j] n] (column-major, original order)
    const int* perm;        // sorted position -> original index
    int row_target;         // -1: none
    double* s_row;
    double* qsum;           // scratch of nsplit x n
};
int hat_splits(int n, int num_sms);
cudaError_t launch_hat_pass(const HatArgs& a, bool geographic, int scale, int nsplit, double* qdiag,
                            cudaStream_t stream);

// Column subsets of X, all of one size, for the w == 1 criterion of variable selection.
struct SubsetList {
    int count;  // columns of each
    unsigned char cols[kMaxP][kMaxP];
};

// out[c] = sum_j Z[j, c] (n x m row-major) with nb fixed partial blocks (part: nb x m).
cudaError_t launch_column_sums(int n, int m, const double* Z, double* part, int nb, double* out, cudaStream_t stream);

// out[4 s .. 4 s + 3] = (tr S, RSS, 0, failures) of the w == 1 model on subset s, from the
// full column sums gall.  partials: 4 doubles per block and subset; first: the device
// array s global_criteria_blocks(n) for s = 0 .. subsets.
int global_criteria_blocks(int n);
cudaError_t launch_global_criteria(int n, int p, const SubsetList& list, int subsets, const double* X, const double* y,
                                   const double* gall, double* partials, const int* first, double* out,
                                   cudaStream_t stream);

// Mixed-precision W.Z contraction on tcgen05 (k_contract_tc.cu).
struct TcArgs {
    int n, mcols, npad, ntiles;   // ntiles: 32-point tiles
    const float4* pts;            // planar: {u_hi, u_lo, v_hi, v_lo}; geographic: 2 float4 (hi/lo unit vector)
    const float4* tb;             // FP32 bound of each 32-point tile (planar box or geographic cap)
    const unsigned char* zimg;    // per tile: [hi | lo] swizzled images, npad x 128 bytes each
    const float* thr;             // per-row threshold, or null for the fixed bandwidth bw
    float bw;
    int kernel, exclude_self, skip, flush_tiles, wpow;
    float2* acc;                  // double-float sums: ceil(n / 128) x npad x 128 (rows in groups of 128)
    float* stage;                 // FP32 staging of one chunk, same layout (single-accumulator form), or null
    double* G;                    // n x ldg FP64 output (first mcols columns)
    int ldg;
    int* err;                     // set to 1 if a bounded wait timed out
    unsigned long long* tiles;    // if not null: += 128 x 32 weight tiles processed
    unsigned long long* prof;     // if not null: += clock64 cycles per phase (kTcProfSlots slots)
    const float* d2c;             // geographic only, optional: the distance cache of launch_fill_d2_sym
    unsigned wait_limit;          // polls of a pipeline wait before it times out (0: the default)
    // Splits of a row block's chunks (0 or 1: none); split s has its own acc and stage, acc_stride
    // elements on, and launch_contract_tc sums them.
    int nsplit;
    size_t acc_stride;
};
// Splits for row blocks that visit about `tiles` tiles each.
int tc_splits(int blocks, int tiles, int flush_tiles, int num_sms);
// Phase slots of TcArgs::prof, summed over CTAs (producer: warp 0 lane 0;
// control: the issuing thread).
enum TcProf {
    kTcProfStageWait,   // producer: waiting for a free weight stage
    kTcProfPointsWait,  // producer: waiting for the tile's point records
    kTcProfWeights,     // producer: weights, split and shared-memory stores
    kTcProfFlush,       // drain warp 0: draining accumulators
    kTcProfAWait,       // control: waiting for the weight tile
    kTcProfZWait,       // control: waiting for the Z tile and a free accumulator
    kTcProfIssue,       // control: MMA issue and Z prefetch
    kTcProfLoop,        // producer: whole tile loop
    kTcProfLoopMax,     // producer: largest tile loop of one CTA (maximum, not a sum)
    kTcProfPrologue,    // producer: kernel start to tile loop
    kTcProfEpilogue,    // producer: tile loop end to kernel end
    kTcProfTilesMax,    // largest number of tiles one CTA processed (maximum, not cycles)
    kTcProfSlots
};
size_t contract_tc_smem_bytes(int npad, int ntiles, int nb, bool cached);
cudaError_t launch_contract_tc(const TcArgs& a, bool geographic, cudaStream_t stream);
// Many contractions in one launch: CTA b computes row block work[b].y of
// segment work[b].x (device arrays; every segment's npad <= max_npad and
// ntiles <= max_ntiles; flush_tiles and the weight kernel are shared).
cudaError_t launch_contract_tc_batch(const TcArgs* segs, const int2* work, int nwork, int max_npad, int max_ntiles,
                                     int flush_tiles, bool geographic, int kernel, cudaStream_t stream);
cudaError_t launch_build_zimg(int n, int mcols, int npad, const double* Z, int ldz, unsigned char* img,
                              cudaStream_t stream);
// Distance cache of the mixed geographic contraction: the FP32 squared
// great-circle distance of every (focus row, data point) pair, exactly the
// value the contraction's weight producer computes, for rows padded to whole
// 128-row blocks and points padded to whole 32-point tiles.  Block (rb, tile)
// is 4096 floats at ((rb * ntiles + tile) * 4096), ordered [quarter 4][half 2]
// [row 128][4 points] so the producer thread of (row, quarter) reads its 8
// points as two float4 and a warp's loads are contiguous; padded pairs hold
// FLT_MAX.  pts: the 2 float4 records per point, padded to whole tiles.
size_t d2_cache_bytes(int n);
// The distance cache of geographic mixed data: every pair's FP32 squared
// distance, block (row block rb of 128 rows, 32-point tile t) of 4096 floats at
// (rb * ntiles + t) * 4096, ordered [quarter 4][half 2][row 128][4 points].
// Each pair is computed once (the FP32 distance is symmetric) and written to
// both rows.  scratch: ceil(n / 128) + 2 ints of device memory.
cudaError_t launch_fill_d2_sym(int n, const float4* pts, float* d2c, int* scratch, int num_sms, cudaStream_t stream);
// D[128 x N] = A[128 x 32] B[N x 32]^T through tcgen05 (device pointers).
cudaError_t launch_tc_selftest(const float* A, const float* B, float* D, int N, int* err, cudaStream_t stream);

// Refinement residual of the mixed path: r_i = X~^T W_i (y~ - X~ beta_i) in
// FP64 arithmetic over the FP32 weights of the contraction (n x p output).
struct RefineArgs {
    int n, p, ntiles, kernel, skip;
    const float4* pts;
    const float4* tb;     // FP32 bound of each 32-point tile
    const double* X;      // n x p row-major (X~)
    const double* y;      // y~
    const double* beta;   // n x p
    const float* thr;
    float bw;
    double* r;            // n x p
    const float* d2c;     // geographic only, optional: the distance cache (the contraction's FP32 d^2)
    const int* low;       // optional: only the 128-row blocks with a mark of launch_normal_residual
};
cudaError_t launch_refine_residual(const RefineArgs& a, bool geographic, cudaStream_t stream);

// Mixed-precision hat pass: the FP32 weights of the tensor-core contraction.
struct HatMixedArgs {
    int n;
    const float4* pts;
    const float4* tb16;
    const float* tile_thr;
    const double* X;
    int p;
    const double* v;
    const float* thr32;
    float bw;
    int kernel;
    const float* d2c;  // geographic only, optional: the distance cache
    double* S;         // as HatArgs
    const int* perm;
    int row_target;
    double* s_row;
    double* qsum;      // scratch of nsplit x n
};
cudaError_t launch_hat_mixed(const HatMixedArgs& a, bool geographic, int nsplit, double* qdiag, cudaStream_t stream);

// Results of the sorted rows in the original order: dst[q][perm[s] + k n] =
// src[q][s p[q] + k] for the first `count` of three.  With musc (p means, then p
// scales) src[0] holds the coefficients of the centred and scaled mixed problem:
// beta_k = s_y beta~_k / scale_k, and the intercept column icol (-1: none) takes
// mu_y and the other columns' means back.
struct UnpermuteArgs {
    int n;
    const int* perm;
    int p[3];
    const double* src[3];
    double* dst[3];
    const double* musc;
    double s_y, mu_y;
    int icol;
};
cudaError_t launch_unpermute(const UnpermuteArgs& a, int count, cudaStream_t stream);

// tile_thr[t] = far-test threshold of the largest r_i (thr, or bw) over tile t of `tile` points.
cudaError_t launch_tile_far_thr(int n, int tile, bool geographic, const double* thr, double bw, float* tile_thr,
                                cudaStream_t stream);

// Maximum pairwise distance (CRSDistance::maxDistance) as an ordered key: key_out[0]
// for planar data, key_out[1] for geographic data (key_out[0] then holds the
// unit-vector form's maximum).  Both keys start at 0; rowmax (geographic only)
// holds n doubles of scratch.  boxes32 / caps32: FP64 bounds of the 32-point tiles.
cudaError_t launch_max_distance(const DevPoints& P, bool geographic, const TileBox* boxes32, const TileCap* caps32,
                                unsigned long long* key_out, double* rowmax, int num_sms, cudaStream_t stream);


// GWRMultiscale hat matrix (k_mgwr.cu).  Matrices are n x n row-major in the
// sorted order; SA holds p of them back to back.
size_t mgwr_hat_all_smem(int p);
// SA_k(i, j) = w_ij x_ik (A_i^-1 x_j)_k and S0(i, j) = sum_k SA_k(i, j) for
// every pair (ainv: n x p x p from the fit's solve).
cudaError_t launch_mgwr_hat_all(const DevPoints& P, bool geographic, const double* X, int p, const double* ainv,
                                const double* thr, double bw, int kernel, double* S0, double* SA, int num_sms,
                                cudaStream_t stream);
// T = SA - S0 over count elements.
cudaError_t launch_mgwr_sub(size_t count, const double* SA, const double* S0, double* T, cudaStream_t stream);
// SA = S (T + I) for the one-variable hat matrix S(i, j) = w_ij v_i x_j, over
// neighbouring data tiles only where the kernel is compact (bisquare, tricube,
// boxcar) (X: the variable, v: A_i^-1 x_i from the fit, both n sorted).  With unless, only
// when *unless is nonzero.
cudaError_t launch_mgwr_hat_update(const DevPoints& P, bool geographic, const float4* tb16, const double* X,
                                   const double* v, const double* thr, double bw, int kernel, const double* T,
                                   double* SA, const int* unless, cudaStream_t stream);
// SA += S (S may be null: no addition); S0 = SA - T over count elements.
cudaError_t launch_mgwr_post(size_t count, double* SA, const double* S, const double* T, double* S0,
                             cudaStream_t stream);
// partials[4 b + 0] / [4 b + 1]: block b's share of tr(S0) and of sum S0_ij^2;
// *nblocks receives the block count (at most max_blocks).
cudaError_t launch_mgwr_traces(int n, const double* S0, double* partials, int max_blocks, int* nblocks,
                               cudaStream_t stream);

}  // namespace gwgpu
