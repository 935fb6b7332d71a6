// Internal declarations shared by the segpu CUDA sources (not installed).
//
// Device data layout
//  - Field values: double[nVertsTotal][ndofs] in the reference's vertex
//    order (x fastest, periodic duplicates stored), so that host uploads and
//    downloads are single copies and the SL gathers read an element's
//    (N+1)^2 block as N+1 contiguous rows of N+1 values.
//  - Solver vectors ("unknowns"): the reference's vector ordering, which on
//    SE's regular Cartesian meshes is always a row-major rectangle of the
//    vertex grid: rows [lo_y, hi_y), columns [lo_x, hi_x). Dirichlet and
//    periodic-duplicate vertices are not unknowns.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

#define SE_MAXN 12
#define SE_MAXN1 (SE_MAXN + 1)

namespace seg {

// Everything a kernel needs to know about one mesh (passed by value; lives
// in the kernel parameter bank).
struct MeshDev {
  int N;
  int nEls[2];
  int nVerts[2];
  int periodic[2];
  double min[2], max[2], dx[2];
  double two_over_dx[2];  // 2.0/dx, rounded as the reference rounds it
  double inv_dx[2];       // 1.0/dx
  int snaps;  // every vertex's coordinates give back that vertex (element search and node snap)
  double span[2];         // max - min
  double nspan[2];        // min - max
  double abcissa[SE_MAXN1];
  double lambda[SE_MAXN1];  // 1 / prod_{k != j} (x_j - x_k): Lagrange product weights
  double w[SE_MAXN1];       // GLL weights
  double dC[SE_MAXN1 * SE_MAXN1];  // cardinal derivative matrix, row = point
};

// One direction of the tensor-product operator on the unknown grid.
struct Dir {
  int nE, N, nV;
  int periodic;
  int lo, hi;  // unknown vertex range [lo, hi)
};

// A = alpha (W x W) + beta[0] (Kx x W) + beta[1] (W x Ky): the assembled
// c*Mass + s*Laplacian of SE on a uniform Cartesian GLL mesh, with Kh the
// 1-D reference-element stiffness and W the assembled 1-D GLL weights.
struct OpDev {
  Dir d[2];
  int G[2];  // unknowns per direction
  double alpha;
  double beta[2];
  double Kh[SE_MAXN1 * SE_MAXN1];
  double w[SE_MAXN1];
  // Spectral vanishing viscosity (HelmholtzEqn with svvCutoff != 0):
  // + gamma (Sv along x (x) Tv along y), the assembled 1-D element matrices
  // S = (F D)^T diag(w) (F D) and T = F^T diag(w) F of the modal filter F;
  // gamma == 0: no such term (and Sv, Tv unused).
  double gamma;
  double Sv[SE_MAXN1 * SE_MAXN1];
  double Tv[SE_MAXN1 * SE_MAXN1];
};

// Device-side error bits (a single unsigned word per library instance).
enum : unsigned {
  KERR_DOMAIN = 1u,            // departure point outside the mesh after the wrap
  KERR_BARRIER_TIMEOUT = 2u,   // a grid barrier wait gave up
  KERR_BAD_CONFIG = 4u,
};

// ---- exact-rounding arithmetic: the reference's coordinate operations, one
// IEEE operation at a time, never contracted into FMAs.
__device__ __forceinline__ double xadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double xsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double xmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double xdiv(double a, double b) { return __ddiv_rn(a, b); }

// ---- double-double arithmetic (error-free transformations: Knuth's TwoSum;
// TwoProd with an FMA): a pair (hi, lo) carries a value to about twice double
// precision. The _rn intrinsics keep each operation one IEEE operation (the
// compiler must not fuse a product into a following sum here).
__device__ __forceinline__ void two_sum(double a, double b, double& s, double& e) {
  s = __dadd_rn(a, b);
  const double bb = __dsub_rn(s, a);
  e = __dadd_rn(__dsub_rn(a, __dsub_rn(s, bb)), __dsub_rn(b, bb));
}
__device__ __forceinline__ void dd_add(double& hi, double& lo, double x) {
  double s, e;
  two_sum(hi, x, s, e);
  hi = s;
  lo += e;
}
__device__ __forceinline__ void dd_fma(double& hi, double& lo, double a, double b) {
  const double p = __dmul_rn(a, b);
  const double pe = fma(a, b, -p);  // exact: a*b - p
  dd_add(hi, lo, p);
  lo += pe;
}

constexpr int kSms = 148;  // of a B200
// Largest y extent of a grid: more rows of blocks take several launches.
constexpr int kGridRows = 65535;

// ---------------------------------------------------------------------------
// Host launch wrappers (defined in sl.cu / linsys.cu). All take the stream.

// SL advection. field: [Nv][ndofs]; vel/vel_prev: [Nv][2]; out: [Nv][ndofs].
// field_prev == nullptr selects the first-order scheme. dep_el/dep_xy are
// optional recordings of the departure elements/points (all vertices). mix
// (second order, nullable): work for the half-level velocities, 4 doubles a
// vertex; without it they are formed at every gathered vertex.
cudaError_t launch_sl(const MeshDev& m, int ndofs, const double* field, const double* vel,
                      const double* field_prev, const double* vel_prev, double* mix, double dt,
                      double* out, int* dep_el, double* dep_xy, unsigned* err, cudaStream_t s);
// Gathered values of one interpolation over the mesh, nv (N+1)^2, from which
// the second-order advection forms the half-level velocities once per vertex
// (a launch more) instead of at every gathered one: at 37,249 vertices, p = 6
// (1.8M) 16.0 us against 16.5, p = 3 (0.6M) 11.8 against 8.3; at 295,425
// vertices, p = 6 54 against 65.
constexpr size_t kSlMixMin = (size_t)2 << 20;
// Mesh::GlobalToLocal at points (device arrays).
cudaError_t launch_global_to_local(const MeshDev& m, const double* pts, int npts, int* el,
                                   double* lc, cudaStream_t s);
// Field::InterpGlobal at points (device arrays).
cudaError_t launch_interp_global(const MeshDev& m, int ndofs, const double* vals,
                                 const double* pts, int npts, double* out, cudaStream_t s);
// NavierStokesEqn pressure step (sl.cu): kind 0 out = div(a) (a 2
// components), kind 2 out = div(a) * 1.5 * 10.0, kind 1 out = a - dt grad p;
// derivatives as InterpDerivsGlobal at the vertices. err (may be null) gets
// KERR_BAD_CONFIG if a vertex does not snap to an element's nodes.
cudaError_t launch_ns_pressure(const MeshDev& m, int kind, const double* a, const double* p,
                               double dt, double* out, unsigned* err, cudaStream_t s);
// Component dof of a 2-component field to (to_scalar) or from a scalar field.
cudaError_t launch_component(int nv, int to_scalar, int dof, double* two, double* one,
                             cudaStream_t s);
// Two-layer QG step pieces (sl.cu): GenPV; pointwise combinations (kind 0
// Helmholtz rhs, 1 Poisson rhs, 2 stream functions and vorticities); SolveQ
// with the dissipation rhs over the unknowns of (dx, dy). grad is
// vel-layout (-d/dy, d/dx) of omegaHat from launch_gen_vel.
cudaError_t launch_gen_pv(const MeshDev& m, const double* omega, const double* psi_i,
                          const double* psi_j, double F, double beta, double* alpha, cudaStream_t s);
cudaError_t launch_qg_combine(const MeshDev& m, int kind, const double* a, const double* b,
                              const double* t, const double* c, double F1, double F2, double cb,
                              double* out0, double* out1, double* out2, double* out3,
                              cudaStream_t s);
cudaError_t launch_qg_solve_q(const MeshDev& m, const Dir& dx, const Dir& dy, double dt,
                              const double* q, const double* tau, const double* omh,
                              const double* grad, const double* tau_e, double rF, double Ei,
                              double nu, double a, double* alpha, cudaStream_t s);
// vel[Nv][2] = (-d psi/dy, d psi/dx) at every vertex (GenVel of SE's QG models).
cudaError_t launch_gen_vel(const MeshDev& m, const double* psi, double* vel, unsigned* err,
                           cudaStream_t s);
// Field::PeriodicUpdate.
cudaError_t launch_periodic_update(const MeshDev& m, int ndofs, double* vals, cudaStream_t s);
// Quadrature sums over all elements: sum detJ*w*a (Integrate) or, with
// b != nullptr, sums of detJ*w*(a-b)^2 and detJ*w*b^2 (FieldError).
// Results land in out2[0..1] (device), deterministic order.
cudaError_t launch_quadrature(const MeshDev& m, int ndofs, int dof, const double* a,
                              const double* b, double* scratch, int nscratch, double* out2,
                              cudaStream_t s);
// Max over vertices of |v|^2 (CalcTimeStep), deterministic.
cudaError_t launch_max_speed_sq(int nv, const double* vel, double* scratch, int nscratch,
                                double* out, cudaStream_t s);

// Linear-system pieces.
// y = A x, element-structured (apply.cu); the reduced-precision form reads
// x in FP16 (fp16 != 0) or BF16 and computes and writes FP32.
cudaError_t launch_op_apply(const OpDev& op, const double* x, double* y, cudaStream_t s);
cudaError_t launch_op_apply_low(const OpDev& op, int fp16, const void* x, float* y, cudaStream_t s);
// r = b - A x with per-block partial sums (partial[2*block]: (w r)^2 or, when
// natural, r w r; and r^2) over residual_blocks(op) blocks (cg.cu).
cudaError_t launch_residual(const OpDev& op, const double* x, const double* b, double* r,
                            const double* w, int natural, double* partial, cudaStream_t s);
// The same residual with the FDM refinement loop's tail fused in: the block
// that finishes last (arrival counter *count, zero between launches) sums
// the partials in block order into res[0..1], runs the convergence test on
// the loop state and sets the loop's while-condition h.
// split_hi/split_lo (nullable): also write r's TF32 hi/lo split, rows of
// split_pitch FP32 (the tensor-core inverse's input).
struct FdmParams;
struct FdmState;
struct ResTail {
  double* res;
  unsigned* count;
  const FdmParams* p;
  FdmState* st;
  cudaGraphConditionalHandle h;
};
cudaError_t launch_residual_check(const OpDev& op, const double* x, const double* b, double* r,
                                  const double* w, int natural, double* partial, double* res,
                                  unsigned* count, const FdmParams* p, FdmState* st,
                                  cudaGraphConditionalHandle h, cudaStream_t s,
                                  float* split_hi = nullptr, float* split_lo = nullptr,
                                  int split_pitch = 0);
// The element-factored residual of orders 4 to 8 without an SVV term
// (apply.cu); false when the operator needs the general kernel.
bool residual_ef_supported(const OpDev& op);
// Partial-sum pairs launch_residual (with b and partial given) writes.
int residual_partial_blocks(const OpDev& op);
cudaError_t launch_residual_ef(const OpDev& op, const double* x, const double* b, double* r,
                               const double* w, int natural, double* partial, const ResTail& tail,
                               float* split_hi, float* split_lo, int split_pitch, cudaStream_t s);
int residual_blocks(const OpDev& op);
cudaError_t launch_op_diag(const OpDev& op, double* d, cudaStream_t s);
// f = Mass*rhs over the unknowns (FieldRHS + Vector::Assemble), plus lift.
cudaError_t launch_rhs_assemble(const OpDev& op, const MeshDev& m, const double* rhs_vals,
                                const double* lift, double* f, cudaStream_t s);
// lift = -A[unknowns, Dirichlet] * sol_vals[Dirichlet].
cudaError_t launch_lift(const OpDev& op, const MeshDev& m, const double* sol_vals, double* lift,
                        cudaStream_t s);
// dst[0, n) = src[0, n) on the stream (device arrays that do not overlap).
cudaError_t launch_copy(double* dst, const double* src, size_t n, cudaStream_t s);
// sol_vals[unknown vertices and their periodic copies] = x; with st and
// st_host (the device address of a mapped page-locked buffer) also
// *st_host = *st.
cudaError_t launch_update_field(const OpDev& op, const MeshDev& m, const double* x,
                                double* sol_vals, cudaStream_t s, const FdmState* st = nullptr,
                                FdmState* st_host = nullptr);

// Persistent CG over a batch of solves.
struct CgSolve {
  OpDev op;
  const double* b;  // right-hand side (unknowns)
  double *x, *r, *z, *p0, *p1, *w;
  double* dinv;     // Jacobi inverse (streaming mode only)
  double rtol, atol, dtol;
  int max_it;
  int norm_type;
  int remove_null;
  int n;  // unknowns
  // segment range of this solve in the partial-sum table
  int seg_begin, seg_end;
  // state (written by the kernel)
  double beta, betaold, dpi, dpiold, rnorm0, ttol, dp, bcoef, a, zmean;
  int its, reason, done, pbuf;
};
struct CgTile {
  int solve;
  int x0, y0;  // first unknown column/row of the tile
  int seg;     // partial-sum segment this tile accumulates into
};
struct CgBatch {
  CgSolve* solves;  // device array
  int nsolves;
  const CgTile* tiles;  // device array, grouped by block (contiguous chunks)
  const int* block_tile_begin;  // [grid+1]
  double* partials;  // [2][nseg][4]: double-buffered by pass parity
  int nseg;
  unsigned* bar_count;
  unsigned* bar_gen;
  int* n_active;
  unsigned* err;
};
constexpr int kCgTileX = 32;
constexpr int kCgTileY = 16;
constexpr int kCgThreads = kCgTileX * kCgTileY;
// Shared memory of the standalone operator apply for order maxN.
size_t cg_smem_bytes(int maxN);
// Tiles a block may own in the register-resident CG mode.
constexpr int kCgResidentTiles = 4;
// Dynamic shared memory of one CG block (order N, nsolves per launch).
size_t cg_dyn_smem_bytes(int N, int nsolves);
// Blocks of kCgThreads that can be co-resident for the CG kernel.
int cg_max_grid(int device, int N, bool resident, int nsolves, int lowp = 0);
// Persistent CG over a batch of same-order solves; resident needs every block
// to own at most kCgResidentTiles tiles.
// lowp: 0 the FP64 apply; 1 (BF16) or 2 (FP16): the CG's direction vector
// rounded to that type for the operator apply, computed in FP32 (orders 4 to
// 8, no SVV term); dots, updates and the other vectors stay FP64.
cudaError_t launch_cg(const CgBatch& batch, int grid, int N, bool resident, cudaStream_t s,
                      int lowp = 0);

// CG with the whole iteration state on the chip (cg_patch.cu): a solve cut
// into gx x gy patches of elements, one block each.
struct PatchPkt {  // a value and its sequence number, stored and read as one 16-byte word
  double v;
  unsigned long long seq;
};
struct PatchSolve {
  Dir d[2];
  int G0;             // unknowns per row
  int n;              // unknowns
  double alpha, bx, by;
  const double* b;
  double* x;
  double rtol, atol, dtol;
  int max_it, norm_type, remove_null;
  int gx, gy, cta0;   // patches, first block of this solve
  int edge_stride;    // packets of one patch edge, whole lines
  int pad;
  PatchPkt* slots;    // sum packets: 3 arrays of one line per patch (128-byte aligned)
  PatchPkt* edges;    // 4 edge_stride gx gy edge packets
  unsigned long long seq0;  // first sequence number: above any used on these packets before,
                            // with room for the reductions of max_it iterations
};
struct PatchResult {
  double dp, rnorm0, beta;
  int its, reason;
  unsigned long long err;  // seq0 of the launch whose wait gave up
};
struct PatchPlan {
  int gx, gy, edge_stride;
  bool in_registers;  // every block's nodes fit the kernel form with all state in registers
  int cluster;        // the blocks are one thread-block cluster
  size_t smem;
  double cost;  // modelled cycles of an iteration's work
};
struct PatchLaunch {
  int N, blocks;
  bool in_registers, cluster;
  size_t smem;
  const PatchSolve* one;     // host: the solve of a single-solve launch
  const PatchSolve* solves;  // device: a batch's solves (then one is null)
  const int* cta_solve;      // device: solve of each block (batch)
  PatchResult* res;          // device, one per solve
  const double* Kh;          // host: (N+1)^2 element stiffness and N+1 weights
  const double* w;
};
constexpr int kPatchThreads = 512;
constexpr int kPatchMaxBlocks = 160;
constexpr int kPatchMaxCluster = 16;
constexpr int kPatchLine = 8;  // packets of a 128-byte line
constexpr int kPatchSmemMax = 224 * 1024;
// The cut of a solve of its own over at most max_blocks blocks, as one cluster
// where that is estimated faster; false: it does not fit on the chip (or has
// an SVV term).
bool patch_plan_single(const OpDev& op, int max_blocks, PatchPlan* out);
// The best cut for every block count 0..max_blocks (gx == 0: it does not fit).
void patch_plan_table(const OpDev& op, int max_blocks, PatchPlan* out);
// Shared memory of a plan's blocks in one of the two kernel forms.
size_t patch_smem_bytes(const OpDev& op, const PatchPlan& p, bool in_registers);
// Sum and edge packets of a plan.
inline size_t patch_packets(const PatchPlan& p) {
  return (size_t)p.gx * p.gy * (3 * kPatchLine + 4 * (size_t)p.edge_stride);
}
cudaError_t launch_cg_patch(const PatchLaunch& L, cudaStream_t s);

// Device-resident parameters and state of an FDM refinement loop.
struct FdmParams {
  double rtol, atol, dtol;
  int max_it, pad;
};
struct FdmState {
  double rnorm0, ttol, dp, best;
  int its, reason, stalled;
  unsigned kerr;  // KERR_* bits of the loop's kernels (zeroed by the loop's set-up)
};
// Set up the loop from res = {norm^2 of f, .}: rnorm0, tolerance, the
// iteration-0 test; sets the while-condition (1 = iterate).
cudaError_t launch_fdm_init(const FdmParams* p, FdmState* st, const double* res,
                            cudaGraphConditionalHandle h, cudaStream_t s);
// The prologue of an FDM solve in one launch (linsys.cu): f as
// launch_rhs_assemble, r = f, x = 0, res = {norm^2 of f (weights w, natural
// or not), |f|^2} and the loop's set-up as launch_fdm_init. partial holds at
// least 2 * npart doubles; count is zero on entry and on return.
cudaError_t launch_fdm_prologue(const OpDev& op, const MeshDev& m, const double* rhs_vals,
                                const double* lift, double* f, double* r, double* x,
                                const double* w, int natural, double* partial, int npart,
                                double* res, unsigned* count, const FdmParams* p, FdmState* st,
                                cudaGraphConditionalHandle h, cudaStream_t s);
// After a refinement step: iteration count, the residual tests (RTOL, ATOL,
// DTOL, NANORINF, ITS, and stagnation at the rounding floor) and the
// while-condition.
cudaError_t launch_fdm_check(const FdmParams* p, FdmState* st, const double* res,
                             cudaGraphConditionalHandle h, cudaStream_t s);

// FDM products on the tcgen05 tensor cores (tc_gemm.cu): D (M x N) = A B with
// A = (a_hi + a_lo) stored [M][K] (pitch a_pitch) and B stored transposed as
// (b_hi + b_lo) [N][K] (pitch b_pitch), FP32 pairs whose hi parts are TF32
// numbers; three kind::tf32 MMAs per K step (Ah Bh + Ah Bl + Al Bh). Element
// (m, n) of D goes to [n * pitch + m]: kind TC_EPI_SPLIT stores the hi/lo
// split of D, TC_EPI_DIVIDE that of D / (alpha + bm lm[m] + bn ln[n]) (0 where
// the divisor is at most null_tol in magnitude), TC_EPI_ACC64 adds D to an
// FP64 array. Pitches are multiples of 4; bases 16-byte aligned; err must be
// set (KERR_BARRIER_TIMEOUT when a bounded wait gave up).
enum { TC_EPI_SPLIT = 0, TC_EPI_DIVIDE = 1, TC_EPI_ACC64 = 2 };
struct TcEpi {
  int M, N, K;
  float *out_hi, *out_lo;  // SPLIT / DIVIDE: the next product's operand pair
  int pitch;
  double* out64;           // ACC64
  const double *lm, *ln;   // DIVIDE
  double alpha, bm, bn, null_tol;
  unsigned* err;
};
// A product planned once per buffer set (tile shape, tensor maps), launched
// as often as needed.
struct TcPlan {
  CUtensorMap maps[4];
  TcEpi e;
  int epi, bn, ck;
};
cudaError_t tc_plan(TcPlan* p, int epi, const float* a_hi, const float* a_lo, int a_pitch,
                    const float* b_hi, const float* b_lo, int b_pitch, const TcEpi& e);
cudaError_t launch_tc_plan(const TcPlan& p, cudaStream_t s);
// hi/lo split of an FP64 [rows][cols] array (leading dimension ld) into FP32
// arrays of the given pitch: hi = x rounded to TF32, lo = x - hi in FP32.
cudaError_t launch_tc_split(const double* x, int rows, int cols, int ld, float* hi, float* lo,
                            int pitch, cudaStream_t s);

// One periodic direction of nel = 2^logn equal elements of order p in Bloch
// form (bloch.cu): V [nel][p][p] complex, row i column k, the W-orthonormal
// eigenvectors of wavenumber m; mu [nel][p] their eigenvalues; tw [nel/2]
// the FFT twiddles exp(-2 pi i j / nel).
struct BlochDir {
  int nel, p, logn;
  const double2* V;
  const double* mu;
  const double2* tw;
};
// x (= or +=) A^{-1} in for a doubly periodic system by Bloch waves (three
// launches); xh: bloch_spectrum_elems complex work. Shared memory limits:
// 16 p nel bytes (x direction) and 32 p nel bytes (y) each at most 48 KB.
// gate (nullable): a refinement loop's state; when its reason is set on
// the device, in is read as zero (the step adds nothing).
cudaError_t launch_bloch_inverse(const BlochDir& bx, const BlochDir& by, double alpha, double cx,
                                 double cy, double null_tol, const double* in, double* out,
                                 bool accumulate, double2* xh, const FdmState* gate,
                                 cudaStream_t s);
size_t bloch_spectrum_elems(const BlochDir& bx, const BlochDir& by);

// A direction of the FP64 dense inverse. Where the direction is its own mirror
// image (periodic, or two ends of the same kind) every eigenvector is even or
// odd about the reflection i -> n-1-i (periodic: n-i mod n): `on`. A folded
// vector holds the ge sums over mirrored pairs (and the fixed points) in slots
// [0, ge), then the go differences in [os, os + go); the eigenvector matrix
// becomes an even block of ge modes and an odd one of go, half the
// multiplications. os and len (the folded length) are even, so that rows of
// folded arrays and of the blocks start on 16-byte boundaries.
struct FoldDir {
  int n, ge, go, os, len, on, periodic;
};
// A direction's square factor in an FP64 product: the even block (ge x ge,
// pitch os) and after it the odd block (go x go, pitch len - os).
enum { FDM_FACTOR_B = 1, FDM_FACTOR_A = 2 };
// The low modes of a direction that the FP64 inverse carries apart from the
// backward products: slots [0, even) and [split, split + odd).
constexpr int kFdmLow = 8;
struct FdmLowMap {
  int even, odd, split;
};
// C = A B on folded arrays ([y.len][x.len]) in FP64, one operand the factor of
// a direction (`which`: B that of x, or A that of y); with lx the spectral
// divide by alpha + bx lx[col] + by ly[row] (|divisor| <= null_tol gives 0)
// and, with zlow, the low modes moved into zlow[8][8] (0 left in C). Where no
// direction is folded the first product can read the caller's array (lda, any
// alignment) and the last write it (ldc): with low_y, C (= or +=, accumulate)
// gets A B + sum_ab low_y[row][a] zlow[a][b] low_x[col][b], the low modes'
// eigenvectors ([n][8]), in double-double, rounded once; zeros (or nothing
// added) when gate && *gate != 0.
struct FdmProduct {
  const double *A, *B;
  double* C;
  FoldDir x, y;
  int which, lda, ldc;
  const int* gate;
  const double *lx, *ly;
  double alpha, bx, by, null_tol;
  double* zlow;
  FdmLowMap low_r, low_c;
  const double *low_x, *low_y;
  int accumulate;
};
cudaError_t launch_fdm_dgemm(const FdmProduct& p, cudaStream_t s);
// out ([dy.len][dx.len]) = in ([dy.n][dx.n]) folded along both directions (a
// direction that is not `on` stays as it is); zeros when *gate != 0 (fdm.cu).
cudaError_t launch_fdm_fold(const FoldDir& dx, const FoldDir& dy, const double* in, double* out,
                            const int* gate, cudaStream_t s);
// out (= or +=) the unfolded `in` plus the low modes: sum_ab ly[row][a]
// zlow[a][b] lx[col][b], ly and lx the low modes' eigenvectors ([n][8]), the
// sums in double-double, rounded once.
cudaError_t launch_fdm_unfold(const FoldDir& dx, const FoldDir& dy, const double* in, double* out,
                              bool accumulate, const double* zlow, const double* lx,
                              const double* ly, cudaStream_t s);
// C = A B (row-major, leading dimensions lda/ldb/ldc) on the tensor cores
// (gemm.cu). prec: 1 TF32 on FP32 data, 2 BF16. epi: 0 store,
// 1 store after the spectral divide by alpha + bx lx[col] + by ly[row]
// (|divisor| <= null_tol gives 0), 2 accumulate into FP64 C scaled by *cmax
// (cmax == nullptr: 1). a_fp64: A is FP64 (scaled by 1/*amax when amax is
// given); c_fp64: C is FP64 (required for epi 2).
cudaError_t launch_fdm_gemm(int prec, int epi, const void* A, int a_fp64, const void* B, void* C,
                            int c_fp64, int M, int N, int K, int lda, int ldb, int ldc,
                            const double* amax, const double* cmax, const double* lx,
                            const double* ly, double alpha, double bx, double by, double null_tol,
                            cudaStream_t s);

// Fast-diagonalization pieces (fdm.cu). prec: 0 FP64, 1 FP32, 2 BF16.
cudaError_t launch_spectral_divide(int prec, void* v, int gx, int gy, const double* lx,
                                   const double* ly, double alpha, double bx, double by,
                                   double null_tol, cudaStream_t s);
// y = x / max (max read from device memory; 0 leaves y = 0).
cudaError_t launch_to_low(int prec, const double* x, void* y, size_t n, const double* max,
                          cudaStream_t s);
// x += y * max.
cudaError_t launch_add_low(int prec, double* x, const void* y, size_t n, const double* max,
                           cudaStream_t s);
// out2 = {sum (w r)^2 or, natural != 0, sum r w r; sum r^2} (w == nullptr:
// w = 1), deterministic.
cudaError_t launch_norms(const double* r, const double* w, size_t n, int natural, double* partial,
                         int npart, double* out2, cudaStream_t s);
// Sum np pairs of partials into out2 (deterministic order).
cudaError_t launch_norm_final(const double* partial, int np, double* out2, cudaStream_t s);
cudaError_t launch_maxabs(const double* x, size_t n, double* partial, int npart, double* out,
                          cudaStream_t s);
cudaError_t launch_sub(const double* b, const double* y, double* r, size_t n, cudaStream_t s);
cudaError_t launch_invert(double* x, size_t n, cudaStream_t s);
// C = A^T (Bh + Bl) in double-double for n x n row-major matrices, returned
// as Ch + Cl (Bl may be null); set-up only.
cudaError_t launch_dd_gemm_tn(int n, const double* A, const double* Bh, const double* Bl,
                              double* Ch, double* Cl, cudaStream_t s);
// y = a y + b x (a == 0: y = b x, y not read)
cudaError_t launch_axpby(double* y, double a, double b, const double* x, size_t n,
                         cudaStream_t s);
// f -= (sum f / sum d) d with d = 1 / dinv: the right-hand side that Jacobi
// CG with the constant null space projected out of every preconditioned
// residual converges to (its limit solves A x = f - c d, c = sum f / sum d).
cudaError_t launch_project_null(double* f, const double* dinv, size_t n, double* partial,
                                int npart, double* sum2, cudaStream_t s);
cudaError_t launch_remove_mean(double* x, size_t n, double* partial, int npart, double* sum2,
                               cudaStream_t s);

}  // namespace seg
