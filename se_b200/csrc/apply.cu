// Matrix-free operator apply y = A x of SE's assembled Helmholtz/Poisson
// operator on the unknown grid, element-factored, sm_100a.
//
// A = alpha (W_y x W_x) + beta_x (W_y x K_x) + beta_y (K_y x W_x), with K the
// assembled 1-D stiffness and W the assembled 1-D GLL weights (linsys.cu).
// Along one grid row the assembled K_x is the element matrix Kh (order N,
// (N+1) x (N+1)) applied to every element's N+1 nodes, the two contributions
// at a node shared by neighbouring elements summed. A block of 256 threads
// owns a tile of EX x 4 elements (EX = 64 / N) and
//   1. stages x over the tile plus N vertices to the left and below and one
//      to the right and above, as the arithmetic type in shared memory;
//   2. rows: the item (row, element) reads the 2N+1 values of its element and
//      of the one to the left and writes wy beta_x (K_x u) of the element's
//      first N nodes;
//   3. columns: the item (column, element) does the same along y, adds the
//      mass term and the row part, and writes y for its N nodes.
// The stiffness products run by even/odd halves (kh.cuh) with coefficients in
// the kernel parameters, the beta factors folded in.
//
// Almost every tile of a large mesh is interior: all staged vertices are
// unknowns, nothing wraps, every element and its left and lower neighbours
// exist. Its path has no conditions: a staged row is one contiguous run of the
// unknown array (one address a row, copies at fixed offsets from it) and the
// weights are the element's own. The others take the general path (a
// neighbour element that does not exist contributes nothing, by a flag and not
// by the zero fill, because its own node carries a value), each direction's
// conditions apart: in a mesh not much wider than a tile, where no tile is
// interior, most have none along y. All compute the same sums in the same
// order, every output by one thread: the result does not depend on scheduling.
//
// Types: FP64 (x, arithmetic, y), staged by 8-byte cp.async; the reduced-
// precision apply (x in BF16 or FP16, operator and arithmetic in FP32, y in
// FP32), staged through registers, four values a load where every row starts
// on an 8-byte boundary.
//
// What bounds it: HBM, with instruction issue close behind. Measured, FP64: 37.7M
// unknowns, p = 8, 121 us (4990 GB/s, 0.76 of the measured copy rate; 159 us
// with every tile on the general path and full products); 3.06M unknowns,
// p = 10, 17.3 us (56 us on the FP64 tensor cores, whose 8-wide steps pad
// 11-wide elements, with a host wait for its bounded TMA waits); p = 3, 12 and
// 11: 31, 28 and 25 us against 92, 104 and 138. BF16, 37.7M unknowns, p = 8:
// 78 us against 117. Without interior tiles: 7 x 50,000 elements, p = 5,
// between walls 47 us (70 with both directions' conditions in every tile),
// BF16 43 (66).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cstdint>
#include <cstring>

#include "common.cuh"
#include "fdm_ctl.cuh"
#include "kh.cuh"

namespace seg {
namespace {

__device__ __forceinline__ float to_a(__nv_bfloat16 v, float) { return __bfloat162float(v); }
__device__ __forceinline__ float to_a(__half v, float) { return __half2float(v); }

// Unknown index of vertex g along d (-1: Dirichlet or outside), one wrap for
// periodic directions.
__device__ __forceinline__ int unk(const Dir& d, int g) {
  if (d.periodic) {
    const int L = d.nV - 1;
    if (g < 0)
      g += L;
    else if (g >= L)
      g -= L;
  } else if (g < 0 || g >= d.nV) {
    return -1;
  }
  return (g >= d.lo && g < d.hi) ? g - d.lo : -1;
}

// Assembled 1-D weight of vertex (element e, node a).
template <int N, class A>
__device__ __forceinline__ A wsum(const Dir& d, const A* w, int e, int a) {
  A s = A(0);
  if (e < d.nE) s += w[a];
  if (a == 0 && (e > 0 || d.periodic)) s += w[N];
  return s;
}

// Tile of an order: EX elements (TX vertices) by four element rows, at most
// one row item and one column item a thread; odd pitches keep a warp's
// column-wise shared-memory reads free of conflicts.
template <int N>
struct EfTile {
  static constexpr int EX = 64 / N;      // elements per tile row
  static constexpr int TX = EX * N;      // output vertices per tile row
  static constexpr int SW = TX + N + 1;  // staged vertices per row
  static constexpr int W = SW | 1;       // staged row pitch (odd)
  static constexpr int OXP = (TX + 1) | 1;  // x-pass output pitch (odd)
  static constexpr int TY = 4 * N;       // output rows per tile
  static constexpr int ITEMS = EX * TY;  // x-pass (= y-pass) items, one per thread
  static_assert(ITEMS <= 256 && TX * (TY / N) == ITEMS && TY % N == 0, "tile shape");
  static_assert(SW > 64 && SW <= 96, "staging columns");
};
constexpr int kEfThreads = 256, kEfWarps = kEfThreads / 32;

// The apply's tile: R times four element rows, up to R items a thread and pass.
template <int N, int R>
struct ElTile : EfTile<N> {
  static constexpr int TY = 4 * N * R;
  static constexpr int H = TY + N + 1;
  static constexpr int ITEMS = EfTile<N>::EX * TY;
};

// Whether the staged range of a tile along d lies inside the unknowns and all
// elements it touches exist.
__device__ __forceinline__ bool inside(const Dir& d, int first, int last) {
  return first >= d.lo && last < d.hi && (d.periodic || last < d.nV);
}

// Whether all outputs [first, first + n) of a tile along d are unknowns whose
// elements and left (lower) neighbours exist.
__device__ __forceinline__ bool all_outputs(const Dir& d, int first, int n) {
  return first >= d.lo && first + n <= d.hi && (d.periodic || first > 0);
}

// Stage the tile's vertices and its N-vertex halo to the left and below into
// X (zero where a vertex is no unknown): warp w takes rows w, w + 8, ...;
// lane l columns l, l + 32, l + 64; all copies issued before the wait.
template <int N, int H>
__device__ __forceinline__ void ef_stage(const Dir& dx, const Dir& dy, int G0,
                                         const double* __restrict__ x, double* X, int gx0,
                                         int gy0) {
  typedef EfTile<N> T;
  constexpr int SW = T::SW, W = T::W;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int cu[3];
#pragma unroll
  for (int q = 0; q < 3; q++) {
    const int i = lane + 32 * q;
    cu[q] = i < SW ? unk(dx, gx0 - N + i) : -1;
  }
#pragma unroll
  for (int r = 0; r < (H + kEfWarps - 1) / kEfWarps; r++) {
    const int j = warp + kEfWarps * r;
    if (j < H) {
      const int uy = unk(dy, gy0 - N + j);
      const double* rowp = x + (size_t)(uy < 0 ? 0 : uy) * G0;
#pragma unroll
      for (int q = 0; q < 3; q++) {
        const int i = lane + 32 * q;
        if (i < SW) {
          const bool ok = uy >= 0 && cu[q] >= 0;
          const double* src = ok ? rowp + cu[q] : x;
          const unsigned dst = (unsigned)__cvta_generic_to_shared(X + j * W + i);
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(dst), "l"(src),
                       "r"(ok ? 8 : 0));
        }
      }
    }
  }
  asm volatile("cp.async.commit_group;\n" ::);
  asm volatile("cp.async.wait_group 0;\n" ::);
}

// Everything the apply needs, by value (the kernel parameter bank).
template <int N, class A>
struct ElArgs {
  Dir dx, dy;
  int G0, G1;
  A cx[Eo<N>::NC], cy[Eo<N>::NC];  // beta_x Kh, beta_y Kh by even/odd halves
  A lx[N + 1], ly[N + 1];          // their last rows: the left / lower element's part
  A w[N + 1], alpha;
};

// Interior staging, FP64: one address a row, three copies at fixed offsets.
template <int N, int R>
__device__ __forceinline__ void stage_interior(const ElArgs<N, double>& op, const double* x,
                                               double* X, int gx0, int gy0, int) {
  typedef ElTile<N, R> T;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double* src = x + (size_t)(gy0 - N - op.dy.lo + warp) * op.G0 + (gx0 - N - op.dx.lo + lane);
  unsigned dst = (unsigned)__cvta_generic_to_shared(X + warp * T::W + lane);
  const size_t step = (size_t)kEfWarps * op.G0;
#pragma unroll
  for (int r = 0; r < (T::H + kEfWarps - 1) / kEfWarps; r++) {
    if (r < T::H / kEfWarps || warp + r * kEfWarps < T::H) {
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst), "l"(src));
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst + 256), "l"(src + 32));
      if (lane < T::SW - 64)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst + 512), "l"(src + 64));
    }
    src += step;
    dst += kEfWarps * T::W * 8;
  }
  asm volatile("cp.async.commit_group;\n" ::);
  asm volatile("cp.async.wait_group 0;\n" ::);
}

// Four 16-bit values of a load as FP32.
__device__ __forceinline__ void unpack4(uint2 q, float (&f)[4], __nv_bfloat16) {
  f[0] = __uint_as_float(q.x << 16);
  f[1] = __uint_as_float(q.x & 0xffff0000u);
  f[2] = __uint_as_float(q.y << 16);
  f[3] = __uint_as_float(q.y & 0xffff0000u);
}
__device__ __forceinline__ void unpack4(uint2 q, float (&f)[4], __half) {
  const __half2 a = *reinterpret_cast<const __half2*>(&q.x), b = *reinterpret_cast<const __half2*>(&q.y);
  const float2 u = __half22float2(a), v = __half22float2(b);
  f[0] = u.x;
  f[1] = u.y;
  f[2] = v.x;
  f[3] = v.y;
}

// Interior staging, 16-bit x: quads != 0 when every row starts on an 8-byte
// boundary at the same offset (rows a multiple of four unknowns long, x
// aligned): loads of four values from the boundary at or before the row's
// first vertex, quads - 1 values further left. The staged row then starts
// quads - 1 floats into its pitch.
template <int N, int R, class TI>
__device__ __forceinline__ void stage_interior(const ElArgs<N, float>& op, const TI* x, float* X,
                                               int gx0, int gy0, int quads) {
  typedef ElTile<N, R> T;
  constexpr int W = (T::SW + 3) | 1;
  const size_t q0 = (size_t)(gy0 - N - op.dy.lo) * op.G0 + (gx0 - N - op.dx.lo);
  if (quads) {
    constexpr int NQ = (T::SW + 3 + 3) / 4;  // loads that cover a row at any offset
    // a thread loads one column of quads, RP rows apart
    constexpr int RP = kEfThreads / NQ, S = (T::H + RP - 1) / RP;
    const int j0 = threadIdx.x / NQ, i = threadIdx.x - j0 * NQ;
    if (j0 >= RP) return;
    const uint2* src = reinterpret_cast<const uint2*>(x + (q0 - (quads - 1))) +
                       (size_t)j0 * (op.G0 / 4) + i;
    const size_t step = (size_t)RP * (op.G0 / 4);
    uint2 v[S];
#pragma unroll
    for (int s = 0; s < S; s++) {
      if (j0 + s * RP < T::H) v[s] = __ldg(src);
      src += step;
    }
    float* dst = X + j0 * W + 4 * i;
#pragma unroll
    for (int s = 0; s < S; s++) {
      if (j0 + s * RP < T::H) {
        float f[4];
        unpack4(v[s], f, TI());
#pragma unroll
        for (int q = 0; q < 4; q++)
          if (4 * i + q < W) dst[q] = f[q];
      }
      dst += RP * W;
    }
    return;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const TI* src = x + q0 + (size_t)warp * op.G0 + lane;
  float* dst = X + warp * W + lane;
  const size_t step = (size_t)kEfWarps * op.G0;
  constexpr int Q = (T::H + kEfWarps - 1) / kEfWarps;
  TI v[Q][3];
#pragma unroll
  for (int r = 0; r < Q; r++) {
    if (warp + r * kEfWarps < T::H) {
      v[r][0] = src[0];
      v[r][1] = src[32];
      if (lane < T::SW - 64) v[r][2] = src[64];
    }
    src += step;
  }
#pragma unroll
  for (int r = 0; r < Q; r++) {
    if (warp + r * kEfWarps < T::H) {
      dst[0] = to_a(v[r][0], 0.f);
      dst[32] = to_a(v[r][1], 0.f);
      if (lane < T::SW - 64) dst[64] = to_a(v[r][2], 0.f);
    }
    dst += kEfWarps * W;
  }
}

// General staging: every vertex mapped, zero where there is no unknown (the
// loads of a 16-bit tile issued before any is used). YIN: the staged rows are
// consecutive rows of unknowns, only the columns need mapping (a mesh not
// much wider than a tile consists of such tiles).
template <int N, int R, bool YIN>
__device__ __forceinline__ void stage_general(const ElArgs<N, double>& op, const double* x,
                                              double* X, int gx0, int gy0) {
  typedef ElTile<N, R> T;
  if constexpr (!YIN) {
    ef_stage<N, T::H>(op.dx, op.dy, op.G0, x, X, gx0, gy0);
  } else {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double* src[3];
    int bytes[3];
    const double* row0 = x + (size_t)(gy0 - N - op.dy.lo + warp) * op.G0;
#pragma unroll
    for (int q = 0; q < 3; q++) {
      const int cu = lane + 32 * q < T::SW ? unk(op.dx, gx0 - N + lane + 32 * q) : -1;
      src[q] = row0 + max(cu, 0);
      bytes[q] = cu >= 0 ? 8 : 0;
    }
    unsigned dst = (unsigned)__cvta_generic_to_shared(X + warp * T::W + lane);
    const size_t step = (size_t)kEfWarps * op.G0;
#pragma unroll
    for (int r = 0; r < (T::H + kEfWarps - 1) / kEfWarps; r++) {
      if (r < T::H / kEfWarps || warp + r * kEfWarps < T::H) {
#pragma unroll
        for (int q = 0; q < 3; q++) {
          if (lane + 32 * q < T::SW)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(dst + 256 * q),
                         "l"(src[q]), "r"(bytes[q]));
          src[q] += step;
        }
      }
      dst += kEfWarps * T::W * 8;
    }
    asm volatile("cp.async.commit_group;\n" ::);
    asm volatile("cp.async.wait_group 0;\n" ::);
  }
}
template <int N, int R, bool YIN, class TI>
__device__ __forceinline__ void stage_general(const ElArgs<N, float>& op, const TI* x, float* X,
                                              int gx0, int gy0) {
  typedef ElTile<N, R> T;
  constexpr int W = (T::SW + 3) | 1, Q = (T::H + kEfWarps - 1) / kEfWarps;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int cu[3];
#pragma unroll
  for (int q = 0; q < 3; q++)
    cu[q] = lane + 32 * q < T::SW ? unk(op.dx, gx0 - N + lane + 32 * q) : -1;
  const TI* row = x + (YIN ? (size_t)(gy0 - N - op.dy.lo + warp) * op.G0 : 0);
  const size_t step = (size_t)kEfWarps * op.G0;
  TI v[Q][3];
#pragma unroll
  for (int r = 0; r < Q; r++) {
    const int j = warp + r * kEfWarps;
    bool in = j < T::H;
    if constexpr (!YIN) {
      const int uy = in ? unk(op.dy, gy0 - N + j) : -1;
      in = uy >= 0;
      row = x + (size_t)(in ? uy : 0) * op.G0;
    }
#pragma unroll
    for (int q = 0; q < 3; q++) v[r][q] = in && cu[q] >= 0 ? row[cu[q]] : TI(0.f);
    if constexpr (YIN) row += step;
  }
  float* dst = X + warp * W + lane;
#pragma unroll
  for (int r = 0; r < Q; r++) {
    if (warp + r * kEfWarps < T::H) {
#pragma unroll
      for (int q = 0; q < 3; q++)
        if (lane + 32 * q < T::SW) dst[32 * q] = to_a(v[r][q], 0.f);
    }
    dst += kEfWarps * W;
  }
}

// Row and column passes on the staged tile (row j, column i at X[j * W + i]).
// XIN, YIN: along x, y every output is an unknown and every element and its
// left (lower) neighbour exists.
template <int N, int R, class A, class TO, int W, bool XIN, bool YIN>
__device__ __forceinline__ void el_passes(const ElArgs<N, A>& op, const A* X, A* OX, const A* sw,
                                          int gx0, int gy0, TO* __restrict__ y) {
  typedef ElTile<N, R> T;
  constexpr int OXP = T::OXP, TX = T::TX, TY = T::TY;
  const int tid = threadIdx.x;
#pragma unroll
  for (int q = 0; q < R; q++) {  // item = (element e, row r)
    const int it = tid + q * kEfThreads, r = it % TY, e = it / TY;
    // an item past the mesh's end has no output
    if (it >= T::ITEMS || (!XIN && gx0 + e * N >= op.dx.hi) || (!YIN && gy0 + r >= op.dy.hi)) continue;
    const A* row = X + (r + N) * W + e * N;  // left element's first node
    A l[N], v[N + 1], o[N + 1];
#pragma unroll
    for (int k = 0; k < N; k++) l[k] = row[k];
#pragma unroll
    for (int k = 0; k <= N; k++) v[k] = row[N + k];
    eo_product<N, false>(op.cx, v, o);
    A t = op.lx[N] * v[0];
#pragma unroll
    for (int k = 0; k < N; k++) t = fma(op.lx[k], l[k], t);
    A wy;
    if constexpr (XIN) {
      o[0] += t;
    } else {
      const int ex = gx0 / N + e;
      const bool own = ex < op.dx.nE, left = ex > 0 || op.dx.periodic;
      if (!own) {
#pragma unroll
        for (int k = 0; k < N; k++) o[k] = A(0);
      }
      if (left && ex <= op.dx.nE) o[0] += t;
    }
    if constexpr (YIN) {
      wy = sw[r % N];
    } else {
      const int ey = gy0 / N + r / N, a = r % N;
      wy = (ey < op.dy.nE ? op.w[a] : A(0)) +
           (a == 0 && (ey > 0 || op.dy.periodic) ? op.w[N] : A(0));
    }
#pragma unroll
    for (int a = 0; a < N; a++) OX[r * OXP + e * N + a] = wy * o[a];
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < R; q++) {  // item = (element row e, column c), consecutive columns per warp
    const int it = tid + q * kEfThreads, c = it % TX, e = it / TX;
    if (it >= T::ITEMS) continue;
    if (!XIN && (gx0 + c < op.dx.lo || gx0 + c >= op.dx.hi)) continue;
    if (!YIN && gy0 + e * N >= op.dy.hi) continue;
    const A* col = X + (e * N) * W + c + N;  // lower element's first node
    A l[N], v[N + 1], o[N + 1];
#pragma unroll
    for (int k = 0; k < N; k++) l[k] = col[k * W];
#pragma unroll
    for (int k = 0; k <= N; k++) v[k] = col[(N + k) * W];
    eo_product<N, false>(op.cy, v, o);
    A t = op.ly[N] * v[0];
#pragma unroll
    for (int k = 0; k < N; k++) t = fma(op.ly[k], l[k], t);
    const A* oxp = OX + (e * N) * OXP + c;
    // y = wx (alpha wy x + beta_y (Ky x)) + wy beta_x (Kx x)
    A wx;
    if constexpr (XIN) {
      wx = sw[c % N];
    } else {
      const int gx = gx0 + c, ex = gx / N, b = gx % N;
      wx = (ex < op.dx.nE ? op.w[b] : A(0)) +
           (b == 0 && (ex > 0 || op.dx.periodic) ? op.w[N] : A(0));
    }
    if constexpr (YIN) {
      o[0] += t;
      const size_t ld = (size_t)op.G0;
      TO* yp = y + (size_t)(gy0 + e * N - op.dy.lo) * ld + (gx0 + c - op.dx.lo);
#pragma unroll
      for (int a = 0; a < N; a++) {
        const A wa = op.alpha * (a == 0 ? op.w[0] + op.w[N] : op.w[a]);
        *yp = (TO)fma(wx, fma(wa, v[a], o[a]), oxp[a * OXP]);
        yp += ld;
      }
    } else {
      const int ey = gy0 / N + e;
      const bool own = ey < op.dy.nE, low = (ey > 0 || op.dy.periodic) && ey <= op.dy.nE;
      if (!own) {
#pragma unroll
        for (int k = 0; k < N; k++) o[k] = A(0);
      }
      if (low) o[0] += t;
#pragma unroll
      for (int a = 0; a < N; a++) {
        const int gy = gy0 + e * N + a;
        A wa = (own ? op.w[a] : A(0));
        if (a == 0) wa = (own ? op.w[0] : A(0)) + (low ? op.w[N] : A(0));
        const A r = fma(wx, fma(op.alpha * wa, v[a], o[a]), oxp[a * OXP]);
        if (gy >= op.dy.lo && gy < op.dy.hi)
          y[(size_t)(gy - op.dy.lo) * op.G0 + (gx0 + c - op.dx.lo)] = (TO)r;
      }
    }
  }
}

// quads: x in 16 bits with rows a multiple of four long and an 8-byte aligned
// base. y0: the first row of vertices of this launch.
template <int N, int R, class TI, class A, class TO, int MINB>
__global__ void __launch_bounds__(kEfThreads, MINB)
    apply_el_kernel(const __grid_constant__ ElArgs<N, A> op, const TI* __restrict__ x,
                    TO* __restrict__ y, int quads, int y0) {
  typedef ElTile<N, R> T;
  constexpr bool LOW = sizeof(TI) != sizeof(A);
  constexpr int W = LOW ? (T::SW + 3) | 1 : T::W;
  extern __shared__ __align__(16) unsigned char el_smem[];
  A* X = reinterpret_cast<A*>(el_smem);  // vertices (gx0-N .. gx0+TX) x (gy0-N .. gy0+TY)
  A* OX = X + T::H * W;                  // row-pass results of the tile's vertices
  A* sw = OX + T::TY * T::OXP;           // assembled weights of an element's first N nodes
  const int gx0 = blockIdx.x * T::TX, gy0 = blockIdx.y * T::TY + y0;
  if (threadIdx.x < N)
    sw[threadIdx.x] = threadIdx.x == 0 ? op.w[0] + op.w[N] : op.w[threadIdx.x];
  bool interior = inside(op.dx, gx0 - N, gx0 + T::TX) && inside(op.dy, gy0 - N, gy0 + T::TY);
  int shift = 0;
  if (LOW && quads && interior) {
    // offset of the row's first value from the boundary before it; the loads
    // past the row's end must stay inside the array
    shift = (gx0 - N - op.dx.lo) & 3;
    const size_t last = (size_t)(gy0 + T::TY - op.dy.lo) * op.G0 + (gx0 - N - op.dx.lo - shift);
    if (last + (T::SW + 6) / 4 * 4 > (size_t)op.G0 * op.G1) interior = false;
  }
  if (interior) {
    stage_interior<N, R>(op, x, X, gx0, gy0, LOW && quads ? shift + 1 : 0);
  } else {
    shift = 0;
    if (inside(op.dy, gy0 - N, gy0 + T::TY))
      stage_general<N, R, true>(op, x, X, gx0, gy0);
    else
      stage_general<N, R, false>(op, x, X, gx0, gy0);
  }
  __syncthreads();
  // (a tile at a periodic seam has general staging and plain passes)
  const bool xin = all_outputs(op.dx, gx0, T::TX), yin = all_outputs(op.dy, gy0, T::TY);
  if (xin && yin)
    el_passes<N, R, A, TO, W, true, true>(op, X + shift, OX, sw, gx0, gy0, y);
  else if (yin)
    el_passes<N, R, A, TO, W, false, true>(op, X, OX, sw, gx0, gy0, y);
  else
    el_passes<N, R, A, TO, W, false, false>(op, X, OX, sw, gx0, gy0, y);
}

template <int N, int R, class TI, class A, class TO>
cudaError_t launch_tile(const OpDev& od, const TI* x, TO* y, cudaStream_t s) {
  typedef ElTile<N, R> T;
  constexpr bool LOW = sizeof(TI) != sizeof(A);
  constexpr int W = LOW ? (T::SW + 3) | 1 : T::W;
  // blocks per SM: the most without spills and with no kernel slower (bf16,
  // p = 8: 5 blocks 84 us, 8 blocks 78; FP64, p = 4: 5 blocks 64, 6 blocks 62)
  constexpr int MINB = LOW ? (N >= 9 ? 5 : 8) : N >= 11 ? 3 : N >= 7 ? 4 : 6;
  ElArgs<N, A> op;
  op.dx = od.d[0];
  op.dy = od.d[1];
  op.G0 = od.G[0];
  op.G1 = od.G[1];
  eo_coefs<N>(od.Kh, od.beta[0], op.cx);
  eo_coefs<N>(od.Kh, od.beta[1], op.cy);
  for (int k = 0; k <= N; k++) {
    op.lx[k] = (A)(od.beta[0] * od.Kh[N * (N + 1) + k]);
    op.ly[k] = (A)(od.beta[1] * od.Kh[N * (N + 1) + k]);
    op.w[k] = (A)od.w[k];
  }
  op.alpha = (A)od.alpha;
  constexpr size_t smem = sizeof(A) * ((size_t)T::H * W + (size_t)T::TY * T::OXP + N);
  if (smem > 48 * 1024) {
    static bool attr[64] = {};  // per instantiation and device
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!attr[dev]) {
      e = cudaFuncSetAttribute(apply_el_kernel<N, R, TI, A, TO, MINB>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
      attr[dev] = true;
    }
  }
  const int quads = LOW && od.G[0] % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 7) == 0;
  const int rows = (od.d[1].hi + T::TY - 1) / T::TY;
  for (int r = 0; r < rows; r += kGridRows) {
    const dim3 grid((od.d[0].hi + T::TX - 1) / T::TX, std::min(rows - r, kGridRows));
    apply_el_kernel<N, R, TI, A, TO, MINB><<<grid, kEfThreads, smem, s>>>(op, x, y, quads, r * T::TY);
  }
  return cudaGetLastError();
}

template <int N, class TI, class A, class TO>
cudaError_t launch_el(const OpDev& od, const TI* x, TO* y, cudaStream_t s) {
  // Four times the rows a tile where that leaves a wave of blocks: a 16-bit
  // tile of a low order has little work beside its fixed costs. Order 2 at
  // 2000 x 2000 elements 40 us against 60; order 4 in a mesh of one tile's
  // width, 5 x 30,000 elements, 14.4 us against 20.5.
  if constexpr (sizeof(TI) != sizeof(A) && N <= 4) {
    typedef ElTile<N, 1> T;
    const long tx = (od.d[0].hi + T::TX - 1) / T::TX, ty = (od.d[1].hi + T::TY - 1) / T::TY;
    if ((N == 2 || tx == 1) && tx * ty > 8 * kSms) return launch_tile<N, 4, TI, A, TO>(od, x, y, s);
  }
  return launch_tile<N, 1, TI, A, TO>(od, x, y, s);
}

// ------------------------------- refinement residual, orders 4 to 8 ----
// r = b - A x on the apply's tile with TY / kResSplit output rows: the
// stiffness sums of both passes, the combination and the subtraction in
// double-double (the stiffness rows sum to zero, so the taps cancel and a
// plain FP64 sum loses the digits a 1e-10 residual needs), rounded once.
// Each element row (x pass) and column (y pass) is shared by kResSplit
// thread groups, warp-uniform, each forming a contiguous share of its N
// outputs in the same order as one thread would: twice the blocks of half
// the depth for this latency-bound kernel, and the same bits. Per-block
// partial sums of (w r)^2 (or r w r when natural) and r^2; the block that
// finishes last sums the partials in block order and runs the FDM loop's
// convergence test (ResTail). Optionally also writes r's TF32 hi/lo split
// for the tensor-core inverse.
constexpr int kResSplit = 2;
template <int N>
struct ResTile {
  typedef EfTile<N> E;
  static constexpr int EX = E::EX, TX = E::TX, W = E::W, OXP = E::OXP;
  static constexpr int TY = E::TY / kResSplit;   // output rows: 16, 14, 12, 10, 8
  static constexpr int H = TY + N + 1;           // staged rows
  static constexpr int ITEMS = EX * TY;          // rows (x pass) = columns (y pass)
  static constexpr int GROUP = kEfThreads / kResSplit;  // threads of one share
  static constexpr int CH = (N + kResSplit - 1) / kResSplit;  // outputs of a share
  static_assert(TY % N == 0 && ITEMS <= GROUP && GROUP % 32 == 0, "residual tile shape");
};

// x pass of outputs [A0, A1) of one element row: v = the row's 2N+1 staged
// values (left element, shared node, own element).
template <int N, int A0, int A1>
__device__ __forceinline__ void res_xpass(const OpDev& op, const double* row, bool own, bool left,
                                          double* OXH, double* OXL) {
  constexpr int n = N + 1;
  double v[2 * N + 1];
#pragma unroll
  for (int k = (A0 == 0 ? 0 : N); k <= 2 * N; k++) v[k] = row[k];
#pragma unroll
  for (int a = A0; a < A1; a++) {
    double hi = 0.0, lo = 0.0;
    if (own) {
#pragma unroll
      for (int q = 0; q < n; q++) dd_fma(hi, lo, op.Kh[a * n + q], v[N + q]);
    }
    if (A0 == 0 && a == 0 && left) {
      double h2 = 0.0, l2 = 0.0;
#pragma unroll
      for (int q = 0; q < n; q++) dd_fma(h2, l2, op.Kh[N * n + q], v[q]);
      dd_add(hi, lo, h2);
      lo += l2;
    }
    OXH[a] = hi;
    OXL[a] = lo;
  }
}

// y pass, combination and residual of outputs [A0, A1) of one element
// column; accumulates the norm partials.
template <int N, int A0, int A1>
__device__ __forceinline__ void res_ypass(const OpDev& op, const double* col, const double* OXH,
                                          const double* OXL, const double* sw, int c, int e,
                                          int gx, int gy0, bool own, bool left,
                                          const double* __restrict__ b, double* __restrict__ rout,
                                          const double* __restrict__ wv, int natural,
                                          double& acc0, double& acc1, float* __restrict__ sp_hi,
                                          float* __restrict__ sp_lo, int sp_pitch) {
  typedef ResTile<N> T;
  constexpr int n = N + 1, W = T::W, OXP = T::OXP;
  const Dir& dx = op.d[0];
  const Dir& dy = op.d[1];
  double v[2 * N + 1];
#pragma unroll
  for (int k = (A0 == 0 ? 0 : N); k <= 2 * N; k++) v[k] = col[k * W];
  double yh[A1 - A0], yl[A1 - A0];
#pragma unroll
  for (int a = A0; a < A1; a++) {
    double hi = 0.0, lo = 0.0;
    if (own) {
#pragma unroll
      for (int q = 0; q < n; q++) dd_fma(hi, lo, op.Kh[a * n + q], v[N + q]);
    }
    if (A0 == 0 && a == 0 && left) {
      double h2 = 0.0, l2 = 0.0;
#pragma unroll
      for (int q = 0; q < n; q++) dd_fma(h2, l2, op.Kh[N * n + q], v[q]);
      dd_add(hi, lo, h2);
      lo += l2;
    }
    yh[a - A0] = hi;
    yl[a - A0] = lo;
  }
  if (gx < dx.lo || gx >= dx.hi) return;
  const double wx = wsum<N>(dx, sw, gx / N, gx % N);
  const double w0 = (own ? op.w[0] : 0.0) + (left ? op.w[N] : 0.0);
  const int gyb = gy0 + e * N;
  const size_t ux = (size_t)(gx - dx.lo);
#pragma unroll
  for (int a = A0; a < A1; a++) {
    const int gy = gyb + a;
    if (gy < dy.lo || gy >= dy.hi) continue;
    const double wy = a == 0 ? w0 : op.w[a];
    const size_t k = (size_t)(gy - dy.lo) * op.G[0] + ux;
    const double cm = -op.alpha * wx * wy, cx = -op.beta[0] * wy, cy = -op.beta[1] * wx;
    double hi = b[k], lo = 0.0;
    dd_fma(hi, lo, cm, v[N + a]);
    dd_fma(hi, lo, cx, OXH[(e * N + a) * OXP + c]);
    lo = fma(cx, OXL[(e * N + a) * OXP + c], lo);
    dd_fma(hi, lo, cy, yh[a - A0]);
    lo = fma(cy, yl[a - A0], lo);
    const double rv = hi + lo;
    rout[k] = rv;
    const double z = wv ? rv * wv[k] : rv;
    acc0 += natural ? z * rv : z * z;
    acc1 += rv * rv;
    if (sp_hi) {
      uint32_t h;
      asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(h) : "f"((float)rv));
      const float fh = __uint_as_float(h);
      const size_t o = (size_t)(gy - dy.lo) * sp_pitch + ux;
      sp_hi[o] = fh;
      sp_lo[o] = (float)(rv - (double)fh);
    }
  }
}

template <int N>
__global__ void __launch_bounds__(kEfThreads, 2)
    residual_ef_kernel(const OpDev op, const double* __restrict__ x, const double* __restrict__ b,
                       double* __restrict__ rout, const double* __restrict__ wv, int natural,
                       double* __restrict__ partial, const ResTail tail, float* __restrict__ sp_hi,
                       float* __restrict__ sp_lo, int sp_pitch) {
  typedef ResTile<N> T;
  constexpr int W = T::W, OXP = T::OXP, TX = T::TX, TY = T::TY, H = T::H, CH = T::CH;
  extern __shared__ __align__(16) double efsm[];
  double* X = efsm;              // staged vertices
  double* OXH = X + H * W;       // x-pass stiffness sums, high parts
  double* OXL = OXH + TY * OXP;  // and low parts
  double* sw = OXL + TY * OXP;
  __shared__ double red[kEfWarps][2];
  __shared__ unsigned last;
  const Dir& dx = op.d[0];
  const Dir& dy = op.d[1];
  const int gx0 = blockIdx.x * TX, gy0 = blockIdx.y * TY;
  const int tid = threadIdx.x;
  // share of the outputs (warp-uniform) and item of this thread
  const int sub = tid / T::GROUP, item = tid - sub * T::GROUP;
  if (tid <= N) sw[tid] = op.w[tid];
  ef_stage<N, H>(dx, dy, op.G[0], x, X, gx0, gy0);
  __syncthreads();
  if (item < T::ITEMS) {  // x pass
    const int r = item % TY, e = item / TY;
    const int ex = gx0 / N + e;
    const double* row = X + (r + N) * W + e * N;
    const bool own = ex < dx.nE, left = ex > 0 || dx.periodic;
    double* oh = OXH + r * OXP + e * N;
    double* ol = OXL + r * OXP + e * N;
    if constexpr (kResSplit == 1)
      res_xpass<N, 0, N>(op, row, own, left, oh, ol);
    else if (sub == 0)
      res_xpass<N, 0, CH>(op, row, own, left, oh, ol);
    else
      res_xpass<N, CH, N>(op, row, own, left, oh, ol);
  }
  __syncthreads();
  double acc0 = 0.0, acc1 = 0.0;
  if (item < T::ITEMS) {  // y pass, the combination and the residual
    const int c = item % TX, e = item / TX;
    const int ey = gy0 / N + e;
    const double* col = X + (e * N) * W + c + N;
    const bool own = ey < dy.nE, left = ey > 0 || dy.periodic;
    if constexpr (kResSplit == 1)
      res_ypass<N, 0, N>(op, col, OXH, OXL, sw, c, e, gx0 + c, gy0, own, left, b, rout, wv,
                         natural, acc0, acc1, sp_hi, sp_lo, sp_pitch);
    else if (sub == 0)
      res_ypass<N, 0, CH>(op, col, OXH, OXL, sw, c, e, gx0 + c, gy0, own, left, b, rout, wv,
                          natural, acc0, acc1, sp_hi, sp_lo, sp_pitch);
    else
      res_ypass<N, CH, N>(op, col, OXH, OXL, sw, c, e, gx0 + c, gy0, own, left, b, rout, wv,
                          natural, acc0, acc1, sp_hi, sp_lo, sp_pitch);
  }
  // block sums in a fixed order
  const int lane = tid & 31, warp = tid >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    acc0 += __shfl_down_sync(0xffffffffu, acc0, o);
    acc1 += __shfl_down_sync(0xffffffffu, acc1, o);
  }
  if (lane == 0) {
    red[warp][0] = acc0;
    red[warp][1] = acc1;
  }
  __syncthreads();
  const unsigned blk = blockIdx.y * gridDim.x + blockIdx.x, nb = gridDim.x * gridDim.y;
  if (tid == 0) {
    double s0 = 0.0, s1 = 0.0;
#pragma unroll
    for (int q = 0; q < kEfWarps; q++) {
      s0 += red[q][0];
      s1 += red[q][1];
    }
    partial[2 * blk] = s0;
    partial[2 * blk + 1] = s1;
  }
  if (!tail.count) return;
  // the last block to finish sums the partials in block order and runs the
  // refinement step's convergence test (no block waits for another)
  __threadfence();
  __syncthreads();
  if (tid == 0) last = atomicAdd(tail.count, 1u) == nb - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  double s0 = 0.0, s1 = 0.0;
  for (unsigned k = tid; k < nb; k += kEfThreads) {
    s0 += __ldcg(partial + 2 * k);
    s1 += __ldcg(partial + 2 * k + 1);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s0 += __shfl_down_sync(0xffffffffu, s0, o);
    s1 += __shfl_down_sync(0xffffffffu, s1, o);
  }
  __syncthreads();
  if (lane == 0) {
    red[warp][0] = s0;
    red[warp][1] = s1;
  }
  __syncthreads();
  if (tid == 0) {
    double t0 = 0.0, t1 = 0.0;
#pragma unroll
    for (int q = 0; q < kEfWarps; q++) {
      t0 += red[q][0];
      t1 += red[q][1];
    }
    tail.res[0] = t0;
    tail.res[1] = t1;
    *tail.count = 0u;
    fdm_check_state(tail.p, tail.st, t0, tail.h);
  }
}

template <int N>
cudaError_t launch_res_ef(const OpDev& op, const double* x, const double* b, double* r,
                          const double* w, int natural, double* partial, const ResTail& tail,
                          float* sh, float* sl, int sp, cudaStream_t s) {
  typedef ResTile<N> T;
  constexpr size_t smem = sizeof(double) * ((size_t)T::H * T::W + 2 * (size_t)T::TY * T::OXP + 16);
  if (smem > 48 * 1024) {
    static bool attr[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!attr[dev]) {
      e = cudaFuncSetAttribute(residual_ef_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)smem);
      if (e != cudaSuccess) return e;
      attr[dev] = true;
    }
  }
  const dim3 grid((op.d[0].hi + T::TX - 1) / T::TX, (op.d[1].hi + T::TY - 1) / T::TY);
  residual_ef_kernel<N><<<grid, kEfThreads, smem, s>>>(op, x, b, r, w, natural, partial, tail, sh,
                                                       sl, sp);
  return cudaGetLastError();
}

}  // namespace

bool residual_ef_supported(const OpDev& op) {
  return op.gamma == 0.0 && op.d[0].N >= 4 && op.d[0].N <= 8;
}

namespace {
template <int N>
int res_ef_blocks(const OpDev& op) {
  typedef ResTile<N> T;
  return ((op.d[0].hi + T::TX - 1) / T::TX) * ((op.d[1].hi + T::TY - 1) / T::TY);
}
}  // namespace

int residual_partial_blocks(const OpDev& op) {
  if (!residual_ef_supported(op)) return residual_blocks(op);
  switch (op.d[0].N) {
    case 4: return res_ef_blocks<4>(op);
    case 5: return res_ef_blocks<5>(op);
    case 6: return res_ef_blocks<6>(op);
    case 7: return res_ef_blocks<7>(op);
    default: return res_ef_blocks<8>(op);
  }
}

cudaError_t launch_residual_ef(const OpDev& op, const double* x, const double* b, double* r,
                               const double* w, int natural, double* partial, const ResTail& tail,
                               float* split_hi, float* split_lo, int split_pitch, cudaStream_t s) {
  if (!residual_ef_supported(op) || !b || !partial) return cudaErrorInvalidValue;
  switch (op.d[0].N) {
    case 4: return launch_res_ef<4>(op, x, b, r, w, natural, partial, tail, split_hi, split_lo, split_pitch, s);
    case 5: return launch_res_ef<5>(op, x, b, r, w, natural, partial, tail, split_hi, split_lo, split_pitch, s);
    case 6: return launch_res_ef<6>(op, x, b, r, w, natural, partial, tail, split_hi, split_lo, split_pitch, s);
    case 7: return launch_res_ef<7>(op, x, b, r, w, natural, partial, tail, split_hi, split_lo, split_pitch, s);
    default: return launch_res_ef<8>(op, x, b, r, w, natural, partial, tail, split_hi, split_lo, split_pitch, s);
  }
}

#define SE_ORDERS(CALL)                                                                   \
  switch (op.d[0].N) {                                                                    \
    CALL(2) CALL(3) CALL(4) CALL(5) CALL(6) CALL(7) CALL(8) CALL(9) CALL(10) CALL(11) CALL(12) \
    default:                                                                              \
      return cudaErrorInvalidValue;                                                       \
  }
#define SE_APPLY_N(n) \
  case n:             \
    return launch_el<n, double, double, double>(op, x, y, s);
cudaError_t launch_op_apply(const OpDev& op, const double* x, double* y, cudaStream_t s) {
  // an SVV term (dense element blocks) is applied by the CG kernel's staged
  // per-unknown form, which carries it
  if (op.gamma != 0.0) return launch_residual(op, x, nullptr, y, nullptr, 0, nullptr, s);
  SE_ORDERS(SE_APPLY_N)
}
#undef SE_APPLY_N

#define SE_APPLY_LOW_N(n)                                                              \
  case n:                                                                              \
    return fp16 ? launch_el<n, __half, float, float>(op, (const __half*)x, y, s)       \
                : launch_el<n, __nv_bfloat16, float, float>(op, (const __nv_bfloat16*)x, y, s);
cudaError_t launch_op_apply_low(const OpDev& op, int fp16, const void* x, float* y, cudaStream_t s) {
  if (op.gamma != 0.0) return cudaErrorNotSupported;  // no SVV term in the low-precision apply
  SE_ORDERS(SE_APPLY_LOW_N)
}
#undef SE_APPLY_LOW_N
#undef SE_ORDERS

}  // namespace seg
