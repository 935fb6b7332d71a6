// Jacobi-preconditioned CG with the whole iteration state on the chip, sm_100a.
//
// A solve's elements are cut by a gx x gy grid into rectangular patches, one
// block each. A block keeps its patch's nodes for the whole solve: r in
// registers, x, the direction p, the Jacobi inverse and the two stiffness
// products in shared memory. A node on the line between two patches is held
// by both, with the same bits on either side. Memory sees two things per
// iteration:
//   * edge packets: at a line between patches the 1-D stiffness sum of a node
//     has one part from each side's element; each block publishes its part of
//     every edge node and reads the other's (a few hundred doubles a block);
//   * sum packets: a block's part of a dot product, read by every block of
//     the solve and added in the same order everywhere.
// A packet is 16 bytes, the value and a sequence number in one atomic store,
// so that a reader needs no fence, no flag and no barrier: waiting for the
// packets IS the grid barrier. A slot is reused only after another reduction
// over all blocks of the solve has completed, which no block joins before it
// has read the slot. Every block's sum packets have a 128-byte line of their
// own: with eight writers to a line an all-to-all sum over 148 blocks took
// 5100 cycles, with one 3150 (2440 over 64 blocks).
//
// One iteration (PETSc's KSPCG with PCJACOBI, the same tests and reasons as
// the streaming kernel in cg.cu):
//   A  p = z + b p; per element row and per element column the stiffness
//      product (one thread each, even/odd halves: (N+1)^2 / 2 FMAs instead of
//      (N+1)^2), edge packets, and p . A p as the sum of the element energies
//      (no assembled A p is needed for it); reduction 1;
//   B  A p assembled at each node from the two products and the edge
//      packets, x += a p, r -= a A p, z = D^-1 r, norms; reduction 2.
// With the constant null space removed, the mean of z is a third reduction.
//
// A small solve's blocks form one thread-block cluster and exchange the same
// values through distributed shared memory instead (CL).
//
// What bounds it: latency. At 64x64 elements, p = 8 (262,144 unknowns, 143
// patches) an iteration takes 6.4 us: about 1.5 us for each of the two
// reductions (store to L2, poll), 0.8 us for the stiffness products, 1 us for
// the node updates, the rest block sums and scalars; the streaming kernel
// took 20.4 us. At 16x16 elements, p = 6: 2.6 us as a cluster of 16 blocks,
// 4.1 us as 64 blocks through L2, 11.4 us with the streaming kernel.
// Several solves of one order share a launch as independent teams of blocks
// that never wait for one another.
//
// Every wait is bounded (kPatchPolls polls); a block whose wait gives up
// records the launch's sequence number in the error word and leaves.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "common.cuh"
#include "kh.cuh"

namespace seg {
namespace {

constexpr int kPT = kPatchThreads;
constexpr int kWarps = kPT / 32;
constexpr int kPatchK = 8;     // nodes per thread at most: their residuals stay in registers
constexpr int kPatchRegs = 4;  // nodes per thread whose whole state stays in registers
constexpr int kLine = kPatchLine;
constexpr int kPatchPolls = 1 << 22;

template <int N>
struct PatchArgs {
  PatchSolve one;            // the solve of a single-solve launch
  const PatchSolve* solves;  // a batch's solves (nullptr: one)
  const int* cta_solve;      // solve of each block (batch)
  PatchResult* res;
  double cf[Eo<N>::NC];  // even/odd halves of Kh (kh.cuh)
  double w[N + 1], kd[N + 1];  // GLL weights, stiffness diagonal
};

__device__ __forceinline__ void put(PatchPkt* p, double v, unsigned long long seq) {
  asm volatile(
      "{\n .reg .b128 q;\n mov.b128 q, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], q;\n}\n" ::"l"(p),
      "l"(__double_as_longlong(v)), "l"(seq)
      : "memory");
}
__device__ __forceinline__ bool get(const PatchPkt* p, unsigned long long seq, double& v) {
  long long b;
  unsigned long long s;
  asm volatile(
      "{\n .reg .b128 q;\n ld.relaxed.gpu.global.b128 q, [%2];\n mov.b128 {%0, %1}, q;\n}\n"
      : "=l"(b), "=l"(s)
      : "l"(p)
      : "memory");
  v = __longlong_as_double(b);
  return s == seq;
}

// ---- cluster form: stores into the other blocks' shared memory ----
__device__ __forceinline__ unsigned peer_address(const void* p, int rank) {
  unsigned a = (unsigned)__cvta_generic_to_shared(p), r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
// (st.async: the bytes count on the receiving block's mbarrier when they have
// landed, so that neither side needs a fence; a cluster barrier over plain
// stores took about 1100 cycles, this about 300)
__device__ __forceinline__ void store_peer(unsigned at, double v, unsigned bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(at),
               "l"(__double_as_longlong(v)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void put_peer(double2* p, int rank, double a, double b,
                                         unsigned long long* bar) {
  asm volatile(
      "st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(
          peer_address(p, rank)),
      "l"(__double_as_longlong(a)), "l"(__double_as_longlong(b)), "r"(peer_address(bar, rank))
      : "memory");
}
__device__ __forceinline__ void expect_bytes(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool wait_bytes(unsigned long long* bar, unsigned parity) {
  for (int k = 0; k < kPatchPolls; k++) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], "
        "%2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"((unsigned)__cvta_generic_to_shared(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}
__device__ __forceinline__ void cluster_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;"
               ::: "memory");
}
// Sum of the blocks' values in the inbox, by one warp, in a fixed order.
template <int NV>
__device__ __forceinline__ void sum_inbox(const double2* in, int G, double* out) {
  const int l = threadIdx.x & 31;
  const double2 v = l < G ? in[l] : make_double2(0.0, 0.0);
#pragma unroll
  for (int q = 0; q < NV; q++) {
    double s = q ? v.y : v.x;
#pragma unroll
    for (int o = kPatchMaxCluster / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    out[q] = s;
  }
}

// Sum over a solve's blocks of NV values, by one warp, in a fixed order; the
// packet of block c, value q is slots[c * kLine + q]. False: a wait gave up.
template <int NV>
__device__ __forceinline__ bool sum_packets(const PatchPkt* slots, int G, unsigned long long seq,
                                            double* out) {
  constexpr int C = (kPatchMaxBlocks + 31) / 32;
  const int l = threadIdx.x & 31;
  double v[C][NV];
  bool here = false;
  // every load of a poll issued before any is looked at
  for (int polls = 0; polls < kPatchPolls && !here; polls++) {
    bool got = true;
#pragma unroll
    for (int c = 0; c < C; c++)
      if (32 * c < G) {
        const PatchPkt* p = slots + (size_t)min(l + 32 * c, G - 1) * kLine;
#pragma unroll
        for (int q = 0; q < NV; q++) got = get(p + q, seq, v[c][q]) && got;
      }
    here = __all_sync(0xffffffffu, got);
  }
#pragma unroll
  for (int q = 0; q < NV; q++) {
    double s = 0.0;
#pragma unroll
    for (int c = 0; c < C; c++)
      if (l + 32 * c < G) s += v[c][q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    out[q] = s;
  }
  return here;
}

// Unknown index of unwrapped vertex g along d (-1: Dirichlet or outside).
__device__ __forceinline__ int unk1(const Dir& d, int g) {
  if (d.periodic) {
    const int L = d.nV - 1;
    if (g >= L) g -= L;
  }
  return (g >= d.lo && g < d.hi) ? g - d.lo : -1;
}

// Assembled 1-D weight and stiffness diagonal at vertex g.
template <int N>
__device__ __forceinline__ void assembled(const Dir& d, const double* w, const double* kd, int g,
                                          double& ws, double& ks) {
  if (d.periodic && g >= d.nV - 1) g -= d.nV - 1;
  const int e = g / N, a = g - e * N;
  ws = ks = 0.0;
  if (e < d.nE) {
    ws += w[a];
    ks += kd[a];
  }
  if (a == 0 && (e > 0 || d.periodic)) {
    ws += w[N];
    ks += kd[N];
  }
}

template <int NV>
__device__ __forceinline__ void warp_sum(double (&v)[NV]) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int q = 0; q < NV; q++) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
}

// Block sum of NV values (fixed order); valid in every lane of warp 0. One
// block barrier inside; red is [NV][kWarps].
template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV], double2* red2) {
  double* red = reinterpret_cast<double*>(red2);
  warp_sum<NV>(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0)
#pragma unroll
    for (int q = 0; q < NV; q++) red[q * kWarps + w] = v[q];
  __syncthreads();
  if (w == 0) {
    // every lane adds the warps' sums as a tree: shorter than more shuffles
#pragma unroll
    for (int q = 0; q < NV; q++) {
      double t[kWarps];
#pragma unroll
      for (int k = 0; k < kWarps; k += 2) {
        const double2 d = red2[(q * kWarps + k) / 2];
        t[k] = d.x;
        t[k + 1] = d.y;
      }
#pragma unroll
      for (int o = kWarps / 2; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < o; k++) t[k] += t[k + o];
      v[q] = t[0];
    }
  }
}

// K: nodes per thread at most. Up to kPatchRegs of them keep x, the Jacobi
// inverse, p and the mass coefficient in registers beside r; more keep those
// in shared memory.
//
// CL: the solve's blocks are one thread-block cluster (at most 16). The edge
// sums are then stored straight into the neighbour's shared memory and the
// dot products into every block's inbox, each with its bytes counted on the
// receiver's mbarrier, in place of the packets; the argument for reusing them
// is the same.
template <int N, int K, bool CL>
__global__ void __launch_bounds__(kPT, 1) cg_patch_kernel(const __grid_constant__ PatchArgs<N> A) {
  constexpr bool REG = K <= kPatchRegs;
  extern __shared__ double sm[];
  __shared__ PatchSolve S;
  __shared__ double2 red[kWarps];
  // scalars of the iteration, written by thread 0
  __shared__ struct {
    double beta, betaold, dpi, a, b, rnorm0, ttol, nn, zmean, cproj;
    double lo2, hi2;  // squares between which the norm decides nothing
    int its, reason, done, ok;
  } c;
  __shared__ PatchPkt *edge_out[4], *edge_in[4];
  // CL: where this block's edge sums go (shared address in the neighbour, 0:
  // the mesh ends here; doubles from one to the next), the sums that arrive
  __shared__ unsigned edge_at[4], edge_bar[4];
  __shared__ int edge_step[4];
  __shared__ unsigned long long arrived[3];  // of the sums A (with the edges), B, M
  __shared__ double2 inbox[3][kPatchMaxCluster];
  const int tid = threadIdx.x, warp = tid >> 5;
  const int si = A.cta_solve ? A.cta_solve[blockIdx.x] : 0;
  {
    const int* src = reinterpret_cast<const int*>(A.solves ? A.solves + si : &A.one);
    int* dst = reinterpret_cast<int*>(&S);
    for (int k = tid; k < (int)(sizeof(PatchSolve) / sizeof(int)); k += kPT) dst[k] = src[k];
    if (tid == 0) {
      c.beta = c.betaold = c.dpi = c.a = c.b = c.rnorm0 = c.ttol = c.nn = c.zmean = c.cproj = c.lo2 = c.hi2 = 0.0;
      c.its = c.reason = c.done = 0;
      c.ok = 1;
    }
  }
  __syncthreads();
  const Dir dx = S.d[0], dy = S.d[1];
  const int rank = blockIdx.x - S.cta0;
  const int pxi = rank % S.gx, pyi = rank / S.gx;
  const int ex0 = dx.nE * pxi / S.gx, ey0 = dy.nE * pyi / S.gy;
  const int nex = dx.nE * (pxi + 1) / S.gx - ex0, ney = dy.nE * (pyi + 1) / S.gy - ey0;
  const int PX = nex * N + 1, PY = ney * N + 1, pitch = PX | 1, nodes = PX * PY;
  const int vx0 = ex0 * N, vy0 = ey0 * N;
  double* P = sm;                 // direction, [PY][pitch]
  double* KX = P + PY * pitch;    // x stiffness products: parts of the element right of a node
  double* KY = KX + PY * pitch;   // y stiffness products: parts of the element above
  double* DI = KY + PY * pitch;   // Jacobi inverse and solution (!REG)
  double* X = DI + PY * pitch;
  double* RX = REG ? DI : X + PY * pitch;  // [nex+1][PY]: parts of the element left of node column e N
  double* RY = RX + (nex + 1) * PY;  // [ney+1][PX]: parts of the element below node row e N
  double* wx = RY + (ney + 1) * PX;
  double* wy = wx + PX;
  double* bwy = wy + PY;     // beta_x wy
  double* bwx = bwy + PY;    // beta_y wx
  double* ex_row = bwx + PX;  // beta_x wy of the rows this block owns (else 0)
  double* ey_col = ex_row + PY;
  double* kdx = ey_col + PX;  // assembled 1-D stiffness diagonals
  double* kdy = kdx + PX;

  // edges of this block (left, right, bottom, top): where its packets go, and
  // where those of the facing edge come from (nullptr: the mesh ends here)
  if (tid < 4) {
    const int side = tid, last = side < 2 ? S.gx - 1 : S.gy - 1, at = side < 2 ? pxi : pyi;
    const int step = side < 2 ? 1 : S.gx, periodic = side < 2 ? dx.periodic : dy.periodic;
    int nb;
    if (side & 1)
      nb = at < last ? rank + step : (periodic ? rank - last * step : -1);
    else
      nb = at > 0 ? rank - step : (periodic ? rank + last * step : -1);
    const size_t EM = S.edge_stride;
    if constexpr (CL) {
      // the neighbour's arrays (its patch may be one element wider or higher)
      unsigned at = 0;
      int st = 1;
      if (nb >= 0) {
        const int nx = nb % S.gx, ny = nb / S.gx;
        const int bx = dx.nE * (nx + 1) / S.gx - dx.nE * nx / S.gx;
        const int by = dy.nE * (ny + 1) / S.gy - dy.nE * ny / S.gy;
        const int qx = bx * N + 1, qy = by * N + 1, qp = qx | 1, a = qy * qp;
        const int rx = (REG ? 3 : 5) * a;  // P, KX, KY (DI, X), then RX, RY
        const int off = side == 0   ? a + bx * N
                        : side == 1 ? rx
                        : side == 2 ? 2 * a + by * N * qp
                                    : rx + (bx + 1) * qy;
        st = side == 0 ? qp : 1;
        at = peer_address(sm + off, nb);
        edge_bar[side] = peer_address(&arrived[0], nb);
      }
      edge_at[side] = at;
      edge_step[side] = st;
    } else {
      edge_out[side] = nb >= 0 ? S.edges + ((size_t)rank * 4 + side) * EM : nullptr;
      edge_in[side] = nb >= 0 ? S.edges + ((size_t)nb * 4 + (side ^ 1)) * EM : nullptr;
    }
  }

  // tables
  for (int t = tid; t < PX + PY; t += kPT) {
    double ws, ks;
    if (t < PX) {
      assembled<N>(dx, A.w, A.kd, vx0 + t, ws, ks);
      wx[t] = ws;
      bwx[t] = S.by * ws;
      kdx[t] = ks;
      ey_col[t] = (t < PX - 1 || (!dx.periodic && pxi == S.gx - 1)) ? S.by * ws : 0.0;
    } else {
      const int j = t - PX;
      assembled<N>(dy, A.w, A.kd, vy0 + j, ws, ks);
      wy[j] = ws;
      bwy[j] = S.bx * ws;
      kdy[j] = ks;
      ex_row[j] = (j < PY - 1 || (!dy.periodic && pyi == S.gy - 1)) ? S.bx * ws : 0.0;
    }
  }
  __syncthreads();

  for (int t = tid; t < (REG ? 3 : 5) * PY * pitch; t += kPT) P[t] = 0.0;
  for (int t = tid; t < (nex + 1) * PY; t += kPT) RX[t] = 0.0;
  for (int t = tid; t < (ney + 1) * PX; t += kPT) RY[t] = 0.0;
  if constexpr (CL) {
    if (tid == 0) {
      for (int k = 0; k < 3; k++)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(
            (unsigned)__cvta_generic_to_shared(&arrived[k])) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    cluster_sync();  // no block stores into another before it has cleared its arrays
  } else {
    __syncthreads();
  }

  // per-thread nodes: packed (unknown, own, j, i), residual and (REG) x, D^-1,
  // p, alpha wx wy
  constexpr int KR = REG ? K : 1;
  double r[K], xr[KR], dr[KR], pr[KR], mr[KR];
  unsigned ij[K];
  constexpr unsigned kUnk = 0x80000000u, kOwn = 0x40000000u;
  auto node_i = [](unsigned q) { return (int)(q & 0x3fffu); };
  auto node_j = [](unsigned q) { return (int)((q >> 14) & 0x3fffu); };
  auto diag = [&](unsigned q) {
    const int i = node_i(q), j = node_j(q);
    return S.alpha * wx[i] * wy[j] + S.bx * kdx[i] * wy[j] + S.by * wx[i] * kdy[j];
  };
#pragma unroll
  for (int k = 0; k < K; k++) {
    const int n = tid + k * kPT;
    r[k] = 0.0;
    if constexpr (REG) xr[k] = dr[k] = pr[k] = mr[k] = 0.0;
    ij[k] = 0;
    if (n < nodes) {
      const int j = n / PX, i = n - j * PX;
      const int ux = unk1(dx, vx0 + i), uy = unk1(dy, vy0 + j);
      unsigned f = (unsigned)(i | (j << 14));
      if (ux >= 0 && uy >= 0) {
        f |= kUnk;
        // the last column / row of nodes is the next patch's first
        if ((i < PX - 1 || (!dx.periodic && pxi == S.gx - 1)) &&
            (j < PY - 1 || (!dy.periodic && pyi == S.gy - 1)))
          f |= kOwn;
        r[k] = S.b[(size_t)uy * S.G0 + ux];
      }
      ij[k] = f;
    }
  }

  // sum packets, one line a block
  enum { SUM_A = 0, SUM_B = 1, SUM_M = 2 };
  auto slot = [&](int k) { return S.slots + k * kLine * S.gx * S.gy; };
  unsigned long long seq = S.seq0;
  const int nt = S.norm_type;

  // CL, warp 0: the block's two values to every block's inbox, then every
  // block's (and extra bytes: the edge sums) in
  unsigned parity = 0;  // bit k: of arrived[k]
  auto exchange = [&](int k, double v0, double v1, unsigned extra) {
    const int G = S.gx * S.gy;
    if (tid == 0) expect_bytes(&arrived[k], 16u * (unsigned)G + extra);
    if (tid < G) put_peer(&inbox[k][rank], tid, v0, v1, &arrived[k]);
    __syncwarp();
    const bool ok = wait_bytes(&arrived[k], (parity >> k) & 1u);
    parity ^= 1u << k;
    return __all_sync(0xffffffffu, ok) != 0;
  };

  // A block's NV sums out, then (warp 0) every block's in: `then` runs on
  // thread 0 with the totals. Ends with a block barrier; false: gave up.
  auto reduce2 = [&](int slots, double v0, double v1, auto&& then) {
    double v[2] = {v0, v1};
    block_sum<2>(v, red);
    if (warp == 0) {
      double t[2];
      bool ok;
      if constexpr (CL) {
        ok = exchange(slots, v[0], v[1], 0);
        sum_inbox<2>(inbox[slots], S.gx * S.gy, t);
      } else {
        if (tid < 2) put(slot(slots) + kLine * rank + tid, tid ? v[1] : v[0], seq);
        ok = sum_packets<2>(slot(slots), S.gx * S.gy, seq, t);
      }
      if (tid == 0) {
        if (!ok) c.ok = 0;
        then(t[0], t[1]);
      }
    }
    __syncthreads();
    seq++;
    return c.ok != 0;
  };
  auto reduce1 = [&](int slots, double v0, auto&& then) {
    double v[1] = {v0};
    block_sum<1>(v, red);
    if (warp == 0) {
      double t[1];
      bool ok;
      if constexpr (CL) {
        ok = exchange(slots, v[0], 0.0, 0);
        sum_inbox<1>(inbox[slots], S.gx * S.gy, t);
      } else {
        if (tid == 0) put(slot(slots) + kLine * rank, v[0], seq);
        ok = sum_packets<1>(slot(slots), S.gx * S.gy, seq, t);
      }
      if (tid == 0) {
        if (!ok) c.ok = 0;
        then(t[0]);
      }
    }
    __syncthreads();
    seq++;
    return c.ok != 0;
  };
  // the last common step of a cluster's blocks, on every way out: none leaves
  // while another may store into it (one that gave up early waits here for
  // the others, whose waits for it run out)
  auto leave = [&]() {
    if constexpr (CL) cluster_sync();
  };
  auto give_up = [&]() {
    leave();
    if (tid == 0) atomicExch(&A.res[si].err, S.seq0);
  };
  // KSPConvergedDefault on the norm at iteration n (thread 0). nn is the
  // squared norm (or its signed form, natural); a square clear of both
  // thresholds decides nothing and spares the root, which is long on the path
  // every block waits for.
  auto converged = [&](int n, double nn) {
    c.nn = nn;
    if (n > 0 && nn > c.lo2 && nn < c.hi2) return;
    const double dp = sqrt(nt == 2 ? fabs(nn) : nn);
    if (!(dp == dp) || isinf(dp)) {
      c.reason = -9;
      c.done = 1;
      return;
    }
    if (n == 0) {
      c.rnorm0 = dp;
      c.ttol = fmax(S.rtol * dp, S.atol);
      const double up = S.dtol * dp;
      // only where the squares are far from under- and overflow
      if (nt != 2 && c.ttol > 1e-140 && up < 1e140 && up > 1e-140) {
        c.lo2 = c.ttol * c.ttol * (1.0 + 1e-12);
        c.hi2 = up * up * (1.0 - 1e-12);
      }
    }
    if (dp <= c.ttol) {
      c.reason = dp < S.atol ? 3 : 2;
      c.done = 1;
    } else if (n > 0 && dp >= S.dtol * c.rnorm0) {
      c.reason = -4;
      c.done = 1;
    }
  };

  // a node's word, opaque to the compiler: it would otherwise keep every
  // node's addresses in registers across the iteration loop (and spill)
  auto node = [&](int k) {
    unsigned f = ij[k];
    asm volatile("" : "+r"(f));
    return f;
  };

  // right-hand side off the operator's range (remove_null == 2): f -= (sum f
  // / sum d) d
  if (S.remove_null == 2) {
    double s0 = 0.0, s1 = 0.0;
#pragma unroll
    for (int k = 0; k < K; k++) {
      const unsigned f = node(k);
      if (!(f & kOwn)) continue;
      s0 += r[k];
      s1 += diag(f);
    }
    if (!reduce2(SUM_A, s0, s1, [&](double t0, double t1) { c.cproj = t0 / t1; })) {
      give_up();
      return;
    }
  }
  double s_zr = 0.0, s_n = 0.0, s_z = 0.0;
  {
    const double cp = c.cproj;
#pragma unroll
    for (int k = 0; k < K; k++) {
      const unsigned f = node(k);
      if (!(f & kUnk)) continue;
      const double d = diag(f);
      r[k] = r[k] - cp * d;
      const double di = 1.0 / d;
      if constexpr (REG) {
        dr[k] = di;
        mr[k] = S.alpha * wx[node_i(f)] * wy[node_j(f)];
      } else {
        DI[node_j(f) * pitch + node_i(f)] = di;
      }
      const double z = r[k] * di;
      if (f & kOwn) {
        s_zr += z * r[k];
        s_n += nt == 1 ? r[k] * r[k] : z * z;
        s_z += z;
      }
    }
  }
  auto dinv = [&](int k, int q) {
    if constexpr (REG)
      return dr[k];
    else
      return DI[q];
  };
  // z with its mean removed: the sums again
  auto mean_sums = [&]() -> bool {
    const double n = (double)S.n;
    if (!reduce1(SUM_M, s_z, [&](double t) { c.zmean = t / n; })) return false;
    const double zm = c.zmean;
    s_zr = s_n = 0.0;
#pragma unroll
    for (int k = 0; k < K; k++) {
      const unsigned f = node(k);
      if (!(f & kOwn)) continue;
      const double z = r[k] * dinv(k, node_j(f) * pitch + node_i(f)) - zm;
      s_zr += z * r[k];
      s_n += nt == 1 ? r[k] * r[k] : z * z;
    }
    return true;
  };
  bool good = S.remove_null ? mean_sums() : true;
  good = good && reduce2(SUM_B, s_zr, s_n, [&](double zr, double nn) {
    converged(0, nt == 2 ? zr : nn);
    c.beta = zr;
    if (!c.done && S.max_it <= 0) {
      c.reason = -3;
      c.done = 1;
    }
    if (!c.done && c.beta == 0.0) {
      c.reason = 3;
      c.done = 1;
    }
  });

  // this thread's first item of the stiffness passes: x items (row j, element
  // e) from thread 0, y items (column i, element e) from the next whole warp
  const int nxi = nex * PY, nxp = (nxi + 31) & ~31, nit = nxp + ney * PX;

  // this block's part of an edge node's stiffness sum, to the other side
  auto edge_sum = [&](int side, int at, double v) {
    if constexpr (CL) {
      if (edge_at[side])
        store_peer(edge_at[side] + 8u * (unsigned)(at * edge_step[side]), v, edge_bar[side]);
    } else {
      if (edge_out[side]) put(edge_out[side] + at, v, seq);
    }
  };

  while (good && !c.done) {
    // ---- A: direction, stiffness products, energies ----
    double acc[1] = {0.0};
    {
      const double b = c.b, zm = c.zmean;
      const bool first = c.its == 0;
#pragma unroll
      for (int k = 0; k < K; k++) {
        const unsigned f = node(k);
        if (!(f & kUnk)) continue;
        const int i = node_i(f), j = node_j(f), q = j * pitch + i;
        const double z = r[k] * dinv(k, q) - zm;
        double p, m;
        if constexpr (REG) {
          p = first ? z : fma(b, pr[k], z);
          pr[k] = p;
          m = mr[k];
        } else {
          p = first ? z : fma(b, P[q], z);
          m = S.alpha * wx[i] * wy[j];
        }
        P[q] = p;
        if (f & kOwn) acc[0] = fma(m * p, p, acc[0]);
      }
    }
    __syncthreads();
    for (int it = tid; it < nit; it += kPT) {
      if (it < nxp) {
        if (it >= nxi) continue;
        const int e = it / PY, j = it - e * PY;
        const double* u = P + j * pitch + e * N;
        double v[N + 1], o[N + 1];
#pragma unroll
        for (int k = 0; k <= N; k++) v[k] = u[k];
        const double en = eo_product<N, true>(A.cf, v, o);
        acc[0] = fma(ex_row[j], en, acc[0]);
        if (e == 0) edge_sum(0, j, o[0]);
        if (e == nex - 1) edge_sum(1, j, o[N]);
        double* kx = KX + j * pitch + e * N;
#pragma unroll
        for (int k = 0; k < N; k++) kx[k] = o[k];
        RX[(e + 1) * PY + j] = o[N];
      } else {
        const int t = it - nxp, e = t / PX, i = t - e * PX;
        const double* u = P + (e * N) * pitch + i;
        double v[N + 1], o[N + 1];
#pragma unroll
        for (int k = 0; k <= N; k++) v[k] = u[k * pitch];
        const double en = eo_product<N, true>(A.cf, v, o);
        acc[0] = fma(ey_col[i], en, acc[0]);
        if (e == 0) edge_sum(2, i, o[0]);
        if (e == ney - 1) edge_sum(3, i, o[N]);
        double* ky = KY + (e * N) * pitch + i;
#pragma unroll
        for (int k = 0; k < N; k++) ky[k * pitch] = o[k];
        RY[(e + 1) * PX + i] = o[N];
      }
    }
    block_sum<1>(acc, red);
    if (warp == 0) {
      double t[1];
      bool ok;
      if constexpr (CL) {
        const unsigned edges = (edge_at[0] ? PY : 0) + (edge_at[1] ? PY : 0) +
                               (edge_at[2] ? PX : 0) + (edge_at[3] ? PX : 0);
        ok = exchange(SUM_A, acc[0], 0.0, 8u * edges);
        sum_inbox<1>(inbox[SUM_A], S.gx * S.gy, t);
      } else {
        if (tid == 0) put(slot(SUM_A) + kLine * rank, acc[0], seq);
        ok = sum_packets<1>(slot(SUM_A), S.gx * S.gy, seq, t);
      }
      if (tid == 0) {
        if (!ok) c.ok = 0;
        const double dpi = t[0], old = c.dpi;
        c.dpi = dpi;
        c.betaold = c.beta;
        if (dpi == 0.0 || (c.its > 0 && dpi * old <= 0.0)) {
          c.reason = -10;
          c.done = 1;
        } else {
          c.a = c.beta / dpi;
        }
      }
    } else if constexpr (!CL) {
      // the other warps collect the edge packets meanwhile
      for (int t = tid - 32; t < 2 * (PX + PY); t += kPT - 32) {
        const int side = t < 2 * PY ? (t < PY ? 0 : 1) : (t < 2 * PY + PX ? 2 : 3);
        const int q = t - (side < 2 ? side * PY : 2 * PY + (side - 2) * PX);
        const PatchPkt* src = edge_in[side];
        if (!src) continue;
        src += q;
        double* dst = side == 0   ? RX + q
                      : side == 1 ? KX + q * pitch + nex * N
                      : side == 2 ? RY + q
                                  : KY + (ney * N) * pitch + q;
        double v;
        int polls = 0;
        bool ok;
        while (!(ok = get(src, seq, v)))
          if (++polls > kPatchPolls) break;
        if (!ok) c.ok = 0;
        *dst = v;
      }
    }
    __syncthreads();
    seq++;
    if (!c.ok) break;
    if (c.done) break;

    // ---- B: A p at every node, update, norms ----
    s_zr = s_n = s_z = 0.0;
    {
      const double a = c.a;
#pragma unroll
      for (int k = 0; k < K; k++) {
        const unsigned f = node(k);
        if (!(f & kUnk)) continue;
        const int i = node_i(f), j = node_j(f), q = j * pitch + i;
        const int ei = i / N, ej = j / N;
        double kx = KX[q], ky = KY[q];
        if (ei * N == i) kx += RX[ei * PY + j];
        if (ej * N == j) ky += RY[ej * PX + i];
        double p, m;
        if constexpr (REG) {
          p = pr[k];
          m = mr[k];
          xr[k] = fma(a, p, xr[k]);
        } else {
          p = P[q];
          m = S.alpha * wx[i] * wy[j];
          X[q] = fma(a, p, X[q]);
        }
        const double w = m * p + bwy[j] * kx + bwx[i] * ky;
        r[k] = fma(-a, w, r[k]);
        const double z = r[k] * dinv(k, q);
        if (f & kOwn) {
          s_zr += z * r[k];
          s_n += nt == 1 ? r[k] * r[k] : z * z;
          s_z += z;
        }
      }
    }
    if (S.remove_null) good = mean_sums();
    good = good && reduce2(SUM_B, s_zr, s_n, [&](double zr, double nn) {
      c.its += 1;
      converged(c.its, nt == 2 ? zr : nn);
      if (!c.done) {
        if (zr == 0.0) {
          c.reason = 3;
          c.done = 1;
        } else if (zr * c.betaold < 0.0) {
          c.reason = -8;
          c.done = 1;
        } else if (c.its >= S.max_it) {
          c.reason = -3;
          c.done = 1;
        } else {
          c.beta = zr;
          c.b = zr / c.betaold;
        }
      }
    });
  }
  if (!c.ok) {
    give_up();
    return;
  }
  leave();
#pragma unroll
  for (int k = 0; k < K; k++) {
    const unsigned f = node(k);
    if (!(f & kOwn)) continue;
    const int ux = unk1(dx, vx0 + node_i(f)), uy = unk1(dy, vy0 + node_j(f));
    double v;
    if constexpr (REG)
      v = xr[k];
    else
      v = X[node_j(f) * pitch + node_i(f)];
    S.x[(size_t)uy * S.G0 + ux] = v;
  }
  if (rank == 0 && tid == 0) {
    PatchResult& o = A.res[si];
    o.dp = sqrt(nt == 2 ? fabs(c.nn) : c.nn);
    o.rnorm0 = c.rnorm0;
    o.beta = c.beta;
    o.its = c.its;
    o.reason = c.reason;
  }
}

size_t patch_smem(int N, int nex, int ney, bool regs) {
  const size_t PX = (size_t)nex * N + 1, PY = (size_t)ney * N + 1, pitch = PX | 1;
  return sizeof(double) *
         ((regs ? 3 : 5) * PY * pitch + (nex + 1) * PY + (ney + 1) * PX + 4 * (PX + PY));
}

// clusters (cluster form only): how many of these clusters the device holds,
// instead of a launch.
template <int N>
cudaError_t launch_n(const PatchLaunch& L, cudaStream_t s, int* clusters) {
  constexpr int n = N + 1;
  PatchArgs<N> A;
  std::memset(&A, 0, sizeof(A));
  if (L.one) A.one = *L.one;
  A.solves = L.solves;
  A.cta_solve = L.cta_solve;
  A.res = L.res;
  eo_coefs<N>(L.Kh, 1.0, A.cf);
  for (int a = 0; a < n; a++) {
    A.w[a] = L.w[a];
    A.kd[a] = L.Kh[a * n + a];
  }
  const void* f =
      L.cluster ? (L.in_registers ? (const void*)cg_patch_kernel<N, kPatchRegs, true>
                                  : (const void*)cg_patch_kernel<N, kPatchK, true>)
                : (L.in_registers ? (const void*)cg_patch_kernel<N, kPatchRegs, false>
                                  : (const void*)cg_patch_kernel<N, kPatchK, false>);
  cudaError_t e =
      cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, kPatchSmemMax);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg;
  std::memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(L.blocks);
  cfg.blockDim = dim3(kPT);
  cfg.dynamicSmemBytes = L.smem;
  cfg.stream = s;
  cudaLaunchAttribute at;
  std::memset(&at, 0, sizeof(at));
  if (L.cluster) {
    if ((e = cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)) !=
        cudaSuccess)
      return e;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = L.blocks;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
  } else {
    at.id = cudaLaunchAttributeCooperative;
    at.val.cooperative = 1;
  }
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  if (clusters) return cudaOccupancyMaxActiveClusters(clusters, f, &cfg);
  void* args[] = {&A};
  return cudaLaunchKernelExC(&cfg, f, args);
}

}  // namespace

// The cut of one solve over at most max_blocks blocks that makes the slowest
// block's iteration shortest: its stiffness items (about 1.25 cycles each with
// four FP64 pipes) and nodes, plus a little for every block that the
// reductions read.
void patch_plan_table(const OpDev& op, int max_blocks, PatchPlan* out) {
  const int N = op.d[0].N, cap = std::min(max_blocks, kPatchMaxBlocks);
  for (int g = 0; g <= max_blocks; g++) {
    std::memset(&out[g], 0, sizeof(PatchPlan));
    out[g].cost = 1e300;
  }
  if (op.gamma != 0.0 || N < 2 || N > SE_MAXN) return;
  for (int gx = 1; gx <= std::min(cap, op.d[0].nE); gx++)
    for (int gy = 1; gy <= std::min(cap / gx, op.d[1].nE); gy++) {
      const int mx = (op.d[0].nE + gx - 1) / gx, my = (op.d[1].nE + gy - 1) / gy;
      const long px = (long)mx * N + 1, py = (long)my * N + 1;
      if (px * py > (long)kPT * kPatchK) continue;
      const bool regs = px * py <= (long)kPT * kPatchRegs;
      // room for the other kernel form too: a batch may mix cuts of both
      if (patch_smem(N, mx, my, false) > kPatchSmemMax) continue;
      const size_t sm = patch_smem(N, mx, my, regs);
      const double items = (double)(mx * py + my * px);
      const double rounds = std::ceil((items + 31) / kPT);
      const double t = (0.9 + 0.06 * N) * items + 250 * rounds + 0.8 * px * py + 3.0 * gx * gy;
      PatchPlan& p = out[gx * gy];
      if (t < p.cost) p = {gx, gy, (int)(std::max(px, py) + kLine - 1) / kLine * kLine, regs, 0, sm, t};
    }
  for (int g = 1; g <= max_blocks; g++)
    if (out[g - 1].cost <= out[g].cost) out[g] = out[g - 1];
}

size_t patch_smem_bytes(const OpDev& op, const PatchPlan& p, bool in_registers) {
  return patch_smem(op.d[0].N, (op.d[0].nE + p.gx - 1) / p.gx, (op.d[1].nE + p.gy - 1) / p.gy,
                    in_registers);
}

namespace {
cudaError_t dispatch(const PatchLaunch& L, cudaStream_t s, int* clusters) {
  switch (L.N) {
    case 2: return launch_n<2>(L, s, clusters);
    case 3: return launch_n<3>(L, s, clusters);
    case 4: return launch_n<4>(L, s, clusters);
    case 5: return launch_n<5>(L, s, clusters);
    case 6: return launch_n<6>(L, s, clusters);
    case 7: return launch_n<7>(L, s, clusters);
    case 8: return launch_n<8>(L, s, clusters);
    case 9: return launch_n<9>(L, s, clusters);
    case 10: return launch_n<10>(L, s, clusters);
    case 11: return launch_n<11>(L, s, clusters);
    case 12: return launch_n<12>(L, s, clusters);
    default: return cudaErrorInvalidValue;
  }
}
}  // namespace

cudaError_t launch_cg_patch(const PatchLaunch& L, cudaStream_t s) { return dispatch(L, s, nullptr); }

// The cost model's cycles count work; times 1.8 and with 6700 cycles of
// latency (reductions through L2, block sums, scalars) they matched 16x16
// p = 6 over 64 blocks (7900) and 64x64 p = 8 over 143 (12000); inside a
// cluster the latency is about 3100 (16x16 p = 6 over 16 blocks: 5000). So
// systems up to 21,000 to 37,000 unknowns, by order and element counts, run as a
// cluster. What fits a grid runs
// as one: with the state in shared memory (more than 2048 nodes a block) an
// iteration takes 7.3 us at 322,560 unknowns, p = 8 (streaming 26.1), 8.3 at
// 518,400, p = 6 (31.7), 10.6 at 484,416, p = 12 (39.4).
bool patch_plan_single(const OpDev& op, int max_blocks, PatchPlan* out) {
  max_blocks = std::min(max_blocks, kPatchMaxBlocks);
  PatchPlan t[kPatchMaxBlocks + 1];
  patch_plan_table(op, max_blocks, t);
  *out = t[max_blocks];
  if (out->gx == 0) return false;
  const double grid = 1.8 * out->cost + 6700.0;
  // t improves with the block count: the largest cluster first
  for (int g = std::min(kPatchMaxCluster, max_blocks); g > 0; g--) {
    PatchPlan p = t[g];
    if (p.gx == 0 || 1.8 * p.cost + 3100.0 >= grid) break;
    if (p.gx * p.gy != g) continue;  // the same cut as a smaller count's
    p.cluster = 1;
    PatchLaunch L;
    std::memset(&L, 0, sizeof(L));
    L.N = op.d[0].N;
    L.blocks = g;
    L.in_registers = p.in_registers;
    L.cluster = true;
    L.smem = p.smem;
    L.Kh = op.Kh;
    L.w = op.w;
    int held = 0;
    if (dispatch(L, 0, &held) == cudaSuccess && held > 0) {
      *out = p;
      break;
    }
    cudaGetLastError();
  }
  return true;
}

}  // namespace seg
