// Dense GEMMs of the fast-diagonalization solve (fdm.cu / api.cu), written
// for the solve's CUDA graph: one kernel launch per product, no workspace,
// no library-internal nodes, so the products can sit inside the graph's
// conditional refinement loop.
//
// C (M x N) = A (M x K) * B (K x N), all row-major with leading dimensions,
// on the tensor cores through warp-level MMA:
//   FP64 data, m16n8k8 f64 MMA (Blackwell's FP64 tensor path; there is no FP64
//   kind of the tcgen05 MMA), FP64 accumulation (launch_fdm_dgemm);
//   P = 1  FP32 data rounded to TF32, m16n8k8 tf32 MMA, FP32 accumulation;
//   P = 2  BF16 data, m16n8k16 bf16 MMA, FP32 accumulation (launch_fdm_gemm).
//
// Low precision: 32 x 32 tiles while a grid of 64 x 64 tiles would leave SMs
// idle, 64 x 64 above that, 2 x 2 warps; operands pass through registers
// (converted, and the FP64 first operand scaled, on the way) into
// double-buffered shared memory, from rows of any length. Epilogues: store;
// store after the spectral divide C[l][k] /= alpha + bx lx[k] + by ly[l]
// (entries whose divisor is below null_tol in magnitude -- the null mode --
// become 0); accumulate into an FP64 C with an optional scale read from device
// memory.
//
// FP64: one operand is a direction's factor. Where the direction is folded
// (FoldDir, fdm.cu) that factor is block-diagonal, an even and an odd block
// stored one after the other, and the product two of half the depth in one
// launch; a block of threads works inside one of them. Tiles of 32 x 24, 32 or
// 40 by 4 warps that split each K stage and sum their partial tiles in warp
// order; 64 x 64 by 2 x 2 warps where an unfolded array of that size covers the
// SMs with them (a folded one may not: its two parts' partial tiles). Operands
// stream through a multi-stage pipeline of 16-byte copies, so rows start on
// even offsets: folded arrays and factors are laid out that way, and only the
// input of an inverse that does not fold may not be (D_FIRST, 8-byte copies).
// The divide moves the low modes of both directions out of C into zlow
// (8 x 8), leaving zeros: a smooth solution's largest coefficients, which the
// unfolding, or the last product where nothing is folded (D_FINISH), adds back
// in double-double so that the products' rounding of them does not dominate
// the solve's first residual.
#include <cuda_bf16.h>

#include <cstdint>

#include "common.cuh"

namespace seg {
namespace {

constexpr int kThreads = 128;

template <int P>
struct Tr;
template <>
struct Tr<1> {
  typedef uint32_t S;  // TF32 bit patterns
  typedef float Acc;
  enum { BK = 32, KS = 8, AP = 4, BP = 8 };
};
template <>
struct Tr<2> {
  typedef __nv_bfloat16 S;
  typedef float Acc;
  enum { BK = 32, KS = 16, AP = 8, BP = 8 };
};

__device__ __forceinline__ float as_f(float x) { return x; }
__device__ __forceinline__ float as_f(__nv_bfloat16 x) { return __bfloat162float(x); }

__device__ __forceinline__ uint32_t to_tf32(float f) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(f));
  return r;
}

// Element of an operand in the shared-memory type of precision P; `scale`
// multiplies FP64 inputs (the FDM's 1/max|r| normalisation).
template <int P, class T>
__device__ __forceinline__ typename Tr<P>::S to_s(T x, double scale) {
  float f;
  if constexpr (sizeof(T) == 8)
    f = (float)(x * scale);
  else
    f = as_f(x);
  if constexpr (P == 1)
    return to_tf32(f);
  else
    return __float2bfloat16_rn(f);
}

__device__ __forceinline__ void mma_f64(double (&c)[4], const double (&a)[4], const double (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ __forceinline__ uint32_t pack_bf16(__nv_bfloat16 lo, __nv_bfloat16 hi) {
  return (uint32_t)__bfloat16_as_ushort(lo) | ((uint32_t)__bfloat16_as_ushort(hi) << 16);
}

template <class TA, class TB, class TC>
struct GemmArgs {
  const TA* A;
  const TB* B;
  TC* C;
  int M, N, K, lda, ldb, ldc;
  const double* amax;  // A scale 1/max (FP64 A only), nullptr: 1
  const double* cmax;  // accumulate scale, nullptr: 1
  const double *lx, *ly;
  double alpha, bx, by, null_tol;
};

// Place of mode m among the low modes carried apart (-1: not one).
__device__ __forceinline__ int low_mode(const FdmLowMap& l, int m) {
  if (m < l.even) return m;
  const int o = m - l.split;
  return o >= 0 && o < l.odd ? kFdmLow / 2 + o : -1;
}

enum { EPI_STORE = 0, EPI_DIVIDE = 1, EPI_ACCUM = 2 };

// Low-precision products (P = 1, 2): BM x BN block tile of 2 x 2 warps,
// operands converted (and the FP64 first operand scaled) on the way from
// global memory through registers into double-buffered shared memory.
template <int P, int kBM, int kBN, class TA, class TB, class TC, int EPI>
__global__ void __launch_bounds__(kThreads) fdm_gemm_kernel(const GemmArgs<TA, TB, TC> g) {
  typedef typename Tr<P>::S S;
  typedef typename Tr<P>::Acc Acc;
  constexpr int BK = Tr<P>::BK, KS = Tr<P>::KS;
  constexpr int AS = BK + Tr<P>::AP, BS = kBN + Tr<P>::BP;
  constexpr int AE = kBM * BK / kThreads, BE = BK * kBN / kThreads;
  constexpr int MT = kBM / 32, NT = kBN / 16;  // m16n8 tiles per warp
  __shared__ __align__(16) S As[2][kBM * AS];
  __shared__ __align__(16) S Bs[2][BK * BS];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gq = lane >> 2, tq = lane & 3;
  const int wm = (warp >> 1) * (kBM / 2), wn = (warp & 1) * (kBN / 2);
  const int m0 = blockIdx.y * kBM, n0 = blockIdx.x * kBN;
  double ascale = 1.0;
  if (g.amax) {
    const double m = *g.amax;
    ascale = m > 0.0 ? 1.0 / m : 0.0;
  }

  S ra[AE], rb[BE];
  auto load = [&](int k0) {
#pragma unroll
    for (int r = 0; r < AE; r++) {
      const int e = tid + r * kThreads;
      const int row = e / BK, col = e % BK;
      const int gr = m0 + row, gc = k0 + col;
      ra[r] = (gr < g.M && gc < g.K) ? to_s<P>(g.A[(size_t)gr * g.lda + gc], ascale)
                                     : to_s<P>(0.0, 1.0);
    }
#pragma unroll
    for (int r = 0; r < BE; r++) {
      const int e = tid + r * kThreads;
      const int row = e / kBN, col = e % kBN;
      const int gr = k0 + row, gc = n0 + col;
      rb[r] = (gr < g.K && gc < g.N) ? to_s<P>(g.B[(size_t)gr * g.ldb + gc], 1.0) : to_s<P>(0.0, 1.0);
    }
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int r = 0; r < AE; r++) {
      const int e = tid + r * kThreads;
      As[buf][(e / BK) * AS + e % BK] = ra[r];
    }
#pragma unroll
    for (int r = 0; r < BE; r++) {
      const int e = tid + r * kThreads;
      Bs[buf][(e / kBN) * BS + e % kBN] = rb[r];
    }
  };

  Acc acc[MT][NT][4];
#pragma unroll
  for (int i = 0; i < MT; i++)
#pragma unroll
    for (int j = 0; j < NT; j++)
#pragma unroll
      for (int q = 0; q < 4; q++) acc[i][j][q] = Acc(0);

  const int KT = (g.K + BK - 1) / BK;
  load(0);
  store(0);
  __syncthreads();
  for (int kt = 0; kt < KT; kt++) {
    const int buf = kt & 1;
    if (kt + 1 < KT) load((kt + 1) * BK);
    const S* as = As[buf];
    const S* bs = Bs[buf];
#pragma unroll
    for (int kk = 0; kk < BK; kk += KS) {
      if constexpr (P == 1) {
        S a[MT][4], b[NT][2];
#pragma unroll
        for (int mt = 0; mt < MT; mt++) {
          const int r0 = wm + mt * 16 + gq;
          a[mt][0] = as[r0 * AS + kk + tq];
          a[mt][1] = as[(r0 + 8) * AS + kk + tq];
          a[mt][2] = as[r0 * AS + kk + tq + 4];
          a[mt][3] = as[(r0 + 8) * AS + kk + tq + 4];
        }
#pragma unroll
        for (int nt = 0; nt < NT; nt++) {
          const int c0 = wn + nt * 8 + gq;
          b[nt][0] = bs[(kk + tq) * BS + c0];
          b[nt][1] = bs[(kk + tq + 4) * BS + c0];
        }
#pragma unroll
        for (int mt = 0; mt < MT; mt++)
#pragma unroll
          for (int nt = 0; nt < NT; nt++) {
            mma_tf32(acc[mt][nt], a[mt], b[nt]);
          }
      } else {
        uint32_t a[MT][4], b[NT][2];
#pragma unroll
        for (int mt = 0; mt < MT; mt++) {
          const int r0 = wm + mt * 16 + gq;
          a[mt][0] = *reinterpret_cast<const uint32_t*>(&as[r0 * AS + kk + 2 * tq]);
          a[mt][1] = *reinterpret_cast<const uint32_t*>(&as[(r0 + 8) * AS + kk + 2 * tq]);
          a[mt][2] = *reinterpret_cast<const uint32_t*>(&as[r0 * AS + kk + 2 * tq + 8]);
          a[mt][3] = *reinterpret_cast<const uint32_t*>(&as[(r0 + 8) * AS + kk + 2 * tq + 8]);
        }
#pragma unroll
        for (int nt = 0; nt < NT; nt++) {
          const int c0 = wn + nt * 8 + gq;
          b[nt][0] = pack_bf16(bs[(kk + 2 * tq) * BS + c0], bs[(kk + 2 * tq + 1) * BS + c0]);
          b[nt][1] = pack_bf16(bs[(kk + 2 * tq + 8) * BS + c0], bs[(kk + 2 * tq + 9) * BS + c0]);
        }
#pragma unroll
        for (int mt = 0; mt < MT; mt++)
#pragma unroll
          for (int nt = 0; nt < NT; nt++) mma_bf16(acc[mt][nt], a[mt], b[nt]);
      }
    }
    if (kt + 1 < KT) store(buf ^ 1);
    __syncthreads();
  }

  double cscale = 1.0;
  if (EPI == EPI_ACCUM && g.cmax) cscale = *g.cmax;
#pragma unroll
  for (int mt = 0; mt < MT; mt++)
#pragma unroll
    for (int nt = 0; nt < NT; nt++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int r = m0 + wm + mt * 16 + gq + 8 * h;
        if (r >= g.M) continue;
#pragma unroll
        for (int q = 0; q < 2; q++) {
          const int c = n0 + wn + nt * 8 + 2 * tq + q;
          if (c >= g.N) continue;
          double v = (double)acc[mt][nt][2 * h + q];
          TC* dst = g.C + (size_t)r * g.ldc + c;
          if constexpr (EPI == EPI_DIVIDE) {
            const double d = g.alpha + g.bx * g.lx[c] + g.by * g.ly[r];
            v = fabs(d) <= g.null_tol ? 0.0 : v / d;
          }
          if constexpr (EPI == EPI_ACCUM) {
            *dst += v * cscale;
          } else {
            if constexpr (sizeof(TC) == 8)
              *dst = v;
            else if constexpr (sizeof(TC) == 4)
              *dst = (float)v;
            else
              *dst = __float2bfloat16_rn((float)v);
          }
        }
      }
}

// ---------------------------------------------------------------------------
// FP64 products: multi-stage cp.async pipeline (16-byte copies with zero fill;
// 8-byte ones held the products at a third of the FP64 rate), BM x BN block tile of WM x WN warps, each warp
// (BM/WM) x (BN/WN) in m16n8 MMA tiles.
template <int BM_, int BN_, int WM_, int WN_, int ST_, int BK_ = 16>
struct DCfg {
  static constexpr int BM = BM_, BN = BN_, WM = WM_, WN = WN_, ST = ST_;
  static constexpr int BK = BK_, AS = BK + 4, BS = BN + 8;
  static constexpr int THREADS = WM * WN * 32;
  static constexpr int MT = BM / WM / 16, NT = BN / WN / 8;
  static constexpr int A_ELEMS = BM * AS, B_ELEMS = BK * BS;
  static constexpr size_t SMEM = (size_t)ST * (A_ELEMS + B_ELEMS) * sizeof(double);
};

// Epilogues of the FP64 products. D_FIRST stores as D_STORE and reads its A
// (rows of any pitch and alignment) by 8-byte copies.
enum { D_STORE = 0, D_FIRST, D_DIVIDE, D_FINISH };

__device__ __forceinline__ void cp_async8(void* smem, const void* gmem, bool valid) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(sa), "l"(gmem),
               "r"(valid ? 8 : 0));
}
// Copies n (0, 1 or 2) doubles and zeros for the rest of 16 bytes.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, int n) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(gmem), "r"(8 * n));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// The output tile of a block and the operands it multiplies: A[row * lda + k]
// and B[k * ldb + column] for k < K, rows below m_end, columns below n_end; a
// block of threads works inside one part (even or odd) of either direction.
struct DTile {
  const double *A, *B;
  int m0, n0, m_end, n_end, K, lda, ldb;
};
template <int BM, int BN>
__device__ __forceinline__ DTile tile_of(const FdmProduct& g) {
  const FoldDir &x = g.x, &y = g.y;
  const int nt = (x.ge + BN - 1) / BN, mt = (y.ge + BM - 1) / BM;
  const bool xo = (int)blockIdx.x >= nt, yo = (int)blockIdx.y >= mt;
  DTile t;
  t.n0 = xo ? x.os + ((int)blockIdx.x - nt) * BN : (int)blockIdx.x * BN;
  t.m0 = yo ? y.os + ((int)blockIdx.y - mt) * BM : (int)blockIdx.y * BM;
  t.n_end = xo ? x.os + x.go : x.ge;
  t.m_end = yo ? y.os + y.go : y.ge;
  t.lda = g.lda;
  t.ldb = x.len;
  t.A = g.A;
  t.B = g.B;
  if (g.which == FDM_FACTOR_B) {
    t.K = xo ? x.go : x.ge;
    t.ldb = xo ? x.len - x.os : x.os;
    if (xo) {
      t.A += x.os;
      t.B += (ptrdiff_t)x.ge * x.os - x.os;
    }
  } else {
    t.K = yo ? y.go : y.ge;
    t.lda = yo ? y.len - y.os : y.os;
    if (yo) {
      t.A += (ptrdiff_t)y.ge * y.os - (ptrdiff_t)y.os * t.lda;
      t.B += (ptrdiff_t)y.os * t.ldb;
    }
  }
  return t;
}
template <int BM, int BN>
dim3 tile_grid(const FdmProduct& g) {
  auto cut = [](const FoldDir& d, int b) { return (d.ge + b - 1) / b + (d.go + b - 1) / b; };
  return dim3(cut(g.x, BN), cut(g.y, BM));
}

// A stage's operands in 16-byte copies (two values; one and a zero at an odd
// end, zeros beyond).
template <class C, int EPI>
__device__ __forceinline__ void load_stage(const FdmProduct& g, const DTile& t, int k0, double* as,
                                           double* bs) {
  constexpr int AC = C::BK / 2, BC = C::BN / 2;
  static_assert(C::BM * AC % C::THREADS == 0 && C::BK * BC % C::THREADS == 0 && C::AS % 2 == 0 &&
                    C::BS % 2 == 0, "stage copies");
#pragma unroll
  for (int e = 0; e < C::BM * AC / C::THREADS; e++) {
    const int q = threadIdx.x + e * C::THREADS, row = q / AC, col = q % AC * 2;
    const int gr = t.m0 + row, gc = k0 + col;
    const int n = gr < t.m_end ? min(2, t.K - gc) : 0;
    if constexpr (EPI == D_FIRST) {
      const double* src = t.A + (ptrdiff_t)gr * t.lda + gc;
      cp_async8(as + row * C::AS + col, n > 0 ? src : g.A, n > 0);
      cp_async8(as + row * C::AS + col + 1, n > 1 ? src + 1 : g.A, n > 1);
    } else {
      cp_async16(as + row * C::AS + col, n > 0 ? t.A + (ptrdiff_t)gr * t.lda + gc : g.A, max(n, 0));
    }
  }
#pragma unroll
  for (int e = 0; e < C::BK * BC / C::THREADS; e++) {
    const int q = threadIdx.x + e * C::THREADS, row = q / BC, col = q % BC * 2;
    const int gr = k0 + row, gc = t.n0 + col;
    const int n = gr < t.K ? min(2, t.n_end - gc) : 0;
    cp_async16(bs + row * C::BS + col, n > 0 ? t.B + (ptrdiff_t)gr * t.ldb + gc : g.B, max(n, 0));
  }
}

// The operands of D_FINISH's low modes that one thread loads, when the kernel
// starts (they do not depend on the product), so that their latency hides
// behind the main loop: one zlow entry, its share of the tile's rows of low_y,
// and low_x of the output column whose entries of U it forms (entries tid,
// tid + THREADS, ... of the 8 x BN block, all in column tid % BN).
template <class C>
struct LowRegs {
  static constexpr int L = kFdmLow;
  static_assert(C::THREADS >= L * L && C::BM * L % C::THREADS == 0, "low modes' thread map");
  static constexpr int AL = C::BM * L / C::THREADS;
  // doubles in shared memory: zlow, low_y's rows, U = zlow low_x^T as hi and lo
  enum { SIZE = L * L + C::BM * L + 2 * L * C::BN };
  double z, al[AL], ex[L];

  __device__ __forceinline__ void load(const FdmProduct& g, const DTile& t) {
    const int tid = threadIdx.x, gc = t.n0 + tid % C::BN;
    z = tid < L * L ? g.zlow[tid] : 0.0;
#pragma unroll
    for (int q = 0; q < AL; q++) {
      const int e = tid + q * C::THREADS, gr = t.m0 + e / L;
      al[q] = gr < t.m_end ? g.low_y[(size_t)gr * L + e % L] : 0.0;
    }
#pragma unroll
    for (int b = 0; b < L; b++) ex[b] = gc < t.n_end ? g.low_x[(size_t)gc * L + b] : 0.0;
  }
  // To shared memory, and U formed there; ends with the block synchronised.
  __device__ __forceinline__ void stage(double* sm) const {
    static_assert(C::THREADS % C::BN == 0, "low modes' thread map");
    const int tid = threadIdx.x, c = tid % C::BN;
    double *al_s = sm + L * L, *uh = al_s + C::BM * L, *ul = uh + L * C::BN;
    if (tid < L * L) sm[tid] = z;
#pragma unroll
    for (int q = 0; q < AL; q++) al_s[tid + q * C::THREADS] = al[q];
    __syncthreads();
#pragma unroll
    for (int q = 0; q < L * C::BN / C::THREADS; q++) {
      const int a = (tid + q * C::THREADS) / C::BN;
      double h = 0.0, l = 0.0;
#pragma unroll
      for (int b = 0; b < L; b++) dd_fma(h, l, sm[a * L + b], ex[b]);
      uh[a * C::BN + c] = h;
      ul[a * C::BN + c] = l;
    }
    __syncthreads();
  }
  // v, the low modes and the old value (accumulate) at tile row r, column c.
  static __device__ __forceinline__ double add(const double* sm, int r, int c, double v, double old) {
    const double *al_s = sm + L * L + r * L, *uh = sm + L * L + C::BM * L, *ul = uh + L * C::BN;
    double h = 0.0, l = 0.0;
#pragma unroll
    for (int a = 0; a < L; a++) {
      dd_fma(h, l, al_s[a], uh[a * C::BN + c]);
      l = fma(al_s[a], ul[a * C::BN + c], l);
    }
    dd_add(h, l, v);
    dd_add(h, l, old);
    return h + l;
  }
};

// v, the product's output at (row, column), as the epilogue stores it.
template <class C, int EPI>
__device__ __forceinline__ void store_out(const FdmProduct& g, const DTile& t, const double* low,
                                          bool closed, int row, int col, double v) {
  double* dst = g.C + (size_t)row * g.ldc + col;
  if constexpr (EPI == D_DIVIDE) {
    const double d = g.alpha + g.bx * g.lx[col] + g.by * g.ly[row];
    v = fabs(d) <= g.null_tol ? 0.0 : v / d;
    const int lr = low_mode(g.low_r, row), lc = low_mode(g.low_c, col);
    if (lr >= 0 && lc >= 0) {
      g.zlow[lr * kFdmLow + lc] = v;
      v = 0.0;
    }
  } else if constexpr (EPI == D_FINISH) {
    const double old = g.accumulate ? *dst : 0.0;
    v = closed ? old : LowRegs<C>::add(low, row - t.m0, col - t.n0, v, old);
  }
  *dst = v;
}

template <class C, int EPI>
__global__ void __launch_bounds__(C::THREADS) fdm_dgemm_kernel(const FdmProduct g) {
  extern __shared__ __align__(16) double dsm[];
  double* As = dsm;
  double* Bs = dsm + C::ST * C::A_ELEMS;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gq = lane >> 2, tq = lane & 3;
  const int wm = (warp / C::WN) * (C::BM / C::WM), wn = (warp % C::WN) * (C::BN / C::WN);
  const DTile t = tile_of<C::BM, C::BN>(g);
  const int m0 = t.m0, n0 = t.n0;
  const int nkt = (t.K + C::BK - 1) / C::BK;
  const bool closed = EPI == D_FINISH && g.gate && *g.gate != 0;
  LowRegs<C> low;
  if constexpr (EPI == D_FINISH) low.load(g, t);

  auto issue = [&](int i) {
    load_stage<C, EPI>(g, t, i * C::BK, As + (i % C::ST) * C::A_ELEMS, Bs + (i % C::ST) * C::B_ELEMS);
  };

  double acc[C::MT][C::NT][4];
#pragma unroll
  for (int i = 0; i < C::MT; i++)
#pragma unroll
    for (int j = 0; j < C::NT; j++)
#pragma unroll
      for (int q = 0; q < 4; q++) acc[i][j][q] = 0.0;

#pragma unroll
  for (int s = 0; s < C::ST - 1; s++) {
    if (s < nkt) issue(s);
    cp_async_commit();
  }
  for (int i = 0; i < nkt; i++) {
    cp_async_wait<C::ST - 2>();
    __syncthreads();
    if (i + C::ST - 1 < nkt) issue(i + C::ST - 1);
    cp_async_commit();
    const double* as = As + (i % C::ST) * C::A_ELEMS;
    const double* bs = Bs + (i % C::ST) * C::B_ELEMS;
#pragma unroll
    for (int kk = 0; kk < C::BK; kk += 8) {
      double a[C::MT][4], b[C::NT][2];
#pragma unroll
      for (int mt = 0; mt < C::MT; mt++) {
        const int r0 = wm + mt * 16 + gq;
        a[mt][0] = as[r0 * C::AS + kk + tq];
        a[mt][1] = as[(r0 + 8) * C::AS + kk + tq];
        a[mt][2] = as[r0 * C::AS + kk + tq + 4];
        a[mt][3] = as[(r0 + 8) * C::AS + kk + tq + 4];
      }
#pragma unroll
      for (int nt = 0; nt < C::NT; nt++) {
        const int c0 = wn + nt * 8 + gq;
        b[nt][0] = bs[(kk + tq) * C::BS + c0];
        b[nt][1] = bs[(kk + tq + 4) * C::BS + c0];
      }
#pragma unroll
      for (int mt = 0; mt < C::MT; mt++)
#pragma unroll
        for (int nt = 0; nt < C::NT; nt++) mma_f64(acc[mt][nt], a[mt], b[nt]);
    }
  }
  cp_async_wait<0>();
  if constexpr (EPI == D_FINISH) {
    static_assert(LowRegs<C>::SIZE * sizeof(double) <= C::SMEM, "low modes exceed the pipeline");
    __syncthreads();  // the pipeline's shared memory is free from here
    low.stage(dsm);
  }
#pragma unroll
  for (int mt = 0; mt < C::MT; mt++)
#pragma unroll
    for (int nt = 0; nt < C::NT; nt++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int r = m0 + wm + mt * 16 + gq + 8 * h;
        if (r >= t.m_end) continue;
#pragma unroll
        for (int q = 0; q < 2; q++) {
          const int c = n0 + wn + nt * 8 + 2 * tq + q;
          if (c < t.n_end) store_out<C, EPI>(g, t, dsm, closed, r, c, acc[mt][nt][2 * h + q]);
        }
      }
}

template <class C, int EPI>
cudaError_t run_d(const FdmProduct& g, cudaStream_t s) {
  if (C::SMEM > 48 * 1024) {
    static bool attr[64] = {};  // per kernel instantiation and device
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!attr[dev]) {
      e = cudaFuncSetAttribute(fdm_dgemm_kernel<C, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)C::SMEM);
      if (e != cudaSuccess) return e;
      attr[dev] = true;
    }
  }
  fdm_dgemm_kernel<C, EPI><<<tile_grid<C::BM, C::BN>(g), C::THREADS, C::SMEM, s>>>(g);
  return cudaGetLastError();
}

// FP64 products split over K inside the block: a 32 x BN output tile per
// block of W warps; stage i holds a (8 W KW)-wide slice of K and warp w
// multiplies its w-th (8 KW)-wide part, so every warp keeps the whole tile's
// 2 NT accumulator fragments (independent MMA chains) and runs 2 NT KW MMAs
// between barriers. At the end the W partial tiles are summed through shared
// memory in warp order (deterministic) and the epilogue is applied.
template <int BN_, int W_, int ST_, int KW_ = 1>
struct KCfg {
  static constexpr int W = W_, ST = ST_, KW = KW_;
  static constexpr int BM = 32, BN = BN_, NT = BN / 8, BK = 8 * W * KW;
  static constexpr int AS = BK + 4, BS = BN + 4, RS = BN + 1;
  static constexpr int THREADS = 32 * W;
  static constexpr int A_ELEMS = BM * AS, B_ELEMS = BK * BS;
  static constexpr int PIPE = ST * (A_ELEMS + B_ELEMS), RED = W * BM * RS;
  static constexpr size_t SMEM = sizeof(double) * (size_t)(PIPE > RED ? PIPE : RED);
};

template <class C, int EPI>
__global__ void __launch_bounds__(C::THREADS) fdm_dgemm_ksplit_kernel(
    const FdmProduct g) {
  extern __shared__ __align__(16) double dsm[];
  double* As = dsm;
  double* Bs = dsm + C::ST * C::A_ELEMS;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gq = lane >> 2, tq = lane & 3;
  const DTile t = tile_of<C::BM, C::BN>(g);
  const int m0 = t.m0, n0 = t.n0;
  const int nkt = (t.K + C::BK - 1) / C::BK;
  const bool closed = EPI == D_FINISH && g.gate && *g.gate != 0;
  LowRegs<C> low;
  if constexpr (EPI == D_FINISH) low.load(g, t);

  auto issue = [&](int i) {
    load_stage<C, EPI>(g, t, i * C::BK, As + (i % C::ST) * C::A_ELEMS, Bs + (i % C::ST) * C::B_ELEMS);
  };

  double acc[2][C::NT][4];
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < C::NT; j++)
#pragma unroll
      for (int q = 0; q < 4; q++) acc[i][j][q] = 0.0;

#pragma unroll
  for (int s = 0; s < C::ST - 1; s++) {
    if (s < nkt) issue(s);
    cp_async_commit();
  }
  for (int i = 0; i < nkt; i++) {
    cp_async_wait<C::ST - 2>();
    __syncthreads();
    if (i + C::ST - 1 < nkt) issue(i + C::ST - 1);
    cp_async_commit();
    const double* as = As + (i % C::ST) * C::A_ELEMS;
    const double* bs = Bs + (i % C::ST) * C::B_ELEMS;
#pragma unroll
    for (int ks = 0; ks < C::KW; ks++) {
      const int kk = (warp * C::KW + ks) * 8;
      double a[2][4], b[C::NT][2];
#pragma unroll
      for (int mt = 0; mt < 2; mt++) {
        const int r0 = mt * 16 + gq;
        a[mt][0] = as[r0 * C::AS + kk + tq];
        a[mt][1] = as[(r0 + 8) * C::AS + kk + tq];
        a[mt][2] = as[r0 * C::AS + kk + tq + 4];
        a[mt][3] = as[(r0 + 8) * C::AS + kk + tq + 4];
      }
#pragma unroll
      for (int nt = 0; nt < C::NT; nt++) {
        const int c0 = nt * 8 + gq;
        b[nt][0] = bs[(kk + tq) * C::BS + c0];
        b[nt][1] = bs[(kk + tq + 4) * C::BS + c0];
      }
#pragma unroll
      for (int mt = 0; mt < 2; mt++)
#pragma unroll
        for (int nt = 0; nt < C::NT; nt++) mma_f64(acc[mt][nt], a[mt], b[nt]);
    }
  }
  cp_async_wait<0>();
  __syncthreads();

  // partial tiles of the W warps, summed in warp order
  double* red = dsm;
#pragma unroll
  for (int mt = 0; mt < 2; mt++)
#pragma unroll
    for (int nt = 0; nt < C::NT; nt++)
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int r = mt * 16 + gq + (q >> 1) * 8, c = nt * 8 + 2 * tq + (q & 1);
        red[(warp * C::BM + r) * C::RS + c] = acc[mt][nt][q];
      }
  if constexpr (EPI == D_FINISH) {
    static_assert((C::RED + LowRegs<C>::SIZE) * sizeof(double) <= C::SMEM, "low modes");
    low.stage(dsm + C::RED);
  }
  __syncthreads();
  for (int e = tid; e < C::BM * C::BN; e += C::THREADS) {
    const int r = e / C::BN, c = e % C::BN;
    if (m0 + r >= t.m_end || n0 + c >= t.n_end) continue;
    double v = red[r * C::RS + c];
#pragma unroll
    for (int w = 1; w < C::W; w++) v += red[(w * C::BM + r) * C::RS + c];
    store_out<C, EPI>(g, t, dsm + C::RED, closed, m0 + r, n0 + c, v);
  }
}

template <class C, int EPI>
cudaError_t run_k(const FdmProduct& g, cudaStream_t s) {
  if (C::SMEM > 48 * 1024) {
    static bool attr[64] = {};  // per kernel instantiation and device
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!attr[dev]) {
      e = cudaFuncSetAttribute(fdm_dgemm_ksplit_kernel<C, EPI>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
      if (e != cudaSuccess) return e;
      attr[dev] = true;
    }
  }
  fdm_dgemm_ksplit_kernel<C, EPI><<<tile_grid<C::BM, C::BN>(g), C::THREADS, C::SMEM, s>>>(g);
  return cudaGetLastError();
}

// Tile shape by problem size: 32 x 32 tiles (four times the blocks) until
// the 64 x 64 grid alone covers the GPU's SMs.
inline bool small_tiles(int M, int N) { return ((M + 63) / 64) * ((N + 63) / 64) < kSms; }

template <int P, class TA, class TB, class TC, int EPI>
cudaError_t run(const GemmArgs<TA, TB, TC>& g, cudaStream_t s) {
  if (g.M <= 0 || g.N <= 0 || g.K <= 0) return cudaErrorInvalidValue;
  if (small_tiles(g.M, g.N)) {
    const dim3 grid((g.N + 31) / 32, (g.M + 31) / 32);
    fdm_gemm_kernel<P, 32, 32, TA, TB, TC, EPI><<<grid, kThreads, 0, s>>>(g);
  } else {
    const dim3 grid((g.N + 63) / 64, (g.M + 63) / 64);
    fdm_gemm_kernel<P, 64, 64, TA, TB, TC, EPI><<<grid, kThreads, 0, s>>>(g);
  }
  return cudaGetLastError();
}

}  // namespace

// prec: 1 TF32 on FP32 data, 2 BF16. Types by role:
//  in:  FP64 for the normalised first product (amax given), else the low type;
//  out: FP64 for accumulate, else the precision's type.
cudaError_t launch_fdm_gemm(int prec, int epi, const void* A, int a_fp64, const void* B, void* C,
                            int c_fp64, int M, int N, int K, int lda, int ldb, int ldc,
                            const double* amax, const double* cmax, const double* lx,
                            const double* ly, double alpha, double bx, double by, double null_tol,
                            cudaStream_t s) {
#define SE_GEMM_ARGS(TA, TB, TC)                                                              \
  GemmArgs<TA, TB, TC> g{(const TA*)A, (const TB*)B, (TC*)C, M, N, K, lda, ldb, ldc, amax, cmax, \
                         lx, ly, alpha, bx, by, null_tol}
  if (prec != 1 && prec != 2) return cudaErrorInvalidValue;  // FP64: launch_fdm_dgemm
  if (prec == 1) {
    if (a_fp64) {
      SE_GEMM_ARGS(double, float, float);
      return run<1, double, float, float, EPI_STORE>(g, s);
    }
    if (c_fp64) {
      SE_GEMM_ARGS(float, float, double);
      return run<1, float, float, double, EPI_ACCUM>(g, s);
    }
    SE_GEMM_ARGS(float, float, float);
    if (epi == EPI_DIVIDE) return run<1, float, float, float, EPI_DIVIDE>(g, s);
    return run<1, float, float, float, EPI_STORE>(g, s);
  }
  typedef __nv_bfloat16 bf;
  if (a_fp64) {
    SE_GEMM_ARGS(double, bf, bf);
    return run<2, double, bf, bf, EPI_STORE>(g, s);
  }
  if (c_fp64) {
    SE_GEMM_ARGS(bf, bf, double);
    return run<2, bf, bf, double, EPI_ACCUM>(g, s);
  }
  SE_GEMM_ARGS(bf, bf, bf);
  if (epi == EPI_DIVIDE) return run<2, bf, bf, bf, EPI_DIVIDE>(g, s);
  return run<2, bf, bf, bf, EPI_STORE>(g, s);
#undef SE_GEMM_ARGS
}

namespace {
template <template <class, int> class Run, class C>
cudaError_t run_epi(const FdmProduct& p, bool wide, cudaStream_t s) {
  if (p.lx) return Run<C, D_DIVIDE>::run(p, s);
  return wide ? Run<C, D_STORE>::run(p, s) : Run<C, D_FIRST>::run(p, s);
}
template <class C, int EPI>
struct RunD {
  static cudaError_t run(const FdmProduct& p, cudaStream_t s) { return run_d<C, EPI>(p, s); }
};
template <class C, int EPI>
struct RunK {
  static cudaError_t run(const FdmProduct& p, cudaStream_t s) { return run_k<C, EPI>(p, s); }
};
}  // namespace

cudaError_t launch_fdm_dgemm(const FdmProduct& p, cudaStream_t s) {
  if (p.x.len <= 0 || p.y.len <= 0 || (p.lx && !p.zlow)) return cudaErrorInvalidValue;
  // 16-byte copies of A: even rows from an aligned base (folded arrays and
  // factors always; the caller's array where it happens to have them)
  const bool wide = p.which == FDM_FACTOR_A ||
                    (p.lda % 2 == 0 && (reinterpret_cast<uintptr_t>(p.A) & 15) == 0);
  typedef DCfg<64, 64, 2, 2, 3> D;
  const bool small = small_tiles(p.y.len, p.x.len);
  if (p.low_y) return small ? run_k<KCfg<32, 4, 3>, D_FINISH>(p, s) : run_d<D, D_FINISH>(p, s);
  if (!small) return run_epi<RunD, D>(p, wide, s);
  // The tile width whose fullest SM multiplies least: a direction's two parts
  // end in partial tiles, and a 301st tile on 148 SMs costs as much as 144
  // more (768 x 383 unknowns, 300 tiles of 32 x 32 20.6 us an x product, 396
  // of 32 x 24 16.1). The 4 stand for a tile's own cost.
  auto load = [&](int bn) {
    const int tiles = ((p.y.ge + 31) / 32 + (p.y.go + 31) / 32) *
                      ((p.x.ge + bn - 1) / bn + (p.x.go + bn - 1) / bn);
    return (tiles + kSms - 1) / kSms * (bn + 4);
  };
  int bn = 32;
  for (int c : {24, 40})
    if (load(c) < load(bn)) bn = c;
  if (bn == 24) return run_epi<RunK, KCfg<24, 4, 3>>(p, wide, s);
  if (bn == 40) return run_epi<RunK, KCfg<40, 4, 3>>(p, wide, s);
  return run_epi<RunK, KCfg<32, 4, 3>>(p, wide, s);
}

}  // namespace seg
