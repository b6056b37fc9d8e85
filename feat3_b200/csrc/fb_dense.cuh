// The small end of the V-cycle as one dense operator.
//
// From the first level of at most kDenseRows rows downwards, the cycle maps the level's right-hand
// side to its correction by a fixed linear operator (damped Jacobi steps, transfers and the direct,
// smoothing or identity coarse solver are linear; the smoothers' skip test, which is absolute, is not, so
// cycles on defects that it could act on run level by level: dense_applies in fb_mg.cu). k_dense_build
// forms it column by column in FP64 when the solver is configured; a cycle then applies it as one
// matrix-vector product (dense_rows) in place of some 2 nu + 3 dependent launches per level, each of
// which costs its latency (2-4 us) for a few KB of work.
// Whole solves with / without it: 2D Q1 129^2 FP64 V(4,4) 0.53 / 0.96 ms, 65^3 FP64 handed over as CSR
// 2.82 / 3.33 ms, 2D Q2 1025^2 on FP16 values 12.0 / 14.0 ms, 513^2 solve and adjoint 4.78 / 6.56 ms, 257^3
// mixed matrix-free 13.26 / 13.84 ms (its coarse cluster then runs one level instead of four); 129^3 FP32
// cycle 0.487 / 0.533 ms. It adds 0.1 to 0.6 ms to a hierarchy's first configuration. In the FP32 and FP16
// forms these levels' matrices enter in FP64 and only the operator is rounded.
#pragma once
#include "fb_sell.cuh"

namespace fb {

// up to 13 MB of FP64 operator: a few microseconds from L2 or HBM
constexpr uint32_t kDenseRows = 1280;
constexpr int kDenseThreads = 512;
constexpr int kDenseMax = 12;

struct DLevel {
  uint32_t n;
  SellView A;            // FP64 values
  CsrView P, R;          // transfers to the next coarser level (not on the last)
  const uint32_t* mask;
  const double* invd;    // omega_J / diag
};

struct DenseArgs {
  DLevel L[kDenseMax];   // L[0] = the level whose operator is formed
  int nlv, nu, coarse;
  double omega;
  const double* cinv;    // inverse of the coarsest filtered system (FB_COARSE_DIRECT), rows of ldc
  uint32_t ldc;
};

// The columns col0 .. col0 + NC - 1 of the operator: the cycle on NC unit vectors, one CTA, all
// vectors in shared memory ([level][rhs, x, y][row][NC]); op is zero before the launch.
template<typename T, int NC>
__global__ void __launch_bounds__(kDenseThreads) k_dense_build(DenseArgs D, T* op, uint32_t ld) {
  extern __shared__ double dsm[];
  const uint32_t col0 = blockIdx.x * NC, tid = threadIdx.x;
  // a Dirichlet entry's column stays zero (half of the 9^3 level's)
  bool inner = false;
  for (uint32_t c = col0; c < col0 + NC && c < D.L[0].n; ++c) inner = inner || !masked(D.L[0].mask, c);
  if (!inner) return;
  const double om = D.omega;
  double* rhs[kDenseMax];
  double* xs[kDenseMax];
  double* ys[kDenseMax];
  double* sol[kDenseMax];
  {
    double* p = dsm;
    for (int l = 0; l < D.nlv; ++l) {
      const size_t s = size_t(D.L[l].n) * NC;
      rhs[l] = p; xs[l] = p + s; ys[l] = p + 2 * s;
      p += 3 * s;
    }
  }
  // A x at a slot row (the thread's column of the NC); empty slots carry column ~0u
  auto product = [&](const DLevel& L, const double* x, uint32_t sr, uint32_t c) {
    const uint32_t ch = sr >> 5, e = L.A.cs[ch] + (sr & 31u), len = L.A.cl[ch];
    const double* val = static_cast<const double*>(L.A.val);
    double s = 0.0;
#pragma unroll 4
    for (uint32_t j = 0; j < len; ++j) {
      const uint32_t cc = __ldg(L.A.col + e + j * 32u);  // an empty slot's value is 0
      s += __ldg(val + e + j * 32u) * x[(cc == 0xffffffffu ? 0u : cc) * NC + c];
    }
    return s;
  };
  auto transfer = [&](const CsrView& A, const double* x, uint32_t row, uint32_t c) {
    const double* val = static_cast<const double*>(A.val);
    const uint32_t end = __ldg(A.rp + row + 1);
    double s = 0.0;
#pragma unroll 4
    for (uint32_t k = __ldg(A.rp + row); k < end; ++k) s += __ldg(val + k) * x[__ldg(A.col + k) * NC + c];
    return s;
  };
  // one pass over the level's slot rows: f(row, column, A x)
  auto each_row = [&](const DLevel& L, const double* x, auto&& f) {
    for (uint32_t i = tid; i < L.n * NC; i += kDenseThreads) {
      const uint32_t sr = i / NC, c = i % NC, row = L.A.perm ? __ldg(L.A.perm + sr) : sr;
      f(row, c, product(L, x, sr, c));
    }
    __syncthreads();
  };
  auto jacobi = [&](const DLevel& L, const double* b, const double* x, double* out) {
    each_row(L, x, [&](uint32_t row, uint32_t c, double s) {
      const size_t i = size_t(row) * NC + c;
      out[i] = masked(L.mask, row) ? x[i] : om * (L.invd[row] * (b[i] - s)) + x[i];
    });
  };
  auto presmooth = [&](int l) {
    const DLevel& L = D.L[l];
    for (uint32_t i = tid; i < L.n * NC; i += kDenseThreads)
      xs[l][i] = masked(L.mask, i / NC) ? 0.0 : om * (L.invd[i / NC] * rhs[l][i]);
    __syncthreads();
    double *cur = xs[l], *oth = ys[l];
    for (int it = 1; it < D.nu; ++it) {
      jacobi(L, rhs[l], cur, oth);
      double* t = cur; cur = oth; oth = t;
    }
    sol[l] = cur;
  };
  for (uint32_t i = tid; i < D.L[0].n * NC; i += kDenseThreads) {
    const uint32_t row = i / NC;
    rhs[0][i] = (row == col0 + i % NC && !masked(D.L[0].mask, row)) ? 1.0 : 0.0;
  }
  __syncthreads();
  for (int l = 0; l + 1 < D.nlv; ++l) {
    const DLevel& L = D.L[l];
    const DLevel& C = D.L[l + 1];
    presmooth(l);
    double* def = sol[l] == xs[l] ? ys[l] : xs[l];
    each_row(L, sol[l], [&](uint32_t row, uint32_t c, double s) {
      const size_t i = size_t(row) * NC + c;
      def[i] = masked(L.mask, row) ? 0.0 : rhs[l][i] - s;
    });
    for (uint32_t i = tid; i < C.n * NC; i += kDenseThreads)
      rhs[l + 1][i] = masked(C.mask, i / NC) ? 0.0 : transfer(L.R, def, i / NC, i % NC);
    __syncthreads();
  }
  {
    const int l = D.nlv - 1;
    const DLevel& L = D.L[l];
    if (D.coarse == FB_COARSE_DIRECT) {
      for (uint32_t i = tid; i < L.n * NC; i += kDenseThreads) {
        const uint32_t row = i / NC, c = i % NC;
        double s = 0.0;
        for (uint32_t j = 0; j < L.n; ++j) s += __ldg(D.cinv + size_t(row) * D.ldc + j) * rhs[l][size_t(j) * NC + c];
        xs[l][i] = s;
      }
      __syncthreads();
      sol[l] = xs[l];
    } else if (D.coarse == FB_COARSE_SMOOTHER) {
      presmooth(l);
    } else {
      for (uint32_t i = tid; i < L.n * NC; i += kDenseThreads) xs[l][i] = masked(L.mask, i / NC) ? 0.0 : rhs[l][i];
      __syncthreads();
      sol[l] = xs[l];
    }
  }
  for (int l = D.nlv - 2; l >= 0; --l) {
    const DLevel& L = D.L[l];
    double *cur = sol[l], *oth = cur == xs[l] ? ys[l] : xs[l];
    for (uint32_t i = tid; i < L.n * NC; i += kDenseThreads)
      if (!masked(L.mask, i / NC)) cur[i] += transfer(L.P, sol[l + 1], i / NC, i % NC);
    __syncthreads();
    for (int it = 0; it < D.nu; ++it) {
      jacobi(L, rhs[l], cur, oth);
      double* t = cur; cur = oth; oth = t;
    }
    sol[l] = cur;
  }
  for (uint32_t i = tid; i < D.L[0].n * NC; i += kDenseThreads)
    if (col0 + i % NC < D.L[0].n) op[size_t(i / NC) * ld + col0 + i % NC] = T(sol[0][i]);
}

// Dense product rows row0, row0 + stride, ... < n by a warp, R rows at a time (their loads in flight
// together); b in shared memory, zeros behind entry n up to ld. 16-byte loads of the
// operator's rows, whose ld is a multiple of 4 with zeros behind column n; summed in FP64, in the same
// order for every caller. out(row, sum) runs in lane 0.
template<int R, typename T, typename Out>
__device__ __forceinline__ void dense_rows(const T* __restrict__ op, uint32_t ld, const T* b, uint32_t n, uint32_t row0,
                                           uint32_t stride, uint32_t lane, Out&& out) {
  constexpr uint32_t NV = 16 / sizeof(T);
  for (uint32_t r = row0; r < n; r += R * stride) {
    double s[R] = {};
#pragma unroll (R > 1 ? 2 : 8)
    for (uint32_t j = lane * NV; j < ld; j += 32 * NV) {
      T a[R][NV], bv[NV];
#pragma unroll
      for (int q = 0; q < R; ++q)
        if (r + q * stride < n)
          *reinterpret_cast<float4*>(a[q]) = __ldg(reinterpret_cast<const float4*>(op + size_t(r + q * stride) * ld + j));
      *reinterpret_cast<float4*>(bv) = *reinterpret_cast<const float4*>(b + j);
#pragma unroll
      for (int q = 0; q < R; ++q)
        if (r + q * stride < n)
#pragma unroll
          for (uint32_t v = 0; v < NV; ++v) s[q] += double(a[q][v]) * double(bv[v]);
    }
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const double t = warp_sum(s[q]);
      if (lane == 0 && r + q * stride < n) out(r + q * stride, t);
    }
  }
}

// dense product x = op b (the coarse direct solve, or the small end of the cycle): one row per warp; b
// staged in shared memory (at most 32 KB: a direct solve of 4096 rows in FP64)
template<typename T>
__global__ void __launch_bounds__(128) k_dense_solve(T* x, const T* __restrict__ op, uint32_t ld, const T* __restrict__ b,
                                                     uint32_t n) {
  extern __shared__ __align__(16) unsigned char dense_sm[];
  T* sb = reinterpret_cast<T*>(dense_sm);
  pdl_wait();
  pdl_trigger();
  for (uint32_t i = threadIdx.x; i < ld; i += 128) sb[i] = i < n ? b[i] : T(0);
  __syncthreads();
  const uint32_t warp = (blockIdx.x * 128 + threadIdx.x) >> 5, nw = gridDim.x * 4;
  dense_rows<1>(op, ld, sb, n, warp, nw, threadIdx.x & 31, [&](uint32_t row, double s) { x[row] = T(s); });
}

}  // namespace fb
