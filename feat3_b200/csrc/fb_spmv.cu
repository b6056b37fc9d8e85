// Sparse matrix-vector products of the operator layer:
//   * CSR  r = b*y + a*A*x   (1 to 32 threads per row, picked from the mean row length)
//   * CSR  r = b*y + a*A^T*x (scatter with FP64/FP32 atomics)
//   * FEAT SELL-C ("ELL") r = b*y + a*A*x (thread per row, chunk-major coalesced streams)
// Each takes 32-bit (IT = uint32_t) or 64-bit (IT = uint64_t, FEAT's default Index) index
// arrays as they are; the 64-bit forms read the caller's arrays directly, no narrowing copy.
#include "fb_sell.cuh"

namespace fb {

// (within 32 registers, 40 for FP32 values with 64-bit indices: 250,000 rows of 27 at random 32 us, 35 with 32)
template<typename T, int G, int P, typename IT>
__global__ void __launch_bounds__(256, sizeof(T) == 4 && sizeof(IT) == 8 ? 6 : 8) k_csr(T* r, T a, const T* __restrict__ x, T b, const T* y,
                                             const T* __restrict__ val, const IT* __restrict__ col,
                                             const IT* __restrict__ rp, uint64_t rows, bool use_y) {
  const uint64_t row = (blockIdx.x * uint64_t(blockDim.x) + threadIdx.x) / G;
  const bool has = row < rows, first = has && threadIdx.x % G == 0;
  T prev(0);
  if (use_y && first) prev = y[row];
  const T sum = csr_rows<G, P, T, T, T>(val, col, x, has ? __ldg(rp + row) : IT(0), has ? __ldg(rp + row + 1) : IT(0));
  if (first) r[row] = use_y ? (sum * a) + (b * prev) : sum * a;
}

template<typename T>
__global__ void k_scale_copy(T* r, const T* y, T b, uint64_t n, bool use_y) {
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n; i += uint64_t(gridDim.x) * blockDim.x)
    r[i] = use_y ? b * y[i] : T(0);
}

template<typename T, typename IT>
__global__ void k_csr_t(T* r, T a, const T* __restrict__ x, const T* __restrict__ val,
                        const IT* __restrict__ col, const IT* __restrict__ rp, uint64_t rows) {
  const uint64_t gid = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
  const uint64_t row = gid / 8;
  const int sub = threadIdx.x % 8;
  if (row >= rows) return;
  const T xa = a * x[row];
  const IT beg = rp[row], end = rp[row + 1];
  if (beg >= end) return;
  // (offsets from the row's start: a position past its end may lie behind the index type's limit)
  for (uint64_t o = sub; o < uint64_t(end - beg); o += 8) {
    const IT k = beg + IT(o);
    atomicAdd(&r[col[k]], val[k] * xa);
  }
}

// FEAT's SELL-C rows, one thread per row; the loads of eight slots are issued together (two memory
// round trips per eight slots). Times over 300 to 400,000 rows of 3 / 9 / 27 entries, C = 8 and 32, against
// one slot at a time: FP32 u32 1.00 / 0.99 / 1.00, FP32 u64 1.00 / 0.89 / 0.77, FP64 u32 0.97 / 0.95 / 0.95,
// FP64 u64 1.02 / 1.02 / 0.85. (The row's chunk found by a 32-bit division or a shift: 1.00 / 0.97 / 1.02, 1.15
// / 1.06 / 0.95, 1.01 / 1.03 / 1.17, 0.96 / 0.97 / 0.94.)
template<typename T, typename IT>
__global__ void __launch_bounds__(256) k_ell(T* r, T a, const T* __restrict__ x, T b, const T* y,
                                             const T* __restrict__ val, const IT* __restrict__ col,
                                             const IT* __restrict__ cs, const IT* __restrict__ cl,
                                             uint32_t C, uint32_t rows, bool use_y) {
  constexpr int U = 8;
  const uint64_t row = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
  if (row >= rows) return;
  const uint64_t c = row / C;
  const IT lane = IT(row % C);
  const IT base = cs[c] + lane, len = cl[c];
  T sum(0);
  IT j = 0;
  for (; j + U <= len; j += U) {
    IT cc[U];
    T vv[U], xx[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const IT k = base + (j + IT(u)) * IT(C);
      cc[u] = col[k];
      vv[u] = val[k];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) xx[u] = x[cc[u]];
#pragma unroll
    for (int u = 0; u < U; ++u) sum += vv[u] * xx[u];
  }
#pragma unroll 4
  for (; j < len; ++j) {
    const IT k = base + j * IT(C);
    sum += val[k] * x[col[k]];
  }
  const T prev = use_y ? y[row] : T(0);
  r[row] = use_y ? (sum * a) + (b * prev) : sum * a;
}

template<typename T, typename IT>
int csr_apply(T* r, T a, const T* x, T b, const T* y, const T* val, const IT* col, const IT* rp,
              uint64_t rows, uint64_t cols, uint64_t nnz, int transposed, cudaStream_t s) {
  const bool use_y = std::fabs(b) >= eps_of<T>();
  const uint64_t nout = transposed ? cols : rows;
  if (nout == 0) return FB_OK;
  if (!r || (use_y && !y) || (rows && (!rp || (nnz && (!val || !col || !x))))) return FB_ERR_INVALID;
  // sizes must fit the index type (rows and columns are indices, nnz a row-pointer value)
  const uint64_t lim = sizeof(IT) == 4 ? 0xffffffffull : ~0ull;
  if (rows > lim || cols > lim || nnz > lim) return FB_ERR_INVALID;
  if (transposed) {
    k_scale_copy<T><<<grid_for(nout, 256) > 16u * kSMs ? 16u * kSMs : grid_for(nout, 256), 256, 0, s>>>(r, y, b, nout, use_y);
    FB_CHECK_LAUNCH();
    if (rows && nnz) {
      k_csr_t<T, IT><<<grid_for(rows * 8, 256), 256, 0, s>>>(r, a, x, val, col, rp, rows);
      FB_CHECK_LAUNCH();
    }
    return FB_OK;
  }
  // Threads per row from the mean row length: about four to seven entries per thread, which loads
  // four at a time (csr_row). Entries of 12 bytes and more (index and value) take twice the threads on
  // long rows. Measured (us, threads per row):
  //   27 entries, 1.03M rows: FP64 u64 82 (8), 90 (4), 127 (16); FP64 u32 72 (8), 75 (4); FP32 u32 58 (4),
  //   75 (8), 135 (16); 16 entries, 1.0M rows, FP64 u64: 60 (4), 68 (8), 82 (2); 9 entries, 1.44M rows,
  //   FP64 u32: 45 (2), 49 (4), 84 (8); 3.4 entries, 2.1M rows, FP32 u32: 17 (1), 33 (2), 51 (4)
  // One entry at a time with 8 threads per row (2 for the last) took 117, 103, 109, 94, 98 and 39 us.
  // The sums per thread (P, csr_row) go by the rounding. FP32 errors against 64 bits over the groups P G, in
  // units of 1e-8: 3D prolongation 2.86 (1), 2.75 (2), 2.74 (4); random rows of 6 entries 4.48 (2), 4.80
  // (4); 2D stencil, 9 entries, 5.03 (2), 5.04 (4), 5.18 (8); 2D restriction, 9, 5.14 (2), 5.03 (4), 4.76
  // (8); random rows of 16 5.56 (4), 5.62 (8), of 27 6.32 (4), 6.04 (8); 3D restriction, 27, 6.46 (4), 6.00 (8).
  const double avg = rows ? double(nnz) / double(rows) : 0.0;
  constexpr bool wide = sizeof(T) + sizeof(IT) >= 12;
  auto launch = [&](auto g, auto p) {
    constexpr int G = decltype(g)::value, P = decltype(p)::value;
    k_csr<T, G, P, IT><<<grid_for(rows * G, 256), 256, 0, s>>>(r, a, x, b, y, val, col, rp, rows, use_y);
  };
  // Few rows: threads enough that most rows are one batch of loads, as long as the matrix is at most some
  // three fillings of the chip with them (one for rows of up to 4 entries). us with / without: 10,000 rows
  // of 7 to 11 entries at random, FP64 u32, 2.13 / 2.89, 2D stencil of 401^2 rows 5.2 / 5.5, 1201^2 (not
  // taken) 45 / 42; 2D Q2 121^2 2.3 / 2.9, 401^2 (not taken) 8.9 / 8.3; 27 entries, FP32 u32, 33^3
  // 3.1 / 3.2, 51^3 6.5 / 6.4; 3D prolongation, FP64 u32, 33^3 2.05 / 2.45, 65^3 (not taken) 4.7 / 4.3.
  using std::integral_constant;
  auto few = [&](uint64_t g) { return rows * g <= (uint64_t(1) << 20); };
  if (avg <= 4.0) {
    if (rows * 2 <= uint64_t(kSMs) * 2048) launch(integral_constant<int, 2>(), integral_constant<int, 1>());
    else launch(integral_constant<int, 1>(), integral_constant<int, 2>());
  } else if (avg <= 8.0) {
    if (avg > 6.0 && few(4)) launch(integral_constant<int, 4>(), integral_constant<int, 1>());
    else launch(integral_constant<int, 2>(), integral_constant<int, 1>());
  } else if (avg <= 12.0) {
    if (few(4)) launch(integral_constant<int, 4>(), integral_constant<int, 1>());
    else launch(integral_constant<int, 2>(), integral_constant<int, 2>());
  } else if (avg <= 20.0) {
    if (few(8)) launch(integral_constant<int, 8>(), integral_constant<int, 1>());
    else launch(integral_constant<int, 4>(), integral_constant<int, 1>());
  } else if (avg <= 32.0) {
    if (wide || few(8)) launch(integral_constant<int, 8>(), integral_constant<int, 1>());
    else launch(integral_constant<int, 4>(), integral_constant<int, 2>());
  } else if (avg <= 64.0) {
    if (wide || few(16)) launch(integral_constant<int, 16>(), integral_constant<int, 1>());
    else launch(integral_constant<int, 8>(), integral_constant<int, 2>());
  } else {
    launch(integral_constant<int, 32>(), integral_constant<int, 1>());
  }
  FB_CHECK_LAUNCH();
  return FB_OK;
}

template<typename T, typename IT>
int ell_apply(T* r, T a, const T* x, T b, const T* y, const T* val, const IT* col, const IT* cs,
              const IT* cl, uint64_t C, uint64_t rows, cudaStream_t s) {
  const bool use_y = std::fabs(b) >= eps_of<T>();
  if (rows == 0) return FB_OK;
  if (!r || (use_y && !y) || !val || !col || !cs || !cl || !x || C == 0 || C > 1024 || rows > 0xffffffffull)
    return FB_ERR_INVALID;
  k_ell<T, IT><<<grid_for(rows, 256), 256, 0, s>>>(r, a, x, b, y, val, col, cs, cl, uint32_t(C), uint32_t(rows), use_y);
  FB_CHECK_LAUNCH();
  return FB_OK;
}

template<typename T, typename IT>
__global__ void k_diag_csr(T* d, const T* __restrict__ val, const IT* __restrict__ col,
                           const IT* __restrict__ rp, uint64_t rows) {
  const uint64_t row = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
  if (row >= rows) return;
  T v(0);
  for (IT k = rp[row]; k < rp[row + 1]; ++k)
    if (col[k] == row) { v = val[k]; break; }
  d[row] = v;
}

template<typename T, typename IT>
__global__ void k_diag_ell(T* d, const T* __restrict__ val, const IT* __restrict__ col,
                           const IT* __restrict__ cs, const IT* __restrict__ cl, uint32_t C, uint64_t rows) {
  const uint64_t row = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
  if (row >= rows) return;
  const uint64_t c = row / C;
  const IT base = cs[c] + IT(row % C);
  T v(0);
  for (IT j = 0; j < cl[c]; ++j) {
    const IT k = base + j * IT(C);
    if (col[k] == row && val[k] != T(0)) { v = val[k]; break; }
  }
  d[row] = v;
}

template<typename T, typename IT>
int diag_csr(T* d, const T* val, const IT* col, const IT* rp, uint64_t rows, cudaStream_t s) {
  if (rows == 0) return FB_OK;
  if (!d || !val || !col || !rp) return FB_ERR_INVALID;
  k_diag_csr<T, IT><<<grid_for(rows, 256), 256, 0, s>>>(d, val, col, rp, rows);
  FB_CHECK_LAUNCH();
  return FB_OK;
}

template<typename T, typename IT>
int diag_ell(T* d, const T* val, const IT* col, const IT* cs, const IT* cl, uint64_t C, uint64_t rows,
             cudaStream_t s) {
  if (rows == 0) return FB_OK;
  if (!d || !val || !col || !cs || !cl || C == 0 || C > 1024) return FB_ERR_INVALID;
  k_diag_ell<T, IT><<<grid_for(rows, 256), 256, 0, s>>>(d, val, col, cs, cl, uint32_t(C), rows);
  FB_CHECK_LAUNCH();
  return FB_OK;
}

}  // namespace fb

using namespace fb;
#define ST(s) ((cudaStream_t)(s))

extern "C" {

int fb_csr_apply_f64(double* r, double a, const double* x, double b, const double* y, const double* val,
                     const uint32_t* col, const uint32_t* rp, uint64_t rows, uint64_t cols, uint64_t nnz,
                     int transposed, fb_stream_t s) {
  return csr_apply<double, uint32_t>(r, a, x, b, y, val, col, rp, rows, cols, nnz, transposed, ST(s));
}
int fb_csr_apply_f32(float* r, float a, const float* x, float b, const float* y, const float* val,
                     const uint32_t* col, const uint32_t* rp, uint64_t rows, uint64_t cols, uint64_t nnz,
                     int transposed, fb_stream_t s) {
  return csr_apply<float, uint32_t>(r, a, x, b, y, val, col, rp, rows, cols, nnz, transposed, ST(s));
}
int fb_csr_apply_f64_u64(double* r, double a, const double* x, double b, const double* y, const double* val,
                         const uint64_t* col, const uint64_t* rp, uint64_t rows, uint64_t cols, uint64_t nnz,
                         int transposed, fb_stream_t s) {
  return csr_apply<double, uint64_t>(r, a, x, b, y, val, col, rp, rows, cols, nnz, transposed, ST(s));
}
int fb_csr_apply_f32_u64(float* r, float a, const float* x, float b, const float* y, const float* val,
                         const uint64_t* col, const uint64_t* rp, uint64_t rows, uint64_t cols, uint64_t nnz,
                         int transposed, fb_stream_t s) {
  return csr_apply<float, uint64_t>(r, a, x, b, y, val, col, rp, rows, cols, nnz, transposed, ST(s));
}
int fb_ell_apply_f64(double* r, double a, const double* x, double b, const double* y, const double* val,
                     const uint32_t* col, const uint32_t* cs, const uint32_t* cl, uint64_t C, uint64_t rows,
                     fb_stream_t s) {
  return ell_apply<double, uint32_t>(r, a, x, b, y, val, col, cs, cl, C, rows, ST(s));
}
int fb_ell_apply_f32(float* r, float a, const float* x, float b, const float* y, const float* val,
                     const uint32_t* col, const uint32_t* cs, const uint32_t* cl, uint64_t C, uint64_t rows,
                     fb_stream_t s) {
  return ell_apply<float, uint32_t>(r, a, x, b, y, val, col, cs, cl, C, rows, ST(s));
}
int fb_ell_apply_f64_u64(double* r, double a, const double* x, double b, const double* y, const double* val,
                         const uint64_t* col, const uint64_t* cs, const uint64_t* cl, uint64_t C, uint64_t rows,
                         fb_stream_t s) {
  return ell_apply<double, uint64_t>(r, a, x, b, y, val, col, cs, cl, C, rows, ST(s));
}
int fb_ell_apply_f32_u64(float* r, float a, const float* x, float b, const float* y, const float* val,
                         const uint64_t* col, const uint64_t* cs, const uint64_t* cl, uint64_t C, uint64_t rows,
                         fb_stream_t s) {
  return ell_apply<float, uint64_t>(r, a, x, b, y, val, col, cs, cl, C, rows, ST(s));
}
int fb_diagonal_csr_f64(double* d, const double* val, const uint32_t* col, const uint32_t* rp, uint64_t rows,
                        fb_stream_t s) {
  return diag_csr<double, uint32_t>(d, val, col, rp, rows, ST(s));
}
int fb_diagonal_csr_f32(float* d, const float* val, const uint32_t* col, const uint32_t* rp, uint64_t rows,
                        fb_stream_t s) {
  return diag_csr<float, uint32_t>(d, val, col, rp, rows, ST(s));
}
int fb_diagonal_csr_f64_u64(double* d, const double* val, const uint64_t* col, const uint64_t* rp, uint64_t rows,
                            fb_stream_t s) {
  return diag_csr<double, uint64_t>(d, val, col, rp, rows, ST(s));
}
int fb_diagonal_csr_f32_u64(float* d, const float* val, const uint64_t* col, const uint64_t* rp, uint64_t rows,
                            fb_stream_t s) {
  return diag_csr<float, uint64_t>(d, val, col, rp, rows, ST(s));
}
int fb_diagonal_ell_f64(double* d, const double* val, const uint32_t* col, const uint32_t* cs, const uint32_t* cl,
                        uint64_t C, uint64_t rows, fb_stream_t s) {
  return diag_ell<double, uint32_t>(d, val, col, cs, cl, C, rows, ST(s));
}
int fb_diagonal_ell_f32(float* d, const float* val, const uint32_t* col, const uint32_t* cs, const uint32_t* cl,
                        uint64_t C, uint64_t rows, fb_stream_t s) {
  return diag_ell<float, uint32_t>(d, val, col, cs, cl, C, rows, ST(s));
}
int fb_diagonal_ell_f64_u64(double* d, const double* val, const uint64_t* col, const uint64_t* cs, const uint64_t* cl,
                            uint64_t C, uint64_t rows, fb_stream_t s) {
  return diag_ell<double, uint64_t>(d, val, col, cs, cl, C, rows, ST(s));
}
int fb_diagonal_ell_f32_u64(float* d, const float* val, const uint64_t* col, const uint64_t* cs, const uint64_t* cl,
                            uint64_t C, uint64_t rows, fb_stream_t s) {
  return diag_ell<float, uint64_t>(d, val, col, cs, cl, C, rows, ST(s));
}

}  // extern "C"
