// Vector kernels of the operator layer: axpy, dot, norm2, component product/invert,
// scale, unit filter, precision conversion, fill. HBM-bound; grid-stride loops with
// 16-byte accesses for aligned vectors beyond the L2.
#include "fb_common.cuh"

#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <vector>

namespace fb {

// ------------------------------------------------------------------ workspace (per device)
namespace {
std::mutex g_ws_mtx;
std::vector<Workspace*> g_ws;  // indexed by device ordinal
}

int workspace_get(Workspace** out) {
  int dev = 0;
  FB_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(g_ws_mtx);
  if ((int)g_ws.size() <= dev) g_ws.resize(dev + 1, nullptr);
  if (!g_ws[dev]) {
    Workspace* w = new Workspace();
    if (cudaMalloc(&w->partials, sizeof(double) * kRedBlocks) != cudaSuccess ||
        cudaMalloc(&w->counter, sizeof(unsigned) * 8) != cudaSuccess ||
        cudaMallocHost(&w->host_result, sizeof(double) * 8) != cudaSuccess) {
      delete w;
      return FB_ERR_ALLOC;
    }
    // one-time initialisation, complete before any stream (blocking or not) can use the counter
    if (cudaMemset(w->counter, 0, sizeof(unsigned) * 8) != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess)
      return FB_ERR_CUDA;
    g_ws[dev] = w;
  }
  *out = g_ws[dev];
  return FB_OK;
}

bool debug_enabled() {
  static int on = -1;
  if (on < 0) { const char* e = std::getenv("FB_DEBUG"); on = (e && e[0] == '1') ? 1 : 0; }
  return on == 1;
}

bool pdl_enabled() {
  static int on = -1;
  if (on < 0) { const char* e = std::getenv("FB_PDL"); on = (e && e[0] == '1') ? 1 : 0; }
  return on == 1;
}

bool check_enabled() {
  static int on = -1;
  if (on < 0) { const char* e = std::getenv("FB_CHECK"); on = ((e && e[0] == '1') || debug_enabled()) ? 1 : 0; }
  return on == 1;
}

cudaError_t debug_sync(cudaStream_t s, const char* file, int line) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &cs) == cudaSuccess && cs != cudaStreamCaptureStatusNone) return cudaSuccess;
  cudaError_t e = cudaStreamSynchronize(s);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) std::fprintf(stderr, "feat3_b200: %s after the launch at %s:%d\n", cudaGetErrorString(e), file, line);
  return e;
}

void debug_report(cudaError_t e, const char* what, const char* file, int line) {
  std::fprintf(stderr, "feat3_b200: %s returned %s at %s:%d\n", what, cudaGetErrorString(e), file, line);
}

// ------------------------------------------------------------------ elementwise kernels
// r = f(x, y) element by element: 16-byte accesses, two in flight per thread and vector (VEC), or one
// value at a time. An element is read before it is written by the same thread, so r may be x or y.
// Bound by its streams: while the L2 holds them, one value at a time is faster. axpy in us, 16-byte accesses
// against one value: FP32, 1.5 / 4 / 6 / 17 million values 3.8 / 5.4 / 7.1 / 31.9 against 3.2 / 5.5 / 7.9 /
// 45.1, FP64 5.7 / 14.7 / 25.5 / 63.0 against 4.0 / 10.8 / 24.9 / 66.9 (12 million 45.8 against 47.8); scale,
// one vector less: FP32 3.1 / 4.7 / 5.9 / 23.3 against 3.0 / 5.1 / 7.0 / 38.5, FP64 4.2 / 7.1 / 12.7 / 44.0
// against 3.6 / 7.5 / 12.7 / 54.5.
template<typename T, typename F, int NIN, bool VEC>
__global__ void __launch_bounds__(256) k_ew(T* r, const T* x, const T* y, uint64_t n, F f) {
  constexpr int NV = VEC ? 16 / sizeof(T) : 1, U = VEC ? 2 : 1;
  struct alignas(VEC ? 16 : sizeof(T)) Pack { T v[NV]; };
  const Pack* px = reinterpret_cast<const Pack*>(x);
  const Pack* py = reinterpret_cast<const Pack*>(y);
  Pack* pr = reinterpret_cast<Pack*>(r);
  const uint64_t np = n / NV, stride = uint64_t(gridDim.x) * blockDim.x;
  const uint64_t tid = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
  auto apply = [&](const Pack& a, const Pack& b) {
    Pack o;
#pragma unroll
    for (int v = 0; v < NV; ++v) o.v[v] = f(a.v[v], b.v[v]);
    return o;
  };
  uint64_t i = tid;
  for (; i + (U - 1) * stride < np; i += U * stride) {
    Pack a[U], b[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      a[u] = px[i + u * stride];
      b[u] = NIN > 1 ? py[i + u * stride] : a[u];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) pr[i + u * stride] = apply(a[u], b[u]);
  }
  for (; i < np; i += stride) pr[i] = apply(px[i], NIN > 1 ? py[i] : px[i]);
  if (VEC && tid < n % NV) {
    const uint64_t k = np * NV + tid;
    r[k] = f(x[k], NIN > 1 ? y[k] : x[k]);
  }
}

template<typename T> struct OpAxpy { T a; __device__ T operator()(T x, T y) const { return a * x + y; } };
template<typename T> struct OpCopy { __device__ T operator()(T x, T) const { return x; } };
template<typename T> struct OpProd { __device__ T operator()(T x, T y) const { return x * y; } };
template<typename T> struct OpInv { T s; __device__ T operator()(T x, T) const { return s / x; } };
template<typename T> struct OpScale { T s; __device__ T operator()(T x, T) const { return s * x; } };

template<typename T>
__global__ void k_set(T* __restrict__ r, T v, uint64_t n) {
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n; i += uint64_t(gridDim.x) * blockDim.x)
    r[i] = v;
}
template<typename D, typename S>
__global__ void k_convert(D* __restrict__ r, const S* __restrict__ x, uint64_t n) {
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n; i += uint64_t(gridDim.x) * blockDim.x)
    r[i] = D(x[i]);
}
template<typename T, typename IT>
__global__ void k_filter_rhs(T* __restrict__ v, const T* __restrict__ sv, const IT* __restrict__ idx, uint64_t ue) {
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < ue; i += uint64_t(gridDim.x) * blockDim.x)
    v[idx[i]] = sv[i];
}
template<typename T, typename IT>
__global__ void k_filter_def(T* __restrict__ v, const IT* __restrict__ idx, uint64_t ue) {
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < ue; i += uint64_t(gridDim.x) * blockDim.x)
    v[idx[i]] = T(0);
}

// dot / sum of squares, FP64 accumulation, deterministic finish. Four loads of each vector in flight per
// thread, of 16 bytes (VEC) or of one value. dot in us, 16-byte loads against one value: FP64, 1.5 / 4 / 17
// million values 6.0 / 8.7 / 46.2 against 5.7 / 8.2 / 41.8, FP32 5.9 / 7.4 / 26.2 against 5.2 / 7.1 / 28.2 (6
// million 8.1 against 8.6); norm: FP64 5.6 / 7.0 / 24.7 against 5.1 / 6.6 / 26.4 (12 million 12.1 against 14.9),
// FP32 5.2 / 6.0 / 9.6 against 5.0 / 6.3 / 10.9. One value at a time and none in flight: FP64, 17 million, 69
// (dot) and 57 (norm). So the FP64 dot never takes 16 bytes.
template<typename T, bool SQUARE, bool SQRT, bool VEC>
__global__ void __launch_bounds__(kRedThreads) k_dot(const T* __restrict__ x, const T* __restrict__ y, uint64_t n,
                                                     double* ws, unsigned* counter, double* out) {
  __shared__ double sh[kRedThreads / 32];
  constexpr int NV = VEC ? 16 / sizeof(T) : 1, U = 4;
  struct alignas(VEC ? 16 : sizeof(T)) Pack { T v[NV]; };
  const Pack* px = reinterpret_cast<const Pack*>(x);
  const Pack* py = reinterpret_cast<const Pack*>(y);
  const uint64_t np = n / NV, stride = uint64_t(gridDim.x) * kRedThreads;
  const uint64_t tid = blockIdx.x * uint64_t(kRedThreads) + threadIdx.x;
  double acc[NV] = {};
  auto add = [&](const Pack& a, const Pack& b) {
#pragma unroll
    for (int v = 0; v < NV; ++v) acc[v] += double(a.v[v]) * double(b.v[v]);
  };
  uint64_t i = tid;
  for (; i + (U - 1) * stride < np; i += U * stride) {
    Pack a[U], b[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      a[u] = px[i + u * stride];
      if (!SQUARE) b[u] = py[i + u * stride];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) add(a[u], SQUARE ? a[u] : b[u]);
  }
  for (; i < np; i += stride) add(px[i], SQUARE ? px[i] : py[i]);
  if (VEC && tid < n % NV) {
    const uint64_t k = np * NV + tid;
    acc[0] += double(x[k]) * double(SQUARE ? x[k] : y[k]);
  }
  double sum = acc[0];
#pragma unroll
  for (int v = 1; v < NV; ++v) sum += acc[v];
  double blk = block_sum<kRedThreads>(sum, sh);
  reduce_finish<kRedThreads>(blk, ws, counter, out, sh, SQRT);
}

constexpr int kEW = 256;
inline unsigned ew_grid(uint64_t n) {
  unsigned g = grid_for(n, kEW);
  return g > 16u * kSMs ? 16u * kSMs : g;
}

// wide accesses: all vectors 16-byte aligned and their streams together longer than `mb` MB, from where on
// they were faster (figures at k_ew and k_dot)
inline bool wide_accesses(uintptr_t addresses, uint64_t bytes, uint64_t mb) {
  return (addresses & 15) == 0 && bytes > mb * 1000000u;
}

template<int NIN, typename T, typename F>
int elementwise(T* r, const T* x, const T* y, uint64_t n, F f, cudaStream_t s) {
  if (n == 0) return FB_OK;
  if (!r || !x || (NIN > 1 && !y)) return FB_ERR_INVALID;
  const uintptr_t at = reinterpret_cast<uintptr_t>(r) | reinterpret_cast<uintptr_t>(x) | (NIN > 1 ? reinterpret_cast<uintptr_t>(y) : 0);
  constexpr uint64_t mb = NIN > 1 ? (sizeof(T) == 4 ? 60 : 150) : (sizeof(T) == 4 ? 28 : 90);
  if (wide_accesses(at, n * sizeof(T) * (NIN + 1), mb)) k_ew<T, F, NIN, true><<<ew_grid((n * sizeof(T) + 15) / 16), kEW, 0, s>>>(r, x, y, n, f);
  else k_ew<T, F, NIN, false><<<ew_grid(n), kEW, 0, s>>>(r, x, y, n, f);
  FB_CHECK_LAUNCH();
  return FB_OK;
}

template<typename T>
int axpy(T* r, T a, const T* x, const T* y, uint64_t n, cudaStream_t s) {
  if (n == 0) return FB_OK;
  if (!r || !y || (!x && std::fabs(double(a)) >= double(eps_of<T>()))) return FB_ERR_INVALID;
  if (std::fabs(a) < eps_of<T>()) return r == y ? FB_OK : elementwise<1>(r, y, (const T*)nullptr, n, OpCopy<T>{}, s);
  return elementwise<2>(r, x, y, n, OpAxpy<T>{a}, s);
}

template<typename T, bool SQUARE, bool SQRT>
int reduce(const T* x, const T* y, uint64_t n, double* result, cudaStream_t s) {
  if (!result || (n > 0 && (!x || (!SQUARE && !y)))) return FB_ERR_INVALID;
  Workspace* ws = nullptr;
  FB_TRY(workspace_get(&ws));
  unsigned g = grid_for(n, kRedThreads);
  if (g > unsigned(kRedBlocks)) g = kRedBlocks;
  constexpr uint64_t mb = SQUARE ? (sizeof(T) == 4 ? 10 : 80) : 40;
  const uintptr_t at = reinterpret_cast<uintptr_t>(x) | (SQUARE ? 0 : reinterpret_cast<uintptr_t>(y));
  const bool vec = (SQUARE || sizeof(T) == 4) && wide_accesses(at, n * sizeof(T) * (SQUARE ? 1 : 2), mb);
  if (vec) k_dot<T, SQUARE, SQRT, true><<<g, kRedThreads, 0, s>>>(x, y, n, ws->partials, ws->counter, result);
  else k_dot<T, SQUARE, SQRT, false><<<g, kRedThreads, 0, s>>>(x, y, n, ws->partials, ws->counter, result);
  FB_CHECK_LAUNCH();
  return FB_OK;
}

template<typename T, bool SQUARE, bool SQRT>
int reduce_sync(const T* x, const T* y, uint64_t n, double* host_result, cudaStream_t s) {
  if (!host_result) return FB_ERR_INVALID;
  Workspace* ws = nullptr;
  FB_TRY(workspace_get(&ws));
  // the kernel writes the scalar to the pinned host word itself (no copy behind it)
  FB_TRY((reduce<T, SQUARE, SQRT>(x, y, n, ws->host_result, s)));
  FB_CUDA(cudaStreamSynchronize(s));
  *host_result = *ws->host_result;
  return FB_OK;
}

template<typename K, typename... A>
int launch_ew(K kern, uint64_t n, cudaStream_t s, A... args) {
  if (n == 0) return FB_OK;
  kern<<<ew_grid(n), kEW, 0, s>>>(args...);
  FB_CHECK_LAUNCH();
  return FB_OK;
}

}  // namespace fb

using namespace fb;
#define ST(s) ((cudaStream_t)(s))

extern "C" {

int fb_axpy_f64(double* r, double a, const double* x, const double* y, uint64_t n, fb_stream_t s) { return axpy<double>(r, a, x, y, n, ST(s)); }
int fb_axpy_f32(float* r, float a, const float* x, const float* y, uint64_t n, fb_stream_t s) { return axpy<float>(r, a, x, y, n, ST(s)); }

int fb_dot_f64(const double* x, const double* y, uint64_t n, double* res, fb_stream_t s) { return reduce<double, false, false>(x, y, n, res, ST(s)); }
int fb_dot_f32(const float* x, const float* y, uint64_t n, double* res, fb_stream_t s) { return reduce<float, false, false>(x, y, n, res, ST(s)); }
int fb_dot_f64_sync(const double* x, const double* y, uint64_t n, double* h, fb_stream_t s) { return reduce_sync<double, false, false>(x, y, n, h, ST(s)); }
int fb_dot_f32_sync(const float* x, const float* y, uint64_t n, double* h, fb_stream_t s) { return reduce_sync<float, false, false>(x, y, n, h, ST(s)); }
int fb_norm2_f64(const double* x, uint64_t n, double* res, fb_stream_t s) { return reduce<double, true, true>(x, x, n, res, ST(s)); }
int fb_norm2_f32(const float* x, uint64_t n, double* res, fb_stream_t s) { return reduce<float, true, true>(x, x, n, res, ST(s)); }
int fb_norm2_f64_sync(const double* x, uint64_t n, double* h, fb_stream_t s) { return reduce_sync<double, true, true>(x, x, n, h, ST(s)); }
int fb_norm2_f32_sync(const float* x, uint64_t n, double* h, fb_stream_t s) { return reduce_sync<float, true, true>(x, x, n, h, ST(s)); }

int fb_component_product_f64(double* r, const double* x, const double* y, uint64_t n, fb_stream_t s) {
  return elementwise<2>(r, x, y, n, OpProd<double>{}, ST(s));
}
int fb_component_product_f32(float* r, const float* x, const float* y, uint64_t n, fb_stream_t s) {
  return elementwise<2>(r, x, y, n, OpProd<float>{}, ST(s));
}
int fb_component_invert_f64(double* r, const double* x, double sc, uint64_t n, fb_stream_t s) {
  return elementwise<1>(r, x, (const double*)nullptr, n, OpInv<double>{sc}, ST(s));
}
int fb_component_invert_f32(float* r, const float* x, float sc, uint64_t n, fb_stream_t s) {
  return elementwise<1>(r, x, (const float*)nullptr, n, OpInv<float>{sc}, ST(s));
}
int fb_scale_f64(double* r, const double* x, double sc, uint64_t n, fb_stream_t s) {
  return elementwise<1>(r, x, (const double*)nullptr, n, OpScale<double>{sc}, ST(s));
}
int fb_scale_f32(float* r, const float* x, float sc, uint64_t n, fb_stream_t s) {
  return elementwise<1>(r, x, (const float*)nullptr, n, OpScale<float>{sc}, ST(s));
}
int fb_unit_filter_rhs_f64(double* v, const double* sv, const uint32_t* idx, uint64_t ue, fb_stream_t s) {
  if (ue && (!v || !sv || !idx)) return FB_ERR_INVALID;
  return launch_ew(k_filter_rhs<double, uint32_t>, ue, ST(s), v, sv, idx, ue);
}
int fb_unit_filter_def_f64(double* v, const uint32_t* idx, uint64_t ue, fb_stream_t s) {
  if (ue && (!v || !idx)) return FB_ERR_INVALID;
  return launch_ew(k_filter_def<double, uint32_t>, ue, ST(s), v, idx, ue);
}
int fb_unit_filter_rhs_f32(float* v, const float* sv, const uint32_t* idx, uint64_t ue, fb_stream_t s) {
  if (ue && (!v || !sv || !idx)) return FB_ERR_INVALID;
  return launch_ew(k_filter_rhs<float, uint32_t>, ue, ST(s), v, sv, idx, ue);
}
int fb_unit_filter_def_f32(float* v, const uint32_t* idx, uint64_t ue, fb_stream_t s) {
  if (ue && (!v || !idx)) return FB_ERR_INVALID;
  return launch_ew(k_filter_def<float, uint32_t>, ue, ST(s), v, idx, ue);
}
int fb_unit_filter_rhs_f64_u64(double* v, const double* sv, const uint64_t* idx, uint64_t ue, fb_stream_t s) {
  if (ue && (!v || !sv || !idx)) return FB_ERR_INVALID;
  return launch_ew(k_filter_rhs<double, uint64_t>, ue, ST(s), v, sv, idx, ue);
}
int fb_unit_filter_def_f64_u64(double* v, const uint64_t* idx, uint64_t ue, fb_stream_t s) {
  if (ue && (!v || !idx)) return FB_ERR_INVALID;
  return launch_ew(k_filter_def<double, uint64_t>, ue, ST(s), v, idx, ue);
}
int fb_unit_filter_rhs_f32_u64(float* v, const float* sv, const uint64_t* idx, uint64_t ue, fb_stream_t s) {
  if (ue && (!v || !sv || !idx)) return FB_ERR_INVALID;
  return launch_ew(k_filter_rhs<float, uint64_t>, ue, ST(s), v, sv, idx, ue);
}
int fb_unit_filter_def_f32_u64(float* v, const uint64_t* idx, uint64_t ue, fb_stream_t s) {
  if (ue && (!v || !idx)) return FB_ERR_INVALID;
  return launch_ew(k_filter_def<float, uint64_t>, ue, ST(s), v, idx, ue);
}
int fb_convert_f64_to_f32(float* d, const double* x, uint64_t n, fb_stream_t s) {
  if (n && (!d || !x)) return FB_ERR_INVALID;
  return launch_ew(k_convert<float, double>, n, ST(s), d, x, n);
}
int fb_convert_f32_to_f64(double* d, const float* x, uint64_t n, fb_stream_t s) {
  if (n && (!d || !x)) return FB_ERR_INVALID;
  return launch_ew(k_convert<double, float>, n, ST(s), d, x, n);
}
int fb_set_f64(double* d, double v, uint64_t n, fb_stream_t s) {
  if (n && !d) return FB_ERR_INVALID;
  return launch_ew(k_set<double>, n, ST(s), d, v, n);
}
int fb_set_f32(float* d, float v, uint64_t n, fb_stream_t s) {
  if (n && !d) return FB_ERR_INVALID;
  return launch_ew(k_set<float>, n, ST(s), d, v, n);
}

const char* fb_version(void) { return "feat3_b200 0.1 (sm_100a)"; }

}  // extern "C"
