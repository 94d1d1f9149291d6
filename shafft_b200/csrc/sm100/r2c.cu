// Real-to-complex and complex-to-real transforms (an extension: the
// reference supports C2C / Z2Z only, docs/limitations.dox:51-60).
//
// A real tensor of dims (d_0, ..., d_{n-1}) with an even last length L is
// read as a complex tensor z of dims (d_0, ..., L/2), z[.., j] = x[.., 2j] +
// i x[.., 2j+1], at no cost (the same bytes).  With H = L/2, J the index over
// the other axes and -J its mirror (every other index negated modulo its
// length), forward (R2C):
//   1. the C2C transform of z over every axis (the library's ordinary plan
//      of dims (d_0, ..., H): its specialised passes apply): Z = DFT(z)
//   2. untangle, for k = 0 .. H (Z[J, H] taken as Z[J, 0]):
//        E = (Z[J, k] + conj(Z[-J, H-k])) / 2     (spectrum of the even samples)
//        O = (Z[J, k] - conj(Z[-J, H-k])) / (2i)  (spectrum of the odd samples)
//        X[J, k] = E + w_L^k O
// Backward (C2R) inverts the untangle with the Hermitian extension
// X[J, k + H] = conj(X[-J, H - k]) folded in,
//        Z[J, k] = (X[J, k] + conj(X[-J, H-k])) + i w_L^{-k} (X[J, k] - conj(X[-J, H-k])),
// then runs the backward C2C of z, whose complex output read as reals is the
// unnormalised real inverse.  The R2C output is the first H + 1 frequencies
// of the last axis (the others follow by Hermitian symmetry), the layout FFTW
// and cuFFT use.  Normalisation (`scale`) is fused into the last step.
#include <cuda_runtime.h>
#include <stdarg.h>
#include <stdio.h>

#include <new>
#include <vector>

#include "../../../include/shafft_sm100.h"
#include "butterflies.cuh"
#include "launch.h"

namespace shafft_sm100 {
namespace {

int rfail(int code, const char* fmt, ...) {
  char msg[256];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(msg, sizeof(msg), fmt, ap);
  va_end(ap);
  return report_error(code, msg);
}

// Other axes of the tensor (all but the last): lengths and row-major
// strides, for the mirror index -J.
struct RDims {
  int n;
  int64_t len[16];
  int64_t stride[16];
};

template <typename I>
__device__ __forceinline__ int64_t mirror_row(const RDims& d, I row) {
  int64_t m = 0;
  for (int a = d.n - 1; a >= 0; --a) {
    const I len = (I)d.len[a], q = row / len, j = row - q * len;
    row = q;
    m += (j ? d.len[a] - (int64_t)j : 0) * d.stride[a];
  }
  return m;
}

// The (un)tangle kernels read and write every element once: with a =
// Z[J, k], b = conj(Z[-J, H-k]), E and O of (J, k) also give the mirror,
// X[J, k] = E + w^k O and X[-J, H-k] = conj(E - w^k O).  A group of 2^logG
// lanes (up to a warp, fewer for short rows) takes one row pair (J, -J), J <=
// -J in row order, and kRcUnroll points a lane of it; the other rows are done
// by their partners, so half of the groups leave at once.  Bound by HBM.  The
// pairing and one 32-bit index division a group in place of several 64-bit
// divisions an element took the untangle
// of 256^3 float32 from 66 to 26 us, the tangle from 62 to 27 on B200.
constexpr int kRcUnroll = 4;

// Row pair and first point of this thread (then every 2^logG-th, kRcUnroll of
// them); false: none.
__device__ __forceinline__ bool rc_item(const RDims& d, int64_t rows, int64_t chunks, int logG, int64_t& r,
                                        int64_t& mr, int64_t& k0) {
  const int64_t item = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> logG;
  if (item >= rows * chunks) return false;
  int64_t c;
  if (rows * chunks < ((int64_t)1 << 32)) {
    const uint32_t q = (uint32_t)item / (uint32_t)chunks;
    r = q;
    c = (uint32_t)item - q * (uint32_t)chunks;
    mr = mirror_row<uint32_t>(d, q);
  } else {
    r = item / chunks;
    c = item - r * chunks;
    mr = mirror_row<int64_t>(d, r);
  }
  k0 = ((c * kRcUnroll) << logG) + (threadIdx.x & ((1 << logG) - 1));
  return r <= mr;
}

// forward untangle: Z (rows x H) -> X (rows x (H + 1)), H = L / 2;
// tw[k] = w_L^k (forward sign), k <= H
template <typename T>
__global__ void __launch_bounds__(256)
    k_r2c_untangle(const typename Cx<T>::type* Z, typename Cx<T>::type* X, int64_t rows, int64_t H, int64_t chunks, int logG,
                   const typename Cx<T>::type* tw, T scale, const RDims d) {
  chain_begin();
  using C = typename Cx<T>::type;
  int64_t r, mr, k0;
  if (!rc_item(d, rows, chunks, logG, r, mr, k0)) return;
  const C* zr = Z + r * H;
  const C* zm = Z + mr * H;
  C* xr = X + r * (H + 1);
  C* xm = X + mr * (H + 1);
  C a[kRcUnroll], b[kRcUnroll], w[kRcUnroll];
#pragma unroll
  for (int u = 0; u < kRcUnroll; ++u) {
    const int64_t k = k0 + ((int64_t)u << logG);
    const bool on = k < H;
    a[u] = on ? zr[k] : C{0, 0};
    b[u] = on ? zm[k == 0 ? 0 : H - k] : C{0, 0};
    w[u] = on ? __ldg(tw + k) : C{0, 0};
  }
#pragma unroll
  for (int u = 0; u < kRcUnroll; ++u) {
    const int64_t k = k0 + ((int64_t)u << logG);
    if (k >= H) continue;
    const C e = C{(a[u].x + b[u].x) * (T)0.5, (a[u].y - b[u].y) * (T)0.5};
    // (a - conj(z)) / (2i) = (a.y + z.y, -(a.x - z.x)) / 2
    const C o = cmul(C{(a[u].y + b[u].y) * (T)0.5, (b[u].x - a[u].x) * (T)0.5}, w[u]);
    // the scale last: one more rounding of the finished value, none inside
    const C p = cscale(cadd(e, o), scale), q = cscale(cconj(csub(e, o)), scale);
    xr[k] = p;
    if (k == 0) xr[H] = cconj(q);  // Z[J, H] is Z[J, 0] and w^H = -1
    if (r != mr) {
      xm[H - k] = q;
      if (k == 0) xm[0] = cconj(p);
    }
  }
}

// backward untangle: X (rows x (H + 1)) -> Z (rows x H): with a = X[J, k], b =
// conj(X[-J, H-k]) (X[J, k + H] by Hermitian symmetry), S = a + b and V = i
// conj(w_L^k) (a - b), Z[J, k] = S + V and Z[-J, H-k] = conj(S - V)
template <typename T>
__global__ void __launch_bounds__(256)
    k_c2r_tangle(const typename Cx<T>::type* X, typename Cx<T>::type* Z, int64_t rows, int64_t H, int64_t chunks, int logG,
                 const typename Cx<T>::type* tw, const RDims d) {
  chain_begin();
  using C = typename Cx<T>::type;
  int64_t r, mr, k0;
  if (!rc_item(d, rows, chunks, logG, r, mr, k0)) return;
  const C* xr = X + r * (H + 1);
  const C* xm = X + mr * (H + 1);
  C* zr = Z + r * H;
  C* zm = Z + mr * H;
  C a[kRcUnroll], b[kRcUnroll], w[kRcUnroll];
#pragma unroll
  for (int u = 0; u < kRcUnroll; ++u) {
    const int64_t k = k0 + ((int64_t)u << logG);
    const bool on = k < H;
    a[u] = on ? xr[k] : C{0, 0};
    b[u] = on ? xm[H - k] : C{0, 0};
    w[u] = on ? __ldg(tw + k) : C{0, 0};
  }
#pragma unroll
  for (int u = 0; u < kRcUnroll; ++u) {
    const int64_t k = k0 + ((int64_t)u << logG);
    if (k >= H) continue;
    const C z = cconj(b[u]);
    const C s = cadd(a[u], z);
    const C wd = cmul(csub(a[u], z), cconj(w[u]));
    const C v = C{-wd.y, wd.x};
    zr[k] = cadd(s, v);
    if (r != mr) {
      if (k != 0) {
        zm[H - k] = cconj(csub(s, v));
      } else {  // Z[-J, 0] of X[-J, 0] and X[J, H]; w^0 = 1
        const C a0 = xm[0], b0 = cconj(xr[H]);
        const C d0 = csub(a0, b0);
        zm[0] = cadd(cadd(a0, b0), C{-d0.y, d0.x});
      }
    }
  }
}

template <typename T>
__global__ void k_r2c_twiddle(typename Cx<T>::type* tw, int64_t L) {
  const int64_t H = L / 2;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k <= H; k += (int64_t)gridDim.x * blockDim.x) {
    double s, c;
    sincospi(-2.0 * (double)k / (double)L, &s, &c);
    tw[k] = typename Cx<T>::type{(T)c, (T)s};
  }
}

unsigned grid_for(int64_t n) {
  const int64_t g = (n + 255) / 256;
  return (unsigned)(g < 148 * 16 ? (g < 1 ? 1 : g) : 148 * 16);
}

// Launch shape over rows of H points (rc_item).
struct RcShape {
  unsigned grid;
  int64_t chunks;
  int logG;
};
RcShape rc_shape(int64_t rows, int64_t H) {
  RcShape s{1, 1, 1};
  while (s.logG < 5 && ((int64_t)kRcUnroll << s.logG) < H) ++s.logG;
  const int64_t step = (int64_t)kRcUnroll << s.logG;
  s.chunks = (H + step - 1) / step;
  s.grid = (unsigned)((rows * s.chunks + (256 >> s.logG) - 1) / (256 >> s.logG));
  return s;
}

}  // namespace
}  // namespace shafft_sm100

using namespace shafft_sm100;

struct shafft_sm100_rplan_s {
  int precision = 0;
  int64_t rows = 0, H = 0;        // rows of the last axis, L / 2
  shafft_sm100_plan full = nullptr;  // C2C over every axis of (..., H)
  RDims dims{};                   // the other axes, for the mirror index
  void* tw = nullptr;             // w_L^k, k <= H
  void* a = nullptr;              // rows x H
};

namespace {

void rplan_free(shafft_sm100_rplan_s* p) {
  if (p->full) shafft_sm100_plan_destroy(p->full);
  if (p->tw) dev_free(p->tw);
  if (p->a) dev_free(p->a);
  delete p;
}

}  // namespace

extern "C" {

int shafft_sm100_rplan_create(shafft_sm100_rplan* out, int ndim, const int64_t* dims, int precision) {
  if (!out || !dims || ndim < 1 || ndim > 16) return rfail(SHAFFT_SM100_EINVAL, "bad real-transform arguments");
  if (precision != 0 && precision != 1) return rfail(SHAFFT_SM100_EINVAL, "bad precision");
  *out = nullptr;
  for (int a = 0; a < ndim; ++a)
    if (dims[a] < 1) return rfail(SHAFFT_SM100_EINVAL, "axis %d has length %lld", a, (long long)dims[a]);
  const int64_t L = dims[ndim - 1];
  if (L % 2) return rfail(SHAFFT_SM100_ENOTSUP, "the last axis (%lld) must have an even length", (long long)L);
  auto* p = new (std::nothrow) shafft_sm100_rplan_s();
  if (!p) return rfail(SHAFFT_SM100_EALLOC, "host allocation failed");
  p->precision = precision;
  p->H = L / 2;
  p->rows = 1;
  p->dims.n = ndim - 1;
  for (int a = ndim - 2; a >= 0; --a) {
    p->dims.len[a] = dims[a];
    p->dims.stride[a] = p->rows;
    p->rows *= dims[a];
  }
  const size_t es = precision ? 16 : 8;
  std::vector<int64_t> half(dims, dims + ndim);
  half[ndim - 1] = p->H;
  int rc = shafft_sm100_plan_create_nd(&p->full, ndim, half.data(), precision);
  if (rc) {
    p->full = nullptr;
    rplan_free(p);
    return rc;
  }
  cudaError_t e = dev_malloc(&p->tw, (size_t)(p->H + 1) * es);
  if (e == cudaSuccess) e = dev_malloc(&p->a, (size_t)(p->rows * p->H) * es);
  if (e != cudaSuccess) {
    cudaGetLastError();
    rplan_free(p);
    return rfail(SHAFFT_SM100_EALLOC, "device allocation for the real transform failed");
  }
  if (precision)
    k_r2c_twiddle<double><<<grid_for(p->H + 1), 256>>>(reinterpret_cast<double2*>(p->tw), L);
  else
    k_r2c_twiddle<float><<<grid_for(p->H + 1), 256>>>(reinterpret_cast<float2*>(p->tw), L);
  e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaStreamSynchronize(nullptr);
  if (e != cudaSuccess) {
    rplan_free(p);
    return rfail(SHAFFT_SM100_ECUDA, "real-transform twiddles: %s", cudaGetErrorString(e));
  }
  *out = p;
  return 0;
}

int shafft_sm100_rplan_destroy(shafft_sm100_rplan p) {
  if (p) rplan_free(p);
  return 0;
}

int64_t shafft_sm100_rplan_spectrum_elements(shafft_sm100_rplan p) {
  return p ? p->rows * (p->H + 1) : 0;
}

int shafft_sm100_execute_r2c(shafft_sm100_rplan p, void* real_in, void* spec_out, double scale, void* stream) {
  if (!p || !real_in || !spec_out) return rfail(SHAFFT_SM100_EINVAL, "null argument");
  if (real_in == spec_out) return rfail(SHAFFT_SM100_EINVAL, "input and output must be distinct buffers");
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const int rc = shafft_sm100_execute(p->full, real_in, p->a, 0, 1.0, stream);
  if (rc) return rc;
  const RcShape g = rc_shape(p->rows, p->H);
  cudaError_t e;
  if (p->precision)
    e = launch_chained(
        k_r2c_untangle<double>, g.grid, 256, 0, s,
        reinterpret_cast<const double2*>(p->a),
        reinterpret_cast<double2*>(spec_out), p->rows, p->H, g.chunks, g.logG,
        reinterpret_cast<const double2*>(p->tw), scale, p->dims);
  else
    e = launch_chained(
        k_r2c_untangle<float>, g.grid, 256, 0, s,
        reinterpret_cast<const float2*>(p->a),
        reinterpret_cast<float2*>(spec_out), p->rows, p->H, g.chunks, g.logG,
        reinterpret_cast<const float2*>(p->tw), (float)scale, p->dims);
  if (e != cudaSuccess) return rfail(SHAFFT_SM100_ECUDA, "untangle launch: %s", cudaGetErrorString(e));
  return 0;
}

int shafft_sm100_execute_c2r(shafft_sm100_rplan p, void* spec_in, void* real_out, double scale, void* stream) {
  if (!p || !spec_in || !real_out) return rfail(SHAFFT_SM100_EINVAL, "null argument");
  if (real_out == spec_in) return rfail(SHAFFT_SM100_EINVAL, "input and output must be distinct buffers");
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const RcShape g = rc_shape(p->rows, p->H);
  cudaError_t e;
  if (p->precision)
    e = launch_chained(
        k_c2r_tangle<double>, g.grid, 256, 0, s,
        reinterpret_cast<const double2*>(spec_in), reinterpret_cast<double2*>(p->a), p->rows, p->H, g.chunks, g.logG,
        reinterpret_cast<const double2*>(p->tw), p->dims);
  else
    e = launch_chained(
        k_c2r_tangle<float>, g.grid, 256, 0, s,
        reinterpret_cast<const float2*>(spec_in), reinterpret_cast<float2*>(p->a), p->rows, p->H, g.chunks, g.logG,
        reinterpret_cast<const float2*>(p->tw), p->dims);
  if (e != cudaSuccess) return rfail(SHAFFT_SM100_ECUDA, "tangle launch: %s", cudaGetErrorString(e));
  return shafft_sm100_execute(p->full, p->a, real_out, 1, scale, stream);
}

}  // extern "C"
