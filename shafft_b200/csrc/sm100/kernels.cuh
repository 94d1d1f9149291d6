// Direct-DFT pass, element-wise kernels and table generation of the sm_100a
// C2C FFT backend.
//
// k_fft_direct -- one HBM pass of batched length-L DFTs on W-wide tiles for
// lengths with a prime factor above 13: the tile is loaded in natural order
// and every output is an O(L) sum, evaluated in pairs (direct_store).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "butterflies.cuh"
#include "mix.cuh"
#include "pass.h"

namespace shafft_sm100 {

// One output of a direct-DFT tile, with the pass's fused post-twiddle,
// scale and output conjugation.
template <typename T, typename C>
__device__ __forceinline__ void direct_put(const PassGeom& g, const PassTables<C>& tb, C* out, C y, int k, int w,
                                           int64_t bout, int64_t w0, int64_t tconst, T scale) {
  if (g.tw_mode == TW_POST) {
    const int64_t tt = (g.tw_dim == 0) ? (w0 + w) : tconst;
    y = cmul(y, tw_n(tb, g.tw_shift, g.tw_mask, (int64_t)k * tt));
  }
  if (g.scale != 1.0) y = cscale(y, scale);
  if (g.conj_out) y.y = -y.y;
  out[bout + (int64_t)w * g.sout[0] + (int64_t)k * g.sk_out] = y;
}

// Direct DFT of the tile held in shared memory (natural order, [n][w] with
// the given pitch), X[k] = sum_n x[n] w^{nk} with w = exp(-2 pi i / L),
// evaluated in pairs.  With s[n] = x[n] + x[L-n] and d[n] = x[n] - x[L-n]
// for n = 1 .. h (h = (L-1)/2), and e_k = (-1)^k x[L/2] for even L (0 for
// odd L):
//   X[k]   = x[0] + e_k + sum_n s[n] Re w^{nk} + i sum_n d[n] Im w^{nk}
//   X[L-k] = x[0] + e_k + sum_n s[n] Re w^{nk} - i sum_n d[n] Im w^{nk}
// for k = 1 .. h; X[0] = x[0] + sum_n s[n] + x[L/2] and, for even L,
// X[L/2] = x[0] + sum_n (-1)^n s[n] + (-1)^{L/2} x[L/2].  Each table read
// and each pair of real multiplies then serves two outputs, a quarter of
// the arithmetic of the plain sum; the exponent n*k is reduced modulo L
// incrementally.  Used for lengths with a prime factor above 13 when L is
// small enough that O(L) work per output beats a Bluestein round trip.
// Outputs go straight to HBM with the pass's fused twiddle/scale/conj.
template <typename T, typename C>
__device__ __forceinline__ void direct_store(const PassGeom& g, const PassTables<C>& tb, C* sm, C* out, int L,
                                             int W, int logW, int pitch, int wcount, int64_t bout, int64_t w0,
                                             int64_t tconst) {
  const int h = (L - 1) / 2;
  const bool even = (L & 1) == 0;
  // s and d in place: row n <- s[n], row L-n <- d[n]
  for (int b = threadIdx.x; b < (h << logW); b += kThreads) {
    const int w = b & (W - 1), n = 1 + (b >> logW);
    const C a = sm[n * pitch + w], c = sm[(L - n) * pitch + w];
    sm[n * pitch + w] = C{a.x + c.x, a.y + c.y};
    sm[(L - n) * pitch + w] = C{a.x - c.x, a.y - c.y};
  }
  __syncthreads();
  const T scale = (T)g.scale;
  // item (j, w): j = 0 gives X[0] (and X[L/2] for even L), j = 1 .. h gives
  // X[j] and X[L-j]
  const int items = (h + 1) << logW;
  for (int b = threadIdx.x; b < items; b += kThreads) {
    const int w = b & (W - 1), j = b >> logW;
    if (w >= wcount) continue;
    const C x0 = sm[w];
    const C xh = even ? sm[(L / 2) * pitch + w] : C{0, 0};
    if (j == 0) {
      C y0 = x0, yh = x0;
      T sg = -1;
      for (int n = 1; n <= h; ++n) {
        const C sn = sm[n * pitch + w];
        y0.x += sn.x;
        y0.y += sn.y;
        yh.x += sg * sn.x;
        yh.y += sg * sn.y;
        sg = -sg;
      }
      y0.x += xh.x;
      y0.y += xh.y;
      direct_put<T, C>(g, tb, out, y0, 0, w, bout, w0, tconst, scale);
      if (even) {
        const T e = ((L / 2) & 1) ? (T)-1 : (T)1;
        yh.x += e * xh.x;
        yh.y += e * xh.y;
        direct_put<T, C>(g, tb, out, yh, L / 2, w, bout, w0, tconst, scale);
      }
      continue;
    }
    T px = 0, py = 0, qx = 0, qy = 0;
    int m = 0;
    for (int n = 1; n <= h; ++n) {
      m += j;
      if (m >= L) m -= L;
      const C t = tb.twL[m];
      const C sn = sm[n * pitch + w], dn = sm[(L - n) * pitch + w];
      px += sn.x * t.x;
      py += sn.y * t.x;
      qx += dn.x * t.y;
      qy += dn.y * t.y;
    }
    const T e = (j & 1) ? (T)-1 : (T)1;
    const T bx = x0.x + e * xh.x + px, by = x0.y + e * xh.y + py;
    direct_put<T, C>(g, tb, out, C{bx - qy, by + qx}, j, w, bout, w0, tconst, scale);
    direct_put<T, C>(g, tb, out, C{bx + qy, by - qx}, L - j, w, bout, w0, tconst, scale);
  }
}

// One tile of a direct-DFT pass.  `sm` holds L * pitch elements.
template <typename T>
__device__ __forceinline__ void direct_tile(const PassGeom& g, const typename Cx<T>::type* in,
                                            typename Cx<T>::type* out,
                                            const PassTables<typename Cx<T>::type>& tb, int64_t tile,
                                            typename Cx<T>::type* sm) {
  using C = typename Cx<T>::type;
  const int L = g.L, W = g.W;
  const TileAt at = tile_at(g, tile);
  const int total = L << g.logW;
  for (int b = threadIdx.x; b < total; b += kThreads) {
    int w, n;
    if (g.in_row) {
      n = b % L;
      w = b / L;
    } else {
      w = b & (W - 1);
      n = b >> g.logW;
    }
    C x = (w < at.wcount) ? in[at.bin + (int64_t)w * g.sin[0] + (int64_t)n * g.sn_in] : C{0, 0};
    if (g.conj_in) x.y = -x.y;
    sm[n * g.pitch + w] = x;
  }
  __syncthreads();
  direct_store<T, C>(g, tb, sm, out, L, W, g.logW, g.pitch, at.wcount, at.bout, at.w0, at.tconst);
}

template <typename T>
__global__ void __launch_bounds__(kThreads)
    k_fft_direct(const __grid_constant__ PassGeom g, const typename Cx<T>::type* in,
                 typename Cx<T>::type* out, const __grid_constant__ PassTables<typename Cx<T>::type> tb) {
  using C = typename Cx<T>::type;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  C* sm = reinterpret_cast<C*>(smem_raw);
  for (int64_t tile = blockIdx.x; tile < g.ntiles; tile += gridDim.x) {
    direct_tile<T>(g, in, out, tb, tile, sm);
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Elementwise kernels
// ---------------------------------------------------------------------------

// data[i] = conj?(src[i]) * factor   (normalize, copies)
template <typename T>
__global__ void k_scale_copy(const typename Cx<T>::type* src, typename Cx<T>::type* dst, int64_t n,
                             T factor, int conj) {
  using C = typename Cx<T>::type;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    C x = src[i];
    x.x *= factor;
    x.y *= factor;
    if (conj) x.y = -x.y;
    dst[i] = x;
  }
}

// The Bluestein element-wise steps run on a 2-D grid: blockIdx.y walks the
// batch rows b = o*I + i (one division per row), blockIdx.x/threadIdx.x the
// points of a row in block tiles of kEwUnroll*blockDim points, each thread
// loading its kEwUnroll points before it computes (independent loads in
// flight; the arrays are L2-resident at the lengths Bluestein pads to).
constexpr int kEwUnroll = 4;

// Bluestein modulate: dst[b*M + m] = (m < L) ? conj?(x(o, m, i)) * chirp[m] : 0
// with b = o*I + i and x(o, m, i) = src[(o*L + m)*I + i].
template <typename T>
__global__ void k_bs_modulate(const typename Cx<T>::type* src, typename Cx<T>::type* dst, int64_t L,
                              int64_t M, int64_t I, int64_t rows, const typename Cx<T>::type* chirp,
                              int conj) {
  using C = typename Cx<T>::type;
  const int64_t tile = (int64_t)blockDim.x * kEwUnroll;
  for (int64_t b = blockIdx.y; b < rows; b += gridDim.y) {
    const int64_t o = b / I, i = b - o * I;
    const C* srow = src + o * L * I + i;
    C* drow = dst + b * M;
    for (int64_t base = blockIdx.x * tile + threadIdx.x; base < M; base += gridDim.x * tile) {
      C x[kEwUnroll], w[kEwUnroll];
#pragma unroll
      for (int u = 0; u < kEwUnroll; ++u) {
        const int64_t m = base + (int64_t)u * blockDim.x;
        x[u] = m < L ? srow[m * I] : C{0, 0};
        w[u] = m < L ? chirp[m] : C{0, 0};
      }
#pragma unroll
      for (int u = 0; u < kEwUnroll; ++u) {
        const int64_t m = base + (int64_t)u * blockDim.x;
        if (conj) x[u].y = -x[u].y;
        if (m < M) drow[m] = cmul(x[u], w[u]);
      }
    }
  }
}

// s[b*M + m] = conj(s[b*M + m] * H[m])   (H carries the 1/M of the inverse)
template <typename T>
__global__ void k_bs_mulh(typename Cx<T>::type* s, const typename Cx<T>::type* H, int64_t M,
                          int64_t rows) {
  using C = typename Cx<T>::type;
  const int64_t tile = (int64_t)blockDim.x * kEwUnroll;
  for (int64_t b = blockIdx.y; b < rows; b += gridDim.y) {
    C* row = s + b * M;
    for (int64_t base = blockIdx.x * tile + threadIdx.x; base < M; base += gridDim.x * tile) {
      C x[kEwUnroll], h[kEwUnroll];
#pragma unroll
      for (int u = 0; u < kEwUnroll; ++u) {
        const int64_t m = base + (int64_t)u * blockDim.x;
        x[u] = m < M ? row[m] : C{0, 0};
        h[u] = m < M ? H[m] : C{0, 0};
      }
#pragma unroll
      for (int u = 0; u < kEwUnroll; ++u) {
        const int64_t m = base + (int64_t)u * blockDim.x;
        C y = cmul(x[u], h[u]);
        y.y = -y.y;
        if (m < M) row[m] = y;
      }
    }
  }
}

// Bluestein demodulate: dst(o, k, i) = conj?(chirp[k] * conj(s[b*M + k])) * scale
template <typename T>
__global__ void k_bs_demod(const typename Cx<T>::type* s, typename Cx<T>::type* dst, int64_t L,
                           int64_t M, int64_t I, int64_t rows, const typename Cx<T>::type* chirp,
                           int conj, T scale) {
  using C = typename Cx<T>::type;
  const int64_t tile = (int64_t)blockDim.x * kEwUnroll;
  for (int64_t b = blockIdx.y; b < rows; b += gridDim.y) {
    const int64_t o = b / I, i = b - o * I;
    const C* srow = s + b * M;
    C* drow = dst + o * L * I + i;
    for (int64_t base = blockIdx.x * tile + threadIdx.x; base < L; base += gridDim.x * tile) {
      C v[kEwUnroll], w[kEwUnroll];
#pragma unroll
      for (int u = 0; u < kEwUnroll; ++u) {
        const int64_t k = base + (int64_t)u * blockDim.x;
        v[u] = k < L ? srow[k] : C{0, 0};
        w[u] = k < L ? chirp[k] : C{0, 0};
      }
#pragma unroll
      for (int u = 0; u < kEwUnroll; ++u) {
        const int64_t k = base + (int64_t)u * blockDim.x;
        C a = v[u];
        a.y = -a.y;
        C r = cmul(w[u], a);
        r.x *= scale;
        r.y *= scale;
        if (conj) r.y = -r.y;
        if (k < L) drow[k * I] = r;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Table generation (FP64 phase, rounded once to the storage type)
// ---------------------------------------------------------------------------

// out[i] = exp(-2*pi*i * ((i*mult) mod N) / N), i < count
template <typename T>
__global__ void k_gen_twiddle(typename Cx<T>::type* out, int64_t count, int64_t mult, int64_t N) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < count;
       i += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t m = ((unsigned __int128)(uint64_t)i * (uint64_t)mult) % (uint64_t)N;
    double s, c;
    sincospi(-2.0 * ((double)m / (double)N), &s, &c);
    out[i] = typename Cx<T>::type{(T)c, (T)s};
  }
}

// chirp[m] = exp(-i*pi*(m^2 mod 2L)/L), m < L  (integer phase reduction)
template <typename T>
__global__ void k_gen_chirp(typename Cx<T>::type* out, int64_t L) {
  for (int64_t m = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; m < L;
       m += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t r = ((unsigned __int128)(uint64_t)m * (uint64_t)m) % (uint64_t)(2 * L);
    double s, c;
    sincospi(-((double)r / (double)L), &s, &c);
    out[m] = typename Cx<T>::type{(T)c, (T)s};
  }
}

// Bluestein kernel sequence h (length M): conj(chirp[|j|]) cyclically, zero elsewhere.
template <typename T>
__global__ void k_gen_bs_kernel(typename Cx<T>::type* h, const typename Cx<T>::type* chirp, int64_t L,
                                int64_t M) {
  using C = typename Cx<T>::type;
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < M;
       j += (int64_t)gridDim.x * blockDim.x) {
    C r = C{0, 0};
    if (j < L) {
      r = chirp[j];
      r.y = -r.y;
    } else if (j > M - L) {
      r = chirp[M - j];
      r.y = -r.y;
    }
    h[j] = r;
  }
}

}  // namespace shafft_sm100
