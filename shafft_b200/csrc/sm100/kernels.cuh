// Direct-DFT pass, element-wise kernels and table generation of the sm_100a
// C2C FFT backend.
//
// k_fft_direct -- one HBM pass of batched length-L DFTs on W-wide tiles for
// lengths with a prime factor above 13: the tile is loaded in natural order
// and every output is an O(L) sum, evaluated in pairs (direct_sums).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "butterflies.cuh"
#include "mix.cuh"
#include "pass.h"

namespace shafft_sm100 {

// Cosine c and sine s of a direct DFT, and acc + a * c, acc + a * s on complex
// numbers: for complex64 one packed FMA for both parts (two roundings as of
// two scalar FMAs), whose operand is the factor twice.
template <typename C>
struct DirectTw;
template <>
struct alignas(16) DirectTw<float2> {
  float2 cc, ss;
  __device__ __forceinline__ void set(float2 t) {
    cc = float2{t.x, t.x};
    ss = float2{t.y, t.y};
  }
  static __device__ __forceinline__ float2 fma2(float2 a, float2 tt, float2 acc) {
    float2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(reinterpret_cast<unsigned long long&>(r))
        : "l"(reinterpret_cast<const unsigned long long&>(a)), "l"(reinterpret_cast<const unsigned long long&>(tt)),
          "l"(reinterpret_cast<const unsigned long long&>(acc)));
    return r;
  }
  __device__ __forceinline__ float2 add_c(float2 a, float2 acc) const { return fma2(a, cc, acc); }
  __device__ __forceinline__ float2 add_s(float2 a, float2 acc) const { return fma2(a, ss, acc); }
};
template <>
struct alignas(16) DirectTw<double2> {
  double2 t;
  __device__ __forceinline__ void set(double2 x) { t = x; }
  __device__ __forceinline__ double2 add_c(double2 a, double2 acc) const {
    return double2{fma(a.x, t.x, acc.x), fma(a.y, t.x, acc.y)};
  }
  __device__ __forceinline__ double2 add_s(double2 a, double2 acc) const {
    return double2{fma(a.x, t.y, acc.x), fma(a.y, t.y, acc.y)};
  }
};

// One output of a direct-DFT tile, with the pass's fused post-twiddle,
// scale and output conjugation.
template <typename T, typename C>
__device__ __forceinline__ void direct_put(const PassGeom& g, const PassTables<C>& tb, C* out, C y, int k, int w,
                                           const TileAt& at, T scale) {
  if (g.tw_mode == TW_POST) {
    const int64_t tt = (g.tw_dim == 0) ? (at.w0 + w) : at.tconst;
    y = cmul(y, tw_n(tb, g.tw_shift, g.tw_mask, (int64_t)k * tt));
  }
  y = C{y.x * scale, g.conj_out ? -(y.y * scale) : y.y * scale};
  out[at.bout + (int64_t)w * g.sout[0] + (int64_t)k * g.sk_out] = y;
}

// Sums and stores of a direct-DFT tile: item (jg, wg) is the output pairs
// jg + i * ng (i < J) of the columns wg + c * WG (c < CB).
template <typename T, int J, int CB>
__device__ __forceinline__ void direct_sums(const PassGeom& g, const PassTables<typename Cx<T>::type>& tb,
                                            typename Cx<T>::type* out, const typename Cx<T>::type* sm,
                                            const DirectTw<typename Cx<T>::type>* tw, const TileAt& at) {
  using C = typename Cx<T>::type;
  const int L = g.L, W = g.W, pitch = g.pitch;
  const int h = (L - 1) / 2, half = L / 2, np = half + 1;
  const bool even = (L & 1) == 0;
  const T scale = (T)g.scale;
  const int WG = W >= CB ? W / CB : 1, ng = (np + J - 1) / J;
  const int logWG = W >= CB ? g.logW - (CB == 2 ? 1 : 0) : 0;
  for (int b = threadIdx.x; b < (ng << logWG); b += blockDim.x) {
    const int wg = b & (WG - 1), jg = b >> logWG;
    if (wg >= at.wcount) continue;
    C P[J][CB], Q[J][CB];
    int j[J], m[J];
#pragma unroll
    for (int i = 0; i < J; ++i) {
      j[i] = min(jg + i * ng, half);
      m[i] = 0;
#pragma unroll
      for (int c = 0; c < CB; ++c) P[i][c] = Q[i][c] = C{0, 0};
    }
    auto step = [&](int n) {
      C sn[CB], dn[CB];
#pragma unroll
      for (int c = 0; c < CB; ++c) {
        const int w = min(wg + c * WG, W - 1);
        sn[c] = sm[n * pitch + w];
        dn[c] = sm[(L - n) * pitch + w];
      }
#pragma unroll
      for (int i = 0; i < J; ++i) {
        const uint32_t mi = (uint32_t)(m[i] + j[i]);
        m[i] = (int)min(mi, mi - (uint32_t)L);  // mod L: mi - L wraps to a large number below L
        const DirectTw<C> t = tw[m[i]];
#pragma unroll
        for (int c = 0; c < CB; ++c) {
          P[i][c] = t.add_c(sn[c], P[i][c]);
          Q[i][c] = t.add_s(dn[c], Q[i][c]);
        }
      }
    };
    if constexpr (J == 1) {
#pragma unroll 4  // a lone output pair waits on its own loads
      for (int n = 1; n <= h; ++n) step(n);
    } else {
      for (int n = 1; n <= h; ++n) step(n);
    }
#pragma unroll
    for (int c = 0; c < CB; ++c) {
      const int w = wg + c * WG;
      if (w >= at.wcount) continue;
      const C x0 = sm[w];
      const C xh = even ? sm[half * pitch + w] : C{0, 0};
#pragma unroll
      for (int i = 0; i < J; ++i) {
        const int k = jg + i * ng;
        if (k > half) continue;
        const T e = (k & 1) ? (T)-1 : (T)1;
        const T bx = x0.x + e * xh.x + P[i][c].x, by = x0.y + e * xh.y + P[i][c].y;
        // an output that is its own partner has no sine part: 0 times an
        // infinite input would make it NaN
        const bool own = k == 0 || 2 * k == L;
        const C q = own ? C{0, 0} : Q[i][c];
        direct_put<T, C>(g, tb, out, C{bx - q.y, by + q.x}, k, w, at, scale);
        if (!own) direct_put<T, C>(g, tb, out, C{bx + q.y, by - q.x}, L - k, w, at, scale);
      }
    }
  }
}

// One tile of a direct-DFT pass: X[k] = sum_n x[n] w^{nk}, w = exp(-2 pi i / L),
// evaluated in pairs.  With s[n] = x[n] + x[L-n] and d[n] = x[n] - x[L-n] for
// n = 1 .. h (h = (L-1)/2), and e_k = (-1)^k x[L/2] for even L (0 for odd L):
//   X[k]   = x[0] + e_k + sum_n s[n] Re w^{nk} + i sum_n d[n] Im w^{nk}
//   X[L-k] = x[0] + e_k + sum_n s[n] Re w^{nk} - i sum_n d[n] Im w^{nk}
// for k = 0 .. L/2 (X[0], and X[L/2] of even L, are their own partners): two
// real h x h matrices times the complex columns s and d, a quarter of the
// arithmetic of the plain sum.  Used for lengths with a prime factor above 13
// when L is small enough that O(L) work per output beats a Bluestein round
// trip.
//
// Bound by FP32 / FP64 multiply-adds (about L per point), so a thread keeps
// kDirectJ output pairs of direct_cols columns in registers: each twiddle pair read
// serves the columns and each s, d the outputs, and complex64 sums take one
// packed multiply-add for both parts.  The exponent n*k is reduced modulo L
// incrementally.
//
// `sm` holds the tile, L * pitch elements ([n][w]; rows n and L - n hold s and
// d), rounded up to 16 bytes, then L DirectTw.
template <typename T>
__device__ __forceinline__ void direct_tile(const PassGeom& g, const typename Cx<T>::type* in,
                                            typename Cx<T>::type* out,
                                            const PassTables<typename Cx<T>::type>& tb, int64_t tile,
                                            typename Cx<T>::type* sm) {
  using C = typename Cx<T>::type;
  const int L = g.L, W = g.W, pitch = g.pitch;
  const int half = L / 2;
  const TileAt at = tile_at(g, tile);
  DirectTw<C>* tw = reinterpret_cast<DirectTw<C>*>(
      reinterpret_cast<unsigned char*>(sm) + (((size_t)L * pitch * sizeof(C) + 15) & ~(size_t)15));
  for (int m = threadIdx.x; m < L; m += blockDim.x) tw[m].set(__ldg(tb.twL + m));
  // s and d of the pairs (n, L - n); n = 0 and, for even L, L/2 alone
  const int np = half + 1;
  const T sy = g.conj_in ? (T)-1 : (T)1;
#pragma unroll 2
  for (int b = threadIdx.x; b < (np << g.logW); b += blockDim.x) {
    int w, n;
    if (g.in_row) {
      w = np > 1 ? (int)__umulhi((uint32_t)b, g.mdiv[0]) : b;
      n = b - w * np;
    } else {
      w = b & (W - 1);
      n = b >> g.logW;
    }
    const int n2 = n == 0 ? 0 : L - n;
    const C* p = in + at.bin + (int64_t)w * g.sin[0];
    C x = C{0, 0}, z = C{0, 0};
    if (w < at.wcount) {
      x = p[(int64_t)n * g.sn_in];
      if (n != n2) z = p[(int64_t)n2 * g.sn_in];
    }
    x.y *= sy;
    z.y *= sy;
    if (n == n2) {
      sm[n * pitch + w] = x;
    } else {
      sm[n * pitch + w] = C{x.x + z.x, x.y + z.y};
      sm[n2 * pitch + w] = C{x.x - z.x, x.y - z.y};
    }
  }
  __syncthreads();
  if (g.direct_j == 1)
    direct_sums<T, 1, 1>(g, tb, out, sm, tw, at);
  else
    direct_sums<T, kDirectJ, direct_cols(sizeof(C))>(g, tb, out, sm, tw, at);
}

template <typename T>
__global__ void __launch_bounds__(kThreads)
    k_fft_direct(const __grid_constant__ PassGeom g, const typename Cx<T>::type* in,
                 typename Cx<T>::type* out, const __grid_constant__ PassTables<typename Cx<T>::type> tb) {
  chain_begin();
  using C = typename Cx<T>::type;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  C* sm = reinterpret_cast<C*>(smem_raw);
  for (int64_t tile = blockIdx.x; tile < g.ntiles; tile += gridDim.x) {
    direct_tile<T>(g, in, out, tb, tile, sm);
    __syncthreads();
  }
}

// streaming accesses of 8- and 16-byte vectors
template <typename V>
__device__ __forceinline__ V ld_vec(const V* p) {
  static_assert(sizeof(V) == 16 || sizeof(V) == 8, "vector of 8 or 16 bytes");
  V v;
  if constexpr (sizeof(V) == 16)
    reinterpret_cast<float4&>(v) = __ldcs(reinterpret_cast<const float4*>(p));
  else
    reinterpret_cast<float2&>(v) = __ldcs(reinterpret_cast<const float2*>(p));
  return v;
}
template <typename V>
__device__ __forceinline__ void st_vec(V* p, const V& v) {
  if constexpr (sizeof(V) == 16)
    __stcs(reinterpret_cast<float4*>(p), reinterpret_cast<const float4&>(v));
  else
    __stcs(reinterpret_cast<float2*>(p), reinterpret_cast<const float2&>(v));
}

// ---------------------------------------------------------------------------
// Elementwise kernels
// ---------------------------------------------------------------------------

// dst[i] = conj?(src[i]) * factor   (normalize, copies); src may be dst.
// HBM bound: blocks of kScaleUnroll x 256 vectors of VW elements (16 bytes
// where both buffers start on 16), all loads issued before the first store,
// both streaming.  Measured on B200, 384^3 complex64 in place:
// 165 -> 134 us, 6.75 TB/s (one 8-byte element a step of a grid-stride loop
// before).
constexpr int kScaleUnroll = 4;
template <typename T, int VW>
__global__ void __launch_bounds__(256)
    k_scale_copy(const typename Cx<T>::type* src, typename Cx<T>::type* dst, int64_t n, T fx, T fy) {
  chain_begin();
  using C = typename Cx<T>::type;
  using V = MixChunk<C, VW>;
  const int64_t nv = n / VW;
  const int64_t i0 = (int64_t)blockIdx.x * (256 * kScaleUnroll) + threadIdx.x;
  V x[kScaleUnroll];
#pragma unroll
  for (int u = 0; u < kScaleUnroll; ++u)
    if (i0 + u * 256 < nv) x[u] = ld_vec(reinterpret_cast<const V*>(src) + i0 + u * 256);
#pragma unroll
  for (int u = 0; u < kScaleUnroll; ++u) {
    if (i0 + u * 256 >= nv) continue;
#pragma unroll
    for (int k = 0; k < VW; ++k) x[u].v[k] = C{x[u].v[k].x * fx, x[u].v[k].y * fy};
    st_vec(reinterpret_cast<V*>(dst) + i0 + u * 256, x[u]);
  }
  if (VW > 1 && blockIdx.x == 0 && threadIdx.x < n - nv * VW) {
    const int64_t i = nv * VW + threadIdx.x;
    dst[i] = C{src[i].x * fx, src[i].y * fy};
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
