// Generic HBM pass: batched DFTs of any length that factors into 2, 3, 5, 7,
// 11, 13 (L <= 4096) on tiles of L points x W batch columns, radix sequence
// and strides at run time.
//
// Phase A  every thread loads the R0 inputs of a first-stage butterfly of
//          one chunk (VW neighbouring batch columns), runs the radix-R0
//          butterfly in registers, applies the decimation-in-frequency
//          twiddle and stores the results to the shared tile.
// Phase B  the middle radix stages, in place in the shared tile.
// Phase C  the last radix stage; its outputs go from registers straight to
//          HBM at their natural (digit-unreversed) places, with the four-step
//          post-twiddle, scale and conjugation fused in.
// A length of one radix needs neither the tile nor a barrier.
//
// What bounds it: instructions issued (an HBM-rate pass has about 90 thread
// instructions per complex64 element).  So
//   * a chunk is 16 bytes (VW = 2 complex64 or 1 complex128 column): index
//     arithmetic, twiddles and shared accesses are paid once per chunk
//     (VW = 1 for a complex64 tile of one column);
//   * index divisions by run-time values are one multiply-high (the planner
//     stores the reciprocals), also those that find a tile's place;
//   * radices up to 13 with 6, 9, 10, 12 composed in registers, so that up to
//     1728 points need three stages, i.e. two trips through shared memory;
//   * results are stored from the last stage's registers.
// Measured on B200 against the pass it replaced (per-element shared accesses,
// run-time divisions, radices {2,3,4,5,7,8,11,13,16}, results read back from
// shared memory through a permutation table): 384^3 complex64 forward +
// normalize 2.13 -> 0.83 ms (a pass 650 -> 215 us), 2048^2 complex64 158 ->
// 64 us, 1,488,375 complex128 72 -> 64 us (against compile-time instances of
// its two lengths), 512 uneven batched transforms 5.28 -> 4.23 ms.
//
// The chunk of column c of point p has linear slot s = p * NC + c (NC = W / VW
// chunks a row).  Column tiles at least 8 chunks wide use it as it is: 8 lanes
// always cover one row, i.e. all 128-byte bank groups.  Everything else has
// lanes that walk points (row tiles, narrow tiles), at strides that depend on
// the radices, and folds the higher bits of s into the bank bits (SWZ).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "butterflies.cuh"
#include "pass.h"

namespace shafft_sm100 {

template <typename C>
__device__ __forceinline__ C tw_n(const PassTables<C>& tb, int shift, int64_t mask, int64_t m) {
  const C hi = __ldg(tb.tw_hi + (m >> shift));
  const C lo = __ldg(tb.tw_lo + (m & mask));
  return cmul(hi, lo);
}

// VW complex elements moved as one 8- or 16-byte vector
template <typename C, int VW>
struct alignas(sizeof(C) * VW) MixChunk {
  C v[VW];
};

template <int VW, int BYTES, bool SWZ>
__device__ __forceinline__ int mix_slot(int s) {
  if constexpr (SWZ) {
    constexpr int B = BYTES == 16 ? 3 : 4;  // chunks per 128 bytes
    return s ^ (((s >> B) ^ (s >> (2 * B)) ^ (s >> (3 * B))) & ((1 << B) - 1));
  } else {
    return s;
  }
}

// Position of a tile in its pass.
struct TileAt {
  int64_t w0, bin, bout, tconst;
  int wcount;
};
__device__ __forceinline__ TileAt tile_at(const PassGeom& g, int64_t tile) {
  const TileIdx x = tile_idx(g, tile);
  TileAt a;
  a.w0 = x.tw * g.W;
  const int64_t left = g.ext[0] - a.w0;
  a.wcount = (int)(left < g.W ? left : g.W);
  a.bin = a.w0 * g.sin[0] + x.i1 * g.sin[1] + x.i2 * g.sin[2] + x.i3 * g.sin[3];
  a.bout = a.w0 * g.sout[0] + x.i1 * g.sout[1] + x.i2 * g.sout[2] + x.i3 * g.sout[3];
  a.tconst = g.tw_dim == 1 ? x.i1 : (g.tw_dim == 2 ? x.i2 : (g.tw_dim == 3 ? x.i3 : 0));
  return a;
}

// What every phase of a tile needs.
template <typename T, int VW>
struct MixEnv {
  using C = typename Cx<T>::type;
  const C* in;   // tile origin
  C* out;        // tile origin
  int logNC;
  int wcount;
  int64_t w0, tconst;
  T sy_in, sx, sy;  // imaginary sign at load; real and imaginary factor at store
  bool vin, vout;   // chunks are 16-byte vectors in memory
};

template <int R, typename T, int VW>
__device__ __forceinline__ void mix_load(const PassGeom& g, const MixEnv<T, VW>& e,
                                         typename Cx<T>::type (&v)[VW][R], int c, int j, int m0) {
  using C = typename Cx<T>::type;
  const int wl = e.wcount - c * VW;  // valid columns of this chunk (may exceed VW)
  const int64_t step = (int64_t)m0 * g.sn_in;
  const C* p = e.in + (int64_t)j * g.sn_in + (int64_t)(c * VW) * g.sin[0];
  if (VW > 1 && e.vin && wl >= VW) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const MixChunk<C, VW> q = *reinterpret_cast<const MixChunk<C, VW>*>(p + r * step);
#pragma unroll
      for (int k = 0; k < VW; ++k) v[k][r] = q.v[k];
    }
  } else {
#pragma unroll
    for (int k = 0; k < VW; ++k) {
      const C* q = p + (int64_t)k * g.sin[0];
#pragma unroll
      for (int r = 0; r < R; ++r) v[k][r] = wl > k ? q[r * step] : C{0, 0};
    }
  }
#pragma unroll
  for (int k = 0; k < VW; ++k)
#pragma unroll
    for (int r = 0; r < R; ++r) v[k][r].y *= e.sy_in;
}

// Outputs k0 + r * ks (r < R) of one chunk.  The four-step twiddle w_N^{k t}
// is a running product by w_N^{ks t}, taken afresh from the two-level table
// every kTwAnchor outputs.
template <int R, typename T, int VW>
__device__ __forceinline__ void mix_store(const PassGeom& g, const PassTables<typename Cx<T>::type>& tb,
                                          const MixEnv<T, VW>& e, typename Cx<T>::type (&v)[VW][R], int c, int k0,
                                          int ks) {
  using C = typename Cx<T>::type;
  constexpr int kTwAnchor = 4;
  const int wl = e.wcount - c * VW;
  if (g.tw_mode == TW_POST) {
#pragma unroll
    for (int k = 0; k < VW; ++k) {
      // columns past the edge use the last valid one's exponent (in range of the tables)
      const int64_t t = g.tw_dim == 0 ? e.w0 + min(c * VW + k, e.wcount - 1) : e.tconst;
      const C step = tw_n(tb, g.tw_shift, g.tw_mask, (int64_t)ks * t);
      C cur = C{1, 0};
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if (r % kTwAnchor == 0)
          cur = tw_n(tb, g.tw_shift, g.tw_mask, (int64_t)(k0 + r * ks) * t);
        else
          cur = cmul(cur, step);
        v[k][r] = cmul(v[k][r], cur);
      }
    }
  }
#pragma unroll
  for (int k = 0; k < VW; ++k)
#pragma unroll
    for (int r = 0; r < R; ++r) v[k][r] = C{v[k][r].x * e.sx, v[k][r].y * e.sy};
  const int64_t step = (int64_t)ks * g.sk_out;
  C* p = e.out + (int64_t)k0 * g.sk_out + (int64_t)(c * VW) * g.sout[0];
  if (VW > 1 && e.vout && wl >= VW) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      MixChunk<C, VW> q;
#pragma unroll
      for (int k = 0; k < VW; ++k) q.v[k] = v[k][r];
      *reinterpret_cast<MixChunk<C, VW>*>(p + r * step) = q;
    }
  } else {
#pragma unroll
    for (int k = 0; k < VW; ++k) {
      if (wl <= k) continue;
      C* q = p + (int64_t)k * g.sout[0];
#pragma unroll
      for (int r = 0; r < R; ++r) q[r * step] = v[k][r];
    }
  }
}

template <int R, typename C, int VW>
__device__ __forceinline__ void mix_dft(C (&v)[VW][R]) {
#pragma unroll
  for (int k = 0; k < VW; ++k) dft<R>(v[k]);
}

template <int R, typename C, int VW>
__device__ __forceinline__ void mix_twiddle(const C* twL, C (&v)[VW][R], int j) {
  if (j == 0) return;
#pragma unroll
  for (int r = 1; r < R; ++r) {
    const C w = __ldg(twL + j * r);
#pragma unroll
    for (int k = 0; k < VW; ++k) v[k][r] = cmul(v[k][r], w);
  }
}

template <int R, typename T, int VW, bool SWZ>
__device__ __forceinline__ void mix_first(const PassGeom& g, const PassTables<typename Cx<T>::type>& tb,
                                          const MixEnv<T, VW>& e, MixChunk<typename Cx<T>::type, VW>* sm) {
  using C = typename Cx<T>::type;
  constexpr int BYTES = sizeof(C) * VW;
  const int m0 = g.L / R;
  const int nbf = m0 << e.logNC;
  for (int id = threadIdx.x; id < nbf; id += blockDim.x) {
    int c, j;
    if (g.in_row) {
      c = (int)__umulhi((uint32_t)id, g.mdiv[0]);
      j = id - c * m0;
    } else {
      c = id & ((1 << e.logNC) - 1);
      j = id >> e.logNC;
    }
    C v[VW][R];
    mix_load<R, T, VW>(g, e, v, c, j, m0);
    mix_dft<R, C, VW>(v);
    mix_twiddle<R, C, VW>(tb.twL, v, j);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      MixChunk<C, VW> q;
#pragma unroll
      for (int k = 0; k < VW; ++k) q.v[k] = v[k][r];
      sm[mix_slot<VW, BYTES, SWZ>(((j + r * m0) << e.logNC) + c)] = q;
    }
  }
}

template <int R, typename T, int VW, bool SWZ>
__device__ __forceinline__ void mix_mid(const PassGeom& g, const PassTables<typename Cx<T>::type>& tb, int logNC,
                                        MixChunk<typename Cx<T>::type, VW>* sm, int s, int span, int Ls) {
  using C = typename Cx<T>::type;
  constexpr int BYTES = sizeof(C) * VW;
  const int m = span / R;
  const int nbf = (g.L / R) << logNC;
  const uint32_t mdiv = g.mdiv[s];
  for (int id = threadIdx.x; id < nbf; id += blockDim.x) {
    const int c = id & ((1 << logNC) - 1);
    const int q = id >> logNC;
    const int blk = (int)__umulhi((uint32_t)q, mdiv);
    const int j = q - blk * m;
    const int base = ((blk * span + j) << logNC) + c;
    const int st = m << logNC;
    C v[VW][R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const MixChunk<C, VW> x = sm[mix_slot<VW, BYTES, SWZ>(base + r * st)];
#pragma unroll
      for (int k = 0; k < VW; ++k) v[k][r] = x.v[k];
    }
    mix_dft<R, C, VW>(v);
    mix_twiddle<R, C, VW>(tb.twL, v, j * Ls);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      MixChunk<C, VW> x;
#pragma unroll
      for (int k = 0; k < VW; ++k) x.v[k] = v[k][r];
      sm[mix_slot<VW, BYTES, SWZ>(base + r * st)] = x;
    }
  }
}

template <int R, typename T, int VW, bool SWZ>
__device__ __forceinline__ void mix_last(const PassGeom& g, const PassTables<typename Cx<T>::type>& tb,
                                         const MixEnv<T, VW>& e, const MixChunk<typename Cx<T>::type, VW>* sm) {
  using C = typename Cx<T>::type;
  constexpr int BYTES = sizeof(C) * VW;
  const int ks = g.L / R;  // butterflies a column, and the stride of the last digit in k
  const int nbf = ks << e.logNC;
  for (int id = threadIdx.x; id < nbf; id += blockDim.x) {
    int c, k0, pos;
    if (g.out_row) {
      c = (int)__umulhi((uint32_t)id, g.mdiv[g.nst - 1]);
      k0 = id - c * ks;
      pos = __ldg(tb.k2p + k0);
    } else {
      c = id & ((1 << e.logNC) - 1);
      pos = (id >> e.logNC) * R;
      k0 = __ldg(tb.p2k + pos);
    }
    const int base = (pos << e.logNC) + c;
    C v[VW][R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const MixChunk<C, VW> x = sm[mix_slot<VW, BYTES, SWZ>(base + (r << e.logNC))];
#pragma unroll
      for (int k = 0; k < VW; ++k) v[k][r] = x.v[k];
    }
    mix_dft<R, C, VW>(v);
    mix_store<R, T, VW>(g, tb, e, v, c, k0, ks);
  }
}

// L = R: load, butterfly, store (in place is safe: a thread stores only where
// it loaded)
template <int R, typename T, int VW>
__device__ __forceinline__ void mix_single(const PassGeom& g, const PassTables<typename Cx<T>::type>& tb,
                                           const MixEnv<T, VW>& e) {
  using C = typename Cx<T>::type;
  for (int c = threadIdx.x; c < (1 << e.logNC); c += blockDim.x) {
    if (c * VW >= e.wcount) continue;
    C v[VW][R];
    mix_load<R, T, VW>(g, e, v, c, 0, 1);
    mix_dft<R, C, VW>(v);
    mix_store<R, T, VW>(g, tb, e, v, c, 0, 1);
  }
}

#define SHAFFT_MIX_DISPATCH(RAD, CALL) \
  switch (RAD) {                       \
    case 2: CALL(2); break;            \
    case 3: CALL(3); break;            \
    case 4: CALL(4); break;            \
    case 5: CALL(5); break;            \
    case 6: CALL(6); break;            \
    case 7: CALL(7); break;            \
    case 8: CALL(8); break;            \
    case 9: CALL(9); break;            \
    case 10: CALL(10); break;          \
    case 11: CALL(11); break;          \
    case 12: CALL(12); break;          \
    case 13: CALL(13); break;          \
    default: break;                    \
  }

// One tile.  `smem` holds L * W elements, rounded up to 128 bytes.
template <typename T, int VW, bool SWZ>
__device__ __forceinline__ void mix_tile(const PassGeom& g, const typename Cx<T>::type* in,
                                         typename Cx<T>::type* out,
                                         const PassTables<typename Cx<T>::type>& tb, int64_t tile, void* smem) {
  using C = typename Cx<T>::type;
  MixChunk<C, VW>* sm = reinterpret_cast<MixChunk<C, VW>*>(smem);
  const TileAt at = tile_at(g, tile);
  MixEnv<T, VW> e;
  e.in = in + at.bin;
  e.out = out + at.bout;
  e.logNC = g.logW - (VW == 2 ? 1 : 0);
  e.wcount = at.wcount;
  e.w0 = at.w0;
  e.tconst = at.tconst;
  e.sy_in = g.conj_in ? (T)-1 : (T)1;
  e.sx = (T)g.scale;
  e.sy = g.conj_out ? -(T)g.scale : (T)g.scale;
  // the geometry keeps 16-byte steps; the caller's buffer may start on 8
  e.vin = g.vec_in && (reinterpret_cast<uintptr_t>(in) & 15) == 0;
  e.vout = g.vec_out && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
  if (g.nst == 1) {
#define SHAFFT_CALL(R) mix_single<R, T, VW>(g, tb, e)
    SHAFFT_MIX_DISPATCH(g.L, SHAFFT_CALL)
#undef SHAFFT_CALL
    return;
  }
#define SHAFFT_CALL(R) mix_first<R, T, VW, SWZ>(g, tb, e, sm)
  SHAFFT_MIX_DISPATCH(g.rad[0], SHAFFT_CALL)
#undef SHAFFT_CALL
  __syncthreads();
  int Ls = g.rad[0];
  for (int s = 1; s + 1 < g.nst; ++s) {
    const int span = g.span[s];
#define SHAFFT_CALL(R) mix_mid<R, T, VW, SWZ>(g, tb, e.logNC, sm, s, span, Ls)
    SHAFFT_MIX_DISPATCH(g.rad[s], SHAFFT_CALL)
#undef SHAFFT_CALL
    Ls *= g.rad[s];
    __syncthreads();
  }
#define SHAFFT_CALL(R) mix_last<R, T, VW, SWZ>(g, tb, e, sm)
  SHAFFT_MIX_DISPATCH(g.rad[g.nst - 1], SHAFFT_CALL)
#undef SHAFFT_CALL
}

// 256 threads x 3 CTAs per SM, i.e. at most 85 registers; every instance is
// compiled to 80.  The radix 11 and 13 stages of a chunk need more, and spill:
// 104 bytes a thread (complex64 unpermuted), 60 (permuted), 188 and 268
// (complex128); the one-column complex64 instance does not.
template <typename T, int VW, bool SWZ>
__global__ void __launch_bounds__(kThreads, 3)
    k_fft_mix(const __grid_constant__ PassGeom g, const typename Cx<T>::type* in, typename Cx<T>::type* out,
              const __grid_constant__ PassTables<typename Cx<T>::type> tb) {
  chain_begin();
  extern __shared__ __align__(128) unsigned char smem_raw[];
  for (int64_t tile = blockIdx.x; tile < g.ntiles; tile += gridDim.x) {
    if (tile != blockIdx.x) __syncthreads();  // the previous tile is read out
    mix_tile<T, VW, SWZ>(g, in, out, tb, tile, smem_raw);
  }
}

}  // namespace shafft_sm100
