// Pass descriptors shared by the host planner (plan.cu) and the device
// kernels (kernels.cu).
//
// A "pass" is one kernel launch that reads the whole working tensor from HBM
// once and writes it once.  It performs batched DFTs of length L (L <= 4096)
// along one logical index "n" of a strided view of the tensor:
//
//   input  element (n, b0, b1, b2, b3) at  in  + n*sn_in  + sum_d b_d*sin[d]
//   output element (k, b0, b1, b2, b3) at  out + k*sk_out + sum_d b_d*sout[d]
//
// b0 is the tile dimension: one CTA processes W consecutive b0 values for one
// (b1, b2, b3) tuple, so every load/store instruction of a warp touches W
// consecutive elements when sin[0]/sout[0] == 1 ("column" orientation) or L
// consecutive elements when sn_in/sk_out == 1 ("row" orientation).
//
// Optional extras fused into the same pass:
//   * a four-step twiddle  w_N^{k * t}  with t = b_{tw_dim} on the output; the
//     planner guarantees the exponent is < N so no modular reduction is needed;
//   * conjugation on input / output (backward transforms are computed as
//     conj(F(conj(x))));
//   * a real scale on output (fused normalisation).
#pragma once
#include <stdint.h>

namespace shafft_sm100 {

constexpr int kMaxStages = 8;
constexpr int kMaxPassLen = 4096;
constexpr int kThreads = 256;

enum TwMode : int { TW_NONE = 0, TW_POST = 2 };

struct RadixPlan {
  int n = 0;
  int r[kMaxStages] = {};
};

// Radix sequence of a pass of length L: radices 2 .. 13, the fewest stages
// (each costs a trip through shared memory), among those the smallest
// largest radix (registers), then the smallest sum; largest first.  n = 0
// for L = 1, -1 when L has a prime factor above 13.
RadixPlan radix_plan(int L);

struct alignas(16) PassGeom {
  int L;
  int nst;
  int rad[kMaxStages];
  int span[kMaxStages];       // points a block of stage s spans: L / (rad[0] .. rad[s-1])
  uint32_t mdiv[kMaxStages];  // ceil(2^32 / d): q / d = umulhi(q, mdiv) for q, d < 2^16, with d the
                              // butterflies of a block of stage s (the last stage: of a column); direct
                              // DFT: mdiv[0] for d = L / 2 + 1
  int threads;                // block size of the generic pass (mix_shape)
  int direct_j;               // direct DFT: output pairs a thread works on at a time (1 or kDirectJ)
  int vec_in, vec_out;        // complex64: two neighbouring columns are one aligned 16-byte vector
  int W;       // tile width along b0 (power of two)
  int logW;
  int pitch;   // shared-memory row pitch in elements (generic_pitch): direct DFT: element (p, w) at p*pitch + w
  int in_row;  // 1: lanes walk n at load (sn_in == 1)
  int out_row; // 1: lanes walk k at store (sk_out == 1)
  int64_t ext[4];
  int64_t sin[4];
  int64_t sout[4];
  int64_t sn_in, sk_out;
  int64_t tiles_w;  // ceil(ext[0] / W)
  int64_t ntiles;   // tiles_w * ext[1] * ext[2] * ext[3]
  // division of a tile index < 2^31 by d = tiles_w, ext[1], ext[2]:
  // (umulhi(x, mul) + x) >> sh (tile_idx), with mul and sh as in Granlund and
  // Montgomery, "Division by Invariant Integers using Multiplication" (1994)
  uint32_t tdiv_mul[3];
  uint32_t tdiv_sh[3];
  int tw_mode;
  int tw_dim;
  int tw_shift;     // two-level table split: m = (m >> shift, m & mask)
  int64_t tw_mask;
  int conj_in, conj_out;
  double scale;
  // Bluestein steps fused into a specialised pass (bits; 0 = none):
  //   BS_LOAD_MOD    load x (rows of bs_L, stride 1) into the virtual rows of
  //                  2^bs_logM points: conj_in(x[p]) * chirp[p] for p < bs_L,
  //                  0 beyond (replaces the modulate step before the pass);
  //   BS_STORE_MULH  store conj(y * H[p]) (the spectrum multiply after it);
  //   BS_STORE_DEMOD store conj_out(chirp[p] * conj(y) * scale) to rows of
  //                  bs_L points, p < bs_L only (the demodulate after it);
  // p is the point's position in its virtual row of 2^bs_logM points.
  int bs_mode;
  int bs_logM;
  int64_t bs_L;
  // Block map of a slab / pencil exchange fused into a specialised pass
  // (bits; 0 = none): the pass reads its input (MAP_LOAD) or writes its
  // output (MAP_STORE) in the per-peer block layout of the row-major array
  // [map_outer][2^map_log_n][2^map_log_inner] instead of the natural layout,
  // for an even partition of the n axis into blocks of 2^map_log_q: natural
  // index v = (o*n + k)*inner + i lives in the block layout at
  //   ((p*map_outer + o)*q + k % q)*inner + i,  p = k / q.
  int map_mode;
  int map_log_n, map_log_inner, map_log_q;
  int64_t map_outer;
};

// Indices of a tile: tile = tw + tiles_w * (i1 + ext[1] * (i2 + ext[2] * i3)).
struct TileIdx {
  int64_t tw, i1, i2, i3;
};

// Fields that follow from the others (radices, tile width, extents and
// strides) and the element size: stage spans, reciprocals, block size, vector
// flags.  Call once they are set.
void geom_derive(PassGeom& g, size_t elem);

// Dynamic shared memory of a generic (k_fft_mix) or direct-DFT pass.
size_t pass_smem(const PassGeom& g, size_t elem);

// Outputs a thread of a direct-DFT tile works on at a time: kDirectJ output
// pairs (k, L - k) of direct_cols columns, or one of one where the tiles are
// too few to keep an SM busy that way.
constexpr int kDirectJ = 4;
__host__ __device__ constexpr int direct_cols(size_t elem) { return elem == 8 ? 2 : 1; }

// Block size of a generic (k_fft_mix) or direct-DFT pass, and its estimated
// time (arbitrary units, comparable between widths of one pass).
struct MixShape {
  int threads;
  double time;
  int direct_j = 0;
};
MixShape mix_shape(const PassGeom& g, size_t elem);
MixShape direct_shape(const PassGeom& g, size_t elem);

#ifdef __CUDACC__
// First statement of every kernel launched by launch_chained (launch.h): waits
// until the kernels before it are complete and their writes visible.  No
// launch_dependents: let in early, the next kernel's blocks all went to the
// SMs that ran out of work first (1000 x 1000 complex64 15.7 -> 23.2 us).
__device__ __forceinline__ void chain_begin() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Run-time 64-bit divisions cost a few hundred instructions a thread ahead of
// the tile's first load; tile indices below 2^31 take multiplies instead.
__device__ __forceinline__ TileIdx tile_idx(const PassGeom& g, int64_t tile) {
  TileIdx x;
  if (g.ntiles < ((int64_t)1 << 31)) {
    const uint32_t t = (uint32_t)tile;
    const uint32_t q0 = (__umulhi(t, g.tdiv_mul[0]) + t) >> g.tdiv_sh[0];
    const uint32_t q1 = (__umulhi(q0, g.tdiv_mul[1]) + q0) >> g.tdiv_sh[1];
    const uint32_t q2 = (__umulhi(q1, g.tdiv_mul[2]) + q1) >> g.tdiv_sh[2];
    x.tw = t - q0 * (uint32_t)g.tiles_w;
    x.i1 = q0 - q1 * (uint32_t)g.ext[1];
    x.i2 = q1 - q2 * (uint32_t)g.ext[2];
    x.i3 = q2;
  } else {
    x.tw = tile % g.tiles_w;
    int64_t rest = tile / g.tiles_w;
    x.i1 = rest % g.ext[1];
    rest /= g.ext[1];
    x.i2 = rest % g.ext[2];
    x.i3 = rest / g.ext[2];
  }
  return x;
}
#endif

enum BsMode : int { BS_LOAD_MOD = 1, BS_STORE_MULH = 2, BS_STORE_DEMOD = 4 };
enum MapMode : int { MAP_LOAD = 1, MAP_STORE = 2 };

// Shared-memory row pitch (elements) of a generic or direct-DFT tile
// [L][pitch] whose rows hold W columns.  Direct-DFT passes address the tile by
// it: column-input ones put the W columns of a row on consecutive lanes, so a
// pitch of W keeps their half-warps of 8-byte accesses on distinct banks;
// row-input ones put consecutive rows on consecutive lanes, where with W >= 8
// a pitch of W would put a half-warp on one bank pair, so they get the odd
// pitch W + 1.  Radix passes (k_fft_mix) permute 16-byte chunks instead and
// use L * W elements of the tile; their row tiles of W >= 8 are still sized by
// this rule, one part in W more than they need.
__host__ __device__ constexpr int generic_pitch(int W, bool in_row) {
  return W == 1 ? 1 : ((in_row && W >= 8) ? W + 1 : W);
}

// Device pointers a pass reads besides its input/output.
template <typename C>
struct PassTables {
  const C* twL;            // w_L^m, m < L
  const uint16_t* p2k;     // digit-reversed position -> frequency index
  const uint16_t* k2p;     // frequency index -> position
  const C* tw_hi;          // w_N^{(m >> shift) << shift}
  const C* tw_lo;          // w_N^{m & mask}
  const void* tcB;         // tensor-core passes: split DFT matrix in shared-memory layout
  const C* bs_chirp;       // Bluestein fused into the pass (PassGeom::bs_mode)
  const C* bs_H;
};

}  // namespace shafft_sm100
