// Pieces shared by the tcgen05 forward and backward block kernels: per-tile mask
// metadata, tile classification, TMA descriptor construction, the device status word.
#pragma once
#include <cuda.h>

#include "common.cuh"
#include "ptx_sm100.cuh"

namespace ra {

constexpr int kTileRows = 128;     // rows of one q tile / one kv tile
constexpr int kMaxTiles = 4096;    // most tiles one block (shard) may have along either axis
__host__ __device__ constexpr int tiles_of(int rows) { return (rows + kTileRows - 1) / kTileRows; }

constexpr uint32_t kMaskKinds = RA_MOD_CAUSAL | RA_MOD_SEGMENT | RA_MOD_PREFIX | RA_MOD_WINDOW;
// Score-mods that read the tile summaries (ALiBi reads pos_contig to choose its in-loop form).
constexpr uint32_t kMetaKinds = kMaskKinds | RA_MOD_ALIBI;

// Bits [first, 32 * kWords) / [0, last) of a run of kWords 32-bit words, as this word's part.
__device__ __forceinline__ uint32_t bits_from(int first) {
  return first <= 0 ? 0xffffffffu : (first >= 32 ? 0u : 0xffffffffu << first);
}
__device__ __forceinline__ uint32_t bits_below(int last) { return ~bits_from(last); }

// The bf16 pair in `hi` (the rounded x0, x1) leaves a remainder; this is that remainder as a second
// bf16 pair: hi + lo holds 16 bits of each value.  A value that rounded to infinity keeps lo = 0.
__device__ __forceinline__ uint32_t pack_bf16_rest(uint32_t hi, float x0, float x1) {
  const float h0 = __uint_as_float(hi << 16), h1 = __uint_as_float(hi & 0xffff0000u);
  const float r0 = fabsf(h0) == INFINITY ? 0.f : x0 - h0, r1 = fabsf(h1) == INFINITY ? 0.f : x1 - h1;
  return ptx::pack_bf16(r0, r1);
}

// Which of the 32 * kWords columns of a tile this thread's row sees under the mask kinds: bit c of
// the words = column c.  kRowIsQuery: the row is a query and the columns are keys (forward); else
// the row is a key and the columns are queries (backward, transposed tiles).  Only tiles that mix
// visible and masked pairs come here; the kernels then clear the masked scores in registers.
// What bounds it is issue slots on the path between a score tile and its softmax, so nothing is
// done per (row, column) pair that can be done per row or per column:
//   * columns at contiguous positions (`col_contig`: column c is at col_pos0 + c): causal and
//     window masks are one range of columns per row;
//   * prefix flags: one ballot per 32 columns, shared by all rows of the warp;
//   * segment ids: one ballot per 32 columns for every DISTINCT id among the warp's 32 rows (one
//     or two with packed documents, 32 at worst);
//   * scattered positions: one shuffle and compare per column.
// (The form before this one evaluated the mask per pair on scores in TMEM: about 17,000 cycles for
// a 128 x 128 forward tile, several times the rest of the tile's softmax.)
// All 32 lanes of the warp call it; the column arrays point at the tile's first column and hold `ncols`
// entries from there: columns past them (a ragged last tile) are not read and count as masked.
template <bool kRowIsQuery, int kWords>
__device__ __forceinline__ void visible_columns(uint32_t (&vis)[kWords], uint32_t kinds, int32_t window, int32_t row_pos,
                                                int32_t row_seg, bool row_pre, const int32_t* col_pos,
                                                const int32_t* col_seg, const uint8_t* col_pre, int32_t col_pos0,
                                                bool col_contig, int ncols = 32 * kWords) {
  const int lane = threadIdx.x & 31;
  auto col = [&](int w) { return min(32 * w + lane, ncols - 1); };  // this lane's column of word w, kept inside
  const bool order = (kinds & (RA_MOD_CAUSAL | RA_MOD_PREFIX)) != 0, win = (kinds & RA_MOD_WINDOW) != 0;
  if (!(order || win)) {
#pragma unroll
    for (int w = 0; w < kWords; ++w) vis[w] = 0xffffffffu;
  } else if (col_contig) {
    // columns [first, last) by position order, cut to the window below
    const long long rel = (long long)row_pos - (long long)col_pos0;  // column index at the row's own position
    long long first = 0, last = 32 * kWords;      // causal range
    long long wfirst = 0, wlast = 32 * kWords;    // window range
    if (kRowIsQuery) {
      last = rel + 1;
      wfirst = rel - window + 1;
    } else {
      first = rel;
      wlast = rel + window;
    }
    auto clip = [](long long x) { return (int)(x < 0 ? 0 : (x > 32 * kWords ? 32 * kWords : x)); };
    const int f = order ? clip(first) : 0, l = order ? clip(last) : 32 * kWords;
    const int wf = win ? clip(wfirst) : 0, wl = win ? clip(wlast) : 32 * kWords;
#pragma unroll
    for (int w = 0; w < kWords; ++w) {
      uint32_t m = bits_from(f - 32 * w) & bits_below(l - 32 * w);
      if (kinds & RA_MOD_PREFIX) {
        const uint32_t pre = __ballot_sync(0xffffffffu, col_pre[col(w)] != 0);
        if (row_pre) m |= pre;
      }
      vis[w] = m & bits_from(wf - 32 * w) & bits_below(wl - 32 * w);
    }
  } else {
#pragma unroll
    for (int w = 0; w < kWords; ++w) {
      const int32_t cp = col_pos[col(w)];
      uint32_t m = 0xffffffffu, near = 0xffffffffu;
#pragma unroll 1
      for (int c = 0; c < 32; ++c) {
        const int32_t p = __shfl_sync(0xffffffffu, cp, c);
        const int32_t qp = kRowIsQuery ? row_pos : p, kp = kRowIsQuery ? p : row_pos;
        if (order && kp > qp) m &= ~(1u << c);
        if (win && qp - kp >= window) near &= ~(1u << c);
      }
      if (kinds & RA_MOD_PREFIX) {
        const uint32_t pre = __ballot_sync(0xffffffffu, col_pre[col(w)] != 0);
        if (row_pre) m |= pre;
      }
      vis[w] = m & near;
    }
  }
  if (kinds & RA_MOD_SEGMENT) {
    int32_t cs[kWords];
#pragma unroll
    for (int w = 0; w < kWords; ++w) cs[w] = col_seg[col(w)];
    uint32_t todo = 0xffffffffu;  // rows of the warp whose id has not been looked up yet
#pragma unroll 1
    while (todo) {
      const int32_t id = __shfl_sync(0xffffffffu, row_seg, __ffs(todo) - 1);
      const bool mine = row_seg == id;
#pragma unroll
      for (int w = 0; w < kWords; ++w) {
        const uint32_t same = __ballot_sync(0xffffffffu, cs[w] == id);
        if (mine) vis[w] &= same;
      }
      todo &= ~__ballot_sync(0xffffffffu, mine);
    }
  }
#pragma unroll
  for (int w = 0; w < kWords; ++w) vis[w] &= bits_below(ncols - 32 * w);
}

// Adds a per-pair bias to raw (unscaled) scores that sit in TMEM, in place: this thread's TMEM
// lane, `ncols` columns (a multiple of 16) from `taddr`.  Two biases come this way: ALiBi over
// columns at scattered positions (over contiguous ones it is FMAs in the kernels' loops, one per score in
// the forward and two in the backward), and
// a dense bias tile (RA_MOD_DENSE: the materialised bias_fn result of ring.py:60-61).  Both are
// added divided by the softmax scale, so that the main loops, which multiply by the scale, see
// exactly scale * s + bias.  A rolled loop on purpose: the main loops stay small enough for the
// instruction cache.  The next 16 columns are in flight while the current 16 are worked on.
// kRowIsQuery: as above.  `bias` points at this thread's row and the tile's first column,
// consecutive columns are `bias_col_stride` floats apart (1 in the forward, where a thread reads
// 64 contiguous bytes per 16 columns; the bias row stride in the backward, where the lanes of a
// warp read consecutive floats of one bias row).  `ncols_valid`: positions past it are not read.
template <bool kRowIsQuery>
__device__ __noinline__ void bias_scores_tmem(uint32_t taddr, int ncols, bool alibi, float alibi_over_scale,
                                              int32_t row_pos, const int32_t* col_pos, const float* bias,
                                              int64_t bias_col_stride, float inv_scale, int ncols_valid) {
  uint32_t cur[16], nxt[16];
  ptx::tmem_ld16(taddr, cur);
#pragma unroll 1
  for (int c0 = 0; c0 < ncols; c0 += 16) {
    ptx::tc_wait_ld();
    const bool more = c0 + 16 < ncols;
    if (more) ptx::tmem_ld16(taddr + c0 + 16, nxt);
    if (bias) {
      float bv[16];
      if constexpr (kRowIsQuery) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float4 b4 = __ldg(reinterpret_cast<const float4*>(bias + c0) + j);
          bv[4 * j] = b4.x, bv[4 * j + 1] = b4.y, bv[4 * j + 2] = b4.z, bv[4 * j + 3] = b4.w;
        }
      } else {
#pragma unroll
        for (int e = 0; e < 16; ++e) bv[e] = __ldg(bias + (int64_t)(c0 + e) * bias_col_stride);
      }
#pragma unroll
      for (int e = 0; e < 16; ++e) cur[e] = __float_as_uint(fmaf(bv[e], inv_scale, __uint_as_float(cur[e])));
    }
    if (alibi) {
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const int32_t cp = __ldg(col_pos + min(c0 + e, ncols_valid - 1));
        const int32_t dist = kRowIsQuery ? row_pos - cp : cp - row_pos;  // q_pos - kv_pos
        cur[e] = __float_as_uint(fmaf(-alibi_over_scale, (float)dist, __uint_as_float(cur[e])));
      }
    }
    ptx::tmem_st16(taddr + c0, cur);
    if (more) {
      ptx::tc_wait_ld();
#pragma unroll
      for (int e = 0; e < 16; ++e) cur[e] = nxt[e];
    }
  }
  ptx::tc_wait_st();
}

// Host side -----------------------------------------------------------------------------
// Tensor map over a [b, len, h, d] bf16 tensor with box {64 elements of d, 1 head, 128 rows,
// 1 batch} and the 128-byte swizzle the UMMA descriptors expect.  Returns false (with a
// reason) when the driver refuses the layout.
bool make_tile_map(CUtensorMap* map, const TensorView& t, int b, int len, int h, int d, int box_rows,
                   const char** why);

// Launches the kernel that fills TileMeta[b][n_tiles] for the query side and the key side.
cudaError_t launch_tile_meta(TileMeta* out_q, TileMeta* out_kv, const ModParams& m, int b, int lq, int lk, cudaStream_t s);

// Stream-ordered scratch (tile summaries) from a memory pool of this library, one per device,
// that keeps what it has been given: the default pool hands unused memory back to the driver at
// every synchronisation, and the next call's allocation then costs milliseconds on the stream.
// Free with cudaFreeAsync on the same stream.
cudaError_t scratch_alloc(void** ptr, size_t bytes, cudaStream_t s);

// Device status word of the current device (bit set = a bounded wait ran out).
unsigned int* device_status_word();

// Failure codes OR-ed into the status word.
constexpr uint32_t kStFwdProducer = 1u << 0, kStFwdMma = 1u << 1, kStFwdSoftmax = 1u << 2;
constexpr uint32_t kStBwdProducer = 1u << 8, kStBwdMma = 1u << 9, kStBwdCompute = 1u << 10;

}  // namespace ra
