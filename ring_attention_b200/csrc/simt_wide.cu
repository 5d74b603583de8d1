// fp32 CUDA-core block kernels for head dims 17 to 128: the same contract as the kernels of
// simt_kernels.cu (any lengths, strides and score-mods, fp32 or bf16 inputs, all arithmetic in
// fp32), laid out for the FMA pipe.  What bounded the general kernels here was shared memory: a
// 4 x 4 patch per thread fed by eight 4-byte loads per 16 FMAs, both operands staged again for
// every 32 columns of the head dim, and the mask evaluated per pair on every tile, seen or not.
// Here whole operand tiles are staged once by asynchronous copies, a thread owns R x 4 scores and
// reads its operands as 16-byte vectors in products on packed fp32 pairs,
// and tiles are classified from position / segment ranges, so that only tiles which really mix
// visible and masked pairs look at pairs.
// Measured (device time, general kernels -> these): 1500 x 1500, b 2, h 4, fp32, no mask: d 64 forward
// 372 -> 245 us, backward 830 -> 399 us; d 128: 643 -> 456, 2088 -> 775 us; causal 1024, b 1, h 4, d 64:
// 177 -> 80, 387 -> 95 us.  What bounds it now is the FMA pipe together with the shared-memory reads (25 to
// 33 of 74 TFLOP/s): two (head dims above 64) to four warps per scheduler do not hide them all.
#include <math.h>

#include "common.cuh"
#include "host_util.h"
#include "ptx_sm100.cuh"
#include "tc_common.cuh"

namespace ra {

namespace {

using ptx::fma2;
using ptx::pack2;
using ptx::unpack2;

constexpr int BT = 64;          // rows of a key tile, and of a query tile in the backward
constexpr int PP = BT + 4;      // pitch of the P / dS tiles: 16-byte rows, spread over the banks
constexpr int kClsTiles = 256;  // tiles classified at a time

template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

// Rows [row0, row0 + ROWS) x D_PAD columns of an operand into shared memory as floats, zeros outside
// the tensor, in two halves so that the loads run under what stands between them: `begin` starts them,
// `end` (after it, the tile's old contents no longer read) leaves the tile complete.  fp32 rows on 16-byte
// boundaries go as asynchronous copies (the caller commits and waits); bf16 rows on 16-byte boundaries
// wait in registers, 16 bytes a load (one element a load, complete in `begin`, made the forward at head
// dims above 64 slower than the general kernel: 1000 x 1000, 8 heads, d 96: 370 against 268 us);
// anything else element by element, all in `begin`.
template <typename T, int D_PAD, int NT, int ROWS>
struct Stage {
  static constexpr int P = D_PAD + 4;
  static constexpr int N16 = sizeof(T) == 2 ? ROWS * (D_PAD / 8) / NT : 1;  // 16-byte loads of a thread
  static_assert(sizeof(T) == 4 || ROWS * (D_PAD / 8) % NT == 0, "uneven share");
  uint4 held[N16];
  bool holding = false;

  __device__ __forceinline__ void begin(float* dst, const T* base, int64_t sl, int row0, int nrows, int dim) {
    const bool aligned =
        ((reinterpret_cast<uintptr_t>(base) | (uintptr_t)(sl * sizeof(T)) | (uintptr_t)(dim * sizeof(T))) & 15) == 0;
    if (aligned) {
      if constexpr (sizeof(T) == 4) {
        for (int e = threadIdx.x; e < ROWS * (D_PAD / 4); e += NT) {
          const int r = e / (D_PAD / 4), c = (e % (D_PAD / 4)) * 4;
          const bool in = row0 + r < nrows && c < dim;
          const T* src = in ? base + (int64_t)(row0 + r) * sl + c : base;
          const uint32_t n = in ? 16u : 0u;  // bytes read; the rest of the 16 is zero-filled
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(ptx::smem_u32(dst + r * P + c)), "l"(src), "r"(n)
                       : "memory");
        }
      } else {
        holding = true;
#pragma unroll
        for (int i = 0; i < N16; ++i) {
          const int e = threadIdx.x + i * NT, r = e / (D_PAD / 8), c = (e % (D_PAD / 8)) * 8;
          held[i] = (row0 + r < nrows && c < dim) ? *reinterpret_cast<const uint4*>(base + (int64_t)(row0 + r) * sl + c)
                                                  : make_uint4(0u, 0u, 0u, 0u);
        }
      }
      return;
    }
    for (int e = threadIdx.x; e < ROWS * D_PAD; e += NT) {
      const int r = e / D_PAD, c = e % D_PAD;
      dst[r * P + c] = (row0 + r < nrows && c < dim) ? load_as_float(base + (int64_t)(row0 + r) * sl + c) : 0.f;
    }
  }
  __device__ __forceinline__ void end(float* dst) {
    if constexpr (sizeof(T) == 2) {
      if (!holding) return;
      holding = false;
#pragma unroll
      for (int i = 0; i < N16; ++i) {
        const int e = threadIdx.x + i * NT, r = e / (D_PAD / 8), c = (e % (D_PAD / 8)) * 8;
        const uint4 v = held[i];
        float4* to = reinterpret_cast<float4*>(dst + r * P + c);
        to[0] = make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16),
                            __uint_as_float(v.y & 0xffff0000u));
        to[1] = make_float4(__uint_as_float(v.z << 16), __uint_as_float(v.z & 0xffff0000u), __uint_as_float(v.w << 16),
                            __uint_as_float(v.w & 0xffff0000u));
      }
    }
  }
  __device__ __forceinline__ void whole(float* dst, const T* base, int64_t sl, int row0, int nrows, int dim) {
    begin(dst, base, sl, row0, nrows, dim);
    end(dst);
  }
};

// acc[i][j] += (even, odd) halves of sum_c A[R ty + i][c] * B[tx + 16 j][c] over the first `dim` columns
// (rounded up to 16: the rest are zeros)
template <int D_PAD, int R>
__device__ __forceinline__ void dot_tile(uint64_t (&acc)[R][4], const float* A, const float* B, int dim, int ty, int tx) {
  constexpr int P = D_PAD + 4;
  const int cols = (dim + 15) & ~15;
#pragma unroll 4
  for (int c = 0; c < cols; c += 4) {
    ulonglong2 a[R], b[4];
#pragma unroll
    for (int i = 0; i < R; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(A + (ty * R + i) * P + c);
#pragma unroll
    for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const ulonglong2*>(B + (tx + 16 * j) * P + c);
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = fma2(a[i].y, b[j].y, fma2(a[i].x, b[j].x, acc[i][j]));
  }
}

// out[i][2 cc + {0, 1}] += sum over the tile's 64 entries of W(i, k) * V[k][4 tx + 64 cc ...]; W row-major
// over k (a thread's rows R ty + i), four k at a time.
template <int D_PAD, int R>
__device__ __forceinline__ void mul_rows(uint64_t (&out)[R][D_PAD / 32], const float* W, const float* V, int ty, int tx) {
  constexpr int P = D_PAD + 4, CC = D_PAD / 64;
#pragma unroll 2
  for (int k = 0; k < BT; k += 4) {
    float4 w[R];
#pragma unroll
    for (int i = 0; i < R; ++i) w[i] = *reinterpret_cast<const float4*>(W + (ty * R + i) * PP + k);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      ulonglong2 v[CC];
#pragma unroll
      for (int cc = 0; cc < CC; ++cc) v[cc] = *reinterpret_cast<const ulonglong2*>(V + (k + u) * P + tx * 4 + 64 * cc);
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const float x = u == 0 ? w[i].x : (u == 1 ? w[i].y : (u == 2 ? w[i].z : w[i].w));
        const uint64_t x2 = pack2(x, x);
#pragma unroll
        for (int cc = 0; cc < CC; ++cc) {
          out[i][2 * cc] = fma2(x2, v[cc].x, out[i][2 * cc]);
          out[i][2 * cc + 1] = fma2(x2, v[cc].y, out[i][2 * cc + 1]);
        }
      }
    }
  }
}

// The same with W column-major: the thread's rows are W's columns R ty + i, the sum runs over W's rows.
template <int D_PAD, int R>
__device__ __forceinline__ void mul_cols(uint64_t (&out)[R][D_PAD / 32], const float* W, const float* V, int ty, int tx) {
  constexpr int P = D_PAD + 4, CC = D_PAD / 64;
#pragma unroll 4
  for (int k = 0; k < BT; ++k) {
    float w[R];
#pragma unroll
    for (int i = 0; i < R; i += 4) {
      const float4 t = *reinterpret_cast<const float4*>(W + k * PP + ty * R + i);
      w[i] = t.x, w[i + 1] = t.y, w[i + 2] = t.z, w[i + 3] = t.w;
    }
    ulonglong2 v[CC];
#pragma unroll
    for (int cc = 0; cc < CC; ++cc) v[cc] = *reinterpret_cast<const ulonglong2*>(V + k * P + tx * 4 + 64 * cc);
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const uint64_t x2 = pack2(w[i], w[i]);
#pragma unroll
      for (int cc = 0; cc < CC; ++cc) {
        out[i][2 * cc] = fma2(x2, v[cc].x, out[i][2 * cc]);
        out[i][2 * cc + 1] = fma2(x2, v[cc].y, out[i][2 * cc + 1]);
      }
    }
  }
}

// Score-mod arrays of one side (queries or keys) of a batch element.
struct ModSide {
  const int32_t *pos, *seg;
  const uint8_t* pre;
  int n;
};
__device__ __forceinline__ ModSide q_side(const ModParams& m, int bb, int lq) {
  const int64_t o = (int64_t)bb * lq;
  return {m.q_pos ? m.q_pos + o : nullptr, m.q_seg ? m.q_seg + o : nullptr, m.q_pre ? m.q_pre + o : nullptr, lq};
}
__device__ __forceinline__ ModSide kv_side(const ModParams& m, int bb, int lk) {
  const int64_t o = (int64_t)bb * lk;
  return {m.kv_pos ? m.kv_pos + o : nullptr, m.kv_seg ? m.kv_seg + o : nullptr, m.kv_pre ? m.kv_pre + o : nullptr, lk};
}
__device__ __forceinline__ ModRow mod_row(const ModSide& s, int i) {
  ModRow r{0, 0, false};
  if (i < s.n) {
    if (s.pos) r.pos = s.pos[i];
    if (s.seg) r.seg = s.seg[i];
    if (s.pre) r.pre = s.pre[i] != 0;
  }
  return r;
}

// Range summary of `rows` (at most 64) entries from row0; one warp, every lane gets it.
__device__ __forceinline__ TileMeta tile_meta(const ModSide& s, int row0, int rows, int lane) {
  TileMeta m{INT32_MAX, INT32_MIN, INT32_MAX, INT32_MIN, 0, 1, 0, 0};
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int i = row0 + lane + 32 * u;
    if (lane + 32 * u < rows && i < s.n) {
      const ModRow r = mod_row(s, i);
      m.pos_min = min(m.pos_min, r.pos), m.pos_max = max(m.pos_max, r.pos);
      m.seg_min = min(m.seg_min, r.seg), m.seg_max = max(m.seg_max, r.seg);
      m.pre_any |= r.pre, m.pre_all &= r.pre;
    }
  }
  m.pos_min = __reduce_min_sync(0xffffffffu, m.pos_min), m.pos_max = __reduce_max_sync(0xffffffffu, m.pos_max);
  m.seg_min = __reduce_min_sync(0xffffffffu, m.seg_min), m.seg_max = __reduce_max_sync(0xffffffffu, m.seg_max);
  m.pre_any = __any_sync(0xffffffffu, m.pre_any), m.pre_all = __all_sync(0xffffffffu, m.pre_all);
  return m;
}

constexpr uint32_t kPairMasks = RA_MOD_CAUSAL | RA_MOD_SEGMENT | RA_MOD_PREFIX | RA_MOD_WINDOW;

// Whether a (64 or fewer queries) x (64 keys) tile has a visible pair at all, pair by pair; one warp.
__device__ __noinline__ bool any_visible(uint32_t kinds, int32_t window, const ModSide& q, int q0, int nq, const ModSide& k, int k0) {
  const int lane = threadIdx.x & 31;
  bool any = false;
  for (int u = 0; u < 2; ++u) {
    const int c = k0 + lane + 32 * u;
    if (c >= k.n) continue;
    const ModRow kr = mod_row(k, c);
    for (int r = q0; r < min(q0 + nq, q.n); ++r) {
      const ModRow qr = mod_row(q, r);
      any = any || apply_mod(0.f, kinds & kPairMasks, window, 0.f, qr.pos, qr.seg, qr.pre, kr.pos, kr.seg, kr.pre) == 0.f;
    }
  }
  return __any_sync(0xffffffffu, any);
}

// Classes (classify_tiles) of tiles [first, first + kClsTiles) of one side against this CTA's tile of
// the other.  A dense bias keeps the NaN of rows that see no key (ring.py:146), which a skipped tile
// would not add: there the skip is decided pair by pair, as a promise about every pair.
template <int NT, bool kCtaHasQueries>
__device__ __forceinline__ void classify(uint8_t* cls, const ModParams& mod, const ModSide& q, const ModSide& k, int own0,
                                         int own_rows, int other_rows, int first, int n_tiles) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool masks = (mod.kinds & kPairMasks) != 0, dense = (mod.kinds & RA_MOD_DENSE) != 0;
  TileMeta own;
  if (masks) own = tile_meta(kCtaHasQueries ? q : k, own0, own_rows, lane);
  for (int t = warp; t < kClsTiles && first + t < n_tiles; t += NT / 32) {
    int c = 1;
    const int o0 = (first + t) * other_rows;
    if (masks) {
      const TileMeta other = tile_meta(kCtaHasQueries ? k : q, o0, other_rows, lane);
      c = kCtaHasQueries ? classify_tiles(mod.kinds, mod.window, own, other) : classify_tiles(mod.kinds, mod.window, other, own);
      if (dense && c == 2)
        c = kCtaHasQueries ? (any_visible(mod.kinds, mod.window, q, own0, own_rows, k, o0) ? 2 : 0)
                           : (any_visible(mod.kinds, mod.window, q, o0, other_rows, k, own0) ? 2 : 0);
    }
    if (lane == 0) cls[t] = (uint8_t)c;
  }
}

// Scores of a thread's patch (rows q0 + R ty + i, columns k0 + tx + 16 j): scaled, biased, masked.
template <int R>
__device__ __forceinline__ void score_patch(float (&s)[R][4], const uint64_t (&acc)[R][4], const ModParams& mod, const ModSide& q,
                                            const ModSide& k, float scale, float slope, bool pairs, int bb, int hh, int q0, int k0,
                                            int ty, int tx) {
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float lo, hi;
      unpack2(acc[i][j], lo, hi);
      s[i][j] = (lo + hi) * scale;
    }
  if (mod.kinds & RA_MOD_DENSE) {
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int row = q0 + ty * R + i, col = k0 + tx + 16 * j;
        if (row < q.n && col < k.n)
          s[i][j] += mod.bias[(int64_t)bb * mod.bsb + (int64_t)hh * mod.bsh + (int64_t)row * mod.bsq + col];
      }
  }
  if (pairs) {
    ModRow kr[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) kr[j] = mod_row(k, k0 + tx + 16 * j);
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const ModRow qr = mod_row(q, q0 + ty * R + i);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        s[i][j] = apply_mod(s[i][j], mod.kinds, mod.window, slope, qr.pos, qr.seg, qr.pre, kr[j].pos, kr[j].seg, kr[j].pre);
    }
  }
  if (k0 + BT > k.n) {
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (k0 + tx + 16 * j >= k.n) s[i][j] = -INFINITY;
  }
}

// ---------------------------------------------------------------------------------------
// Forward block (ring.py:58-76).  TY * 16 threads, R * TY query rows.  V of a tile arrives under its
// QK^T, K of the next tile under the softmax and PV.
// ---------------------------------------------------------------------------------------
template <typename T, int D_PAD, int R, int TY>
__global__ void __launch_bounds__(16 * TY, D_PAD == 64 ? 2 : 1) wide_fwd_kernel(const FwdParams p) {
  constexpr int P = D_PAD + 4, BM = R * TY, NT = 16 * TY, NO = D_PAD / 32;
  extern __shared__ __align__(16) float smem[];
  float* Qs = smem;
  float* Ks = Qs + BM * P;
  float* Vs = Ks + BT * P;
  float* Ps = Vs + BT * P;  // [BM][PP]
  __shared__ uint8_t cls[kClsTiles];

  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  // heaviest causal rows first
  const int q0 = (gridDim.x - 1 - blockIdx.x) * BM, hh = blockIdx.y, bb = blockIdx.z;
  const T* qb = (const T*)p.q.ptr + (int64_t)bb * p.q.sb + (int64_t)hh * p.q.sh;
  const T* kb = (const T*)p.k.ptr + (int64_t)bb * p.k.sb + (int64_t)hh * p.k.sh;
  const T* vb = (const T*)p.v.ptr + (int64_t)bb * p.v.sb + (int64_t)hh * p.v.sh;
  const int64_t row_base = ((int64_t)bb * p.h + hh) * p.lq;
  const ModSide qm = q_side(p.mod, bb, p.lq), km = kv_side(p.mod, bb, p.lk);
  const float slope = (p.mod.kinds & RA_MOD_ALIBI) ? p.mod.slopes[hh] : 0.f;

  float m_run[R], l_run[R];  // l: this thread's columns only, summed over the 16 threads of the row at the end
  uint64_t o_acc[R][NO];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int row = q0 + ty * R + i;
    const bool ld = !p.first && row < p.lq;
    m_run[i] = ld ? p.m[row_base + row] : -INFINITY;
    l_run[i] = (ld && tx == 0) ? p.l[row_base + row] : 0.f;
#pragma unroll
    for (int n = 0; n < NO; ++n) {
      float v[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int c = tx * 4 + 64 * (n >> 1) + 2 * (n & 1) + u;
        v[u] = (ld && c < p.dv) ? p.o[(row_base + row) * p.dv + c] : 0.f;
      }
      o_acc[i][n] = pack2(v[0], v[1]);
    }
  }
  Stage<T, D_PAD, NT, BM>().whole(Qs, qb, p.q.sl, q0, p.lq, p.dk);
  Stage<T, D_PAD, NT, BT> stage_k, stage_v;

  const int n_tiles = (p.lk + BT - 1) / BT;
  for (int base = 0; base < n_tiles; base += kClsTiles) {
    __syncthreads();  // the classes of the chunk before, and its buffers, are no longer read
    classify<NT, true>(cls, p.mod, qm, km, q0, BM, BT, base, n_tiles);
    __syncthreads();
    const int end = min(kClsTiles, n_tiles - base);
    auto next = [&](int t) {
      while (t < end && cls[t] == 0) ++t;
      return t;
    };
    int t = next(0);
    if (t < end) stage_k.whole(Ks, kb, p.k.sl, (base + t) * BT, p.lk, p.dk);
    cp_commit();
    while (t < end) {
      const int k0 = (base + t) * BT, tn = next(t + 1);
      stage_v.begin(Vs, vb, p.v.sl, k0, p.lk, p.dv);
      cp_commit();
      cp_wait<1>();
      __syncthreads();
      uint64_t acc[R][4];
#pragma unroll
      for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
      dot_tile<D_PAD, R>(acc, Qs, Ks, p.dk, ty, tx);
      stage_v.end(Vs);
      __syncthreads();
      if (tn < end) stage_k.begin(Ks, kb, p.k.sl, (base + tn) * BT, p.lk, p.dk);
      cp_commit();
      float s[R][4];
      score_patch<R>(s, acc, p.mod, qm, km, p.scale, slope, cls[t] == 2 || (p.mod.kinds & RA_MOD_ALIBI), bb, hh, q0, k0, ty, tx);
#pragma unroll
      for (int i = 0; i < R; ++i) {
        float mx = fmaxf(fmaxf(s[i][0], s[i][1]), fmaxf(s[i][2], s[i][3]));
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float m_new = fmaxf(m_run[i], mx);                                 // ring.py:63
        const float corr = (m_new == -INFINITY) ? 0.f : expf(m_run[i] - m_new);  // ring.py:65-66
        float rs = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float pe = (m_new == -INFINITY) ? 0.f : expf(s[i][j] - m_new);  // ring.py:68-69
          rs += pe;
          Ps[(ty * R + i) * PP + tx + 16 * j] = pe;
        }
        l_run[i] = corr * l_run[i] + rs;  // ring.py:75
        m_run[i] = m_new;
        const uint64_t c2 = pack2(corr, corr);
#pragma unroll
        for (int n = 0; n < NO; ++n) o_acc[i][n] = ptx::mul2(o_acc[i][n], c2);  // ring.py:72
      }
      stage_k.end(Ks);
      cp_wait<1>();
      __syncthreads();
      mul_rows<D_PAD, R>(o_acc, Ps, Vs, ty, tx);
      __syncthreads();
      t = tn;
    }
  }

#pragma unroll
  for (int i = 0; i < R; ++i) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) l_run[i] += __shfl_xor_sync(0xffffffffu, l_run[i], o);
    const int row = q0 + ty * R + i;
    if (row >= p.lq) continue;
    if (tx == 0) {
      p.m[row_base + row] = m_run[i];
      p.l[row_base + row] = l_run[i];
    }
#pragma unroll
    for (int n = 0; n < NO; ++n) {
      float v[2];
      unpack2(o_acc[i][n], v[0], v[1]);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int c = tx * 4 + 64 * (n >> 1) + 2 * (n & 1) + u;
        if (c < p.dv) p.o[(row_base + row) * p.dv + c] = v[u];
      }
    }
  }
}

__device__ __forceinline__ bool rows_aligned(const float* base, int dim) {
  return ((reinterpret_cast<uintptr_t>(base) | (uintptr_t)(dim * 4)) & 15) == 0;
}
// Adds x to columns [c, c + 4) of a row of `dim` floats; `vec`: rows are 16-byte aligned; `atomic`: other
// CTAs add to the same row.
__device__ __forceinline__ void add4(float* row, int c, int dim, const float (&x)[4], bool vec, bool atomic) {
  if (vec) {
    if (c >= dim) return;
    if (atomic) {
      asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(row + c), "f"(x[0]), "f"(x[1]), "f"(x[2]), "f"(x[3])
                   : "memory");
    } else {
      float4 a = *reinterpret_cast<float4*>(row + c);
      a.x += x[0], a.y += x[1], a.z += x[2], a.w += x[3];
      *reinterpret_cast<float4*>(row + c) = a;
    }
  } else {
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (c + u < dim) {
        if (atomic) atomicAdd(row + c + u, x[u]);
        else row[c + u] += x[u];
      }
  }
}

// Adds a thread's R x D_PAD/32 pairs to rows row0 + i of an fp32 [.., rows, dim] accumulator.
template <int D_PAD, int R>
__device__ __forceinline__ void add_rows(float* base, const uint64_t (&v)[R][D_PAD / 32], int row0, int nrows, int dim, int tx,
                                         bool atomic) {
  const bool vec = rows_aligned(base, dim);
#pragma unroll
  for (int i = 0; i < R; ++i) {
    if (row0 + i >= nrows) continue;
#pragma unroll
    for (int cc = 0; cc < D_PAD / 64; ++cc) {
      float x[4];
      unpack2(v[i][2 * cc], x[0], x[1]);
      unpack2(v[i][2 * cc + 1], x[2], x[3]);
      add4(base + (int64_t)(row0 + i) * dim, tx * 4 + 64 * cc, dim, x, vec, atomic);
    }
  }
}

// One split's dK and dV of a key tile: [dK, dV][64][D_PAD].  `used` (an array behind the parts) says which
// parts hold anything: a mask leaves some splits without a visible tile.
template <int D_PAD>
constexpr int64_t kPartFloats = 2 * BT * D_PAD;
template <int D_PAD, int R>
__device__ __forceinline__ void put_rows(float* part, const uint64_t (&v)[R][D_PAD / 32], int row0, int tx) {
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int cc = 0; cc < D_PAD / 64; ++cc)
      *reinterpret_cast<ulonglong2*>(part + (row0 + i) * D_PAD + tx * 4 + 64 * cc) =
          make_ulonglong2(v[i][2 * cc], v[i][2 * cc + 1]);
}

// ---------------------------------------------------------------------------------------
// Backward block (ring.py:140-157).  A CTA owns 64 keys and every `splits`-th query tile: a short
// sequence has too few key tiles for 148 SMs, and the tiles one of them would walk alone are a
// serial chain.  With one split a CTA adds its dK and dV itself; with more each leaves them in a part of its
// own and sum_parts_kernel adds the parts in a fixed order, so that repeated calls give the same bits
// (dQ is added atomically and does not).  Atomic additions of dK and dV instead cost the same; the splits as a
// cluster with the sums in shared memory held every SM until a tile's slowest split was done (causal 1k, d 128:
// 206 against 134 us; a window of 125 of 1000 tokens: 279 against 134 us).
// The next Q and dO tiles arrive under the dQ product.
// ---------------------------------------------------------------------------------------
template <typename T, int D_PAD, int TY>
__global__ void __launch_bounds__(16 * TY, D_PAD == 64 ? 2 : 1) wide_bwd_kernel(const BwdParams p, int splits, float* parts, int* used) {
  constexpr int P = D_PAD + 4, R = BT / TY, NT = 16 * TY, NO = D_PAD / 32;
  extern __shared__ __align__(16) float smem[];
  float* Qs = smem;
  float* Gs = Qs + BT * P;  // dO
  float* Ks = Gs + BT * P;
  float* Vs = Ks + BT * P;
  float* Ps = Vs + BT * P;   // [64 q][PP]
  float* Ds = Ps + BT * PP;  // [64 q][PP]
  __shared__ uint8_t cls[kClsTiles];
  __shared__ float sL[BT], sDelta[BT];

  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int k0 = (int)(blockIdx.x / splits) * BT, split = blockIdx.x % splits, hh = blockIdx.y, bb = blockIdx.z;
  const T* qb = (const T*)p.q.ptr + (int64_t)bb * p.q.sb + (int64_t)hh * p.q.sh;
  const T* kb = (const T*)p.k.ptr + (int64_t)bb * p.k.sb + (int64_t)hh * p.k.sh;
  const T* vb = (const T*)p.v.ptr + (int64_t)bb * p.v.sb + (int64_t)hh * p.v.sh;
  const T* gb = (const T*)p.dout.ptr + (int64_t)bb * p.dout.sb + (int64_t)hh * p.dout.sh;
  const int64_t qrow_base = ((int64_t)bb * p.h + hh) * p.lq, krow_base = ((int64_t)bb * p.h + hh) * p.lk;
  const ModSide qm = q_side(p.mod, bb, p.lq), km = kv_side(p.mod, bb, p.lk);
  const float slope = (p.mod.kinds & RA_MOD_ALIBI) ? p.mod.slopes[hh] : 0.f;
  const bool dense = (p.mod.kinds & RA_MOD_DENSE) != 0;

  uint64_t dk_acc[R][NO], dv_acc[R][NO];  // rows: keys R ty + i
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int n = 0; n < NO; ++n) dk_acc[i][n] = dv_acc[i][n] = 0ull;
  Stage<T, D_PAD, NT, BT>().whole(Ks, kb, p.k.sl, k0, p.lk, p.dk_dim);
  Stage<T, D_PAD, NT, BT>().whole(Vs, vb, p.v.sl, k0, p.lk, p.dv_dim);

  bool any = false;
  const int n_tiles = (p.lq + BT - 1) / BT;
  for (int base = 0; base < n_tiles; base += kClsTiles) {
    __syncthreads();
    classify<NT, false>(cls, p.mod, qm, km, k0, BT, BT, base, n_tiles);
    __syncthreads();
    const int end = min(kClsTiles, n_tiles - base);
    auto next = [&](int t) {  // first tile >= t of this split with a visible pair
      while (t < end && (cls[t] == 0 || (base + t) % splits != split)) ++t;
      return t;
    };
    float L_next = 0.f, delta_next = 0.f;
    auto stage_q = [&](int t) {
      const int q0 = (base + t) * BT;
      Stage<T, D_PAD, NT, BT>().whole(Qs, qb, p.q.sl, q0, p.lq, p.dk_dim);
      Stage<T, D_PAD, NT, BT>().whole(Gs, gb, p.dout.sl, q0, p.lq, p.dv_dim);
      if (tid < BT && q0 + tid < p.lq) {
        L_next = p.lse[qrow_base + q0 + tid];
        delta_next = p.delta[qrow_base + q0 + tid];
      }
    };
    int t = next(0);
    if (t < end) stage_q(t);
    cp_commit();
    any = any || t < end;
    while (t < end) {
      const int q0 = (base + t) * BT, tn = next(t + 1);
      if (tid < BT) {
        sL[tid] = L_next;
        sDelta[tid] = delta_next;
      }
      cp_wait<0>();
      __syncthreads();
      uint64_t acc[R][4], dacc[R][4];  // rows: queries R ty + i, columns: keys tx + 16 j
#pragma unroll
      for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = dacc[i][j] = 0ull;
      dot_tile<D_PAD, R>(acc, Qs, Ks, p.dk_dim, ty, tx);   // S = Q K^T
      dot_tile<D_PAD, R>(dacc, Gs, Vs, p.dv_dim, ty, tx);  // dP = dO V^T
      float s[R][4];
      score_patch<R>(s, acc, p.mod, qm, km, p.scale, slope, cls[t] == 2 || (p.mod.kinds & RA_MOD_ALIBI), bb, hh, q0, k0, ty, tx);
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const int r = ty * R + i;
        const float L = sL[r], dl = sDelta[r];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float pe = 0.f, ds = 0.f;
          if (q0 + r < p.lq && k0 + tx + 16 * j < p.lk) {
            // ring.py:146.  With a dense bias tile a row that saw no key (L = -inf) gives
            // exp(-inf + inf) = NaN exactly like the reference; the compiled-in masks define
            // p = 0 on a masked pair, so such rows contribute nothing.
            const bool masked = s[i][j] == -INFINITY && !dense;
            float lo, hi;
            unpack2(dacc[i][j], lo, hi);
            pe = masked ? 0.f : expf(s[i][j] - L);
            ds = masked ? 0.f : pe * ((lo + hi) - dl) * p.scale;  // ring.py:152
          }
          Ps[r * PP + tx + 16 * j] = pe;
          Ds[r * PP + tx + 16 * j] = ds;
        }
      }
      __syncthreads();
      mul_cols<D_PAD, R>(dv_acc, Ps, Gs, ty, tx);  // dV += P^T dO (ring.py:148)
      mul_cols<D_PAD, R>(dk_acc, Ds, Qs, ty, tx);  // dK += dS^T Q (ring.py:155)
      __syncthreads();
      if (tn < end) stage_q(tn);
      cp_commit();
      uint64_t dq[R][NO];
#pragma unroll
      for (int i = 0; i < R; ++i)
#pragma unroll
        for (int n = 0; n < NO; ++n) dq[i][n] = 0ull;
      mul_rows<D_PAD, R>(dq, Ds, Ks, ty, tx);  // dQ = dS K (ring.py:154)
      add_rows<D_PAD, R>(p.dq + qrow_base * p.dk_dim, dq, q0 + ty * R, p.lq, p.dk_dim, tx, true);
      t = tn;
    }
  }
  cp_wait<0>();
  if (splits == 1) {
    add_rows<D_PAD, R>(p.dk + krow_base * p.dk_dim, dk_acc, k0 + ty * R, p.lk, p.dk_dim, tx, false);
    add_rows<D_PAD, R>(p.dv + krow_base * p.dv_dim, dv_acc, k0 + ty * R, p.lk, p.dv_dim, tx, false);
    return;
  }
  const int64_t part = ((int64_t)bb * p.h + hh) * gridDim.x + blockIdx.x;
  if (tid == 0) used[part] = any;
  if (!any) return;
  put_rows<D_PAD, R>(parts + part * kPartFloats<D_PAD>, dk_acc, ty * R, tx);
  put_rows<D_PAD, R>(parts + part * kPartFloats<D_PAD> + BT * D_PAD, dv_acc, ty * R, tx);
}

// dK, dV += the parts of a key tile.  Four groups of 64 threads add every fourth part each and meet in shared memory:
// an order that depends on the number of splits alone.  blockIdx: key tile, 64 of its 16-byte chunks, (batch, head).
template <int D_PAD>
__global__ void __launch_bounds__(256) sum_parts_kernel(const BwdParams p, int splits, const float* __restrict__ parts,
                                                        const int* __restrict__ used) {
  __shared__ float4 sums[4][64];
  const int k0 = blockIdx.x * BT, i = threadIdx.x & 63, g = threadIdx.x >> 6;
  const int64_t bh = blockIdx.z, first = (bh * gridDim.x + blockIdx.x) * splits;
  const int e = blockIdx.y * 64 + i;  // chunk of [dK, dV][64][D_PAD / 4]
  const float* from = parts + first * kPartFloats<D_PAD> + e * 4;
  float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
  for (int k = g; k < splits; k += 4)
    if (used[first + k]) {
      const float4 v = *reinterpret_cast<const float4*>(from + k * kPartFloats<D_PAD>);
      x.x += v.x, x.y += v.y, x.z += v.z, x.w += v.w;
    }
  sums[g][i] = x;
  __syncthreads();
  const int which = e / (BT * D_PAD / 4), r = e / (D_PAD / 4) % BT, c = e % (D_PAD / 4) * 4;
  const int dim = which ? p.dv_dim : p.dk_dim;
  if (g || k0 + r >= p.lk || c >= dim) return;
  float y[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int j = 0; j < 4; ++j) y[0] += sums[j][i].x, y[1] += sums[j][i].y, y[2] += sums[j][i].z, y[3] += sums[j][i].w;
  float* base = (which ? p.dv : p.dk) + bh * p.lk * dim;
  add4(base + (int64_t)(k0 + r) * dim, c, dim, y, rows_aligned(base, dim), false);
}

// Query splits of a backward: until there are about four CTAs per SM, each with a query tile of its own to look
// at (a mask may leave some without a visible one).
int bwd_splits(int b, int h, int lq, int lk) {
  const int64_t ctas = (int64_t)((lk + BT - 1) / BT) * h * b, q_tiles = (lq + BT - 1) / BT;
  int64_t splits = (4 * 148 + ctas - 1) / ctas;
  if (splits > q_tiles) splits = q_tiles;
  return splits < 1 ? 1 : (int)splits;
}
size_t bwd_parts(int b, int h, int lq, int lk) {
  const int splits = bwd_splits(b, h, lq, lk);
  return splits == 1 ? 0 : (size_t)((lk + BT - 1) / BT) * h * b * splits;
}

template <typename T, int D_PAD, int R, int TY>
cudaError_t launch_fwd(const FwdParams& p, cudaStream_t s) {
  constexpr int BM = R * TY;
  constexpr size_t smem = sizeof(float) * ((BM + 2 * BT) * (D_PAD + 4) + BM * PP);
  auto kern = wide_fwd_kernel<T, D_PAD, R, TY>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  kern<<<dim3((p.lq + BM - 1) / BM, p.h, p.b), 16 * TY, smem, s>>>(p);
  count_launch();
  return cudaGetLastError();
}

template <typename T, int D_PAD, int TY>
cudaError_t launch_bwd(const BwdParams& p, cudaStream_t s) {
  constexpr size_t smem = sizeof(float) * (4 * BT * (D_PAD + 4) + 2 * BT * PP);
  auto kern = wide_bwd_kernel<T, D_PAD, TY>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const unsigned k_tiles = (p.lk + BT - 1) / BT;
  int splits = bwd_splits(p.b, p.h, p.lq, p.lk);
  float* parts = nullptr;
  int* used = nullptr;
  if (splits > 1) {
    const size_t n = bwd_parts(p.b, p.h, p.lq, p.lk);
    if (scratch_alloc((void**)&parts, n * (kPartFloats<D_PAD> * sizeof(float) + sizeof(int)), s) == cudaSuccess) {
      used = reinterpret_cast<int*>(parts + n * kPartFloats<D_PAD>);
    } else {  // no memory for the parts: whole key tiles, which need none
      cudaGetLastError();
      parts = nullptr;
      splits = 1;
    }
  }
  kern<<<dim3(k_tiles * splits, p.h, p.b), 16 * TY, smem, s>>>(p, splits, parts, used);
  count_launch();
  e = cudaGetLastError();
  if (parts) {
    if (e == cudaSuccess) {
      sum_parts_kernel<D_PAD><<<dim3(k_tiles, kPartFloats<D_PAD> / 4 / 64, p.b * p.h), 256, 0, s>>>(p, splits, parts, used);
      count_launch();
      e = cudaGetLastError();
    }
    cudaFreeAsync(parts, s);
  }
  return e;
}

template <typename T>
cudaError_t dispatch_fwd(const FwdParams& p, cudaStream_t s) {
  // 64 query rows per CTA when that fills the chip, 32 otherwise; 256 threads, since more warps hide
  // more of the shared-memory latency than larger patches save (2048 x 2048: 337 -> 320 us, causal 1k:
  // 91 -> 83 us against 128 threads)
  const bool small = (int64_t)((p.lq + 63) / 64) * p.h * p.b < 148;
  if (max(p.dk, p.dv) <= 64) return small ? launch_fwd<T, 64, 2, 16>(p, s) : launch_fwd<T, 64, 4, 16>(p, s);
  return small ? launch_fwd<T, 128, 2, 16>(p, s) : launch_fwd<T, 128, 4, 16>(p, s);
}

template <typename T>
cudaError_t dispatch_bwd(const BwdParams& p, cudaStream_t s) {
  if (max(p.dk_dim, p.dv_dim) > 64) return launch_bwd<T, 128, 16>(p, s);
  // few key tiles: 256 threads shorten a CTA's chain (causal 1k: 117 -> 105 us); many: 128 threads read
  // less shared memory per FMA (2048 x 2048: 710 us against 755)
  const bool small = (int64_t)((p.lk + BT - 1) / BT) * p.h * p.b < 148;
  return small ? launch_bwd<T, 64, 16>(p, s) : launch_bwd<T, 64, 8>(p, s);
}

}  // namespace

cudaError_t simt_wide_fwd(const FwdParams& p, int dtype, cudaStream_t s) {
  return dtype == RA_DTYPE_F32 ? dispatch_fwd<float>(p, s) : dispatch_fwd<__nv_bfloat16>(p, s);
}
size_t simt_bwd_scratch_bytes(int b, int h, int lq, int lk, int dk, int dv) {
  if (!simt_wide_dims(dk, dv)) return 0;
  const size_t floats = dk > 64 || dv > 64 ? kPartFloats<128> : kPartFloats<64>;
  return bwd_parts(b, h, lq, lk) * (floats * sizeof(float) + sizeof(int));
}
cudaError_t simt_wide_bwd(const BwdParams& p, int dtype, cudaStream_t s) {
  return dtype == RA_DTYPE_F32 ? dispatch_bwd<float>(p, s) : dispatch_bwd<__nv_bfloat16>(p, s);
}

}  // namespace ra
