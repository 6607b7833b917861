// Warp-level matrix multiply-accumulate for the pipelined kernels' tiles of at most eight tokens.
//
// A tile of eight tokens is eight columns of mma.sync.m16n8k16: adapter rows (shrink) or outputs (expand) are the
// sixteen rows, tokens the columns, FP32 accumulators.  tcgen05 wants 64 or 128 rows of M with its operands in
// descriptor layouts; here the operands of one instruction are 16 scattered rows against a handful of tokens that sit
// in a stage as the bulk copies left them, and the consumers are bound by the instructions they issue, not by the
// tensor pipe: one mma replaces 64 fused multiply-adds per lane.  Against 64-bit results the error of both forms is that
// of the 16-bit outputs (2.2e-4 to 2.6e-4 in fp16, 1.9e-3 in bf16 on every batch measured).  Chains are short (32 values of
// k, mma_k32), so that the FP32 sums behind them are no worse either: intermediates of fp16 batches that are not the
// nearest value to the 64-bit sum, per thousand at hidden 4096 / 5120 / 8192: FMA 0.8 / 0.9 / 0.9, whole rows in one
// accumulator 1.1 / 1.3 / 1.6, now 0.7 / 0.7 / 0.8.
//
// The dot product's order over k is free, so a fragment takes its k values where they lie: lane (g, t) = (lane / 4,
// lane % 4) loads whole 16-byte vectors of its row and the token operand is loaded the same way, which makes both
// agree on which k sits in which slot.  An output's bits depend on its own row and its own token only - not on how many
// tokens share the tile or where the row sits in the block - so planned, per-token and tensor-parallel calls agree.
#pragma once

#include "lora_common.cuh"

namespace slora {

// d (16 x 8, FP32) += a (16 x 16) * b (16 x 8).  Lane (g, t): a0 / a2 = row g, a1 / a3 = row g + 8 (two k values each;
// a2 / a3 the second half of k), b0 / b1 = column g, d0, d1 = row g columns 2t, 2t + 1, d2, d3 = row g + 8.
template <typename T>
__device__ __forceinline__ void mma_k16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                        uint32_t b1);
template <>
__device__ __forceinline__ void mma_k16<__half>(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                                uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <>
__device__ __forceinline__ void mma_k16<__nv_bfloat16>(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                                       uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, "
      "%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// d = a * b: the first of a chain.
template <typename T>
__device__ __forceinline__ void mma_k16_first(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                              uint32_t b1);
template <>
__device__ __forceinline__ void mma_k16_first<__half>(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                                      uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, "
      "%10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
template <>
__device__ __forceinline__ void mma_k16_first<__nv_bfloat16>(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                                             uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, "
      "%10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
// The 32 values of k that a 16-byte vector per lane holds, from zero: u, v = this lane's vectors of rows g and g + 8, b = of
// column g.  Longer sums add such results with additions of their own: an mma truncates what it adds to its accumulator.
template <typename T>
__device__ __forceinline__ void mma_k32(float (&d)[4], const uint4& u, const uint4& v, const uint4& b) {
  mma_k16_first<T>(d, u.x, v.x, u.y, v.y, b.x, b.y);
  mma_k16<T>(d, u.z, v.z, u.w, v.w, b.z, b.w);
}
// The same with k = 8: a0 = row g, a1 = row g + 8, b0 = column g (two k values each).
template <typename T>
__device__ __forceinline__ void mma_k8(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0);
template <>
__device__ __forceinline__ void mma_k8<__half>(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(b0));
}
template <>
__device__ __forceinline__ void mma_k8<__nv_bfloat16>(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(b0));
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}

// v[i] becomes v[i ^ x] for a lane value x below N (N = 2, 4 or 8; selects, so that v stays in registers).
template <int N>
__device__ __forceinline__ void xor_index(float (&v)[N], int x) {
#pragma unroll
  for (int bit = 1; bit < N; bit <<= 1) {
    const bool swap = (x & bit) != 0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      if ((i & bit) == 0) {
        const float lo = v[i], hi = v[i + bit];
        v[i] = swap ? hi : lo;
        v[i + bit] = swap ? lo : hi;
      }
    }
  }
}

// ------------------------------------------------------------------------------------------------------------
// One warp's share of an expand stage: 2048 flat elements of B = 2048 / R outputs of R values each, R = the rank.
//
// The outputs are cut into NG groups of 8 * VPL.  Row block q of a group is eight outputs, one per g; the order is
// chosen so that lane (g, t) ends up with VPL outputs that lie next to each other - its part of y is one vector - and so
// that the eight rows a load touches fall on different shared-memory banks: block q brings lane g its output q ^ x(g),
// undone by selects afterwards.  Ranks 64 and 128 (rows of 128 bytes and more) need no x: odd rows fetch the halves of
// a 128-byte line in the other order.
// Tokens are columns, and with fewer than eight of them the columns repeat them: all four lanes t of a row then hold
// the same token's values, and each of them finishes (adds to y, stores) another group.
// ------------------------------------------------------------------------------------------------------------
template <int R>
struct ExpandShape {
  static constexpr int NOUT = 2048 / R;
  static constexpr int VPL = R == 8 ? 8 : (R == 16 ? 4 : 2);
  static constexpr int NG = NOUT / (8 * VPL);
};

// x(g): see above.
template <int R>
__device__ __forceinline__ int expand_x(int g) {
  return R == 8 ? g : (R == 16 ? (g & 3) : (R == 32 ? (g & 1) : 0));
}

// First output (inside the chunk) of the VPL this lane owns of group gr of warp cw.
template <int R>
__device__ __forceinline__ int expand_out(int cw, int gr, int g) {
  using S = ExpandShape<R>;
  return cw * S::NOUT + (gr * 8 + g) * S::VPL;
}

// The token operand: the delta rows of the tile's tokens, column g = token g (repeated below eight tokens).
template <int R>
struct DeltaFrag {
  uint32_t w[R <= 8 ? 1 : R / 8];
  __device__ __forceinline__ uint4 vec(int i) const { return make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]); }
};
template <typename T, int R>
__device__ __forceinline__ DeltaFrag<R> load_delta_frag(const T* ds, int tok, int t) {
  DeltaFrag<R> f;
  if constexpr (R == 8) {
    f.w[0] = *reinterpret_cast<const uint32_t*>(ds + tok * 8 + 2 * t);
  } else if constexpr (R == 16) {
    const uint2 v = *reinterpret_cast<const uint2*>(ds + tok * 16 + 4 * t);
    f.w[0] = v.x, f.w[1] = v.y;
  } else {
#pragma unroll
    for (int i = 0; i < R / 32; ++i) {
      const uint4 v = *reinterpret_cast<const uint4*>(ds + tok * R + 8 * (t + 4 * i));
      f.w[4 * i] = v.x, f.w[4 * i + 1] = v.y, f.w[4 * i + 2] = v.z, f.w[4 * i + 3] = v.w;
    }
  }
  return f;
}

// Row blocks 2j and 2j + 1 of group gr against the tokens: d[0..1] = this lane's output of block 2j for its two
// columns, d[2..3] = that of block 2j + 1.  Rows past the chunk's nout outputs repeat the last one.
template <typename T, int R>
__device__ __forceinline__ void expand_block_pair(float (&d)[4], const T* bs, const DeltaFrag<R>& f, int cw, int gr, int j,
                                                  int nout, int g, int t) {
  const int base = expand_out<R>(cw, gr, g);
  const int x = expand_x<R>(g);
  const int o0 = min(base + ((2 * j) ^ x), nout - 1), o1 = min(base + ((2 * j + 1) ^ x), nout - 1);
  if constexpr (R == 16) {
    const uint2 u = *reinterpret_cast<const uint2*>(bs + o0 * 16 + 4 * t);
    const uint2 v = *reinterpret_cast<const uint2*>(bs + o1 * 16 + 4 * t);
    mma_k16_first<T>(d, u.x, v.x, u.y, v.y, f.w[0], f.w[1]);
  } else {
    static_assert(R >= 32, "rank 8 has its own loads");
    if constexpr (R == 32) {
      const uint4 u = *reinterpret_cast<const uint4*>(bs + o0 * 32 + 8 * t);
      const uint4 v = *reinterpret_cast<const uint4*>(bs + o1 * 32 + 8 * t);
      mma_k32<T>(d, u, v, f.vec(0));
    } else {
      const bool odd = g & 1;
#pragma unroll
      for (int i = 0; i < R / 32; i += 2) {
        // two 16-byte vectors of each row, 64 bytes apart; odd rows fetch them in the other order
        const int va = t + 4 * (i + (odd ? 1 : 0)), vb = t + 4 * (i + (odd ? 0 : 1));
        const uint4 ua = *reinterpret_cast<const uint4*>(bs + o0 * R + 8 * va);
        const uint4 ub = *reinterpret_cast<const uint4*>(bs + o0 * R + 8 * vb);
        const uint4 wa = *reinterpret_cast<const uint4*>(bs + o1 * R + 8 * va);
        const uint4 wb = *reinterpret_cast<const uint4*>(bs + o1 * R + 8 * vb);
        const uint4 u0 = odd ? ub : ua, u1 = odd ? ua : ub, v0 = odd ? wb : wa, v1 = odd ? wa : wb;
        float e[4];
        if (i == 0) {
          mma_k32<T>(d, u0, v0, f.vec(0));
        } else {
          mma_k32<T>(e, u0, v0, f.vec(i));
#pragma unroll
          for (int q = 0; q < 4; ++q) d[q] += e[q];
        }
        mma_k32<T>(e, u1, v1, f.vec(i + 1));
#pragma unroll
        for (int q = 0; q < 4; ++q) d[q] += e[q];
      }
    }
  }
}

// All of group gr: acc[b][c] = block b, column 2t + c of this lane.
template <typename T, int R>
__device__ __forceinline__ void expand_group(float (&acc)[ExpandShape<R>::VPL][2], const T* bs,
                                             const DeltaFrag<R>& f, int cw, int gr, int nout, int lane) {
  using S = ExpandShape<R>;
  const int g = lane >> 2, t = lane & 3;
  if constexpr (R == 8) {
    // ldmatrix: four blocks at once, lane l points at row l % 8 of block l / 8
    const int rr = lane & 7, bi = lane >> 3;
    const int base = expand_out<R>(cw, gr, rr);
    const int x = expand_x<R>(rr);
#pragma unroll
    for (int j = 0; j < S::VPL / 4; ++j) {
      const int b = 4 * j + bi;
      const int o = min(base + (b ^ x), nout - 1);
      uint32_t r[4];
      ldmatrix_x4(r, smem_u32(bs + o * 8));
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float d[4] = {0.f, 0.f, 0.f, 0.f};
        mma_k8<T>(d, r[2 * h], r[2 * h + 1], f.w[0]);
        acc[4 * j + 2 * h][0] = d[0], acc[4 * j + 2 * h][1] = d[1];
        acc[4 * j + 2 * h + 1][0] = d[2], acc[4 * j + 2 * h + 1][1] = d[3];
      }
    }
  } else {
#pragma unroll
    for (int j = 0; j < S::VPL / 2; ++j) {
      float d[4];
      expand_block_pair<T, R>(d, bs, f, cw, gr, j, nout, g, t);
      acc[2 * j][0] = d[0], acc[2 * j][1] = d[1];
      acc[2 * j + 1][0] = d[2], acc[2 * j + 1][1] = d[3];
    }
  }
}

// Which tokens and groups a lane finishes when the tile has at most NT tokens (a power of two): TPL tokens starting
// at tok0, in round r the group r * DUP + di.
template <int NT>
struct TokenSplit {
  static constexpr int TPL = NT == 1 ? 1 : 2;
  static constexpr int DUP = NT <= 2 ? 4 : (NT == 4 ? 2 : 1);
  static __device__ __forceinline__ int column(int g, int n) { return min(g & (NT - 1), n - 1); }
  static __device__ __forceinline__ int tok0(int t) { return NT <= 2 ? 0 : (NT == 4 ? 2 * (t & 1) : 2 * t); }
  static __device__ __forceinline__ int di(int t) { return NT <= 2 ? t : (NT == 4 ? t >> 1 : 0); }
};

// Round `r` of a stage: after it acc holds the values of this lane's own group.
template <typename T, int R, int NT>
__device__ __forceinline__ void expand_round(float (&acc)[ExpandShape<R>::VPL][2], const T* bs,
                                             const DeltaFrag<R>& f, int cw, int r, int nout, int lane) {
  using S = ExpandShape<R>;
  using K = TokenSplit<NT>;
  const int di = K::di(lane & 3);
#pragma unroll
  for (int s = 0; s < K::DUP; ++s) {
    if (r * K::DUP + s >= S::NG) break;
    if (s == 0) {
      expand_group<T, R>(acc, bs, f, cw, r * K::DUP, nout, lane);
    } else {
      float other[S::VPL][2];
      expand_group<T, R>(other, bs, f, cw, r * K::DUP + s, nout, lane);
      const bool mine = di == s;
#pragma unroll
      for (int b = 0; b < S::VPL; ++b) {
#pragma unroll
        for (int c = 0; c < K::TPL; ++c) acc[b][c] = mine ? other[b][c] : acc[b][c];
      }
    }
  }
}

// N consecutive 16-bit values as one vector (N in 2, 4, 8), and eight floats from / to them.
template <typename T, int N>
__device__ __forceinline__ void load_vec(float (&f)[N], const T* p) {
  if constexpr (N == 8) {
    const uint4 v = *reinterpret_cast<const uint4*>(p);
    cvt8<T>(v, f);
  } else {
    T e[N];
    if constexpr (N == 4) {
      *reinterpret_cast<uint2*>(e) = *reinterpret_cast<const uint2*>(p);
    } else {
      *reinterpret_cast<uint32_t*>(e) = *reinterpret_cast<const uint32_t*>(p);
    }
#pragma unroll
    for (int i = 0; i < N; ++i) f[i] = to_f32<T>(e[i]);
  }
}
template <typename T, int N>
__device__ __forceinline__ void store_vec(T* p, const float (&f)[N]) {
  __align__(16) T e[N];
#pragma unroll
  for (int i = 0; i < N; ++i) e[i] = from_f32<T>(f[i]);
  if constexpr (N == 8) {
    *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(e);
  } else if constexpr (N == 4) {
    *reinterpret_cast<uint2*>(p) = *reinterpret_cast<const uint2*>(e);
  } else {
    *reinterpret_cast<uint32_t*>(p) = *reinterpret_cast<const uint32_t*>(e);
  }
}

}  // namespace slora
