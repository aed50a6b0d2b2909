// Of the prepare kernel: from the product [Q;K] K^T of a chunk to P and the triangular inverse T = (I+A)^-1, and from T to the
// scaled operand tiles, by the eight warps of a CTA.  The single launch does the same operations in the same order (gdn_fused.cu),
// so both give the same bits, but on a matrix with a row pitch of 68 floats.
//
// The FP32 64x64 matrix (A, then T in place) lies in shared memory without padding, its 16-byte granules permuted within a
// row (granule ^ granule_key(row)): whatever the phases do with it is free of bank conflicts - a row piece per lane (eight
// consecutive rows take eight different granules), the A fragments (ldmatrix, likewise) and the B fragments of the TF32
// products (four rows k..k+3, k a multiple of 4, by eight columns: their keys 0 2 4 6 or 1 3 5 7 spread the four pairs of
// granules over all banks).  With a pitch of 68 floats the B fragments, and with them a third of the kernel's shared-memory
// wavefronts, were conflicts: B1 T8192, 32 heads 120.8 us, 112.6 so (T2048: 38.9 and 37.6).  The single launch is bound by instruction issue and
// has no registers to spare: there this form is 12 to 18 % slower (more address arithmetic per tile).
//
// What lies above the diagonal is not computed, written or read where the consumer can leave it out: the block products
// skip 16x16 blocks of zeros, and the tensor-core products with T as their B operand take, of the 16 tokens j of a K step,
// only the rows i >= j's 16-token block (rows_from).
#pragma once
#include "umma_math.cuh"

namespace gdn_sm100 {
namespace {

constexpr int kMatrixBytes = kChunk * kChunk * 4;

// Shared-memory addresses of the matrix: `matrix` is its base (1024-byte aligned), a row is 256 bytes, and byte column c of row r
// is at (matrix + 256 r + 16 granule_key(r)) ^ c.
__device__ __forceinline__ int granule_key(int row) { return (2 * row + ((row >> 2) & 1)) & 7; }
__device__ __forceinline__ uint32_t matrix_row(uint32_t matrix, int row) { return matrix + row * 256 + granule_key(row) * 16; }
template <class T>
__device__ __forceinline__ T* shared_at(uint32_t address) { return reinterpret_cast<T*>(__cvta_shared_to_generic(address)); }

// Masks and decays on D = [Q;K] K^T (tensor memory, 128 lanes from `d_addr`, 64 columns): P as a BF16 K-major swizzled tile and
// A = tril(beta_i k_i.k_j exp(p_i - p_j), -1) as the FP32 matrix.  A warp owns the TMEM lane quarter (warp & 3; 0, 1: rows of P,
// 2, 3: rows of A) and the column half (warp >> 2); the two warps above the diagonal have nothing to do.  Of A only what the
// solves and products read is right (nothing on or above the diagonal of a 16x16 block, no block above the diagonal); of
// P the 32x32 block above the diagonal is not written.  In the block off the diagonal (rows 32.., columns ..31)
// exp(p_i - p_j) = exp(p_i - p_31) exp(p_31 - p_j): a factor per row and one per column (an exponential takes the
// special-function unit eight cycles per warp).  `pl2` = p log2(e), `ecol` = exp(p_31 - p_j).
// Returns whether this lane's token is no contraction of
// the state: it multiplies it by exp(g_i) (I - beta_i k_i k_i^T), a contraction iff 0 <= beta_i |k_i|^2 <= 2.
__device__ __forceinline__ bool mask_chunk(uint32_t d_addr, const float* pl2, const float* beta, const float* ecol,
                                           uint32_t tile_p, uint32_t matrix, int warp, int lane) {
  const int quarter = warp & 3, half = warp >> 2, i = (quarter & 1) * 32 + lane;
  const bool diagonal = half == (quarter & 1), below = half < (quarter & 1);
  if (!diagonal && !below) return false;
  const uint32_t taddr = d_addr + (uint32_t(quarter * 32) << 16);
  const uint32_t p_row = tile_p + i * 128 + (i & 7) * 16, a_row = matrix_row(matrix, i);
  const float pi = pl2[i], bi = beta[i];
  const float row = quarter < 2 ? kScale : bi, off = below ? fast_exp2(pi - pl2[31]) * row : 0.f;
#pragma unroll 1
  for (int h = half * 2; h < half * 2 + 2; ++h) {
    uint32_t d[16];
    tmem_ld16(taddr + h * 16, d);
    tmem_wait_ld();
    const float4* pj = reinterpret_cast<const float4*>(diagonal ? pl2 + h * 16 : ecol + h * 16);
    if (diagonal) {
#pragma unroll
      for (int q4 = 0; q4 < 4; ++q4) {
        const float4 p4 = pj[q4];
#pragma unroll
        for (int e = 0; e < 4; e += 2) {
          float x0 = __uint_as_float(d[q4 * 4 + e]), x1 = __uint_as_float(d[q4 * 4 + e + 1]), e0, e1;
          sub2(e0, e1, pi, pi, e ? p4.z : p4.x, e ? p4.w : p4.y);
          mul2(x0, x1, x0, x1, row, row);
          mul2(x0, x1, x0, x1, fast_exp2(e0), fast_exp2(e1));
          d[q4 * 4 + e] = __float_as_uint(x0);
          d[q4 * 4 + e + 1] = __float_as_uint(x1);
        }
      }
    } else {
#pragma unroll
      for (int q4 = 0; q4 < 4; ++q4) {
        const float4 p4 = pj[q4];
#pragma unroll
        for (int e = 0; e < 4; e += 2) {
          float x0 = __uint_as_float(d[q4 * 4 + e]), x1 = __uint_as_float(d[q4 * 4 + e + 1]);
          mul2(x0, x1, x0, x1, e ? p4.z : p4.x, e ? p4.w : p4.y);
          mul2(x0, x1, x0, x1, off, off);
          d[q4 * 4 + e] = __float_as_uint(x0);
          d[q4 * 4 + e + 1] = __float_as_uint(x1);
        }
      }
    }
    if (quarter < 2) {
#pragma unroll
      for (int c8 = 0; c8 < 2; ++c8) {
        uint32_t packed[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) packed[e] = pack_bf16(__uint_as_float(d[c8 * 8 + 2 * e]), __uint_as_float(d[c8 * 8 + 2 * e + 1]));
        *shared_at<uint4>(p_row ^ uint32_t((h * 2 + c8) << 4)) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
      }
    } else {
#pragma unroll
      for (int q4 = 0; q4 < 4; ++q4)
        *shared_at<uint4>(a_row ^ uint32_t((h * 4 + q4) << 4)) = make_uint4(d[q4 * 4], d[q4 * 4 + 1], d[q4 * 4 + 2], d[q4 * 4 + 3]);
    }
  }
  if (!diagonal) return false;
  if (quarter < 2) {
    // the piece that holds the diagonal, and the one behind it within the 16x16 block
    uint4* at = shared_at<uint4>(p_row ^ uint32_t((i >> 3) << 4));
    uint4 x = *at;
    const int keep = (i & 7) + 1;                       // columns of the piece on or below the diagonal, two to a word
    x.x &= keep > 1 ? ~0u : 0xffffu;
    x.y &= keep > 3 ? ~0u : (keep == 3 ? 0xffffu : 0u);
    x.z &= keep > 5 ? ~0u : (keep == 5 ? 0xffffu : 0u);
    x.w &= keep > 7 ? ~0u : (keep == 7 ? 0xffffu : 0u);
    *at = x;
    if (!(i & 8)) *shared_at<uint4>(p_row ^ uint32_t(((i >> 3) + 1) << 4)) = make_uint4(0u, 0u, 0u, 0u);
    return false;
  }
  return !(bi >= 0.f && *shared_at<float>(a_row ^ uint32_t(i << 2)) <= 2.f);          // beta_i |k_i|^2 exp(0), as this lane stored it
}

// The two 16x16 solves of 32x32 diagonal block `big`, by one warp: a column per thread (left-looking, in registers); the 16
// threads of a block overwrite it only after all of them have read it.
__device__ __forceinline__ void solve_diagonal(uint32_t matrix, int big, int lane) {
  const int col = lane & 15, block = big * 2 + (lane >> 4);
  // byte column 64 block + 16 j of a row is at its base ^ 64 block ^ 16 (j ^ key): of j ^ key, bit 2 flips between two places
  const uint32_t rows = matrix + block * 16 * 256, even = rows + block * 64, odd = rows + ((block * 64) ^ 64);
  const auto piece = [&](int r, int j4) -> float4 {
    const int c = (j4 >> 2) ^ granule_key(r & 7);
    return *shared_at<const float4>((c & 4 ? odd : even) + r * 256 + (c & 3) * 16);
  };
  float x[16];
#pragma unroll
  for (int r = 0; r < 16; ++r) {
    float acc0 = (r == col) ? 1.f : 0.f, acc1 = 0.f;
#pragma unroll
    for (int j4 = 0; j4 < r; j4 += 4) {
      const float4 a = piece(r, j4);
      if (j4 + 0 < r) acc0 = fmaf(-a.x, x[j4 + 0], acc0);
      if (j4 + 1 < r) acc1 = fmaf(-a.y, x[j4 + 1], acc1);
      if (j4 + 2 < r) acc0 = fmaf(-a.z, x[j4 + 2], acc0);
      if (j4 + 3 < r) acc1 = fmaf(-a.w, x[j4 + 3], acc1);
    }
    x[r] = acc0 + acc1;
  }
  __syncwarp();
  const uint32_t at = rows + ((block * 64) ^ (col << 2));
#pragma unroll
  for (int r = 0; r < 16; ++r) *shared_at<float>((at ^ (granule_key(r & 7) * 16)) + r * 256) = x[r];
}

// Block products T21 = -T22 (A21 T11) at block size 16, then 32, two steps each, as m16n8 tiles in 3xTF32, a tile per warp;
// the scratch is the 32x32 block above the diagonal, which holds nothing.  The four steps share one body (code size), and the
// 16x16 blocks of zeros above the diagonals of T11 and T22 are skipped.  `sync` is a barrier of the eight warps; the last
// step's tiles are not behind one.
template <class Sync>
__device__ __forceinline__ void merge_blocks(uint32_t matrix, bool ok, int warp, int lane, Sync sync) {
  const int g = lane >> 2, t = lane & 3;
  // this lane's places in an A fragment (its row piece), a B fragment (row t, column g) and a D tile at row 0, column 0
  const uint32_t a_lane = matrix_row(matrix, (lane & 7) + ((lane >> 3) & 1) * 8) ^ uint32_t((lane >> 4) << 4);
  const uint32_t b_lane = matrix_row(matrix, t) ^ uint32_t(g << 2), d_lane = matrix_row(matrix, g) ^ uint32_t(t << 3);
#pragma unroll 1
  for (int step = 0; step < 4; ++step) {
    const bool second = step & 1;
    int row, col, a_col, b_row, b_col, k0, k1, d_row, d_col;          // D = A[row.., a_col + k] B[b_row + k, b_col..]
    if (step < 2) {
      const int o = (warp >> 1 & 1) * 32;
      row = o + 16;
      col = (warp & 1) * 8;
      a_col = second ? row : o;
      b_row = second ? o >> 1 : o;
      b_col = second ? 32 + col : o + col;
      d_row = second ? row : o >> 1;
      d_col = second ? o + col : 32 + col;
      k0 = 0;
      k1 = warp < 4 ? 16 : 0;
    } else {
      const int row16 = (warp & 1) * 16;
      col = (warp >> 1) * 8;
      row = 32 + row16;
      a_col = second ? 32 : 0;
      b_row = 0;
      b_col = second ? 32 + col : col;
      d_row = second ? row : row16;
      d_col = second ? col : 32 + col;
      k0 = second ? 0 : col & 16;
      k1 = second ? row16 + 16 : 32;
    }
    if (ok && k0 < k1) {
      const uint32_t a = a_lane + row * 256, b = (b_lane + b_row * 256) ^ uint32_t(b_col << 2), d = (d_lane + d_row * 256) ^ uint32_t(d_col << 2);
      float lh[4] = {}, hl[4] = {}, hh[4] = {};
#pragma unroll 1
      for (int k = k0; k < k1; k += 16) {
#pragma unroll
        for (int u = 0; u < 16; u += 8) {
          float av[4];
          uint32_t ah[4], al[4], bh[2], bl[2];
          load_fragment_a(av, a ^ uint32_t((a_col + k + u) << 2));
          const float bv[2] = {*shared_at<float>(b + (k + u) * 256), *shared_at<float>((b ^ 16) + (k + u + 4) * 256)};      // keys 2 t, 2 t + 1
          split_tf32(av, ah, al);
          split_tf32(bv, bh, bl);
          mma_tf32(lh, al, bh);
          mma_tf32(hl, ah, bl);
          mma_tf32(hh, ah, bh);
        }
      }
      const float sign = second ? -1.f : 1.f;
      *shared_at<float2>(d) = make_float2(sign * ((lh[0] + hl[0]) + hh[0]), sign * ((lh[1] + hl[1]) + hh[1]));
      *shared_at<float2>(d + 8 * 256) = make_float2(sign * ((lh[2] + hl[2]) + hh[2]), sign * ((lh[3] + hl[3]) + hh[3]));
    }
    if (step < 3) sync();
  }
}

// A thread's part of T (row t & 63, 16 columns from (t >> 6) * 16 on), the same scaled per column by `coef` as BF16 hi/lo pieces, and
// their place in a K-major swizzled tile pair, the lo tile `kLo` bytes behind.  The block above the diagonal is left out.
__device__ __forceinline__ bool inverse_part(uint32_t matrix, int t, float4 (&x)[4]) {
  const int row = t & 63, c4 = (t >> 6) * 4;
  if (c4 >= 8 && row < 32) return false;
  const uint32_t at = matrix_row(matrix, row) ^ uint32_t(c4 << 4);
#pragma unroll
  for (int q4 = 0; q4 < 4; ++q4) x[q4] = *shared_at<const float4>(at ^ uint32_t(q4 << 4));
  return true;
}
struct ScaledPart { uint4 hi[2], lo[2]; };
__device__ __forceinline__ ScaledPart scaled_part(const float4 (&x)[4], const float* coef, int t) {
  ScaledPart out;
#pragma unroll
  for (int g8 = 0; g8 < 2; ++g8) {
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int q4 = 0; q4 < 2; ++q4) {
      const float4 y = x[g8 * 2 + q4], c = *reinterpret_cast<const float4*>(coef + (t >> 6) * 16 + (g8 * 2 + q4) * 4);
      float a0, a1, b0, b1;
      mul2(a0, a1, y.x, y.y, c.x, c.y);
      mul2(b0, b1, y.z, y.w, c.z, c.w);
      split_pair(a0, a1, hi[q4 * 2], lo[q4 * 2]);
      split_pair(b0, b1, hi[q4 * 2 + 1], lo[q4 * 2 + 1]);
    }
    out.hi[g8] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    out.lo[g8] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
  }
  return out;
}
template <int kLo>
__device__ __forceinline__ void store_part(const ScaledPart& p, uint32_t tile, int t) {
  const int row = t & 63, c0 = (t >> 6) * 16;
  const uint32_t at = (tile + row * 128 + (row & 7) * 16) ^ uint32_t(c0 << 1);
#pragma unroll
  for (int g8 = 0; g8 < 2; ++g8) {
    *shared_at<uint4>(at ^ uint32_t(g8 << 4)) = p.hi[g8];
    *shared_at<uint4>((at ^ uint32_t(g8 << 4)) + kLo) = p.lo[g8];
  }
}

}  // namespace
}  // namespace gdn_sm100
