// Device arithmetic shared by the tensor-core kernels of this backend (two-kernel path and single-launch forward):
// both produce the same bits, so the operations and their order live in one place.
#pragma once
#include "gdn_common.cuh"
#include "umma.cuh"

namespace gdn_sm100 {
using namespace ptx;
namespace {

constexpr float kLog2e = 1.4426950408889634f;
constexpr int kBox = 8192;            // one TMA box: 64 rows x 128 bytes
constexpr uint32_t kIdescN64 = idesc_bf16(128, 64, false, false);      // A K-major (smem or TMEM), B K-major
constexpr uint32_t kIdescN128BT = idesc_bf16(128, 128, false, true);   // B MN-major
// K step ks (16 tokens j) of a product whose B operand is a lower-triangular K-major [i][j] tile: only rows i from 16 ks on; what lies
// above need not even be written
constexpr uint32_t idesc_rows_from(int ks, bool a_mn_major) { return idesc_bf16(128, 64 - 16 * ks, a_mn_major, false); }
constexpr uint32_t rows_from(int ks) { return uint32_t(ks) * (16 * 128 / 16); }     // their offset in the B descriptor

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Packed FP32 pairs (two IEEE round-to-nearest operations per instruction on sm_100): the arithmetic of the walk's
// chain warps is bound by instruction issue, and these halve its floating-point instruction count bit for bit.
#define GDN_F32X2(name, op)                                                                                      \
  __device__ __forceinline__ void name(float& x0, float& x1, float a0, float a1, float b0, float b1) {          \
    asm("{\n\t.reg .b64 a, b, c;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t" op                       \
        ".rn.f32x2 c, a, b;\n\tmov.b64 {%0, %1}, c;\n\t}"                                                       \
        : "=f"(x0), "=f"(x1) : "f"(a0), "f"(a1), "f"(b0), "f"(b1));                                              \
  }
GDN_F32X2(sub2, "sub")
GDN_F32X2(mul2, "mul")
#undef GDN_F32X2
// d += a b for one m16n8k8 tile with FP32-grade accuracy from TF32 tensor-core products: a ~ ah + al, b ~ bh + bl
// (both parts TF32), d += ah bh + ah bl + al bh (the 3xTF32 scheme the reference uses for these merges,
// tests/wy_cpu.py:10-18).  Fragment layout of mma.m16n8k8: g = lane / 4, t = lane % 4;
// a = {A[g][t], A[g+8][t], A[g][t+4], A[g+8][t+4]}, b = {B[t][g], B[t+4][g]}, d = {D[g][2t], D[g][2t+1], D[g+8][2t], D[g+8][2t+1]}.
// The high part is the operand with its 13 low mantissa bits cleared (a TF32 value), the low part the exact FP32
// remainder, of which the tensor core reads the leading TF32 bits: about 2^-20 relative in all, below the 16 significant
// bits the inverse is later stored with.  Logic and add instructions: the conversion unit stays free for BF16 packing.
template <int kN>
__device__ __forceinline__ void split_tf32(const float (&x)[kN], uint32_t (&hi)[kN], uint32_t (&lo)[kN]) {
#pragma unroll
  for (int i = 0; i < kN; i += 2) {
    hi[i] = __float_as_uint(x[i]) & 0xffffe000u;
    hi[i + 1] = __float_as_uint(x[i + 1]) & 0xffffe000u;
    float l0, l1;
    sub2(l0, l1, x[i], x[i + 1], __uint_as_float(hi[i]), __uint_as_float(hi[i + 1]));
    lo[i] = __float_as_uint(l0);
    lo[i + 1] = __float_as_uint(l1);
  }
}
__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// The A fragment {A[g][t], A[g+8][t], A[g][t+4], A[g+8][t+4]} of a row-major FP32 matrix in shared memory in one instruction:
// a 16-byte row piece of an 8x8 16-bit matrix holds four floats.  `addr` is this lane's row piece (fragment_row).
__device__ __forceinline__ void load_fragment_a(float (&a)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=f"(a[0]), "=f"(a[1]), "=f"(a[2]), "=f"(a[3]) : "r"(addr) : "memory");
}
// row piece of a lane: rows 0..15, columns 0 or 4 (floats, pitch lda)
__device__ __forceinline__ int fragment_row(int lane, int lda) { return ((lane & 7) + ((lane >> 3) & 1) * 8) * lda + (lane >> 4) * 4; }
// One m16n8 tile D = A B over k in [0, 16 kSteps): A at this lane's `a_addr`, B row-major with pitch ldb, b = this lane's
// B[t][g]; of the 16-wide steps those in the mask `steps` are taken.  The three TF32 products of the split run as three chains
// that are added at the end (one chain of dependent products would be three times as long, some 25 cycles each).
template <int kSteps>
__device__ __forceinline__ void tile_row_tf32x3(float (&d)[4], uint32_t a_addr, const float* b, int ldb, int steps) {
  float lh[4] = {}, hl[4] = {}, hh[4] = {};
#pragma unroll
  for (int step = 0; step < kSteps; ++step) {
    if (kSteps > 1 && !(steps >> step & 1)) continue;
#pragma unroll
    for (int k0 = step * 16; k0 < step * 16 + 16; k0 += 8) {
      float av[4];
      uint32_t ah[4], al[4], bh[2], bl[2];
      load_fragment_a(av, a_addr + k0 * 4);
      const float bv[2] = {b[k0 * ldb], b[(k0 + 4) * ldb]};
      split_tf32(av, ah, al);
      split_tf32(bv, bh, bl);
      mma_tf32(lh, al, bh);
      mma_tf32(hl, ah, bl);
      mma_tf32(hh, ah, bh);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) d[i] = (lh[i] + hl[i]) + hh[i];
}
__device__ __forceinline__ float bf16_lo(uint32_t packed) { return __uint_as_float(packed << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t packed) { return __uint_as_float(packed & 0xffff0000u); }
// L2-normalises 32 of the 128 rows of a [Q0 K0 Q1 K1] tile group in place, pass 0 and 1 the 64 Q rows, 2 and 3 the K rows: 256
// threads, 8 per row, each the same swizzled 16-byte slot of the row's two halves; x rsqrt(sum x^2 + 1e-6) rounded to BF16.  The
// sum's order is that of the step in front of the path (prepare_inputs: 16 lanes of 8 values, lanes 8, 4, 2, 1 apart added),
// whose first addition is within a thread here: one of four rounds of shuffles less and half as many of the others (raw projections,
// 32 value heads: 2 x 1500 tokens 97.3 -> 91.1 us, 4 x 4000 305 -> 288).
__device__ __forceinline__ void normalise_rows(uint8_t* tiles, int pass, int t) {
  const int lane8 = t & 7, r = pass * 32 + (t >> 3), row = r & 63;
  uint8_t* slot = tiles + (r < 64 ? 0 : kBox) + row * 128 + ((lane8 ^ (row & 7)) << 4);
  uint32_t x[2][4];
  float square[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint4 v = *reinterpret_cast<const uint4*>(slot + h * 2 * kBox);
    x[h][0] = v.x;
    x[h][1] = v.y;
    x[h][2] = v.z;
    x[h][3] = v.w;
    square[h] = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) square[h] = fmaf(bf16_hi(x[h][e]), bf16_hi(x[h][e]), fmaf(bf16_lo(x[h][e]), bf16_lo(x[h][e]), square[h]));
  }
  float sum = square[0] + square[1];
#pragma unroll
  for (int d = 4; d; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d, 8);
  const float factor = rsqrtf(sum + 1e-6f);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float a, b;
      mul2(a, b, bf16_lo(x[h][e]), bf16_hi(x[h][e]), factor, factor);
      x[h][e] = pack_bf16(a, b);
    }
    *reinterpret_cast<uint4*>(slot + h * 2 * kBox) = make_uint4(x[h][0], x[h][1], x[h][2], x[h][3]);
  }
}
// (x0, x1) ~ hi + lo as packed BF16 pairs
__device__ __forceinline__ void split_pair(float x0, float x1, uint32_t& hi, uint32_t& lo) {
  hi = pack_bf16(x0, x1);
  float l0, l1;
  sub2(l0, l1, x0, x1, bf16_lo(hi), bf16_hi(hi));
  lo = pack_bf16(l0, l1);
}

// kN columns of an accumulator times a factor per column (shared memory, 16-byte aligned)
template <int kN>
__device__ __forceinline__ void scale_columns(uint32_t (&x)[kN], const float* factor) {
#pragma unroll
  for (int q4 = 0; q4 < kN / 4; ++q4) {
    const float4 f = *reinterpret_cast<const float4*>(factor + q4 * 4);
    float a, b;
    mul2(a, b, __uint_as_float(x[q4 * 4]), __uint_as_float(x[q4 * 4 + 1]), f.x, f.y);
    x[q4 * 4] = __float_as_uint(a);
    x[q4 * 4 + 1] = __float_as_uint(b);
    mul2(a, b, __uint_as_float(x[q4 * 4 + 2]), __uint_as_float(x[q4 * 4 + 3]), f.z, f.w);
    x[q4 * 4 + 2] = __float_as_uint(a);
    x[q4 * 4 + 3] = __float_as_uint(b);
  }
}

}  // namespace
}  // namespace gdn_sm100
