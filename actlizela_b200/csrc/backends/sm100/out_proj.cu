// out_proj of the layer's output gate: C[M,N] = A[M,K] W[N,K]^T, BF16 operands, FP32 accumulation, BF16 result
// (the reference's out_proj_gemm / out_proj_gemm_cutlass, csrc/output_gate/output_gate.cu and
// csrc/output_gate/output_gate_cutlass.cu, docs/OUTPUT_GATE.md:17-24: an mma.sync kernel and a CUTLASS SM80 GEMM).
// Here: one tcgen05 kernel.  A CTA owns a tile of C of 128 or 256 rows; both operands are K-major as they lie in memory
// (A row-major, W in the Linear layout [N][K]), so their 64-wide K steps come straight from TMA into 128-byte-swizzled
// shared memory, three or four stages deep; the accumulators live in tensor memory.
// Roles: warp 0 TMA producer, warp 1 MMA issuer (owns the tensor-memory allocation), then four epilogue warps per 128 rows
// (TMEM -> registers -> BF16 -> swizzled tile -> TMA store).  Rows and columns beyond M, N and the K tail
// read as zeros (TMA fill).
#include "actlize_la_sm100.h"
#include "gdn_common.cuh"
#include "umma.cuh"

namespace gdn_sm100 {
using namespace ptx;
namespace {

constexpr int kTileM = 128, kTileK = 64;
constexpr int kOperandBytes = kTileM * kTileK * 2;                 // 16 KB per 128-row operand tile
// Tiles of 128 kRows x kN.  Bound by shared memory, 128 bytes a cycle: a K step of 64 of a 128 x 128 tile is written (32 KB) and
// read by the tensor core (32 KB) in 512 cycles, of a 128 x 256 tile in 768 (512 of products), of a 256 x 256 tile in 1280
// (1024 of products; its two accumulators fill tensor memory), of 256 x 224 in 1184, which fits the turns of some sizes better.  Two
// CTAs of the smallest share an SM, the others have it alone.  K 4096, N 2560, in this order: M 3000 68, 61, 53 and 49 us; M 6000 as
// 128 x 256 121, then 102 and 94; M 8192 165, 148, 147 and 137 (1.25 PFLOP/s).
template <int kN, int kRows> struct GemmLayout {
  static constexpr int kStage = kOperandBytes * kRows + kN * kTileK * 2;
  static constexpr int kStages = kRows == 1 && kN == 256 ? 4 : 3, kPerSm = kN == 128 ? 2 : 1;
  static constexpr int kAccStride = kN == 224 ? 256 : kN, kColumns = kAccStride * kRows;      // tensor memory
  static constexpr int kThreads = 64 + 128 * kRows;
  static constexpr int kBars = kStages * kStage;
  static constexpr int kBytes = kBars + 128 + 1024;
  static constexpr uint32_t kIdesc = idesc_bf16(kTileM, kN, false, false);
  static_assert(kN % 32 == 0 && kRows * (kN / 64) * kOperandBytes <= kBars, "the output tile must fit on the stages");
  static_assert(kPerSm * (kBytes + 1024) <= 227 * 1024 && kPerSm * kColumns <= 512, "shared and tensor memory of one SM");
};

template <int kN, int kRows>
__global__ void __launch_bounds__(GemmLayout<kN, kRows>::kThreads, GemmLayout<kN, kRows>::kPerSm)
out_proj_umma_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_w,
                     const __grid_constant__ CUtensorMap tm_c, __nv_bfloat16* __restrict__ c, int m, int n, int k) {
  using L = GemmLayout<kN, kRows>;
  extern __shared__ __align__(1024) uint8_t raw_smem[];
  uint8_t* sm = raw_smem + ((1024u - (smem_u32(raw_smem) & 1023u)) & 1023u);
  uint64_t* full = reinterpret_cast<uint64_t*>(sm + L::kBars);       // [stages] tiles landed
  uint64_t* empty = full + L::kStages;                               // [stages] tiles consumed
  uint64_t* done = empty + L::kStages;                               // accumulator complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* abort_word = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const AbortFlag abort{abort_word};

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n0 = blockIdx.x * kN, m0 = blockIdx.y * kTileM * kRows;
  const int k_tiles = (k + kTileK - 1) / kTileK;

  if (tid == 0) {
    for (int s = 0; s < L::kStages; ++s) {
      mbar_init(full + s, 1);
      mbar_init(empty + s, 1);
    }
    mbar_init(done, 1);
    *abort_word = 0;
    fence_barrier_init();
  }
  if (warp == 0 && lane == 0) {
    prefetch_tensormap(&tm_a);
    prefetch_tensormap(&tm_w);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, L::kColumns);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  wait_for_previous_kernel();
  dependents_may_start();

  if (warp == 0) {
    if (lane == 0) {
      for (int kt = 0; kt < k_tiles; ++kt) {
        const int s = kt % L::kStages;
        if (kt >= L::kStages && !mbar_wait(empty + s, ((kt / L::kStages) - 1) & 1, abort, 60, kt)) break;
        uint8_t* stage = sm + s * L::kStage;
        mbar_arrive_expect_tx(full + s, L::kStage);
        tma_load_2d(stage, &tm_a, full + s, kt * kTileK, m0);
        tma_load_2d(stage + kOperandBytes * kRows, &tm_w, full + s, kt * kTileK, n0);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    const uint32_t base = __shfl_sync(0xffffffffu, smem_u32(sm), 0);
    if (elect_one()) {
      bool ok = true;
      for (int kt = 0; kt < k_tiles && ok; ++kt) {
        const int s = kt % L::kStages;
        ok = mbar_wait(full + s, (kt / L::kStages) & 1, abort, 61, kt);
        tc_fence_after();
        const uint64_t da = smem_desc(base + s * L::kStage, 16, 1024);
        const uint64_t db = smem_desc(base + s * L::kStage + kOperandBytes * kRows, 16, 1024);
#pragma unroll
        for (int ks = 0; ks < kTileK / 16; ++ks)          // 16 BF16 (32 bytes) along K per instruction
#pragma unroll
          for (int r = 0; r < kRows; ++r)
            mma_ss(tmem + r * L::kAccStride, da + uint64_t(r * (kOperandBytes >> 4) + ks * 2), db + uint64_t(ks * 2), L::kIdesc, (kt | ks) != 0);
        mma_commit(empty + s);
      }
      mma_commit(done);
    }
    __syncwarp();
  } else {
    // epilogue: a warp may only touch the TMEM lane quarter (warp % 4); warps 2..5 cover quarters 2, 3, 0, 1, warps 6..9 those
    // of the second 128 rows
    const int quarter = warp & 3, part = (warp - 2) >> 2;
    // The tile leaves through boxes of 128 rows x 64 columns on the dead stages and TMA stores, which clip it at M and N.
    // (Straight from registers a warp's 16-byte stores go to 32 rows, two to a sector: about 4 us a turn of the wide tiles.)
    const int row = quarter * 32 + lane;
    const bool ok = mbar_wait(done, 0, abort, 62, 0);
    tc_fence_after();
    const uint32_t taddr = tmem + (uint32_t(quarter * 32) << 16) + part * L::kAccStride;
    const bool leader = ((warp - 2) & 3) == 0 && lane == 0;
#pragma unroll 1
    for (int box = 0; box < kN / 64; ++box) {
      uint8_t* tile = sm + (part * (kN / 64) + box) * kOperandBytes;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        if (ok) {
          uint32_t d[32];
          tmem_ld32(taddr + box * 64 + half * 32, d);
          tmem_wait_ld();
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            uint4 o;
            o.x = pack_bf16(__uint_as_float(d[q * 8 + 0]), __uint_as_float(d[q * 8 + 1]));
            o.y = pack_bf16(__uint_as_float(d[q * 8 + 2]), __uint_as_float(d[q * 8 + 3]));
            o.z = pack_bf16(__uint_as_float(d[q * 8 + 4]), __uint_as_float(d[q * 8 + 5]));
            o.w = pack_bf16(__uint_as_float(d[q * 8 + 6]), __uint_as_float(d[q * 8 + 7]));
            *reinterpret_cast<uint4*>(tile + row * 128 + (((half * 4 + q) ^ (row & 7)) << 4)) = o;
          }
        }
      }
      fence_proxy_async_smem();
      asm volatile("bar.sync %0, 128;" ::"r"(1 + part) : "memory");
      if (leader && ok && m0 + part * kTileM < m && n0 + box * 64 < n) {
        tma_store_2d(&tm_c, tile, n0 + box * 64, m0 + part * kTileM);
        tma_store_commit();
      }
    }
    if (kN % 64 && ok) {
      // 32 columns more: too narrow for a box
      uint32_t d[32];
      tmem_ld32(taddr + kN - 32, d);
      tmem_wait_ld();
      const int r = m0 + part * kTileM + row, first = n0 + kN - 32;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (r < m && first + q * 8 < n)      // N is a multiple of 8: a 16-byte piece is inside or outside
          *reinterpret_cast<uint4*>(c + (long long)r * n + first + q * 8) =
              make_uint4(pack_bf16(__uint_as_float(d[q * 8]), __uint_as_float(d[q * 8 + 1])), pack_bf16(__uint_as_float(d[q * 8 + 2]), __uint_as_float(d[q * 8 + 3])),
                         pack_bf16(__uint_as_float(d[q * 8 + 4]), __uint_as_float(d[q * 8 + 5])), pack_bf16(__uint_as_float(d[q * 8 + 6]), __uint_as_float(d[q * 8 + 7])));
    }
    if (leader) tma_store_wait_all();
  }
  if (abort.raised()) {
    for (int i = 0; i < 20; ++i) __nanosleep(100000);   // let copies in flight land before the CTA leaves
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, L::kColumns);
}

// ------------------------------------------------------------------------------------------- few rows: split over K
// With few rows of A (a decode step) the 128 x 128 tiles above are fewer than the SMs, and a CTA walks all of K alone: at
// M 4, K 4096, N 2560 twenty CTAs streamed W, 21 MB, at 0.7 TB/s.  Here the roles are swapped (128 rows of W on the
// tensor-memory lanes, kM rows of A as the N dimension, so that nothing but kM rows is multiplied) and a cluster of CTAs
// splits K: each accumulates its range, leaves its partial tile in its own shared memory, and sums a share of the rows
// over the cluster, in rank order, through distributed shared memory.  Bound by the stream of W (L2 or HBM) and a launch's
// latencies: descriptors are fetched beside the end of the kernel in front, the ranks' partial sums all at once (4 rows, weights from
// HBM: 8.13 us, 7.95 so; 33 rows 9.53 and 9.17).
constexpr int kSkinnyThreads = 192;
template <int kM> struct SkinnyLayout {
  static constexpr int kStage = kOperandBytes + kM * kTileK * 2;             // W tile, A tile
  static constexpr int kStages = kM <= 32 ? 5 : (kM == 64 ? 4 : 3);          // two CTAs per SM
  static constexpr int kBars = kStages * kStage;
  static constexpr int kBytes = kBars + 128 + 1024;
  static_assert(kM * 128 * 4 <= kBars, "the partial tile must fit on the stages");
  static_assert(2 * (kBytes + 1024) <= 227 * 1024, "two CTAs per SM");
};

template <int kM>
__global__ void __launch_bounds__(kSkinnyThreads, 2)
out_proj_skinny_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_w,
                       __nv_bfloat16* __restrict__ c, int m, int n, int k) {
  using L = SkinnyLayout<kM>;
  extern __shared__ __align__(1024) uint8_t raw_smem[];
  uint8_t* sm = raw_smem + ((1024u - (smem_u32(raw_smem) & 1023u)) & 1023u);
  uint64_t* full = reinterpret_cast<uint64_t*>(sm + L::kBars);        // [stages] tiles landed
  uint64_t* empty = full + L::kStages;                                // [stages] tiles consumed
  uint64_t* done = empty + L::kStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* abort_word = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const AbortFlag abort{abort_word};
  constexpr uint32_t kColumns = kM < 32 ? 32 : kM;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = blockIdx.x, split = gridDim.x;                      // the cluster spans the first grid dimension
  const int n0 = blockIdx.y * kTileM, m0 = blockIdx.z * kM;
  const int k_tiles = (k + kTileK - 1) / kTileK;
  const int kt0 = k_tiles * rank / split, kt1 = k_tiles * (rank + 1) / split;

  if (tid == 0) {
    for (int s = 0; s < L::kStages; ++s) {
      mbar_init(full + s, 1);
      mbar_init(empty + s, 1);
    }
    mbar_init(done, 1);
    *abort_word = 0;
    fence_barrier_init();
  }
  if (warp == 0 && lane == 0) {          // beside the end of the kernel in front
    prefetch_tensormap(&tm_a);
    prefetch_tensormap(&tm_w);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, kColumns);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  wait_for_previous_kernel();
  dependents_may_start();

  if (warp == 0) {
    if (lane == 0) {
      for (int kt = kt0; kt < kt1; ++kt) {
        const int i = kt - kt0, s = i % L::kStages;
        if (i >= L::kStages && !mbar_wait(empty + s, ((i / L::kStages) - 1) & 1, abort, 63, kt)) break;
        uint8_t* stage = sm + s * L::kStage;
        mbar_arrive_expect_tx(full + s, L::kStage);
        tma_load_2d(stage, &tm_w, full + s, kt * kTileK, n0);
        tma_load_2d(stage + kOperandBytes, &tm_a, full + s, kt * kTileK, m0);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t base = smem_u32(sm);
      bool ok = true;
      for (int kt = kt0; kt < kt1 && ok; ++kt) {
        const int i = kt - kt0, s = i % L::kStages;
        ok = mbar_wait(full + s, (i / L::kStages) & 1, abort, 64, kt);
        tc_fence_after();
        const uint64_t dw = smem_desc(base + s * L::kStage, 16, 1024), da = smem_desc(base + s * L::kStage + kOperandBytes, 16, 1024);
#pragma unroll
        for (int ks = 0; ks < kTileK / 16; ++ks)
          mma_ss(tmem, dw + uint64_t(ks * 2), da + uint64_t(ks * 2), idesc_bf16(128, kM, false, false), (i | ks) != 0);
        mma_commit(empty + s);
      }
      mma_commit(done);
    }
    __syncwarp();
  } else if (mbar_wait(done, 0, abort, 65, 0)) {
    // the partial tile as [row of A][row of W], over the stages (every tile has been consumed)
    tc_fence_after();
    const int quarter = warp & 3;
    float* part = reinterpret_cast<float*>(sm) + quarter * 32 + lane;
#pragma unroll
    for (int piece = 0; piece < kM / 16; ++piece) {
      uint32_t d[16];
      tmem_ld16(tmem + (uint32_t(quarter * 32) << 16) + piece * 16, d);
      tmem_wait_ld();
#pragma unroll
      for (int j = 0; j < 16; ++j) part[(piece * 16 + j) * 128] = __uint_as_float(d[j]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, kColumns);
  // every CTA of the cluster comes here, also one that gave up a wait
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  {
    // rank r sums rows r, r + split, ...: 64 threads take a row's 128 columns in pairs
    const int pair = tid & 63;
    const bool inside = n0 + pair * 2 < n;
    for (int row = rank + (tid >> 6) * split; row < kM && m0 + row < m; row += 3 * split) {
      const uint32_t at = smem_u32(sm) + (row * 128 + pair * 2) * 4;
      float px[8], py[8];                    // all ranks' partial sums are in flight, then added in rank order
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        px[r] = py[r] = 0.f;
        if (r < split) {
          uint32_t remote;
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(at), "r"(r));
          asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(px[r]), "=f"(py[r]) : "r"(remote) : "memory");
        }
      }
      float x = px[0], y = py[0];
#pragma unroll
      for (int r = 1; r < 8; ++r) {
        x += px[r];
        y += py[r];
      }
      if (inside) *reinterpret_cast<uint32_t*>(c + (long long)(m0 + row) * n + n0 + pair * 2) = pack_bf16(x, y);
    }
  }
  if (abort.raised()) {
    for (int i = 0; i < 20; ++i) __nanosleep(100000);   // let copies in flight land before the CTA leaves
  }
  // nobody leaves while its partial tile may still be read
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int kM>
int launch_skinny(TensorMapEncoder& enc, const void* a, const void* w, void* c, int m, int n, int k, int split, cudaStream_t stream) {
  CUtensorMap tm_a, tm_w;
  if (int rc = enc.bf16_2d(&tm_a, a, uint64_t(k), uint64_t(m), kM)) return rc;
  if (int rc = enc.bf16_2d(&tm_w, w, uint64_t(k), uint64_t(n), kTileM)) return rc;
  cudaLaunchConfig_t launch{};
  launch.gridDim = dim3(split, (n + kTileM - 1) / kTileM, (m + kM - 1) / kM);
  launch.blockDim = dim3(kSkinnyThreads);
  launch.dynamicSmemBytes = SkinnyLayout<kM>::kBytes;
  launch.stream = stream;
  cudaLaunchAttribute attributes[2] = {};
  attributes[0].id = cudaLaunchAttributeClusterDimension;
  attributes[0].val.clusterDim.x = split;
  attributes[0].val.clusterDim.y = attributes[0].val.clusterDim.z = 1;
  attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;      // see launch_early
  attributes[1].val.programmaticStreamSerializationAllowed = 1;
  launch.attrs = attributes;
  launch.numAttrs = 2;
  return int(cudaLaunchKernelEx(&launch, out_proj_skinny_kernel<kM>, tm_a, tm_w, static_cast<__nv_bfloat16*>(c), m, n, k));
}


template <int kN, int kRows>
int launch_tiles(TensorMapEncoder& enc, const void* a, const void* w, void* c, int m, int n, int k, cudaStream_t stream) {
  using L = GemmLayout<kN, kRows>;
  CUtensorMap tm_a, tm_w, tm_c;
  if (int rc = enc.bf16_2d(&tm_c, c, uint64_t(n), uint64_t(m), kTileM)) return rc;
  if (int rc = enc.bf16_2d(&tm_a, a, uint64_t(k), uint64_t(m), kTileM * kRows)) return rc;
  if (int rc = enc.bf16_2d(&tm_w, w, uint64_t(k), uint64_t(n), kN)) return rc;
  return launch_early(out_proj_umma_kernel<kN, kRows>, dim3((n + kN - 1) / kN, (m + kTileM * kRows - 1) / (kTileM * kRows)), L::kThreads,
                      L::kBytes, true, stream, tm_a, tm_w, tm_c, static_cast<__nv_bfloat16*>(c), m, n, k);
}
}  // namespace

GDN_SM100_DEFINE_STATUS_HOOKS(gemm)

int configure_out_proj() {
  if (int rc = tensor_map_encoder().init()) return rc;
  const auto smem = cudaFuncAttributeMaxDynamicSharedMemorySize;
  cudaError_t e = cudaFuncSetAttribute(out_proj_umma_kernel<128, 1>, smem, GemmLayout<128, 1>::kBytes);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(out_proj_umma_kernel<256, 1>, smem, GemmLayout<256, 1>::kBytes);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(out_proj_umma_kernel<256, 2>, smem, GemmLayout<256, 2>::kBytes);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(out_proj_umma_kernel<224, 2>, smem, GemmLayout<224, 2>::kBytes);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(out_proj_skinny_kernel<16>, smem, SkinnyLayout<16>::kBytes);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(out_proj_skinny_kernel<32>, smem, SkinnyLayout<32>::kBytes);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(out_proj_skinny_kernel<64>, smem, SkinnyLayout<64>::kBytes);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(out_proj_skinny_kernel<128>, smem, SkinnyLayout<128>::kBytes);
  return int(e);
}

int launch_out_proj(const void* a, const void* w, void* c, int m, int n, int k, cudaStream_t stream) {
  TensorMapEncoder& enc = tensor_map_encoder();
  if (int rc = enc.init()) return rc;
  // Fewer 128 x 128 tiles than half the CTA slots (two per SM): split K over a cluster, by the largest power of two up to 8
  // that keeps the CTAs within the slots and at least two K steps in each.
  const long long tiles = ((n + kTileM - 1LL) / kTileM) * ((m + 127LL) / 128), k_tiles = (k + kTileK - 1LL) / kTileK;
  int split = 1;
  while (split < 8 && tiles * split * 2 <= 2 * kSms && k_tiles >= 4 * split) split *= 2;
  if (split > 1) {
    if (m <= 16) return launch_skinny<16>(enc, a, w, c, m, n, k, split, stream);
    if (m <= 32) return launch_skinny<32>(enc, a, w, c, m, n, k, split, stream);
    if (m <= 64) return launch_skinny<64>(enc, a, w, c, m, n, k, split, stream);
    return launch_skinny<128>(enc, a, w, c, m, n, k, split, stream);
  }
  // A K step takes an SM 512 cycles for a 128 x 128 tile, 768 for a 128 x 256, 1280 for a 256 x 256 and 1184 for a 256 x 224 one
  // (shared memory, see GemmLayout; measured 0.43 us and 0.69 for the second and third): the form whose turns are the shortest in all.
  // The ends of the turns are not counted.  At K 256 to 1024 (N 1024, 2560, 5120, M 1000 to 16000, calls back to back) the form
  // taken is within 1 % of the fastest of the four at 99 of 108 sizes, wherever it has 256 rows among them.  The others are sizes
  // whose third turn of 128 x 256 tiles is nearly empty, while two 128 x 128 CTAs an SM overlap their ends (M 4000, N 2560:
  // K 256 14.5 us and 12.8 as 128 x 128, K 512 18.4 and 17.3, K 768 22.7 and 22.1, K 1024 26.3 and 26.6).
  const auto cost = [&](long long width, int rows, int cycles) {
    const long long all = ((n + width - 1) / width) * ((m + rows - 1LL) / rows);
    return (all + kSms - 1) / kSms * cycles;
  };
  const long long small = cost(128, 128, 512), wide = cost(256, 128, 768), square = cost(256, 256, 1280), narrow = cost(224, 256, 1184);
  if (square < wide && square < small && square <= narrow) return launch_tiles<256, 2>(enc, a, w, c, m, n, k, stream);
  if (narrow < wide && narrow < small) return launch_tiles<224, 2>(enc, a, w, c, m, n, k, stream);
  return wide < small ? launch_tiles<256, 1>(enc, a, w, c, m, n, k, stream) : launch_tiles<128, 1>(enc, a, w, c, m, n, k, stream);
}

}  // namespace gdn_sm100

using namespace gdn_sm100;

extern "C" int actlize_la_sm100_out_proj(const void* a, const void* w, void* c, int m, int n, int k, void* stream) {
  if (!a || !w || !c || m <= 0 || n <= 0 || k <= 0) return int(cudaErrorInvalidValue);
  if ((n & 7) || (k & 7)) return int(cudaErrorInvalidValue);               // 16-byte rows for TMA and the stores
  if ((reinterpret_cast<uintptr_t>(a) & 15) || (reinterpret_cast<uintptr_t>(w) & 15) || (reinterpret_cast<uintptr_t>(c) & 15))
    return int(cudaErrorInvalidValue);
  if ((m + kTileM - 1) / kTileM > 65535) return int(cudaErrorInvalidValue);
  return launch_out_proj(a, w, c, m, n, k, static_cast<cudaStream_t>(stream));
}
