// Fine (block-sparse) attention on the Blackwell tensor path: TMA tile gathers by block id, tcgen05.mma with accumulators in tensor
// memory, warp-specialised elementwise stages.  This file has the host side, the self-tests and the choice between the kernels:
//   sparse_split.inl     64-row tiles, a tile of the other side per lane half (blocks of 64 tokens; larger ones on small grids or with short routes)
//   sparse_wide.inl      128-row tiles (blocks of 128 and 256 tokens)
//   sparse_umma_bwd.inl  the opt-in backward that forms dS once
//   coarse_umma.inl      the pooled branch
// The softmax of every forward uses a fixed shift, the row maximum over the first live tiles: softmax is shift-invariant, so a later
// score simply gives P = 2^(s-m) > 1, which bf16 and fp32 hold up to 2^127.  If a sum or an output leaves the finite range the tile
// writes NaN into its log-sum-exp rows and the exact warp-level kernel recomputes just those tiles in a follow-up launch.
// Every mbarrier wait is bounded; on a time-out the CTA records an error code in a device status word, stops issuing work, frees
// its tensor memory and returns.
#include <cuda.h>

#include <algorithm>
#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "kernels.h"
#include "umma.cuh"

namespace vsa {

__device__ int g_device_status = 0;

namespace {

using bf16 = __nv_bfloat16;
using namespace umma;

constexpr int kD = 128;
constexpr int kTile = 64;
constexpr int kMaxTiles = 1024;        // live 64-token key tiles per query tile the list can hold
constexpr int kSlab = 64 * 128;        // one TMA box: 64 rows x 128 bytes
constexpr int kPairHalf = 2 * kSlab;   // 128 rows x 128 bytes (one head-dim half of a stacked pair)
constexpr int kPairBytes = 2 * kPairHalf;
constexpr uint32_t kTmemCols = 512;

// ---- host: tensor maps ---------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

// [rows, cols] row-major of a 16-bit element type (cols = 128: q/k/v-like tensors; cols = 64: stored dS tiles), boxes of box_rows
// rows x 64 columns, 128-byte swizzle.
int make_map_of(CUtensorMap* map, CUtensorMapDataType elem, const void* ptr, int64_t rows, const char* what, int cols = kD, int box_rows = 64) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return fail(VSA_ERR_LAUNCH, "%s: cuTensorMapEncodeTiled is not available from the driver", what);
  if (reinterpret_cast<uintptr_t>(ptr) % 16) return fail(VSA_ERR_BAD_ARGUMENT, "%s: pointer is not 16-byte aligned", what);
  if (rows > 0x7fffffffLL) return fail(VSA_ERR_UNSUPPORTED, "%s: %lld rows exceed the TMA coordinate range", what, (long long)rows);
  const cuuint64_t gdim[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t gstride[1] = {(cuuint64_t)cols * 2};
  const cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = fn(map, elem, 2, const_cast<void*>(ptr), gdim, gstride, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(VSA_ERR_LAUNCH, "%s: cuTensorMapEncodeTiled failed with code %d", what, (int)r);
  return VSA_OK;
}

__device__ __forceinline__ void report_timeout(int code) { atomicCAS(&g_device_status, 0, code); }
// all waits of this file poll the status word so that a failure anywhere drains the grid quickly
#define VSA_WAIT(bar_, parity_) mbar_wait((bar_), (parity_), &g_device_status)
#define VSA_WARP_WAIT(bar_, parity_) warp_wait((bar_), (parity_), &g_device_status)
#define VSA_WARP_WAIT2(a_, pa_, b_, pb_) (VSA_WARP_WAIT(a_, pa_) && VSA_WARP_WAIT(b_, pb_))
#define VSA_WARP_WAIT3(a_, pa_, b_, pb_, c_, pc_) (VSA_WARP_WAIT(a_, pa_) && VSA_WARP_WAIT(b_, pb_) && VSA_WARP_WAIT(c_, pc_))
#define VSA_WARP_WAIT_TEST(a_, pa_, b_, pb_, done_) warp_wait_and_test((a_), (pa_), (b_), (pb_), &g_device_status, (done_))

// One 64x128 tile = two boxes (head-dim halves); `dst` is the row offset inside a stacked pair.
__device__ __forceinline__ void load_tile(uint32_t pair_base, int half_rows_off, const CUtensorMap* map, int row,
                                          uint32_t bar) {
  tma_load_2d(pair_base + half_rows_off, map, 0, row, bar);
  tma_load_2d(pair_base + kPairHalf + half_rows_off, map, 64, row, bar);
}

// ---- descriptor / TMEM self-test ---------------------------------------------------------------------
// mode 0: D[128x64] = A[128 x 128 (k contiguous)] * B[64 x 128 (k contiguous)]^T
// mode 1: D[128x64] = A[128 k x 128 m (m contiguous)]^T * B[128 k x 64 n (n contiguous)], B written by threads
__global__ void __launch_bounds__(128) umma_selftest_kernel(const __grid_constant__ CUtensorMap map_a,
                                                            const __grid_constant__ CUtensorMap map_b,
                                                            const bf16* __restrict__ b_raw, float* __restrict__ out,
                                                            int mode) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t sA = base, sB = base + kPairBytes;
  const uint32_t bar_load = base + kPairBytes + 16384, bar_mma = bar_load + 8, tmem_slot = bar_load + 16;
  const int tid = threadIdx.x, warp = tid >> 5;
  if (tid == 0) {
    mbar_init(bar_load, 1);
    mbar_init(bar_mma, 1);
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc(tmem_slot, 64);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(base_ptr + kPairBytes + 16384 + 16);
  bool ok = true;
  if (mode == 1) {   // B rows written by their owner thread as swizzled 128-byte rows
    const uint4* src = reinterpret_cast<const uint4*>(b_raw + tid * 64);
#pragma unroll
    for (int c = 0; c < 8; ++c)
      *reinterpret_cast<uint4*>(base_ptr + kPairBytes + tid * 128 + ((c ^ (tid & 7)) << 4)) = src[c];
    fence_proxy_async_smem();
  }
  __syncthreads();
  if (tid == 0) {
    const uint32_t bytes = kPairBytes + (mode == 0 ? 2 * kSlab : 0);
    mbar_arrive_expect_tx(bar_load, bytes);
    load_tile(sA, 0, &map_a, 0, bar_load);
    load_tile(sA, kSlab, &map_a, 64, bar_load);
    if (mode == 0) {
      tma_load_2d(sB, &map_b, 0, 0, bar_load);
      tma_load_2d(sB + kSlab, &map_b, 64, 0, bar_load);
    }
    ok = VSA_WAIT(bar_load, 0);
    if (ok) {
      tc_fence_after();
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        if (mode == 0) {
          const uint32_t off = (ks >> 2) * kPairHalf + (ks & 3) * 32;
          const uint32_t offb = (ks >> 2) * kSlab + (ks & 3) * 32;
          mma_ss(tmem, smem_desc(sA + off, 16, 1024), smem_desc(sB + offb, 16, 1024), instr_desc(128, 64, 0, 0), ks > 0);
        } else {
          mma_ss(tmem, smem_desc(sA + ks * 2048, kPairHalf, 1024), smem_desc(sB + ks * 2048, 16, 1024),
                 instr_desc(128, 64, 1, 1), ks > 0);
        }
      }
      mma_commit(bar_mma);
    } else {
      report_timeout(101);
    }
  }
  __syncthreads();
  if (VSA_WAIT(bar_mma, 0)) {
    tc_fence_after();
    uint32_t r[32];
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + half * 32, r);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 32; ++j) out[tid * 64 + half * 32 + j] = __uint_as_float(r[j]);
    }
  } else {
    report_timeout(102);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 64);
}

// ---- bounded-wait self-test ---------------------------------------------------------------------------
// One warp waits, with a caller-chosen limit, on a barrier that nothing will ever arrive at.  The wait must give
// up, the code must land in the device status word, and the kernel must return normally: the path every product
// kernel takes when a producer or a tensor-core commit fails to show up, exercised without making anything fail.
constexpr int kSelftestTimeoutCode = 201;
__global__ void __launch_bounds__(32) wait_timeout_selftest_kernel(unsigned long long limit_ns, int* __restrict__ gave_up) {
  __shared__ __align__(8) unsigned long long bar_storage;
  const uint32_t bar = smem_u32(&bar_storage);
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    fence_barrier_init();
  }
  __syncwarp();
  if (threadIdx.x == 0) {
    const bool ok = mbar_wait(bar, 0, &g_device_status, limit_ns);
    if (!ok) report_timeout(kSelftestTimeoutCode);
    *gave_up = ok ? 0 : 1;
  }
}

// [batch, rows, cols] of a 16-bit element type, rows `pitch` elements apart (0: dense); boxes of 64 columns x box_rows rows of one batch slice, 128-byte swizzle.
int make_map3d_of(CUtensorMap* map, CUtensorMapDataType elem, const void* ptr, int64_t batch, int64_t rows, int64_t cols, int box_rows,
               const char* what, int64_t pitch = 0) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return fail(VSA_ERR_LAUNCH, "%s: cuTensorMapEncodeTiled is not available from the driver", what);
  if (pitch == 0) pitch = cols;
  if (reinterpret_cast<uintptr_t>(ptr) % 16 || (pitch * 2) % 16)
    return fail(VSA_ERR_BAD_ARGUMENT, "%s: pointer or row pitch is not 16-byte aligned", what);
  const cuuint64_t gdim[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)batch};
  const cuuint64_t gstride[2] = {(cuuint64_t)pitch * 2, (cuuint64_t)rows * pitch * 2};
  const cuuint32_t box[3] = {64, (cuuint32_t)box_rows, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = fn(map, elem, 3, const_cast<void*>(ptr), gdim, gstride, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(VSA_ERR_LAUNCH, "%s: cuTensorMapEncodeTiled failed with code %d", what, (int)r);
  return VSA_OK;
}

template <typename Kern>
int reserve_smem(Kern kern, int bytes, const char* what, bool two_per_sm = false) {
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess && two_per_sm) e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  if (e != cudaSuccess) return fail(VSA_ERR_LAUNCH, "%s: shared memory: %s", what, cudaGetErrorString(e));
  return VSA_OK;
}

int check_kv_shard(int64_t Lkv, int be, int64_t* kv_shard, const char* what) {
  if (*kv_shard <= 0) *kv_shard = Lkv;
  if (Lkv % *kv_shard || *kv_shard % be)
    return fail(VSA_ERR_BAD_ARGUMENT, "%s: the K/V shard length %lld must divide Lkv = %lld and be a multiple of the block volume %d",
                what, (long long)*kv_shard, (long long)Lkv, be);
  return VSA_OK;
}

}  // namespace

// The kernels of the stored-dS backward walk a block of 64, 128 or 256 tokens as 1, 2 or 4 tiles (their SUB parameter).
#define VSA_BY_BLOCK_VOLUME(be_, launch_, kernel_) \
  return (be_) == 64 ? launch_(kernel_<1>) : (be_) == 128 ? launch_(kernel_<2>) : launch_(kernel_<4>)

// The kernels exist once per 16-bit element type: same code, other input format in the instruction descriptor and
// the tensor maps, other conversions in the epilogues.
namespace tc_bf16 {
using elem_t = __nv_bfloat16;
constexpr uint32_t kInFmt = 1u;
constexpr CUtensorMapDataType kTmaElem = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
constexpr int kDtypeCode = VSA_BF16;
constexpr float kShiftBias = 0.f;
#include "sparse_umma_typed.inl"
}  // namespace tc_bf16
namespace tc_f16 {
using elem_t = __half;
constexpr uint32_t kInFmt = 0u;
constexpr CUtensorMapDataType kTmaElem = CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
constexpr int kDtypeCode = VSA_F16;
// The forward's fixed softmax shift is the first pair's column maximum plus this many binades, so that P = 2^(s - shift)
// of the first pair tops out at 2^-4: fp16 then holds later scores up to 20 binades (13.9 nats) above the first pair's
// maximum before P overflows (and the tile goes to the exact kernel) and keeps scores down to 20 binades below it --
// the middle of fp16's 2^-24 .. 2^16 instead of its top.  The row sum uses the same shift, so O/l and the saved
// statistic are unchanged.  bf16 has 2^127 above the first pair's maximum and needs no bias.
// (The 128-row forward at head dim 64 does without it; see there.)
constexpr float kShiftBias = 4.f;
#include "sparse_umma_typed.inl"
}  // namespace tc_f16

#define VSA_BY_DTYPE(dtype_, call_) ((dtype_) == VSA_F16 ? tc_f16::call_ : tc_bf16::call_)

// ---- host entry points ---------------------------------------------------------------------------------------
// The SM count decides between kernels only; without a device (a query on a build machine) a B200's is assumed.
static int sm_count() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && sms > 0)
    return sms;
  cudaGetLastError();
  return 148;
}

// Head dim 64, blocks of 128 and 256 tokens: whether the 128-row kernels are faster than both the 64-row tcgen05 kernels and
// mma.sync.  us, 64-row / 128-row / mma.sync, blocks of 128, by tiles of 64 a route:
//   [1, 2, 4096, 64], 128 row tiles    forward 8: 11.1 / 12.5 / 11.6, 16: 13.7 / 15.0 / 20.0;  dQ 4: 7.1 / 7.9 / 7.4, 16: 10.3 / 13.0 / 21.4;
//                                      dK/dV 2: 8.9 / 11.4 / 11.8, 16: 17.0 / 26.4 / 35.8: never
//   [1, 4, 4096, 64], 256              forward 6: 12.4 / 12.3 / 11.8, 8: 13.5 / 13.0 / 14.7;  dQ 2: 11.9 / 7.2 / 6.3, 4: 12.7 / 8.3 / 9.7;
//                                      dK/dV 4: 15.7 / 14.6 / 20.3, 6: 17.5 / 19.0 / 26.5 (blocks of 256, 16: 29.7 / 36.8 / 68.7)
//   [1, 3, 8192, 64], 384              forward 12: 23.5 / 25.2 / 24.7, 24: 32.1 / 32.9 / 45.5;  dQ 4: 18.1 / 14.7 / 12.3, 6: 19.9 / 16.5 / 16.5;
//                                      dK/dV 4: 20.5 / 18.2 / 26.9, 16: 36.6 / 37.4 / 62.9
//   [1, 4, 8192, 64], 512              forward 8: 22.9 / 22.8 / 21.4, 10: 24.7 / 24.2 / 25.9, 16: 29.7 / 28.0 / 38.9
//   [1, 12, 16384, 64], 3072           forward, 0.2 s of back-to-back calls (power limit), 12: 136 / 140 / 151, 16: 153 / 154 / 195,
//                                      24: 195 / 183 / 285;  dQ 4: 125 / 85 / 77, 6: 136 / 94 / 106;
//                                      dK/dV 2: 103 / 66 / 61, 4: 132 / 89 / 100, 16: 241 / 190 / 329
// With the pooled gradients (`fused`) dQ crosses earlier while the grid is small: 256 row tiles, 2: 12.9 / 7.7 / 10.4; 640, 4: 31.2 / 22.4 /
// 24.1; 3072, 4: 138 / 92 / 85.
static bool sparse_wide64_pays(SparsePass pass, int64_t tiles, int64_t n, bool fused) {
  const int64_t sms = sm_count(), waves = (tiles + sms - 1) / sms;
  if (waves == 1) return false;
  if (pass == kPassForward) return n >= (waves == 2 ? 8 : waves == 4 ? 10 : 18);
  if (pass == kPassDkdv) return waves > 2 || n < 6;
  return n >= (waves == 2 ? 4 : 6) - (fused && waves <= 8 ? 2 : 0);
}
// Head dim 64 on 64-row tiles: tcgen05 (sparse_split.inl; the forward has two CTAs on an SM, the backward one) or mma.sync, of which
// three or four CTAs share an SM and need little set-up, so that they are faster while a route holds few tiles: the longer, the less
// the 64-row tcgen05 tiles fill their last wave.  us, tcgen05 / mma.sync, blocks of 64, by tiles per route:
//   [1, 2, 4096, 64], 128 row tiles    forward 2: 9.4 / 5.0, 7: 11.7 / 10.9, 8: 11.2 / 11.9;  dQ 1: 6.9 / 3.7, 3: 7.2 / 6.5, 4: 7.1 / 7.6;
//                                      dK/dV 1: 7.4 / 7.0, 2: 8.2 / 8.2, 3: 8.8 / 10.6
//   [1, 4, 4096, 64], 256              forward 7: 13.5 / 13.1, 8: 13.5 / 14.3;  dQ 7: 15.3 / 14.8, 8: 15.0 / 16.3;  dK/dV 2: 13.4 / 11.9, 3: 15.6 / 15.4
//   [1, 3, 8192, 64], 384              forward 10: 22.1 / 21.0, 12: 23.6 / 24.4;  dQ 8: 21.4 / 20.7, 10: 23.0 / 24.9;  dK/dV 4: 22.1 / 21.3, 5: 23.4 / 25.1
//   [1, 5, 8192, 64], 640              forward 8: 29.9 / 28.8, 10: 32.2 / 34.9;  dQ 8: 34.1 / 34.0, 10: 36.9 / 41.4;  dK/dV 5: 34.5 / 33.9, 6: 37.5 / 39.1
//   [1, 12, 8192, 64], 1536            forward 9: 64.7 / 59.9, 10: 63.5 / 65.8;  dQ 9: 80.9 / 78.7, 10: 79.8 / 85.7;  dK/dV 7: 84.6 / 83.2, 8: 89.8 / 93.8
//   [1, 12, 16384, 64], 3072           forward 9: 126 / 114, 10: 124 / 125, 12: 133 / 146;  dQ 9: 162 / 149, 10: 159 / 163;  dK/dV 8: 178 / 172, 9: 187 / 191
// With the pooled gradients (`fused`) mma.sync needs one more launch per gradient, which moves the line on small grids: 128 row tiles,
// dQ 1: 7.4 / 6.3, 2: 7.2 / 7.6, dK/dV 1: 7.4 / 12.0; 256, dQ 5: 15.2 / 14.2, 6: 14.9 / 15.9; 3072, dQ 9: 177 / 156, 12: 184 / 199,
// dK/dV 7: 176 / 168, 8: 185 / 188.  At no point measured is the slower side taken by more than 5 %.
bool sparse_split64_pays(SparsePass pass, int64_t BH, int64_t L, int be, int topk, bool fused) {
  const int64_t n = (int64_t)topk * (be / kTile), sms = sm_count(), tiles = BH * (L / kTile), waves = (tiles + sms - 1) / sms;
  if (pass == kPassForward) return n >= (waves <= 2 ? 8 : waves == 3 ? 12 : 10);
  if (pass == kPassDq) return n >= (waves == 1 ? 4 : waves <= 5 ? 8 : 10) - (fused && waves <= 2 ? 2 : 0);
  if (be > kTile) return true;      // [1, 2, 4096, 64], 2: 8.9 / 11.8; longer routes and larger grids: the 128-row kernels are asked first
  return n >= std::min<int64_t>({waves + 1, 5 + waves / 4, 9}) - (fused ? (waves < 8 ? 2 : 1) : 0);
}

// Whether blocks of 128 and 256 tokens take the 128-row kernels (sparse_wide.inl) or are walked as 64-row tiles (sparse_split.inl).
// A 128-row CTA does twice the rows in less than twice the time, so 64-row tiles are the faster ones where they all are on the SMs at
// once.  us, 64-row / 128-row, head dim 128, full blocks of 128, by tiles of 64 a route (one B200):
//   [1, 2, 4096], 128 row tiles    forward 2: 11.4 / 12.5, 8: 13.3 / 15.6, 32: 20.9 / 24.2;  dQ 7.7 / 8.7, 10.0 / 11.8, 19.0 / 24.4;
//                                  dK/dV 10.2 / 12.3, 15.1 / 20.7, 25.7 / 37.8
// Beyond that the 128-row dQ is faster at every point measured (192 to 11,520 row tiles, 2 to 64 tiles a route), dK/dV at all but a
// few of one or two waves (blocks of 256, [1, 3, 4096], 4: 12.3 / 15.2):
//   [1, 3, 4096], 192              dQ 4: 14.2 / 9.7, 8: 16.9 / 12.1, 32: 33.0 / 24.5;  dK/dV 16.7 / 15.1, 21.7 / 19.8, 40.6 / 42.6
//   [1, 3, 8192], 384              dQ 4: 21.1 / 18.2, 8: 24.9 / 22.7, 32: 48.5 / 47.9;  dK/dV 24.3 / 21.9, 29.7 / 25.7, 62.8 / 62.8
//   [1, 12, 16384], 3072           dQ 4: 156 / 118, 8: 178 / 137, 32: 358 / 296;  dK/dV 155 / 104, 199 / 137, 457 / 350
// The 64-row forward has two CTAs on an SM and less to set up: it is ahead for short routes, and on grids of three to five waves, where
// 128-row CTAs leave half of their last wave empty, for longer ones.  With many waves the board's power limit decides; these are
// times of 0.3 s of back-to-back calls:
//   [1, 4, 4096], 256              forward 4: 13.9 / 14.3, 16: 19.1 / 19.4, 20: 20.9 / 20.5, 32: 26.1 / 25.2, 64: 40.0 / 37.0
//   [1, 5, 8192], 640              forward 4: 33.6 / 36.5, 16: 46.5 / 51.1, 32: 64.7 / 68.7, 40: 75.3 / 76.8, 64: 107 / 104
//   [1, 12, 8192], 1536            forward 16: 104 / 110, 24: 132 / 129, 64: 267 / 236
//   [1, 12, 16384], 3072           forward 16: 198 / 199, 24: 252 / 237, 64: 512 / 449
//   [1, 8, 92160], 11520           forward 16: 729 / 695, 24: 923 / 862, 64: 1883 / 1661
bool sparse_wide_rows(SparsePass pass, int64_t BH, int64_t L, int D, int be, int topk, bool fused) {
  if (be % 128 != 0) return false;
  const int64_t tiles = BH * (L / kTile), n = (int64_t)topk * (be / kTile);
  if (D == 64) return sparse_wide64_pays(pass, tiles, n, fused);
  const int64_t sms = sm_count(), waves = (tiles + sms - 1) / sms;
  return waves > 1 && (pass != kPassForward || n > (waves > 2 && waves <= 5 ? 40 : 16));
}

bool sparse_umma_eligible(int D, int be, int dtype, int topk) {
  if ((dtype != VSA_BF16 && dtype != VSA_F16) || D != 128) return false;
  if (be == 64 || be == 128 || be == 256) return topk * (be / kTile) <= kMaxTiles;
  return false;
}

bool sparse_umma64_eligible(int D, int be, int dtype, int topk) {
  return D == 64 && (be == 64 || be == 128 || be == 256) && (dtype == VSA_BF16 || dtype == VSA_F16) && topk * (be / kTile) <= kMaxTiles;
}

int64_t sparse_ds_workspace_bytes(int64_t BH, int64_t Lq, int be, int topk) {
  const int64_t sub = be / kTile;
  return BH * (Lq / be) * topk * sub * sub * (int64_t)(kTile * kTile * 2);
}

int sparse_fwd_umma(const void* q, const void* k, const void* v, const int32_t* selected, const int32_t* kv_sizes,
                    void* out, float* lse2, int64_t BH, int64_t Lq, int64_t Lkv, int D, int be, int topk, float scale,
                    int dtype, cudaStream_t st, const void* out_c, const void* gate, void* out_comb, int64_t kv_shard,
                    const int32_t* comb_map, int64_t comb_rows, int comb_heads) {
  const RasterMap rm{comb_map, (long long)comb_rows, comb_heads > 0 ? comb_heads : 1};
  return VSA_BY_DTYPE(dtype, sparse_fwd_umma(q, k, v, selected, kv_sizes, out, lse2, BH, Lq, Lkv, D, be, topk, scale, st,
                                             out_c, gate, out_comb, kv_shard, rm));
}

int sparse_dq_umma(const void* dout, const void* q, const void* k, const void* v, const void* out_s,
                   const float* lse2, const int32_t* selected, const int32_t* kv_sizes, float* delta, void* dq,
                   int64_t BH, int64_t Lq, int64_t Lkv, int D, int be, int topk, float scale, int dtype, cudaStream_t st,
                   const void* dq_mean, const int32_t* q_sizes, int64_t kv_shard, const int32_t* out_map,
                   int64_t out_rows, int out_heads) {
  const RasterMap rm{out_map, (long long)out_rows, out_heads > 0 ? out_heads : 1};
  return VSA_BY_DTYPE(dtype, sparse_dq_umma(dout, q, k, v, out_s, lse2, selected, kv_sizes, delta, dq, BH, Lq, Lkv, D, be,
                                            topk, scale, st, dq_mean, q_sizes, kv_shard, rm));
}

int sparse_dkdv_umma(const void* dout, const void* q, const void* k, const void* v, const float* lse2,
                     const float* delta, const int32_t* counts, const int32_t* offsets, const int32_t* inverse,
                     const int32_t* kv_sizes, void* dk, void* dv, int64_t BH, int64_t Lq, int64_t Lkv, int D, int be, int topk,
                     float scale, int dtype, cudaStream_t st, const void* dk_mean, const void* dv_mean, void* ds_ws,
                     int64_t kv_shard, const int32_t* out_map, int64_t out_rows, int out_heads) {
  const RasterMap rm{out_map, (long long)out_rows, out_heads > 0 ? out_heads : 1};
  return VSA_BY_DTYPE(dtype, sparse_dkdv_umma(dout, q, k, v, lse2, delta, counts, offsets, inverse, kv_sizes, dk, dv, BH,
                                              Lq, Lkv, D, be, topk, scale, st, dk_mean, dv_mean, ds_ws, kv_shard, rm));
}

int sparse_dq_from_ds_umma(const void* k, const int32_t* selected, const int32_t* kv_sizes, const void* ds_ws, void* dq,
                           int64_t BH, int64_t Lq, int64_t Lkv, int be, int topk, float scale, int dtype,
                           cudaStream_t st, const void* dq_mean, const int32_t* q_sizes) {
  return VSA_BY_DTYPE(dtype, sparse_dq_from_ds_umma(k, selected, kv_sizes, ds_ws, dq, BH, Lq, Lkv, be, topk, scale, st,
                                                    dq_mean, q_sizes));
}

// ---- pooled attention on tcgen05 ---------------------------------------------------------------------------
// head dim 64: the same kernel, the second 64-column box of a 128-wide tile lies outside the tensor and is zero-filled.
// Block counts are free: what TMA wants is a row pitch of 16 bytes, which the caller gives `probs` and dS.  At 1441 blocks and
// eight slices the pooled forward takes 0.46 ms instead of 0.65 with every product on the CUDA cores, and a training step on
// an 81,000-token raster grid (1380 blocks, eight heads) 25.7 ms instead of 26.5.
bool coarse_umma_eligible(int Kb, int pitch, int D, int dtype) {
  return (dtype == VSA_BF16 || dtype == VSA_F16) && (D == 128 || D == 64) && pitch >= Kb && pitch % 8 == 0;
}

int coarse_fwd_umma(const void* qc, const void* kc, const void* vc, void* scores, void* probs, void* out_c, int64_t BH,
                    int Qb, int Kb, int pitch, int D, float scale, int dtype, cudaStream_t st) {
  return VSA_BY_DTYPE(dtype, coarse_fwd_umma(qc, kc, vc, scores, probs, out_c, BH, Qb, Kb, pitch, D, scale, st));
}

int coarse_bwd_umma(const void* d_out_c, const void* out_c, const void* qc, const void* kc, const void* vc,
                    const void* probs, void* ds, float* rowdot, void* dqc, void* dkc, void* dvc, int64_t BH, int Qb,
                    int Kb, int pitch, int D, float scale, int dtype, cudaStream_t st) {
  return VSA_BY_DTYPE(dtype, coarse_bwd_umma(d_out_c, out_c, qc, kc, vc, probs, ds, rowdot, dqc, dkc, dvc, BH, Qb, Kb, pitch,
                                             D, scale, st));
}

int umma_selftest(const void* a, const void* b, float* out, int mode, cudaStream_t st) {
  CUtensorMap ma, mb;
  int rc;
  if ((rc = make_map_of(&ma, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, a, 128, "selftest (a)"))) return rc;
  if ((rc = make_map_of(&mb, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, mode == 0 ? b : a, mode == 0 ? 64 : 128, "selftest (b)"))) return rc;
  const int smem = kPairBytes + 16384 + 64 + 1024;
  const cudaError_t e = cudaFuncSetAttribute(umma_selftest_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return fail(VSA_ERR_LAUNCH, "selftest: shared memory: %s", cudaGetErrorString(e));
  umma_selftest_kernel<<<1, 128, smem, st>>>(ma, mb, (const bf16*)b, out, mode);
  return check_launch("umma_selftest_kernel");
}

int wait_timeout_selftest(unsigned long long limit_ns, int* gave_up, cudaStream_t st) {
  wait_timeout_selftest_kernel<<<1, 32, 0, st>>>(limit_ns, gave_up);
  return check_launch("wait_timeout_selftest_kernel");
}

int device_status_fetch_and_clear(int* status) {
  int zero = 0;
  cudaError_t e = cudaMemcpyFromSymbol(status, g_device_status, sizeof(int));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_device_status, &zero, sizeof(int));
  if (e != cudaSuccess) return fail(VSA_ERR_LAUNCH, "device status: %s", cudaGetErrorString(e));
  return VSA_OK;
}

}  // namespace vsa
