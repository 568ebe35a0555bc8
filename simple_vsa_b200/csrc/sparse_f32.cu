// Fine attention in fp32 on tiles of 64 query rows x 64 key rows, for blocks of 64, 128 or 256 tokens and head dims 64
// and 128 (the row kernels in generic_kernels.cu keep every other shape).
//
// Bound by the FP32 pipe: 256 threads, a 4 x 4 patch of scores and 4 rows x D/16 dims of the products each, so that a
// 16-byte shared-memory read feeds 8 to 16 multiply-adds.  The row kernels spend a warp reduction per score and re-read
// every K and V row once per query row.  Rows are padded by 16 bytes: the 16 rows that a half-warp reads at once then fall
// into different banks.  Measured against the row kernels, ms for forward / dQ / dK/dV: [1, 4, 4096, 128], topk 8:
// 0.96 / 1.13 / 1.45 -> 0.15 / 0.22 / 0.38 (a fifth to a third of the FP32 peak: one CTA of eight warps per SM at this head
// dim); [1, 2, 1024, 64], topk 4: 0.111 / 0.114 / 0.233 -> 0.033 / 0.038 / 0.083 (32 CTAs for 148 SMs).
#include "common.cuh"
#include "kernels.h"

namespace vsa {
namespace {

constexpr int kT = 64;                 // tile edge
constexpr int kThreads = 256;
constexpr int kPad = kT + 4;           // row pitch of the score tile

template <int D> constexpr int kPitch = D + 4;
template <int D> constexpr int kTileFloats = kT * kPitch<D>;
constexpr int kScoreFloats = kT * kPad;

// A 64 x D tile: registers first (the loads fly under the arithmetic in between), shared memory later.
template <int D>
struct TileRegs {
  static constexpr int N = kT * D / 4 / kThreads;
  float4 r[N];
  __device__ __forceinline__ void fetch(const float* __restrict__ g, int rows, int tid) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int e = tid + i * kThreads, row = e / (D / 4), c = e % (D / 4);
      r[i] = row < rows ? *reinterpret_cast<const float4*>(g + row * D + c * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  __device__ __forceinline__ void put(float* sm, int tid) const {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int e = tid + i * kThreads, row = e / (D / 4), c = e % (D / 4);
      *reinterpret_cast<float4*>(sm + row * kPitch<D> + c * 4) = r[i];
    }
  }
};

// s[i][j] = sum_d a[4 ty + i][d] * b[tx + 16 j][d], summed in pieces of 16: one addition more per 16 products, and a chain of
// 16 + D/16 roundings instead of D (with one chain the result was further from float64 than that of the row kernels, whose
// lanes hold a few products each).
template <int D>
__device__ __forceinline__ void scores(float (&s)[4][4], const float* a, const float* b, int tx, int ty) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 1
  for (int d0 = 0; d0 < D; d0 += 16) {
    float t[4][4] = {};
#pragma unroll
    for (int d = d0; d < d0 + 16; d += 4) {
      float4 x[4], y[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) x[i] = *reinterpret_cast<const float4*>(a + (4 * ty + i) * kPitch<D> + d);
#pragma unroll
      for (int j = 0; j < 4; ++j) y[j] = *reinterpret_cast<const float4*>(b + (tx + 16 * j) * kPitch<D> + d);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          t[i][j] = fmaf(x[i].w, y[j].w, fmaf(x[i].z, y[j].z, fmaf(x[i].y, y[j].y, fmaf(x[i].x, y[j].x, t[i][j]))));
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) s[i][j] += t[i][j];
  }
}

// acc[i][4 h + e] += sum_n p[4 ty + i][n] * b[n][64 h + 4 tx + e]
template <int D>
__device__ __forceinline__ void product(float (&acc)[4][D / 16], const float* p, const float* b, int tx, int ty) {
#pragma unroll 2
  for (int n = 0; n < kT; n += 4) {
    float4 w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = *reinterpret_cast<const float4*>(p + (4 * ty + i) * kPad + n);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
#pragma unroll
      for (int h = 0; h < D / 64; ++h) {
        const float4 x = *reinterpret_cast<const float4*>(b + (n + e) * kPitch<D> + 64 * h + 4 * tx);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float f = e == 0 ? w[i].x : e == 1 ? w[i].y : e == 2 ? w[i].z : w[i].w;
          acc[i][4 * h + 0] = fmaf(f, x.x, acc[i][4 * h + 0]);
          acc[i][4 * h + 1] = fmaf(f, x.y, acc[i][4 * h + 1]);
          acc[i][4 * h + 2] = fmaf(f, x.z, acc[i][4 * h + 2]);
          acc[i][4 * h + 3] = fmaf(f, x.w, acc[i][4 * h + 3]);
        }
      }
    }
  }
}

// Rows from `live` on are padding: they get zeros, not 0 * whatever stood in the rows summed over.
template <int D>
__device__ __forceinline__ void store_rows(float* __restrict__ g, const float (&acc)[4][D / 16], const float (&mul)[4], int tx, int ty,
                                           int live = kT) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int h = 0; h < D / 64; ++h)
      *reinterpret_cast<float4*>(g + (4 * ty + i) * D + 64 * h + 4 * tx) =
          4 * ty + i < live ? make_float4(acc[i][4 * h] * mul[i], acc[i][4 * h + 1] * mul[i], acc[i][4 * h + 2] * mul[i], acc[i][4 * h + 3] * mul[i])
                            : make_float4(0.f, 0.f, 0.f, 0.f);
}

__device__ __forceinline__ float half_warp_max(float x) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, o));
  return x;
}
__device__ __forceinline__ float half_warp_sum(float x) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// Walks the live 64-row key tiles of a query block's route.
struct KeyTiles {
  const int32_t* sel;
  const int32_t* sizes;
  int n, sub, Kb, it;
  long long token;     // first token of the current tile
  int left;            // its live tokens
  __device__ __forceinline__ bool next() {
    for (; ++it < n;) {
      const int kvb = sel[it / sub];
      left = (unsigned)kvb < (unsigned)Kb ? sizes[kvb] - (it % sub) * kT : 0;    // an id outside the table is an empty block
      if (left > 0) {
        left = left > kT ? kT : left;
        token = ((long long)kvb * sub + it % sub) * kT;
        return true;
      }
    }
    return false;
  }
};

template <int D>
__global__ void __launch_bounds__(kThreads)
sparse_fwd_f32_kernel(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v,
                      const int32_t* __restrict__ selected, const int32_t* __restrict__ kv_sizes, float* __restrict__ out,
                      float* __restrict__ lse2, long long Lq, long long Lkv, int be, int topk, float scale) {
  extern __shared__ __align__(16) float f32_sm[];
  float* sq = f32_sm;
  float* sk = sq + kTileFloats<D>;
  float* sv = sk + kTileFloats<D>;
  float* sp = sv + kTileFloats<D>;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const long long bh = blockIdx.y, row0 = bh * Lq + (long long)blockIdx.x * kT;
  const int sub = be / kT, qb = blockIdx.x / sub;
  const float c = scale * kLog2e;
  KeyTiles tiles{selected + (bh * (Lq / be) + qb) * (long long)topk, kv_sizes, topk * sub, sub, (int)(Lkv / be), -1, 0, 0};
  TileRegs<D> rk, rv;
  rk.fetch(q + row0 * D, kT, tid);
  rk.put(sq, tid);
  float acc[4][D / 16] = {}, m[4], l[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    m[i] = -INFINITY;
    l[i] = 0.f;
  }
  bool more = tiles.next();
  if (more) rk.fetch(k + (bh * Lkv + tiles.token) * D, tiles.left, tid);
  while (more) {
    const int left = tiles.left;
    rk.put(sk, tid);
    rv.fetch(v + (bh * Lkv + tiles.token) * D, left, tid);
    __syncthreads();
    float s[4][4];
    scores<D>(s, sq, sk, tx, ty);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float mx = m[i];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[i][j] = tx + 16 * j < left ? s[i][j] * c : -INFINITY;
        mx = fmaxf(mx, s[i][j]);
      }
      mx = half_warp_max(mx);
      const float alpha = exp2f(m[i] - mx);          // m == -inf on the first tile gives 0
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float p = tx + 16 * j < left ? exp2f(s[i][j] - mx) : 0.f;
        sp[(4 * ty + i) * kPad + tx + 16 * j] = p;
        sum += p;
      }
      l[i] = l[i] * alpha + half_warp_sum(sum);
      m[i] = mx;
#pragma unroll
      for (int e = 0; e < D / 16; ++e) acc[i][e] *= alpha;
    }
    rv.put(sv, tid);
    more = tiles.next();
    if (more) rk.fetch(k + (bh * Lkv + tiles.token) * D, tiles.left, tid);
    __syncthreads();
    product<D>(acc, sp, sv, tx, ty);
  }
  float inv[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) inv[i] = 1.f / l[i];
  store_rows<D>(out + row0 * D, acc, inv, tx, ty);
  if (lse2 && tx == 0)
#pragma unroll
    for (int i = 0; i < 4; ++i) lse2[row0 + 4 * ty + i] = m[i] + log2f(l[i]);
}

template <int D>
__global__ void __launch_bounds__(kThreads)
sparse_dq_f32_kernel(const float* __restrict__ dout, const float* __restrict__ q, const float* __restrict__ k,
                     const float* __restrict__ v, const float* __restrict__ out_s, const float* __restrict__ lse2,
                     const int32_t* __restrict__ selected, const int32_t* __restrict__ kv_sizes, float* __restrict__ delta,
                     float* __restrict__ dq, long long Lq, long long Lkv, int be, int topk, float scale) {
  extern __shared__ __align__(16) float f32_sm[];
  float* sq = f32_sm;
  float* sdo = sq + kTileFloats<D>;
  float* sk = sdo + kTileFloats<D>;
  float* sv = sk + kTileFloats<D>;
  float* sp = sv + kTileFloats<D>;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const long long bh = blockIdx.y, row0 = bh * Lq + (long long)blockIdx.x * kT;
  const int sub = be / kT, qb = blockIdx.x / sub;
  const float c = scale * kLog2e;
  KeyTiles tiles{selected + (bh * (Lq / be) + qb) * (long long)topk, kv_sizes, topk * sub, sub, (int)(Lkv / be), -1, 0, 0};
  TileRegs<D> rk, rv;
  rk.fetch(q + row0 * D, kT, tid);
  rk.put(sq, tid);
  rk.fetch(dout + row0 * D, kT, tid);
  rk.put(sdo, tid);
  __syncthreads();
  float acc[4][D / 16] = {}, lse[4], dl[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {      // delta = rowsum(out_s * dout), sixteen threads per row
    const int r = 4 * ty + i;
    float x = 0.f;
#pragma unroll
    for (int d = 0; d < D; d += 16) x = fmaf(out_s[(row0 + r) * D + d + tx], sdo[r * kPitch<D> + d + tx], x);
    dl[i] = half_warp_sum(x);
    lse[i] = lse2[row0 + r];
    if (tx == 0) delta[row0 + r] = dl[i];
  }
  bool more = tiles.next();
  if (more) {
    rk.fetch(k + (bh * Lkv + tiles.token) * D, tiles.left, tid);
    rv.fetch(v + (bh * Lkv + tiles.token) * D, tiles.left, tid);
  }
  while (more) {
    const int left = tiles.left;
    rk.put(sk, tid);
    rv.put(sv, tid);
    __syncthreads();
    more = tiles.next();
    float s[4][4], dp[4][4];
    scores<D>(s, sq, sk, tx, ty);
    scores<D>(dp, sdo, sv, tx, ty);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        sp[(4 * ty + i) * kPad + tx + 16 * j] = tx + 16 * j < left ? exp2f(s[i][j] * c - lse[i]) * (dp[i][j] - dl[i]) * scale : 0.f;
    if (more) {
      rk.fetch(k + (bh * Lkv + tiles.token) * D, tiles.left, tid);
      rv.fetch(v + (bh * Lkv + tiles.token) * D, tiles.left, tid);
    }
    __syncthreads();
    product<D>(acc, sp, sk, tx, ty);
    __syncthreads();
  }
  const float one[4] = {1.f, 1.f, 1.f, 1.f};
  store_rows<D>(dq + row0 * D, acc, one, tx, ty);
}

template <int D>
__global__ void __launch_bounds__(kThreads)
sparse_dkdv_f32_kernel(const float* __restrict__ dout, const float* __restrict__ q, const float* __restrict__ k,
                       const float* __restrict__ v, const float* __restrict__ lse2, const float* __restrict__ delta,
                       const int32_t* __restrict__ counts, const int32_t* __restrict__ offsets,
                       const int32_t* __restrict__ inverse, const int32_t* __restrict__ kv_sizes, float* __restrict__ dk,
                       float* __restrict__ dv, long long Lq, long long Lkv, int be, int topk, float scale) {
  extern __shared__ __align__(16) float f32_sm[];
  float* sk = f32_sm;
  float* sv = sk + kTileFloats<D>;
  float* sq = sv + kTileFloats<D>;
  float* sdo = sq + kTileFloats<D>;
  float* sp = sdo + kTileFloats<D>;
  float* sds = sp + kScoreFloats;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const long long bh = blockIdx.y, row0 = bh * Lkv + (long long)blockIdx.x * kT;
  const int sub = be / kT, kvb = blockIdx.x / sub, Kb = (int)(Lkv / be);
  const float c = scale * kLog2e;
  const int valid = kv_sizes[kvb] - (int)(blockIdx.x % sub) * kT;
  const int n = valid > 0 ? counts[bh * Kb + kvb] * sub : 0;
  const int32_t* inv = inverse + bh * (Lq / be) * (long long)topk + offsets[bh * Kb + kvb];
  auto tile = [&](int i) -> long long { return bh * Lq + (long long)inv[i / sub] * be + (i % sub) * kT; };
  TileRegs<D> rq, rd;
  rq.fetch(k + row0 * D, valid, tid);
  rq.put(sk, tid);
  rq.fetch(v + row0 * D, valid, tid);
  rq.put(sv, tid);
  float ak[4][D / 16] = {}, av[4][D / 16] = {};
  if (n > 0) {
    rq.fetch(q + tile(0) * D, kT, tid);
    rd.fetch(dout + tile(0) * D, kT, tid);
  }
  for (int it = 0; it < n; ++it) {
    const long long r0 = tile(it);
    rq.put(sq, tid);
    rd.put(sdo, tid);
    float lse[4], dl[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      lse[j] = lse2[r0 + tx + 16 * j];
      dl[j] = delta[r0 + tx + 16 * j];
    }
    __syncthreads();
    float s[4][4], dp[4][4];
    scores<D>(s, sk, sq, tx, ty);
    scores<D>(dp, sv, sdo, tx, ty);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float p = 4 * ty + i < valid ? exp2f(s[i][j] * c - lse[j]) : 0.f;
        sp[(4 * ty + i) * kPad + tx + 16 * j] = p;
        sds[(4 * ty + i) * kPad + tx + 16 * j] = 4 * ty + i < valid ? p * (dp[i][j] - dl[j]) : 0.f;
      }
    if (it + 1 < n) {
      rq.fetch(q + tile(it + 1) * D, kT, tid);
      rd.fetch(dout + tile(it + 1) * D, kT, tid);
    }
    __syncthreads();
    product<D>(av, sp, sdo, tx, ty);
    product<D>(ak, sds, sq, tx, ty);
    __syncthreads();
  }
  const float mk[4] = {scale, scale, scale, scale}, mv[4] = {1.f, 1.f, 1.f, 1.f};
  store_rows<D>(dk + row0 * D, ak, mk, tx, ty, valid);
  store_rows<D>(dv + row0 * D, av, mv, tx, ty, valid);
}

template <typename Kern>
int reserve(Kern kern, int floats, const char* what) {
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, floats * 4);
  if (e != cudaSuccess) return fail(VSA_ERR_LAUNCH, "%s: shared memory: %s", what, cudaGetErrorString(e));
  return VSA_OK;
}

template <int D>
int fwd(const float* q, const float* k, const float* v, const int32_t* selected, const int32_t* kv_sizes, float* out,
        float* lse2, dim3 grid, int64_t Lq, int64_t Lkv, int be, int topk, float scale, cudaStream_t st) {
  constexpr int floats = 3 * kTileFloats<D> + kScoreFloats;
  const int rc = reserve(sparse_fwd_f32_kernel<D>, floats, "sparse forward");
  if (rc) return rc;
  sparse_fwd_f32_kernel<D><<<grid, kThreads, floats * 4, st>>>(q, k, v, selected, kv_sizes, out, lse2, Lq, Lkv, be, topk, scale);
  return check_launch("sparse_fwd_f32_kernel");
}

template <int D>
int dq_pass(const float* dout, const float* q, const float* k, const float* v, const float* out_s, const float* lse2,
            const int32_t* selected, const int32_t* kv_sizes, float* delta, float* dq, dim3 grid, int64_t Lq, int64_t Lkv,
            int be, int topk, float scale, cudaStream_t st) {
  constexpr int floats = 4 * kTileFloats<D> + kScoreFloats;
  const int rc = reserve(sparse_dq_f32_kernel<D>, floats, "sparse dQ");
  if (rc) return rc;
  sparse_dq_f32_kernel<D><<<grid, kThreads, floats * 4, st>>>(dout, q, k, v, out_s, lse2, selected, kv_sizes, delta, dq, Lq, Lkv,
                                                              be, topk, scale);
  return check_launch("sparse_dq_f32_kernel");
}

template <int D>
int dkdv_pass(const float* dout, const float* q, const float* k, const float* v, const float* lse2, const float* delta,
              const int32_t* counts, const int32_t* offsets, const int32_t* inverse, const int32_t* kv_sizes, float* dk,
              float* dv, dim3 grid, int64_t Lq, int64_t Lkv, int be, int topk, float scale, cudaStream_t st) {
  constexpr int floats = 4 * kTileFloats<D> + 2 * kScoreFloats;
  const int rc = reserve(sparse_dkdv_f32_kernel<D>, floats, "sparse dK/dV");
  if (rc) return rc;
  sparse_dkdv_f32_kernel<D><<<grid, kThreads, floats * 4, st>>>(dout, q, k, v, lse2, delta, counts, offsets, inverse, kv_sizes,
                                                                dk, dv, Lq, Lkv, be, topk, scale);
  return check_launch("sparse_dkdv_f32_kernel");
}

}  // namespace

bool sparse_f32_eligible(int D, int be, int dtype, int64_t BH, std::initializer_list<const void*> operands) {
  if (dtype != VSA_F32 || (D != 64 && D != 128) || (be != 64 && be != 128 && be != 256) || BH > 65535) return false;
  for (const void* p : operands)
    if (reinterpret_cast<uintptr_t>(p) % 16) return false;       // 16-byte accesses
  return true;
}

int sparse_fwd_f32(const void* q, const void* k, const void* v, const int32_t* selected, const int32_t* kv_sizes, void* out,
                   float* lse2, int64_t BH, int64_t Lq, int64_t Lkv, int D, int be, int topk, float scale, cudaStream_t st) {
  if (BH == 0 || Lq == 0) return VSA_OK;
  const dim3 grid((unsigned)(Lq / kT), (unsigned)BH);
  auto run = D == 64 ? fwd<64> : fwd<128>;
  return run((const float*)q, (const float*)k, (const float*)v, selected, kv_sizes, (float*)out, lse2, grid, Lq, Lkv, be, topk,
             scale, st);
}

int sparse_dq_f32(const void* dout, const void* q, const void* k, const void* v, const void* out_s, const float* lse2,
                  const int32_t* selected, const int32_t* kv_sizes, float* delta, void* dq, int64_t BH, int64_t Lq, int64_t Lkv,
                  int D, int be, int topk, float scale, cudaStream_t st) {
  if (BH == 0 || Lq == 0) return VSA_OK;
  const dim3 grid((unsigned)(Lq / kT), (unsigned)BH);
  auto run = D == 64 ? dq_pass<64> : dq_pass<128>;
  return run((const float*)dout, (const float*)q, (const float*)k, (const float*)v, (const float*)out_s, lse2, selected, kv_sizes,
             delta, (float*)dq, grid, Lq, Lkv, be, topk, scale, st);
}

int sparse_dkdv_f32(const void* dout, const void* q, const void* k, const void* v, const float* lse2, const float* delta,
                    const int32_t* counts, const int32_t* offsets, const int32_t* inverse, const int32_t* kv_sizes, void* dk,
                    void* dv, int64_t BH, int64_t Lq, int64_t Lkv, int D, int be, int topk, float scale, cudaStream_t st) {
  if (BH == 0 || Lkv == 0) return VSA_OK;
  const dim3 grid((unsigned)(Lkv / kT), (unsigned)BH);
  auto run = D == 64 ? dkdv_pass<64> : dkdv_pass<128>;
  return run((const float*)dout, (const float*)q, (const float*)k, (const float*)v, lse2, delta, counts, offsets, inverse, kv_sizes,
             (float*)dk, (float*)dv, grid, Lq, Lkv, be, topk, scale, st);
}

}  // namespace vsa
