// Fine attention for block volumes that are multiples of 128 tokens (128 and 256), forward and backward, on the
// Blackwell tensor path.  Included by sparse_umma_typed.inl, once per 16-bit element type.
//
// 128 consecutive tokens of a block share one route, so the CTA owns 128 rows and they are the M dimension themselves: half the
// streamed bytes of 64-row tiles per score, 64 cycles of tensor work per M128 x N128 x K16, nothing to add in the epilogue.  The
// resident tile (Q; Q and dO; K and V) is the A operand, the streamed tile the B operand, and P / dS never touch shared memory --
// the thread that owns a row (a TMEM lane) packs them over the fp32 scores it has just read, and the second product takes them
// from tensor memory as its A operand:
//   forward  S[128 q x 128 k]  = Q K^T                             O[128 q x D]  += P V
//   dQ       S = Q K^T,  dP = dO V^T  (128 q x 128 k)              dQ[128 q x D] += dS K
//   dK/dV    S^T = K Q^T, dP^T = V dO^T  (128 k x 64 q)            dV[128 k x D] += P^T dO,  dK += dS^T Q
// Shared-memory bytes per 128 x 128 scores at D = 128 (128 B/clk): forward 160 KB, dQ 224, dK/dV 320; tensor work 1024 / 1536 / 2560
// cycles; exponentials 1024 cycles (16 per clock and SM) in every pass.
//
// Measured, ms for forward / dQ / dK/dV: with transposed 64-token tiles (mma.sync at D = 64) -> these kernels -> whole-warp waits
// and MMAs under elect.sync:
//   [1, 8, 92160, 128], blocks of 128, topk 90:   5.77 / 8.11 / 9.69  -> 3.55 / 5.80 / 7.13 -> 3.37 / 5.20 / 6.92
//   [1, 12, 16384, 128], blocks of 128, topk 16:                         0.277 / 0.387 / 0.381 -> 0.259 / 0.287 / 0.351
// What bounds them: the chain product -> elementwise -> product of a tile, of which three (forward) and two (backward) are in
// flight; at 92k tokens the backward is within 10 % of what a long cuBLAS GEMM sustains under the board's power limit.
//
// The softmax shift of the forward is the row maximum over the first live key tile, as in the 64-row kernels (a row
// is one thread here, so it needs no exchange between lanes); rows that leave the finite range are marked the same
// way, 64 rows at a time, for the exact kernel.
constexpr int kWRows = 128;                       // rows of a wide tile
constexpr int kWHalf = kWRows * 128;              // 64 head dims of a wide tile: 128 rows x 128 bytes
constexpr int kWMaxTiles = kMaxTiles / 2;         // live 128-token key tiles per query tile

int make_wide_map(CUtensorMap* map, const void* ptr, int64_t rows, int dim, int box_rows, const char* what) {
  return make_map_of(map, kTmaElem, ptr, rows, what, dim, box_rows);
}

// D[128 x N] = A[128 x HD] B[N x HD]^T, both K-major; halves of 64 head dims A_HALF / B_HALF bytes apart.
template <int HD, int N, int B_HALF>
__device__ __forceinline__ void wide_issue_scores(uint32_t d_tmem, uint32_t a_tile, uint32_t b_tile) {
  constexpr uint32_t idesc = instr_desc(128, N, 0, 0, kInFmt);
  constexpr uint32_t hi = desc_hi(1024);
  const uint32_t a0 = desc_lo(a_tile, 16), b0 = desc_lo(b_tile, 16);
#pragma unroll
  for (int ks = 0; ks < HD / 16; ++ks)
    mma_ss(d_tmem, desc_pack(a0 + (uint32_t)(((ks >> 2) * kWHalf + (ks & 3) * 32) >> 4), hi),
           desc_pack(b0 + (uint32_t)(((ks >> 2) * B_HALF + (ks & 3) * 32) >> 4), hi), idesc, ks > 0 ? 1u : 0u);
}
// D[128 x HD] (+)= A[128 x ROWS] (tensor memory, 16-bit) B[ROWS x HD] (dims contiguous).  The A columns were written by
// column groups of GROUP scores each, every group packing its half-width result at the start of its own columns.
template <int HD, int ROWS, int GROUP, int TILE = ROWS>
__device__ __forceinline__ void wide_issue_product(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_tile, bool accumulate) {
  constexpr uint32_t idesc = instr_desc(128, HD, 0, 1, kInFmt);
  constexpr uint32_t hi = desc_hi(1024);
  const uint32_t b0 = desc_lo(b_tile, TILE * 128);
  const uint32_t acc0 = accumulate ? 1u : 0u;
#pragma unroll
  for (int ks = 0; ks < ROWS / 16; ++ks)
    mma_ts(d_tmem, a_tmem + (uint32_t)((ks * 16 / GROUP) * GROUP + (ks * 16 % GROUP) / 2), desc_pack(b0 + (uint32_t)(ks * 128), hi),
           idesc, ks > 0 ? 1u : acc0);
}
// Eight fp32 values (as register words) rounded to the element type, 16 bytes.
__device__ __forceinline__ uint4 wide_pack8(const uint32_t* r) {
  return make_uint4(Elem<elem_t>::pack(__uint_as_float(r[0]), __uint_as_float(r[1])), Elem<elem_t>::pack(__uint_as_float(r[2]), __uint_as_float(r[3])),
                    Elem<elem_t>::pack(__uint_as_float(r[4]), __uint_as_float(r[5])), Elem<elem_t>::pack(__uint_as_float(r[6]), __uint_as_float(r[7])));
}
// N accumulator columns plus N values that every row receives.
template <int N>
__device__ __forceinline__ void wide_add_mean(uint32_t (&acc)[N], const float* mean) {
#pragma unroll
  for (int i = 0; i < N / 4; ++i) {
    const float4 m = reinterpret_cast<const float4*>(mean)[i];
    acc[4 * i] = __float_as_uint(__uint_as_float(acc[4 * i]) + m.x);
    acc[4 * i + 1] = __float_as_uint(__uint_as_float(acc[4 * i + 1]) + m.y);
    acc[4 * i + 2] = __float_as_uint(__uint_as_float(acc[4 * i + 2]) + m.z);
    acc[4 * i + 3] = __float_as_uint(__uint_as_float(acc[4 * i + 3]) + m.w);
  }
}
// HD/64 boxes of `rows` x 128 bytes, all on one barrier (the caller has announced the bytes).
template <int HD>
__device__ __forceinline__ void wide_load(uint32_t dst, const CUtensorMap* map, int row, uint32_t half_bytes, uint32_t bar) {
#pragma unroll
  for (int h = 0; h < HD / 64; ++h) tma_load_2d(dst + h * half_bytes, map, h * 64, row, bar);
}

// Live key tiles of a query block in routing order: (row of the tile in the K/V tensors) / 128 << 8 | live tokens.
// Called by the whole CTA; ends with a barrier.  Ids outside the key table and empty tiles are dropped.
__device__ __forceinline__ void wide_tile_list(uint32_t* list, volatile uint32_t* n_live_out, const int32_t* sel,
                                               const int32_t* kv_sizes, int topk, int sub, int Kb, long long bh,
                                               long long BH, long long kv_shard, int tid, int threads) {
  const int n_iter = topk * sub;
  for (int it = tid; it < n_iter; it += threads) {
    const int slot = it / sub, part = it - slot * sub;
    const int kvb = sel[slot];
    int left = (unsigned)kvb < (unsigned)Kb ? kv_sizes[kvb] - part * kWRows : 0;
    left = left > kWRows ? kWRows : left;
    list[it] = left > 0 ? (uint32_t)(kv_tensor_row(bh, BH, ((long long)kvb * sub + part) * kWRows, kv_shard) >> 7) << 8 | (uint32_t)left : 0u;
  }
  __syncthreads();
  if (tid < 32) {
    int n_live = 0;
    for (int it0 = 0; it0 < n_iter; it0 += 32) {
      const uint32_t e = it0 + tid < n_iter ? list[it0 + tid] : 0u;
      const unsigned live = __ballot_sync(0xffffffffu, e != 0u);
      __syncwarp();
      if (e != 0u) list[n_live + __popc(live & ((1u << tid) - 1u))] = e;
      n_live += __popc(live);
      __syncwarp();
    }
    if (tid == 0) *n_live_out = (uint32_t)n_live;
  }
  __syncthreads();
}

// ------------------------------------------------------------------------------------------------------
// forward
// ------------------------------------------------------------------------------------------------------
// Softmax groups of four warps; group g works on tiles g, g+3, ... in its own accumulator.  Three: with two, 3.96 -> 4.36 ms
// on the 92k shape above.
constexpr int kWfGroups = 3;
constexpr int kWfEwThreads = 128 * kWfGroups;
constexpr int kWfThreads = 128 + kWfEwThreads;
template <int HD>
struct WfSmem {
  static constexpr uint32_t tile = HD * 256;                      // 128 rows
  static constexpr int stages = 3;                                // of K and of V
  static constexpr uint32_t q = 0;
  static constexpr uint32_t k = q + tile;
  static constexpr uint32_t v = k + stages * tile;
  static constexpr uint32_t list = v + stages * tile;             // uint32 [kWMaxTiles]
  static constexpr uint32_t m_row = list + 4 * kWMaxTiles;        // float [128]
  static constexpr uint32_t bars = m_row + 512;
  static constexpr uint32_t misc = bars + 32 * 8;
  static constexpr uint32_t total = misc + 32;
};
static_assert(WfSmem<128>::total <= 232448, "shared memory of the wide forward");
enum WfBar { WF_Q_FULL = 0, WF_K_FULL = 1, WF_K_EMPTY = 4, WF_V_FULL = 7, WF_V_EMPTY = 10, WF_S_FULL = 13, WF_S_EMPTY = 16,
             WF_P_FULL = 19, WF_P2_FULL = 22, WF_M_FULL = 25, WF_O_FULL = 26 };

template <int HD>
__global__ void __launch_bounds__(kWfThreads, 1)
sparse_fwd_wide_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                       const __grid_constant__ CUtensorMap map_v, const int32_t* __restrict__ selected,
                       const int32_t* __restrict__ kv_sizes, elem_t* __restrict__ out, float* __restrict__ lse2,
                       const elem_t* __restrict__ out_c, const elem_t* __restrict__ gate, elem_t* __restrict__ out_comb,
                       long long Lq, long long Lkv, long long kv_shard, int be, int topk, float scale, RasterMap comb_map) {
  using Sm = WfSmem<HD>;
  extern __shared__ __align__(1024) uint8_t wide_smem[];
  if (*(volatile int*)&g_device_status != 0) return;
  uint8_t* sm = wide_smem;
  const uint32_t base = smem_u32(sm);
  if (base & 1023u) {                              // the operand layouts need it; the whole 227 KB leave no room to round up
    if (threadIdx.x == 0) report_timeout(49);
    return;
  }
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int qtile = blockIdx.x;
  const long long bh = blockIdx.y;
  const int sub = be / kWRows, Qb = (int)(Lq / be);
  const int qb = qtile / sub;
  const long long row0 = bh * Lq + (long long)qtile * kWRows;
  const float c = scale * kLog2e;
  uint32_t* list = reinterpret_cast<uint32_t*>(sm + Sm::list);
  float* m_row = reinterpret_cast<float*>(sm + Sm::m_row);
  volatile uint32_t* misc = reinterpret_cast<volatile uint32_t*>(sm + Sm::misc);   // tmem base, live tiles, redo flags
  auto bar = [&](int i) -> uint32_t { return base + Sm::bars + 8u * i; };

  if (tid == 0) {
    mbar_init(bar(WF_Q_FULL), 1);
    for (int i = 0; i < 3; ++i) {
      mbar_init(bar(WF_K_FULL + i), 1);
      mbar_init(bar(WF_K_EMPTY + i), 1);
      mbar_init(bar(WF_V_FULL + i), 1);
      mbar_init(bar(WF_V_EMPTY + i), 1);
      mbar_init(bar(WF_S_FULL + i), 1);
      mbar_init(bar(WF_S_EMPTY + i), 1);
      mbar_init(bar(WF_P_FULL + i), 4);        // the first and the second 64 keys of a tile
      mbar_init(bar(WF_P2_FULL + i), 4);
    }
    mbar_init(bar(WF_M_FULL), 4);
    mbar_init(bar(WF_O_FULL), 1);
    misc[2] = 0u;
    misc[3] = 0u;
    fence_barrier_init();
    tma_prefetch_desc(&map_k);
    tma_prefetch_desc(&map_v);
    mbar_arrive_expect_tx(bar(WF_Q_FULL), Sm::tile);
    wide_load<HD>(base + Sm::q, &map_q, (int)row0, kWHalf, bar(WF_Q_FULL));
  }
  if (warp == 1) {
    tmem_alloc(base + Sm::misc, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  wide_tile_list(list, misc + 1, selected + (bh * Qb + qb) * (long long)topk, kv_sizes, topk, sub, (int)(Lkv / be), bh,
                 gridDim.y, kv_shard, tid, kWfThreads);
  tc_fence_after();
  const uint32_t tmem = misc[0];
  const int n_tiles = (int)misc[1];
  const uint32_t tmem_o = tmem + 128 * kWfGroups;
  bool ok = true;

  if (warp >= 4) {          // 3 x 152 + 56 registers are the four groups' 128 at launch
    registers_inc<152>();
    // softmax: a thread owns query row `row`; group g takes every third key tile, in its own accumulator
    const int quarter = warp & 3, g = (warp - 4) >> 2;
    const int row = quarter * 32 + lane, st = tid - 128;
    const uint32_t s_addr = tmem + 128 * g + ((uint32_t)(quarter * 32) << 16);
    float2 lsum = make_float2(0.f, 0.f);
    float neg_m = 0.f;
    for (int p = g; p < n_tiles && ok; p += kWfGroups) {
      const uint32_t ph = (p / kWfGroups) & 1;
      const int valid = (int)(list[p] & 255u);
      ok = VSA_WARP_WAIT(bar(WF_S_FULL + g), ph);
      if (!ok) break;
      tc_fence_after();
      if (p == 0) {          // the row's shift: maximum over the first live key tile
        float m = -INFINITY;
#pragma unroll 1
        for (int j = 0; j < 4; ++j) {
          uint32_t sv[32];
          tmem_ld(s_addr + 32 * j, sv);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) m = fmaxf(m, 32 * j + i < valid ? __uint_as_float(sv[i]) * c : -INFINITY);
        }
        // Head dim 64 keeps fp16's precision at the bottom: the online softmax of the mma.sync kernels, which it shares its
        // shapes with, has its largest P at 1, and P below 2^-14 lose bits.  With four binades less under the maximum the
        // error against float64 rose 6 % where one key outweighs 8000 others by 10 nats (2.62e-4 -> 2.77e-4), and doubled at
        // 12.  Scores 16 binades above the first tile's maximum go to the exact kernel (20 with the bias).
        if (HD != 64) m += kShiftBias;
        m_row[row] = m;
        neg_m = -m;
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(WF_M_FULL));
      } else if (p == g) {
        ok = VSA_WARP_WAIT(bar(WF_M_FULL), 0);
        if (!ok) break;
        neg_m = -m_row[row];
      }
      if (valid < kWRows) {  // padding rows of V meet P = 0 in the product: they must be finite (0 * NaN)
        const int s = p % Sm::stages;
        ok = VSA_WARP_WAIT(bar(WF_V_FULL + s), (p / Sm::stages) & 1);
        if (!ok) break;
        if (row >= valid) {
          uint8_t* vrow = sm + Sm::v + s * Sm::tile + row * 128;
#pragma unroll
          for (int ch = 0; ch < HD / 8; ++ch)
            *reinterpret_cast<uint4*>(vrow + (ch >> 3) * kWHalf + ((ch ^ row) & 7) * 16) = make_uint4(0, 0, 0, 0);   // all banks
        }
        fence_proxy_async_smem();
      }
      const float2 c2 = make_float2(c, c), m2 = make_float2(neg_m, neg_m);
      // P is handed over in two halves, so that its product starts under the second: 3.82 -> 3.55 ms and 1.04 -> 0.99 ms on the
      // first two shapes above.
      // P over scores that this thread has already read.  Full and ragged tiles are separate code: with one body the
      // compiler turned the mask into two more instructions per score for every tile.
      auto exponentiate = [&](auto ragged) {
        uint32_t sv[2][32], pk[16];
        tmem_ld(s_addr, sv[0]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          tmem_ld_wait();
          if (j < 3) tmem_ld(s_addr + 32 * (j + 1), sv[(j + 1) & 1]);
          const uint32_t* x32 = sv[j & 1];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float2 x = fma2(word_pair(x32 + 2 * i), c2, m2);
            float2 e = make_float2(fast_exp2(x.x), fast_exp2(x.y));
            if (decltype(ragged)::value) {     // scores of padding keys come from whatever sits in K there: select
              if (32 * j + 2 * i >= valid) e.x = 0.f;
              if (32 * j + 2 * i + 1 >= valid) e.y = 0.f;
            }
            lsum = add2(lsum, e);
            pk[i] = Elem<elem_t>::pack(e.x, e.y);
          }
          tmem_st(s_addr + 16 * j, pk);
          if (j & 1) {
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar((j == 1 ? WF_P_FULL : WF_P2_FULL) + g));
          }
        }
      };
      if (valid == kWRows) exponentiate(std::false_type{});
      else exponentiate(std::true_type{});
    }
    if (!ok && lane == 0) report_timeout(43);

    // Every MMA is done and all of shared memory is free; with no live tile nobody else has waited for the load of Q, over
    // which the rows are staged below.
    if (ok) ok = VSA_WARP_WAIT(bar(n_tiles > 0 ? WF_O_FULL : WF_Q_FULL), 0);
    if (!ok && lane == 0) report_timeout(44);
    tc_fence_after();
    float* l_part = reinterpret_cast<float*>(sm + Sm::k);              // [groups][128]
    l_part[g * kWRows + row] = lsum.x + lsum.y;
    named_barrier(1, kWfEwThreads);
    float l = l_part[row];
#pragma unroll
    for (int i = 1; i < kWfGroups; ++i) l += l_part[i * kWRows + row];
    bool finite = l <= 3.0e38f;
    uint8_t* stage = sm + Sm::q;                                       // [128 rows][HD], 16-byte chunks xor row
    for (int j = g; j < HD / 32; j += kWfGroups) {
      uint32_t ov[32];
      if (ok && n_tiles > 0) {
        tmem_ld(tmem_o + ((uint32_t)(quarter * 32) << 16) + 32 * j, ov);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const float o = __uint_as_float(ov[i]) / l;
          finite = finite && fabsf(o) <= 3.0e38f;
          ov[i] = __float_as_uint(o);
        }
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) ov[i] = n_tiles == 0 ? 0x7fc00000u : 0u;
      }
#pragma unroll
      for (int q4 = 0; q4 < 4; ++q4)
        *reinterpret_cast<uint4*>(stage + row * (HD * 2) + (((4 * j + q4) ^ (row & 7)) << 4)) = wide_pack8(ov + 8 * q4);
    }
    if (!finite) misc[2 + (row >> 6)] = 1u;
    named_barrier(1, kWfEwThreads);
    for (int i = st; i < kWRows * HD / 8; i += kWfEwThreads) {
      const int r = i / (HD / 8), ch = i % (HD / 8);
      const uint4 sv = *reinterpret_cast<const uint4*>(stage + r * (HD * 2) + ((ch ^ (r & 7)) << 4));
      *reinterpret_cast<uint4*>(out + (row0 + r) * HD + ch * 8) = sv;
      if (out_comb != nullptr) {   // gated combine with the pooled branch on the way out
        const long long crow = comb_map.map == nullptr ? row0 + r : raster_row(comb_map, bh, (long long)qtile * kWRows + r);
        if (crow >= 0) {
          const uint4 cv = *reinterpret_cast<const uint4*>(out_c + (bh * Qb + qb) * (long long)HD + ch * 8);
          uint4 gv = make_uint4(0, 0, 0, 0);
          if (gate != nullptr) gv = *reinterpret_cast<const uint4*>(gate + crow * HD + ch * 8);
          *reinterpret_cast<uint4*>(out_comb + crow * HD + ch * 8) = combine_x8<elem_t>(sv, cv, gv, gate != nullptr);
        }
      }
    }
    if (g == 0) {
      const bool redo = (misc[2 + (row >> 6)] != 0u) && ok;
      lse2[row0 + row] = (redo || n_tiles == 0) ? NAN : m_row[row] + log2f(l);
    }
  } else {
    registers_dec<56>();
    if (warp == 0 || warp == 1) {
      const bool is_k = warp == 0;
      const CUtensorMap* map = is_k ? &map_k : &map_v;
      const int full0 = is_k ? WF_K_FULL : WF_V_FULL, empty0 = is_k ? WF_K_EMPTY : WF_V_EMPTY;
      const uint32_t ring = base + (is_k ? Sm::k : Sm::v);
      for (int p = 0; p < n_tiles; ++p) {
        const int s = p % Sm::stages;
        const int row = (int)(list[p] >> 8) << 7;
        ok = VSA_WARP_WAIT(bar(empty0 + s), ((p / Sm::stages) & 1) ^ 1);
        if (!ok) break;
        if (elect_one()) {
          mbar_arrive_expect_tx(bar(full0 + s), Sm::tile);
          wide_load<HD>(ring + s * Sm::tile, map, row, kWHalf, bar(full0 + s));
        }
        __syncwarp();
      }
      if (!ok && lane == 0) report_timeout(41);
    } else if (warp == 2) {
      // S = Q K^T
      ok = VSA_WARP_WAIT(bar(WF_Q_FULL), 0);
      for (int p = 0; p < n_tiles && ok; ++p) {
        const int s = p % Sm::stages, b = p % kWfGroups;
        ok = VSA_WARP_WAIT(bar(WF_K_FULL + s), (p / Sm::stages) & 1) && VSA_WARP_WAIT(bar(WF_S_EMPTY + b), ((p / kWfGroups) & 1) ^ 1);
        if (!ok) break;
        tc_fence_after();
        if (elect_one()) {
          wide_issue_scores<HD, 128, kWHalf>(tmem + b * 128, base + Sm::q, base + Sm::k + s * Sm::tile);
          mma_commit(bar(WF_K_EMPTY + s));
          mma_commit(bar(WF_S_FULL + b));
        }
        __syncwarp();
      }
      if (!ok && lane == 0) report_timeout(42);
    } else if (warp == 3) {
      // O += P V
      for (int p = 0; p < n_tiles && ok; ++p) {
        const int s = p % Sm::stages, b = p % kWfGroups;
        ok = VSA_WARP_WAIT(bar(WF_V_FULL + s), (p / Sm::stages) & 1) && VSA_WARP_WAIT(bar(WF_P_FULL + b), (p / kWfGroups) & 1);
        if (!ok) break;
        tc_fence_after();
        if (elect_one()) {
          wide_issue_product<HD, 64, 128, 128>(tmem_o, tmem + b * 128, base + Sm::v + s * Sm::tile, p > 0);
        }
        __syncwarp();
        ok = VSA_WARP_WAIT(bar(WF_P2_FULL + b), (p / kWfGroups) & 1);
        if (!ok) break;
        tc_fence_after();
        if (elect_one()) {
          wide_issue_product<HD, 64, 128, 128>(tmem_o, tmem + b * 128 + 32, base + Sm::v + s * Sm::tile + 64 * 128, true);
          mma_commit(bar(WF_V_EMPTY + s));
          mma_commit(bar(WF_S_EMPTY + b));
        }
        __syncwarp();
      }
      if (ok && elect_one()) mma_commit(bar(WF_O_FULL));
      __syncwarp();
      if (!ok && lane == 0) report_timeout(45);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, kTmemCols);
}

// ------------------------------------------------------------------------------------------------------
// dQ
// ------------------------------------------------------------------------------------------------------
// Score columns of a thread.  All sixteen warps share a tile: two sets of eight on alternate tiles with 64 columns a thread
// took 6.2 ms instead of 5.6 on the 92k shape above (spills, and dP has one accumulator for both).
constexpr int kWqCols = 32;
constexpr int kWqGroups = kWRows / kWqCols;
constexpr int kWqEwThreads = 128 * kWqGroups;
constexpr int kWqThreads = 128 + kWqEwThreads;
template <int HD>
struct WqSmem {
  static constexpr uint32_t tile = HD * 256;
  static constexpr int k_stages = 3, v_stages = 2;
  static constexpr uint32_t q = 0;
  static constexpr uint32_t d_o = q + tile;
  static constexpr uint32_t k = d_o + tile;
  static constexpr uint32_t v = k + k_stages * tile;
  static constexpr uint32_t list = v + v_stages * tile;
  static constexpr uint32_t delta = list + 4 * kWMaxTiles;        // float [128]
  static constexpr uint32_t bars = delta + 512;
  static constexpr uint32_t misc = bars + 32 * 8;
  static constexpr uint32_t total = misc + 32;
};
static_assert(WqSmem<128>::total <= 232448, "shared memory of the wide dQ pass");
enum WqBar { WQ_QDO_FULL = 0, WQ_K_FULL = 1, WQ_K_EMPTY = 4, WQ_V_FULL = 7, WQ_V_EMPTY = 9, WQ_S_FULL = 11, WQ_S_EMPTY = 13,
             WQ_DP_FULL = 15, WQ_DP_EMPTY = 16, WQ_DS_FULL = 17, WQ_ACC_FULL = 19 };

template <int HD>
__global__ void __launch_bounds__(kWqThreads, 1)
sparse_dq_wide_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_do,
                      const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                      const elem_t* __restrict__ dout, const elem_t* __restrict__ out_s, const float* __restrict__ lse2,
                      const int32_t* __restrict__ selected, const int32_t* __restrict__ kv_sizes,
                      float* __restrict__ delta, elem_t* __restrict__ dq, const elem_t* __restrict__ mean_grad,
                      const int32_t* __restrict__ q_sizes, long long Lq, long long Lkv, long long kv_shard, int be, int topk,
                      float scale, RasterMap out_map) {
  using Sm = WqSmem<HD>;
  extern __shared__ __align__(1024) uint8_t wide_smem[];
  if (*(volatile int*)&g_device_status != 0) return;
  uint8_t* sm = wide_smem;
  const uint32_t base = smem_u32(sm);
  if (base & 1023u) {
    if (threadIdx.x == 0) report_timeout(59);
    return;
  }
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int qtile = blockIdx.x;
  const long long bh = blockIdx.y;
  const int sub = be / kWRows, Qb = (int)(Lq / be);
  const int qb = qtile / sub;
  const long long row0 = bh * Lq + (long long)qtile * kWRows;
  const float c = scale * kLog2e;
  uint32_t* list = reinterpret_cast<uint32_t*>(sm + Sm::list);
  volatile uint32_t* misc = reinterpret_cast<volatile uint32_t*>(sm + Sm::misc);
  auto bar = [&](int i) -> uint32_t { return base + Sm::bars + 8u * i; };
  const bool elementwise = warp >= 4;
  const int quarter = warp & 3, cg = (warp - 4) >> 2, row = quarter * 32 + lane;

  if (tid == 0) {
    mbar_init(bar(WQ_QDO_FULL), 1);
    for (int i = 0; i < Sm::k_stages; ++i) {
      mbar_init(bar(WQ_K_FULL + i), 1);
      mbar_init(bar(WQ_K_EMPTY + i), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar(WQ_V_FULL + i), 1);
      mbar_init(bar(WQ_V_EMPTY + i), 1);
      mbar_init(bar(WQ_S_FULL + i), 1);
      mbar_init(bar(WQ_S_EMPTY + i), 1);
      mbar_init(bar(WQ_DS_FULL + i), 4 * kWqGroups);
    }
    mbar_init(bar(WQ_DP_FULL), 1);
    mbar_init(bar(WQ_DP_EMPTY), 4 * kWqGroups);
    mbar_init(bar(WQ_ACC_FULL), 1);
    fence_barrier_init();
    tma_prefetch_desc(&map_k);
    tma_prefetch_desc(&map_v);
    mbar_arrive_expect_tx(bar(WQ_QDO_FULL), 2 * Sm::tile);
    wide_load<HD>(base + Sm::q, &map_q, (int)row0, kWHalf, bar(WQ_QDO_FULL));
    wide_load<HD>(base + Sm::d_o, &map_do, (int)row0, kWHalf, bar(WQ_QDO_FULL));
  }
  // delta = rowsum(out_s * dout): kWqGroups neighbouring threads per row
  float* s_delta = reinterpret_cast<float*>(sm + Sm::delta);
  if (elementwise) {
    const int st = tid - 128, r = st / kWqGroups, part = st % kWqGroups;
    constexpr int kDims = HD / kWqGroups;
    const uint4* po = reinterpret_cast<const uint4*>(out_s + (row0 + r) * HD + part * kDims);
    const uint4* pd = reinterpret_cast<const uint4*>(dout + (row0 + r) * HD + part * kDims);
    float acc = 0.f;
#pragma unroll
    for (int i = 0; i < kDims / 8; ++i) {
      const uint4 a = po[i], b = pd[i];
      const elem_t* ea = reinterpret_cast<const elem_t*>(&a);
      const elem_t* eb = reinterpret_cast<const elem_t*>(&b);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc = fmaf(Elem<elem_t>::to(ea[j]), Elem<elem_t>::to(eb[j]), acc);
    }
#pragma unroll
    for (int o = 1; o < kWqGroups; o <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (part == 0) {
      s_delta[r] = acc;
      delta[row0 + r] = acc;
    }
  }
  if (warp == 1) {
    tmem_alloc(base + Sm::misc, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  const float dl = elementwise ? s_delta[row] : 0.f;
  const float neg_lse = elementwise ? log2f(fabsf(scale)) - lse2[row0 + row] : 0.f;   // 2^(s c - lse) * |scale| in one exponential
  wide_tile_list(list, misc + 1, selected + (bh * Qb + qb) * (long long)topk, kv_sizes, topk, sub, (int)(Lkv / be), bh,
                 gridDim.y, kv_shard, tid, kWqThreads);
  tc_fence_after();
  const uint32_t tmem = misc[0];
  const int n_tiles = (int)misc[1];
  // S (later dS) in two accumulators, dP in one that is free again as soon as it has been read, dQ behind them
  const uint32_t tmem_dp = tmem + 256, tmem_acc = tmem + 384;
  bool ok = true;

  if (warp == 0) {
    for (int p = 0; p < n_tiles; ++p) {
      const int sk = p % Sm::k_stages, sv = p % Sm::v_stages;
      const int krow = (int)(list[p] >> 8) << 7;
      ok = VSA_WARP_WAIT(bar(WQ_K_EMPTY + sk), ((p / Sm::k_stages) & 1) ^ 1);
      if (!ok) break;
      if (elect_one()) {
        mbar_arrive_expect_tx(bar(WQ_K_FULL + sk), Sm::tile);
        wide_load<HD>(base + Sm::k + sk * Sm::tile, &map_k, krow, kWHalf, bar(WQ_K_FULL + sk));
      }
      __syncwarp();
      ok = VSA_WARP_WAIT(bar(WQ_V_EMPTY + sv), ((p / Sm::v_stages) & 1) ^ 1);
      if (!ok) break;
      if (elect_one()) {
        mbar_arrive_expect_tx(bar(WQ_V_FULL + sv), Sm::tile);
        wide_load<HD>(base + Sm::v + sv * Sm::tile, &map_v, krow, kWHalf, bar(WQ_V_FULL + sv));
      }
      __syncwarp();
    }
    if (!ok && lane == 0) report_timeout(51);
  } else if (warp == 2) {
    // S = Q K^T
    ok = VSA_WARP_WAIT(bar(WQ_QDO_FULL), 0);
    for (int p = 0; p < n_tiles && ok; ++p) {
      const int s = p % Sm::k_stages, b = p & 1;
      ok = VSA_WARP_WAIT(bar(WQ_K_FULL + s), (p / Sm::k_stages) & 1) && VSA_WARP_WAIT(bar(WQ_S_EMPTY + b), ((p >> 1) & 1) ^ 1);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
        wide_issue_scores<HD, 128, kWHalf>(tmem + b * 128, base + Sm::q, base + Sm::k + s * Sm::tile);
        mma_commit(bar(WQ_S_FULL + b));
      }
      __syncwarp();
    }
    if (!ok && lane == 0) report_timeout(52);
  } else if (warp == 1) {
    // dP = dO V^T
    ok = VSA_WARP_WAIT(bar(WQ_QDO_FULL), 0);
    for (int p = 0; p < n_tiles && ok; ++p) {
      const int s = p % Sm::v_stages;
      ok = VSA_WARP_WAIT(bar(WQ_V_FULL + s), (p / Sm::v_stages) & 1) && VSA_WARP_WAIT(bar(WQ_DP_EMPTY), (p & 1) ^ 1);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
        wide_issue_scores<HD, 128, kWHalf>(tmem_dp, base + Sm::d_o, base + Sm::v + s * Sm::tile);
        mma_commit(bar(WQ_V_EMPTY + s));
        mma_commit(bar(WQ_DP_FULL));
      }
      __syncwarp();
    }
    if (!ok && lane == 0) report_timeout(56);
  } else if (warp == 3) {
    // dQ += dS K
    for (int p = 0; p < n_tiles && ok; ++p) {
      const int s = p % Sm::k_stages, b = p & 1;
      ok = VSA_WARP_WAIT(bar(WQ_K_FULL + s), (p / Sm::k_stages) & 1) && VSA_WARP_WAIT(bar(WQ_DS_FULL + b), (p >> 1) & 1);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
        wide_issue_product<HD, 128, kWqCols>(tmem_acc, tmem + b * 128, base + Sm::k + s * Sm::tile, p > 0);
        mma_commit(bar(WQ_K_EMPTY + s));
        mma_commit(bar(WQ_S_EMPTY + b));
      }
      __syncwarp();
    }
    if (ok && elect_one()) mma_commit(bar(WQ_ACC_FULL));
    __syncwarp();
    if (!ok && lane == 0) report_timeout(53);
  } else {
    const int c0 = cg * kWqCols, st = tid - 128;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const float2 c2 = make_float2(c, c), l2 = make_float2(neg_lse, neg_lse), d2 = make_float2(-dl, -dl);
    for (int p = 0; p < n_tiles && ok; ++p) {
      const int b = p & 1;
      const int valid = (int)(list[p] & 255u);
      ok = VSA_WARP_WAIT(bar(WQ_S_FULL + b), (p >> 1) & 1);
      if (!ok) break;
      tc_fence_after();
      const uint32_t s_addr = tmem + b * 128 + lane_addr + c0;
      uint32_t sv[kWqCols];
      tmem_ld(s_addr, sv);
      tmem_ld_wait();
      if (valid < kWRows && cg == 0) {   // padding rows of K meet dS = 0 in the product: finite, please (S has completed)
        if (row >= valid) {
          uint8_t* krow = sm + Sm::k + (p % Sm::k_stages) * Sm::tile + row * 128;
#pragma unroll
          for (int ch = 0; ch < HD / 8; ++ch)
            *reinterpret_cast<uint4*>(krow + (ch >> 3) * kWHalf + ((ch ^ row) & 7) * 16) = make_uint4(0, 0, 0, 0);
        }
        fence_proxy_async_smem();
      }
      float2 pf[kWqCols / 2];            // 2^(S c - lse) * |scale|
#pragma unroll
      for (int i = 0; i < kWqCols / 2; ++i) {
        const float2 x = fma2(word_pair(sv + 2 * i), c2, l2);
        pf[i] = make_float2(fast_exp2(x.x), fast_exp2(x.y));
      }
      ok = VSA_WARP_WAIT(bar(WQ_DP_FULL), p & 1);
      if (!ok) break;
      tc_fence_after();
      uint32_t dv[kWqCols];
      tmem_ld(tmem_dp + lane_addr + c0, dv);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(WQ_DP_EMPTY));
      uint32_t pk[kWqCols / 2];
#pragma unroll
      for (int i = 0; i < kWqCols / 2; ++i) {
        const float2 y = mul2(pf[i], add2(word_pair(dv + 2 * i), d2));
        pk[i] = Elem<elem_t>::pack(y.x, y.y);
      }
      if (valid < kWRows) {              // scores of padding keys come from whatever sits in K and V there
#pragma unroll
        for (int i = 0; i < kWqCols / 2; ++i) {
          if (c0 + 2 * i >= valid) pk[i] = 0u;
          else if (c0 + 2 * i + 1 >= valid) pk[i] &= 0xffffu;
        }
      }
      tmem_st(s_addr, pk);               // over this thread's own scores
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(WQ_DS_FULL + b));
    }
    // block-mean backward folded in: query row r of the block also receives dmean[block] / max(size, 1) while r < size
    float mean = 0.f;
    bool mean_row = false;
    if (mean_grad != nullptr) {
      const int size = q_sizes[qb];
      mean_row = row < size - (qtile % sub) * kWRows;
      if (st < HD) mean = Elem<elem_t>::to(mean_grad[(bh * Qb + qb) * (long long)HD + st]) / (float)(size > 1 ? size : 1);
    }
    if (!ok && lane == 0) report_timeout(54);
    // as in the forward: Q, over which dQ is staged, may still be landing when the route has no live tile
    if (ok) ok = VSA_WARP_WAIT(bar(n_tiles > 0 ? WQ_ACC_FULL : WQ_QDO_FULL), 0);
    if (!ok && lane == 0) report_timeout(55);
    tc_fence_after();
    if (st < HD) s_delta[st] = mean;       // every row's delta has long been read
    named_barrier(1, kWqEwThreads);
    uint8_t* stage = sm + Sm::q;
    for (int j = cg; j < HD / 32; j += kWqGroups) {
      uint32_t av[32];
      if (ok && n_tiles > 0) {
        tmem_ld(tmem_acc + lane_addr + 32 * j, av);
        tmem_ld_wait();
        if (scale < 0.f) {
#pragma unroll
          for (int i = 0; i < 32; ++i) av[i] ^= 0x80000000u;
        }
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) av[i] = 0u;
      }
      if (mean_row) wide_add_mean(av, s_delta + 32 * j);
#pragma unroll
      for (int q4 = 0; q4 < 4; ++q4)
        *reinterpret_cast<uint4*>(stage + row * (HD * 2) + (((4 * j + q4) ^ (row & 7)) << 4)) = wide_pack8(av + 8 * q4);
    }
    named_barrier(1, kWqEwThreads);
    for (int i = st; i < kWRows * HD / 8; i += kWqEwThreads) {
      const int r = i / (HD / 8), ch = i % (HD / 8);
      const long long drow = out_map.map == nullptr ? row0 + r : raster_row(out_map, bh, (long long)qtile * kWRows + r);
      if (drow >= 0)
        *reinterpret_cast<uint4*>(dq + drow * HD + ch * 8) = *reinterpret_cast<const uint4*>(stage + r * (HD * 2) + ((ch ^ (r & 7)) << 4));
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, kTmemCols);
}

// ------------------------------------------------------------------------------------------------------
// dK / dV: lanes = 128 key rows, columns = 64 query rows of a streamed tile
// ------------------------------------------------------------------------------------------------------
// 32 columns a thread, eight warps per tile; two sets of eight on alternate tiles measured 7.5 ms instead of 7.2.
constexpr int kWkCols = 32;
constexpr int kWkGroups = kTile / kWkCols;
constexpr int kWkEwThreads = 128 * kWkGroups;
constexpr int kWkThreads = 128 + kWkEwThreads;
template <int HD>
struct WkSmem {
  static constexpr uint32_t tile = HD * 256;          // 128 resident rows
  static constexpr uint32_t part = HD * 128;          // 64 streamed rows
  static constexpr int q_stages = 5, do_stages = 5;
  static constexpr uint32_t k = 0;
  static constexpr uint32_t v = k + tile;
  static constexpr uint32_t q = v + tile;
  static constexpr uint32_t d_o = q + q_stages * part;
  static constexpr uint32_t stats = d_o + do_stages * part;       // per Q stage: lse [64], delta [64]
  static constexpr uint32_t bars = stats + q_stages * 512;
  static constexpr uint32_t misc = bars + 40 * 8;
  static constexpr uint32_t total = misc + 32;
};
static_assert(WkSmem<128>::total <= 232448, "shared memory of the wide dK/dV pass");
enum WkBar { WK_KV_FULL = 0, WK_Q_FULL = 1, WK_Q_EMPTY = 6, WK_DO_FULL = 11, WK_DO_EMPTY = 16, WK_S_FULL = 21, WK_S_EMPTY = 23,
             WK_DP_FULL = 25, WK_DP_EMPTY = 27, WK_P_FULL = 29, WK_DS_FULL = 31, WK_ACC_FULL = 33 };

template <int HD>
__global__ void __launch_bounds__(kWkThreads, 1)
sparse_dkdv_wide_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_do,
                        const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                        const float* __restrict__ lse2, const float* __restrict__ delta,
                        const int32_t* __restrict__ counts, const int32_t* __restrict__ offsets,
                        const int32_t* __restrict__ inverse, const int32_t* __restrict__ kv_sizes,
                        elem_t* __restrict__ dk, elem_t* __restrict__ dv, const elem_t* __restrict__ mean_grad_k,
                        const elem_t* __restrict__ mean_grad_v, long long Lq, long long Lkv, long long kv_shard, int be,
                        int topk, float scale, RasterMap out_map) {
  using Sm = WkSmem<HD>;
  extern __shared__ __align__(1024) uint8_t wide_smem[];
  if (*(volatile int*)&g_device_status != 0) return;
  uint8_t* sm = wide_smem;
  const uint32_t base = smem_u32(sm);
  if (base & 1023u) {
    if (threadIdx.x == 0) report_timeout(69);
    return;
  }
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int ktile = blockIdx.x;
  const long long bh = blockIdx.y;
  const int sub = be / kWRows, qsub = be / kTile;
  const int Kb = (int)(Lkv / be), Qb = (int)(Lq / be);
  const int kvb = ktile / sub;
  const int size = kv_sizes[kvb];
  int valid = size - (ktile % sub) * kWRows;
  valid = valid < 0 ? 0 : (valid > kWRows ? kWRows : valid);
  const long long krow0 = kv_tensor_row(bh, gridDim.y, (long long)ktile * kWRows, kv_shard);
  const int32_t* inv = inverse + bh * (long long)Qb * topk + offsets[bh * Kb + kvb];
  const int n_tiles = valid > 0 ? counts[bh * Kb + kvb] * qsub : 0;
  const float c = scale * kLog2e;
  const long long q_row_base = bh * Lq;
  const float mean_inv = 1.f / (float)(size > 1 ? size : 1);
  const long long mean_off = (bh * Kb + kvb) * (long long)HD;

  if (n_tiles == 0) {   // nobody selected this tile, or it is all padding: pooled gradient only
    for (int i = tid; i < kWRows * HD / 8; i += (int)blockDim.x) {
      const int r = i / (HD / 8), ch = i % (HD / 8);
      const long long drow = out_map.map == nullptr ? krow0 + r : raster_row(out_map, bh, (long long)ktile * kWRows + r);
      if (drow < 0) continue;
      uint4 ok4 = make_uint4(0, 0, 0, 0), ov4 = make_uint4(0, 0, 0, 0);
      if (mean_grad_k != nullptr && r < valid) {
        elem_t* ek = reinterpret_cast<elem_t*>(&ok4);
        elem_t* ev = reinterpret_cast<elem_t*>(&ov4);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          ek[e] = Elem<elem_t>::from(Elem<elem_t>::to(mean_grad_k[mean_off + ch * 8 + e]) * mean_inv);
          ev[e] = Elem<elem_t>::from(Elem<elem_t>::to(mean_grad_v[mean_off + ch * 8 + e]) * mean_inv);
        }
      }
      *reinterpret_cast<uint4*>(dk + drow * HD + ch * 8) = ok4;
      *reinterpret_cast<uint4*>(dv + drow * HD + ch * 8) = ov4;
    }
    return;
  }
  volatile uint32_t* misc = reinterpret_cast<volatile uint32_t*>(sm + Sm::misc);
  auto bar = [&](int i) -> uint32_t { return base + Sm::bars + 8u * i; };
  // tensor row of the i-th 64-row query tile that selected this key block
  auto tile_row = [&](int i) -> long long { return q_row_base + (long long)inv[i / qsub] * be + (i % qsub) * kTile; };

  if (tid == 0) {
    mbar_init(bar(WK_KV_FULL), 1);
    for (int i = 0; i < Sm::q_stages; ++i) {
      mbar_init(bar(WK_Q_FULL + i), 33);       // the TMA boxes' lane and 32 lanes' copies of the statistics
      mbar_init(bar(WK_Q_EMPTY + i), 1);
    }
    for (int i = 0; i < Sm::do_stages; ++i) {
      mbar_init(bar(WK_DO_FULL + i), 1);
      mbar_init(bar(WK_DO_EMPTY + i), 2);      // read by the dP products of one issuer and the dV products of the other
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar(WK_S_FULL + i), 1);
      mbar_init(bar(WK_S_EMPTY + i), 1);
      mbar_init(bar(WK_DP_FULL + i), 1);
      mbar_init(bar(WK_DP_EMPTY + i), 1);
      mbar_init(bar(WK_P_FULL + i), 4 * kWkGroups);
      mbar_init(bar(WK_DS_FULL + i), 4 * kWkGroups);
    }
    mbar_init(bar(WK_ACC_FULL), 1);
    fence_barrier_init();
    tma_prefetch_desc(&map_q);
    tma_prefetch_desc(&map_do);
    mbar_arrive_expect_tx(bar(WK_KV_FULL), 2 * Sm::tile);
    wide_load<HD>(base + Sm::k, &map_k, (int)krow0, kWHalf, bar(WK_KV_FULL));
    wide_load<HD>(base + Sm::v, &map_v, (int)krow0, kWHalf, bar(WK_KV_FULL));
  }
  if (warp == 1) {
    tmem_alloc(base + Sm::misc, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = misc[0];
  // two buffers of (S^T 64 columns, dP^T 64 columns), P^T and dS^T packed over them; then dK and dV
  const uint32_t tmem_dk = tmem + 256, tmem_dv = tmem + 384;
  bool ok = true;

  if (warp == 0) {       // dO tiles; Q tiles and the statistics of their rows
    for (int p = 0; p < n_tiles; ++p) {
      const int sq = p % Sm::q_stages, sd = p % Sm::do_stages;
      const long long row = tile_row(p);
      ok = VSA_WARP_WAIT2(bar(WK_Q_EMPTY + sq), ((p / Sm::q_stages) & 1) ^ 1, bar(WK_DO_EMPTY + sd), ((p / Sm::do_stages) & 1) ^ 1);
      if (!ok) break;
      const uint32_t st = base + Sm::stats + sq * 512 + lane * 4;
      cp_async4(st, lse2 + row + lane);
      cp_async4(st + 128, lse2 + row + 32 + lane);
      cp_async4(st + 256, delta + row + lane);
      cp_async4(st + 384, delta + row + 32 + lane);
      cp_async_arrive_noinc(bar(WK_Q_FULL + sq));
      if (lane == 0) {
        mbar_arrive_expect_tx(bar(WK_Q_FULL + sq), Sm::part);
        wide_load<HD>(base + Sm::q + sq * Sm::part, &map_q, (int)row, kSlab, bar(WK_Q_FULL + sq));
        mbar_arrive_expect_tx(bar(WK_DO_FULL + sd), Sm::part);
        wide_load<HD>(base + Sm::d_o + sd * Sm::part, &map_do, (int)row, kSlab, bar(WK_DO_FULL + sd));
      }
    }
    if (!ok && lane == 0) report_timeout(61);
  } else if (warp == 2) {
    // S^T = K Q^T
    ok = VSA_WARP_WAIT(bar(WK_KV_FULL), 0);
    for (int p = 0; p < n_tiles && ok; ++p) {
      const int s = p % Sm::q_stages, b = p & 1;
      ok = VSA_WARP_WAIT(bar(WK_Q_FULL + s), (p / Sm::q_stages) & 1) && VSA_WARP_WAIT(bar(WK_S_EMPTY + b), ((p >> 1) & 1) ^ 1);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
        wide_issue_scores<HD, 64, kSlab>(tmem + b * 128, base + Sm::k, base + Sm::q + s * Sm::part);
        mma_commit(bar(WK_S_FULL + b));
      }
      __syncwarp();
    }
    if (!ok && lane == 0) report_timeout(62);
  } else if (warp == 1) {
    // dP^T = V dO^T
    ok = VSA_WARP_WAIT(bar(WK_KV_FULL), 0);
    for (int p = 0; p < n_tiles && ok; ++p) {
      const int s = p % Sm::do_stages, b = p & 1;
      ok = VSA_WARP_WAIT(bar(WK_DO_FULL + s), (p / Sm::do_stages) & 1) && VSA_WARP_WAIT(bar(WK_DP_EMPTY + b), ((p >> 1) & 1) ^ 1);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
        wide_issue_scores<HD, 64, kSlab>(tmem + b * 128 + 64, base + Sm::v, base + Sm::d_o + s * Sm::part);
        mma_commit(bar(WK_DO_EMPTY + s));
        mma_commit(bar(WK_DP_FULL + b));
      }
      __syncwarp();
    }
    if (!ok && lane == 0) report_timeout(66);
  } else if (warp == 3) {
    // dV += P^T dO, dK += dS^T Q
    for (int p = 0; p < n_tiles && ok; ++p) {
      const int sq = p % Sm::q_stages, sd = p % Sm::do_stages, b = p & 1;
      const uint32_t ph = (p >> 1) & 1;
      ok = VSA_WARP_WAIT(bar(WK_DO_FULL + sd), (p / Sm::do_stages) & 1) && VSA_WARP_WAIT(bar(WK_P_FULL + b), ph);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
        wide_issue_product<HD, 64, kWkCols>(tmem_dv, tmem + b * 128, base + Sm::d_o + sd * Sm::part, p > 0);
        mma_commit(bar(WK_DO_EMPTY + sd));
        mma_commit(bar(WK_S_EMPTY + b));
      }
      __syncwarp();
      ok = VSA_WARP_WAIT(bar(WK_DS_FULL + b), ph);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
        wide_issue_product<HD, 64, kWkCols>(tmem_dk, tmem + b * 128 + 64, base + Sm::q + sq * Sm::part, p > 0);
        mma_commit(bar(WK_Q_EMPTY + sq));
        mma_commit(bar(WK_DP_EMPTY + b));
      }
      __syncwarp();
    }
    if (ok && elect_one()) mma_commit(bar(WK_ACC_FULL));
    __syncwarp();
    if (!ok && lane == 0) report_timeout(63);
  } else {
    const int quarter = warp & 3, cg = (warp - 4) >> 2;
    const int row = quarter * 32 + lane, c0 = cg * kWkCols, st = tid - 128;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const bool live = row < valid;
    float mean = 0.f;                       // one of the 2 x HD values that a live row receives from the pooled gradients
    if (mean_grad_k != nullptr && st < 2 * HD) mean = Elem<elem_t>::to(st < HD ? mean_grad_k[mean_off + st] : mean_grad_v[mean_off + st - HD]) * mean_inv;
    const float2 c2 = make_float2(-c, -c), m1 = make_float2(-1.f, -1.f);
    for (int p = 0; p < n_tiles && ok; ++p) {
      const int b = p & 1, sq = p % Sm::q_stages;
      const uint32_t ph = (p >> 1) & 1;
      ok = VSA_WARP_WAIT2(bar(WK_S_FULL + b), ph, bar(WK_Q_FULL + sq), (p / Sm::q_stages) & 1);
      if (!ok) break;
      tc_fence_after();
      const float4* s_lse = reinterpret_cast<const float4*>(sm + Sm::stats + sq * 512 + c0 * 4);
      const uint32_t s_addr = tmem + b * 128 + lane_addr + c0;
      uint32_t sv[kWkCols];
      tmem_ld(s_addr, sv);
      tmem_ld_wait();
      float2 pf[kWkCols / 2];
      uint32_t pk[kWkCols / 2];
#pragma unroll
      for (int i = 0; i < kWkCols / 4; ++i) {
        const float4 l4 = s_lse[i];
        // lse - S c, negated in the exponential: the packed operations have no sign of their own to spend on the statistics
        const float2 x = fma2(word_pair(sv + 4 * i), c2, make_float2(l4.x, l4.y));
        const float2 y = fma2(word_pair(sv + 4 * i + 2), c2, make_float2(l4.z, l4.w));
        pf[2 * i] = make_float2(fast_exp2(-x.x), fast_exp2(-x.y));
        pf[2 * i + 1] = make_float2(fast_exp2(-y.x), fast_exp2(-y.y));
        // a padding key row: its scores come from whatever sits in K there
        pk[2 * i] = live ? Elem<elem_t>::pack(pf[2 * i].x, pf[2 * i].y) : 0u;
        pk[2 * i + 1] = live ? Elem<elem_t>::pack(pf[2 * i + 1].x, pf[2 * i + 1].y) : 0u;
      }
      tmem_st(s_addr, pk);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(WK_P_FULL + b));
      ok = VSA_WARP_WAIT(bar(WK_DP_FULL + b), ph);
      if (!ok) break;
      tc_fence_after();
      uint32_t dvv[kWkCols];
      tmem_ld(s_addr + 64, dvv);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < kWkCols / 4; ++i) {
        const float4 d4 = s_lse[16 + i];       // delta: 64 floats behind the statistics
        const float2 x = mul2(pf[2 * i], fma2(word_pair(dvv + 4 * i), m1, make_float2(d4.x, d4.y)));      // -dS
        const float2 y = mul2(pf[2 * i + 1], fma2(word_pair(dvv + 4 * i + 2), m1, make_float2(d4.z, d4.w)));
        pk[2 * i] = live ? Elem<elem_t>::pack(x.x, x.y) : 0u;
        pk[2 * i + 1] = live ? Elem<elem_t>::pack(y.x, y.y) : 0u;
      }
      tmem_st(s_addr + 64, pk);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(WK_DS_FULL + b));
    }
    if (!ok && lane == 0) report_timeout(64);
    if (ok) ok = VSA_WARP_WAIT(bar(WK_ACC_FULL), 0);
    if (!ok && lane == 0) report_timeout(65);
    tc_fence_after();
    uint8_t* stage_k = sm + Sm::k;          // every MMA is done: dK over K, dV over V
    uint8_t* stage_v = sm + Sm::v;
    float* s_mean = reinterpret_cast<float*>(sm + Sm::stats);
    if (st < 2 * HD) s_mean[st] = mean;
    named_barrier(1, kWkEwThreads);
    for (int j = cg; j < 2 * (HD / 32); j += kWkGroups) {
      const bool is_k = j < HD / 32;
      const int jj = is_k ? j : j - HD / 32;
      uint32_t av[32];
      if (ok) {
        tmem_ld((is_k ? tmem_dk : tmem_dv) + lane_addr + 32 * jj, av);
        tmem_ld_wait();
        if (is_k) {
#pragma unroll
          for (int i = 0; i < 32; ++i) av[i] = __float_as_uint(__uint_as_float(av[i]) * -scale);      // the products summed -dS
        }
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) av[i] = 0u;
      }
      if (mean_grad_k != nullptr && live) wide_add_mean(av, s_mean + 32 * j);
#pragma unroll
      for (int q4 = 0; q4 < 4; ++q4)
        *reinterpret_cast<uint4*>((is_k ? stage_k : stage_v) + row * (HD * 2) + (((4 * jj + q4) ^ (row & 7)) << 4)) = wide_pack8(av + 8 * q4);
    }
    named_barrier(1, kWkEwThreads);
    for (int i = st; i < kWRows * HD / 8; i += kWkEwThreads) {
      const int r = i / (HD / 8), ch = i % (HD / 8);
      const long long drow = out_map.map == nullptr ? krow0 + r : raster_row(out_map, bh, (long long)ktile * kWRows + r);
      if (drow < 0) continue;
      const uint32_t off = r * (HD * 2) + ((ch ^ (r & 7)) << 4);
      *reinterpret_cast<uint4*>(dk + drow * HD + ch * 8) = *reinterpret_cast<const uint4*>(stage_k + off);
      *reinterpret_cast<uint4*>(dv + drow * HD + ch * 8) = *reinterpret_cast<const uint4*>(stage_v + off);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, kTmemCols);
}

// ---- host launchers of the 128-row kernels -----------------------------------------------------------------------
// Taken for block volumes that are multiples of 128, where sparse_wide_rows says so.
template <int HD>
int launch_fwd_wide(const void* q, const void* k, const void* v, const int32_t* selected, const int32_t* kv_sizes, void* out,
                    float* lse2, int64_t BH, int64_t Lq, int64_t Lkv, int be, int topk, float scale, cudaStream_t st,
                    const void* out_c, const void* gate, void* out_comb, int64_t kv_shard, RasterMap comb_map) {
  CUtensorMap mq, mk, mv;
  int rc;
  if ((rc = make_wide_map(&mq, q, BH * Lq, HD, kWRows, "sparse forward (q)"))) return rc;
  if ((rc = make_wide_map(&mk, k, BH * Lkv, HD, kWRows, "sparse forward (k)"))) return rc;
  if ((rc = make_wide_map(&mv, v, BH * Lkv, HD, kWRows, "sparse forward (v)"))) return rc;
  const int smem = WfSmem<HD>::total;
  if ((rc = reserve_smem(sparse_fwd_wide_kernel<HD>, smem, "sparse forward"))) return rc;
  sparse_fwd_wide_kernel<HD><<<dim3((unsigned)(Lq / kWRows), (unsigned)BH), kWfThreads, smem, st>>>(
      mq, mk, mv, selected, kv_sizes, (elem_t*)out, lse2, (const elem_t*)out_c, (const elem_t*)gate, (elem_t*)out_comb, Lq, Lkv,
      kv_shard, be, topk, scale, comb_map);
  return check_launch("sparse_fwd_wide_kernel");
}

template <int HD>
int launch_dq_wide(const void* dout, const void* q, const void* k, const void* v, const void* out_s, const float* lse2,
                   const int32_t* selected, const int32_t* kv_sizes, float* delta, void* dq, int64_t BH, int64_t Lq,
                   int64_t Lkv, int be, int topk, float scale, cudaStream_t st, const void* dq_mean, const int32_t* q_sizes,
                   int64_t kv_shard, RasterMap out_map) {
  CUtensorMap mq, mdo, mk, mv;
  int rc;
  if ((rc = make_wide_map(&mq, q, BH * Lq, HD, kWRows, "sparse dQ (q)"))) return rc;
  if ((rc = make_wide_map(&mdo, dout, BH * Lq, HD, kWRows, "sparse dQ (dout)"))) return rc;
  if ((rc = make_wide_map(&mk, k, BH * Lkv, HD, kWRows, "sparse dQ (k)"))) return rc;
  if ((rc = make_wide_map(&mv, v, BH * Lkv, HD, kWRows, "sparse dQ (v)"))) return rc;
  const int smem = WqSmem<HD>::total;
  if ((rc = reserve_smem(sparse_dq_wide_kernel<HD>, smem, "sparse dQ"))) return rc;
  sparse_dq_wide_kernel<HD><<<dim3((unsigned)(Lq / kWRows), (unsigned)BH), kWqThreads, smem, st>>>(
      mq, mdo, mk, mv, (const elem_t*)dout, (const elem_t*)out_s, lse2, selected, kv_sizes, delta, (elem_t*)dq,
      (const elem_t*)dq_mean, q_sizes, Lq, Lkv, kv_shard, be, topk, scale, out_map);
  return check_launch("sparse_dq_wide_kernel");
}

template <int HD>
int launch_dkdv_wide(const void* dout, const void* q, const void* k, const void* v, const float* lse2, const float* delta,
                     const int32_t* counts, const int32_t* offsets, const int32_t* inverse, const int32_t* kv_sizes, void* dk,
                     void* dv, int64_t BH, int64_t Lq, int64_t Lkv, int be, int topk, float scale, cudaStream_t st,
                     const void* dk_mean, const void* dv_mean, int64_t kv_shard, RasterMap out_map) {
  CUtensorMap mq, mdo, mk, mv;
  int rc;
  if ((rc = make_wide_map(&mq, q, BH * Lq, HD, kTile, "sparse dK/dV (q)"))) return rc;
  if ((rc = make_wide_map(&mdo, dout, BH * Lq, HD, kTile, "sparse dK/dV (dout)"))) return rc;
  if ((rc = make_wide_map(&mk, k, BH * Lkv, HD, kWRows, "sparse dK/dV (k)"))) return rc;
  if ((rc = make_wide_map(&mv, v, BH * Lkv, HD, kWRows, "sparse dK/dV (v)"))) return rc;
  const int smem = WkSmem<HD>::total;
  if ((rc = reserve_smem(sparse_dkdv_wide_kernel<HD>, smem, "sparse dK/dV"))) return rc;
  sparse_dkdv_wide_kernel<HD><<<dim3((unsigned)(Lkv / kWRows), (unsigned)BH), kWkThreads, smem, st>>>(
      mq, mdo, mk, mv, lse2, delta, counts, offsets, inverse, kv_sizes, (elem_t*)dk, (elem_t*)dv, (const elem_t*)dk_mean,
      (const elem_t*)dv_mean, Lq, Lkv, kv_shard, be, topk, scale, out_map);
  return check_launch("sparse_dkdv_wide_kernel");
}
