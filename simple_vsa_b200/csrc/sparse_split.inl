// Fine attention on 64-row tiles with the two lane halves of tensor memory on different tiles of the other side.  Included by
// sparse_umma_typed.inl, once per 16-bit element type.
//
// tcgen05.mma.ws with M = 64 spreads its result over all 128 lanes: lanes 0-63 hold the first half of the N columns, lanes
// 64-127 the second half, and an A operand in tensor memory is read by each lane half from its own lanes (checked on the
// device, bit for bit, with different operands in the two halves).  With N covering a PAIR of 64-token tiles the halves
// therefore work on different tiles, and the second product is two products at once:
//   forward  S [64 rows x 64 keys | 64 keys] = Q [K tile 2p | K tile 2p+1]^T     O  [64 x D | D] += [P | P] [V tile 2p | V tile 2p+1]
//   dQ       S, dP = dO [V | V]^T                                                dQ [64 x D | D] += [dS | dS] [K | K]
//   dK/dV    S^T = K [Q tile 2p | Q tile 2p+1]^T, dP^T = V [dO | dO]^T           dV += [P^T | P^T] [dO | dO],  dK += [dS^T | dS^T] [Q | Q]
// A lane is one row of the resident tile and one parity of the tiles that stream by.  P and dS never leave tensor memory, row
// statistics of the resident side are thread-local, and the two partial results are added once, in the epilogue.
//
// Why not the 128 x 64 products on transposed operands that these kernels replace: those read 6 KB of shared memory per 32 cycles
// of tensor work and pass P / dS through it, 176 / 224 / 288 KB a pair at D = 128 (forward / dQ / dK/dV, 64 KB of TMA writes
// among them).  Here it is 136 / 160 / 208 KB: operands in tensor memory cost no shared-memory reads, and one MMA (47 cycles for
// M64 x N128 x K16, 76 for N256) reads 4 KB or 8 KB of B alone.  At 90 pairs a tile a pair takes 847 / 1318 / 1690 cycles, set-up
// and drain included, with operand reads at 67 / 57 / 68 % of their peak and the tensor pipe at 60 / 58 / 61 % ([1, 8, 92160, 128],
// topk 180): what bounds it is the chain product -> elementwise -> product, and 10,000 to 12,000 cycles of set-up and drain a tile.

// Live 64-token key tiles of a query block in routing order: row of the tile in the K/V tensors (a multiple of 64) << 1 | live
// tokens.  Called by the whole CTA; ends with a barrier.  Ids outside the key table and empty tiles are dropped.
__device__ __forceinline__ void split_tile_list(uint32_t* list, volatile uint32_t* n_live_out, const int32_t* sel,
                                                const int32_t* kv_sizes, int topk, int sub, int Kb, long long bh,
                                                long long BH, long long kv_shard, int tid, int threads) {
  const int n_iter = topk * sub;
  for (int it = tid; it < n_iter; it += threads) {
    const int slot = it / sub, part = it - slot * sub;
    const int kvb = sel[slot];
    int left = (unsigned)kvb < (unsigned)Kb ? kv_sizes[kvb] - part * kTile : 0;
    left = left > kTile ? kTile : left;
    list[it] = left > 0 ? (uint32_t)kv_tensor_row(bh, BH, ((long long)kvb * sub + part) * kTile, kv_shard) << 1 | (uint32_t)left : 0u;
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
__device__ __forceinline__ int split_row(uint32_t entry) { return (int)(entry >> 7) << 6; }
__device__ __forceinline__ int split_valid(uint32_t entry) { return (int)(entry & 127u); }

// [rows, dim] row-major, boxes of box_rows rows x all head dims that land as one [box_rows][128 bytes] slab per 64 dims.
int make_slab_map(CUtensorMap* map, const void* ptr, int64_t rows, int dim, int box_rows, const char* what) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return fail(VSA_ERR_LAUNCH, "%s: cuTensorMapEncodeTiled is not available from the driver", what);
  if (reinterpret_cast<uintptr_t>(ptr) % 16) return fail(VSA_ERR_BAD_ARGUMENT, "%s: pointer is not 16-byte aligned", what);
  if (rows > 0x7fffffffLL) return fail(VSA_ERR_UNSUPPORTED, "%s: %lld rows exceed the TMA coordinate range", what, (long long)rows);
  const cuuint64_t gdim[3] = {64, (cuuint64_t)rows, (cuuint64_t)(dim / 64)};
  const cuuint64_t gstride[2] = {(cuuint64_t)dim * 2, 128};
  const cuuint32_t box[3] = {64, (cuuint32_t)box_rows, (cuuint32_t)(dim / 64)};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = fn(map, kTmaElem, 3, const_cast<void*>(ptr), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(VSA_ERR_LAUNCH, "%s: cuTensorMapEncodeTiled failed with code %d", what, (int)r);
  return VSA_OK;
}

// [64 x 64 | 64 x 64] (+)= A [64 x 64 head dims] (tensor memory) times 64 head dims of a pair of tiles: 128 rows x 128 bytes, K-major.
__device__ __forceinline__ void split_issue_scores_ts(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_part, bool accumulate) {
  constexpr uint32_t idesc = instr_desc(64, 128, 0, 0, kInFmt);
  constexpr uint32_t hi = desc_hi(1024);
  const uint32_t b0 = desc_lo(b_part, 16), acc0 = accumulate ? 1u : 0u;
#pragma unroll
  for (int ks = 0; ks < 4; ++ks) mma_ws_ts(d_tmem, a_tmem + 8 * ks, desc_pack(b0 + 2 * ks, hi), idesc, ks > 0 ? 1u : acc0);
}
// [64 x 64 | 64 x 64 head dims] (+)= [A | A] (64 x 64 each, tensor memory) times the same part read along its rows: the two
// tiles are the two halves of the N columns.
__device__ __forceinline__ void split_issue_product(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_part, bool accumulate) {
  constexpr uint32_t idesc = instr_desc(64, 128, 0, 1, kInFmt);
  constexpr uint32_t hi = desc_hi(1024);
  const uint32_t b0 = desc_lo(b_part, kSlab), acc0 = accumulate ? 1u : 0u;
#pragma unroll
  for (int ks = 0; ks < 4; ++ks) mma_ws_ts(d_tmem, a_tmem + 8 * ks, desc_pack(b0 + 128 * ks, hi), idesc, ks > 0 ? 1u : acc0);
}

// Accumulator columns [begin, begin + W) of the 64 rows, the two lane halves added: each thread finishes W/2 of them for its
// row and stages them as 16-bit values, [64 rows][HD] with 16-byte chunks xor row.  128 threads (a warp per lane quarter) on
// named barrier `id`; `exchange`: 64 * W * 4 bytes that nothing else uses any more.  `finish` works on N sums from column c.
template <int HD, int W, typename Finish>
__device__ __forceinline__ void split_add_halves(uint32_t acc, bool have, uint8_t* exchange, uint8_t* stage, int begin, int half,
                                                 int r, int id, Finish&& finish) {
  constexpr int kMine = W / 2, N = kMine < 32 ? kMine : 32;
  uint8_t* give = exchange + half * (64 * kMine * 4) + r * (kMine * 4);
  const uint8_t* take = exchange + (half ^ 1) * (64 * kMine * 4) + r * (kMine * 4);
  constexpr int kSwz = kMine / 4 < 8 ? kMine / 4 - 1 : 7;
  if (have) {
#pragma unroll
    for (int j = 0; j < kMine / N; ++j) {
      uint32_t ov[N];
      tmem_ld(acc + begin + (half ^ 1) * kMine + N * j, ov);
      tmem_ld_wait();
#pragma unroll
      for (int q4 = 0; q4 < N / 4; ++q4)
        *reinterpret_cast<uint4*>(give + (((N / 4 * j + q4) ^ (r & kSwz)) << 4)) = make_uint4(ov[4 * q4], ov[4 * q4 + 1], ov[4 * q4 + 2], ov[4 * q4 + 3]);
    }
  }
  named_barrier(id, 128);
#pragma unroll
  for (int j = 0; j < kMine / N; ++j) {
    const int c0 = begin + half * kMine + N * j;
    uint32_t ov[N];
    if (have) {
      tmem_ld(acc + c0, ov);
      tmem_ld_wait();
#pragma unroll
      for (int q4 = 0; q4 < N / 4; ++q4) {
        const float4 o = *reinterpret_cast<const float4*>(take + (((N / 4 * j + q4) ^ (r & kSwz)) << 4));
        ov[4 * q4] = __float_as_uint(__uint_as_float(ov[4 * q4]) + o.x);
        ov[4 * q4 + 1] = __float_as_uint(__uint_as_float(ov[4 * q4 + 1]) + o.y);
        ov[4 * q4 + 2] = __float_as_uint(__uint_as_float(ov[4 * q4 + 2]) + o.z);
        ov[4 * q4 + 3] = __float_as_uint(__uint_as_float(ov[4 * q4 + 3]) + o.w);
      }
    } else {
#pragma unroll
      for (int i = 0; i < N; ++i) ov[i] = 0u;
    }
    finish(ov, c0);
#pragma unroll
    for (int q8 = 0; q8 < N / 8; ++q8)
      *reinterpret_cast<uint4*>(stage + r * (HD * 2) + (((c0 / 8 + q8) ^ (r & 7)) << 4)) = wide_pack8(ov + 8 * q8);
  }
  named_barrier(id, 128);
}
// Row r of a slab (64 head dims, TMA's 128-byte swizzle) to 32 columns of this thread's lane, two 16-bit values each.  Read from
// shared memory: fetched by each thread from global memory, a row of 256 bytes per lane, Q and dO took 14,000 cycles to get here.
__device__ __forceinline__ void split_store_row(uint32_t taddr, const uint8_t* slab, int r) {
  uint32_t w[2][16];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint4 x = *reinterpret_cast<const uint4*>(slab + r * 128 + ((i ^ (r & 7)) << 4));
    w[i >> 2][4 * (i & 3)] = x.x;
    w[i >> 2][4 * (i & 3) + 1] = x.y;
    w[i >> 2][4 * (i & 3) + 2] = x.z;
    w[i >> 2][4 * (i & 3) + 3] = x.w;
  }
  tmem_st(taddr, w[0]);
  tmem_st(taddr + 16, w[1]);
}
// A row of HD values, stored as slabs of 128 bytes `slab` bytes apart, becomes zero.  Lanes of a warp hold consecutive rows:
// the chunk order differs between them, so that eight lanes cover all banks (30 % ragged tiles: 558 -> 452 us of forward).
template <int HD>
__device__ __forceinline__ void split_zero_row(uint8_t* row, int r, uint32_t slab) {
#pragma unroll
  for (int ch = 0; ch < HD / 8; ++ch)
    *reinterpret_cast<uint4*>(row + (ch >> 3) * slab + (((ch ^ r) & 7) << 4)) = make_uint4(0, 0, 0, 0);
}

// ------------------------------------------------------------------------------------------------------
// forward
// ------------------------------------------------------------------------------------------------------
// Two CTAs share an SM, 113 KB and 256 columns each: what one spends on its tile list, its first loads and its epilogue is the
// other's steady state, and the chain product -> softmax -> product of one pair runs under the other CTA's.  K and V pairs arrive
// in parts of 16 KB (K: 64 head dims of both tiles; V: 32 keys of both tiles at D = 128), a ring of three parts each.  P has
// columns of its own, so the score columns are free as soon as they have been read.  Half of Q sits in tensor memory, which is
// what its columns allow beside O (128), S (64) and P (32).
// The softmax shift of a row is its maximum over the first live pair, as in the 128-row kernels; rows that leave the finite range
// send the tile to the exact kernel.
constexpr int kSfThreads = 256;
constexpr int kSfStages = 3;                        // parts of K and of V in flight
template <int HD>
struct SfSmem {
  static constexpr uint32_t part = 16384;
  static constexpr uint32_t k = 0;                                // part: 64 head dims of both tiles, 128 rows x 128 bytes
  static constexpr uint32_t v = k + kSfStages * part;             // part: 64*64/HD keys of both tiles, all head dims
  static constexpr uint32_t q = v + kSfStages * part;             // head dims 64..127 of Q (0..63 are in tensor memory)
  static constexpr uint32_t list = q + (HD / 64 - 1) * kSlab;     // uint32 [kMaxTiles]
  static constexpr uint32_t m_row = list + 4 * kMaxTiles;         // float [64]
  static constexpr uint32_t l_part = m_row + 256;                 // float [128]
  static constexpr uint32_t bars = l_part + 512;
  static constexpr uint32_t misc = bars + 24 * 8;
  static constexpr uint32_t total = misc + 32;
};
static_assert(SfSmem<128>::total + 1024 <= 115712, "two CTAs of the forward share an SM");
enum SfBar { SF_Q_FULL = 0, SF_QT_FULL = 1, SF_K_FULL = 2, SF_K_EMPTY = 5, SF_V_FULL = 8, SF_V_EMPTY = 11, SF_S_FULL = 14,
             SF_S_EMPTY = 15, SF_P_FULL = 16, SF_P_EMPTY = 17, SF_O_FULL = 18 };
constexpr uint32_t kSfTmem = 256;                   // O 128 columns, S 64, P 32, Q 32

template <int HD>
__global__ void __launch_bounds__(kSfThreads, 2)
sparse_fwd_split_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                        const __grid_constant__ CUtensorMap map_v, const int32_t* __restrict__ selected,
                        const int32_t* __restrict__ kv_sizes, elem_t* __restrict__ out, float* __restrict__ lse2,
                        const elem_t* __restrict__ out_c, const elem_t* __restrict__ gate, elem_t* __restrict__ out_comb,
                        long long Lq, long long Lkv, long long kv_shard, int sub, int topk, float scale, RasterMap comb_map) {
  using Sm = SfSmem<HD>;
  constexpr int kParts = HD / 64;
  constexpr int kVRows = 64 / kParts;               // keys of each tile in a part of V
  // Head dim 64 takes the place of an online softmax, whose largest P is 1 exactly; with P rounded under a fixed shift the output was
  // 2-3 % further from float64.  Its O leaves 64 columns free, so what the rounding of P loses is kept there, in the element type,
  // and multiplied too.
  constexpr bool kSplitP = HD == 64;
  constexpr uint32_t kQStage = Sm::v + (kSfStages - 1) * Sm::part;     // Q on its way to tensor memory, in the last part of V
  extern __shared__ uint8_t smem_raw[];
  if (*(volatile int*)&g_device_status != 0) return;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* sm = smem_raw + (base - smem_u32(smem_raw));
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int qtile = blockIdx.x;
  const long long bh = blockIdx.y, BH = gridDim.y;
  const int Qb = (int)(Lq / (kTile * sub)), qb = qtile / sub;
  const long long row0 = bh * Lq + (long long)qtile * kTile;
  const float c = scale * kLog2e;
  uint32_t* list = reinterpret_cast<uint32_t*>(sm + Sm::list);
  float* m_row = reinterpret_cast<float*>(sm + Sm::m_row);
  volatile uint32_t* misc = reinterpret_cast<volatile uint32_t*>(sm + Sm::misc);   // tmem base, live tiles, redo flag
  auto bar = [&](int i) -> uint32_t { return base + Sm::bars + 8u * i; };

  if (tid == 0) {
    mbar_init(bar(SF_Q_FULL), 1);
    mbar_init(bar(SF_QT_FULL), 4);
    for (int i = 0; i < kSfStages; ++i) {
      mbar_init(bar(SF_K_FULL + i), 2);
      mbar_init(bar(SF_K_EMPTY + i), 1);
      mbar_init(bar(SF_V_FULL + i), 2);
      mbar_init(bar(SF_V_EMPTY + i), 1);
    }
    mbar_init(bar(SF_S_FULL), 1);
    mbar_init(bar(SF_S_EMPTY), 4);
    mbar_init(bar(SF_P_FULL), 4);
    mbar_init(bar(SF_P_EMPTY), 1);
    mbar_init(bar(SF_O_FULL), 1);
    misc[2] = 0u;
    fence_barrier_init();
    tma_prefetch_desc(&map_k);
    tma_prefetch_desc(&map_v);
    mbar_arrive_expect_tx(bar(SF_Q_FULL), HD * 128);
    tma_load_2d(base + kQStage, &map_q, 0, (int)row0, bar(SF_Q_FULL));
    if (HD > 64) tma_load_2d(base + Sm::q, &map_q, 64, (int)row0, bar(SF_Q_FULL));
  }
  if (warp == 2) {
    tmem_alloc(base + Sm::misc, kSfTmem);
    tmem_relinquish();
  }
  tc_fence_before();
  split_tile_list(list, misc + 1, selected + (bh * Qb + qb) * (long long)topk, kv_sizes, topk, sub, (int)(Lkv / (kTile * sub)),
                  bh, BH, kv_shard, tid, kSfThreads);
  tc_fence_after();
  const uint32_t tmem_o = misc[0], tmem_s = tmem_o + 128, tmem_p = tmem_o + 192, tmem_q = tmem_o + 224;
  const uint32_t tmem_plo = tmem_o + 64;            // head dim 64: what P lost in rounding
  const int n_live = (int)misc[1], n_pairs = (n_live + 1) >> 1;
  bool ok = true;

  if (warp < 2) {
    // producers: the two tiles of a pair on two lanes; the second one of an odd tail lies outside the tensor, i.e. is zero
    const bool is_k = warp == 0;
    const CUtensorMap* map = is_k ? &map_k : &map_v;
    const int full0 = is_k ? SF_K_FULL : SF_V_FULL, empty0 = is_k ? SF_K_EMPTY : SF_V_EMPTY;
    const uint32_t ring = base + (is_k ? Sm::k : Sm::v);
    for (int i = 0; i < n_pairs * kParts; ++i) {
      const int s = i % kSfStages, idx = 2 * (i / kParts) + lane, h = i % kParts;
      ok = VSA_WARP_WAIT(bar(empty0 + s), ((i / kSfStages) & 1) ^ 1) && (is_k || i != kSfStages - 1 || VSA_WARP_WAIT(bar(SF_QT_FULL), 0));
      if (!ok) break;
      if (lane < 2) {
        const int row = idx < n_live ? split_row(list[idx]) : (int)(BH * Lkv);
        mbar_arrive_expect_tx(bar(full0 + s), Sm::part / 2);
        const uint32_t dst = ring + s * Sm::part + lane * (Sm::part / 2);
        if (is_k)
          tma_load_2d(dst, map, h * 64, row, bar(full0 + s));
        else
          tma_load_3d(dst, map, 0, row + h * kVRows, 0, bar(full0 + s));
      }
      __syncwarp();
    }
    if (!ok && lane == 0) report_timeout(is_k ? 71 : 72);
  } else if (warp == 2) {
    // S = Q K^T
    constexpr uint32_t idesc = instr_desc(64, 128, 0, 0, kInFmt);
    constexpr uint32_t hi = desc_hi(1024);
    const uint32_t aq = desc_lo(base + Sm::q, 16);
    ok = VSA_WARP_WAIT2(bar(SF_Q_FULL), 0, bar(SF_QT_FULL), 0);
    for (int p = 0; p < n_pairs && ok; ++p) {
      const int i0 = p * kParts, i1 = i0 + kParts - 1;
      ok = VSA_WARP_WAIT3(bar(SF_K_FULL + i0 % kSfStages), (i0 / kSfStages) & 1, bar(SF_K_FULL + i1 % kSfStages),
                          (i1 / kSfStages) & 1, bar(SF_S_EMPTY), (p & 1) ^ 1);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int h = 0; h < kParts; ++h) {
          const int s = (i0 + h) % kSfStages;
          const uint32_t b0 = desc_lo(base + Sm::k + s * Sm::part, 16);
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) {
            if (h == 0)
              mma_ws_ts(tmem_s, tmem_q + 8 * ks, desc_pack(b0 + 2 * ks, hi), idesc, ks > 0 ? 1u : 0u);
            else
              mma_ws_ss(tmem_s, desc_pack(aq + 2 * ks, hi), desc_pack(b0 + 2 * ks, hi), idesc, 1u);
          }
          mma_commit(bar(SF_K_EMPTY + s));
        }
        mma_commit(bar(SF_S_FULL));
      }
      __syncwarp();
    }
    if (!ok && lane == 0) report_timeout(73);
  } else if (warp == 3) {
    // O += P V
    constexpr uint32_t idesc = instr_desc(64, 2 * HD, 0, 1, kInFmt);
    constexpr uint32_t hi = desc_hi(1024);
    for (int p = 0; p < n_pairs && ok; ++p) {
      const int i0 = p * kParts, i1 = i0 + kParts - 1;
      ok = VSA_WARP_WAIT3(bar(SF_V_FULL + i0 % kSfStages), (i0 / kSfStages) & 1, bar(SF_V_FULL + i1 % kSfStages),
                          (i1 / kSfStages) & 1, bar(SF_P_FULL), p & 1);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int h = 0; h < kParts; ++h) {
          const int s = (i0 + h) % kSfStages;
          const uint32_t b0 = desc_lo(base + Sm::v + s * Sm::part, kVRows * 128);
#pragma unroll
          for (int ks = 0; ks < kVRows / 16; ++ks) {
            mma_ws_ts(tmem_o, tmem_p + 8 * (h * (kVRows / 16) + ks), desc_pack(b0 + 128 * ks, hi), idesc, p > 0 || h > 0 || ks > 0 ? 1u : 0u);
            if (kSplitP) mma_ws_ts(tmem_o, tmem_plo + 8 * ks, desc_pack(b0 + 128 * ks, hi), idesc, 1u);
          }
          mma_commit(bar(SF_V_EMPTY + s));
        }
        mma_commit(bar(SF_P_EMPTY));
      }
      __syncwarp();
    }
    if (ok && elect_one()) mma_commit(bar(SF_O_FULL));
    __syncwarp();
    if (!ok && lane == 0) report_timeout(74);
  } else {
    // softmax: a thread owns query row r on the tiles of one parity
    const int quarter = warp & 3, half = quarter >> 1, r = (quarter & 1) * 32 + lane, st = tid - 128;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    ok = VSA_WARP_WAIT(bar(SF_Q_FULL), 0);
    split_store_row(tmem_q + lane_addr, sm + kQStage, r);     // the same in both halves
    tmem_st_wait();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(SF_QT_FULL));
    float2 lsum = make_float2(0.f, 0.f);
    float neg_m = 0.f;
    bool shifted = n_pairs == 0;
    for (int p = 0; p < n_pairs && ok; ++p) {
      const int idx = 2 * p + half;
      const int valid = idx < n_live ? split_valid(list[idx]) : 0;
      ok = VSA_WARP_WAIT(bar(SF_S_FULL), p & 1);
      if (!ok) break;
      tc_fence_after();
      uint32_t sv[2][32];
      tmem_ld(tmem_s + lane_addr, sv[0]);
      tmem_ld(tmem_s + lane_addr + 32, sv[1]);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(SF_S_EMPTY));
      if (p == 0) {          // the row's shift: maximum over the first pair of live tiles
        float m = -INFINITY;
#pragma unroll
        for (int i = 0; i < 64; ++i) m = fmaxf(m, i < valid ? __uint_as_float(sv[i >> 5][i & 31]) * c : -INFINITY);
        if (half == 0) m_row[r] = m;
        named_barrier(1, 128);
        if (half == 1) {
          m = fmaxf(m, m_row[r]) + (HD != 64 ? kShiftBias : 0.f);     // head dim 64: see the 128-row forward
          m_row[r] = m;
        }
        named_barrier(1, 128);
        neg_m = -m_row[r];
        shifted = true;
      }
      const float2 c2 = make_float2(c, c), m2 = make_float2(neg_m, neg_m);
      uint32_t pk[2][16], lo[2][16];
      // full and ragged tiles are separate code: a mask costs two more instructions per score
      auto exponentiate = [&](auto ragged) {
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const float2 x = fma2(word_pair(&sv[i >> 4][2 * (i & 15)]), c2, m2);
          float2 e = make_float2(fast_exp2(x.x), fast_exp2(x.y));
          if (decltype(ragged)::value) {     // scores of padding keys come from whatever sits in K there: select
            if (2 * i >= valid) e.x = 0.f;
            if (2 * i + 1 >= valid) e.y = 0.f;
          }
          lsum = add2(lsum, e);
          const uint32_t w = Elem<elem_t>::pack(e.x, e.y);
          if (kSplitP) {
            const float2 rounded = Elem<elem_t>::unpack(w);
            lo[i >> 4][i & 15] = Elem<elem_t>::pack(e.x - rounded.x, e.y - rounded.y);
          }
          pk[i >> 4][i & 15] = w;
        }
      };
      if (valid == kTile) exponentiate(std::false_type{});
      else exponentiate(std::true_type{});
      ok = VSA_WARP_WAIT(bar(SF_P_EMPTY), (p & 1) ^ 1);
      if (!ok) break;
      tc_fence_after();
      if (valid < kTile && idx < n_live) {
        // Padding rows of V meet P = 0 in the product: they must be finite (0 * NaN).  Not before P V of the last pair has completed:
        // only then has the part's slot been filled for every earlier pair, so that this parity can mean nothing but this pair.
        const int i = p * kParts + r / kVRows, s = i % kSfStages;
        ok = VSA_WARP_WAIT(bar(SF_V_FULL + s), (i / kSfStages) & 1);
        if (!ok) break;
        if (r >= valid) split_zero_row<HD>(sm + Sm::v + s * Sm::part + half * (Sm::part / 2) + (r % kVRows) * 128, r, kVRows * 128);
        fence_proxy_async_smem();
      }
      tmem_st(tmem_p + lane_addr, pk[0]);
      tmem_st(tmem_p + lane_addr + 16, pk[1]);
      if (kSplitP) {
        tmem_st(tmem_plo + lane_addr, lo[0]);
        tmem_st(tmem_plo + lane_addr + 16, lo[1]);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(SF_P_FULL));
    }
    if (!ok && lane == 0) report_timeout(75);
    if (!shifted) {          // a wait that ran out: the barriers that the other warps may be in
      named_barrier(1, 128);
      named_barrier(1, 128);
    }
    if (ok && n_pairs > 0) ok = VSA_WARP_WAIT(bar(SF_O_FULL), 0);
    if (!ok && lane == 0) report_timeout(76);
    tc_fence_after();
    // add the two halves: each thread finishes half of the head dims of its row.  Every MMA is done, the rings are free.
    float* l_part = reinterpret_cast<float*>(sm + Sm::l_part);
    l_part[st] = lsum.x + lsum.y;
    uint8_t* stage = sm + 64 * HD * 4;
    float l = 0.f;
    bool finite = true;
    split_add_halves<HD, HD>(tmem_o + lane_addr, ok && n_pairs > 0, sm, stage, 0, half, r, 1, [&](auto& ov, int) {
      l = l_part[r] + l_part[64 + r];
      finite = finite && l <= 3.0e38f;
#pragma unroll
      for (auto& w : ov) {
        const float o = __uint_as_float(w) / l;
        finite = finite && fabsf(o) <= 3.0e38f;
        w = n_pairs == 0 ? 0x7fc00000u : __float_as_uint(o);
      }
      if (!finite) misc[2] = 1u;
    });
    for (int i = st; i < kTile * HD / 8; i += 128) {
      const int rr = i / (HD / 8), ch = i % (HD / 8);
      const uint4 ov = *reinterpret_cast<const uint4*>(stage + rr * (HD * 2) + ((ch ^ (rr & 7)) << 4));
      *reinterpret_cast<uint4*>(out + (row0 + rr) * HD + ch * 8) = ov;
      if (out_comb != nullptr) {   // gated combine with the pooled branch on the way out
        const long long crow = comb_map.map == nullptr ? row0 + rr : raster_row(comb_map, bh, (long long)qtile * kTile + rr);
        if (crow >= 0) {
          const uint4 cv = *reinterpret_cast<const uint4*>(out_c + (bh * Qb + qb) * (long long)HD + ch * 8);
          uint4 gv = make_uint4(0, 0, 0, 0);
          if (gate != nullptr) gv = *reinterpret_cast<const uint4*>(gate + crow * HD + ch * 8);
          *reinterpret_cast<uint4*>(out_comb + crow * HD + ch * 8) = combine_x8<elem_t>(ov, cv, gv, gate != nullptr);
        }
      }
    }
    if (half == 0) {
      const bool redo = misc[2] != 0u && ok;
      lse2[row0 + r] = (redo || n_pairs == 0) ? NAN : m_row[r] + log2f(l);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 2) tmem_dealloc(misc[0], kSfTmem);
}

template <int HD>
int launch_fwd_split(const void* q, const void* k, const void* v, const int32_t* selected, const int32_t* kv_sizes, void* out,
                     float* lse2, int64_t BH, int64_t Lq, int64_t Lkv, int be, int topk, float scale, cudaStream_t st,
                     const void* out_c, const void* gate, void* out_comb, int64_t kv_shard, RasterMap comb_map) {
  CUtensorMap mq, mk, mv;
  int rc;
  if ((rc = make_wide_map(&mq, q, BH * Lq, HD, kTile, "sparse forward (q)"))) return rc;
  if ((rc = make_wide_map(&mk, k, BH * Lkv, HD, kTile, "sparse forward (k)"))) return rc;
  if ((rc = make_slab_map(&mv, v, BH * Lkv, HD, 64 * 64 / HD, "sparse forward (v)"))) return rc;
  const int smem = SfSmem<HD>::total + 1024;
  if ((rc = reserve_smem(sparse_fwd_split_kernel<HD>, smem, "sparse forward", true))) return rc;
  sparse_fwd_split_kernel<HD><<<dim3((unsigned)(Lq / kTile), (unsigned)BH), kSfThreads, smem, st>>>(
      mq, mk, mv, selected, kv_sizes, (elem_t*)out, lse2, (const elem_t*)out_c, (const elem_t*)gate, (elem_t*)out_comb, Lq, Lkv,
      kv_shard, be / kTile, topk, scale, comb_map);
  return check_launch("sparse_fwd_split_kernel");
}

// ------------------------------------------------------------------------------------------------------
// dQ
// ------------------------------------------------------------------------------------------------------
// One CTA per SM.  Q and dO live in tensor memory, so all of shared memory is K (four pairs) and V (two and a half).  Two
// elementwise groups of four warps take alternate pairs, 64 scores a thread.  S, dP (two buffers) and dS (two) have columns of
// their own: score columns are free as soon as a group has read them.
constexpr int kSqThreads = 512;                     // warps 0-3 and 12-15: loads and MMA issue; 4-11: elementwise
template <int HD>
struct SqSmem {
  static constexpr uint32_t part = 16384;                         // 64 head dims of a pair: 128 rows x 128 bytes
  static constexpr uint32_t pair = (HD / 64) * part;
  static constexpr int k_stages = 4, v_parts = 5;
  static constexpr uint32_t k = 0;
  static constexpr uint32_t v = k + k_stages * pair;
  static constexpr uint32_t list = v + v_parts * part;            // uint32 [kMaxTiles]
  static constexpr uint32_t mean = list + 4 * kMaxTiles;          // float [HD]: what a live row receives from the pooled gradient
  static constexpr uint32_t delta = mean + HD * 4;                // float [64]
  static constexpr uint32_t bars = delta + 256;
  static constexpr uint32_t misc = bars + 40 * 8;
  static constexpr uint32_t total = misc + 32;
};
static_assert(SqSmem<128>::total + 1024 <= 232448, "shared memory of the split dQ pass");
enum SqBar { SQ_QT_FULL = 0, SQ_DOT_FULL = 1, SQ_K_FULL = 2, SQ_K_EMPTY = 6, SQ_V_FULL = 10, SQ_V_EMPTY = 15, SQ_S_FULL = 20,
             SQ_S_EMPTY = 22, SQ_DP_FULL = 23, SQ_DP_EMPTY = 25, SQ_DS_FULL = 27, SQ_DS_EMPTY = 29, SQ_ACC_FULL = 31, SQ_QDO_FULL = 32 };

template <int HD>
__global__ void __launch_bounds__(kSqThreads, 1)
sparse_dq_split_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_do,
                       const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                       const elem_t* __restrict__ dout, const elem_t* __restrict__ out_s, const float* __restrict__ lse2,
                       const int32_t* __restrict__ selected, const int32_t* __restrict__ kv_sizes, float* __restrict__ delta,
                       elem_t* __restrict__ dq, const elem_t* __restrict__ mean_grad, const int32_t* __restrict__ q_sizes,
                       long long Lq, long long Lkv, long long kv_shard, int sub, int topk, float scale, RasterMap out_map) {
  using Sm = SqSmem<HD>;
  constexpr int kParts = HD / 64;
  constexpr uint32_t kStage = Sm::k + (Sm::k_stages - 1) * Sm::pair;      // Q and dO on their way to tensor memory, in the last K stage
  extern __shared__ uint8_t smem_raw[];
  if (*(volatile int*)&g_device_status != 0) return;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* sm = smem_raw + (base - smem_u32(smem_raw));
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int qtile = blockIdx.x;
  const long long bh = blockIdx.y, BH = gridDim.y;
  const int Qb = (int)(Lq / (kTile * sub)), qb = qtile / sub;
  const long long row0 = bh * Lq + (long long)qtile * kTile;
  const float c = scale * kLog2e;
  uint32_t* list = reinterpret_cast<uint32_t*>(sm + Sm::list);
  volatile uint32_t* misc = reinterpret_cast<volatile uint32_t*>(sm + Sm::misc);
  auto bar = [&](int i) -> uint32_t { return base + Sm::bars + 8u * i; };

  if (tid == 0) {
    mbar_init(bar(SQ_QT_FULL), 4);
    mbar_init(bar(SQ_DOT_FULL), 4);
    for (int i = 0; i < Sm::k_stages; ++i) {
      mbar_init(bar(SQ_K_FULL + i), 2 * kParts);
      mbar_init(bar(SQ_K_EMPTY + i), 1);
    }
    for (int i = 0; i < Sm::v_parts; ++i) {
      mbar_init(bar(SQ_V_FULL + i), 2);
      mbar_init(bar(SQ_V_EMPTY + i), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar(SQ_S_FULL + i), 1);       // by parity of the pair, for the group that takes it; the columns are the same
      mbar_init(bar(SQ_DP_FULL + i), 1);
      mbar_init(bar(SQ_DP_EMPTY + i), 4);
      mbar_init(bar(SQ_DS_FULL + i), 4);
      mbar_init(bar(SQ_DS_EMPTY + i), 1);
    }
    mbar_init(bar(SQ_S_EMPTY), 4);
    mbar_init(bar(SQ_ACC_FULL), 1);
    mbar_init(bar(SQ_QDO_FULL), 1);
    fence_barrier_init();
    tma_prefetch_desc(&map_k);
    tma_prefetch_desc(&map_v);
    mbar_arrive_expect_tx(bar(SQ_QDO_FULL), 2 * HD * 128);
    wide_load<HD>(base + kStage, &map_q, (int)row0, kSlab, bar(SQ_QDO_FULL));
    wide_load<HD>(base + kStage + HD * 128, &map_do, (int)row0, kSlab, bar(SQ_QDO_FULL));
  }
  if (warp == 12) {
    tmem_alloc(base + Sm::misc, kTmemCols);
    tmem_relinquish();
  }
  // delta = rowsum(out_s * dout): four neighbouring threads per row
  float* s_delta = reinterpret_cast<float*>(sm + Sm::delta);
  if (warp >= 4 && warp < 12) {
    const int row = (tid - 128) >> 2, part = tid & 3;
    const uint4* po = reinterpret_cast<const uint4*>(out_s + (row0 + row) * HD + part * (HD / 4));
    const uint4* pd = reinterpret_cast<const uint4*>(dout + (row0 + row) * HD + part * (HD / 4));
    float acc = 0.f;
#pragma unroll
    for (int i = 0; i < HD / 32; ++i) {
      const uint4 a = po[i], b = pd[i];
      const elem_t* ea = reinterpret_cast<const elem_t*>(&a);
      const elem_t* eb = reinterpret_cast<const elem_t*>(&b);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc = fmaf(Elem<elem_t>::to(ea[j]), Elem<elem_t>::to(eb[j]), acc);
    }
    acc += __shfl_xor_sync(0xffffffffu, acc, 1);
    acc += __shfl_xor_sync(0xffffffffu, acc, 2);
    if (part == 0) {
      s_delta[row] = acc;
      delta[row0 + row] = acc;
    }
  }
  // block-mean backward folded in: query row r of the block also receives dmean[block] / max(size, 1) while r < size
  float* s_mean = reinterpret_cast<float*>(sm + Sm::mean);
  int rows_live = 0;
  if (mean_grad != nullptr) {
    const int size = q_sizes[qb];
    rows_live = size - (qtile % sub) * kTile;
    if (tid < HD) s_mean[tid] = Elem<elem_t>::to(mean_grad[(bh * Qb + qb) * (long long)HD + tid]) / (float)(size > 1 ? size : 1);
  }
  tc_fence_before();
  split_tile_list(list, misc + 1, selected + (bh * Qb + qb) * (long long)topk, kv_sizes, topk, sub, (int)(Lkv / (kTile * sub)),
                  bh, BH, kv_shard, tid, kSqThreads);
  tc_fence_after();
  const uint32_t tmem = misc[0];
  const uint32_t tmem_acc = tmem, tmem_s = tmem + 128, tmem_dp = tmem + 192, tmem_ds = tmem + 320, tmem_q = tmem + 384, tmem_do = tmem + 448;
  const int n_live = (int)misc[1], n_pairs = (n_live + 1) >> 1;
  bool ok = true;

  if (warp >= 4 && warp < 12) {
    registers_inc<192>();
    const int quarter = warp & 3, half = quarter >> 1, r = (quarter & 1) * 32 + lane, g = (warp - 4) >> 2;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const float dl = s_delta[r], neg_lse = log2f(fabsf(scale)) - lse2[row0 + r];      // 2^(s c - lse) * |scale| in one exponential
    ok = VSA_WARP_WAIT(bar(SQ_QDO_FULL), 0);
#pragma unroll
    for (int h = 0; h < kParts; ++h)        // group 0 brings Q, group 1 dO
      split_store_row((g == 0 ? tmem_q : tmem_do) + lane_addr + 32 * h, sm + kStage + g * (HD * 128) + h * kSlab, r);
    tmem_st_wait();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(g == 0 ? SQ_QT_FULL : SQ_DOT_FULL));
    const float2 c2 = make_float2(c, c), l2 = make_float2(neg_lse, neg_lse), d2 = make_float2(-dl, -dl);
    for (int p = g; p < n_pairs && ok; p += 2) {
      const uint32_t ph = (p >> 1) & 1;
      const int idx = 2 * p + half;
      const int valid = idx < n_live ? split_valid(list[idx]) : 0;
      ok = VSA_WARP_WAIT(bar(SQ_S_FULL + g), ph);
      if (!ok) break;
      tc_fence_after();
      float2 pf[32];
      {
        uint32_t sv[2][32];
        tmem_ld(tmem_s + lane_addr, sv[0]);
        tmem_ld(tmem_s + lane_addr + 32, sv[1]);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(SQ_S_EMPTY));
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const float2 x = fma2(word_pair(&sv[i >> 4][2 * (i & 15)]), c2, l2);
          pf[i] = make_float2(fast_exp2(x.x), fast_exp2(x.y));          // 2^(S c - lse) * |scale|
        }
      }
      if (valid < kTile && idx < n_live) {   // padding rows of K meet dS = 0 in the product: finite, please (S has completed)
        if (r >= valid) split_zero_row<HD>(sm + Sm::k + (p % Sm::k_stages) * Sm::pair + (half * 64 + r) * 128, r, Sm::part);
        fence_proxy_async_smem();
      }
      ok = VSA_WARP_WAIT(bar(SQ_DP_FULL + g), ph);
      if (!ok) break;
      tc_fence_after();
      uint32_t pk[2][16];
      {
        uint32_t dv[2][32];
        tmem_ld(tmem_dp + 64 * g + lane_addr, dv[0]);
        tmem_ld(tmem_dp + 64 * g + lane_addr + 32, dv[1]);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(SQ_DP_EMPTY + g));
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const float2 y = mul2(pf[i], add2(word_pair(&dv[i >> 4][2 * (i & 15)]), d2));
          pk[i >> 4][i & 15] = Elem<elem_t>::pack(y.x, y.y);
        }
      }
      if (valid < kTile) {              // scores of padding keys come from whatever sits in K and V there
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          if (2 * i >= valid) pk[i >> 4][i & 15] = 0u;
          else if (2 * i + 1 >= valid) pk[i >> 4][i & 15] &= 0xffffu;
        }
      }
      ok = VSA_WARP_WAIT(bar(SQ_DS_EMPTY + g), ph ^ 1);
      if (!ok) break;
      tc_fence_after();
      tmem_st(tmem_ds + 32 * g + lane_addr, pk[0]);
      tmem_st(tmem_ds + 32 * g + lane_addr + 16, pk[1]);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(SQ_DS_FULL + g));
    }
    if (!ok && lane == 0) report_timeout(86);
    if (ok && n_pairs > 0) ok = VSA_WARP_WAIT(bar(SQ_ACC_FULL), 0);
    if (!ok && lane == 0) report_timeout(87);
    tc_fence_after();
    // a group finishes half of the head dims; every MMA is done, the rings are free
    constexpr int W = HD / 2;
    uint8_t* stage = sm + 2 * 64 * W * 4;
    split_add_halves<HD, W>(tmem_acc + lane_addr, ok && n_pairs > 0, sm + g * (64 * W * 4), stage, g * W, half, r, 1 + g,
                            [&](auto& ov, int c0) {
      if (scale < 0.f) {
#pragma unroll
        for (auto& w : ov) w ^= 0x80000000u;
      }
      if (r < rows_live) wide_add_mean(ov, s_mean + c0);
    });
    for (int i = (warp & 3) * 32 + lane; i < kTile * W / 8; i += 128) {
      const int rr = i / (W / 8), ch = g * (W / 8) + i % (W / 8);
      const long long drow = out_map.map == nullptr ? row0 + rr : raster_row(out_map, bh, (long long)qtile * kTile + rr);
      if (drow >= 0)
        *reinterpret_cast<uint4*>(dq + drow * HD + ch * 8) = *reinterpret_cast<const uint4*>(stage + rr * (HD * 2) + ((ch ^ (rr & 7)) << 4));
    }
  } else {
    registers_dec<64>();
    if (warp == 0) {          // K pairs: a lane per tile and 64 head dims
      for (int p = 0; p < n_pairs; ++p) {
        const int s = p % Sm::k_stages, idx = 2 * p + (lane & 1), h = lane >> 1;
        const int row = idx < n_live ? split_row(list[idx]) : (int)(BH * Lkv);       // outside the tensor: zeros
        ok = VSA_WARP_WAIT(bar(SQ_K_EMPTY + s), ((p / Sm::k_stages) & 1) ^ 1) &&
             (p != Sm::k_stages - 1 || VSA_WARP_WAIT2(bar(SQ_QT_FULL), 0, bar(SQ_DOT_FULL), 0));
        if (!ok) break;
        if (lane < 2 * kParts) {
          mbar_arrive_expect_tx(bar(SQ_K_FULL + s), kSlab);
          tma_load_2d(base + Sm::k + s * Sm::pair + h * Sm::part + (lane & 1) * kSlab, &map_k, h * 64, row, bar(SQ_K_FULL + s));
        }
        __syncwarp();
      }
      if (!ok && lane == 0) report_timeout(81);
    } else if (warp == 1) {   // V pairs
      for (int p = 0; p < n_pairs; ++p) {
        const int idx = 2 * p + (lane & 1), h = lane >> 1, i0 = p * kParts, i1 = i0 + kParts - 1, s = (i0 + h) % Sm::v_parts;
        const int row = idx < n_live ? split_row(list[idx]) : (int)(BH * Lkv);
        ok = VSA_WARP_WAIT2(bar(SQ_V_EMPTY + i0 % Sm::v_parts), ((i0 / Sm::v_parts) & 1) ^ 1, bar(SQ_V_EMPTY + i1 % Sm::v_parts),
                            ((i1 / Sm::v_parts) & 1) ^ 1);
        if (!ok) break;
        if (lane < 2 * kParts) {
          mbar_arrive_expect_tx(bar(SQ_V_FULL + s), kSlab);
          tma_load_2d(base + Sm::v + s * Sm::part + (lane & 1) * kSlab, &map_v, h * 64, row, bar(SQ_V_FULL + s));
        }
        __syncwarp();
      }
      if (!ok && lane == 0) report_timeout(82);
    } else if (warp == 2) {   // S = Q K^T
      ok = VSA_WARP_WAIT(bar(SQ_QT_FULL), 0);
      for (int p = 0; p < n_pairs && ok; ++p) {
        const int s = p % Sm::k_stages;
        ok = VSA_WARP_WAIT2(bar(SQ_K_FULL + s), (p / Sm::k_stages) & 1, bar(SQ_S_EMPTY), (p & 1) ^ 1);
        if (!ok) break;
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int h = 0; h < kParts; ++h)
            split_issue_scores_ts(tmem_s, tmem_q + 32 * h, base + Sm::k + s * Sm::pair + h * Sm::part, h > 0);
          mma_commit(bar(SQ_S_FULL + (p & 1)));
        }
        __syncwarp();
      }
      if (!ok && lane == 0) report_timeout(83);
    } else if (warp == 3) {   // dP = dO V^T
      ok = VSA_WARP_WAIT(bar(SQ_DOT_FULL), 0);
      for (int p = 0; p < n_pairs && ok; ++p) {
        const int i0 = p * kParts, i1 = i0 + kParts - 1, b = p & 1;
        ok = VSA_WARP_WAIT3(bar(SQ_V_FULL + i0 % Sm::v_parts), (i0 / Sm::v_parts) & 1, bar(SQ_V_FULL + i1 % Sm::v_parts),
                            (i1 / Sm::v_parts) & 1, bar(SQ_DP_EMPTY + b), ((p >> 1) & 1) ^ 1);
        if (!ok) break;
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int h = 0; h < kParts; ++h) {
            const int s = (i0 + h) % Sm::v_parts;
            split_issue_scores_ts(tmem_dp + 64 * b, tmem_do + 32 * h, base + Sm::v + s * Sm::part, h > 0);
            mma_commit(bar(SQ_V_EMPTY + s));
          }
          mma_commit(bar(SQ_DP_FULL + b));
        }
        __syncwarp();
      }
      if (!ok && lane == 0) report_timeout(84);
    } else if (warp == 12) {  // dQ += dS K
      for (int p = 0; p < n_pairs && ok; ++p) {
        const int s = p % Sm::k_stages, b = p & 1;
        ok = VSA_WARP_WAIT2(bar(SQ_K_FULL + s), (p / Sm::k_stages) & 1, bar(SQ_DS_FULL + b), (p >> 1) & 1);
        if (!ok) break;
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int h = 0; h < kParts; ++h)
            split_issue_product(tmem_acc + 64 * h, tmem_ds + 32 * b, base + Sm::k + s * Sm::pair + h * Sm::part, p > 0);
          mma_commit(bar(SQ_K_EMPTY + s));
          mma_commit(bar(SQ_DS_EMPTY + b));
        }
        __syncwarp();
      }
      if (ok && elect_one()) mma_commit(bar(SQ_ACC_FULL));
      __syncwarp();
      if (!ok && lane == 0) report_timeout(85);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 12) tmem_dealloc(tmem, kTmemCols);
}

template <int HD>
int launch_dq_split(const void* dout, const void* q, const void* k, const void* v, const void* out_s, const float* lse2,
                    const int32_t* selected, const int32_t* kv_sizes, float* delta, void* dq, int64_t BH, int64_t Lq,
                    int64_t Lkv, int be, int topk, float scale, cudaStream_t st, const void* dq_mean, const int32_t* q_sizes,
                    int64_t kv_shard, RasterMap out_map) {
  CUtensorMap mq, mdo, mk, mv;
  int rc;
  if ((rc = make_wide_map(&mq, q, BH * Lq, HD, kTile, "sparse dQ (q)"))) return rc;
  if ((rc = make_wide_map(&mdo, dout, BH * Lq, HD, kTile, "sparse dQ (dout)"))) return rc;
  if ((rc = make_wide_map(&mk, k, BH * Lkv, HD, kTile, "sparse dQ (k)"))) return rc;
  if ((rc = make_wide_map(&mv, v, BH * Lkv, HD, kTile, "sparse dQ (v)"))) return rc;
  const int smem = SqSmem<HD>::total + 1024;
  if ((rc = reserve_smem(sparse_dq_split_kernel<HD>, smem, "sparse dQ"))) return rc;
  sparse_dq_split_kernel<HD><<<dim3((unsigned)(Lq / kTile), (unsigned)BH), kSqThreads, smem, st>>>(
      mq, mdo, mk, mv, (const elem_t*)dout, (const elem_t*)out_s, lse2, selected, kv_sizes, delta, (elem_t*)dq,
      (const elem_t*)dq_mean, q_sizes, Lq, Lkv, kv_shard, be / kTile, topk, scale, out_map);
  return check_launch("sparse_dq_split_kernel");
}

// ------------------------------------------------------------------------------------------------------
// dK / dV: lanes = 64 key rows x parity of the query tile, columns = its 64 query rows
// ------------------------------------------------------------------------------------------------------
// One CTA per SM.  dK and dV (256 columns), S, dP (64 each), P, dS (32 each) and V (64) fill tensor memory, so K is read from
// shared memory by its products.  All eight elementwise warps share a pair, 32 scores a thread: what bounds the pass is how long a
// Q pair is held (load -> S -> P -> dS -> dK), three pairs being what fits, and two groups on alternate pairs hold it longer.
constexpr int kSkThreads = 512;
template <int HD>
struct SkSmem {
  static constexpr uint32_t part = 16384;
  static constexpr uint32_t pair = (HD / 64) * part;
  static constexpr int q_stages = 3, do_stages = 3;               // pairs
  static constexpr uint32_t k = 0;                                // resident K tile, [HD/64][64 rows][128 bytes]
  static constexpr uint32_t q = k + HD * 128;
  static constexpr uint32_t d_o = q + q_stages * pair;
  static constexpr uint32_t stats = d_o + do_stages * pair;       // per Q stage and tile: lse [64], delta [64]
  static constexpr uint32_t mean = stats + q_stages * 1024;        // float [2][HD]: what a live row receives from the pooled gradients
  static constexpr uint32_t bars = mean + 2 * HD * 4;
  static constexpr uint32_t misc = bars + 32 * 8;
  static constexpr uint32_t total = misc + 32;
};
static_assert(SkSmem<128>::total + 1024 <= 232448, "shared memory of the split dK/dV pass");
enum SkBar { SK_K_FULL = 0, SK_V_FULL = 1, SK_VT_FULL = 2, SK_Q_FULL = 3, SK_Q_EMPTY = 7, SK_DO_FULL = 11, SK_DO_EMPTY = 14,
             SK_S_FULL = 17, SK_S_EMPTY, SK_DP_FULL, SK_DP_EMPTY, SK_P_FULL, SK_P_EMPTY, SK_DS_FULL, SK_DS_EMPTY, SK_ACC_FULL };

template <int HD>
__global__ void __launch_bounds__(kSkThreads, 1)
sparse_dkdv_split_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_do,
                         const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                         const float* __restrict__ lse2, const float* __restrict__ delta, const int32_t* __restrict__ counts,
                         const int32_t* __restrict__ offsets, const int32_t* __restrict__ inverse,
                         const int32_t* __restrict__ kv_sizes, elem_t* __restrict__ dk, elem_t* __restrict__ dv,
                         const elem_t* __restrict__ mean_grad_k, const elem_t* __restrict__ mean_grad_v, long long Lq,
                         long long Lkv, long long kv_shard, int sub, int topk, float scale, RasterMap out_map) {
  using Sm = SkSmem<HD>;
  constexpr int kParts = HD / 64;
  constexpr uint32_t kStage = Sm::d_o + (Sm::do_stages - 1) * Sm::pair;      // V on its way to tensor memory, in the last dO stage
  extern __shared__ uint8_t smem_raw[];
  if (*(volatile int*)&g_device_status != 0) return;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* sm = smem_raw + (base - smem_u32(smem_raw));
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int ktile = blockIdx.x;
  const long long bh = blockIdx.y, BH = gridDim.y;
  const int be = kTile * sub, Kb = (int)(Lkv / be), Qb = (int)(Lq / be);
  const int kvb = ktile / sub;
  const int size = kv_sizes[kvb];
  int valid = size - (ktile % sub) * kTile;
  valid = valid < 0 ? 0 : (valid > kTile ? kTile : valid);
  const long long krow0 = kv_tensor_row(bh, BH, (long long)ktile * kTile, kv_shard);
  const int32_t* inv = inverse + bh * (long long)Qb * topk + offsets[bh * Kb + kvb];
  const int n_tiles = valid > 0 ? counts[bh * Kb + kvb] * sub : 0, n_pairs = (n_tiles + 1) >> 1;
  const float c = scale * kLog2e;
  const float mean_inv = 1.f / (float)(size > 1 ? size : 1);
  const long long mean_off = (bh * Kb + kvb) * (long long)HD;

  if (n_tiles == 0) {   // nobody selected this tile, or it is all padding: pooled gradient only
    for (int i = tid; i < kTile * HD / 8; i += kSkThreads) {
      const int rr = i / (HD / 8), ch = i % (HD / 8);
      const long long drow = out_map.map == nullptr ? krow0 + rr : raster_row(out_map, bh, (long long)ktile * kTile + rr);
      if (drow < 0) continue;
      uint4 ok4 = make_uint4(0, 0, 0, 0), ov4 = make_uint4(0, 0, 0, 0);
      if (mean_grad_k != nullptr && rr < valid) {
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
  auto tile_row = [&](int i) -> long long { return bh * Lq + (long long)inv[i / sub] * be + (i % sub) * kTile; };

  if (tid == 0) {
    mbar_init(bar(SK_K_FULL), 1);
    mbar_init(bar(SK_V_FULL), 1);
    mbar_init(bar(SK_VT_FULL), 4 * kParts);
    for (int i = 0; i < Sm::q_stages; ++i) {
      mbar_init(bar(SK_Q_FULL + i), 2 * kParts + 32);      // the boxes' lanes and 32 lanes' copies of the statistics
      mbar_init(bar(SK_Q_EMPTY + i), 1);
    }
    for (int i = 0; i < Sm::do_stages; ++i) {
      mbar_init(bar(SK_DO_FULL + i), 2 * kParts);
      mbar_init(bar(SK_DO_EMPTY + i), 2);                  // read by the dP products of one issuer and the dV products of another
    }
    mbar_init(bar(SK_S_FULL), 1);
    mbar_init(bar(SK_S_EMPTY), 8);
    mbar_init(bar(SK_DP_FULL), 1);
    mbar_init(bar(SK_DP_EMPTY), 8);
    mbar_init(bar(SK_P_FULL), 8);
    mbar_init(bar(SK_P_EMPTY), 1);
    mbar_init(bar(SK_DS_FULL), 8);
    mbar_init(bar(SK_DS_EMPTY), 1);
    mbar_init(bar(SK_ACC_FULL), 2);
    fence_barrier_init();
    tma_prefetch_desc(&map_q);
    tma_prefetch_desc(&map_do);
    mbar_arrive_expect_tx(bar(SK_K_FULL), HD * 128);
    wide_load<HD>(base + Sm::k, &map_k, (int)krow0, kSlab, bar(SK_K_FULL));
    mbar_arrive_expect_tx(bar(SK_V_FULL), HD * 128);
    wide_load<HD>(base + kStage, &map_v, (int)krow0, kSlab, bar(SK_V_FULL));
  }
  if (warp == 12) {
    tmem_alloc(base + Sm::misc, kTmemCols);
    tmem_relinquish();
  }
  float* s_mean = reinterpret_cast<float*>(sm + Sm::mean);
  if (mean_grad_k != nullptr && tid < 2 * HD)
    s_mean[tid] = Elem<elem_t>::to(tid < HD ? mean_grad_k[mean_off + tid] : mean_grad_v[mean_off + tid - HD]) * mean_inv;
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = misc[0];
  const uint32_t tmem_dk = tmem, tmem_dv = tmem + 128, tmem_s = tmem + 256, tmem_dp = tmem + 320, tmem_p = tmem + 384,
                 tmem_ds = tmem + 416, tmem_v = tmem + 448;
  bool ok = true;

  if (warp >= 4 && warp < 12) {
    const int quarter = warp & 3, half = quarter >> 1, r = (quarter & 1) * 32 + lane, g = (warp - 4) >> 2, c0 = 32 * g;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const bool live = r < valid;
    if (g < kParts) {
      ok = VSA_WARP_WAIT(bar(SK_V_FULL), 0);
      split_store_row(tmem_v + 32 * g + lane_addr, sm + kStage + g * kSlab, r);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(SK_VT_FULL));
    }
    const float2 c2 = make_float2(-c, -c), m1 = make_float2(-1.f, -1.f);
    for (int p = 0; p < n_pairs && ok; ++p) {
      const int s = p % Sm::q_stages;
      const uint32_t ph = p & 1;
      ok = VSA_WARP_WAIT2(bar(SK_Q_FULL + s), (p / Sm::q_stages) & 1, bar(SK_S_FULL), ph);
      if (!ok) break;
      tc_fence_after();
      const float4* s_lse = reinterpret_cast<const float4*>(sm + Sm::stats + s * 1024 + half * 512 + c0 * 4);
      float2 pf[16];
      uint32_t pk[16];
      {
        uint32_t sv[32];
        tmem_ld(tmem_s + lane_addr + c0, sv);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(SK_S_EMPTY));
#pragma unroll
        for (int i = 0; i < 8; ++i) {
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
      }
      ok = VSA_WARP_WAIT(bar(SK_P_EMPTY), ph ^ 1);
      if (!ok) break;
      tc_fence_after();
      tmem_st(tmem_p + lane_addr + 16 * g, pk);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(SK_P_FULL));
      ok = VSA_WARP_WAIT(bar(SK_DP_FULL), ph);
      if (!ok) break;
      tc_fence_after();
      {
        uint32_t dvv[32];
        tmem_ld(tmem_dp + lane_addr + c0, dvv);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(SK_DP_EMPTY));
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4 d4 = s_lse[16 + i];       // delta: 64 floats behind the statistics
          const float2 x = mul2(pf[2 * i], fma2(word_pair(dvv + 4 * i), m1, make_float2(d4.x, d4.y)));      // -dS
          const float2 y = mul2(pf[2 * i + 1], fma2(word_pair(dvv + 4 * i + 2), m1, make_float2(d4.z, d4.w)));
          pk[2 * i] = live ? Elem<elem_t>::pack(x.x, x.y) : 0u;
          pk[2 * i + 1] = live ? Elem<elem_t>::pack(y.x, y.y) : 0u;
        }
      }
      ok = VSA_WARP_WAIT(bar(SK_DS_EMPTY), ph ^ 1);
      if (!ok) break;
      tc_fence_after();
      tmem_st(tmem_ds + lane_addr + 16 * g, pk);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(SK_DS_FULL));
    }
    if (!ok && lane == 0) report_timeout(96);
    if (ok) ok = VSA_WARP_WAIT(bar(SK_ACC_FULL), 0);
    if (!ok && lane == 0) report_timeout(97);
    tc_fence_after();
    // group 0 finishes dK, group 1 dV; every MMA is done, the rings are free
    uint8_t* mine = sm + Sm::q + g * (64 * HD * 6);
    uint8_t* stage = mine + 64 * HD * 4;
    split_add_halves<HD, HD>((g == 0 ? tmem_dk : tmem_dv) + lane_addr, ok, mine, stage, 0, half, r, 1 + g, [&](auto& ov, int col) {
      if (g == 0) {
#pragma unroll
        for (auto& w : ov) w = __float_as_uint(__uint_as_float(w) * -scale);      // the products summed -dS
      }
      if (mean_grad_k != nullptr && live) wide_add_mean(ov, s_mean + g * HD + col);
    });
    elem_t* dst = g == 0 ? dk : dv;
    for (int i = (warp & 3) * 32 + lane; i < kTile * HD / 8; i += 128) {
      const int rr = i / (HD / 8), ch = i % (HD / 8);
      const long long drow = out_map.map == nullptr ? krow0 + rr : raster_row(out_map, bh, (long long)ktile * kTile + rr);
      if (drow >= 0) *reinterpret_cast<uint4*>(dst + drow * HD + ch * 8) = *reinterpret_cast<const uint4*>(stage + rr * (HD * 2) + ((ch ^ (rr & 7)) << 4));
    }
  } else if (warp == 0) {   // Q pairs with the statistics of their rows; a lane per tile and 64 head dims
    for (int p = 0; p < n_pairs; ++p) {
      const int s = p % Sm::q_stages, h = lane >> 1;
      // The second half of an odd tail is the first one's Q again, with statistics that make P = 2^-inf = 0 of any score that the
      // first half has a probability for; zero rows would make NaN of an infinite key.  Its dO lies outside the tensor, i.e. is zero.
      const bool second = 2 * p + 1 < n_tiles;
      const long long row_a = tile_row(2 * p), row_b = second ? tile_row(2 * p + 1) : row_a;
      ok = VSA_WARP_WAIT(bar(SK_Q_EMPTY + s), ((p / Sm::q_stages) & 1) ^ 1);
      if (!ok) break;
      const uint32_t st = base + Sm::stats + s * 1024 + lane * 4;
      cp_async4(st, lse2 + row_a + lane);
      cp_async4(st + 128, lse2 + row_a + 32 + lane);
      cp_async4(st + 256, delta + row_a + lane);
      cp_async4(st + 384, delta + row_a + 32 + lane);
      if (second) {
        cp_async4(st + 512, lse2 + row_b + lane);
        cp_async4(st + 640, lse2 + row_b + 32 + lane);
        cp_async4(st + 768, delta + row_b + lane);
        cp_async4(st + 896, delta + row_b + 32 + lane);
      } else {
        float* f = reinterpret_cast<float*>(sm + Sm::stats + s * 1024 + 512);
        f[lane] = f[32 + lane] = INFINITY;
        f[64 + lane] = f[96 + lane] = 0.f;
        __syncwarp();                                      // ordered by the arrivals of the boxes' lanes
      }
      cp_async_arrive_noinc(bar(SK_Q_FULL + s));
      if (lane < 2 * kParts) {
        mbar_arrive_expect_tx(bar(SK_Q_FULL + s), kSlab);
        tma_load_2d(base + Sm::q + s * Sm::pair + h * Sm::part + (lane & 1) * kSlab, &map_q, h * 64, (int)(lane & 1 ? row_b : row_a), bar(SK_Q_FULL + s));
      }
      __syncwarp();
    }
    if (!ok && lane == 0) report_timeout(91);
  } else if (warp == 1) {   // dO pairs
    for (int p = 0; p < n_pairs; ++p) {
      const int s = p % Sm::do_stages, h = lane >> 1, i = 2 * p + (lane & 1);
      const int row = (int)(i < n_tiles ? tile_row(i) : BH * Lq);
      ok = VSA_WARP_WAIT(bar(SK_DO_EMPTY + s), ((p / Sm::do_stages) & 1) ^ 1) && (p != Sm::do_stages - 1 || VSA_WARP_WAIT(bar(SK_VT_FULL), 0));
      if (!ok) break;
      if (lane < 2 * kParts) {
        mbar_arrive_expect_tx(bar(SK_DO_FULL + s), kSlab);
        tma_load_2d(base + Sm::d_o + s * Sm::pair + h * Sm::part + (lane & 1) * kSlab, &map_do, h * 64, row, bar(SK_DO_FULL + s));
      }
      __syncwarp();
    }
    if (!ok && lane == 0) report_timeout(92);
  } else if (warp == 2) {   // S^T = K Q^T
    constexpr uint32_t idesc = instr_desc(64, 128, 0, 0, kInFmt);
    constexpr uint32_t hi = desc_hi(1024);
    const uint32_t a0 = desc_lo(base + Sm::k, 16);
    ok = VSA_WARP_WAIT(bar(SK_K_FULL), 0);
    for (int p = 0; p < n_pairs && ok; ++p) {
      const int s = p % Sm::q_stages;
      ok = VSA_WARP_WAIT2(bar(SK_Q_FULL + s), (p / Sm::q_stages) & 1, bar(SK_S_EMPTY), (p & 1) ^ 1);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
        const uint32_t b0 = desc_lo(base + Sm::q + s * Sm::pair, 16);
#pragma unroll
        for (int ks = 0; ks < HD / 16; ++ks)
          mma_ws_ss(tmem_s, desc_pack(a0 + (uint32_t)(((ks >> 2) * kSlab + (ks & 3) * 32) >> 4), hi),
                    desc_pack(b0 + (uint32_t)(((ks >> 2) * Sm::part + (ks & 3) * 32) >> 4), hi), idesc, ks > 0 ? 1u : 0u);
        mma_commit(bar(SK_S_FULL));
      }
      __syncwarp();
    }
    if (!ok && lane == 0) report_timeout(93);
  } else if (warp == 3) {   // dP^T = V dO^T
    ok = VSA_WARP_WAIT(bar(SK_VT_FULL), 0);
    for (int p = 0; p < n_pairs && ok; ++p) {
      const int s = p % Sm::do_stages;
      ok = VSA_WARP_WAIT2(bar(SK_DO_FULL + s), (p / Sm::do_stages) & 1, bar(SK_DP_EMPTY), (p & 1) ^ 1);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int h = 0; h < kParts; ++h)
          split_issue_scores_ts(tmem_dp, tmem_v + 32 * h, base + Sm::d_o + s * Sm::pair + h * Sm::part, h > 0);
        mma_commit(bar(SK_DO_EMPTY + s));
        mma_commit(bar(SK_DP_FULL));
      }
      __syncwarp();
    }
    if (!ok && lane == 0) report_timeout(94);
  } else if (warp == 12) {  // dV += P^T dO
    for (int p = 0; p < n_pairs && ok; ++p) {
      const int s = p % Sm::do_stages;
      ok = VSA_WARP_WAIT2(bar(SK_DO_FULL + s), (p / Sm::do_stages) & 1, bar(SK_P_FULL), p & 1);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int h = 0; h < kParts; ++h)
          split_issue_product(tmem_dv + 64 * h, tmem_p, base + Sm::d_o + s * Sm::pair + h * Sm::part, p > 0);
        mma_commit(bar(SK_DO_EMPTY + s));
        mma_commit(bar(SK_P_EMPTY));
      }
      __syncwarp();
    }
    if (ok && elect_one()) mma_commit(bar(SK_ACC_FULL));
    __syncwarp();
    if (!ok && lane == 0) report_timeout(95);
  } else if (warp == 13) {  // dK += dS^T Q
    for (int p = 0; p < n_pairs && ok; ++p) {
      const int s = p % Sm::q_stages;
      ok = VSA_WARP_WAIT2(bar(SK_Q_FULL + s), (p / Sm::q_stages) & 1, bar(SK_DS_FULL), p & 1);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int h = 0; h < kParts; ++h)
          split_issue_product(tmem_dk + 64 * h, tmem_ds, base + Sm::q + s * Sm::pair + h * Sm::part, p > 0);
        mma_commit(bar(SK_Q_EMPTY + s));
        mma_commit(bar(SK_DS_EMPTY));
      }
      __syncwarp();
    }
    if (ok && elect_one()) mma_commit(bar(SK_ACC_FULL));
    __syncwarp();
    if (!ok && lane == 0) report_timeout(98);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 12) tmem_dealloc(tmem, kTmemCols);
}

template <int HD>
int launch_dkdv_split(const void* dout, const void* q, const void* k, const void* v, const float* lse2, const float* delta,
                      const int32_t* counts, const int32_t* offsets, const int32_t* inverse, const int32_t* kv_sizes, void* dk,
                      void* dv, int64_t BH, int64_t Lq, int64_t Lkv, int be, int topk, float scale, cudaStream_t st,
                      const void* dk_mean, const void* dv_mean, int64_t kv_shard, RasterMap out_map) {
  CUtensorMap mq, mdo, mk, mv;
  int rc;
  if ((rc = make_wide_map(&mq, q, BH * Lq, HD, kTile, "sparse dK/dV (q)"))) return rc;
  if ((rc = make_wide_map(&mdo, dout, BH * Lq, HD, kTile, "sparse dK/dV (dout)"))) return rc;
  if ((rc = make_wide_map(&mk, k, BH * Lkv, HD, kTile, "sparse dK/dV (k)"))) return rc;
  if ((rc = make_wide_map(&mv, v, BH * Lkv, HD, kTile, "sparse dK/dV (v)"))) return rc;
  const int smem = SkSmem<HD>::total + 1024;
  if ((rc = reserve_smem(sparse_dkdv_split_kernel<HD>, smem, "sparse dK/dV"))) return rc;
  sparse_dkdv_split_kernel<HD><<<dim3((unsigned)(Lkv / kTile), (unsigned)BH), kSkThreads, smem, st>>>(
      mq, mdo, mk, mv, lse2, delta, counts, offsets, inverse, kv_sizes, (elem_t*)dk, (elem_t*)dv, (const elem_t*)dk_mean,
      (const elem_t*)dv_mean, Lq, Lkv, kv_shard, be / kTile, topk, scale, out_map);
  return check_launch("sparse_dkdv_split_kernel");
}
