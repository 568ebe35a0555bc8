// The backward that forms dS once (opt-in) on the Blackwell tensor path.  Included by sparse_umma_typed.inl.
//
// The key-owned pass works on transposed, 128-row products, per PAIR of query tiles that selected this key tile (lanes = 128 query
// rows, columns = 64 key tokens):
//      S  = Q2 K^T                   dP = dO2 V^T
//      P  = 2^(S c - lse[row]),      dS = P * (dP - delta[row])   (elementwise, statistics per LANE)
//      dV^T [128 dims x 64 keys] += dO2^T P          dK^T += Q2^T dS          (dK^T * scale at the end)
// P / dS are written by the thread that owns their row, once, as a swizzled 128-byte shared-memory row (N-major B operand), and dS
// goes to memory from the same registers; a query-owned pass then multiplies it by K.  Roles of the first: warp 0 and 1 = TMA
// producers (four lanes, one box each), warp 2 = issuer of the S MMAs, warp 3 = issuer of the gradient MMAs, warps 4-11 = elementwise
// (a TMEM lane quarter x 32 of the 64 columns each), warp 12 = issuer of the dP MMAs.

// Every operand byte is read by an MMA once or twice per pair, close to the shared-memory bandwidth limit; eight wider elementwise
// warps disturb that pipe less than sixteen narrow ones.
constexpr int kBwCols = 32;
constexpr int kBwWarps = 4 * (64 / kBwCols);
constexpr int kBwEwThreads = 32 * kBwWarps;
constexpr int kBwdThreads = 128 + kBwEwThreads + 32;   // ... plus the dP issuer, the last warp
constexpr int kDpWarp = 4 + kBwWarps;

// ------------------------------------------------------------------------------------------------------
// dK / dV
// ------------------------------------------------------------------------------------------------------
constexpr int kDkBufs = 2;     // (S, dP) accumulator pairs in flight: 2 x 128 columns, then dK^T and dV^T
// A Q2 pair stays in shared memory from its score MMA (the first of a pair) to its dK MMA (the last), across the
// whole elementwise stage, and a reload takes ~1500 cycles on top, so Q2 gets three stages; dO2 gets two and is
// released as early as the data flow allows: S and dP signal the elementwise warps separately, the warps turn S
// into P while the dP MMAs still run and publish P before they look at dP, and dV^T (which needs only P) is
// issued and committed on its own, ahead of dS and dK^T.  P and dS have one buffer each (written by pair p+1 only
// after the MMA of pair p that reads them has completed, checked right before the stores).
constexpr int kDkQStages = 3;
struct DkSmem {
  static constexpr uint32_t k = 0;                                // 16 KB
  static constexpr uint32_t v = k + 2 * kSlab;                    // 16 KB
  static constexpr uint32_t q = v + 2 * kSlab;                    // kDkQStages x 32 KB  (pairs of query tiles)
  static constexpr uint32_t d_o = q + kDkQStages * kPairBytes;    // 2 x 32 KB
  static constexpr uint32_t p = d_o + 2 * kPairBytes;             // 16 KB
  static constexpr uint32_t ds = p + kPairHalf;                   // 16 KB
  static constexpr uint32_t bars = ds + kPairHalf;
  static constexpr uint32_t misc = bars + 32 * 8;
  static constexpr uint32_t total = misc + 64;
};
enum DkBar { DK_KV_FULL = 0, DK_Q_FULL = 1, DK_DO_FULL = 4, DK_Q_EMPTY = 6, DK_DO_EMPTY = 9, DK_P_FULL = 11,
             DK_P_EMPTY = 12, DK_DS_FULL = 13, DK_DS_EMPTY = 14, DK_ACC_FULL = 15, DK_S_FULL = 16,
             DK_DP_FULL = 16 + kDkBufs, DK_S_EMPTY = 16 + 2 * kDkBufs };

// The rows of `inverse` hold packed edges (query block << kEdgeSlotBits | slot in that block's route)
// and every dS tile (64 query rows x 64 key tokens, 8 KB) is written to `ds_ws` at tile index
// ((edge * SUB + query sub-tile) * SUB + key sub-tile), edge = (slice * Qb + query block) * topk + slot, for the
// dQ pass that only multiplies it by K (sparse_dq_from_ds_kernel below) instead of recomputing S and dP.
// Layout of a stored tile: [8 chunks of 8 key tokens][64 query rows][16 bytes] -- the order in which the rows'
// owner threads hold it (a warp's 32 rows of one chunk are 512 contiguous bytes: fully coalesced stores straight
// from registers), and at the same time the un-swizzled K-major operand layout of tcgen05 (8 rows x 16 bytes per
// core matrix), so the dQ pass copies the 8 KB verbatim into shared memory and multiplies.
constexpr int kEdgeSlotBits = 11;
template <int SUB>
__global__ void __launch_bounds__(kBwdThreads, 1)
sparse_dkdv_ds_umma_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_do,
                        const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                        const float* __restrict__ lse2, const float* __restrict__ delta,
                        const int32_t* __restrict__ counts, const int32_t* __restrict__ offsets,
                        const int32_t* __restrict__ inverse, const int32_t* __restrict__ kv_sizes,
                        elem_t* __restrict__ dk, elem_t* __restrict__ dv, const elem_t* __restrict__ mean_grad_k,
                        const elem_t* __restrict__ mean_grad_v, elem_t* __restrict__ ds_ws, long long Lq, long long Lkv,
                        long long kv_shard, int topk, float scale, RasterMap out_map) {
  extern __shared__ uint8_t smem_raw[];
  if (*(volatile int*)&g_device_status != 0) return;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* sm = smem_raw + (base - smem_u32(smem_raw));
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int ktile = blockIdx.x;
  const long long bh = blockIdx.y;
  const int Kb = (int)(Lkv / (kTile * SUB)), Qb = (int)(Lq / (kTile * SUB));
  const int kvb = ktile / SUB, sub = ktile % SUB;
  int valid = kv_sizes[kvb] - sub * kTile;
  valid = valid < 0 ? 0 : (valid > kTile ? kTile : valid);
  const long long krow0 = kv_tensor_row(bh, gridDim.y, (long long)ktile * kTile, kv_shard);   // K, V, dK, dV rows of this tile
  const int cnt = counts[bh * Kb + kvb];
  const int32_t* inv = inverse + bh * (long long)Qb * topk + offsets[bh * Kb + kvb];
  const int n_tiles = valid > 0 ? cnt * SUB : 0;
  const int n_pairs = (n_tiles + 1) >> 1;
  const float c = scale * kLog2e;
  const long long q_row_base = bh * Lq;

  // block-mean backward folded in (optional): key row r of the block also receives dmean[block] / max(size, 1)
  // while r < size (vsa/fused_common.py:62-103 of the reference)
  const float mean_inv = 1.f / (float)(kv_sizes[kvb] > 1 ? kv_sizes[kvb] : 1);
  const long long mean_off = (bh * Kb + kvb) * (long long)kD;
  if (n_pairs == 0) {   // nobody selected this tile, or it is all padding: no fine gradient, no pipeline
    for (int i = tid; i < 1024; i += (int)blockDim.x) {
      const long long drow = out_map.map == nullptr ? krow0 + (i >> 4) : raster_row(out_map, bh, (long long)ktile * kTile + (i >> 4));
      if (drow < 0) continue;
      uint4 ok4 = make_uint4(0, 0, 0, 0), ov4 = make_uint4(0, 0, 0, 0);
      if (mean_grad_k != nullptr && (i >> 4) < valid) {     // 16 chunks of eight dims per row
        elem_t* ek = reinterpret_cast<elem_t*>(&ok4);
        elem_t* ev = reinterpret_cast<elem_t*>(&ov4);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          ek[e] = Elem<elem_t>::from(Elem<elem_t>::to(mean_grad_k[mean_off + (i & 15) * 8 + e]) * mean_inv);
          ev[e] = Elem<elem_t>::from(Elem<elem_t>::to(mean_grad_v[mean_off + (i & 15) * 8 + e]) * mean_inv);
        }
      }
      *reinterpret_cast<uint4*>(dk + drow * kD + (i & 15) * 8) = ok4;
      *reinterpret_cast<uint4*>(dv + drow * kD + (i & 15) * 8) = ov4;
    }
    return;
  }
  volatile uint32_t* misc = reinterpret_cast<volatile uint32_t*>(sm + DkSmem::misc);
  auto bar = [&](int i) -> uint32_t { return base + DkSmem::bars + 8u * i; };
  // row (inside this batch-head slice) of the i-th query tile that selected this key block
  auto tile_row = [&](int i) -> int {
    const int e = inv[i / SUB];
    return (e >> kEdgeSlotBits) * (kTile * SUB) + (i % SUB) * kTile;
  };
  // index of the dS tile of the i-th in-edge query tile
  auto ds_tile = [&](int i) -> long long {
    const int e = inv[i / SUB];
    const long long edge = (bh * Qb + (e >> kEdgeSlotBits)) * (long long)topk + (e & ((1 << kEdgeSlotBits) - 1));
    return (edge * SUB + (i % SUB)) * SUB + sub;
  };

  if (tid == 0) {
    mbar_init(bar(DK_KV_FULL), 1);
    for (int i = 0; i < kDkQStages; ++i) {
      mbar_init(bar(DK_Q_FULL + i), 4);
      mbar_init(bar(DK_Q_EMPTY + i), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar(DK_DO_FULL + i), 4);
      mbar_init(bar(DK_DO_EMPTY + i), 2);    // read by the dP MMAs of one issuer and the dV^T MMAs of the other
    }
    mbar_init(bar(DK_P_FULL), kBwWarps);
    mbar_init(bar(DK_P_EMPTY), 1);
    mbar_init(bar(DK_DS_FULL), kBwWarps);
    mbar_init(bar(DK_DS_EMPTY), 1);
    for (int i = 0; i < kDkBufs; ++i) {
      mbar_init(bar(DK_S_FULL + i), 1);
      mbar_init(bar(DK_DP_FULL + i), 1);
      mbar_init(bar(DK_S_EMPTY + i), kBwWarps);
    }
    mbar_init(bar(DK_ACC_FULL), 1);
    fence_barrier_init();
    tma_prefetch_desc(&map_q);
    tma_prefetch_desc(&map_do);
    // the tile's own K and V, resident for the whole CTA: in flight before anything else
    mbar_arrive_expect_tx(bar(DK_KV_FULL), 4 * kSlab);
    tma_load_2d(base + DkSmem::k, &map_k, 0, (int)krow0, bar(DK_KV_FULL));
    tma_load_2d(base + DkSmem::k + kSlab, &map_k, 64, (int)krow0, bar(DK_KV_FULL));
    tma_load_2d(base + DkSmem::v, &map_v, 0, (int)krow0, bar(DK_KV_FULL));
    tma_load_2d(base + DkSmem::v + kSlab, &map_v, 64, (int)krow0, bar(DK_KV_FULL));
  }
  if (warp == 1) {
    tmem_alloc(base + DkSmem::misc, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = misc[0];
  const uint32_t tmem_dk = tmem + 128 * kDkBufs, tmem_dv = tmem_dk + 64;
  bool ok = true;

  if (warp == 0 || warp == 1) {
    const bool is_q = warp == 0;
    const int which = lane & 1, dhalf = (lane >> 1) & 1;
    const CUtensorMap* map = is_q ? &map_q : &map_do;
    const int full0 = is_q ? DK_Q_FULL : DK_DO_FULL, empty0 = is_q ? DK_Q_EMPTY : DK_DO_EMPTY;
    const uint32_t ring = base + (is_q ? DkSmem::q : DkSmem::d_o);
    const int depth = is_q ? kDkQStages : 2;
    for (int p = 0; p < n_pairs; ++p) {
      const int s = p % depth;
      const uint32_t ph = (p / depth) & 1;
      int idx = 2 * p + which;
      if (idx >= n_tiles) idx = 2 * p;                  // odd tail: repeat the tile (its rows are masked)
      const int row = (int)(q_row_base + tile_row(idx));
      ok = VSA_WARP_WAIT(bar(empty0 + s), ph ^ 1);
      if (!ok) break;
      if (lane < 4) {
        mbar_arrive_expect_tx(bar(full0 + s), kSlab);
        tma_load_2d(ring + s * kPairBytes + dhalf * kPairHalf + which * kSlab, map, dhalf * 64, row, bar(full0 + s));
      }
    }
    if (!ok && lane == 0) report_timeout(21);
  } else if (warp == 2) {
    // scores: S = Q2 K^T
    ok = VSA_WARP_WAIT(bar(DK_KV_FULL), 0);
    for (int p = 0; p < n_pairs && ok; ++p) {
      const int qs = p % kDkQStages, b = p % kDkBufs;
      ok = VSA_WARP_WAIT(bar(DK_Q_FULL + qs), (p / kDkQStages) & 1) &&
           VSA_WARP_WAIT(bar(DK_S_EMPTY + b), ((p / kDkBufs) & 1) ^ 1);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
        issue_kmajor(tmem + b * 128, base + DkSmem::q + qs * kPairBytes, base + DkSmem::k);
        mma_commit(bar(DK_S_FULL + b));
      }
      __syncwarp();
    }
    if (!ok && lane == 0) report_timeout(22);
  } else if (warp == kDpWarp) {
    // dP = dO2 V^T from a thread of its own: dO2 has two stages only and must not hold back the next S
    ok = VSA_WARP_WAIT(bar(DK_KV_FULL), 0);
    for (int p = 0; p < n_pairs && ok; ++p) {
      const int s = p & 1, b = p % kDkBufs;
      ok = VSA_WARP_WAIT(bar(DK_DO_FULL + s), (p >> 1) & 1) && VSA_WARP_WAIT(bar(DK_S_EMPTY + b), ((p / kDkBufs) & 1) ^ 1);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
        issue_kmajor(tmem + b * 128 + 64, base + DkSmem::d_o + s * kPairBytes, base + DkSmem::v);
        mma_commit(bar(DK_DP_FULL + b));
        mma_commit(bar(DK_DO_EMPTY + s));      // a commit covers the MMAs of the committing thread only: dP here, dV^T there
      }
      __syncwarp();
    }
    if (!ok && lane == 0) report_timeout(26);
  } else if (warp == 3) {
    // dV^T += dO2^T P and dK^T += Q2^T dS
    for (int p = 0; p < n_pairs && ok; ++p) {
      const int qs = p % kDkQStages, s = p & 1;
      const uint32_t ph = (p >> 1) & 1;
      ok = VSA_WARP_WAIT(bar(DK_DO_FULL + s), ph) && VSA_WARP_WAIT(bar(DK_P_FULL), p & 1);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
        issue_mnmajor(tmem_dv, base + DkSmem::d_o + s * kPairBytes, base + DkSmem::p, p > 0);
        mma_commit(bar(DK_P_EMPTY));
        mma_commit(bar(DK_DO_EMPTY + s));      // second of two arrivals: the other issuer commits its dP reads of the stage
      }
      __syncwarp();
      ok = VSA_WARP_WAIT(bar(DK_Q_FULL + qs), (p / kDkQStages) & 1) && VSA_WARP_WAIT(bar(DK_DS_FULL), p & 1);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
        issue_mnmajor(tmem_dk, base + DkSmem::q + qs * kPairBytes, base + DkSmem::ds, p > 0);
        mma_commit(bar(DK_Q_EMPTY + qs));
        mma_commit(bar(DK_DS_EMPTY));
      }
      __syncwarp();
    }
    if (ok && elect_one()) mma_commit(bar(DK_ACC_FULL));
    __syncwarp();
    if (!ok && lane == 0) report_timeout(23);
  } else {
    // elementwise warps: lane t = query row of the pair, kBwCols of the 64 key tokens (columns c0..)
    const float2 c2 = make_float2(c, c);
    const int quarter = warp & 3;
    const int cg = (warp - 4) >> 2;
    const int c0 = cg * kBwCols;
    const int t = quarter * 32 + lane;
    const int half = t >> 6, r = t & 63;
    const int st = tid - 128;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const bool ragged = valid < kTile;      // same for the whole CTA: key columns >= valid are padding
    // statistics of this lane's query row, fetched one pair ahead of their use.  A row that does not exist (the
    // repeated tile of an odd tail) gets lse = +inf, i.e. P = 0 exactly, and delta = 0, so dS = 0 * finite = 0.
    float lse_n = INFINITY, dl_n = 0.f;
    long long dst_n = -1;                    // tile index of this lane's dS row in the coming pair
    if (half < n_tiles) {
      const long long row = q_row_base + tile_row(half) + r;
      lse_n = lse2[row];
      dl_n = delta[row];
      dst_n = ds_tile(half);
    }
    uint8_t* prow = sm + DkSmem::p + t * 128;
    uint8_t* grow = sm + DkSmem::ds + t * 128;
    for (int p = 0; p < n_pairs && ok; ++p) {
      const int b = p % kDkBufs;
      const float lse = lse_n, dl = dl_n;
      const long long dst = dst_n;
      {
        const int nidx = 2 * (p + 1) + half;
        lse_n = INFINITY;
        dl_n = 0.f;
        dst_n = -1;
        if (nidx < n_tiles) {
          const long long row = q_row_base + tile_row(nidx) + r;
          lse_n = lse2[row];
          dl_n = delta[row];
          dst_n = ds_tile(nidx);
        }
      }
      // ---- P from S, published before dP is even looked at (the dP MMAs are still running)
      bool p_free, ds_free;       // looked at together with the blocking waits: usually already true
      ok = VSA_WARP_WAIT_TEST(bar(DK_S_FULL + b), (p / kDkBufs) & 1, bar(DK_P_EMPTY), (p & 1) ^ 1, &p_free);
      if (!ok) break;
      tc_fence_after();
      uint32_t sv[kBwCols];
      tmem_ld(tmem + b * 128 + lane_addr + c0, sv);
      tmem_ld_wait();
      float pf[kBwCols];
      if (!ragged) {
#pragma unroll
        for (int j = 0; j < kBwCols / 2; ++j) {
          const float2 x = fma2(word_pair(sv + 2 * j), c2, make_float2(-lse, -lse));
          pf[2 * j] = fast_exp2(x.x);
          pf[2 * j + 1] = fast_exp2(x.y);
        }
      } else {   // scores of a padding column come from whatever sits in K there: select, do not multiply
#pragma unroll
        for (int j = 0; j < kBwCols; ++j)
          pf[j] = (c0 + j) < valid ? fast_exp2(fmaf(__uint_as_float(sv[j]), c, -lse)) : 0.f;
      }
      if (!p_free) ok = VSA_WARP_WAIT(bar(DK_P_EMPTY), (p & 1) ^ 1);      // dV^T of the previous pair has read the buffer
      if (!ok) break;
#pragma unroll
      for (int ch = 0; ch < kBwCols / 8; ++ch)
        *reinterpret_cast<uint4*>(prow + ((((kBwCols / 8) * cg + ch) ^ (t & 7)) << 4)) =
            make_uint4(Elem<elem_t>::pack(pf[8 * ch], pf[8 * ch + 1]), Elem<elem_t>::pack(pf[8 * ch + 2], pf[8 * ch + 3]),
                       Elem<elem_t>::pack(pf[8 * ch + 4], pf[8 * ch + 5]), Elem<elem_t>::pack(pf[8 * ch + 6], pf[8 * ch + 7]));
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(DK_P_FULL));
      // ---- dS = P * (dP - delta)
      ok = VSA_WARP_WAIT_TEST(bar(DK_DP_FULL + b), (p / kDkBufs) & 1, bar(DK_DS_EMPTY), (p & 1) ^ 1, &ds_free);
      if (!ok) break;
      tc_fence_after();
      uint32_t dvv[kBwCols];
      tmem_ld(tmem + b * 128 + 64 + lane_addr + c0, dvv);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(DK_S_EMPTY + b));       // both accumulators of this buffer have been read
      uint32_t pg[kBwCols / 2];
      if (!ragged) {
#pragma unroll
        for (int j2 = 0; j2 < kBwCols / 2; ++j2) {
          const float2 x = mul2(make_float2(pf[2 * j2], pf[2 * j2 + 1]), add2(word_pair(dvv + 2 * j2), make_float2(-dl, -dl)));
          pg[j2] = Elem<elem_t>::pack(x.x, x.y);
        }
      } else {   // dP of a padding column comes from whatever sits in V there
#pragma unroll
        for (int j2 = 0; j2 < kBwCols / 2; ++j2) {
          const float g0 = (c0 + 2 * j2) < valid ? pf[2 * j2] * (__uint_as_float(dvv[2 * j2]) - dl) : 0.f;
          const float g1 = (c0 + 2 * j2 + 1) < valid ? pf[2 * j2 + 1] * (__uint_as_float(dvv[2 * j2 + 1]) - dl) : 0.f;
          pg[j2] = Elem<elem_t>::pack(g0, g1);
        }
      }
      if (dst >= 0) {   // chunk-major tile: chunk c of row r at c * 1024 + r * 16 bytes
        uint4* g = reinterpret_cast<uint4*>(ds_ws + dst * (kTile * kTile)) + ((kBwCols / 8) * cg) * kTile + r;
#pragma unroll
        for (int ch = 0; ch < kBwCols / 8; ++ch)
          __stcs(g + ch * kTile, make_uint4(pg[4 * ch], pg[4 * ch + 1], pg[4 * ch + 2], pg[4 * ch + 3]));
      }
      if (!ds_free) ok = VSA_WARP_WAIT(bar(DK_DS_EMPTY), (p & 1) ^ 1);     // dK^T of the previous pair has read the buffer
      if (!ok) break;
#pragma unroll
      for (int ch = 0; ch < kBwCols / 8; ++ch)
        *reinterpret_cast<uint4*>(grow + ((((kBwCols / 8) * cg + ch) ^ (t & 7)) << 4)) =
            make_uint4(pg[4 * ch], pg[4 * ch + 1], pg[4 * ch + 2], pg[4 * ch + 3]);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(DK_DS_FULL));
    }
    if (!ok && lane == 0) report_timeout(24);
    if (ok) ok = VSA_WARP_WAIT(bar(DK_ACC_FULL), 0);
    if (!ok && lane == 0) report_timeout(25);
    tc_fence_after();
    elem_t* stage_k = reinterpret_cast<elem_t*>(sm + DkSmem::q);          // [64 key rows][128 dims] each; all MMAs done
    elem_t* stage_v = stage_k + kTile * kD;
    if (ok) {
      uint32_t ak[kBwCols], av[kBwCols];
      tmem_ld(tmem_dk + lane_addr + c0, ak);
      tmem_ld(tmem_dv + lane_addr + c0, av);
      tmem_ld_wait();
      float gmk = 0.f, gmv = 0.f;            // lane t is the head dim here, a column a key row
      if (mean_grad_k != nullptr) {
        gmk = Elem<elem_t>::to(mean_grad_k[mean_off + t]) * mean_inv;
        gmv = Elem<elem_t>::to(mean_grad_v[mean_off + t]) * mean_inv;
      }
#pragma unroll
      for (int j = 0; j < kBwCols; ++j) {
        const bool row_live = (c0 + j) < valid;
        stage_k[(c0 + j) * kD + t] = Elem<elem_t>::from(__uint_as_float(ak[j]) * scale + (row_live ? gmk : 0.f));
        stage_v[(c0 + j) * kD + t] = Elem<elem_t>::from(__uint_as_float(av[j]) + (row_live ? gmv : 0.f));
      }
    } else {
      for (int j = 0; j < kBwCols; ++j) {
        stage_k[(c0 + j) * kD + t] = Elem<elem_t>::from(0.f);
        stage_v[(c0 + j) * kD + t] = Elem<elem_t>::from(0.f);
      }
    }
    named_barrier(1, kBwEwThreads);
#pragma unroll
    for (int i = 0; i < 1024 / kBwEwThreads; ++i) {
      const int cidx = st + kBwEwThreads * i;
      const int row = cidx >> 4, ch = cidx & 15;
      const long long drow = out_map.map == nullptr ? krow0 + row : raster_row(out_map, bh, (long long)ktile * kTile + row);
      if (drow >= 0) {
        *reinterpret_cast<uint4*>(dk + drow * kD + ch * 8) = *reinterpret_cast<const uint4*>(stage_k + row * kD + ch * 8);
        *reinterpret_cast<uint4*>(dv + drow * kD + ch * 8) = *reinterpret_cast<const uint4*>(stage_v + row * kD + ch * 8);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, kTmemCols);
}

// ------------------------------------------------------------------------------------------------------
// dQ from stored dS:  dQ^T [128 dims x 64 query rows] = scale * sum over the selected key tiles of K^T dS^T
// ------------------------------------------------------------------------------------------------------
// The key-owned pass above has already formed every dS tile; this query-owned pass only streams, per selected
// key tile, the K tile (16 KB) and the dS tile (8 KB) and issues four M128 x N64 x K16 MMAs: no scores, no
// exponentials, no elementwise stage.  It is bound by how fast TMA brings the 24 KB in, so the ring is deep.
// Roles: warp 0 = TMA producer of the K tiles (two lanes, one box each), warp 1 = MMA issuer (owns the tensor
// memory; the whole warp zero-fills the padding rows of a ragged K tile first), warps 2-5 = epilogue, warps 6-7 =
// loaders of the dS tiles with plain asynchronous 16-byte copies: one SM's TMA unit moves ~50 bytes per clock in
// 8 KB boxes, the load/store path adds its own bandwidth beside it, and a dS tile is a verbatim 8 KB copy.
constexpr int kDsStages = 8;
constexpr int kDsStageBytes = 3 * kSlab;        // K head-dim half 0 | K head-dim half 1 | dS
constexpr int kDsLoaders = 64;                  // threads that copy dS tiles
constexpr int kDsThreads = 192 + kDsLoaders;
struct DqdsSmem {
  static constexpr uint32_t ring = 0;
  static constexpr uint32_t tile_row = ring + kDsStages * kDsStageBytes;   // int32 [kMaxTiles]
  static constexpr uint32_t tile_it = tile_row + 4 * kMaxTiles;            // uint16 [kMaxTiles]: position in the route
  static constexpr uint32_t tile_valid = tile_it + 2 * kMaxTiles;          // uint8 [kMaxTiles]
  static constexpr uint32_t bars = tile_valid + kMaxTiles;
  static constexpr uint32_t misc = bars + 32 * 8;
  static constexpr uint32_t total = misc + 64;
};
enum DqdsBar { DD_FULL = 0, DD_EMPTY = kDsStages, DD_ACC_FULL = 2 * kDsStages };

template <int SUB>
__global__ void __launch_bounds__(kDsThreads, 1)
sparse_dq_from_ds_kernel(const __grid_constant__ CUtensorMap map_k, const elem_t* __restrict__ ds_ws,
                         const int32_t* __restrict__ selected, const int32_t* __restrict__ kv_sizes,
                         elem_t* __restrict__ dq, const elem_t* __restrict__ mean_grad, const int32_t* __restrict__ q_sizes,
                         long long Lq, long long Lkv, int topk, float scale) {
  extern __shared__ uint8_t smem_raw[];
  if (*(volatile int*)&g_device_status != 0) return;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* sm = smem_raw + (base - smem_u32(smem_raw));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int qtile = blockIdx.x;
  const long long bh = blockIdx.y;
  const int Qb = (int)(Lq / (kTile * SUB)), Kb = (int)(Lkv / (kTile * SUB));
  const int qb = qtile / SUB, qsub = qtile % SUB;
  const int32_t* sel = selected + (bh * Qb + qb) * (long long)topk;
  const int n_iter = topk * SUB;
  const long long qrow0 = bh * Lq + (long long)qtile * kTile;
  const long long edge0 = (bh * Qb + qb) * (long long)topk;

  int32_t* tile_row = reinterpret_cast<int32_t*>(sm + DqdsSmem::tile_row);
  uint16_t* tile_it = reinterpret_cast<uint16_t*>(sm + DqdsSmem::tile_it);
  uint8_t* tile_valid = sm + DqdsSmem::tile_valid;
  volatile uint32_t* misc = reinterpret_cast<volatile uint32_t*>(sm + DqdsSmem::misc);
  auto bar = [&](int i) -> uint32_t { return base + DqdsSmem::bars + 8u * i; };

  if (tid == 0) {
    for (int i = 0; i < kDsStages; ++i) {
      mbar_init(bar(DD_FULL + i), 2 + kDsLoaders);     // two TMA lanes and every loader thread
      mbar_init(bar(DD_EMPTY + i), 1);
    }
    mbar_init(bar(DD_ACC_FULL), 1);
    fence_barrier_init();
    tma_prefetch_desc(&map_k);
  }
  for (int it = tid; it < n_iter; it += kDsThreads) {
    const int kvb = sel[it / SUB];
    const int left = (unsigned)kvb < (unsigned)Kb ? kv_sizes[kvb] - (it % SUB) * kTile : 0;   // an id outside the table is an empty tile
    tile_valid[it] = (uint8_t)(left < 0 ? 0 : (left > kTile ? kTile : left));
    tile_row[it] = kvb * (kTile * SUB) + (it % SUB) * kTile;
    tile_it[it] = (uint16_t)it;
  }
  __syncthreads();
  if (warp == 2) {   // squeeze out the empty tiles in place, keeping the routing order
    int n_live = 0;
    for (int it0 = 0; it0 < n_iter; it0 += 32) {
      const int it = it0 + lane;
      const int valid = it < n_iter ? (int)tile_valid[it] : 0;
      const int row = it < n_iter ? tile_row[it] : 0;
      const unsigned live = __ballot_sync(0xffffffffu, valid > 0);
      __syncwarp();
      if (valid > 0) {
        const int pos = n_live + __popc(live & ((1u << lane) - 1u));
        tile_row[pos] = row;
        tile_valid[pos] = (uint8_t)valid;
        tile_it[pos] = (uint16_t)it;
      }
      n_live += __popc(live);
      __syncwarp();
    }
    if (lane == 0) misc[1] = (uint32_t)n_live;
  }
  if (warp == 1) {
    tmem_alloc(base + DqdsSmem::misc, 64);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = misc[0];
  const int n_live = (int)misc[1];
  const long long kv_row_base = bh * Lkv;
  bool ok = true;

  if (warp == 0) {
    for (int i = 0; i < n_live; ++i) {
      const int s = i % kDsStages;
      ok = VSA_WARP_WAIT(bar(DD_EMPTY + s), ((i / kDsStages) & 1) ^ 1);
      if (!ok) break;
      if (lane < 2) {
        const uint32_t dst = base + DqdsSmem::ring + s * kDsStageBytes + lane * kSlab;
        mbar_arrive_expect_tx(bar(DD_FULL + s), kSlab);
        tma_load_2d(dst, &map_k, lane * 64, (int)(kv_row_base + tile_row[i]), bar(DD_FULL + s));
      }
    }
    if (!ok && lane == 0) report_timeout(31);
  } else if (warp >= 6) {
    const int lt = tid - 192;                          // 64 threads x 8 copies of 16 bytes = one 8 KB tile
    for (int i = 0; i < n_live; ++i) {
      const int s = i % kDsStages;
      ok = VSA_WARP_WAIT(bar(DD_EMPTY + s), ((i / kDsStages) & 1) ^ 1);
      if (!ok) break;
      const int it = tile_it[i];
      const long long tile = ((edge0 + it / SUB) * SUB + qsub) * SUB + (it % SUB);
      const uint8_t* src = reinterpret_cast<const uint8_t*>(ds_ws + tile * (kTile * kTile)) + lt * 16;
      const uint32_t dst = base + DqdsSmem::ring + s * kDsStageBytes + 2 * kSlab + lt * 16;
#pragma unroll
      for (int j = 0; j < kSlab / (16 * kDsLoaders); ++j) cp_async16(dst + j * 16 * kDsLoaders, src + j * 16 * kDsLoaders);
      cp_async_arrive_noinc(bar(DD_FULL + s));
    }
    if (!ok && lane == 0) report_timeout(34);
  } else if (warp == 1) {
    constexpr uint32_t idesc = instr_desc(128, 64, 1, 0, kInFmt);     // A = K^T (dims contiguous), B = dS (keys contiguous)
    constexpr uint32_t hi = desc_hi(1024);
    // B: un-swizzled K-major, core matrices of 8 query rows x 16 bytes; the next 8 rows 128 bytes on, the next
    // 8 key tokens (chunk) 1024 bytes on; one MMA consumes two chunks
    constexpr uint32_t hi_b = desc_hi_noswizzle(128);
    // Two tiles per trip: a wait on an mbarrier costs a shared-memory round trip of a few hundred cycles however
    // long ago it flipped, more than the four MMAs of a tile; two lanes look at two stages at once.
    for (int i0 = 0; i0 < n_live; i0 += 2) {
      const int n_here = n_live - i0 >= 2 ? 2 : 1;
      const int s0 = i0 % kDsStages, s1 = (i0 + 1) % kDsStages;
      if (n_here == 2)
        ok = VSA_WARP_WAIT2(bar(DD_FULL + s0), (i0 / kDsStages) & 1, bar(DD_FULL + s1), ((i0 + 1) / kDsStages) & 1);
      else
        ok = VSA_WARP_WAIT(bar(DD_FULL + s0), (i0 / kDsStages) & 1);
      if (!ok) break;
      for (int h = 0; h < n_here; ++h) {
        const int valid = tile_valid[i0 + h];
        if (valid < kTile) {
          // rows of K beyond a ragged tile's size meet dS = 0 in the product; they must be finite zeros (0 * NaN)
          uint8_t* kst = sm + DqdsSmem::ring + (h ? s1 : s0) * kDsStageBytes;
          for (int r = valid + (lane >> 4); r < kTile; r += 2) {
            const int ch = lane & 15;                 // 16 chunks of 16 bytes: both head-dim halves of the row
            *reinterpret_cast<uint4*>(kst + (ch >> 3) * kSlab + r * 128 + (ch & 7) * 16) = make_uint4(0, 0, 0, 0);
          }
          __syncwarp();
        }
      }
      if (lane == 0) {
        // the dS tiles were written by ordinary asynchronous copies (and padding rows by this warp); the tensor
        // core reads through the async proxy
        fence_proxy_async_smem();
        tc_fence_after();
        for (int h = 0; h < n_here; ++h) {
          const int s = h ? s1 : s0;
          const uint32_t stage = base + DqdsSmem::ring + s * kDsStageBytes;
          const uint32_t a0 = desc_lo(stage, kSlab), b0 = desc_lo(stage + 2 * kSlab, 1024);
#pragma unroll
          for (int ks = 0; ks < 4; ++ks)
            mma_ss(tmem, desc_pack(a0 + (uint32_t)(ks * 128), hi), desc_pack(b0 + (uint32_t)(ks * 128), hi_b), idesc,
                   (i0 + h > 0 || ks > 0) ? 1u : 0u);
          mma_commit(bar(DD_EMPTY + s));
        }
      }
      __syncwarp();
    }
    if (lane == 0) {
      if (ok) mma_commit(bar(DD_ACC_FULL));
      else report_timeout(32);
    }
  } else {
    // epilogue: lane t = head dim, a column = a query row
    const int quarter = warp & 3;
    const int t = quarter * 32 + lane;
    const int st = tid - 64;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    float gm = 0.f;
    int rows_live = 0;
    if (mean_grad != nullptr) {   // block-mean backward folded in, as in the recomputing dQ kernel
      const int size = q_sizes[qb];
      gm = Elem<elem_t>::to(mean_grad[(bh * Qb + qb) * (long long)kD + t]) / (float)(size > 1 ? size : 1);
      rows_live = size - qsub * kTile;
    }
    if (n_live > 0) ok = VSA_WARP_WAIT(bar(DD_ACC_FULL), 0);
    if (!ok && lane == 0) report_timeout(33);
    tc_fence_after();
    elem_t* stage = reinterpret_cast<elem_t*>(sm + DqdsSmem::ring);     // [64 query rows][128 dims]; every MMA is done
#pragma unroll
    for (int hcol = 0; hcol < 2; ++hcol) {
      uint32_t av[32];
      if (ok && n_live > 0) {
        tmem_ld(tmem + lane_addr + hcol * 32, av);
        tmem_ld_wait();
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) av[j] = 0u;
      }
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const int c = hcol * 32 + j;
        stage[c * kD + t] = Elem<elem_t>::from(__uint_as_float(av[j]) * scale + (c < rows_live ? gm : 0.f));
      }
    }
    named_barrier(1, 128);
    elem_t* og = dq + qrow0 * kD;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int cidx = st + 128 * i;
      const int row = cidx >> 4, ch = cidx & 15;
      *reinterpret_cast<uint4*>(og + row * kD + ch * 8) = *reinterpret_cast<const uint4*>(stage + row * kD + ch * 8);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, 64);
}
