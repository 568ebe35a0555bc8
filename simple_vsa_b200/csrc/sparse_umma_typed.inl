// Tensor-path kernels and their launchers for ONE 16-bit element type.  The including file opens a namespace,
// defines there
//     elem_t      the element type (__nv_bfloat16 or __half),
//     kInFmt      its code in the tcgen05 instruction descriptor (1 = bf16, 0 = fp16),
//     kTmaElem    its CUtensorMapDataType,
//     kDtypeCode  its VSA_* dtype code,
//     kShiftBias  binades added to the forward's fixed softmax shift (centres P in the type's exponent range),
// and includes this file; everything else (tiling, barriers, pipelines, tensor-memory use) is the same for both.
int make_map(CUtensorMap* map, const void* ptr, int64_t rows, const char* what, int cols = kD) {
  return make_map_of(map, kTmaElem, ptr, rows, what, cols);
}
int make_map3d(CUtensorMap* map, const void* ptr, int64_t batch, int64_t rows, int64_t cols, int box_rows, const char* what,
               int64_t pitch = 0) {
  return make_map3d_of(map, kTmaElem, ptr, batch, rows, cols, box_rows, what, pitch);
}

// 8 MMAs over the 128-wide reduction, both operands reduction-contiguous ("K-major").
// a_pair: a stacked pair [2 halves][128 rows][128 B]; b_tile: one tile [2 halves][64 rows][128 B].
// Descriptors are advanced with one 32-bit add each (offsets in 16-byte units are compile-time constants).
__device__ __forceinline__ void issue_kmajor(uint32_t d_tmem, uint32_t a_pair, uint32_t b_tile) {
  constexpr uint32_t idesc = instr_desc(128, 64, 0, 0, kInFmt);
  constexpr uint32_t hi = desc_hi(1024);
  const uint32_t a0 = desc_lo(a_pair, 16), b0 = desc_lo(b_tile, 16);
#pragma unroll
  for (int ks = 0; ks < 8; ++ks)
    mma_ss(d_tmem, desc_pack(a0 + (uint32_t)(((ks >> 2) * kPairHalf + (ks & 3) * 32) >> 4), hi),
           desc_pack(b0 + (uint32_t)(((ks >> 2) * kSlab + (ks & 3) * 32) >> 4), hi), idesc, ks > 0 ? 1u : 0u);
}
// 8 MMAs over 128 rows of reduction, both operands output-contiguous ("MN-major"):
// D[128 dims x 64] (+)= a_pair^T [128 dims x 128 rows] * b_rows [128 rows x 64].
__device__ __forceinline__ void issue_mnmajor(uint32_t d_tmem, uint32_t a_pair, uint32_t b_rows, bool accumulate) {
  constexpr uint32_t idesc = instr_desc(128, 64, 1, 1, kInFmt);
  constexpr uint32_t hi = desc_hi(1024);
  const uint32_t a0 = desc_lo(a_pair, kPairHalf), b0 = desc_lo(b_rows, 16);
  const uint32_t acc0 = accumulate ? 1u : 0u;
#pragma unroll
  for (int ks = 0; ks < 8; ++ks)
    mma_ss(d_tmem, desc_pack(a0 + (uint32_t)(ks * 128), hi), desc_pack(b0 + (uint32_t)(ks * 128), hi), idesc,
           ks > 0 ? 1u : acc0);
}

#include "sparse_umma_bwd.inl"
#include "sparse_wide.inl"
#include "sparse_split.inl"
#include "coarse_umma.inl"

// ---- host launchers of this element type ----------------------------------------------------------------------
int sparse_fwd_umma(const void* q, const void* k, const void* v, const int32_t* selected, const int32_t* kv_sizes,
                    void* out, float* lse2, int64_t BH, int64_t Lq, int64_t Lkv, int D, int be, int topk, float scale,
                    cudaStream_t st, const void* out_c, const void* gate, void* out_comb, int64_t kv_shard,
                    RasterMap comb_map) {
  if (BH == 0 || Lq == 0) return VSA_OK;
  { const int rc0 = check_kv_shard(Lkv, be, &kv_shard, "sparse forward"); if (rc0) return rc0; }
  if (BH > 65535) return fail(VSA_ERR_UNSUPPORTED, "sparse forward: batch*heads %lld exceeds 65535", (long long)BH);
  if (sparse_wide_rows(kPassForward, BH, Lq, D, be, topk, false))
    return D == 64 ? launch_fwd_wide<64>(q, k, v, selected, kv_sizes, out, lse2, BH, Lq, Lkv, be, topk, scale, st, out_c, gate, out_comb, kv_shard, comb_map)
                   : launch_fwd_wide<128>(q, k, v, selected, kv_sizes, out, lse2, BH, Lq, Lkv, be, topk, scale, st, out_c, gate, out_comb, kv_shard, comb_map);
  return D == 64 ? launch_fwd_split<64>(q, k, v, selected, kv_sizes, out, lse2, BH, Lq, Lkv, be, topk, scale, st, out_c, gate, out_comb, kv_shard, comb_map)
                 : launch_fwd_split<128>(q, k, v, selected, kv_sizes, out, lse2, BH, Lq, Lkv, be, topk, scale, st, out_c, gate, out_comb, kv_shard, comb_map);
}

int sparse_dq_umma(const void* dout, const void* q, const void* k, const void* v, const void* out_s,
                   const float* lse2, const int32_t* selected, const int32_t* kv_sizes, float* delta, void* dq,
                   int64_t BH, int64_t Lq, int64_t Lkv, int D, int be, int topk, float scale, cudaStream_t st,
                   const void* dq_mean, const int32_t* q_sizes, int64_t kv_shard, RasterMap out_map) {
  if (BH == 0 || Lq == 0) return VSA_OK;
  if (BH > 65535) return fail(VSA_ERR_UNSUPPORTED, "sparse dQ: batch*heads %lld exceeds 65535", (long long)BH);
  { const int rc0 = check_kv_shard(Lkv, be, &kv_shard, "sparse dQ"); if (rc0) return rc0; }
  if (sparse_wide_rows(kPassDq, BH, Lq, D, be, topk, dq_mean != nullptr))
    return D == 64 ? launch_dq_wide<64>(dout, q, k, v, out_s, lse2, selected, kv_sizes, delta, dq, BH, Lq, Lkv, be, topk, scale, st, dq_mean, q_sizes, kv_shard, out_map)
                   : launch_dq_wide<128>(dout, q, k, v, out_s, lse2, selected, kv_sizes, delta, dq, BH, Lq, Lkv, be, topk, scale, st, dq_mean, q_sizes, kv_shard, out_map);
  return D == 64 ? launch_dq_split<64>(dout, q, k, v, out_s, lse2, selected, kv_sizes, delta, dq, BH, Lq, Lkv, be, topk, scale, st, dq_mean, q_sizes, kv_shard, out_map)
                 : launch_dq_split<128>(dout, q, k, v, out_s, lse2, selected, kv_sizes, delta, dq, BH, Lq, Lkv, be, topk, scale, st, dq_mean, q_sizes, kv_shard, out_map);
}

int sparse_dkdv_umma(const void* dout, const void* q, const void* k, const void* v, const float* lse2,
                     const float* delta, const int32_t* counts, const int32_t* offsets, const int32_t* inverse,
                     const int32_t* kv_sizes, void* dk, void* dv, int64_t BH, int64_t Lq, int64_t Lkv, int D, int be, int topk,
                     float scale, cudaStream_t st, const void* dk_mean, const void* dv_mean, void* ds_ws,
                     int64_t kv_shard, RasterMap out_map) {
  if (BH == 0 || Lkv == 0) return VSA_OK;
  if (BH > 65535) return fail(VSA_ERR_UNSUPPORTED, "sparse dK/dV: batch*heads %lld exceeds 65535", (long long)BH);
  { const int rc0 = check_kv_shard(Lkv, be, &kv_shard, "sparse dK/dV"); if (rc0) return rc0; }
  if (ds_ws && topk > (1 << kEdgeSlotBits))
    return fail(VSA_ERR_UNSUPPORTED, "sparse dK/dV: packed edges hold at most %d routes per query block", 1 << kEdgeSlotBits);
  CUtensorMap mq, mdo, mk, mv;
  int rc;
  if (!ds_ws && sparse_wide_rows(kPassDkdv, BH, Lkv, D, be, topk, dk_mean != nullptr))
    return D == 64 ? launch_dkdv_wide<64>(dout, q, k, v, lse2, delta, counts, offsets, inverse, kv_sizes, dk, dv, BH, Lq, Lkv, be, topk, scale, st, dk_mean, dv_mean, kv_shard, out_map)
                   : launch_dkdv_wide<128>(dout, q, k, v, lse2, delta, counts, offsets, inverse, kv_sizes, dk, dv, BH, Lq, Lkv, be, topk, scale, st, dk_mean, dv_mean, kv_shard, out_map);
  if (ds_ws == nullptr)
    return D == 64 ? launch_dkdv_split<64>(dout, q, k, v, lse2, delta, counts, offsets, inverse, kv_sizes, dk, dv, BH, Lq, Lkv, be, topk, scale, st, dk_mean, dv_mean, kv_shard, out_map)
                   : launch_dkdv_split<128>(dout, q, k, v, lse2, delta, counts, offsets, inverse, kv_sizes, dk, dv, BH, Lq, Lkv, be, topk, scale, st, dk_mean, dv_mean, kv_shard, out_map);
  if ((rc = make_map(&mq, q, BH * Lq, "sparse dK/dV (q)"))) return rc;
  if ((rc = make_map(&mdo, dout, BH * Lq, "sparse dK/dV (dout)"))) return rc;
  if ((rc = make_map(&mk, k, BH * Lkv, "sparse dK/dV (k)"))) return rc;
  if ((rc = make_map(&mv, v, BH * Lkv, "sparse dK/dV (v)"))) return rc;
  if (reinterpret_cast<uintptr_t>(ds_ws) % 16)
    return fail(VSA_ERR_BAD_ARGUMENT, "sparse dK/dV: the dS workspace is not 16-byte aligned");
  const int smem = DkSmem::total + 1024;
  dim3 grid((unsigned)(Lkv / kTile), (unsigned)BH);
  auto launch = [&](auto kern) -> int {
    if ((rc = reserve_smem(kern, smem, "sparse dK/dV"))) return rc;
    kern<<<grid, kBwdThreads, smem, st>>>(mq, mdo, mk, mv, lse2, delta, counts, offsets, inverse, kv_sizes, (elem_t*)dk,
                                          (elem_t*)dv, (const elem_t*)dk_mean, (const elem_t*)dv_mean, (elem_t*)ds_ws, Lq, Lkv,
                                          kv_shard, topk, scale, out_map);
    return check_launch("sparse_dkdv_ds_umma_kernel");
  };
  VSA_BY_BLOCK_VOLUME(be, launch, sparse_dkdv_ds_umma_kernel);
}

int sparse_dq_from_ds_umma(const void* k, const int32_t* selected, const int32_t* kv_sizes, const void* ds_ws, void* dq,
                           int64_t BH, int64_t Lq, int64_t Lkv, int be, int topk, float scale, cudaStream_t st,
                           const void* dq_mean, const int32_t* q_sizes) {
  if (BH == 0 || Lq == 0) return VSA_OK;
  if (BH > 65535) return fail(VSA_ERR_UNSUPPORTED, "sparse dQ: batch*heads %lld exceeds 65535", (long long)BH);
  if (reinterpret_cast<uintptr_t>(ds_ws) % 16)
    return fail(VSA_ERR_BAD_ARGUMENT, "sparse dQ: the dS workspace is not 16-byte aligned");
  CUtensorMap mk;
  int rc;
  if ((rc = make_map(&mk, k, BH * Lkv, "sparse dQ (k)"))) return rc;
  const int smem = DqdsSmem::total + 1024;
  dim3 grid((unsigned)(Lq / kTile), (unsigned)BH);
  auto launch = [&](auto kern) -> int {
    if ((rc = reserve_smem(kern, smem, "sparse dQ"))) return rc;
    kern<<<grid, kDsThreads, smem, st>>>(mk, (const elem_t*)ds_ws, selected, kv_sizes, (elem_t*)dq, (const elem_t*)dq_mean,
                                         q_sizes, Lq, Lkv, topk, scale);
    return check_launch("sparse_dq_from_ds_kernel");
  };
  VSA_BY_BLOCK_VOLUME(be, launch, sparse_dq_from_ds_kernel);
}

// C[batch, M, N] = A * B.  a_rows/a_cols and b_rows/b_cols describe the operands as stored in memory; a_pitch and c_pitch
// (0: dense) are the row pitches of A and of C (and of `probs`).
template <int A_MN, int B_MN, int EPI>
int launch_gemm(const void* A, int64_t a_rows, int64_t a_cols, int64_t a_pitch, const void* B, int64_t b_rows, int64_t b_cols,
                void* C, int64_t c_pitch, int64_t batch, int M, int N, int K, float scale, const void* probs,
                const float* rowdot, cudaStream_t st, const char* what) {
  if (batch == 0 || M == 0 || N == 0) return VSA_OK;
  if (batch > 65535) return fail(VSA_ERR_UNSUPPORTED, "%s: batch*heads %lld exceeds 65535", what, (long long)batch);
  CUtensorMap ma, mb;
  int rc;
  if ((rc = make_map3d(&ma, A, batch, a_rows, a_cols, A_MN ? 64 : 128, what, a_pitch))) return rc;
  if ((rc = make_map3d(&mb, B, batch, b_rows, b_cols, B_MN ? 64 : 128, what))) return rc;
  const int smem = GemmSmem::total + 1024;
  auto kern = coarse_gemm_umma_kernel<A_MN, B_MN, EPI>;
  if ((rc = reserve_smem(kern, smem, what))) return rc;
  dim3 grid((unsigned)((N + 127) / 128), (unsigned)((M + 127) / 128), (unsigned)batch);
  kern<<<grid, 192, smem, st>>>(ma, mb, (elem_t*)C, M, N, K, (int)(c_pitch ? c_pitch : N), scale, (const elem_t*)probs, rowdot);
  return check_launch(what);
}

// The scores keep the operator's dense layout.  Unless both block counts are multiples of 8 their product runs on the CUDA cores:
// the wide stores want rows of 16 bytes (Kb % 8 == 0), and a sum taken in another order can turn a rounding, and with it a tie
// at the edge of the Top-K, so an odd Qb alone does not move a shape either.  It is one product of six.
int coarse_fwd_umma(const void* qc, const void* kc, const void* vc, void* scores, void* probs, void* out_c, int64_t BH,
                    int Qb, int Kb, int pitch, int D, float scale, cudaStream_t st) {
  int rc = Qb % 8 == 0 && Kb % 8 == 0
               ? launch_gemm<0, 0, kEpiScores>(qc, Qb, D, 0, kc, Kb, D, scores, 0, BH, Qb, Kb, D, scale, nullptr, nullptr, st,
                                               "pooled scores")
               : coarse_scores(qc, kc, scores, BH, Qb, Kb, D, scale, kDtypeCode, st);
  if (rc) return rc;
  if ((rc = softmax_rows(scores, probs, BH * Qb, Kb, pitch, kDtypeCode, st))) return rc;
  return launch_gemm<0, 1, kEpiStore>(probs, Qb, Kb, pitch, vc, Kb, D, out_c, 0, BH, Qb, D, Kb, 1.f, nullptr, nullptr, st,
                                      "pooled output");
}

int coarse_bwd_umma(const void* d_out_c, const void* out_c, const void* qc, const void* kc, const void* vc,
                    const void* probs, void* ds, float* rowdot, void* dqc, void* dkc, void* dvc, int64_t BH, int Qb,
                    int Kb, int pitch, int D, float scale, cudaStream_t st) {
  int rc = rowdot_rows(d_out_c, out_c, rowdot, BH * Qb, D, kDtypeCode, st);
  if (rc) return rc;
  // dV_c[Kb,D] = P^T dO_c : A = P stored [Qb rows (reduction), Kb cols (M)], B = dO_c stored [Qb rows, D cols]
  if ((rc = launch_gemm<1, 1, kEpiStore>(probs, Qb, Kb, pitch, d_out_c, Qb, D, dvc, 0, BH, Kb, D, Qb, 1.f, nullptr, nullptr,
                                         st, "pooled dV")))
    return rc;
  // dS[Qb,Kb] = P * (dO_c v_c^T - rowdot) * scale
  if ((rc = launch_gemm<0, 0, kEpiSoftmaxBwd>(d_out_c, Qb, D, 0, vc, Kb, D, ds, pitch, BH, Qb, Kb, D, scale, probs, rowdot,
                                              st, "pooled dS")))
    return rc;
  // dQ_c[Qb,D] = dS k_c
  if ((rc = launch_gemm<0, 1, kEpiStore>(ds, Qb, Kb, pitch, kc, Kb, D, dqc, 0, BH, Qb, D, Kb, 1.f, nullptr, nullptr, st,
                                         "pooled dQ")))
    return rc;
  // dK_c[Kb,D] = dS^T q_c
  return launch_gemm<1, 1, kEpiStore>(ds, Qb, Kb, pitch, qc, Qb, D, dkc, 0, BH, Kb, D, Qb, 1.f, nullptr, nullptr, st,
                                      "pooled dK");
}
