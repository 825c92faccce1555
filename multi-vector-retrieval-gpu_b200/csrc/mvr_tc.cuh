// mvr_tc.cuh -- launchers of the tensor-core (tcgen05) kernels (mvr_tc.cu).
#pragma once
#include <cuda_runtime.h>
#include "mvr_common.cuh"
#include "mvr_plan.hpp"

namespace mvr {

cudaError_t configure_tc_kernels();
cudaError_t make_bf16(const float *in, size_t n, void *out, cudaStream_t st);

// bucket-weight tables of the tensor-memory MaxSim kernels (make_tm_weights):
//  BF16 (1-, 2-bit): w[0] / w[1] = low / high bytes of the BF16 weights;
//  FP8 2-bit: w[0] = the 4 E4M3 weights;
//  FP8 4-bit: w[0..1] = |E4M3| of weights 0..7, w[2..3] of weights 8..15,
//             w[4..5] byte j: bit 6 = sign of weight j, bit 7 = of weight 8 + j
struct TmWeights {
  uint32_t w[6];
};
TmWeights make_tm_weights(uint32_t n_bit, const float *weight, bool fp8);

// BF16 MaxSim on the tensor cores; cen_perm: [C + 1][128] BF16 centroid rows in the
// kernels' K order, the last zero (make_centroid_perm); lut_bf16: [256][8/b] BF16
// weights of a residual byte (4 and 8 bits); x_bound: upper bound on the norm of
// every decoded doc token; wait_ns as launch_rerank_ws.  Queries of up to
// kBf16SplitTok tokens: BF16 centroid and BF16 weights contribute separately, where
// split (bf16_split_supported; c_min: the smallest non-zero centroid norm); otherwise their BF16-rounded sum.
constexpr uint32_t kBf16SplitTok = 32;
bool bf16_split_supported(uint32_t n_bit, float x_bound, float c_min);
// largest and smallest non-zero L2 norm of the centroid rows (NaN: none); d_tmp: two
// device words of scratch; synchronises st
cudaError_t centroid_norm_range(const float *cen, uint32_t n_cent, unsigned *d_tmp, float *c_max,
                                float *c_min, cudaStream_t st);
cudaError_t make_centroid_perm(const float *cen, uint32_t n_cent, uint32_t n_bit, void *out,
                               cudaStream_t st);
cudaError_t launch_rerank_bf16(const DevIndex &ix, const void *cen_perm, const void *lut_bf16,
                               const TmWeights &tw, const float *q, const uint64_t *q_off,
                               uint32_t n_query, const uint32_t *short_id,
                               const uint32_t *n_short, uint32_t probe_topk, int semantics,
                               uint32_t nq_min, uint32_t nq_max, float x_bound, bool split,
                               float *approx, unsigned *err, int n_sm, cudaStream_t st,
                               int *n_launch, uint64_t wait_ns);
// E4M3 centroid rows [C][128] in the FP8 kernel's K order (2- and 4-bit codes)
bool fp8_rerank_supported(uint32_t n_bit);
cudaError_t make_centroid_fp8(const float *cen, uint32_t n_cent, uint32_t n_bit, void *out,
                              cudaStream_t st);

// FP8 (E4M3) MaxSim, warp-specialised (producer / decoders / MMA / epilogue
// over a shared-memory ring fed by bulk copies): cen8 as above with one zero
// row appended (row n_centroid); the vq code array must be readable 16 bytes
// past its last code.  wait_ns bounds every pipeline wait of the kernel (on
// expiry it stops and sets bit 4 of *err); nq_min / nq_max: fewest and most
// tokens of a query; set_docs: shortlisted docs per CTA (0: by the grid).
cudaError_t launch_rerank_ws(const DevIndex &ix, const void *cen8, const TmWeights &tw,
                             const float *q, const uint64_t *q_off, uint32_t n_query,
                             const uint32_t *short_id, const uint32_t *n_short,
                             uint32_t probe_topk, int semantics, uint32_t nq_min, uint32_t nq_max,
                             float x_bound, float *approx, unsigned *err, int n_sm,
                             cudaStream_t st, int *n_launch, uint64_t wait_ns, uint32_t set_docs);
// shortlisted docs per CTA the FP8 kernel is built for (32, 64, 128, 256)
bool ws_docs_supported(uint32_t docs);

// Learned-pruner features of every shortlisted doc with the FP8 kernel's
// centroid part only: feat [n_query][probe_topk][33] = per query token the
// best E4M3 centroid score q.c over the doc's tokens, then log(doc length).
// Queries of up to 32 tokens.
cudaError_t launch_prune_features(const DevIndex &ix, const void *cen8, const float *q,
                                  const uint64_t *q_off, uint32_t n_query,
                                  const uint32_t *short_id, const uint32_t *n_short,
                                  uint32_t probe_topk, float x_bound, float *feat, unsigned *err,
                                  cudaStream_t st, int *n_launch, uint64_t wait_ns);
// The docs the rerank takes after the pruner (see mvr_tc.cu).
cudaError_t launch_prune_choose(const DevIndex &ix, const uint32_t *short_id,
                                const uint32_t *n_short, const uint32_t *kept_id,
                                const float *kept_s, uint32_t n_query, uint32_t probe_topk,
                                uint32_t keep, uint32_t R, float margin, uint32_t *fin_id,
                                uint32_t *n_fin, uint32_t *qstat,
                                unsigned long long *n_fallback, cudaStream_t st, int *n_launch);
// The learned pruner's MLP on the tensor cores: pred [n_query][probe_topk]
// from the features of the rows d < n_short[query]; wts / vecs: the weights
// prepared by prune_prepare (prune_weight_bytes() bytes / 769 floats).
size_t prune_weight_bytes();
cudaError_t prune_prepare(const float *params, uint8_t *wts, float *vecs, cudaStream_t st);
cudaError_t launch_prune_mlp(const float *feat, const uint32_t *n_short, uint32_t n_query,
                             uint32_t probe_topk, const uint8_t *wts, const float *vecs,
                             float *pred, unsigned *err, int n_sm, cudaStream_t st,
                             int *n_launch);

// pre-swizzled BF16 tiles of 64 centroids (n_tiles = C_pad / 64, an even count)
cudaError_t make_centroid_tiles(const float *cen, uint32_t n_cent, uint32_t n_tiles, void *out,
                                cudaStream_t st);

// Buffers of a centroid-scoring launch (probe_plan, mvr_plan.hpp)
struct ProbeBufs {
  float4 *ent;        // [n_ent] listed groups of 8 centroids: their BF16 scores
  uint32_t *gid;      // [n_gid] ... and the group's index
  uint32_t *cnt;      // [n_cnt] their count (above cap: the list overflowed)
  float *eps2;        // [n_tok] twice the token's BF16 error bound
  uint32_t *flags;    // [n_flag] count of flagged tokens, scan counters, the tokens
  uint32_t *part_id;  // [n_part] the exact scan's partial lists
  float *part_s;
};
// bounds[2] of probe_tc_kernel: max |c| and max |c - bf16(c)| over the centroids
cudaError_t make_centroid_bounds(const float *cen, uint32_t n_cent, float *bounds,
                                 cudaStream_t st);
// bounds: the largest norm of a doc token's weights, and of their BF16 rounding errors
cudaError_t make_weight_bounds(const DevIndex &ix, float *bounds, int n_sm, cudaStream_t st);
// top nprobe (1..32) per token, (score desc, id asc), equal to an exact FP32
// scan's; cen_sw: swizzled BF16 tiles (make_centroid_tiles), cen: [C][128],
// cen_t: [128][n_cent_pad]
cudaError_t launch_probe(const float *q, uint32_t n_tok, const void *cen_sw, const float *cen,
                         const float *cen_t, uint32_t n_cent, uint32_t n_cent_pad,
                         const float *bounds, uint32_t nprobe, const ProbePlan &p,
                         const ProbeBufs &w, uint32_t *out_id, float *out_s, int n_sm,
                         unsigned *err, cudaStream_t st, int *n_launch);

}  // namespace mvr
