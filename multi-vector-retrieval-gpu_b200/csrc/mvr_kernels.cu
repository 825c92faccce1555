// mvr_kernels.cu -- the plain FP32 search kernels of libmvr (sm_100a).
//
// Stage map (reference -> kernel):
//   centroid scoring S = Q.C^T + 1 and per-token top-nprobe
//       (GenerateVQScoreCandidatePP.hpp:118-179: cuBLAS SGEMM, thrust +1,
//        RAFT select_k)                       -> mvr_tc.cu, probe_scan_kernel
//   IVF gather, candidate flag/compaction, max-over-probes, sum over tokens,
//   top-probe_topk shortlist (FilterPP.hpp:19-142, 267-398)
//                                             -> filter_kernel
//   VQ/residual gather, decompress, SGEMM, max over doc tokens, sum over
//   query tokens (RerankPP.hpp:16-161, 368-475) -> rerank_kernel
//   host std::sort of the shortlist (IGPGPURetrievalPP.hpp:153-161)
//                                             -> topk_kernel
//
// Every dot product is a sequential __fmaf_rn chain over d = 0..127 from
// 0.0f, every other add is a single rounded FP32 add and every sum runs in a
// fixed order, so results are bit-identical to the CPU oracle's canonical
// arithmetic and independent of launch shape.
#include "mvr_common.cuh"
#include "mvr_kernels.cuh"

#include <cuda_bf16.h>

#include <algorithm>
#include <cfloat>

namespace mvr {

// ---------------------------------------------------------------------
// small helpers
// ---------------------------------------------------------------------
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async4(void *smem, const void *gmem) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;\n" ::);
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

constexpr unsigned kFull = 0xffffffffu;

// Insert (s, id) into the sorted per-warp list held one entry per lane
// (lanes < np).  thr is the list's worst entry, uniform across the warp.
__device__ __forceinline__ void warp_list_insert(float &ls, uint32_t &lid,
                                                 float &thr_s, uint32_t &thr_id,
                                                 float ns, uint32_t nid,
                                                 int lane, int np) {
  const bool ahead = lane < np && better(ls, lid, ns, nid);
  const int pos = __popc(__ballot_sync(kFull, ahead));
  const float up_s = __shfl_up_sync(kFull, ls, 1);
  const uint32_t up_id = __shfl_up_sync(kFull, lid, 1);
  if (lane > pos) {
    ls = up_s;
    lid = up_id;
  } else if (lane == pos) {
    ls = ns;
    lid = nid;
  }
  thr_s = __shfl_sync(kFull, ls, np - 1);
  thr_id = __shfl_sync(kFull, lid, np - 1);
}

// ---------------------------------------------------------------------
// K1 fallback: exact S = Q.C^T + 1 and top-nprobe of the tokens that the
// tensor-core scan flagged (mvr_tc.cu: a list that overflowed, a bound that is
// not finite), by FP32 chains over every centroid.  flags[0] = their count,
// flags[2 ..] one arrival counter per 64-token tile (zeroed by the caller),
// flags[list_at ..] the tokens.  A persistent grid of one CTA per SM takes
// (token tile, centroid split) items; few tiles are split over the centroids
// so that the grid has work, and the last CTA of a tile merges its partial
// lists.  With nothing flagged, the usual case, every CTA returns at once.
// Item = 64 tokens x (tiles_per_split * 128) centroids, 256 threads.
// Thread (warp w, lane l): tokens w*8..w*8+7, centroids l*4..l*4+3 of the
// current 128-wide tile.  Qs[k][64] and double-buffered Cs[k][128] in smem.
// ---------------------------------------------------------------------
constexpr int kProbeTokTile = 64;
constexpr int kProbeCenTile = 128;
constexpr size_t kProbeSmem =
    (size_t)(kDim * kProbeTokTile + 2 * kDim * kProbeCenTile) * sizeof(float);

__global__ void __launch_bounds__(256, 1)
probe_scan_kernel(const float *__restrict__ q, const float *__restrict__ ct, uint32_t n_cent,
                  uint32_t n_cent_pad, uint32_t nprobe, uint32_t *__restrict__ flags,
                  uint32_t list_at, uint32_t *__restrict__ part_id, float *__restrict__ part_s,
                  uint32_t *__restrict__ out_id, float *__restrict__ out_s) {
  extern __shared__ __align__(16) float smem[];
  float *Qs = smem;                          // [128][64]
  float *Cs = smem + kDim * kProbeTokTile;   // [2][128][128]
  __shared__ uint32_t s_last;
  const uint32_t n_tok = flags[0];
  if (n_tok == 0) return;
  const uint32_t *list = flags + list_at;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int np = (int)nprobe;
  const uint32_t n_tiles = n_cent_pad / kProbeCenTile;
  const uint32_t tok_tiles = (n_tok + kProbeTokTile - 1) / kProbeTokTile;
  uint32_t splits = min(n_tiles, max(1u, gridDim.x / tok_tiles));
  const uint32_t tiles_per_split = (n_tiles + splits - 1) / splits;
  splits = (n_tiles + tiles_per_split - 1) / tiles_per_split;

  auto load_tile = [&](uint32_t tile, int buf) {
    float *dst = Cs + buf * kDim * kProbeCenTile;
    const float *src = ct + (size_t)tile * kProbeCenTile;
    // 128 rows x 32 chunks of 16 B
#pragma unroll
    for (int i = 0; i < (kDim * kProbeCenTile / 4) / 256; i++) {
      const int ch = tid + i * 256;
      const int k = ch >> 5, c4 = ch & 31;
      cp_async16(dst + k * kProbeCenTile + c4 * 4, src + (size_t)k * n_cent_pad + c4 * 4);
    }
    cp_async_commit();
  };

  for (uint32_t item = blockIdx.x; item < tok_tiles * splits; item += gridDim.x) {
    const uint32_t tt = item / splits, t0 = tt * kProbeTokTile;
    const uint32_t tile_begin = (item % splits) * tiles_per_split;
    const uint32_t tile_end = min(n_tiles, tile_begin + tiles_per_split);
    for (int i = tid; i < kProbeTokTile * (kDim / 4); i += 256) {
      const int t = i % kProbeTokTile, k4 = i / kProbeTokTile;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (t0 + t < n_tok)
        v = __ldg(reinterpret_cast<const float4 *>(q + (size_t)list[t0 + t] * kDim) + k4);
      Qs[(k4 * 4 + 0) * kProbeTokTile + t] = v.x;
      Qs[(k4 * 4 + 1) * kProbeTokTile + t] = v.y;
      Qs[(k4 * 4 + 2) * kProbeTokTile + t] = v.z;
      Qs[(k4 * 4 + 3) * kProbeTokTile + t] = v.w;
    }
    float Ls[8], thr_s[8];
    uint32_t Lid[8], thr_id[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
      Ls[i] = -INFINITY; Lid[i] = 0xffffffffu;
      thr_s[i] = -INFINITY; thr_id[i] = 0xffffffffu;
    }

    load_tile(tile_begin, 0);
    for (uint32_t tile = tile_begin; tile < tile_end; tile++) {
      const int buf = (tile - tile_begin) & 1;
      if (tile + 1 < tile_end) {
        load_tile(tile + 1, buf ^ 1);
        cp_async_wait<1>();
      } else {
        cp_async_wait<0>();
      }
      __syncthreads();

      float acc[8][4];
#pragma unroll
      for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0.0f;
      const float *qs = Qs + warp * 8;
      const float *cs = Cs + buf * kDim * kProbeCenTile + lane * 4;
#pragma unroll 4
      for (int k = 0; k < kDim; k++) {
        const float4 a0 = *reinterpret_cast<const float4 *>(qs + k * kProbeTokTile);
        const float4 a1 = *reinterpret_cast<const float4 *>(qs + k * kProbeTokTile + 4);
        const float4 b = *reinterpret_cast<const float4 *>(cs + k * kProbeCenTile);
        const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
        const float bb[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
          for (int j = 0; j < 4; j++) acc[i][j] = __fmaf_rn(a[i], bb[j], acc[i][j]);
      }

      const uint32_t c0 = tile * kProbeCenTile + lane * 4;
#pragma unroll
      for (int i = 0; i < 8; i++) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const float s = __fadd_rn(acc[i][j], 1.0f);
          const uint32_t id = c0 + j;
          const bool cand = id < n_cent && better(s, id, thr_s[i], thr_id[i]);
          unsigned m = __ballot_sync(kFull, cand);
          while (m) {
            const int src = __ffs(m) - 1;
            m &= m - 1;
            const float ns = __shfl_sync(kFull, s, src);
            const uint32_t nid = __shfl_sync(kFull, id, src);
            if (better(ns, nid, thr_s[i], thr_id[i]))
              warp_list_insert(Ls[i], Lid[i], thr_s[i], thr_id[i], ns, nid, lane, np);
          }
        }
      }
      __syncthreads();
    }

    if (splits == 1) {
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const uint32_t t = t0 + warp * 8 + i;
        if (t < n_tok && lane < np) {
          out_id[(size_t)list[t] * nprobe + lane] = Lid[i];
          out_s[(size_t)list[t] * nprobe + lane] = Ls[i];
        }
      }
    } else {
      // items are at most gridDim.x here: one partial slot of 64 lists each
#pragma unroll
      for (int i = 0; i < 8; i++) {
        if (lane < np) {
          const size_t at = ((size_t)item * kProbeTokTile + warp * 8 + i) * nprobe + lane;
          part_id[at] = Lid[i];
          part_s[at] = Ls[i];
        }
      }
      __threadfence();
      __syncthreads();
      if (tid == 0) s_last = atomicAdd(flags + 2 + tt, 1u) == splits - 1 ? 1u : 0u;
      __syncthreads();
      if (s_last) {
        __threadfence();
        for (int i = 0; i < 8; i++) {
          const uint32_t t = t0 + warp * 8 + i;
          if (t >= n_tok) break;
          float ls = -INFINITY, ts = -INFINITY;
          uint32_t lid = 0xffffffffu, tid_ = 0xffffffffu;
          for (uint32_t sp = 0; sp < splits; sp++) {
            const size_t base =
                (((size_t)tt * splits + sp) * kProbeTokTile + warp * 8 + i) * nprobe;
            float ps = -INFINITY;
            uint32_t pid = 0xffffffffu;
            if (lane < np) { ps = __ldcg(part_s + base + lane); pid = __ldcg(part_id + base + lane); }
            for (int e = 0; e < np; e++) {
              const float ns = __shfl_sync(kFull, ps, e);
              const uint32_t nid = __shfl_sync(kFull, pid, e);
              if (!better(ns, nid, ts, tid_)) break;  // partial lists are sorted
              warp_list_insert(ls, lid, ts, tid_, ns, nid, lane, np);
            }
          }
          if (lane < np) {
            out_id[(size_t)list[t] * nprobe + lane] = lid;
            out_s[(size_t)list[t] * nprobe + lane] = ls;
          }
        }
      }
    }
  }
}

// ---------------------------------------------------------------------
// K2: candidate filter + shortlist, one CTA per query.
//
// Phase A visits the probed lists rank by rank (all tokens' j-th probe, then
// j+1, ...; probes are sorted best-first) so that the first visit of
// (doc, token) carries the max over probes; the rank j is recorded in a
// per-slot byte table rank[doc][token] (0xff = unvisited).  A doc enters the
// candidate set the first time any token visits it (per-slot epoch stamps,
// no O(n_item) reset).  Phase B sums the per-token maxima exactly (2^-32
// fixed point, rounded once to FP32) and restores the touched rank rows to
// 0xff.  Phase C/D radix-select the top
// probe_topk candidates by the 64-bit key (score desc, id asc).
// ---------------------------------------------------------------------
constexpr int kFilterThreads = 1024;
constexpr int kFilterCluster = 4;  // CTAs (SMs) per query of the rank-table filter

// v * 2^32 rounded to nearest-even, clamped to +-2^62 (exact for |v| >= 2^-9):
// the approximate score is the exact sum of these terms, rounded once to FP32
__device__ __forceinline__ long long to_fixed(float v) {
  double x = (double)v * 4294967296.0;
  x = fmin(fmax(x, -4611686018427387904.0), 4611686018427387904.0);
  return __double2ll_rn(x);
}
__device__ __forceinline__ float from_fixed(long long a) {
  return __ll2float_rn(a) * (1.0f / 4294967296.0f);
}

__device__ __forceinline__ uint32_t find_seg(const uint32_t *pref, int n, uint32_t e) {
  // largest i in [0, n) with pref[i] <= e   (pref[0] = 0, non-decreasing)
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (pref[mid] <= e) lo = mid; else hi = mid - 1;
  }
  return (uint32_t)lo;
}

// Cluster form: CL CTAs (one cluster) share one query.  Each CTA takes an
// interleaved share of every rank's list entries, of the candidates and of
// the keys; the candidate counter, the shortlist counter and the radix-select
// histograms are combined through distributed shared memory (CTA 0 holds the
// counters), and cluster barriers order the phases.  Splitting a query over
// CL SMs keeps only n_sm / CL queries' rank rows and stamps in flight, a
// working set that stays in L2.  CL = 1 is the single-CTA kernel.
template <int CL>
__device__ __forceinline__ void filter_sync() {
  if constexpr (CL == 1) {
    __syncthreads();
  } else {
    __threadfence();  // rank bytes / stamps / keys live in global memory
    asm volatile("barrier.cluster.arrive.release.aligned;\n"
                 "barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
  }
}

// the same for data in shared memory alone (cluster-scope ordering)
template <int CL>
__device__ __forceinline__ void cluster_sync() {
  if constexpr (CL == 1) {
    __syncthreads();
  } else {
    asm volatile("barrier.cluster.arrive.release.aligned;\n"
                 "barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
  }
}

template <int CL>
__device__ __forceinline__ uint32_t *cl_ptr(uint32_t *p, uint32_t rank) {
  if constexpr (CL == 1) {
    return p;
  } else {
    uint32_t *r;
    asm volatile("mapa.u64 %0, %1, %2;\n" : "=l"(r) : "l"(p), "r"(rank));
    return r;
  }
}

constexpr int kSelU = 8;  // candidate keys per thread in flight in the select passes

// Shared-memory state of select_emit.
constexpr uint32_t kSelBins = 4096;  // bins of a pass (12 bits of the key)
constexpr uint32_t kSelList = 512;   // keys of the boundary bin that are ranked directly
struct SelectSmem {
  uint32_t *hist;   // [kSelBins]
  uint64_t *list;   // [kSelList], CTA 0's is the cluster's
  uint32_t *wsum;   // [32]
  uint32_t *bin, *need, *cnt, *n_list;
};
constexpr size_t kSelSmem = kSelBins * sizeof(uint32_t) + kSelList * sizeof(uint64_t);

// Phases C/D of the filter: the probe_topk largest 64-bit keys among
// key[0, n_cand) as the (unordered) shortlist of query b.  Radix passes of 12
// bits, high to low, find the bin that the cut falls into, until that bin is
// taken whole or holds at most kSelList keys; the emission pass writes every
// key above it and collects its keys, which are then ranked among themselves.
// Scores take 8 exponent bits, so the first pass spreads them over some 30
// bins: plain shared atomics without the match_any that 8-bit digits needed,
// and usually one pass before the emission instead of three.  With CL > 1 the
// CL CTAs of a cluster each take an interleaved share of the keys and add
// their histograms through distributed shared memory; g_sel / g_stok are CTA
// 0's counters.  Bound: latency, two reads of the keys at one CTA per query.
// 1,184 queries of 31,000 candidates: 465 -> 235 us; one query of 34,000: 64 ->
// 32 us, of 1,065: 15 -> 7 us.
template <int CL>
__device__ void select_emit(const DevIndex &ix, const uint64_t *__restrict__ key, uint32_t n_cand,
                            uint32_t probe_topk, uint32_t b, uint32_t cr, const SelectSmem &sm,
                            uint32_t *g_sel, uint32_t *g_stok, uint32_t *__restrict__ short_id,
                            float *__restrict__ short_approx) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t cstride = CL * kFilterThreads;
  const unsigned lt_mask = (1u << lane) - 1u;
  const bool cut = n_cand > probe_topk;
  uint64_t prefix = 0;
  int shift = 64;  // key bits below the prefix
  bool whole = true;
  uint32_t need = probe_topk;
  if (tid == 0) *sm.n_list = 0;
  // ---- phase C: the bin that holds the cut ----
  while (cut) {
    const int width = min(12, shift);
    const int up = shift;  // prefix = key >> up so far
    shift -= width;
    const uint32_t mask = (1u << width) - 1u;
    for (uint32_t i = tid; i < kSelBins; i += kFilterThreads) sm.hist[i] = 0;
    __syncthreads();
    // kSelU keys per thread in flight
    for (uint32_t i0 = cr * kFilterThreads; i0 < n_cand; i0 += kSelU * cstride) {
      uint64_t kv[kSelU];
#pragma unroll
      for (int u = 0; u < kSelU; u++) {
        const uint32_t i = i0 + u * cstride + tid;
        kv[u] = i < n_cand ? key[i] : 0ull;
      }
#pragma unroll
      for (int u = 0; u < kSelU; u++) {
        const uint32_t i = i0 + u * cstride + tid;
        if (i < n_cand && (up == 64 || (kv[u] >> up) == prefix))
          atomicAdd(&sm.hist[(uint32_t)(kv[u] >> shift) & mask], 1u);
      }
    }
    cluster_sync<CL>();  // every CTA's histogram of this pass complete
    // thread t owns bins 4095 - 4t .. 4092 - 4t (high to low), summed over the cluster
    uint32_t c[4] = {0, 0, 0, 0}, sum = 0;
    for (int r = 0; r < CL; r++) {
      const uint32_t *hr = cl_ptr<CL>(sm.hist, (uint32_t)r);
#pragma unroll
      for (int u = 0; u < 4; u++) c[u] += hr[kSelBins - 1 - 4 * tid - u];
    }
#pragma unroll
    for (int u = 0; u < 4; u++) sum += c[u];
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) sm.wsum[warp] = incl;
    __syncthreads();
    uint32_t above = incl - sum;
    for (int w = 0; w < warp; w++) above += sm.wsum[w];
    if (above < need && need <= above + sum) {
#pragma unroll
      for (int u = 0; u < 4; u++) {
        if (above < need && need <= above + c[u]) {
          *sm.bin = kSelBins - 1 - 4 * tid - u;
          *sm.need = need - above;
          *sm.cnt = c[u];
        }
        above += c[u];
      }
    }
    cluster_sync<CL>();  // the result, and every CTA done with the histograms
    prefix = (prefix << width) | *sm.bin;
    need = *sm.need;
    const uint32_t cnt = *sm.cnt;
    whole = cnt == need;
    if (whole || cnt <= kSelList) break;
  }

  // ---- phase D: emit the shortlist (unordered) ----
  auto emit = [&](bool sel, uint64_t k) {  // whole warps
    const unsigned m = __ballot_sync(kFull, sel);
    if (!m) return;
    uint32_t base = 0;
    if (lane == __ffs(m) - 1) base = atomicAdd(g_sel, (uint32_t)__popc(m));
    base = __shfl_sync(kFull, base, __ffs(m) - 1);
    const uint32_t pos = base + __popc(m & lt_mask);
    if (sel && pos < probe_topk) {
      short_id[(size_t)b * probe_topk + pos] = key_id(k);
      short_approx[(size_t)b * probe_topk + pos] = key_score(k);
    }
  };
  uint64_t *list = cut && !whole ? reinterpret_cast<uint64_t *>(cl_ptr<CL>((uint32_t *)sm.list, 0)) : nullptr;
  uint32_t *g_list = cl_ptr<CL>(sm.n_list, 0);
  if constexpr (CL > 1) cluster_sync<CL>();  // CTA 0's list counter is zero
  for (uint32_t j0 = cr * kFilterThreads; j0 < n_cand; j0 += kSelU * cstride) {
    uint64_t kv[kSelU];
#pragma unroll
    for (int u = 0; u < kSelU; u++) {
      const uint32_t i = j0 + u * cstride + tid;
      kv[u] = i < n_cand ? key[i] : 0ull;
    }
#pragma unroll
    for (int u = 0; u < kSelU; u++) {
      const uint32_t i = j0 + u * cstride + tid;
      const bool in = i < n_cand;
      const uint64_t kp = cut ? kv[u] >> shift : 1ull;
      emit(in && (kp > prefix || (whole && kp == prefix)), kv[u]);
      if (in && list && kp == prefix) list[atomicAdd(g_list, 1u)] = kv[u];
    }
  }
  if (list) cluster_sync<CL>();
  if (list && cr == 0) {  // the `need` largest of the boundary bin's keys
    const uint32_t n = *sm.n_list;
    const uint32_t mine = tid < kSelList ? tid : kSelList;  // kSelList <= kFilterThreads
    if ((uint32_t)(warp * 32) < n) {
      const bool has = mine < n;
      const uint64_t k = has ? sm.list[mine] : 0ull;
      uint32_t rank = 0;
      for (uint32_t i = 0; i < n; i++) rank += sm.list[i] > k ? 1u : 0u;
      emit(has && rank < need, k);
    }
  }
  // tokens of the shortlist (after the emission: a length per emitted key
  // there put a dependent load into every step of it)
  cluster_sync<CL>();
  const uint32_t n_sel = min(*(volatile uint32_t *)g_sel, probe_topk);
  uint32_t len = 0;
  for (uint32_t i = cr * kFilterThreads + tid; i < n_sel; i += cstride)
    len += ix.item_n_vec[__ldcg(short_id + (size_t)b * probe_topk + i)];
  len = __reduce_add_sync(kFull, len);
  if (lane == 0 && len) atomicAdd(g_stok, len);
}

template <int CL>
__global__ void __launch_bounds__(kFilterThreads, 1)
filter_kernel(DevIndex ix, const uint32_t *__restrict__ probe_id,
              const float *__restrict__ probe_s, uint32_t nprobe,
              const uint64_t *__restrict__ q_off, uint32_t probe_topk,
              FilterScratch scr, const uint32_t *__restrict__ epoch_base, uint32_t epoch_add,
              uint32_t *__restrict__ short_id, float *__restrict__ short_approx,
              uint32_t *__restrict__ n_short_out, uint32_t *__restrict__ qstat,
              uint32_t *__restrict__ only_if, int impute) {
  // the probes' scores, offsets and sizes; the select phase reuses their space
  constexpr int kProbes = kMaxQueryTok * kMaxProbe;
  __shared__ __align__(16) unsigned char pool[kProbes * 20];
  static_assert(sizeof(pool) >= kSelSmem, "select state");
  long long *pfix = reinterpret_cast<long long *>(pool);
  uint64_t *lof = reinterpret_cast<uint64_t *>(pool) + kProbes;
  uint32_t *lsz = reinterpret_cast<uint32_t *>(pool) + 4 * kProbes;
  __shared__ long long impf[kMaxQueryTok];  // imputed score of an unmatched token (0: off)
  __shared__ uint32_t pref[kMaxQueryTok + 1];
  __shared__ uint32_t s_ncand, s_sel, s_stok, s_nlist;     // CTA 0's copies are the cluster's
  __shared__ uint32_t s_wsum[32], s_bin, s_need, s_cnt, s_entries;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n_warp = blockDim.x >> 5;
  uint32_t cr = 0;
  if constexpr (CL > 1) asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(cr));
  const uint32_t b = blockIdx.x / CL;
  // fallback use: only the queries whose hash-table filter overflowed (the
  // flag is the same for every CTA of the cluster, read before any barrier;
  // it stays set until the next batch's hash filter clears it)
  if (only_if && only_if[b] == 0) return;
  // stamp epoch of this launch: a device counter (so that a replayed CUDA
  // graph sees a fresh epoch) plus the caller's offset
  const uint32_t epoch = (epoch_base ? *epoch_base : 0u) + epoch_add;
  const uint64_t tok0 = q_off[b];
  const uint32_t nq = (uint32_t)(q_off[b + 1] - tok0);
  uint32_t *stamp = scr.stamp + (size_t)b * scr.n_item;
  uint8_t *rank = scr.rank + (size_t)b * scr.n_item * scr.rank_stride;
  uint64_t *key = scr.key + (size_t)b * scr.n_item;
  uint32_t *g_ncand = cl_ptr<CL>(&s_ncand, 0), *g_sel = cl_ptr<CL>(&s_sel, 0),
           *g_stok = cl_ptr<CL>(&s_stok, 0);
  const unsigned lt_mask = (1u << lane) - 1u;

  // probe scores (fixed point) and list sizes / offsets of every probe
  // (probe id 0xffffffff = no finite score)
  for (uint32_t i = tid; i < nq * nprobe; i += blockDim.x) {
    const uint32_t c = probe_id[tok0 * nprobe + i];
    pfix[i] = to_fixed(probe_s[tok0 * nprobe + i]);
    lsz[i] = c < ix.n_centroid ? ix.ivf_size[c] : 0u;
    lof[i] = c < ix.n_centroid ? ix.ivf_off[c] : 0ull;
  }
  for (uint32_t t = tid; t < nq; t += blockDim.x)
    impf[t] = impute ? to_fixed(probe_s[(tok0 + t) * nprobe + nprobe - 1]) : 0ll;
  if (tid == 0) { s_ncand = 0; s_sel = 0; s_stok = 0; s_entries = 0; }
  filter_sync<CL>();  // counters of CTA 0 initialised before any remote update

  // ---- phase A: scatter probed lists rank by rank ----
  const uint32_t gwarp = cr * n_warp + warp, gstride = CL * n_warp * 128;
  for (uint32_t j = 0; j < nprobe; j++) {
    if (warp == 0) {  // exclusive prefix of the nq list sizes of rank j
      const uint32_t s0 = (uint32_t)lane < nq ? lsz[lane * nprobe + j] : 0u;
      const uint32_t s1 = (uint32_t)lane + 32 < nq ? lsz[(lane + 32) * nprobe + j] : 0u;
      uint32_t i0 = s0, i1 = s1;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v0 = __shfl_up_sync(kFull, i0, o), v1 = __shfl_up_sync(kFull, i1, o);
        if (lane >= o) { i0 += v0; i1 += v1; }
      }
      const uint32_t tot0 = __shfl_sync(kFull, i0, 31);
      if ((uint32_t)lane < nq) pref[lane] = i0 - s0;
      if ((uint32_t)lane + 32 < nq) pref[lane + 32] = tot0 + i1 - s1;
      if (lane == 31) {
        const uint32_t total = tot0 + i1;
        pref[nq] = total;
        s_entries += total;
      }
    }
    __syncthreads();
    const uint32_t total = pref[nq];
    // 4 entries per lane in flight: independent list-id and rank-byte loads
    for (uint32_t e0 = gwarp * 128; e0 < total; e0 += gstride) {
      uint32_t item[4], tt[4];
      uint8_t rv[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const uint32_t e = e0 + u * 32 + lane;
        tt[u] = 0xffffffffu;
        if (e < total) {
          const uint32_t t = find_seg(pref, (int)nq, e);
          tt[u] = t;
          item[u] = ix.ivf_ids[lof[t * nprobe + j] + (e - pref[t])];
        }
      }
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (tt[u] != 0xffffffffu) rv[u] = rank[(size_t)item[u] * scr.rank_stride + tt[u]];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        bool fresh = false;
        if (tt[u] != 0xffffffffu && rv[u] == 0xff) {
          rank[(size_t)item[u] * scr.rank_stride + tt[u]] = (uint8_t)j;
          fresh = atomicExch(stamp + item[u], epoch) != epoch;
        }
        // warp-aggregated append to the cluster's candidate list
        const unsigned m = __ballot_sync(kFull, fresh);
        if (m) {
          uint32_t base = 0;
          if (lane == __ffs(m) - 1) base = atomicAdd(g_ncand, (uint32_t)__popc(m));
          base = __shfl_sync(kFull, base, __ffs(m) - 1);
          if (fresh) key[base + __popc(m & lt_mask)] = item[u];
        }
      }
    }
    filter_sync<CL>();
  }
  const uint32_t n_cand = *g_ncand;

  // ---- phase B: approximate score, restore rank rows (2 candidates in flight) ----
  const uint32_t cstride = CL * blockDim.x;
  for (uint32_t i0 = cr * blockDim.x + tid; i0 < n_cand; i0 += 2 * cstride) {
    long long ps_acc[2] = {0, 0};
    uint32_t item[2];
    uint8_t *row[2];
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const uint32_t i = i0 + u * cstride;
      item[u] = i < n_cand ? (uint32_t)key[i] : 0u;
      row[u] = rank + (size_t)item[u] * scr.rank_stride;
    }
    for (uint32_t t0 = 0; t0 < nq; t0 += 16) {
      uint4 w[2];
#pragma unroll
      for (int u = 0; u < 2; u++)
        if (i0 + u * cstride < n_cand) w[u] = *reinterpret_cast<uint4 *>(row[u] + t0);
#pragma unroll
      for (int u = 0; u < 2; u++) {
        if (i0 + u * cstride >= n_cand) continue;
        const uint8_t *bytes = reinterpret_cast<const uint8_t *>(&w[u]);
        long long s = ps_acc[u];
#pragma unroll
        for (int v = 0; v < 16; v++) {
          const uint32_t t = t0 + v;
          if (t < nq) s += bytes[v] != 0xff ? pfix[t * nprobe + bytes[v]] : impf[t];
        }
        ps_acc[u] = s;
        *reinterpret_cast<uint4 *>(row[u] + t0) = make_uint4(~0u, ~0u, ~0u, ~0u);
      }
    }
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const uint32_t i = i0 + u * cstride;
      if (i < n_cand) key[i] = make_key(from_fixed(ps_acc[u]), item[u]);
    }
  }
  filter_sync<CL>();

  // ---- phases C/D: radix select + emit ----
  SelectSmem sm{reinterpret_cast<uint32_t *>(pool),
                reinterpret_cast<uint64_t *>(pool) + kSelBins / 2, s_wsum, &s_bin, &s_need, &s_cnt,
                &s_nlist};
  select_emit<CL>(ix, key, n_cand, probe_topk, b, cr, sm, g_sel, g_stok, short_id, short_approx);
  filter_sync<CL>();
  if (cr == 0 && tid == 0) {
    n_short_out[b] = min(s_sel, probe_topk);
    qstat[b * 3 + 0] = n_cand;
    qstat[b * 3 + 1] = s_entries;
    qstat[b * 3 + 2] = s_stok;
  }
}

// ---------------------------------------------------------------------
// Hash-table filter (main search path).  P = hash_parts(...) CTAs
// share a query; CTA p owns the docs [p * n_item / P, (p + 1) * n_item / P) and keeps one
// shared-memory hash-table slot per candidate doc of its range: doc id, the
// mask of query tokens that have visited it and the exact fixed-point sum of
// the first-visit probe scores.  The IVF lists are sorted by doc id, so the
// CTA's part of each probed list is the contiguous sub-list given by the
// index's partition table (ivf_part).  Warp w walks token w's sub-lists in
// probe-rank order (probes are sorted best-first), so the token's first
// visit of a doc carries the max over its probes; different tokens only meet
// in the order-free atomics (OR of the mask, integer add of the score).
// score = sum over tokens of those maxima, the same value the rank-table
// filter computes.  Each candidate's 64-bit (score, id) key goes to the
// query's key array, from which filter_select_kernel takes the shortlist.  A
// CTA whose range holds more than kHashFill candidates marks the query in
// scr.ovf and the rank-table filter redoes that query.
// ---------------------------------------------------------------------
constexpr uint32_t kHashLog = 13, kHashCap = 1u << kHashLog;  // slots per CTA
static_assert(kHashFill + 1024 <= kHashCap, "the fill limit must keep >= 1024 slots empty");
constexpr uint32_t kEmpty = 0xffffffffu;

__host__ __device__ constexpr size_t hash_smem_bytes(int mw) {
  return (size_t)kHashCap * (4 + 4 * mw + 8);
}

template <int MW>
__global__ void __launch_bounds__(kFilterThreads, 1)
filter_hash_kernel(DevIndex ix, const uint32_t *__restrict__ probe_id,
                   const float *__restrict__ probe_s, uint32_t nprobe,
                   const uint64_t *__restrict__ q_off, const uint64_t *__restrict__ cta_off,
                   uint32_t n_query, FilterScratch scr, uint32_t *__restrict__ qstat, int impute) {
  extern __shared__ __align__(16) uint8_t hsm[];
  uint32_t *tkey = reinterpret_cast<uint32_t *>(hsm);                      // [cap]
  uint32_t *tmask = tkey + kHashCap;                                       // [cap][MW]
  unsigned long long *tacc = reinterpret_cast<unsigned long long *>(tmask + kHashCap * MW);
  __shared__ long long pfix[kMaxQueryTok * kMaxProbe];
  __shared__ uint32_t lsz[kMaxQueryTok * kMaxProbe];   // this CTA's sub-list sizes
  __shared__ uint64_t lof[kMaxQueryTok * kMaxProbe];   // and offsets in ivf_ids
  __shared__ long long impf[kMaxQueryTok];  // imputed score of an unmatched token (0: off)
  __shared__ long long s_imp;               // sum of impf over the query's tokens
  __shared__ uint32_t s_fill, s_ovf, s_entries, s_b, s_kbase;
  __shared__ uint32_t s_wsum[32];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n_warp = blockDim.x >> 5;
  // this CTA's query and doc range: cta_off[b] <= blockIdx.x < cta_off[b + 1]
  for (uint32_t i = tid; i < n_query; i += blockDim.x)
    if (cta_off[i] <= blockIdx.x && blockIdx.x < cta_off[i + 1]) s_b = i;
  __syncthreads();
  const uint32_t b = s_b;
  const uint32_t part = blockIdx.x - (uint32_t)cta_off[b];
  const uint32_t pstep = (uint32_t)kHashParts / (uint32_t)(cta_off[b + 1] - cta_off[b]);
  const uint64_t tok0 = q_off[b];
  const uint32_t nq = (uint32_t)(q_off[b + 1] - tok0);

  {  // 16-byte stores: keys empty, masks and scores 0
    uint4 *t4 = reinterpret_cast<uint4 *>(hsm);
    constexpr uint32_t kKeys4 = kHashCap / 4, kAll4 = (uint32_t)(hash_smem_bytes(MW) / 16);
    for (uint32_t i = tid; i < kAll4; i += kFilterThreads) {
      const uint32_t x = i < kKeys4 ? kEmpty : 0u;
      t4[i] = make_uint4(x, x, x, x);
    }
  }
  if (tid == 0) { s_fill = 0; s_ovf = 0; s_entries = 0; }
  for (uint32_t t = tid; t < nq; t += blockDim.x)
    impf[t] = impute ? to_fixed(probe_s[(tok0 + t) * nprobe + nprobe - 1]) : 0ll;
  __syncthreads();
  if (tid == 0) {  // fixed order: the same integer in every CTA
    long long a = 0;
    for (uint32_t t = 0; t < nq; t++) a += impf[t];
    s_imp = a;
  }
  uint32_t ent = 0;
  for (uint32_t i = tid; i < nq * nprobe; i += blockDim.x) {
    const uint32_t c = probe_id[tok0 * nprobe + i];
    pfix[i] = to_fixed(probe_s[tok0 * nprobe + i]);
    uint32_t p0 = 0, p1 = 0;
    uint64_t o = 0;
    if (c < ix.n_centroid) {
      const uint32_t *pt = ix.ivf_part + (size_t)c * (kHashParts + 1) + part * pstep;
      p0 = pt[0];
      p1 = pt[pstep];
      o = ix.ivf_off[c];
      ent += ix.ivf_size[c];
    }
    lsz[i] = p1 - p0;
    lof[i] = o + p0;
  }
  if (part == 0) {
    ent = __reduce_add_sync(kFull, ent);
    if (lane == 0 && ent) atomicAdd(&s_entries, ent);
  }
  __syncthreads();

  for (uint32_t t = warp; t < nq; t += n_warp) {
    const uint32_t bit = 1u << (t & 31), word = t >> 5;
    for (uint32_t j = 0; j < nprobe; j++) {
      const uint32_t sz = lsz[t * nprobe + j];
      const uint32_t *ids = ix.ivf_ids + lof[t * nprobe + j];
      // first visit: the probe score replaces the token's imputed score
      const unsigned long long add = (unsigned long long)(pfix[t * nprobe + j] - impf[t]);
      // 4 entries per lane in flight (the loads are independent; the
      // entries of one probe carry the same score, so their order is free)
      for (uint32_t p0 = 0; p0 < sz; p0 += 128) {
        // a CTA past its fill limit stops: its query is redone by the
        // rank-table filter
        if (__any_sync(kFull, *reinterpret_cast<volatile uint32_t *>(&s_ovf) != 0u)) break;
        uint32_t its[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const uint32_t p = p0 + lane + 32u * u;
          its[u] = p < sz ? __ldg(ids + p) : kEmpty;
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
          // a range's share of a list is often shorter than a round (50 entries
          // of 128 at 1M docs, 65,536 lists and 8 ranges): stop where it ends
          if (p0 + 32u * u >= sz) break;
          const uint32_t it = its[u];
          // find or insert `it` (linear probing; the walk is bounded by the
          // table size, and a CTA stops inserting once its fill count passes
          // the limit)
          uint32_t slot = kEmpty;
          bool inserted = false;
          if (it != kEmpty) {
            uint32_t h = (it * 2654435769u) >> (32 - kHashLog);
            for (uint32_t step = 0; step < kHashCap; step++) {
              const uint32_t k = *reinterpret_cast<volatile uint32_t *>(&tkey[h]);
              if (k == it) { slot = h; break; }
              if (k == kEmpty) {
                const uint32_t old = atomicCAS(&tkey[h], kEmpty, it);
                if (old == kEmpty) { slot = h; inserted = true; break; }
                if (old == it) { slot = h; break; }
              }
              h = (h + 1) & (kHashCap - 1);
            }
            if (slot == kEmpty) s_ovf = 1;  // the table is full
          }
          // the fill count (distinct docs inserted): one shared atomic per
          // warp and round instead of one per insert on a single address
          const unsigned ins = __ballot_sync(kFull, inserted);
          if (lane == 0 && ins) {
            const uint32_t n = (uint32_t)__popc(ins);
            if (atomicAdd(&s_fill, n) + n > kHashFill) s_ovf = 1;
          }
          if (slot == kEmpty) continue;
          const uint32_t old = atomicOr(&tmask[slot * MW + word], bit);
          if (!(old & bit)) atomicAdd(&tacc[slot], add);
        }
      }
      __syncwarp();  // rank j of token t before rank j + 1
    }
  }
  __syncthreads();

  // emit this CTA's candidates as (score, id) keys (at most kHashFill per CTA:
  // an overflowed CTA emits none, its query is redone by the rank-table
  // filter).  One global atomic per CTA reserves the CTA's key range: each
  // thread counts its slots (tid, tid + blockDim, ...), a block scan gives
  // its offset, and it writes its keys there.
  uint64_t *key = scr.hkey + (size_t)b * scr.key_stride;
  if (!s_ovf) {
    uint32_t mine = 0;
    for (uint32_t sl = tid; sl < kHashCap; sl += blockDim.x) mine += tkey[sl] != kEmpty ? 1u : 0u;
    uint32_t inc = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(kFull, inc, o);
      if (lane >= o) inc += v;
    }
    if (lane == 31) s_wsum[warp] = inc;
    __syncthreads();
    if (warp == 0) {
      uint32_t w = lane < n_warp ? s_wsum[lane] : 0u, wi = w;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(kFull, wi, o);
        if (lane >= o) wi += v;
      }
      if (lane < n_warp) s_wsum[lane] = wi - w;  // exclusive warp offsets
      if (lane == 31) s_kbase = wi ? atomicAdd(scr.qcnt + b, wi) : 0u;
    }
    __syncthreads();
    uint32_t pos = s_kbase + s_wsum[warp] + inc - mine;
    for (uint32_t sl = tid; sl < kHashCap; sl += blockDim.x) {
      const uint32_t k = tkey[sl];
      if (k != kEmpty) key[pos++] = make_key(from_fixed((long long)tacc[sl] + s_imp), k);
    }
  }
  if (tid == 0) {
    if (s_ovf) atomicOr(scr.ovf + b, 1u);
    if (part == 0) qstat[b * 3 + 1] = s_entries;
  }
}

// ivf_part[c][p] = first position of list c whose doc id is >= p * n_item / P
// (p = 0..P): the doc-range sub-lists of the hash filter.
__global__ void ivf_part_kernel(const uint64_t *__restrict__ ivf_off,
                                const uint32_t *__restrict__ ivf_size,
                                const uint32_t *__restrict__ ivf_ids, uint32_t n_cent,
                                uint32_t n_item, uint32_t *__restrict__ out) {
  const size_t n = (size_t)n_cent * (kHashParts + 1);
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const uint32_t c = (uint32_t)(i / (kHashParts + 1)), p = (uint32_t)(i % (kHashParts + 1));
    const uint32_t bound = (uint32_t)((uint64_t)p * n_item / kHashParts);
    const uint32_t *l = ivf_ids + ivf_off[c];
    uint32_t lo = 0, hi = ivf_size[c];
    while (lo < hi) {
      const uint32_t mid = (lo + hi) >> 1;
      if (l[mid] < bound) lo = mid + 1; else hi = mid;
    }
    out[i] = lo;
  }
}

cudaError_t make_ivf_part(const DevIndex &ix, uint32_t *out, cudaStream_t st) {
  ivf_part_kernel<<<592, 256, 0, st>>>(ix.ivf_off, ix.ivf_size, ix.ivf_ids, ix.n_centroid,
                                       ix.n_item, out);
  return cudaGetLastError();
}

// Shortlist of every query from the keys filter_hash_kernel emitted; resets
// the query's key counter for the next batch and advances the fallback's stamp
// epoch by the launches that may follow.
__global__ void __launch_bounds__(kFilterThreads, 1)
filter_select_kernel(DevIndex ix, uint32_t probe_topk, FilterScratch scr,
                     uint32_t *__restrict__ short_id, float *__restrict__ short_approx,
                     uint32_t *__restrict__ n_short_out, uint32_t *__restrict__ qstat,
                     uint32_t *__restrict__ epoch, uint32_t n_epoch) {
  __shared__ __align__(16) uint32_t hist[kSelBins];
  __shared__ __align__(16) uint64_t list[kSelList];
  __shared__ uint32_t s_wsum[32], s_sel, s_stok, s_bin, s_need, s_cnt, s_nlist;
  const uint32_t b = blockIdx.x;
  const uint32_t n_cand = scr.qcnt[b];
  if (threadIdx.x == 0) { s_sel = 0; s_stok = 0; }
  __syncthreads();
  SelectSmem sm{hist, list, s_wsum, &s_bin, &s_need, &s_cnt, &s_nlist};
  select_emit<1>(ix, scr.hkey + (size_t)b * scr.key_stride, n_cand, probe_topk, b, 0, sm, &s_sel,
                 &s_stok, short_id, short_approx);
  __syncthreads();
  if (threadIdx.x == 0) {
    n_short_out[b] = min(s_sel, probe_topk);
    qstat[b * 3 + 0] = n_cand;
    qstat[b * 3 + 2] = s_stok;
    scr.qcnt[b] = 0;
    if (b == 0) *epoch += n_epoch;  // the rank-table fallback's, which runs next
  }
}

// ---------------------------------------------------------------------
// K3: decompress + exact MaxSim of up to kRkDocs shortlisted docs of one query.
//
// The docs' tokens, doc after doc, form a stream of 128-token tiles; each of
// the CTA's 4 warps takes every 4th tile and works alone (no barrier inside a
// tile).  Lane l owns the tile's tokens l, l + 32, l + 64, l + 96 and all
// query tokens of the pass (16 or 32): it decodes its own tokens in registers,
// x = centroid + W[bucket] (one rounded FP32 add), and accumulates them with
// fma.rn.f32x2, two query tokens per instruction (each half a rounded FP32
// fma, so every dot product is the sequential __fmaf_rn chain over
// d = 0..127 from 0.0f and the scores are bit-identical to the canonical
// arithmetic).  Per dimension a lane reads NQ query values (broadcast
// LDS.128) for 4 NQ FMAs.
//
// Centroid rows come through shared memory in chunks of 16 dimensions, two
// stages per warp: 4 lanes copy a token's 64 bytes (cp.async), so a copy
// instruction touches 8 cache lines instead of the 32 of a row per lane, and
// the 16-byte parts are swizzled so that both the copies and the lanes' reads
// of their own rows spread over all banks.  Residual bytes (one load per
// token and chunk) are in registers a chunk ahead, the next tile's codes two
// chunks ahead.
//
// With KT = 1 a tile is 32 tokens, one per lane, whose centroid rows come at once
// (8 chunks in the space of 2 of 128 tokens): the short chain of a small grid.
//
// After a tile: per doc of the tile, the max over the lane's tokens of that
// doc and a REDUX over the warp for every query token, folded into
// best[doc][query token] by atomicMax.  Queries of more than 32 tokens run in
// two passes; a pass of at most 16 query tokens takes the 16-wide body.
//
// Bound: the FMA pipe (a token of a 32-token query is 32 cycles of an SM's 128
// lanes), 60 % busy by the counters at 2 warps per scheduler and 255
// registers; three warps of 3 tokens per lane spilled (12.2 ms where this
// takes 8.8).  400 queries x 1500 docs of 70 tokens, 2 bits: 12.8 ms with
// scalar FFMA and separate decoder warps -> 8.8 ms, 39 TFLOP/s.
// ---------------------------------------------------------------------
constexpr int kRkDocs = 64;       // most shortlisted docs per CTA
constexpr int kRkT = 4;           // doc tokens per lane (KT = 1: 1)
constexpr int kRkTile = 32 * kRkT;  // doc tokens per warp and tile
constexpr int kRkChunk = 16;      // dimensions per stage
constexpr int kRkStages = 2;
constexpr int kRkQ = 32;          // query tokens per pass
constexpr int kRkWarps = 4;
constexpr int kRkThreads = 32 * kRkWarps;  // two CTAs per SM, up to 255 registers a thread
constexpr int kRkNch = kDim / kRkChunk;    // chunks per tile

// copies of the weight table, so that lanes reading different weights of a
// large table meet fewer bank conflicts (1 is conflict-free up to 32 entries)
__host__ __device__ constexpr int rk_wcopies(int n_bit) { return n_bit <= 4 ? 1 : 8; }

__host__ __device__ constexpr size_t rk_smem_bytes(int n_bit) {
  return (size_t)kRkWarps * kRkStages * kRkTile * kRkChunk * sizeof(float) +  // centroid chunks
         (size_t)kDim * kRkQ * sizeof(float) +                                // query tokens
         (size_t)(1 << n_bit) * rk_wcopies(n_bit) * sizeof(float) +           // weights
         (size_t)kRkDocs * (kRkQ + 1) * sizeof(int);                          // best[doc][q]
}

// 4-dimension groups of a chunk per loop body.  All four unrolled miss the
// instruction cache at 1 and 2 bits (400 queries x 1500 docs at 2 bits: 9.2,
// 8.8 and 9.6 ms with 1, 2 and 4 groups a body), two spill at 4 bits (600
// queries x 40 docs: 1.32, 1.59, 1.35 ms), and at 8 bits only the unrolled
// form knows which register a group's codes are in (200 x 400: 2.12, 2.12, 1.79 ms).
__host__ __device__ constexpr int rk_unroll(int n_bit) { return n_bit <= 2 ? 2 : n_bit == 4 ? 1 : 4; }

__device__ __forceinline__ uint64_t dup_f32x2(float x) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %1};\n" : "=l"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// What a warp needs of its CTA's docs and buffers (shared memory).
struct RkCta {
  const float *Qs;         // [128 dims][32 query tokens]
  const float *wtab;       // [2^NBIT][copies]
  float *xs;               // this warp's stages [kRkStages][128 tokens][16 dims], swizzled
  uint32_t *codes;         // this warp's vq codes [2 tile parities][kRkTile]
  uint64_t *toks;          // ... and token indexes
  int *best;               // [kRkDocs][kRkQ + 1]
  const uint32_t *d_pref;  // [nd + 1] token offsets of the docs
  const uint64_t *d_off;   // [nd] first token of each doc
  uint32_t nd, T;          // docs and tokens of the CTA
};

// One pass of one warp over its tiles: NQ query tokens (rows 0 .. NQ - 1 of Qs).
template <int NBIT, int NQ, int KT>
__device__ __forceinline__ void rk_warp_pass(const DevIndex &ix, const RkCta &c, uint32_t nq_pass) {
  constexpr int CB = kRkChunk * NBIT / 8;  // residual bytes per token and chunk
  constexpr int RW = (CB + 3) / 4;         // ... in 32-bit words
  constexpr uint32_t MASK = (1u << NBIT) - 1u;
  constexpr int TILE = 32 * KT;
  static_assert(KT == kRkT || kRkStages * kRkT == kRkNch * KT,
                "chunks in two stages, or a whole tile of rows at once");
  constexpr int WC = rk_wcopies(NBIT);
  const int lane = threadIdx.x & 31;
  const uint32_t warp = threadIdx.x >> 5;
  const uint32_t n_tiles = (c.T + TILE - 1) / TILE;
  if (warp >= n_tiles) return;
  const float *wt = c.wtab + (lane & (WC - 1));

  uint32_t docs4 = 0, docs4_n = 0;  // doc of each of the lane's tokens, a byte each (255: none)
  // tile tl's tokens of this lane into the buffers of parity pr (the codes by
  // cp.async); past the last token: the last one again (loaded, never counted)
  auto locate = [&](uint32_t tl, uint32_t pr) {
    docs4_n = 0;
#pragma unroll
    for (int j = 0; j < KT; j++) {
      const uint32_t g = TILE * tl + 32u * j + lane, gt = min(g, c.T - 1u);
      const uint32_t d = find_seg(c.d_pref, (int)c.nd, gt);
      docs4_n |= (g < c.T ? d : 255u) << (8 * j);
      const uint64_t v = c.d_off[d] + (gt - c.d_pref[d]);
      c.toks[pr * TILE + 32 * j + lane] = v;
      cp_async4(&c.codes[pr * TILE + 32 * j + lane], ix.vq_code + v);
    }
    cp_async_commit();
  };
  uint32_t res[KT][RW], res_n[KT][RW];
  auto load_res = [&](uint32_t ch, uint32_t pr) {
#pragma unroll
    for (int j = 0; j < KT; j++) {
      const uint8_t *rp =
          ix.residual + c.toks[pr * TILE + 32 * j + lane] * (kDim * NBIT / 8) + ch * CB;
      if constexpr (CB == 2) {
        res_n[j][0] = __ldg(reinterpret_cast<const unsigned short *>(rp));
      } else if constexpr (CB == 4) {
        res_n[j][0] = __ldg(reinterpret_cast<const uint32_t *>(rp));
      } else if constexpr (CB == 8) {
        const uint2 t = __ldg(reinterpret_cast<const uint2 *>(rp));
        res_n[j][0] = t.x;
        res_n[j][1] = t.y;
      } else {
        const uint4 t = __ldg(reinterpret_cast<const uint4 *>(rp));
        res_n[j][0] = t.x;
        res_n[j][1] = t.y;
        res_n[j][2] = t.z;
        res_n[j][3] = t.w;
      }
    }
  };
  // chunk ch of the tile of parity pr into stage st: lane copies 16-byte part
  // lane % 4 of tokens lane / 4, lane / 4 + 8, ...
  auto copy_chunk = [&](uint32_t ch, uint32_t pr, uint32_t st) {
    const uint32_t part = lane & 3u;
    float *dst = c.xs + st * (TILE * kRkChunk);
    const float *src = ix.centroid + ch * kRkChunk + part * 4u;
#pragma unroll
    for (int i = 0; i < TILE / 8; i++) {
      const uint32_t p = 8u * i + (lane >> 2);
      const uint32_t cd = c.codes[pr * TILE + p];
      cp_async16(dst + p * kRkChunk + ((part ^ ((p >> 1) & 3u)) << 2), src + (size_t)cd * kDim);
    }
    cp_async_commit();
  };

  locate(warp, 0);
  cp_async_wait<0>();
  __syncwarp();
  auto copy_first = [&](uint32_t pr, uint32_t st) {  // of a tile: a chunk, or all of them
    if constexpr (KT == kRkT) {
      copy_chunk(0, pr, st);
    } else {
#pragma unroll
      for (uint32_t ch = 0; ch < (uint32_t)kRkNch; ch++) copy_chunk(ch, pr, ch);
    }
    load_res(0, pr);
  };
  copy_first(0, 0);
  uint32_t par = 0;
  for (uint32_t tl = warp; tl < n_tiles; tl += kRkWarps) {
    const bool more = tl + kRkWarps < n_tiles;
    docs4 = docs4_n;
    uint64_t acc[NQ / 2][KT];
#pragma unroll
    for (int i = 0; i < NQ / 2; i++)
#pragma unroll
      for (int j = 0; j < KT; j++) acc[i][j] = 0ull;
#pragma unroll 1
    for (uint32_t ch = 0; ch < (uint32_t)kRkNch; ch++) {
#pragma unroll
      for (int j = 0; j < KT; j++)
#pragma unroll
        for (int w = 0; w < RW; w++) res[j][w] = res_n[j][w];
      const uint32_t st = KT == kRkT ? ch & 1u : ch;
      if (KT == kRkT || ch == 0) {
        cp_async_wait<0>();
        __syncwarp();  // chunk ch landed for every lane; every lane is done with the other stage
      }
      if (ch + 1 < (uint32_t)kRkNch) {
        if constexpr (KT == kRkT) copy_chunk(ch + 1, par, st ^ 1u);
        load_res(ch + 1, par);
        if (ch == (KT == kRkT ? kRkNch - 2 : 0) && more) locate(tl + kRkWarps, par ^ 1u);
      } else if (KT == kRkT && more) {
        par ^= 1u;
        copy_first(par, st ^ 1u);
      }
      const float *xr = c.xs + st * (TILE * kRkChunk) + lane * kRkChunk;
      const float *qr = c.Qs + ch * (kRkChunk * kRkQ);
#pragma unroll rk_unroll(NBIT)
      for (int g = 0; g < kRkChunk / 4; g++) {
        float x[KT][4];  // [token][dim of the group]
#pragma unroll
        for (int j = 0; j < KT; j++) {
          // token 32 j + lane: (p >> 1) & 3 is (lane >> 1) & 3
          const float4 v = *reinterpret_cast<const float4 *>(
              xr + j * 32 * kRkChunk + (((uint32_t)g ^ ((lane >> 1) & 3u)) << 2));
          const float cv[4] = {v.x, v.y, v.z, v.w};
          // the group's 4 codes: bytes in order, most significant bits first
          uint32_t bits;
          if constexpr (NBIT == 1) bits = (res[j][0] >> (8 * (g >> 1) + 4 - 4 * (g & 1))) & 15u;
          else if constexpr (NBIT == 2) bits = (res[j][0] >> (8 * g)) & 255u;
          else if constexpr (NBIT == 4) bits = (g & 2 ? res[j][1] : res[j][0]) >> (16 * (g & 1));
          else bits = g & 2 ? (g & 1 ? res[j][3] : res[j][2]) : (g & 1 ? res[j][1] : res[j][0]);
#pragma unroll
          for (int u = 0; u < 4; u++) {
            const int gbit = NBIT == 1 ? 3 - u : 8 * (u * NBIT / 8) + 8 - NBIT * (u % (8 / NBIT) + 1);
            x[j][u] = __fadd_rn(cv[u], wt[((bits >> gbit) & MASK) * WC]);
          }
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
          uint64_t xx[KT];
#pragma unroll
          for (int j = 0; j < KT; j++) xx[j] = dup_f32x2(x[j][u]);
          const ulonglong2 *qp = reinterpret_cast<const ulonglong2 *>(qr + (4 * g + u) * kRkQ);
#pragma unroll
          for (int i = 0; i < NQ / 4; i++) {
            const ulonglong2 a = qp[i];
#pragma unroll
            for (int j = 0; j < KT; j++) {
              acc[2 * i][j] = fma_f32x2(a.x, xx[j], acc[2 * i][j]);
              acc[2 * i + 1][j] = fma_f32x2(a.y, xx[j], acc[2 * i + 1][j]);
            }
          }
        }
      }
    }
    if (KT != kRkT && more) {
      par ^= 1u;
      cp_async_wait<0>();
      __syncwarp();  // the next tile's codes landed; every lane is done with this one's rows
      copy_first(par, 0);
    }
    // per doc of the tile: max over its tokens for every query token (lane q
    // ends up with query token q's)
    uint32_t d = __reduce_min_sync(kFull, docs4 & 0xffu);
    const uint32_t d_last = find_seg(c.d_pref, (int)c.nd, min(c.T, TILE * (tl + 1)) - 1u);
#pragma unroll 1
    for (; d <= d_last; d++) {
      bool in[KT];
#pragma unroll
      for (int j = 0; j < KT; j++) in[j] = ((docs4 >> (8 * j)) & 0xffu) == d;
      int mine = f2si(-INFINITY);
#pragma unroll
      for (int i = 0; i < NQ / 2; i++) {
        int lo = f2si(-INFINITY), hi = lo;
#pragma unroll
        for (int j = 0; j < KT; j++) {
          if (in[j]) {
            lo = max(lo, f2si(__uint_as_float((uint32_t)acc[i][j])));
            hi = max(hi, f2si(__uint_as_float((uint32_t)(acc[i][j] >> 32))));
          }
        }
        lo = __reduce_max_sync(kFull, lo);
        hi = __reduce_max_sync(kFull, hi);
        mine = lane == 2 * i ? lo : lane == 2 * i + 1 ? hi : mine;
      }
      if ((uint32_t)lane < nq_pass) atomicMax(&c.best[d * (kRkQ + 1) + lane], mine);
    }
  }
}

template <int NBIT, int KT>
__global__ void __launch_bounds__(kRkThreads, 2)
rerank_kernel(DevIndex ix, const float *__restrict__ q, const uint64_t *__restrict__ q_off,
              const uint32_t *__restrict__ short_id, const uint32_t *__restrict__ n_short,
              uint32_t probe_topk, uint32_t docs, int semantics, float *__restrict__ exact) {
  constexpr int VPB = 8 / NBIT;  // values per residual byte
  constexpr int WC = rk_wcopies(NBIT);
  extern __shared__ __align__(16) float smem[];
  float *xs = smem;                                             // [warps][stages][128][16]
  float *Qs = xs + kRkWarps * kRkStages * kRkTile * kRkChunk;   // [128 dims][32 query tokens]
  float *wtab = Qs + kDim * kRkQ;                               // [2^NBIT][WC]
  int *best = reinterpret_cast<int *>(wtab + (1 << NBIT) * WC);  // [kRkDocs][33]
  __shared__ uint32_t d_len[kRkDocs], d_pref[kRkDocs + 1];
  __shared__ uint64_t d_off[kRkDocs];
  __shared__ uint32_t codes[kRkWarps][2 * kRkTile];
  __shared__ uint64_t toks[kRkWarps][2 * kRkTile];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t b = blockIdx.y;
  const uint32_t ns = n_short[b];
  const uint32_t d0 = blockIdx.x * docs;
  if (d0 >= ns) return;
  const uint32_t nd = min(docs, ns - d0);
  const uint64_t tok0 = q_off[b];
  const uint32_t nq = (uint32_t)(q_off[b + 1] - tok0);

  if (tid < (int)nd) {
    const uint32_t it = short_id[(size_t)b * probe_topk + d0 + tid];
    d_len[tid] = ix.item_n_vec[it];
    d_off[tid] = ix.item_off[it];
  }
  for (int i = tid; i < (1 << NBIT) * WC; i += kRkThreads) {
    // bucket v sits in the top NBIT bits of byte v << (8 - NBIT), position 0
    const uint32_t v = (uint32_t)i / WC;
    wtab[i] = ix.lut[((v << (8 - NBIT)) & 0xffu) * VPB];
  }
  __syncthreads();
  if (warp == 0) {  // token offsets of the docs (warp scan)
    uint32_t carry = 0;
    if (lane == 0) d_pref[0] = 0;
    for (uint32_t base = 0; base < nd; base += 32) {
      uint32_t v = base + lane < nd ? d_len[base + lane] : 0u;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(kFull, v, o);
        if (lane >= o) v += t;
      }
      if (base + lane < nd) d_pref[base + lane + 1] = carry + v;
      carry += __shfl_sync(kFull, v, 31);
    }
  }
  const RkCta cta{Qs, wtab, xs + warp * (kRkStages * kRkTile * kRkChunk), codes[warp], toks[warp],
                  best, d_pref, d_off, nd, 0u};
  float sum = 0.0f;  // doc tid's score so far (token order)
  for (uint32_t t0 = 0; t0 < nq; t0 += kRkQ) {
    const uint32_t np = min((uint32_t)kRkQ, nq - t0);
    // query tokens t0 .. t0 + 31 -> Qs[dim][token] (zero past the last token)
    for (int i = tid; i < kDim / 4 * kRkQ; i += kRkThreads) {
      const int j = i % kRkQ, k4 = i / kRkQ;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if ((uint32_t)j < np) v = __ldg(reinterpret_cast<const float4 *>(q + (tok0 + t0 + j) * kDim) + k4);
      Qs[(4 * k4 + 0) * kRkQ + j] = v.x;
      Qs[(4 * k4 + 1) * kRkQ + j] = v.y;
      Qs[(4 * k4 + 2) * kRkQ + j] = v.z;
      Qs[(4 * k4 + 3) * kRkQ + j] = v.w;
    }
    for (int i = tid; i < (int)nd * (kRkQ + 1); i += kRkThreads) best[i] = f2si(-INFINITY);
    __syncthreads();
    RkCta pc = cta;
    pc.T = d_pref[nd];
    if (np <= 16) rk_warp_pass<NBIT, 16, KT>(ix, pc, np);
    else rk_warp_pass<NBIT, 32, KT>(ix, pc, np);
    __syncthreads();
    if (tid < (int)nd) {
      const bool clamp = semantics == 1 && d_len[tid] < ix.max_item_n_vec;
      for (uint32_t t = 0; t < np; t++) {
        float m = si2f(best[tid * (kRkQ + 1) + t]);
        if (clamp) m = fmaxf(m, 0.0f);
        sum = __fadd_rn(sum, m);
      }
    }
    __syncthreads();  // Qs and best are rewritten by the next pass
  }
  if (tid < (int)nd) exact[(size_t)b * probe_topk + d0 + tid] = sum;
}

// ---------------------------------------------------------------------
// Which shortlisted docs an exact FP32 search has to score: those whose BF16
// MaxSim (approx) reaches the topk-th best of the query less twice a bound E on
// |BF16 - exact MaxSim|.  topk docs have exact scores of at least (the topk-th
// best approx - E), and a doc below the cut has an exact score under that.
// Per query token, with X a bound on |x| and dX on |x - BF16 x| of every decoded
// doc token x = c + W (dX: the centroids' and weights' own rounding errors, and for
// queries of more than split_tok tokens, whose kernel rounds the sum, a relative
// 2^-8), the error of a dot product is at most
//   |q - bf16(q)| X + |bf16(q)| dX + 2^-13 |q| X,
// the last term for both sides' FP32 accumulation; 2^-14 max(1, 4 max|q| X)
// covers an accumulator that starts at an offset of up to 2.04 max|q| X (the kernels'
// offset: at most 2 x 1.02 max|q| x_bound, which the index sets to X or less).  The max
// over a doc's tokens and the clamp at 0 enlarge no error, the sum over query
// tokens adds them up.  A bound that is not finite keeps every doc.  One CTA per
// query, the approximate scores' order keys in shared memory.
// ---------------------------------------------------------------------
constexpr int kReachThreads = 512;
__host__ __device__ constexpr size_t reach_smem(uint32_t probe_topk) {
  return (size_t)probe_topk * sizeof(uint32_t) + 4096 * sizeof(uint32_t);
}

__global__ void __launch_bounds__(kReachThreads)
maxsim_reach_kernel(const float *__restrict__ q, const uint64_t *__restrict__ q_off,
                    const uint32_t *__restrict__ short_id, const float *__restrict__ approx,
                    const uint32_t *__restrict__ n_short, uint32_t probe_topk, uint32_t topk,
                    const float *__restrict__ bounds, uint32_t split_tok, uint32_t *__restrict__ out_id, uint32_t *__restrict__ n_out) {
  extern __shared__ uint32_t rsm[];
  uint32_t *ord = rsm, *hist = rsm + probe_topk;  // [probe_topk], [4096]
  __shared__ float s_e[kMaxQueryTok], s_q[kMaxQueryTok];
  __shared__ uint32_t s_wsum[kReachThreads / 32], s_bin, s_need, s_n;
  __shared__ float s_thr;
  const uint32_t b = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t n = min(n_short[b], probe_topk);
  const uint64_t tok0 = q_off[b];
  const uint32_t nq = (uint32_t)(q_off[b + 1] - tok0);
  const size_t row = (size_t)b * probe_topk;
  for (uint32_t i = tid; i < n; i += kReachThreads) ord[i] = f2ord(approx[row + i]);
  if (tid == 0) s_n = 0;
  const float X = (bounds[0] + bounds[2]) * (1.0f + 0x1p-10f);
  const float dX = (bounds[1] + bounds[3]) * (1.0f + 0x1p-10f) + (nq > split_tok ? X * 0x1.02p-8f : 0.0f);
  for (uint32_t t = warp; t < nq; t += kReachThreads / 32) {
    const float4 v = __ldg(reinterpret_cast<const float4 *>(q + (tok0 + t) * kDim) + lane);
    const float x[4] = {v.x, v.y, v.z, v.w};
    float nn = 0.0f, nb = 0.0f, dd = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const float r = __bfloat162float(__float2bfloat16_rn(x[i]));
      nn = fmaf(x[i], x[i], nn);
      nb = fmaf(r, r, nb);
      dd = fmaf(x[i] - r, x[i] - r, dd);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      nn += __shfl_xor_sync(kFull, nn, o);
      nb += __shfl_xor_sync(kFull, nb, o);
      dd += __shfl_xor_sync(kFull, dd, o);
    }
    if (lane == 0) {
      s_e[t] = sqrtf(dd) * X + sqrtf(nb) * dX + sqrtf(nn) * X * 0x1p-13f;
      s_q[t] = sqrtf(nn);
    }
  }
  __syncthreads();
  if (n > topk) {
    // the topk-th largest order key: radix passes of 12, 12 and 8 bits
    uint32_t prefix = 0, need = topk;
    int shift = 32;
    while (shift > 0) {
      const int up = shift, width = min(12, shift);
      shift -= width;
      for (uint32_t i = tid; i < 4096; i += kReachThreads) hist[i] = 0;
      __syncthreads();
      for (uint32_t i = tid; i < n; i += kReachThreads) {
        const uint32_t k = ord[i];
        if (up == 32 || (k >> up) == prefix) atomicAdd(&hist[(k >> shift) & ((1u << width) - 1u)], 1u);
      }
      __syncthreads();
      uint32_t c[8], sum = 0;  // bins 4095 - 8 tid .. 4088 - 8 tid, high to low
#pragma unroll
      for (int u = 0; u < 8; u++) {
        c[u] = hist[4095 - 8 * tid - u];
        sum += c[u];
      }
      uint32_t incl = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += v;
      }
      if (lane == 31) s_wsum[warp] = incl;
      __syncthreads();
      uint32_t above = incl - sum;
      for (int w = 0; w < warp; w++) above += s_wsum[w];
      if (above < need && need <= above + sum) {
#pragma unroll
        for (int u = 0; u < 8; u++) {
          if (above < need && need <= above + c[u]) {
            s_bin = 4095 - 8 * tid - u;
            s_need = need - above;
          }
          above += c[u];
        }
      }
      __syncthreads();
      prefix = (prefix << width) | s_bin;
      need = s_need;
    }
    if (tid == 0) {
      float e = 0.0f, qm = 0.0f;
      for (uint32_t t = 0; t < nq; t++) {
        e += s_e[t];
        qm = fmaxf(qm, s_q[t]);
      }
      e = (e + (float)nq * 0x1p-14f * fmaxf(1.0f, 4.0f * qm * X)) * (1.0f + 0x1p-10f);
      s_thr = e < 1e30f ? __fsub_rd(ord2f(prefix), 2.0f * e) : -INFINITY;
    }
  } else if (tid == 0) {
    s_thr = -INFINITY;
  }
  __syncthreads();
  const float thr = s_thr;
  for (uint32_t i0 = 0; i0 < n; i0 += kReachThreads) {
    const uint32_t i = i0 + tid;
    const bool keep = i < n && !(ord2f(ord[i]) < thr);
    const unsigned m = __ballot_sync(kFull, keep);
    uint32_t at = 0;
    if (lane == 0 && m) at = atomicAdd(&s_n, (uint32_t)__popc(m));
    at = __shfl_sync(kFull, at, 0) + __popc(m & ((1u << lane) - 1u));
    if (keep) out_id[row + at] = short_id[row + i];
  }
  __syncthreads();
  if (tid == 0) n_out[b] = s_n;
}

// ---------------------------------------------------------------------
// K4: final top-k of the reranked shortlist (bitonic sort of 64-bit keys).
// ---------------------------------------------------------------------
__global__ void __launch_bounds__(512)
topk_kernel(const uint32_t *__restrict__ short_id, const float *__restrict__ exact,
            const uint32_t *__restrict__ n_short, uint32_t probe_topk,
            uint32_t n_pad, uint32_t topk, float *__restrict__ out_s,
            uint32_t *__restrict__ out_id, uint32_t *__restrict__ n_out) {
  extern __shared__ uint64_t keys[];
  const uint32_t b = blockIdx.x;
  const uint32_t n = n_short[b];
  if (n_out && threadIdx.x == 0) n_out[b] = min(n, topk);
  for (uint32_t i = threadIdx.x; i < n_pad; i += blockDim.x)
    keys[i] = i < n ? make_key(exact[(size_t)b * probe_topk + i], short_id[(size_t)b * probe_topk + i]) : 0ull;
  __syncthreads();
  for (uint32_t k = 2; k <= n_pad; k <<= 1) {
    for (uint32_t j = k >> 1; j > 0; j >>= 1) {
      for (uint32_t i = threadIdx.x; i < n_pad; i += blockDim.x) {
        const uint32_t l = i ^ j;
        if (l > i) {
          const uint64_t a = keys[i], c = keys[l];
          const bool desc = (i & k) == 0;
          if (desc ? (a < c) : (a > c)) { keys[i] = c; keys[l] = a; }
        }
      }
      __syncthreads();
    }
  }
  for (uint32_t i = threadIdx.x; i < topk; i += blockDim.x) {
    if (i < n) {
      out_s[(size_t)b * topk + i] = key_score(keys[i]);
      out_id[(size_t)b * topk + i] = key_id(keys[i]);
    } else {
      out_s[(size_t)b * topk + i] = -INFINITY;
      out_id[(size_t)b * topk + i] = 0xffffffffu;
    }
  }
}

// ---------------------------------------------------------------------
// K4 for k well below the list length: the same sorted top-k by a radix
// select of the k-th largest key in shared memory (8-bit digits, high to
// low, stopping once the boundary digit is unique), a compaction of the k
// keys at or above it (the keys are unique: exactly k), and a bitonic sort
// of those k only.  Same output as topk_kernel.
// ---------------------------------------------------------------------
__global__ void __launch_bounds__(512)
topk_select_kernel(const uint32_t *__restrict__ short_id, const float *__restrict__ exact,
                   const uint32_t *__restrict__ n_short, uint32_t probe_topk, uint32_t k_pad,
                   uint32_t topk, float *__restrict__ out_s, uint32_t *__restrict__ out_id,
                   uint32_t *__restrict__ n_out) {
  extern __shared__ uint64_t keys[];  // [probe_topk] keys, then [k_pad] selected
  uint64_t *sel = keys + probe_topk;
  __shared__ uint32_t hist[256];
  __shared__ uint32_t s_digit, s_need, s_done, s_cnt;
  const uint32_t b = blockIdx.x;
  const uint32_t n = min(n_short[b], probe_topk);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (n_out && tid == 0) n_out[b] = min(n, topk);
  for (uint32_t i = tid; i < n; i += blockDim.x)
    keys[i] = make_key(exact[(size_t)b * probe_topk + i], short_id[(size_t)b * probe_topk + i]);
  for (uint32_t i = tid; i < k_pad; i += blockDim.x) sel[i] = 0ull;
  if (tid == 0) s_cnt = 0;
  uint64_t prefix = 0, mask = 0;
  if (n > topk) {
    uint32_t need = topk;
    for (int pass = 0; pass < 8; pass++) {
      const int shift = 56 - 8 * pass;
      for (int i = tid; i < 256; i += blockDim.x) hist[i] = 0;
      __syncthreads();
      for (uint32_t i0 = 0; i0 < n; i0 += blockDim.x) {
        const uint32_t i = i0 + tid;
        uint32_t dig = 256;
        if (i < n && (keys[i] & mask) == prefix) dig = (uint32_t)(keys[i] >> shift) & 0xffu;
        const unsigned grp = __match_any_sync(kFull, dig);
        if (dig < 256 && lane == __ffs(grp) - 1) atomicAdd(&hist[dig], (uint32_t)__popc(grp));
      }
      __syncthreads();
      if (warp == 0) {  // lane l owns bins 255-8l .. 248-8l (high to low)
        uint32_t cnt[8], sum = 0;
#pragma unroll
        for (int u = 0; u < 8; u++) {
          cnt[u] = hist[255 - 8 * lane - u];
          sum += cnt[u];
        }
        uint32_t incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t v = __shfl_up_sync(kFull, incl, o);
          if (lane >= o) incl += v;
        }
        const uint32_t excl = incl - sum;
        if (excl < need && need <= incl) {
          uint32_t above = excl;
#pragma unroll
          for (int u = 0; u < 8; u++) {
            if (above < need && need <= above + cnt[u]) {
              s_digit = 255 - 8 * lane - u;
              s_need = need - above;
              s_done = (need - above == cnt[u]) ? 1u : 0u;
            }
            above += cnt[u];
          }
        }
      }
      __syncthreads();
      prefix |= (uint64_t)s_digit << shift;
      mask |= (uint64_t)0xff << shift;
      need = s_need;
      if (s_done) break;
    }
  }
  __syncthreads();
  // the top keys (all n when n <= topk), unordered, then sorted descending
  for (uint32_t i = tid; i < n; i += blockDim.x)
    if ((keys[i] & mask) >= prefix) sel[atomicAdd(&s_cnt, 1u)] = keys[i];
  __syncthreads();
  for (uint32_t kk = 2; kk <= k_pad; kk <<= 1) {
    for (uint32_t j = kk >> 1; j > 0; j >>= 1) {
      for (uint32_t i = tid; i < k_pad; i += blockDim.x) {
        const uint32_t l = i ^ j;
        if (l > i) {
          const uint64_t a = sel[i], c = sel[l];
          const bool desc = (i & kk) == 0;
          if (desc ? (a < c) : (a > c)) { sel[i] = c; sel[l] = a; }
        }
      }
      __syncthreads();
    }
  }
  for (uint32_t i = tid; i < topk; i += blockDim.x) {
    if (i < n) {
      out_s[(size_t)b * topk + i] = key_score(sel[i]);
      out_id[(size_t)b * topk + i] = key_id(sel[i]);
    } else {
      out_s[(size_t)b * topk + i] = -INFINITY;
      out_id[(size_t)b * topk + i] = 0xffffffffu;
    }
  }
}

// ---------------------------------------------------------------------
// host-side launchers
// ---------------------------------------------------------------------
cudaError_t configure_kernels() {
  cudaError_t e = cudaFuncSetAttribute(probe_scan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kProbeSmem);
  if (e != cudaSuccess) return e;
#define MVR_RK_ATTR(NB, KT)                                                                     \
  e = cudaFuncSetAttribute(rerank_kernel<NB, KT>, cudaFuncAttributeMaxDynamicSharedMemorySize,  \
                           (int)rk_smem_bytes(NB));                                             \
  if (e != cudaSuccess) return e;
  MVR_RK_ATTR(1, 1) MVR_RK_ATTR(1, 4)
  MVR_RK_ATTR(2, 1) MVR_RK_ATTR(2, 4)
  MVR_RK_ATTR(4, 1) MVR_RK_ATTR(4, 4)
  MVR_RK_ATTR(8, 1) MVR_RK_ATTR(8, 4)
#undef MVR_RK_ATTR
  e = cudaFuncSetAttribute(filter_hash_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)hash_smem_bytes(1));
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(filter_hash_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)hash_smem_bytes(2));
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(topk_select_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)((kMaxShort + kMaxShort / 4) * sizeof(uint64_t)));
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(maxsim_reach_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)reach_smem(kMaxShort));
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(topk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)(kMaxShort * sizeof(uint64_t)));
}

cudaError_t launch_probe_scan(const float *q, const float *cen_t, uint32_t n_cent,
                              uint32_t n_cent_pad, uint32_t nprobe, uint32_t *flags,
                              uint32_t list_at, uint32_t *part_id, float *part_s,
                              uint32_t *out_id, float *out_s, int n_sm, cudaStream_t st,
                              int *n_launch) {
  probe_scan_kernel<<<n_sm, 256, kProbeSmem, st>>>(q, cen_t, n_cent, n_cent_pad, nprobe, flags,
                                                   list_at, part_id, part_s, out_id, out_s);
  *n_launch += 1;
  return cudaGetLastError();
}

cudaError_t launch_filter(const DevIndex &ix, const uint32_t *probe_id,
                          const float *probe_s, uint32_t nprobe,
                          const uint64_t *q_off, uint32_t n_query,
                          uint32_t probe_topk, const FilterScratch &scr,
                          uint32_t epoch, uint32_t *short_id,
                          float *short_approx, uint32_t *n_short,
                          uint32_t *qstat, cudaStream_t st, int *n_launch) {
  filter_kernel<1><<<n_query, kFilterThreads, 0, st>>>(ix, probe_id, probe_s, nprobe, q_off,
                                                       probe_topk, scr, nullptr, epoch, short_id,
                                                       short_approx, n_short, qstat, nullptr, 0);
  *n_launch += 1;
  return cudaGetLastError();
}

cudaError_t launch_filter_cluster(const DevIndex &ix, const uint32_t *probe_id,
                                  const float *probe_s, uint32_t nprobe,
                                  const uint64_t *q_off, uint32_t n_query,
                                  uint32_t probe_topk, const FilterScratch &scr,
                                  const uint32_t *epoch_base, uint32_t epoch_add,
                                  uint32_t *short_id, float *short_approx, uint32_t *n_short,
                                  uint32_t *qstat, cudaStream_t st, int *n_launch,
                                  uint32_t *only_if, int impute) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(n_query * kFilterCluster, 1, 1);
  cfg.blockDim = dim3(kFilterThreads, 1, 1);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kFilterCluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, filter_kernel<kFilterCluster>, ix, probe_id, probe_s,
                                     nprobe, q_off, probe_topk, scr, epoch_base, epoch_add,
                                     short_id, short_approx, n_short, qstat, only_if, impute);
  *n_launch += 1;
  return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t launch_filter_hash(const DevIndex &ix, const uint32_t *probe_id,
                               const float *probe_s, uint32_t nprobe,
                               const uint64_t *q_off, const uint64_t *cta_off, uint32_t n_cta,
                               uint32_t n_query, uint32_t fb_slots,
                               uint32_t probe_topk, const FilterScratch &scr,
                               uint32_t *epoch, uint32_t *short_id,
                               float *short_approx, uint32_t *n_short,
                               uint32_t *qstat, cudaStream_t st, int *n_launch, int impute) {
  cudaError_t e = cudaMemsetAsync(scr.ovf, 0, (size_t)n_query * sizeof(uint32_t), st);
  if (e != cudaSuccess) return e;
  if (scr.rank_stride <= 32)
    filter_hash_kernel<1><<<n_cta, kFilterThreads, hash_smem_bytes(1), st>>>(
        ix, probe_id, probe_s, nprobe, q_off, cta_off, n_query, scr, qstat, impute);
  else
    filter_hash_kernel<2><<<n_cta, kFilterThreads, hash_smem_bytes(2), st>>>(
        ix, probe_id, probe_s, nprobe, q_off, cta_off, n_query, scr, qstat, impute);
  // one CTA per query also where queries are few: clusters of 4 and 8 CTAs took
  // 18 and 42 us where it takes 7 (1,065 candidates), 38 and 79 us where it takes
  // 32 (34,000), their histograms and counters being remote
  filter_select_kernel<<<n_query, kFilterThreads, 0, st>>>(ix, probe_topk, scr, short_id,
                                                          short_approx, n_short, qstat, epoch,
                                                          (n_query + fb_slots - 1) / fb_slots);
  *n_launch += 2;
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  // queries whose candidates overflowed a hash table: rank-table filter, in
  // chunks of fb_slots queries over its fb_slots scratch slots; chunk c takes the
  // stamp epoch *epoch - c of those that the select kernel advanced it by
  uint32_t c = 0;
  for (uint32_t q0 = 0; q0 < n_query; q0 += fb_slots, c++) {
    const uint32_t cnt = n_query - q0 < fb_slots ? n_query - q0 : fb_slots;
    e = launch_filter_cluster(ix, probe_id, probe_s, nprobe, q_off + q0, cnt, probe_topk, scr,
                              epoch, 0u - c, short_id + (size_t)q0 * probe_topk,
                              short_approx + (size_t)q0 * probe_topk, n_short + q0,
                              qstat + (size_t)q0 * 3, st, n_launch, scr.ovf + q0, impute);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// Shortlisted docs per CTA of the exact rerank: kRkDocs for grids that fill the GPU
// several times over, fewer while n_query * windows stays within two waves of CTAs:
// a wide window would leave most SMs idle (one query, 200 docs: 232 us in 4 CTAs,
// 25 us in 50; 40 docs: 34 us in 10, 23 us in 40).  With up to kRkNarrow docs a CTA
// the tiles are 32 tokens wide, so that a doc occupies its 4 warps (40 docs of 4
// queries: 34 -> 20 us, of 16 queries: 58 -> 43 us); with 4 docs the wide tiles are
// the faster ones (of 37 queries: 55 against 76 us).
constexpr uint32_t kRkNarrow = 2;
static uint32_t rerank_docs(uint32_t n_query, uint32_t n_docs, uint32_t most, int n_sm) {
  uint32_t docs = most;
  while (docs > 1 &&
         (uint64_t)n_query * ((n_docs + docs / 2 - 1) / (docs / 2)) <= 4ull * (uint32_t)n_sm)
    docs /= 2;
  return docs;
}

cudaError_t launch_rerank(const DevIndex &ix, const float *q, const uint64_t *q_off,
                          uint32_t n_query, const uint32_t *short_id,
                          const uint32_t *n_short, uint32_t probe_topk,
                          int semantics, float *exact, int n_sm, cudaStream_t st,
                          int *n_launch, uint32_t most_docs) {
  if (n_query == 0 || probe_topk == 0) return cudaSuccess;
  const uint32_t docs = rerank_docs(n_query, probe_topk, std::min<uint32_t>(most_docs, kRkDocs), n_sm);
  dim3 grid((probe_topk + docs - 1) / docs, n_query);
  const size_t sm = rk_smem_bytes((int)ix.n_bit);
  const bool narrow = docs <= kRkNarrow;
#define MVR_RK(NB)                                                                              \
  if (narrow)                                                                                   \
    rerank_kernel<NB, 1><<<grid, kRkThreads, sm, st>>>(ix, q, q_off, short_id, n_short,         \
                                                       probe_topk, docs, semantics, exact);     \
  else                                                                                          \
    rerank_kernel<NB, kRkT><<<grid, kRkThreads, sm, st>>>(ix, q, q_off, short_id, n_short,      \
                                                          probe_topk, docs, semantics, exact)
  switch (ix.n_bit) {
    case 1: MVR_RK(1); break;
    case 2: MVR_RK(2); break;
    case 4: MVR_RK(4); break;
    case 8: MVR_RK(8); break;
    default: return cudaErrorInvalidValue;
  }
#undef MVR_RK
  *n_launch += 1;
  return cudaGetLastError();
}

cudaError_t launch_maxsim_reach(const float *q, const uint64_t *q_off, uint32_t n_query,
                                const uint32_t *short_id, const float *approx,
                                const uint32_t *n_short, uint32_t probe_topk, uint32_t topk,
                                const float *bounds, uint32_t split_tok, uint32_t *out_id,
                                uint32_t *n_out, cudaStream_t st, int *n_launch) {
  maxsim_reach_kernel<<<n_query, kReachThreads, reach_smem(probe_topk), st>>>(
      q, q_off, short_id, approx, n_short, probe_topk, topk, bounds, split_tok, out_id, n_out);
  *n_launch += 1;
  return cudaGetLastError();
}

cudaError_t launch_topk(const uint32_t *short_id, const float *exact,
                        const uint32_t *n_short, uint32_t n_query,
                        uint32_t probe_topk, uint32_t topk, float *out_s,
                        uint32_t *out_id, uint32_t *n_out, cudaStream_t st, int *n_launch) {
  uint32_t n_pad = 1;
  while (n_pad < probe_topk) n_pad <<= 1;
  uint32_t k_pad = 1;
  while (k_pad < topk) k_pad <<= 1;
  if (probe_topk >= 512 && 4 * topk <= probe_topk) {
    // select, then sort only the k best
    topk_select_kernel<<<n_query, 512, (probe_topk + k_pad) * sizeof(uint64_t), st>>>(
        short_id, exact, n_short, probe_topk, k_pad, topk, out_s, out_id, n_out);
  } else {
    topk_kernel<<<n_query, 512, n_pad * sizeof(uint64_t), st>>>(short_id, exact, n_short,
                                                              probe_topk, n_pad, topk, out_s,
                                                              out_id, n_out);
  }
  *n_launch += 1;
  return cudaGetLastError();
}

}  // namespace mvr
