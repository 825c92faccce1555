// mvr_aux.cu -- index-side kernels of libmvr: centroid transpose for the
// probe kernel, standalone decode (decompression / bucket unpack with the
// rerank decoder's bit layout) and the index-build kernels (residual packing,
// FP64 k-means accumulation).
#include "mvr_aux.cuh"

#include <algorithm>
#include <cstring>
#include <vector>

namespace mvr {

// ct[k][c] = centroid[c][k] for c < C, 0 for C <= c < C_pad.
__global__ void transpose_centroid_kernel(const float *__restrict__ cen, uint32_t n_cent,
                                          uint32_t n_cent_pad, float *__restrict__ ct) {
  __shared__ float tile[32][33];
  const uint32_t c0 = blockIdx.x * 32, k0 = blockIdx.y * 32;
  const int tx = threadIdx.x, ty = threadIdx.y;  // 32 x 8
  for (int r = ty; r < 32; r += 8) {
    const uint32_t c = c0 + r, k = k0 + tx;
    tile[r][tx] = (c < n_cent) ? cen[(size_t)c * kDim + k] : 0.0f;
  }
  __syncthreads();
  for (int r = ty; r < 32; r += 8) {
    const uint32_t k = k0 + r, c = c0 + tx;
    if (c < n_cent_pad) ct[(size_t)k * n_cent_pad + c] = tile[tx][r];
  }
}

cudaError_t launch_transpose_centroid(const float *cen, uint32_t n_cent, uint32_t n_cent_pad,
                                      float *ct, cudaStream_t st) {
  dim3 grid(n_cent_pad / 32, kDim / 32), block(32, 8);
  transpose_centroid_kernel<<<grid, block, 0, st>>>(cen, n_cent, n_cent_pad, ct);
  return cudaGetLastError();
}

// value i of a packed byte (MSB-first): (byte >> (8 - b*(i+1))) & (2^b - 1)
__device__ __forceinline__ uint32_t bucket_of(const uint8_t *res, uint32_t d, uint32_t n_bit) {
  const uint32_t vpb = 8u / n_bit;
  const uint32_t byte = res[d / vpb];
  const uint32_t i = d % vpb;
  return (byte >> (8u - n_bit * (i + 1u))) & ((1u << n_bit) - 1u);
}

__global__ void decompress_kernel(DevIndex ix, const uint64_t *__restrict__ vec_id, uint64_t n,
                                  float *__restrict__ out) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n * kDim) return;
  const uint64_t t = i / kDim;
  const uint32_t d = (uint32_t)(i % kDim);
  const uint64_t v = vec_id[t];
  const uint8_t *res = ix.residual + v * ix.bytes_per_vec;
  const uint32_t vpb = 8u / ix.n_bit;
  const float w = ix.lut[(uint32_t)res[d / vpb] * vpb + d % vpb];
  out[i] = __fadd_rn(ix.centroid[(size_t)ix.vq_code[v] * kDim + d], w);
}

__global__ void unpack_kernel(DevIndex ix, const uint64_t *__restrict__ vec_id, uint64_t n,
                              uint8_t *__restrict__ out) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n * kDim) return;
  const uint64_t t = i / kDim;
  const uint32_t d = (uint32_t)(i % kDim);
  out[i] = (uint8_t)bucket_of(ix.residual + vec_id[t] * ix.bytes_per_vec, d, ix.n_bit);
}

cudaError_t launch_decompress(const DevIndex &ix, const uint64_t *vec_id, uint64_t n, float *out,
                              cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  const uint64_t tot = n * kDim;
  decompress_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(ix, vec_id, n, out);
  return cudaGetLastError();
}

cudaError_t launch_unpack(const DevIndex &ix, const uint64_t *vec_id, uint64_t n, uint8_t *out,
                          cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  const uint64_t tot = n * kDim;
  unpack_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(ix, vec_id, n, out);
  return cudaGetLastError();
}

// One thread per packed byte: bucket = #cutoffs <= (vec - centroid) for each
// of its 8/n_bit values, packed MSB-first (compressSQCode semantics).
__global__ void pack_residual_kernel(const float *__restrict__ vec, uint64_t n_vec,
                                     const float *__restrict__ cen, const uint32_t *__restrict__ code,
                                     Cutoffs cut, uint32_t n_bit, uint8_t *__restrict__ out) {
  const uint32_t vpb = 8u / n_bit;
  const uint32_t bpv = kDim / vpb;
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_vec * bpv) return;
  const uint64_t v = i / bpv;
  const uint32_t p = (uint32_t)(i % bpv);
  const float *x = vec + v * kDim;
  const float *c = cen + (size_t)code[v] * kDim;
  const uint32_t n_cut = (1u << n_bit) - 1u;
  uint32_t byte = 0;
  for (uint32_t u = 0; u < vpb; u++) {
    const uint32_t d = p * vpb + u;
    const float e = __fsub_rn(x[d], c[d]);
    uint32_t bk = n_cut;
    for (uint32_t k = 0; k < n_cut; k++)
      if (cut.v[k] > e) { bk = k; break; }
    byte = (byte << n_bit) | bk;
  }
  out[i] = (uint8_t)byte;
}

cudaError_t launch_pack_residual(const float *vec, uint64_t n_vec, const float *cen,
                                 const uint32_t *code, const Cutoffs &cut, uint32_t n_bit,
                                 uint8_t *out, cudaStream_t st) {
  const uint64_t tot = n_vec * (kDim / (8u / n_bit));
  if (tot == 0) return cudaSuccess;
  pack_residual_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(vec, n_vec, cen, code, cut, n_bit, out);
  return cudaGetLastError();
}

// sum[code[i]][d] += vec[i][d] in FP64; count[code[i]] += 1.  One warp per
// token, 4 dims per lane.
__global__ void kmeans_accumulate_kernel(const float *__restrict__ vec, uint64_t n_vec,
                                         const uint32_t *__restrict__ code, double *__restrict__ sum,
                                         unsigned long long *__restrict__ count) {
  const uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= n_vec) return;
  const uint32_t c = code[w];
  const float4 x = reinterpret_cast<const float4 *>(vec + w * kDim)[lane];
  double *s = sum + (size_t)c * kDim + lane * 4;
  atomicAdd(s + 0, (double)x.x);
  atomicAdd(s + 1, (double)x.y);
  atomicAdd(s + 2, (double)x.z);
  atomicAdd(s + 3, (double)x.w);
  if (lane == 0) atomicAdd(count + c, 1ull);
}

cudaError_t launch_kmeans_accumulate(const float *vec, uint64_t n_vec, const uint32_t *code,
                                     double *sum, uint64_t *count, cudaStream_t st) {
  if (n_vec == 0) return cudaSuccess;
  const uint64_t threads = n_vec * 32;
  kmeans_accumulate_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, st>>>(
      vec, n_vec, code, sum, reinterpret_cast<unsigned long long *>(count));
  return cudaGetLastError();
}

// Order statistics of the residual errors e = vec[i][d] - centroid[code[i]][d]
// (one rounded FP32 subtraction, as the codec computes them), without
// materialising them: e is mapped to a 32-bit key whose unsigned order is the
// float order, and three passes over the vectors count 12, 10 and 10 of its
// bits, the later ones only for keys under a prefix that holds a wanted rank.
//
// A warp takes a token, 4 dimensions a lane (16-byte loads of the vector and
// of its centroid row), and counts in shared memory: residuals crowd into a
// few hundred prefixes, where 64-bit global atomics queue on one address.
// Prefixes beyond the kHistSlots that shared memory holds (8-bit codes have 511
// ranks) count in global memory.  Bound: a pass reads the vectors once (300,007
// tokens, 154 MB: 24 us), plus a shared atomic per counted value: 37, 60 and 63
// us for the 7 ranks of 2-bit codes, where the builder's bisection over
// materialised keys took 50 ms.
__device__ __forceinline__ uint32_t order_key(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

constexpr int kHiBits = 12, kLoBits = 10;       // 12 + 10 + 10 = 32
constexpr uint32_t kHiBins = 1u << kHiBits, kLoBins = 1u << kLoBits;
constexpr uint32_t kHistSlots = 40;             // prefixes counted in shared memory
constexpr uint16_t kNoSlot = 0xffff;

// 4 floats, one load where both arrays start on 16 bytes
__device__ __forceinline__ float4 load4(const float *p, bool aligned) {
  if (aligned) return __ldg(reinterpret_cast<const float4 *>(p));
  return make_float4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3));
}

// PASS 0: hist[key >> 20].  PASS 1: prefixes key >> 20, their next 10 bits.
// PASS 2: prefixes key >> 10, the last 10 bits.  slot1 [4096] / slot2
// [n1][1024]: the slot of a prefix (kNoSlot: not wanted); hist of passes 1 and
// 2: [slots][1024].
template <int PASS>
__global__ void __launch_bounds__(512)
residual_hist_kernel(const float *__restrict__ vec, uint64_t n_vec, const float *__restrict__ cen,
                     const uint32_t *__restrict__ code, bool aligned, const uint16_t *__restrict__ slot1,
                     const uint16_t *__restrict__ slot2, uint32_t n_slot,
                     unsigned long long *__restrict__ hist) {
  extern __shared__ uint32_t sh[];
  const uint32_t held = PASS == 0 ? kHiBins : min(n_slot, kHistSlots) * kLoBins;
  for (uint32_t i = threadIdx.x; i < held; i += blockDim.x) sh[i] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const uint64_t w0 = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t v = w0; v < n_vec; v += nw) {
    const float4 x = load4(vec + v * kDim + 4 * lane, aligned);
    const float4 c = load4(cen + (size_t)code[v] * kDim + 4 * lane, aligned);
    const float e[4] = {__fsub_rn(x.x, c.x), __fsub_rn(x.y, c.y), __fsub_rn(x.z, c.z),
                        __fsub_rn(x.w, c.w)};
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const uint32_t k = order_key(e[u]);
      if constexpr (PASS == 0) {
        atomicAdd(&sh[k >> 20], 1u);
      } else {
        uint32_t sl = slot1[k >> 20], bin = (k >> 10) & (kLoBins - 1u);
        if constexpr (PASS == 2) {
          if (sl != kNoSlot) sl = slot2[(size_t)sl * kLoBins + bin];
          bin = k & (kLoBins - 1u);
        }
        if (sl == kNoSlot) continue;
        if (sl < kHistSlots) atomicAdd(&sh[sl * kLoBins + bin], 1u);
        else atomicAdd(hist + (size_t)sl * kLoBins + bin, 1ull);
      }
    }
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < held; i += blockDim.x)
    if (sh[i]) atomicAdd(hist + i, (unsigned long long)sh[i]);
}

cudaError_t residual_select(const float *vec, uint64_t n_vec, const float *cen,
                            const uint32_t *code, const uint64_t *rank, uint32_t n_rank,
                            float *out, cudaStream_t st) {
  if (n_rank == 0) return cudaSuccess;
  const uint64_t n = n_vec * kDim;
  for (uint32_t r = 0; r < n_rank; r++)
    if (rank[r] >= n) return cudaErrorInvalidValue;
  // one allocation: [hist][slot1][slot2], sized for n_rank distinct prefixes
  const size_t hist_n = std::max<size_t>(kHiBins, (size_t)n_rank * kLoBins);
  const size_t slot2_n = (size_t)n_rank * kLoBins;
  uint8_t *buf = nullptr;
  cudaError_t e = cudaMalloc(&buf, hist_n * 8 + kHiBins * 2 + slot2_n * 2);
  if (e != cudaSuccess) return e;
  auto *hist = reinterpret_cast<unsigned long long *>(buf);
  auto *slot1 = reinterpret_cast<uint16_t *>(buf + hist_n * 8);
  uint16_t *slot2 = slot1 + kHiBins;
  const unsigned grid = 148u * 4u;
  const bool aligned = (((uintptr_t)vec | (uintptr_t)cen) & 15) == 0;
  std::vector<unsigned long long> h(hist_n);
  std::vector<uint32_t> prefix(n_rank, 0), slot_of(n_rank, 0);
  std::vector<uint64_t> below(n_rank, 0);  // keys under smaller prefixes
  std::vector<uint16_t> table;
  uint32_t n_slot = 1;
  for (int pass = 0; pass < 3 && e == cudaSuccess; pass++) {
    const size_t bins = pass == 0 ? kHiBins : kLoBins;
    const size_t smem = pass == 0 ? kHiBins * 4 : (size_t)std::min(n_slot, kHistSlots) * kLoBins * 4;
    e = cudaMemsetAsync(hist, 0, n_slot * bins * 8, st);
    if (e == cudaSuccess) {
      if (pass == 0) {
        residual_hist_kernel<0><<<grid, 512, smem, st>>>(vec, n_vec, cen, code, aligned, slot1, slot2, 1, hist);
      } else {
        e = pass == 1 ? cudaFuncSetAttribute(residual_hist_kernel<1>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)(kHistSlots * kLoBins * 4))
                      : cudaFuncSetAttribute(residual_hist_kernel<2>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)(kHistSlots * kLoBins * 4));
        if (e == cudaSuccess) {
          if (pass == 1)
            residual_hist_kernel<1><<<grid, 512, smem, st>>>(vec, n_vec, cen, code, aligned, slot1, slot2, n_slot, hist);
          else
            residual_hist_kernel<2><<<grid, 512, smem, st>>>(vec, n_vec, cen, code, aligned, slot1, slot2, n_slot, hist);
        }
      }
      if (e == cudaSuccess) e = cudaGetLastError();
    }
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(h.data(), hist, n_slot * bins * 8, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) break;
    // the bin of every rank under its prefix; the distinct longer prefixes
    // become the next pass's slots
    table.assign(pass == 0 ? kHiBins : n_slot * kLoBins, kNoSlot);
    uint32_t next = 0;
    for (uint32_t r = 0; r < n_rank; r++) {
      const unsigned long long *g = h.data() + (size_t)slot_of[r] * bins;
      uint32_t b = 0;
      while (below[r] + g[b] <= rank[r]) below[r] += g[b++];
      prefix[r] = pass == 0 ? b : (prefix[r] << kLoBits) | b;
      uint16_t &t = table[(size_t)slot_of[r] * bins + b];
      if (t == kNoSlot) t = (uint16_t)next++;
      slot_of[r] = t;
    }
    n_slot = next;
    if (pass < 2)
      e = cudaMemcpyAsync(pass == 0 ? slot1 : slot2, table.data(), table.size() * 2,
                          cudaMemcpyHostToDevice, st);
  }
  if (e == cudaSuccess) {
    for (uint32_t r = 0; r < n_rank; r++) {
      const uint32_t k = prefix[r];
      const uint32_t u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
      std::memcpy(&out[r], &u, 4);
    }
  }
  cudaFree(buf);
  return e;
}

// out[q][d] = sum over the query's tokens of the max over the doc's tokens of
// s[token][doc token]: one warp per (query, doc), 16 query tokens at a time
// (32 at a time took 214 registers and left too few warps: 16.6 ms below).
// Each lane keeps its own columns' maximum for every one of the 16 tokens, and
// a transposing reduction (16 exchanges where 16 separate ones would take 80)
// leaves token t's maximum in lane t.  NaN scores carry through, empty docs are
// -inf.  Bound: reading s once.  64 queries x 32 tokens against 1.4M tokens, FP64
// (23 GB): scatter_reduce with its atomics 68 ms -> 7.0 ms.
template <class T>
__device__ __forceinline__ T nan_max(T a, T b) {
  return b > a || b != b ? b : a;
}

template <class T>
__global__ void __launch_bounds__(256, 3)
segment_maxsum_kernel(const T *__restrict__ s, uint64_t ld, const int64_t *__restrict__ q_off,
                      uint32_t n_query, const int64_t *__restrict__ d_off, uint32_t n_doc,
                      T *__restrict__ out) {
  constexpr int NT = 16;  // query tokens at a time
  const int lane = threadIdx.x & 31;
  const uint64_t n = (uint64_t)n_query * n_doc;
  for (uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < n;
       w += ((uint64_t)gridDim.x * blockDim.x) >> 5) {
    const uint32_t q = (uint32_t)(w / n_doc), d = (uint32_t)(w % n_doc);
    const int64_t c0 = d_off[d], c1 = d_off[d + 1];
    T sum = 0;
    for (int64_t t0 = q_off[q]; t0 < q_off[q + 1]; t0 += NT) {
      const int nt = (int)min((int64_t)NT, q_off[q + 1] - t0);
      const T *row = s + (uint64_t)t0 * ld;
      T m[NT];
#pragma unroll
      for (int t = 0; t < NT; t++) m[t] = -INFINITY;
      for (int64_t c = c0 + lane; c < c1; c += 32) {
        T v[NT];  // all rows' loads in flight; past the last token its row again
#pragma unroll
        for (int t = 0; t < NT; t++) v[t] = __ldg(row + (uint64_t)min(t, nt - 1) * ld + c);
#pragma unroll
        for (int t = 0; t < NT; t++) m[t] = nan_max(m[t], v[t]);
      }
      // step o: lanes with bit o set keep the upper half of the tokens left
#pragma unroll
      for (int o = NT / 2; o > 0; o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < o; i++) {
          const T give = up ? m[i] : m[i + o], keep = up ? m[i + o] : m[i];
          m[i] = nan_max(keep, __shfl_xor_sync(0xffffffffu, give, o));
        }
      }
      m[0] = nan_max(m[0], __shfl_xor_sync(0xffffffffu, m[0], NT));
      T v = (lane & (NT - 1)) < nt ? m[0] : (T)0;
#pragma unroll
      for (int o = NT / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      sum += v;
    }
    if (lane == 0) out[w] = sum;
  }
}

cudaError_t launch_segment_maxsum(const void *s, bool f64, uint64_t ld, const int64_t *q_off,
                                  uint32_t n_query, const int64_t *d_off, uint32_t n_doc,
                                  void *out, cudaStream_t st) {
  const uint64_t n = (uint64_t)n_query * n_doc;
  if (n == 0) return cudaSuccess;
  const unsigned grid = (unsigned)std::min<uint64_t>((n + 7) / 8, 148u * 64u);
  if (f64)
    segment_maxsum_kernel<double><<<grid, 256, 0, st>>>((const double *)s, ld, q_off, n_query,
                                                        d_off, n_doc, (double *)out);
  else
    segment_maxsum_kernel<float><<<grid, 256, 0, st>>>((const float *)s, ld, q_off, n_query, d_off,
                                                       n_doc, (float *)out);
  return cudaGetLastError();
}

}  // namespace mvr
