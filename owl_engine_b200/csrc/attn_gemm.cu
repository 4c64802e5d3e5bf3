// Helpers of the GEMM-form prefill attention (long prompts): the two contractions of causal attention run as tcgen05 GEMMs
// (gemm_dense.cu), these kernels do what lies between them.
//
//   owl_kv_gather       paged K / V of one sequence and layer (e4m3, int8 + scales, or fp16 words)
//                         -> K  bf16 [hkv][ctx_pad][hd]   (rows = keys: the B operand of S = Q K^T, k-major)
//                            Vt fp16 [hkv][hd][ctx_pad]   (rows = dims: the B operand of O = P V,   k-major)
//                       ctx_pad is a multiple of 64; the padding columns / rows are written as zeros
//   owl_causal_softmax  S fp16 [rows][ld] -> P fp16 in place: row r sees keys < pos0 + r + 1, softmax(scale * s), zeros elsewhere
//
// Role in the reference: the FlashInfer prefill kernels of crates/kernels/cu/attn (fused form); on this part the tensor cores
// are reached through tcgen05 GEMMs, and below a few thousand keys the fused warp-level kernel of attn.cu stays in use.
#include <cuda_fp8.h>
#include "common.cuh"

namespace owl {

constexpr int AG_PAGE = 16;

// 16 elements of a pool row as floats. FMT 0: e4m3, 1: int8 (times the row's scale), 2: fp16 words
template <int FMT>
__device__ __forceinline__ void ag_floats(const uint4* raw, float scale, float* v) {
  const uint32_t w[8] = {raw[0].x, raw[0].y, raw[0].z, raw[0].w, raw[FMT == 2].x, raw[FMT == 2].y, raw[FMT == 2].z, raw[FMT == 2].w};
#pragma unroll
  for (int i = 0; i < (FMT == 2 ? 8 : 4); ++i) {
    if (FMT == 2) {
      const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
      v[2 * i] = f.x; v[2 * i + 1] = f.y;
    } else if (FMT == 1) {
#pragma unroll
      for (int k = 0; k < 4; ++k) v[4 * i + k] = (float)(int8_t)(w[i] >> (8 * k)) * scale;
    } else {
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const __half2 h = __half2(__nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(w[i] >> (16 * k)), __NV_E4M3));
        const float2 f = __half22float2(h);
        v[4 * i + 2 * k] = f.x; v[4 * i + 2 * k + 1] = f.y;
      }
    }
  }
}

// Bound by memory: a key and head is read once (512 bytes of e4m3) and written once (1 KB). grid (ctx_pad / 64, hkv), 256 threads: 64
// keys of one head; a thread takes 16 dims (16-byte loads) of two neighbouring keys at a time, stores K as it is and puts V as pairs
// of keys into shared memory, [dim][32 pairs], from which a dim's 64 keys leave as one line. A pair lies at place
// pair ^ 2 * (dim / 16): the 16 lanes that write one pair hold dims 16 apart, which would be one bank. ANY: pools or keys that do not
// begin at a multiple of 16 bytes (views; an allocation of their own always does), read byte by byte and stored value by value.
// 34,768 e4m3 keys, 4 heads: 38 us, 32 at copy bandwidth; byte loads and 2-byte stores of 16 keys a CTA took 214.
constexpr int AG_KEYS = 64;
template <bool ANY>
__device__ __forceinline__ uint4 ag_load(const uint8_t* p) {
  if (!ANY) return __ldg(reinterpret_cast<const uint4*>(p));
  uint32_t w[4] = {0, 0, 0, 0};
#pragma unroll
  for (int i = 0; i < 16; ++i) w[i >> 2] |= (uint32_t)__ldg(p + i) << (8 * (i & 3));
  return make_uint4(w[0], w[1], w[2], w[3]);
}
template <int FMT, bool ANY>
__global__ void __launch_bounds__(256) kv_gather_kernel(const uint8_t* __restrict__ k_pool, const uint8_t* __restrict__ v_pool,
                                                        const float* __restrict__ k_scale, const float* __restrict__ v_scale,
                                                        const int* __restrict__ bt, int ctx, int ctx_pad, int hkv,
                                                        __nv_bfloat16* __restrict__ kout, __half* __restrict__ vt) {
  constexpr int HD = 256, ESZ = FMT == 2 ? 2 : 1, RAW = ESZ;        // 16-byte words per 16 elements
  __shared__ __align__(16) uint32_t vs[HD][AG_KEYS / 2];
  const int key0 = blockIdx.x * AG_KEYS, h = blockIdx.y, l16 = threadIdx.x & 15;
  uint4 kr[4][RAW], vr[4][RAW];
  float ks[4], vsc[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {           // keys 2 * (16 * (i / 2) + thread / 16) + i % 2
    const int key = key0 + (i >> 1) * 32 + (threadIdx.x >> 4) * 2 + (i & 1);
    const bool live = key < ctx;
    const size_t row = live ? ((size_t)bt[key / AG_PAGE] * AG_PAGE + key % AG_PAGE) * hkv + h : 0;
    ks[i] = FMT == 1 && live ? k_scale[row] : 1.f;
    vsc[i] = FMT == 1 && live ? v_scale[row] : 1.f;
#pragma unroll
    for (int r = 0; r < RAW; ++r) {
      kr[i][r] = live ? ag_load<ANY>(k_pool + row * HD * ESZ + (l16 * RAW + r) * 16) : make_uint4(0, 0, 0, 0);
      vr[i][r] = live ? ag_load<ANY>(v_pool + row * HD * ESZ + (l16 * RAW + r) * 16) : make_uint4(0, 0, 0, 0);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int key = key0 + (i >> 1) * 32 + (threadIdx.x >> 4) * 2 + (i & 1);
    float f[16];
    ag_floats<FMT>(kr[i], ks[i], f);
    __nv_bfloat16* kd = kout + ((size_t)h * ctx_pad + key) * HD + l16 * 16;
    if (ANY) {
#pragma unroll
      for (int k = 0; k < 16; ++k) kd[k] = __float2bfloat16(f[k]);
      continue;
    }
    uint4* ko = reinterpret_cast<uint4*>(kd);
    ko[0] = make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
    ko[1] = make_uint4(pack_bf16(f[8], f[9]), pack_bf16(f[10], f[11]), pack_bf16(f[12], f[13]), pack_bf16(f[14], f[15]));
  }
#pragma unroll
  for (int i = 0; i < 4; i += 2) {
    const int pair = (i >> 1) * 16 + (threadIdx.x >> 4);
    float a[16], b[16];
    ag_floats<FMT>(vr[i], vsc[i], a);
    ag_floats<FMT>(vr[i + 1], vsc[i + 1], b);
#pragma unroll
    for (int k = 0; k < 16; ++k) vs[l16 * 16 + k][pair ^ (2 * l16)] = pack_f16(a[k], b[k]);
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 8; ++i) {           // 8 lanes take the 64 keys of a dim
    const int d = i * 32 + (threadIdx.x >> 3), q = threadIdx.x & 7, sw = 2 * (d >> 4);
    uint4 u = *reinterpret_cast<const uint4*>(&vs[d][(4 * q) ^ (sw & ~3)]);
    if (sw & 2) u = make_uint4(u.z, u.w, u.x, u.y);
    reinterpret_cast<uint4*>(vt + ((size_t)h * HD + d) * ctx_pad + key0)[q] = u;
  }
}

// one CTA (256 threads) per score row; three passes over the row (max, sum, write)
__global__ void __launch_bounds__(256) causal_softmax_kernel(__half* __restrict__ s, int ld, int ncols, int pos0, float scale_log2,
                                                             int rpt, float* __restrict__ inv_sum) {
  __shared__ float red[32];
  const int r = blockIdx.x;
  __half* row = s + (size_t)r * ld;
  const int limit = min(pos0 + r / rpt + 1, ncols);
  float mx = -INFINITY;
  for (int c = threadIdx.x; c < limit; c += blockDim.x) mx = fmaxf(mx, __half2float(row[c]));
  mx = block_max(mx, red);
  float sum = 0.f;
  for (int c = threadIdx.x; c < limit; c += blockDim.x) sum += exp2f((__half2float(row[c]) - mx) * scale_log2);
  sum = block_sum(sum, red);
  for (int c = threadIdx.x; c < ncols; c += blockDim.x)
    row[c] = __float2half_rn(c < limit ? exp2f((__half2float(row[c]) - mx) * scale_log2) : 0.f);
  if (threadIdx.x == 0) inv_sum[r] = 1.f / sum;
}

// The row staged in shared memory (rows up to ~100 k keys): one vectorised read of the scores, one exponential per element, one
// vectorised write. The probabilities are left UNNORMALISED (largest = 1, which keeps them in the fp16 normal range however many
// keys a row sees); 1 / sum goes to inv_sum[row] and is applied to the output row after O = P V. ld and ncols are multiples of
// 8; dynamic shared memory = ncols halves.
__global__ void __launch_bounds__(512) causal_softmax_smem_kernel(__half* __restrict__ s, int ld, int ncols, int pos0, float scale_log2,
                                                                  int rpt, float* __restrict__ inv_sum) {
  extern __shared__ __align__(16) __half srow[];
  __shared__ float red[32];
  const int r = blockIdx.x;
  __half* row = s + (size_t)r * ld;
  const int limit = min(pos0 + r / rpt + 1, ncols);
  const int nfull = limit >> 3, nv = (limit + 7) >> 3, nv_all = ncols >> 3;   // fully visible chunks / chunks with a visible key / all
  __half2 m2 = __float2half2_rn(-65504.f);
  for (int c = threadIdx.x; c < nv; c += blockDim.x) {
    const uint4 u = reinterpret_cast<const uint4*>(row)[c];
    reinterpret_cast<uint4*>(srow)[c] = u;
    const __half2* h2 = reinterpret_cast<const __half2*>(&u);
    if (c < nfull) {
      m2 = __hmax2(m2, __hmax2(__hmax2(h2[0], h2[1]), __hmax2(h2[2], h2[3])));
    } else {
      const __half* h = reinterpret_cast<const __half*>(&u);
      for (int i = 0; i < limit - c * 8; ++i) m2 = __hmax2(m2, __half2half2(h[i]));
    }
  }
  const float mx = block_max(fmaxf(__low2float(m2), __high2float(m2)), red);
  const float bias = -mx * scale_log2;
  float sum = 0.f;
  for (int c = threadIdx.x; c < nv_all; c += blockDim.x) {
    uint4 u = make_uint4(0u, 0u, 0u, 0u);
    if (c < nv) {
      u = reinterpret_cast<const uint4*>(srow)[c];
      __half2* h2 = reinterpret_cast<__half2*>(&u);
      if (c < nfull) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 f = __half22float2(h2[i]);
          const float e0 = exp2f(fmaf(f.x, scale_log2, bias)), e1 = exp2f(fmaf(f.y, scale_log2, bias));
          sum += e0 + e1;
          h2[i] = __floats2half2_rn(e0, e1);
        }
      } else {
        __half* h = reinterpret_cast<__half*>(&u);
        for (int i = 0; i < 8; ++i) {
          const float e = c * 8 + i < limit ? exp2f(fmaf(__half2float(h[i]), scale_log2, bias)) : 0.f;
          sum += e;
          h[i] = __float2half_rn(e);
        }
      }
    }
    reinterpret_cast<uint4*>(row)[c] = u;
  }
  sum = block_sum(sum, red);
  if (threadIdx.x == 0) inv_sum[r] = 1.f / sum;
}

// y = o * sigmoid(gate): o bf16 [rows][HD], gate from the q projection output ([q_h | gate_h] per head, row stride ldq); y bf16 or
// fp16 [rows][HD]. grid (HD / 8 / 256 rounded up, rows).
__global__ void __launch_bounds__(256) attn_gate_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ qraw,
                                                        int ldq, int D, void* __restrict__ out, int HD, int out_f16, int gq,
                                                        const float* __restrict__ inv_sum) {
  pdl_launch_dependents();
  pdl_wait();
  const int row = blockIdx.y, c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= (HD >> 3)) return;
  const int e = c * 8, head = e / D, off = e % D;
  // gq > 0: o is stacked per kv head, [hkv][rows][gq][D] (the grouped GEMM's output); else [rows][HD]
  const __nv_bfloat16* src = gq > 0 ? o + ((((size_t)(head / gq) * gridDim.y + row) * gq + head % gq) * D + off)
                                    : o + (size_t)row * HD + e;
  const uint4 a = *reinterpret_cast<const uint4*>(src);
  // softmax denominator of this (token, head): same stacking as the grouped rows, or [head][rows] for the flat layout
  const float nrm = !inv_sum ? 1.f : gq > 0 ? inv_sum[((size_t)(head / gq) * gridDim.y + row) * gq + head % gq]
                                            : inv_sum[(size_t)head * gridDim.y + row];
  const uint4 g = *reinterpret_cast<const uint4*>(qraw + (size_t)row * ldq + (size_t)head * 2 * D + D + off);
  const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, gw[4] = {g.x, g.y, g.z, g.w};
  uint32_t r[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float y0 = nrm * bf16_lo(aw[i]) / (1.f + __expf(-bf16_lo(gw[i]))), y1 = nrm * bf16_hi(aw[i]) / (1.f + __expf(-bf16_hi(gw[i])));
    r[i] = out_f16 ? pack_f16(y0, y1) : pack_bf16(y0, y1);
  }
  reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(out) + (size_t)row * HD)[c] = make_uint4(r[0], r[1], r[2], r[3]);
}

}  // namespace owl
using namespace owl;

// q bf16 [rows][hq][D] -> qg [hkv][rows][gq][D]: the q heads of one kv head become consecutive rows of one GEMM operand.
__global__ void __launch_bounds__(256) q_group_kernel(const uint4* __restrict__ q, uint4* __restrict__ qg, int hq, int gq, int cpd) {
  pdl_launch_dependents();
  pdl_wait();
  const int row = blockIdx.y, rows = gridDim.y, c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= hq * cpd) return;
  const int head = c / cpd, off = c % cpd;
  qg[(((size_t)(head / gq) * rows + row) * gq + head % gq) * cpd + off] = q[(size_t)row * hq * cpd + c];
}

OWL_API int owl_q_group(const void* q, void* qg, int rows, int hq, int hkv, int D, cudaStream_t st) {
  if (rows < 1 || hkv < 1 || hq % hkv || (D & 7) || !q || !qg) return OWL_ERR_BAD_ARG;
  const int cpd = D / 8;
  return launch_dep(rows, q_group_kernel, dim3((hq * cpd + 255) / 256, rows), dim3(256), 0, st, (const uint4*)q, (uint4*)qg, hq, hq / hkv, cpd);
}

// gq > 0: `o` is the grouped layout [hkv][rows][gq][D]; gq = 0: [rows][HD].
OWL_API int owl_attn_gate(const void* o, const void* qraw, int ldq, int D, void* out, int rows, int HD, int out_f16, int gq,
                          const void* inv_sum, cudaStream_t st) {
  if (rows < 1 || (HD & 7) || (D & 7) || (ldq & 7) || !o || !qraw || !out || gq < 0) return OWL_ERR_BAD_ARG;
  return launch_dep(rows, attn_gate_kernel, dim3((HD / 8 + 255) / 256, rows), dim3(256), 0, st, (const __nv_bfloat16*)o, (const __nv_bfloat16*)qraw,
                    ldq, D, out, HD, out_f16, gq, (const float*)inv_sum);
}

// bt: the sequence's block-table row (int32 page numbers). fmt: 0 e4m3, 1 int8 with k_scale / v_scale [pages][16][hkv], 2 fp16.
OWL_API int owl_kv_gather(const void* k_pool, const void* v_pool, const void* k_scale, const void* v_scale, int fmt, const void* bt,
                          int ctx, int ctx_pad, int hkv, int hd, void* k_out, void* vt_out, cudaStream_t st) {
  if (hd != 256 || ctx < 1 || ctx_pad < ctx || (ctx_pad & 63) || hkv < 1 || fmt < 0 || fmt > 2 || (fmt == 1 && (!k_scale || !v_scale)))
    return OWL_ERR_BAD_ARG;
  if ((reinterpret_cast<uintptr_t>(vt_out) & 15) || (reinterpret_cast<uintptr_t>(k_out) & 1)) return OWL_ERR_BAD_ARG;
  const bool any = (reinterpret_cast<uintptr_t>(k_pool) | reinterpret_cast<uintptr_t>(v_pool) | reinterpret_cast<uintptr_t>(k_out)) & 15;
  const dim3 grid(ctx_pad / AG_KEYS, hkv);
  auto kernel = fmt == 0 ? (any ? kv_gather_kernel<0, true> : kv_gather_kernel<0, false>)
              : fmt == 1 ? (any ? kv_gather_kernel<1, true> : kv_gather_kernel<1, false>)
                         : (any ? kv_gather_kernel<2, true> : kv_gather_kernel<2, false>);
  kernel<<<grid, 256, 0, st>>>((const uint8_t*)k_pool, (const uint8_t*)v_pool, (const float*)k_scale, (const float*)v_scale, (const int*)bt, ctx,
                               ctx_pad, hkv, (__nv_bfloat16*)k_out, (__half*)vt_out);
  OWL_LAUNCH_CHECK();
  return OWL_OK;
}

// s: fp16 [rows][ld]; columns [0, ncols) are rewritten (probabilities, zeros past the causal limit pos0 + r + 1).
// rows_per_tok consecutive rows belong to one query token (the q heads of a kv head stacked per token).
// The probabilities are written unnormalised (row maximum = 1); inv_sum[row] = 1 / (row sum) scales the row of O = P V.
OWL_API int owl_causal_softmax(void* s, int rows, int ld, int ncols, int pos0, float scale, int rows_per_tok, void* inv_sum,
                               cudaStream_t st) {
  if (rows < 1 || ncols < 1 || ld < ncols || pos0 < 0 || rows_per_tok < 1 || !inv_sum) return OWL_ERR_BAD_ARG;
  const size_t smem = (size_t)ncols * 2;
  if (!(ld & 7) && !(ncols & 7) && !(reinterpret_cast<uintptr_t>(s) & 15) && smem <= 200 * 1024) {
    static SmemLimit limit;
    const int lrc = limit.raise(causal_softmax_smem_kernel, 200 * 1024);
    if (lrc != OWL_OK) return lrc;
    causal_softmax_smem_kernel<<<rows, 512, smem, st>>>((__half*)s, ld, ncols, pos0, scale * 1.4426950408889634f, rows_per_tok,
                                                        (float*)inv_sum);
  } else {
    causal_softmax_kernel<<<rows, 256, 0, st>>>((__half*)s, ld, ncols, pos0, scale * 1.4426950408889634f, rows_per_tok, (float*)inv_sum);
  }
  OWL_LAUNCH_CHECK();
  return OWL_OK;
}
