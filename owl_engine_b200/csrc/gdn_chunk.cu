// Chunked (WY representation) gated delta rule for prefill on tensor cores.
//
// The serial rule per v-head   S <- e^{g_t} S;  d_t = beta_t (v_t - k_t^T S);  S += k_t d_t^T;  o_t = scale q_t^T S
// is evaluated 64 tokens at a time. With gc = cumsum(g) inside a chunk, D_ij = e^{gc_i - gc_j},
//   A'  = strictly_lower(beta_i (k_i . k_j) D_ij)          T = (I + A')^-1
//   u   = T (beta v)             w = T (beta e^{gc} k)     attn = lower(scale (q_i . k_j) D_ij)
//   v'  = u - w S                o = (scale e^{gc} q) S + attn v'
//   S  <- e^{gc_last} S + (e^{gc_last - gc} k)^T v'
// (every exponential has a non-positive argument). Two kernels:
//   gdn_chunk_prep_kernel  one CTA per (chunk, v-head), all chunks in parallel: the 64x64 products and the two 64x128
//                          products on mma.sync (bf16 in, fp32 accumulate), the triangular inverse by forward substitution
//                          with four threads per column; writes w, u, scaled q, scaled k and attn
//   gdn_chunk_scan_kernel  one CTA per (v-head, part of the value columns), the chunks in order: three small tensor-core
//                          products per chunk against the fp32 state kept in MMA accumulator registers (a bf16 copy in
//                          shared memory is the B operand), operands prefetched one chunk ahead with cp.async
// Every tile stays in the row order it has in global memory; the products that need it the other way round read it with
// ldmatrix.trans. Before that the tiles were transposed through shared memory (8-way bank conflicts) and the fragments
// fetched word by word, and the inverse ran one column per thread through 2016 dependent steps: 168 us (preparation) and
// 117 us (recurrence) a layer at 2048 tokens x 48 heads; memory traffic would take 31 and 20 us. The operands, their rounding
// and the order of every sum are those of that form: the outputs are the same bits.
// followed by the gated RMSNorm kernel of gdn.cu. q and k arrive l2-normalised from the convolution kernel.
//
// Reference counterpart: the chunk-64 delta-rule kernels (cumsum, kkt, solve_tril, wu, h, o) that the reference compiles
// ahead of time from a Triton fork (crates/kernels/triton/gdn_chunked_*), launched around a state transpose. Tiles of 64
// rows are below the tcgen05 instruction shapes that pay (M = 128 per CTA), so this family stays on warp-level MMA.
#include "common.cuh"

namespace owl {

constexpr int CK_C = 64;            // chunk length
constexpr int CK_D = 128;           // head dim (k and v)
constexpr int CK_LD = CK_D + 8;     // row stride of [64][128] bf16 tiles (68 words: conflict-free fragment loads)
constexpr int CK_LT = CK_C + 8;     // row stride of [*][64] bf16 tiles
constexpr int CK_NC = 64;           // most value columns per CTA of the recurrence kernel

__device__ __forceinline__ void mma_bf16(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// Fragments through ldmatrix; ld in elements (rows of 16-byte multiples, 16 bytes past a multiple of 128: conflict-free).
__device__ __forceinline__ void ldm4(uint32_t* r, const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)) : "memory");
}
__device__ __forceinline__ void ldm4t(uint32_t* r, const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)) : "memory");
}
// A (16 x 16) of a tile stored [m][k] / [k][m]; B (16 x 16: two n-tiles, registers 0-1 and 2-3) stored [n][k] / [k][n]
__device__ __forceinline__ void frag_a(uint32_t* r, const __nv_bfloat16* s, int ld, int m0, int k0, int l) {
  ldm4(r, s + (m0 + (l & 15)) * ld + k0 + (l >> 4) * 8);
}
__device__ __forceinline__ void frag_at(uint32_t* r, const __nv_bfloat16* s, int ld, int m0, int k0, int l) {
  ldm4t(r, s + (k0 + (l & 7) + (l >> 4) * 8) * ld + m0 + ((l >> 3) & 1) * 8);
}
__device__ __forceinline__ void frag_b(uint32_t* r, const __nv_bfloat16* s, int ld, int n0, int k0, int l) {
  ldm4(r, s + (n0 + (l & 7) + (l >> 4) * 8) * ld + k0 + ((l >> 3) & 1) * 8);
}
__device__ __forceinline__ void frag_bt(uint32_t* r, const __nv_bfloat16* s, int ld, int n0, int k0, int l) {
  ldm4t(r, s + (k0 + (l & 15)) * ld + n0 + (l >> 4) * 8);
}
__device__ __forceinline__ void ck_cp16(void* smem_dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem_dst)), "l"(src) : "memory");
}

struct GdnChunkParams {
  const __nv_bfloat16* qkv;     // [T][conv_dim]: q | k (nk heads each, l2-normalised) | v (nv heads)
  const __nv_bfloat16* ab;      // [T][ldab]: a (nv) | b (nv)
  const float* a_log; const float* dt_bias;
  float* state;                 // [slots][nv][128 k][128 v]
  float* raw;                   // [T][nv * 128] un-normalised outputs
  __nv_bfloat16* w;             // [Tpad][nv][128]
  float* u;                     // [Tpad][nv][128] (fp32: v' = u - w S cancels)
  __nv_bfloat16* qg;            // [Tpad][nv][128]   scale e^{gc} q
  __nv_bfloat16* kd;            // [nv][chunks][64][128]   e^{gc_last - gc} k
  __nv_bfloat16* attn;          // [nv][chunks][64][64]
  float* eglast;                // [nv][chunks]
  int ldab, nk, nv, T, slot, use_state, chunks;
};

// ---- preparation: one CTA per (chunk, v-head), 256 threads, three CTAs per SM -------------------------------------------
struct PrepSmem {
  __nv_bfloat16 k[CK_C][CK_LD];       // k rows, later beta e^{gc} k
  __nv_bfloat16 v[CK_C][CK_LD];       // v rows, then beta v
  union {
    __nv_bfloat16 q[CK_C][CK_LD];
    __nv_bfloat16 tb[CK_C][CK_LT];    // T as bf16 (q is consumed by then)
  };
  float at[CK_C][CK_C + 4];           // A'^T (column j of A' is row j)
  float g[CK_C], gc[CK_C], beta[CK_C], eg[CK_C], el[CK_C];       // eg: e^{gc}, el: e^{gc_last - gc}
};
__device__ __forceinline__ uint4 scale_bf16x8(const uint4& u, float s) {
  return make_uint4(pack_bf16(bf16_lo(u.x) * s, bf16_hi(u.x) * s), pack_bf16(bf16_lo(u.y) * s, bf16_hi(u.y) * s),
                    pack_bf16(bf16_lo(u.z) * s, bf16_hi(u.z) * s), pack_bf16(bf16_lo(u.w) * s, bf16_hi(u.w) * s));
}
__device__ __forceinline__ uint4 scale2_bf16x8(const uint4& u, float s, float e) {      // (x s) e
  return make_uint4(pack_bf16(bf16_lo(u.x) * s * e, bf16_hi(u.x) * s * e), pack_bf16(bf16_lo(u.y) * s * e, bf16_hi(u.y) * s * e),
                    pack_bf16(bf16_lo(u.z) * s * e, bf16_hi(u.z) * s * e), pack_bf16(bf16_lo(u.w) * s * e, bf16_hi(u.w) * s * e));
}
__global__ void __launch_bounds__(256, 3) gdn_chunk_prep_kernel(GdnChunkParams p) {
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ __align__(16) uint8_t ck_smem[];
  PrepSmem& sm = *reinterpret_cast<PrepSmem*>(ck_smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
  const int c = blockIdx.x, h = blockIdx.y, R = p.nv / p.nk, hk = h / R;
  const int K = p.nk * CK_D, V = p.nv * CK_D, conv_dim = 2 * K + V, r0 = c * CK_C;
  const float scale = rsqrtf((float)CK_D);
  // 1. tiles (zero rows past T) and per-token scalars
  for (int i = tid; i < CK_C * 16; i += 256) {
    const int t = i >> 4, piece = (i & 15) * 8, r = r0 + t;
    if (r < p.T) {
      const __nv_bfloat16* xr = p.qkv + (size_t)r * conv_dim;
      ck_cp16(&sm.q[t][piece], xr + hk * CK_D + piece);
      ck_cp16(&sm.k[t][piece], xr + K + hk * CK_D + piece);
      ck_cp16(&sm.v[t][piece], xr + 2 * K + h * CK_D + piece);
    } else {
      const uint4 z = make_uint4(0, 0, 0, 0);
      *reinterpret_cast<uint4*>(&sm.q[t][piece]) = z;
      *reinterpret_cast<uint4*>(&sm.k[t][piece]) = z;
      *reinterpret_cast<uint4*>(&sm.v[t][piece]) = z;
    }
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  if (tid < CK_C) {
    const int r = r0 + tid;
    float gg = 0.f, bb = 0.f;
    if (r < p.T) {
      const float a = __bfloat162float(p.ab[(size_t)r * p.ldab + h]);
      const float b = __bfloat162float(p.ab[(size_t)r * p.ldab + p.nv + h]);
      gg = -__expf(p.a_log[h]) * softplus_f(a + p.dt_bias[h]);
      bb = sigmoid_f(b);
    }
    sm.g[tid] = gg;
    sm.beta[tid] = bb;
  }
  __syncthreads();
  if (tid == 0) {
    float4 gv[CK_C / 4];
#pragma unroll
    for (int i = 0; i < CK_C / 4; ++i) gv[i] = *reinterpret_cast<const float4*>(&sm.g[i * 4]);
    float acc = 0.f;
#pragma unroll
    for (int i = 0; i < CK_C / 4; ++i) {
      float4 o;
      acc += gv[i].x; o.x = acc; acc += gv[i].y; o.y = acc; acc += gv[i].z; o.z = acc; acc += gv[i].w; o.w = acc;
      *reinterpret_cast<float4*>(&sm.gc[i * 4]) = o;
    }
    p.eglast[(size_t)h * p.chunks + c] = __expf(acc);
  }
  __syncthreads();
  if (tid < CK_C) {
    sm.eg[tid] = __expf(sm.gc[tid]);
    sm.el[tid] = __expf(sm.gc[CK_C - 1] - sm.gc[tid]);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  // 2. scaled q rows and scaled k rows to global, beta v in place
  for (int i = tid; i < CK_C * 16; i += 256) {
    const int t = i >> 4, d = (i & 15) * 8;
    *reinterpret_cast<uint4*>(p.qg + ((size_t)(r0 + t) * p.nv + h) * CK_D + d) =
        scale_bf16x8(*reinterpret_cast<const uint4*>(&sm.q[t][d]), scale * sm.eg[t]);
    *reinterpret_cast<uint4*>(p.kd + (((size_t)h * p.chunks + c) * CK_C + t) * CK_D + d) =
        scale_bf16x8(*reinterpret_cast<const uint4*>(&sm.k[t][d]), sm.el[t]);
    uint4* v = reinterpret_cast<uint4*>(&sm.v[t][d]);
    *v = scale_bf16x8(*v, sm.beta[t]);
  }
  // 3. k k^T and q k^T (64 x 64 x 128): warp -> rows 16 (warp & 3), columns 32 (warp >> 2)
  {
    const int m0 = (warp & 3) * 16, nh = (warp >> 2) * 32;
    float kk[4][4], qk[4][4];
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) kk[n][i] = qk[n][i] = 0.f;
#pragma unroll
    for (int ks = 0; ks < CK_D / 16; ++ks) {
      uint32_t ak[4], aq[4];
      frag_a(ak, &sm.k[0][0], CK_LD, m0, ks * 16, lane);
      frag_a(aq, &sm.q[0][0], CK_LD, m0, ks * 16, lane);
#pragma unroll
      for (int n = 0; n < 4; n += 2) {
        uint32_t b[4];
        frag_b(b, &sm.k[0][0], CK_LD, nh + n * 8, ks * 16, lane);
        mma_bf16(kk[n], ak[0], ak[1], ak[2], ak[3], b[0], b[1]);
        mma_bf16(qk[n], aq[0], aq[1], aq[2], aq[3], b[0], b[1]);
        mma_bf16(kk[n + 1], ak[0], ak[1], ak[2], ak[3], b[2], b[3]);
        mma_bf16(qk[n + 1], aq[0], aq[1], aq[2], aq[3], b[2], b[3]);
      }
    }
    __nv_bfloat16* at = p.attn + ((size_t)h * p.chunks + c) * CK_C * CK_C;
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int i = m0 + g + half * 8, j = nh + n * 8 + 2 * t4;
        float av[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int jj = j + e;
          const float dec = jj <= i ? __expf(sm.gc[i] - sm.gc[jj]) : 0.f;
          sm.at[jj][i] = jj < i ? sm.beta[i] * kk[n][half * 2 + e] * dec : 0.f;
          av[e] = scale * qk[n][half * 2 + e] * dec;
        }
        *reinterpret_cast<uint32_t*>(at + i * CK_C + j) = pack_bf16(av[0], av[1]);
      }
  }
  __syncthreads();                    // q and k rows are consumed
  for (int i = tid; i < CK_C * 16; i += 256) {
    const int t = i >> 4, d = (i & 15) * 8;
    uint4* k = reinterpret_cast<uint4*>(&sm.k[t][d]);
    *k = scale2_bf16x8(*k, sm.beta[t], sm.eg[t]);
  }
  // 4. T = (I + A')^-1 by forward substitution. Four threads share column c; thread r holds rows 16 q + 4 r + e. When row j is
  // final, its holder tells the other three, and every later row takes its term: per element the terms come in order of j.
  {
    const int cc = tid >> 2, r = tid & 3;
    float acc[4][4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[q][e] = (16 * q + 4 * r + e == cc) ? 1.f : 0.f;
#pragma unroll
    for (int j = 0; j < CK_C - 1; ++j) {
      const float x = __shfl_sync(0xffffffffu, acc[j >> 4][j & 3], (lane & ~3) | ((j >> 2) & 3));
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (16 * q + 15 <= j) continue;
        const float4 a = *reinterpret_cast<const float4*>(&sm.at[j][16 * q + 4 * r]);
        const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (16 * q > j || 16 * q + 4 * r + e > j) acc[q][e] -= av[e] * x;
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int e = 0; e < 4; ++e) sm.tb[16 * q + 4 * r + e][cc] = __float2bfloat16(acc[q][e]);
  }
  __syncthreads();
  // 5. u = T (beta v), w = T (beta e^{gc} k)  (64 x 128 x 64): warp -> rows 16 (warp & 3), columns 64 (warp >> 2)
  {
    const int m0 = (warp & 3) * 16, nh = (warp >> 2) * 64;
    float uu[8][4], ww[8][4];
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) uu[n][i] = ww[n][i] = 0.f;
#pragma unroll
    for (int ks = 0; ks < CK_C / 16; ++ks) {
      uint32_t a[4];
      frag_a(a, &sm.tb[0][0], CK_LT, m0, ks * 16, lane);
#pragma unroll
      for (int n = 0; n < 8; n += 2) {
        uint32_t bv[4], bk[4];
        frag_bt(bv, &sm.v[0][0], CK_LD, nh + n * 8, ks * 16, lane);
        frag_bt(bk, &sm.k[0][0], CK_LD, nh + n * 8, ks * 16, lane);
        mma_bf16(uu[n], a[0], a[1], a[2], a[3], bv[0], bv[1]);
        mma_bf16(ww[n], a[0], a[1], a[2], a[3], bk[0], bk[1]);
        mma_bf16(uu[n + 1], a[0], a[1], a[2], a[3], bv[2], bv[3]);
        mma_bf16(ww[n + 1], a[0], a[1], a[2], a[3], bk[2], bk[3]);
      }
    }
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const size_t o = ((size_t)(r0 + m0 + g + half * 8) * p.nv + h) * CK_D + nh + n * 8 + 2 * t4;
        *reinterpret_cast<float2*>(p.u + o) = make_float2(uu[n][half * 2], uu[n][half * 2 + 1]);
        *reinterpret_cast<uint32_t*>(p.w + o) = pack_bf16(ww[n][half * 2], ww[n][half * 2 + 1]);
      }
  }
}

// ---- the recurrence over chunks: one CTA per (v-head, part of the value columns), 256 threads ----------------------------
// Bound by the chain of chunks, of which each takes 1.7 us with next to no products in it. The only split is by columns: into as many
// parts (2, 3, 4 or 8, of whole 8-column tiles) as leave every CTA an SM of its own; a part reads the other operands again, from L2.
// us a layer at 2048 tokens, two parts / the rule's: 48 heads 92 / 82 (three), 32 heads 90 / 64 (four), 16 heads 90 / 53 (eight; the 0.8B
// model's prompt of 2048 tokens 6.9 / 6.2 ms). The number of tiles is a template argument: as a variable it cost two parts 25 us. What
// lost: warps 8 to 15 for the outputs, so that 0 to 7 walk the chain alone (99 against 92 us): the state's fragments are read twice.
struct ScanBuf {
  __nv_bfloat16 w[CK_C][CK_LD];
  __nv_bfloat16 qg[CK_C][CK_LD];
  __nv_bfloat16 kd[CK_C][CK_LD];
  __nv_bfloat16 attn[CK_C][CK_LT];
  float u[CK_C][CK_NC + 4];         // this CTA's 64 columns (fp32)
};
struct ScanSmem {
  ScanBuf buf[2];
  __nv_bfloat16 s[CK_D][CK_LT];     // the state as bf16: [k][value column]
  __nv_bfloat16 vn[CK_C][CK_LT];    // v': [token][value column]
};
// Column tiles tile0 .. tile0 + NT - 1 (8 columns each) of one head.
template <int NT>
__device__ __forceinline__ void gdn_scan_part(const GdnChunkParams& p, int tile0) {
  constexpr int H1 = (NT + 1) / 2;                  // tiles of warps 0 to 3; warps 4 to 7 have one less of an odd number
  extern __shared__ __align__(16) uint8_t ck_smem[];
  ScanSmem& sm = *reinterpret_cast<ScanSmem*>(ck_smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
  const int h = blockIdx.x, V = p.nv * CK_D, cb = tile0 * 8;
  // state rows 16 warp .. +15, all columns of the part
  float S[NT][4];
  float* sp = p.state + ((size_t)p.slot * p.nv + h) * CK_D * CK_D;
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int k = warp * 16 + g + half * 8, col = cb + n * 8 + 2 * t4;
      const float2 v = p.use_state ? *reinterpret_cast<const float2*>(sp + (size_t)k * CK_D + col) : make_float2(0.f, 0.f);
      S[n][half * 2] = v.x;
      S[n][half * 2 + 1] = v.y;
    }
  auto issue = [&](int c) {
    if (c < p.chunks) {
      ScanBuf& b = sm.buf[c & 1];
      const int r0 = c * CK_C;
      for (int i = tid; i < CK_C * 16; i += 256) {
        const int t = i >> 4, piece = (i & 15) * 8;
        const size_t o = ((size_t)(r0 + t) * p.nv + h) * CK_D + piece;
        ck_cp16(&b.w[t][piece], p.w + o);
        ck_cp16(&b.qg[t][piece], p.qg + o);
        ck_cp16(&b.kd[t][piece], p.kd + (((size_t)h * p.chunks + c) * CK_C + t) * CK_D + piece);
        if (NT == 8 || piece < NT * 16) ck_cp16(&b.u[t][piece / 2], p.u + ((size_t)(r0 + t) * p.nv + h) * CK_D + cb + piece / 2);
      }
      for (int i = tid; i < CK_C * 8; i += 256) {
        const int t = i >> 3, piece = (i & 7) * 8;
        ck_cp16(&b.attn[t][piece], p.attn + (((size_t)h * p.chunks + c) * CK_C + t) * CK_C + piece);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  issue(0);
  for (int c = 0; c < p.chunks; ++c) {
    ScanBuf& b = sm.buf[c & 1];
    const int r0 = c * CK_C;
    const float eg = p.eglast[(size_t)h * p.chunks + c];
    // the state as the B operand of this chunk (the last reads of s are two barriers back)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int half = 0; half < 2; ++half)
        *reinterpret_cast<uint32_t*>(&sm.s[warp * 16 + g + half * 8][n * 8 + 2 * t4]) = pack_bf16(S[n][half * 2], S[n][half * 2 + 1]);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                 // chunk c and the state copy are visible; everyone is done with chunk c - 1
    issue(c + 1);
    // v' = u - w S and o = qg S: warp -> rows 16 (warp & 3), the first or second half of the column tiles (mine, from nh); K = 128
    const int m0 = (warp & 3) * 16, nh = (warp >> 2) * H1 * 8;
    const bool last = NT % 2 == 0 || warp < 4;       // this warp has a tile H1 - 1
    float pv[H1][4], ov[H1][4];
#pragma unroll
    for (int n = 0; n < H1; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) pv[n][i] = ov[n][i] = 0.f;
#pragma unroll
    for (int ks = 0; ks < CK_D / 16; ++ks) {
      uint32_t aw[4], aq[4];
      frag_a(aw, &b.w[0][0], CK_LD, m0, ks * 16, lane);
      frag_a(aq, &b.qg[0][0], CK_LD, m0, ks * 16, lane);
#pragma unroll
      for (int n = 0; n < H1; n += 2) {
        if (n == H1 - 1 && !last) continue;
        uint32_t bs[4];
        frag_bt(bs, &sm.s[0][0], CK_LT, nh + n * 8, ks * 16, lane);
        mma_bf16(pv[n], aw[0], aw[1], aw[2], aw[3], bs[0], bs[1]);
        mma_bf16(ov[n], aq[0], aq[1], aq[2], aq[3], bs[0], bs[1]);
        if (n + 1 == H1 || (n + 1 == H1 - 1 && !last)) continue;
        mma_bf16(pv[n + 1], aw[0], aw[1], aw[2], aw[3], bs[2], bs[3]);
        mma_bf16(ov[n + 1], aq[0], aq[1], aq[2], aq[3], bs[2], bs[3]);
      }
    }
#pragma unroll
    for (int n = 0; n < H1; ++n)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        if (n == H1 - 1 && !last) continue;
        const int i = m0 + g + half * 8, col = nh + n * 8 + 2 * t4;
        const float2 uw = *reinterpret_cast<const float2*>(&b.u[i][col]);
        *reinterpret_cast<uint32_t*>(&sm.vn[i][col]) = pack_bf16(uw.x - pv[n][half * 2], uw.y - pv[n][half * 2 + 1]);
      }
    __syncthreads();
    // S <- e^{gc_last} S + (e^{gc_last - gc} k)^T v': warp -> state rows 16 warp .. +15, all columns
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) S[n][i] *= eg;
    // and o += attn v'  (K = 64 tokens)
#pragma unroll
    for (int ks = 0; ks < CK_C / 16; ++ks) {
      uint32_t a[4], ak[4];
      frag_at(ak, &b.kd[0][0], CK_LD, warp * 16, ks * 16, lane);
      frag_a(a, &b.attn[0][0], CK_LT, m0, ks * 16, lane);
#pragma unroll
      for (int n = 0; n < NT; n += 2) {
        uint32_t bv[4];
        frag_bt(bv, &sm.vn[0][0], CK_LT, n * 8, ks * 16, lane);
        mma_bf16(S[n], ak[0], ak[1], ak[2], ak[3], bv[0], bv[1]);
        if (n + 1 == NT) continue;
        mma_bf16(S[n + 1], ak[0], ak[1], ak[2], ak[3], bv[2], bv[3]);
      }
#pragma unroll
      for (int n = 0; n < H1; n += 2) {
        if (n == H1 - 1 && !last) continue;
        uint32_t bv[4];
        frag_bt(bv, &sm.vn[0][0], CK_LT, nh + n * 8, ks * 16, lane);
        mma_bf16(ov[n], a[0], a[1], a[2], a[3], bv[0], bv[1]);
        if (n + 1 == H1 || (n + 1 == H1 - 1 && !last)) continue;
        mma_bf16(ov[n + 1], a[0], a[1], a[2], a[3], bv[2], bv[3]);
      }
    }
#pragma unroll
    for (int n = 0; n < H1; ++n)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int r = r0 + m0 + g + half * 8;
        if (r < p.T && (n < H1 - 1 || last))
          *reinterpret_cast<float2*>(p.raw + (size_t)r * V + h * CK_D + cb + nh + n * 8 + 2 * t4) =
              make_float2(ov[n][half * 2], ov[n][half * 2 + 1]);
      }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int k = warp * 16 + g + half * 8, col = cb + n * 8 + 2 * t4;
      *reinterpret_cast<float2*>(sp + (size_t)k * CK_D + col) = make_float2(S[n][half * 2], S[n][half * 2 + 1]);
    }
}
template <int PARTS>
__global__ void __launch_bounds__(256) gdn_chunk_scan_kernel(GdnChunkParams p) {
  pdl_launch_dependents();
  pdl_wait();
  const int tile0 = (int)blockIdx.y * 16 / PARTS;
  if (PARTS == 3 && blockIdx.y == 2) gdn_scan_part<6>(p, tile0);
  else gdn_scan_part<16 / PARTS>(p, tile0);
}

}  // namespace owl
using namespace owl;

static long long ck_work_bytes(int T, int nv) {
  const long long chunks = (T + CK_C - 1) / CK_C, tpad = chunks * CK_C;
  return tpad * nv * CK_D * 2 * 4 + (long long)nv * chunks * CK_D * CK_C * 2 + (long long)nv * chunks * CK_C * CK_C * 2 +
         (long long)nv * chunks * 4 + 1024;
}
// Bytes of the work buffer for T tokens and nv value heads -> *out_bytes (long long).
OWL_API int owl_gdn_chunk_work_bytes(int T, int nv, void* out_bytes) {
  if (T < 1 || nv < 1 || !out_bytes) return OWL_ERR_BAD_ARG;
  *reinterpret_cast<long long*>(out_bytes) = ck_work_bytes(T, nv);
  return OWL_OK;
}

// raw: float [T][nv * 128] (un-normalised outputs, input of the gated norm); work: owl_gdn_chunk_work_bytes(T, nv) bytes.
OWL_API int owl_gdn_chunk_scan(const void* qkv, const void* ab, int ldab, const void* a_log, const void* dt_bias, void* state,
                               int slot, void* raw, void* work, long long work_bytes, int T, int nk, int nv, int use_state,
                               cudaStream_t st) {
  if (T < 1 || nk < 1 || nv % nk || !raw || !work || work_bytes < ck_work_bytes(T, nv) ||
      (reinterpret_cast<uintptr_t>(work) & 255))
    return OWL_ERR_BAD_ARG;
  const int fit = sm_count() / nv, parts = fit >= 8 ? 8 : fit >= 4 ? 4 : fit == 3 ? 3 : 2;
  auto scan = parts == 8 ? gdn_chunk_scan_kernel<8> : parts == 4 ? gdn_chunk_scan_kernel<4> : parts == 3 ? gdn_chunk_scan_kernel<3> : gdn_chunk_scan_kernel<2>;
  static SmemLimit prep_limit, scan_limit[9];
  int lrc = prep_limit.raise(gdn_chunk_prep_kernel, (int)sizeof(PrepSmem));
  if (lrc == OWL_OK) lrc = scan_limit[parts].raise(scan, (int)sizeof(ScanSmem));
  if (lrc != OWL_OK) return lrc;
  GdnChunkParams p = {};
  p.qkv = (const __nv_bfloat16*)qkv; p.ab = (const __nv_bfloat16*)ab; p.a_log = (const float*)a_log; p.dt_bias = (const float*)dt_bias;
  p.state = (float*)state; p.raw = (float*)raw; p.ldab = ldab; p.nk = nk; p.nv = nv; p.T = T; p.slot = slot; p.use_state = use_state;
  p.chunks = (T + CK_C - 1) / CK_C;
  const size_t tpad = (size_t)p.chunks * CK_C, rows = tpad * nv * CK_D;
  auto* base = reinterpret_cast<__nv_bfloat16*>(work);
  p.u = reinterpret_cast<float*>(base);                 // 2 * rows bf16-sized elements
  p.w = base + 2 * rows; p.qg = base + 3 * rows;
  p.kd = base + 4 * rows;
  p.attn = p.kd + (size_t)nv * p.chunks * CK_D * CK_C;
  p.eglast = reinterpret_cast<float*>(p.attn + (size_t)nv * p.chunks * CK_C * CK_C);
  const int rc = launch_dep(T, gdn_chunk_prep_kernel, dim3(p.chunks, nv), dim3(256), sizeof(PrepSmem), st, p);
  if (rc != OWL_OK) return rc;
  return launch_dep(T, scan, dim3(nv, parts), dim3(256), sizeof(ScanSmem), st, p);
}
