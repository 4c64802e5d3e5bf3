// Weight-streaming projections for 1..32 rows (decode, verify, short prompts) on the 16-bit warp-level tensor path.
//
//   owl_w4_mma    : C[M,N] = X[M,K] . dequant(W4)[N,K]^T      int4 records, group 32 / 128 (slice-major, see gemv.cu)
//   owl_nvfp4_mma : C[M,N] = X[M,K] . dequant(NVFP4)[N,K]^T   codes and block scales as stored in the checkpoint
//   both with store / residual add / silu(gate) * up epilogues and, beside the matrix, a few dense bf16 rows (the GDN a / b
//   projections) computed by CTAs of the same grid
//
// No dequantisation: a nibble masked in place (q & 0x000f000f, q & 0x00f000f0, and the same on q >> 8) IS a pair of bf16
// subnormals n * 2^-133 and 16 n * 2^-133 (subnormals and the first binade lie on one line), and the tensor path keeps
// them. The activations come as bf16 times 2^64 (an exponent shift: exact, and the activations under the x16 nibbles
// carry 2^60), so a product is an exact 12-bit integer times a power of two, accumulated in fp32 per group:
//     y += s * (dot - z * sum(x)).
// The integer arm (gemv.cu) rounds the activations to 15 bits, needs two MMAs per 32 k and converts its int32 sums; this
// one rounds nothing before the fp32 sums. Activations of magnitude 2^63 and above become infinite here, and below about 2^-57 fp32
// ends under the products; prompts and the one-token arm carry activations as fp16, whose range is inside that.
// NVFP4: the codes are converted to fp16 pairs by the conversion unit (6.6 clocks a word of eight; moving their bits to the
// sign and exponent places of a bf16 took 15 integer instructions, 19 clocks) and multiplied by the block scale (4 x 2
// significant bits: exact in fp16); the activations are fp16 with a power of two per 128 that the sums are rescaled by.
//
// What bounds it: 0.53 bytes per weight over HBM. An SM receives about 23.5 bytes per clock, one 1088-byte record per 185
// clocks and sub-core; per record this kernel issues 40 mask / shift instructions (two clocks each), 8 MMAs per 8 rows at 8
// clocks each, and about 30 others. Up to 8 rows the stream and the launch-to-launch dependency (about 4 us) are the bound,
// at 32 rows the MMAs and the shared-memory reads of their fragments.
//
// Shape of the work. A CTA is 4 warps x 2 row tiles = 128 rows over one part of k; the KS parts of a row block form a
// thread-block cluster and reduce through distributed shared memory in rank order, so a row's sums have one order that
// depends on N, K and the device's SMs only: a row computes the same bits whatever the number of rows in the step. KS is chosen so that
// one wave of CTAs (4 per SM) covers the matrix: the 5120-row projections would leave 108 SMs idle otherwise. Two row tiles
// per warp halve the activation bytes per weight byte. The activations come in MMA fragment order (actpack.cuh, ACT_FRAG) and
// ride in the same ring of asynchronous copies as the weights, shared by the CTA's warps: read through L1 instead, their L2
// latency was exposed four times a record.
//
// Measured (one B200, graph of dependent launches over rotating weights, group 128; HBM time of the weights; 1 / 8 / 32 rows):
//   16384 x 5120  6.7 us: 10.5 / 10.8 / 25.3    5120 x 6144   2.5 us: 6.9 / 7.0 / 14.6
//   34816 x 5120 14.2 us: 18.8 / 19.5 / 44.0    5120 x 17408  7.1 us: 12.9 / 13.1 / 28.5
// (the integer arm in a step of 8 / 32 rows: 23 / 82 us on average over the four; the NVFP4 GEMV 88 us at 4 rows, here 20.)
//
// Role in the reference: the Marlin W4A16 decode path and the NVFP4 GEMV (crates/kernels/cu/marlin/*,
// crates/kernels/cu/nvfp4/nvfp4_gemv.cu).
#include <cuda_fp8.h>
#include "common.cuh"
#include "actpack.cuh"

namespace owl {

enum { MF_G128 = 0, MF_G32 = 1, MF_NV4 = 2 };
enum { MEPI_STORE = 0, MEPI_RESIDUAL = 1, MEPI_SILU_MUL = 2 };
constexpr int MM_WARPS = 4;       // warps per CTA
constexpr int MM_R = 2;           // row tiles (16 rows) per warp
constexpr int MM_TILES = MM_WARPS * MM_R;

struct MmaParams {
  const uint8_t* w;               // int4: record stream; NVFP4: codes [N][K/2]
  const uint8_t* sf;              // NVFP4: e4m3 block scales [N][K/16]
  const float* row_scale;         // NVFP4, optional: fp32 [N]
  const uint4* x;                 // ACT_FRAG chunks
  const float4* xs;               // ACT_FRAG (scale, sum) pairs of two tokens
  __nv_bfloat16* out;
  const __nv_bfloat16* residual;
  const __nv_bfloat16* ab_w;      // optional dense rows [ab_rows][K] ...
  const __nv_bfloat16* ab_x;      // ... times plain bf16 rows [M][K]
  __nv_bfloat16* ab_out;          // [M][ab_ld]
  float out_scale;
  int M, N, K, ldo, n_tiles, ab_rows, ab_ld, ab_blocks;
};

__device__ __forceinline__ void mm_bf16(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mm_bf16_z(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void mm_f16(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mm_f16_z(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ uint32_t mm_mul2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
// eight e2m1 codes -> four fp16 pairs
__device__ __forceinline__ void mm_e2m1x8(uint32_t q, uint32_t* d) {
  asm("{\n\t.reg .b8 a, b, c, d;\n\tmov.b32 {a, b, c, d}, %4;\n\tcvt.rn.f16x2.e2m1x2 %0, a;\n\tcvt.rn.f16x2.e2m1x2 %1, b;\n\t"
      "cvt.rn.f16x2.e2m1x2 %2, c;\n\tcvt.rn.f16x2.e2m1x2 %3, d;\n\t}"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(q));
}
__device__ __forceinline__ void mm_cp16(uint32_t smem_dst, const void* gsrc) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_dst), "l"(gsrc) : "memory");
}
// The same for rows of which a stage takes 64 bytes: the rest of the line is fetched along (NVFP4: 3 % at 4 rows).
__device__ __forceinline__ void mm_cp16_ahead(uint32_t smem_dst, const void* gsrc) {
  asm volatile("cp.async.cg.shared.global.L2::256B [%0], [%1], 16;" ::"r"(smem_dst), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void mm_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void mm_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void cl_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cl_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t cl_map(uint32_t addr, int rank) {
  uint32_t d;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(addr), "r"(rank));
  return d;
}
__device__ __forceinline__ void cl_store2(uint32_t addr, float a, float b) {
  asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(a), "f"(b) : "memory");
}

// bytes of one tile's record in the ring (NVFP4: 16 rows x 64 code bytes, then 16 rows x 8 scale bytes)
template <int FMT> __host__ __device__ constexpr int mm_rec() { return FMT == MF_G128 ? 1088 : FMT == MF_G32 ? 1280 : 1152; }
__host__ __device__ constexpr int mm_red_ld(int mt) { return mt * 8 + 2; }
// One ring stage: the record of every tile, the activation fragments of the record column, their (scale, sum) pairs.
template <int FMT> __host__ __device__ constexpr int mm_pairs() { return FMT == MF_G32 ? 4 : 1; }
template <int FMT, int MT> __host__ __device__ constexpr int mm_stage() {
  return MM_TILES * mm_rec<FMT>() + MT * (2048 + mm_pairs<FMT>() * 64);
}
// The partial tiles arrive in a buffer behind the ring, or in the ring's own bytes where both would cost a stage too many.
template <int MT> __host__ __device__ constexpr int mm_in_bytes() { return MM_TILES * 16 * mm_red_ld(MT) * 4; }
template <int FMT, int MT, int CT> __host__ __device__ constexpr bool mm_alias() { return FMT != MF_NV4 && MT > 2 && (CT == 4 || (FMT == MF_G32 && MT == 4)); }
// Token blocks per pass over a record's nibbles: above 16 rows the int4 forms of four CTAs per SM unpack a record twice, which
// keeps the sums of one pass in the registers that leaves (34816 x 5120, 20 / 32 rows: 34 / 44 us against 37 / 45 in two waves of
// three; 16384 x 5120: 20 / 25 against 24 / 29). With three CTAs per SM one pass is faster (5120 x 17408, 32 rows: 28.5 against
// 31.4), but for 32 rows of group 32, whose sums spill (37 against 40).
template <int FMT, int MT, int CT> __host__ __device__ constexpr int mm_pass() {
  return FMT != MF_NV4 && MT > 2 && (CT == 4 || (FMT == MF_G32 && MT == 4)) ? 2 : MT;
}
// Ring stages: what CT resident CTAs per SM leave room for.
template <int FMT, int MT, int CT> __host__ __device__ constexpr int mm_stages() {
  return (227 * 1024 / CT - 1024 - (mm_alias<FMT, MT, CT>() ? 0 : mm_in_bytes<MT>())) / mm_stage<FMT, MT>();
}
template <int FMT, int MT, int CT> __host__ __device__ constexpr int mm_ring() { return mm_stages<FMT, MT, CT>() * mm_stage<FMT, MT>(); }
template <int FMT, int MT, int CT> constexpr int mm_smem() {
  return mm_ring<FMT, MT, CT>() + (mm_alias<FMT, MT, CT>() ? 0 : mm_in_bytes<MT>());
}

// Every CTA of the cluster owns 8 / KS of the row block's tiles. The CTAs push their partial tiles into the owners' buffers
// [rank][tile][16 rows][mm_red_ld] (posted stores: reading the peers' buffers instead cost a round trip per peer and a second
// barrier before the exit), and the owner adds them in rank order.
template <int MT, int KS>
__device__ __forceinline__ void mm_reduce(const MmaParams& p, int epi, const float* in, int rank, int nt0) {
  constexpr int LD = mm_red_ld(MT), PER = MM_TILES / KS;
  const int M = p.M;
  for (int i = threadIdx.x; i < PER * M * 8; i += MM_WARPS * 32) {
    const int rp = i & 7, tok = (i >> 3) % M, tl = (i >> 3) / M, nt = nt0 + rank * PER + tl;
    if (nt >= p.n_tiles) continue;
    const int ra = epi == MEPI_SILU_MUL ? rp : 2 * rp, rb = epi == MEPI_SILU_MUL ? rp + 8 : 2 * rp + 1;
    float a = 0.f, b = 0.f;
#pragma unroll
    for (int q = 0; q < KS; ++q) {
      a += in[((q * PER + tl) * 16 + ra) * LD + tok];
      b += in[((q * PER + tl) * 16 + rb) * LD + tok];
    }
    float sa = p.out_scale, sb = sa;
    if (p.row_scale) { sa *= p.row_scale[nt * 16 + ra]; sb *= p.row_scale[nt * 16 + rb]; }
    a *= sa; b *= sb;
    if (epi == MEPI_SILU_MUL) {
      p.out[(size_t)tok * p.ldo + nt * 8 + rp] = __float2bfloat16(silu_f(a) * b);
    } else {
      const size_t o = (size_t)tok * p.ldo + nt * 16 + 2 * rp;
      if (epi == MEPI_RESIDUAL) {
        const uint32_t rr = *reinterpret_cast<const uint32_t*>(p.residual + o);
        a += bf16_lo(rr); b += bf16_hi(rr);
      }
      *reinterpret_cast<uint32_t*>(p.out + o) = pack_bf16(a, b);
    }
  }
}

// Dense bf16 rows: 16 rows per cluster, rank and warp split k.
template <int MT>
__device__ __forceinline__ void mm_dense_block(const MmaParams& p, float* red, int KS, int rank, int blk) {
  constexpr int LD = mm_red_ld(MT);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int parts = KS * MM_WARPS, part = rank * MM_WARPS + warp;
  const int nc = p.K / 32;                            // 32-k steps: 8 k per lane quarter
  const int c0 = part * nc / parts, c1 = (part + 1) * nc / parts;
  const int r0 = min(blk * 16 + g, p.ab_rows - 1), r1 = min(blk * 16 + g + 8, p.ab_rows - 1);
  const uint4* w0 = reinterpret_cast<const uint4*>(p.ab_w + (size_t)r0 * p.K) + t;
  const uint4* w1 = reinterpret_cast<const uint4*>(p.ab_w + (size_t)r1 * p.K) + t;
  float acc[MT][4];
#pragma unroll
  for (int m = 0; m < MT; ++m) acc[m][0] = acc[m][1] = acc[m][2] = acc[m][3] = 0.f;
  const uint4* xr[MT];
#pragma unroll
  for (int m = 0; m < MT; ++m) xr[m] = reinterpret_cast<const uint4*>(p.ab_x + (size_t)min(m * 8 + g, p.M - 1) * p.K) + t;
#pragma unroll 4
  for (int c = c0; c < c1; ++c) {
    const uint4 a = w0[c * 4], b = w1[c * 4];
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      const uint4 xv = xr[m][c * 4];
      mm_bf16(acc[m], a.x, b.x, a.y, b.y, xv.x, xv.y);
      mm_bf16(acc[m], a.z, b.z, a.w, b.w, xv.z, xv.w);
    }
  }
#pragma unroll
  for (int m = 0; m < MT; ++m) {
    float* r = red + (warp * 16 + g) * LD + m * 8 + 2 * t;
    *reinterpret_cast<float2*>(r) = make_float2(acc[m][0], acc[m][1]);
    *reinterpret_cast<float2*>(r + 8 * LD) = make_float2(acc[m][2], acc[m][3]);
  }
  __syncthreads();
  float* in = red + MM_WARPS * 16 * LD;               // [rank][16 rows][LD] of rank 0
  const uint32_t dst = cl_map(smem_u32(in) + rank * 16 * LD * 4, 0);
  cl_wait();
  for (int i = threadIdx.x; i < 16 * MT * 4; i += MM_WARPS * 32) {
    const int row = i / (MT * 4), c = (i % (MT * 4)) * 2;
    float a = 0.f, b = 0.f;
#pragma unroll
    for (int s = 0; s < MM_WARPS; ++s) { a += red[(s * 16 + row) * LD + c]; b += red[(s * 16 + row) * LD + c + 1]; }
    cl_store2(dst + (row * LD + c) * 4, a, b);
  }
  cl_arrive();
  cl_wait();
  if (rank == 0) {
    for (int i = threadIdx.x; i < p.M * 16; i += MM_WARPS * 32) {
      const int row = i & 15, tok = i >> 4;
      if (blk * 16 + row >= p.ab_rows) continue;
      float a = 0.f;
      for (int q = 0; q < KS; ++q) a += in[(q * 16 + row) * LD + tok];
      p.ab_out[(size_t)tok * p.ab_ld + blk * 16 + row] = __float2bfloat16(a);
    }
  }
}

// grid KS * (ab_blocks + row blocks), cluster KS. A8: the activations are 8-bit integers with a scale per (token, group).
template <int FMT, int MT, bool A8, int CT>
__global__ void __launch_bounds__(MM_WARPS * 32, CT) w4_mma_kernel(MmaParams p, int epi, int KS) {
  constexpr int REC = mm_rec<FMT>(), STAGE = mm_stage<FMT, MT>(), LD = mm_red_ld(MT), S = mm_stages<FMT, MT, CT>();
  constexpr int GPR = mm_pairs<FMT>();                  // groups per record
  constexpr int XOFF = MM_TILES * REC, SOFF = XOFF + MT * 2048;      // of the fragments and the pairs in a stage
  extern __shared__ __align__(128) uint8_t smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int rank = KS > 1 ? (int)(blockIdx.x % KS) : 0;
  cl_arrive();                          // the peers run before anything is stored in their shared memory
  const int blk = (int)(blockIdx.x / KS) - p.ab_blocks;
  if (blk < 0) {
    pdl_launch_dependents();
    pdl_wait();
    mm_dense_block<MT>(p, reinterpret_cast<float*>(smem), KS, rank, blk + p.ab_blocks);
    return;
  }
  const int nt0 = blk * MM_TILES, KT = p.K >> 7;
  // this warp's tiles (past the end: the last tile again, never stored)
  const int ta = min(nt0 + warp * MM_R, p.n_tiles - 1), tb = min(nt0 + warp * MM_R + 1, p.n_tiles - 1);
  const int kb = rank * KT / KS, total = (rank + 1) * KT / KS - kb;
  const uint8_t* ring = smem + warp * MM_R * REC;         // this warp's records of stage 0
  const uint32_t ring_s = smem_u32(ring) + lane * 16, x_s = smem_u32(smem) + XOFF + threadIdx.x * 16;
  int to_issue = total, x_issue = total;

  // ---- fetch side ----------------------------------------------------------------------------------------------
  // int4: record (tile, kt) lies in k slice s = the eighth of the record columns that holds kt, at
  // (n_tiles * kt0_s + tile * rpi_s + kt - kt0_s). NVFP4: 16 rows of 64 code bytes (4 lanes x 16 per row) and 8 scale bytes.
  int sl = 0, left = 0;
  const uint8_t *src_a = nullptr, *src_b = nullptr, *sfp = nullptr;
  size_t row8 = 0;
  auto enter_slice = [&](int kt) {      // positions the fetch pointers at record column kt of slice sl
    const int k0 = sl * KT / 8, rpi = (sl + 1) * KT / 8 - k0;
    src_a = p.w + ((size_t)p.n_tiles * k0 + (size_t)ta * rpi + (kt - k0)) * REC + lane * 16;
    src_b = src_a + (size_t)(tb - ta) * rpi * REC;
    left = rpi - (kt - k0);
  };
  if (FMT == MF_NV4) {
    row8 = (size_t)8 * (p.K >> 1);
    src_a = p.w + (size_t)(ta * 16 + g) * (p.K >> 1) + (size_t)kb * 64 + t * 16;
    src_b = src_a + (size_t)(tb - ta) * 2 * row8;
    // scales: lane L copies the 8 bytes of row L % 16 of tile L / 16
    sfp = p.sf + (size_t)((lane < 16 ? ta : tb) * 16 + (lane & 15)) * (p.K >> 4) + (size_t)kb * 8;
  } else if (total > 0) {
    while ((sl + 1) * KT / 8 <= kb) ++sl;
    enter_slice(kb);
  }
  auto issue = [&](uint32_t st) {
    if (to_issue > 0) {
      if (FMT == MF_NV4) {
        mm_cp16_ahead(ring_s + st, src_a);
        mm_cp16_ahead(ring_s + st + 512, src_a + row8);
        mm_cp16_ahead(ring_s + st + REC, src_b);
        mm_cp16_ahead(ring_s + st + REC + 512, src_b + row8);
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(ring_s - lane * 16 + st + (lane >> 4) * REC + 1024 + (lane & 15) * 8),
                     "l"(sfp) : "memory");
        src_a += 64;
        src_b += 64;
        sfp += 8;
      } else {
        mm_cp16(ring_s + st, src_a);
        mm_cp16(ring_s + st + 512, src_a + 512);
        if (lane < (REC - 1024) / 16) mm_cp16(ring_s + st + 1024, src_a + 1024);
        mm_cp16(ring_s + st + REC, src_b);
        mm_cp16(ring_s + st + REC + 512, src_b + 512);
        if (lane < (REC - 1024) / 16) mm_cp16(ring_s + st + REC + 1024, src_b + 1024);
        src_a += REC;
        src_b += REC;
        if (--left == 0 && to_issue > 1) {
          ++sl;
          while ((sl + 1) * KT / 8 == sl * KT / 8) ++sl;      // empty slices of a narrow matrix
          enter_slice(sl * KT / 8);
        }
      }
    }
    --to_issue;
  };
  const size_t xm = (size_t)KT * 128, xsm = (size_t)KT * GPR * 4;          // 16-byte words per block of 8 tokens
  const uint4* xp = p.x + (size_t)kb * 128 + threadIdx.x;             // the 128 threads copy one block of 8 tokens at a time
  const float4* xsp = p.xs + (size_t)kb * GPR * 4 + (GPR ? threadIdx.x % (GPR * 4) : 0) + (GPR ? threadIdx.x / (GPR * 4) : 0) * xsm;
  auto issue_x = [&](uint32_t st) {
    if (x_issue > 0) {
#pragma unroll
      for (int m = 0; m < MT; ++m) mm_cp16(x_s + st + m * 2048, xp + m * xm);
      if (GPR && (int)threadIdx.x < MT * GPR * 4) mm_cp16(x_s + st + MT * 2048, xsp);
      xp += 128;
      xsp += GPR * 4;
    }
    --x_issue;
    mm_commit();
  };
  // the weights do not depend on the previous kernel: the stream starts before the dependency wait
#pragma unroll
  for (int j = 0; j < S - 1; ++j) issue(j * STAGE);
  pdl_launch_dependents();
  pdl_wait();
#pragma unroll
  for (int j = 0; j < S - 1; ++j) issue_x(j * STAGE);

  float acc[MM_R][MT][4];
#pragma unroll
  for (int r = 0; r < MM_R; ++r)
#pragma unroll
    for (int m = 0; m < MT; ++m) acc[r][m][0] = acc[r][m][1] = acc[r][m][2] = acc[r][m][3] = 0.f;
  uint32_t st_c = 0, st_i = (S - 1) * STAGE;
  for (int j = 0; j < total; ++j) {
    mm_wait<S - 2>();
    __syncthreads();                    // everybody's copies of the stage, and everybody left the stage refilled next
    issue(st_i);
    issue_x(st_i);
    st_i = st_i == (S - 1) * STAGE ? 0u : st_i + STAGE;
    const uint8_t* rec = ring + st_c;
    const uint4* xf = reinterpret_cast<const uint4*>(smem + st_c + XOFF) + lane;
    const float4* xg = reinterpret_cast<const float4*>(smem + st_c + SOFF) + t;
    st_c = st_c == (S - 1) * STAGE ? 0u : st_c + STAGE;
    uint4 lo[MM_R], hi[MM_R];
#pragma unroll
    for (int r = 0; r < MM_R; ++r) {
      lo[r] = *reinterpret_cast<const uint4*>(rec + r * REC + lane * 16);
      hi[r] = *reinterpret_cast<const uint4*>(rec + r * REC + 512 + lane * 16);
    }
    if constexpr (FMT == MF_NV4) {
      // this lane's blocks: 16-k blocks 2t and 2t + 1 of rows g and g + 8
      uint32_t sc[MM_R][2][2];          // [tile][row half][block]: the scale in both halves of an fp16 pair
#pragma unroll
      for (int r = 0; r < MM_R; ++r)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint16_t b2 = *reinterpret_cast<const uint16_t*>(rec + r * REC + 1024 + (g + 8 * h) * 8 + 2 * t);
          const __half2 s2 = __half2(__nv_cvt_fp8x2_to_halfraw2(b2, __NV_E4M3));
          const __half2 s0 = __low2half2(s2), s1 = __high2half2(s2);
          sc[r][h][0] = *reinterpret_cast<const uint32_t*>(&s0);
          sc[r][h][1] = *reinterpret_cast<const uint32_t*>(&s1);
        }
      float dot[MM_R][MT][4];
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        uint32_t fa[MM_R][8];
#pragma unroll
        for (int r = 0; r < MM_R; ++r)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const uint4& u = h ? hi[r] : lo[r];
            uint32_t d[4];
            mm_e2m1x8(w == 0 ? u.x : w == 1 ? u.y : w == 2 ? u.z : u.w, d);
#pragma unroll
            for (int i = 0; i < 4; ++i) fa[r][2 * i + h] = mm_mul2(d[i], sc[r][h][w >> 1]);
          }
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          const uint4 xv = xf[m * 128 + w * 32];
#pragma unroll
          for (int r = 0; r < MM_R; ++r) {
            if (w == 0) mm_f16_z(dot[r][m], fa[r][0], fa[r][1], fa[r][2], fa[r][3], xv.x, xv.y);
            else mm_f16(dot[r][m], fa[r][0], fa[r][1], fa[r][2], fa[r][3], xv.x, xv.y);
          }
#pragma unroll
          for (int r = 0; r < MM_R; ++r) mm_f16(dot[r][m], fa[r][4], fa[r][5], fa[r][6], fa[r][7], xv.z, xv.w);
        }
      }
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        const float4 xv = xg[m * 4];     // the powers of two of tokens 2t and 2t + 1
#pragma unroll
        for (int r = 0; r < MM_R; ++r) {
          acc[r][m][0] = fmaf(dot[r][m][0], xv.x, acc[r][m][0]);
          acc[r][m][1] = fmaf(dot[r][m][1], xv.z, acc[r][m][1]);
          acc[r][m][2] = fmaf(dot[r][m][2], xv.x, acc[r][m][2]);
          acc[r][m][3] = fmaf(dot[r][m][3], xv.z, acc[r][m][3]);
        }
      }
    } else {
      constexpr bool G32 = FMT == MF_G32;
      constexpr int MP = mm_pass<FMT, MT, CT>();
#pragma unroll
      for (int mb = 0; mb < MT; mb += MP) {
      float dot[MM_R][MP][4];
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        uint32_t fa[MM_R][8];
#pragma unroll
        for (int r = 0; r < MM_R; ++r)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const uint4& u = h ? hi[r] : lo[r];
            uint32_t q = w == 0 ? u.x : w == 1 ? u.y : w == 2 ? u.z : u.w;
            fa[r][0 + h] = q & 0x000f000fu;
            fa[r][2 + h] = q & 0x00f000f0u;
            q >>= 8;
            fa[r][4 + h] = q & 0x000f000fu;
            fa[r][6 + h] = q & 0x00f000f0u;
          }
        const bool first = G32 || w == 0, last = G32 || w == 3;
#pragma unroll
        for (int m = 0; m < MP && mb + m < MT; ++m) {
          const uint4 xv = xf[(mb + m) * 128 + w * 32];
#pragma unroll
          for (int r = 0; r < MM_R; ++r) {
            if (first) mm_bf16_z(dot[r][m], fa[r][0], fa[r][1], fa[r][2], fa[r][3], xv.x, xv.y);
            else mm_bf16(dot[r][m], fa[r][0], fa[r][1], fa[r][2], fa[r][3], xv.x, xv.y);
          }
#pragma unroll
          for (int r = 0; r < MM_R; ++r) mm_bf16(dot[r][m], fa[r][4], fa[r][5], fa[r][6], fa[r][7], xv.z, xv.w);
        }
        if (last) {
          const int q = G32 ? w : 0;
          float2 s0[MM_R], s1[MM_R];      // (scale, zero) of rows g and g + 8
#pragma unroll
          for (int r = 0; r < MM_R; ++r) {
            s0[r] = __half22float2(*reinterpret_cast<const __half2*>(rec + r * REC + 1024 + q * 64 + g * 4));
            s1[r] = __half22float2(*reinterpret_cast<const __half2*>(rec + r * REC + 1024 + q * 64 + 32 + g * 4));
          }
#pragma unroll
          for (int m = 0; m < MP && mb + m < MT; ++m) {
            const float4 xv = xg[(mb + m) * GPR * 4 + q * 4];       // (scale, sum) of tokens 2t and 2t + 1
#pragma unroll
            for (int r = 0; r < MM_R; ++r) {
              float* d = dot[r][m];
              if (A8) { d[0] *= xv.x; d[1] *= xv.z; d[2] *= xv.x; d[3] *= xv.z; }
              float* o = acc[r][mb + m];
              o[0] = fmaf(s0[r].x, fmaf(-s0[r].y, xv.y, d[0]), o[0]);
              o[1] = fmaf(s0[r].x, fmaf(-s0[r].y, xv.w, d[1]), o[1]);
              o[2] = fmaf(s1[r].x, fmaf(-s1[r].y, xv.y, d[2]), o[2]);
              o[3] = fmaf(s1[r].x, fmaf(-s1[r].y, xv.w, d[3]), o[3]);
            }
          }
        }
      }
      }
    }
  }
  mm_wait<0>();
  cl_wait();
  float* in = reinterpret_cast<float*>(smem + (mm_alias<FMT, MT, CT>() ? 0 : mm_ring<FMT, MT, CT>()));
  if (mm_alias<FMT, MT, CT>()) { cl_arrive(); cl_wait(); }      // every ring of the cluster is drained
  const int per = MM_TILES / KS;
  const uint32_t in_s = smem_u32(in) + ((rank * per * 16 + g) * LD + 2 * t) * 4;
#pragma unroll
  for (int r = 0; r < MM_R; ++r) {
    const int tl = warp * MM_R + r;
    const uint32_t dst = cl_map(in_s, tl / per) + (tl % per) * 16 * LD * 4;
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      cl_store2(dst + m * 32, acc[r][m][0], acc[r][m][1]);
      cl_store2(dst + 8 * LD * 4 + m * 32, acc[r][m][2], acc[r][m][3]);
    }
  }
  cl_arrive();
  cl_wait();
  switch (KS) {
    case 1: mm_reduce<MT, 1>(p, epi, in, rank, nt0); break;
    case 2: mm_reduce<MT, 2>(p, epi, in, rank, nt0); break;
    case 4: mm_reduce<MT, 4>(p, epi, in, rank, nt0); break;
    default: mm_reduce<MT, 8>(p, epi, in, rank, nt0); break;
  }
}

template <int FMT, int MT, bool A8, int CT>
static int launch_mma(const MmaParams& p, int epi, int KS, int blocks, int pdl, cudaStream_t st) {
  auto kernel = w4_mma_kernel<FMT, MT, A8, CT>;
  constexpr int smem = mm_smem<FMT, MT, CT>();
  static SmemLimit limit;
  const int lrc = limit.raise(kernel, smem);
  if (lrc != OWL_OK) return lrc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(KS * blocks);
  cfg.blockDim = dim3(MM_WARPS * 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  int na = 0;
  attr[na].id = cudaLaunchAttributeClusterDimension;
  attr[na].val.clusterDim.x = KS; attr[na].val.clusterDim.y = 1; attr[na].val.clusterDim.z = 1;
  ++na;
  if (pdl) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, p, epi, KS);
  if (e != cudaSuccess) return (int)OWL_ERR_LAUNCH * 1000 - (int)e;
  return OWL_OK;
}

template <int FMT, bool A8>
static int dispatch_mma(MmaParams& p, int epi, int pdl, cudaStream_t st) {
  p.ab_blocks = (p.ab_rows + 15) / 16;
  const int row_blocks = (p.n_tiles + MM_TILES - 1) / MM_TILES;
  const int blocks = row_blocks + p.ab_blocks, sms = sm_count();
  // k parts: as many as one wave of four CTAs per SM holds, each of at least two record columns; independent of M. With one
  // column a part is all start-up and exchange (8192 x 1024, group 128, 1 / 8 / 32 rows: 8 parts 4.6 / 5.0 / 11.6 us, 4 parts 3.8 /
  // 4.0 / 8.1; a column more loses where it takes CTAs away: 1024 x 2048 2.8 -> 3.1).
  int KS = 8;
  while (KS > 1 && (row_blocks * KS > 4 * sms || 2 * KS > (p.K >> 7))) KS >>= 1;
  // Grids of up to three CTAs per SM run with three resident and a deeper ring: with four slots per SM the scheduler fills
  // some SMs with four CTAs and others with two (5120 x 17408, one row: 12.9 against 15.3 us). NVFP4 above 16 rows has registers
  // for three only.
  const bool three = KS * blocks <= 3 * sms;
  switch ((p.M + 7) / 8) {
    case 1: return three ? launch_mma<FMT, 1, A8, 3>(p, epi, KS, blocks, pdl, st) : launch_mma<FMT, 1, A8, 4>(p, epi, KS, blocks, pdl, st);
    case 2: return three ? launch_mma<FMT, 2, A8, 3>(p, epi, KS, blocks, pdl, st) : launch_mma<FMT, 2, A8, 4>(p, epi, KS, blocks, pdl, st);
    case 3: return three || FMT == MF_NV4 ? launch_mma<FMT, 3, A8, 3>(p, epi, KS, blocks, pdl, st) : launch_mma<FMT, 3, A8, FMT == MF_NV4 ? 3 : 4>(p, epi, KS, blocks, pdl, st);
    default: return three || FMT == MF_NV4 ? launch_mma<FMT, 4, A8, 3>(p, epi, KS, blocks, pdl, st) : launch_mma<FMT, 4, A8, FMT == MF_NV4 ? 3 : 4>(p, epi, KS, blocks, pdl, st);
  }
}

static bool mma_args_ok(const void* x, const void* out, const void* residual, const void* ab_w, const void* ab_x, const void* ab_out,
                        int ab_rows, int ab_ld, int M, int N, int K, int ldo, int epi) {
  if (M < 1 || M > 32 || N < 16 || (N & 15) || K < 128 || (K & 127) || epi < 0 || epi > MEPI_SILU_MUL || !x || !out || (ldo & 1) ||
      ab_rows < 0 || (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(out) & 3))
    return false;
  if (epi == MEPI_RESIDUAL && (!residual || (reinterpret_cast<uintptr_t>(residual) & 3))) return false;
  if (ab_rows > 0 && (!ab_w || !ab_x || !ab_out || ab_ld < ab_rows || (reinterpret_cast<uintptr_t>(ab_w) & 15) ||
                      (reinterpret_cast<uintptr_t>(ab_x) & 15)))
    return false;
  return true;
}

}  // namespace owl
using namespace owl;

// x / xs: activations packed with ACT_FRAG (and ACT_A8 when a8). epi: 0 store, 1 out = residual + y (same row stride), 2
// silu(gate) * up with gate / up rows interleaved in eights. ab_*: optional dense bf16 rows [ab_rows][K] times the plain bf16
// rows ab_x [M][K] -> ab_out [M][ab_ld].
OWL_API int owl_w4_mma(const void* records, const void* x, const void* xs, void* out, const void* residual, const void* ab_w,
                       const void* ab_x, void* ab_out, int ab_rows, int ab_ld, int M, int N, int K, int ldo, int group, int epi,
                       int a8, int pdl, cudaStream_t st) {
  if (!records || !xs || (group != 32 && group != 128) || (reinterpret_cast<uintptr_t>(records) & 15) ||
      (reinterpret_cast<uintptr_t>(xs) & 15) ||
      !mma_args_ok(x, out, residual, ab_w, ab_x, ab_out, ab_rows, ab_ld, M, N, K, ldo, epi))
    return OWL_ERR_BAD_ARG;
  MmaParams p = {};
  p.w = (const uint8_t*)records; p.x = (const uint4*)x; p.xs = (const float4*)xs; p.out = (__nv_bfloat16*)out;
  p.residual = (const __nv_bfloat16*)residual; p.ab_w = (const __nv_bfloat16*)ab_w; p.ab_x = (const __nv_bfloat16*)ab_x;
  p.ab_out = (__nv_bfloat16*)ab_out; p.ab_rows = ab_rows; p.ab_ld = ab_ld;
  p.out_scale = ACT_FRAG_UNIT; p.M = M; p.N = N; p.K = K; p.ldo = ldo; p.n_tiles = N / 16;
  if (group == 128) return a8 ? dispatch_mma<MF_G128, true>(p, epi, pdl, st) : dispatch_mma<MF_G128, false>(p, epi, pdl, st);
  return a8 ? dispatch_mma<MF_G32, true>(p, epi, pdl, st) : dispatch_mma<MF_G32, false>(p, epi, pdl, st);
}

// codes [N][K/2], sf [N][K/16], y = alpha * row_scale[n] * sum; x / xs: activations packed with ACT_FRAG | ACT_NV.
OWL_API int owl_nvfp4_mma(const void* codes, const void* sf, float alpha, const void* row_scale, const void* x, const void* xs, void* out,
                          const void* residual, const void* ab_w, const void* ab_x, void* ab_out, int ab_rows, int ab_ld, int M,
                          int N, int K, int ldo, int epi, int pdl, cudaStream_t st) {
  if (!codes || !sf || !xs || ((reinterpret_cast<uintptr_t>(codes) | reinterpret_cast<uintptr_t>(xs)) & 15) ||
      (reinterpret_cast<uintptr_t>(sf) & 7) ||
      !mma_args_ok(x, out, residual, ab_w, ab_x, ab_out, ab_rows, ab_ld, M, N, K, ldo, epi))
    return OWL_ERR_BAD_ARG;
  MmaParams p = {};
  p.w = (const uint8_t*)codes; p.sf = (const uint8_t*)sf; p.row_scale = (const float*)row_scale; p.x = (const uint4*)x;
  p.xs = (const float4*)xs; p.out = (__nv_bfloat16*)out; p.residual = (const __nv_bfloat16*)residual;
  p.ab_w = (const __nv_bfloat16*)ab_w; p.ab_x = (const __nv_bfloat16*)ab_x; p.ab_out = (__nv_bfloat16*)ab_out;
  p.ab_rows = ab_rows; p.ab_ld = ab_ld; p.out_scale = alpha; p.M = M; p.N = N; p.K = K; p.ldo = ldo; p.n_tiles = N / 16;
  return dispatch_mma<MF_NV4, false>(p, epi, pdl, st);
}
