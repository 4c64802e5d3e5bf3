// Weight-streaming projections for 1..32 rows (decode, verify) on tcgen05, the weights unpacked into tensor memory.
//
//   owl_w4_tm    : C[M,N] = X[M,K] . dequant(W4)[N,K]^T      int4 records, group 32 / 128 (slice-major, see gemv.cu)
//   owl_nvfp4_tm : C[M,N] = X[M,K] . dequant(NVFP4)[N,K]^T   codes and block scales as stored in the checkpoint
//   both with store / residual add / silu(gate) * up epilogues and, beside the matrix, a few dense bf16 rows (the GDN a / b
//   projections) computed by CTAs of the same grid
//
// The arithmetic is that of gemv_mma.cu: a masked nibble IS a bf16 subnormal (tcgen05 keeps them), the activations are bf16 times
// 2^64 (2^60 under the nibbles that carry a factor 16), each group's products are summed in fp32 and folded in as
//     y += s * (dot - z * sum(x));
// NVFP4 codes become fp16 times their block scale (exact), the activations fp16 with a power of two per 128.
//
// Why tensor memory: at 32 rows the warp-level MMAs of gemv_mma.cu alone take 256 clocks a record and sub-core (a record's share of
// HBM is 185), and each needs its fragments through registers. Here a row of the block is a thread: it reads its 64 bytes of a
// record column, masks them (5 instructions a word of eight) and stores them to tensor memory as the A operand, tcgen05.mma takes
// the tokens from shared memory (N = 16 or 32: 11 / 17 clocks an instruction, issued by a whole warp with an elected lane), and the
// sums of each group come back to the thread of the row, which holds its scale.
//
// Measured (one B200, graph of dependent launches over rotating weights; HBM time; 1 / 32 rows here, 1 / 32 rows in gemv_mma.cu), us:
//   group 128 16384 x 5120  6.8: 17.2 / 20.9, 11.2 / 26.2    34816 x 5120 14.5: 30.2 / 37.4, 19.9 / 45.4
//             5120 x 6144   2.6: 10.6 / 12.3,  6.8 / 13.7    5120 x 17408  7.2: 20.2 / 23.1, 13.2 / 28.7
//   group 32  16384 x 5120  8.0: 22.9 / 30.2, 13.5 / 33.5    NVFP4 16384 x 5120 7.2: 18.6 / 22.0, 17.4 / 33.7
// What bounds it: a step takes about 550 clocks (group 32 with two reader sets 950: they read four groups' sums back), of which HBM
// would need 370. No pipe is full; each hand-over (unpack -> MMA -> read back -> unpack) costs 100 to 250 clocks of barrier latency,
// the unpacking warps that share a scheduler with the issuing one lag, and three sets of unpacking warps are slower than two
// (16384 x 5120, one row: 19.1 us). Up to 24 rows gemv_mma.cu is the faster form.
//
// Roles of a CTA (one per SM, walking units of 128 rows x a part of k; a step is a record column, 128 k):
//   warp 0       activations of a step: bulk copies of the fragment blocks (8 tokens x 128 k, the 64-byte swizzle of the MMA's B
//                operand) and their sums
//   warp 1       8 MMAs a step, into the accumulators of one (group 128, NVFP4) or four (group 32) groups, two steps deep
//   warps 2-9    two sets of four: set s unpacks steps s, s + 2, ... into one of four stages of tensor memory, each warp 32 rows, from a ring of
//                its own that cp.async fills; the weights do not depend on the kernel before, so the rings fill before the wait
//   warps 10-17  read a step's sums back (a warp: 32 rows x 16 tokens) and keep y in registers
// The k parts of a row block form a cluster and push their partial sums to the part that owns the rows; KS depends on N, K,
// the number of dense rows beside the matrix and the device's SMs, not on M: a row computes the same bits in every step that takes this form.
//
// Every mbarrier wait is bounded; on a timeout the CTA records an error code, the roles leave their loops, copies in flight are
// waited for and TMEM is freed.
//
// Role in the reference: the Marlin W4A16 decode path and the NVFP4 GEMV (crates/kernels/cu/marlin/*,
// crates/kernels/cu/nvfp4/nvfp4_gemv.cu).
#include <cuda_fp8.h>
#include "common.cuh"
#include "actpack.cuh"

namespace owl {

__device__ int g_gemv_tm_status = 0;

enum { TF_G128 = 0, TF_G32 = 1, TF_NV4 = 2 };
enum { TEPI_STORE = 0, TEPI_RESIDUAL = 1, TEPI_SILU_MUL = 2 };
constexpr int TM_SETS = 2, TM_AS = 4, TM_DEQ = 4 * TM_SETS, TM_RB = 8, TM_FIRST_RB = 2 + TM_DEQ, TM_THREADS = (2 + TM_DEQ + TM_RB) * 32;
constexpr int TM_XPOOL = 48 * 1024, TM_XMAX = 16;            // shared memory of the activations' ring, and its longest
constexpr int TM_A_COLS = 64, TM_ACC = TM_AS * TM_A_COLS;    // tensor memory: stages of weights, then the accumulators
constexpr int TM_LD = 36;                                    // floats of a row of partial sums
constexpr int TM_IN = 3 * 48 * TM_LD * 4;                    // partial sums of the rows a CTA owns, from every part
template <int F> __host__ __device__ constexpr int tm_gpr() { return F == TF_G32 ? 4 : 1; }
template <int F> __host__ __device__ constexpr int tm_rec() { return F == TF_G128 ? 1088 : F == TF_G32 ? 1280 : 1152; }
template <int F> __host__ __device__ constexpr int tm_raw() { return F == TF_G32 ? 6 : 8; }      // ring slots (two tiles each) of a warp
// Steps of accumulators: at most TM_AS, since a reader that lags further would take the parity of a later round of `done` for its own.
template <int F> __host__ __device__ constexpr int tm_slots() { return F == TF_G32 ? 2 : 4; }
// Steps whose weight scales are kept: a set that writes those of step `it` has seen the MMAs of step it - TM_AS done, which had waited for
// the readers of step it - TM_AS - slots.
template <int F> __host__ __device__ constexpr int tm_info() { return 8; }
struct TmCtl {
  // full_a / full_x: a step's weights (an arrival per warp of the set) and activations are here; done: its sums are there (the MMAs'
  // commit, and an arrival that passes on what full_a and full_x showed); acc_free / empty_x: the readers have the sums, and are
  // through with the step's activations
  uint64_t full_a[TM_AS], done[TM_AS], full_x[TM_XMAX], empty_x[TM_XMAX], acc_free[4];
  uint32_t tmem_base;
  volatile int abort_flag;
};
// Activations, their sums, weight scales, weights, partial sums; the control block lies behind them.
template <int F> __host__ __device__ constexpr int tm_ctl_off() {
  return TM_XPOOL + TM_XPOOL / 2048 * tm_gpr<F>() * 64 + tm_info<F>() * tm_gpr<F>() * 512 + TM_DEQ * tm_raw<F>() * 2 * tm_rec<F>() + TM_IN;
}
static_assert(tm_ctl_off<TF_G128>() % 8 == 0 && tm_ctl_off<TF_G32>() % 8 == 0 && tm_ctl_off<TF_NV4>() % 8 == 0, "mbarriers");
// 1024 bytes let the base be rounded up to the swizzle's boundary, from wherever dynamic shared memory begins.
template <int F> constexpr int tm_smem() { return tm_ctl_off<F>() + (int)sizeof(TmCtl) + 1024; }

struct TmParams {
  const uint8_t* w;               // int4: record stream; NVFP4: codes [N][K/2]
  const uint8_t* sf;              // NVFP4: e4m3 block scales [N][K/16]
  const float* row_scale;         // NVFP4, optional: fp32 [N]
  const uint8_t* x;               // ACT_TM blocks
  const uint8_t* xs;              // ACT_TM scales and sums
  __nv_bfloat16* out;
  const __nv_bfloat16* residual;
  const __nv_bfloat16* ab_w;      // optional dense rows [ab_rows][K] ...
  const __nv_bfloat16* ab_x;      // ... times plain bf16 rows [M][K]
  __nv_bfloat16* ab_out;          // [M][ab_ld]
  float out_scale;
  int M, N, K, ldo, n_tiles, row_blocks, ab_rows, ab_ld, ab_blocks, epi;
};
__device__ __forceinline__ bool tm_wait(uint64_t* bar, uint32_t parity, TmCtl* c, int code) {
  return mbar_wait_bounded(bar, parity, &c->abort_flag, &g_gemv_tm_status, code);
}
__device__ __forceinline__ bool tm_wait_warp(uint64_t* bar, uint32_t parity, TmCtl* c, int code) {
  return mbar_wait_warp<true>(bar, parity, &c->abort_flag, &g_gemv_tm_status, code);
}
__device__ __forceinline__ void tm_cp16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void tm_cp16_ahead(uint32_t dst, const void* src) {       // rows of which a step takes 64 bytes
  asm volatile("cp.async.cg.shared.global.L2::256B [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
// By a whole warp: an elected lane issues (one lane by itself took 150 clocks a copy)
__device__ __forceinline__ void tm_bulk_warp(uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
               "@q cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n\t}"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
// A load that stays where it is written, before the arrival that gives its slot back (see the readers).
__device__ __forceinline__ float4 tm_ld4(uint32_t addr) {
  float4 v;
  asm volatile("ld.volatile.shared::cta.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void tm_cl_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void tm_cl_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void tm_push4(uint32_t addr, int rank, float a, float b, float c, float d) {
  asm volatile("{\n\t.reg .b32 r;\n\tmapa.shared::cluster.u32 r, %0, %1;\n\tst.shared::cluster.v4.f32 [r], {%2, %3, %4, %5};\n\t}"
               ::"r"(addr), "r"(rank), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
// (a, b) = (a, b) * (s, s) + (c, d), both halves in one instruction
__device__ __forceinline__ void tm_fma2(float& d0, float& d1, float a0, float a1, float b0, float b1, float c0, float c1) {
  asm("{\n\t.reg .b64 a, b, c, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
      "fma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(d0), "=f"(d1) : "f"(a0), "f"(a1), "f"(b0), "f"(b1), "f"(c0), "f"(c1));
}
__device__ __forceinline__ void tm_mma_bf16(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// eight e2m1 codes -> four fp16 pairs
__device__ __forceinline__ void tm_e2m1x8(uint32_t q, uint32_t* d) {
  asm("{\n\t.reg .b8 a, b, c, d;\n\tmov.b32 {a, b, c, d}, %4;\n\tcvt.rn.f16x2.e2m1x2 %0, a;\n\tcvt.rn.f16x2.e2m1x2 %1, b;\n\t"
      "cvt.rn.f16x2.e2m1x2 %2, c;\n\tcvt.rn.f16x2.e2m1x2 %3, d;\n\t}"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(q));
}
__device__ __forceinline__ uint32_t tm_mul2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ void tm_st16(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                 "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
// The B operand of a fragment block: 8 tokens x 32 k as rows of 64 bytes with the 64-byte swizzle, blocks of 8 tokens 2048 bytes apart.
__device__ __forceinline__ uint64_t tm_desc(uint32_t smem_addr) {
  return (uint64_t)((smem_addr & 0x3ffffu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(2048 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)4 << 61);
}

// Dense bf16 rows, 16 by one CTA: the unpacking warps split k.
__device__ __noinline__ void tm_dense_block(const TmParams& p, float* red, int blk) {
  constexpr int LD = 34;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int nc = p.K / 32;                            // 32-k steps: 8 k per lane quarter
  if (warp < TM_DEQ) {
    const int c0 = warp * nc / TM_DEQ, c1 = (warp + 1) * nc / TM_DEQ;
    const int r0 = min(blk * 16 + g, p.ab_rows - 1), r1 = min(blk * 16 + g + 8, p.ab_rows - 1);
    const uint4* w0 = reinterpret_cast<const uint4*>(p.ab_w + (size_t)r0 * p.K) + t;
    const uint4* w1 = reinterpret_cast<const uint4*>(p.ab_w + (size_t)r1 * p.K) + t;
    float acc[4][4];
    const uint4* xr[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      acc[m][0] = acc[m][1] = acc[m][2] = acc[m][3] = 0.f;
      xr[m] = reinterpret_cast<const uint4*>(p.ab_x + (size_t)min(m * 8 + g, p.M - 1) * p.K) + t;
    }
#pragma unroll 2
    for (int c = c0; c < c1; ++c) {
      const uint4 a = w0[c * 4], b = w1[c * 4];
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        if (m * 8 >= p.M) break;
        const uint4 xv = xr[m][c * 4];
        tm_mma_bf16(acc[m], a.x, b.x, a.y, b.y, xv.x, xv.y);
        tm_mma_bf16(acc[m], a.z, b.z, a.w, b.w, xv.z, xv.w);
      }
    }
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      float* r = red + (warp * 16 + g) * LD + m * 8 + 2 * t;
      *reinterpret_cast<float2*>(r) = make_float2(acc[m][0], acc[m][1]);
      *reinterpret_cast<float2*>(r + 8 * LD) = make_float2(acc[m][2], acc[m][3]);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < p.M * 16; i += TM_THREADS) {
    const int row = i & 15, tok = i >> 4;
    if (blk * 16 + row >= p.ab_rows) continue;
    float a = 0.f;
#pragma unroll
    for (int s = 0; s < TM_DEQ; ++s) a += red[(s * 16 + row) * LD + tok];
    p.ab_out[(size_t)tok * p.ab_ld + blk * 16 + row] = __float2bfloat16(a);
  }
}

// grid: KS * (row blocks walked side by side + ab_blocks), cluster KS; the last ab_blocks clusters take the dense rows. A8: the
// activations are 8-bit integers with a scale per (token, group).
template <int F, bool A8>
__global__ void __launch_bounds__(TM_THREADS, 1) w4_tm_kernel(TmParams p, int KS) {
  constexpr int REC = tm_rec<F>(), GPR = tm_gpr<F>(), RAW = tm_raw<F>(), SLOTS = tm_slots<F>(), INFO = tm_info<F>();
  static_assert(SLOTS <= TM_AS && INFO >= TM_AS + SLOTS, "scales are read after the step's accumulators were given back");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* raw_all = base + TM_XPOOL;
  uint8_t* side_all = raw_all + TM_DEQ * RAW * 2 * REC;                // (scale, zero) [step % INFO][group][128 rows]
  uint8_t* sums_all = side_all + INFO * GPR * 512;                  // [stage][block of 8 tokens][group][8 scales, 8 sums]
  float* in = reinterpret_cast<float*>(sums_all + TM_XPOOL / 2048 * GPR * 64);
  TmCtl* ctl = reinterpret_cast<TmCtl*>(base + tm_ctl_off<F>());
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int KT = p.K >> 7;
  const int rank = blockIdx.x % KS, cl = blockIdx.x / KS, n_cl = gridDim.x / KS - p.ab_blocks;
  if (cl >= n_cl) {
    if (rank == 0) {
      pdl_launch_dependents();
      pdl_wait();
      tm_dense_block(p, reinterpret_cast<float*>(smem_raw), cl - n_cl);
    }
    return;
  }
  const int kb = rank * KT / KS, ke = (rank + 1) * KT / KS, len = ke - kb;
  const int units = (p.row_blocks - cl + n_cl - 1) / n_cl, total = units * len;
  const int MT = (p.M + 7) >> 3, rb_sets = p.M > 16 ? 2 : 1;
  const int xbytes = MT * 2048, sbytes = MT * GPR * 64, SX = min(TM_XMAX, TM_XPOOL / xbytes);

  if (threadIdx.x == 0) {
    for (int s = 0; s < TM_AS; ++s) { mbar_init(&ctl->full_a[s], 4); mbar_init(&ctl->done[s], 2); }
    for (int s = 0; s < TM_XMAX; ++s) { mbar_init(&ctl->full_x[s], 1); mbar_init(&ctl->empty_x[s], 4 * rb_sets); }
    for (int a = 0; a < SLOTS; ++a) mbar_init(&ctl->acc_free[a], 4 * rb_sets);
    ctl->abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(&ctl->tmem_base, 512);
    tmem_relinquish();
  }
  if (KS > 1) tm_cl_arrive();           // the peers run before anything is stored in their shared memory
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, ctl->tmem_base, 0);
  const bool reader = warp >= TM_FIRST_RB;
  const int q4 = warp & 3, h = (warp - TM_FIRST_RB) >> 2;      // readers: TMEM lane quarter, half of the tokens
  const int RM = (8 + KS - 1) / KS * 16;                       // rows of a part's block in `in`

  // the rows this CTA owns: their sum in part order to memory, by n threads
  auto emit = [&](int rb, int i0, int n) {
    const int t0 = rank * 8 / KS, nt = (rank + 1) * 8 / KS - t0, M = p.M;
#pragma unroll 1
    for (int i = i0; i < nt * M * 8; i += n) {
      const int rp = i & 7, tok = (i >> 3) % M, tl = (i >> 3) / M, tile = rb * 8 + t0 + tl;
      if (tile >= p.n_tiles) continue;
      const int ra = p.epi == TEPI_SILU_MUL ? rp : 2 * rp, rc = p.epi == TEPI_SILU_MUL ? rp + 8 : 2 * rp + 1;
      float a = 0.f, b = 0.f;
#pragma unroll 1
      for (int q = 0; q < KS; ++q) {
        a += in[((size_t)q * RM + tl * 16 + ra) * TM_LD + tok];
        b += in[((size_t)q * RM + tl * 16 + rc) * TM_LD + tok];
      }
      float sa = p.out_scale, sb = sa;
      if (p.row_scale) { sa *= p.row_scale[tile * 16 + ra]; sb *= p.row_scale[tile * 16 + rc]; }
      a *= sa; b *= sb;
      if (p.epi == TEPI_SILU_MUL) {
        p.out[(size_t)tok * p.ldo + tile * 8 + rp] = __float2bfloat16(silu_f(a) * b);
      } else {
        const size_t o = (size_t)tok * p.ldo + tile * 16 + 2 * rp;
        if (p.epi == TEPI_RESIDUAL) {
          const uint32_t rr = *reinterpret_cast<const uint32_t*>(p.residual + o);
          a += bf16_lo(rr); b += bf16_hi(rr);
        }
        *reinterpret_cast<uint32_t*>(p.out + o) = pack_bf16(a, b);
      }
    }
  };

  if (warp == 0) {
    pdl_launch_dependents();
    pdl_wait();                          // the kernel before writes the activations
    const uint32_t xb = smem_u32(base), sb = smem_u32(sums_all);
    int it = 0, s = 0;
    uint32_t ph = 1;
    bool ok = true;
    for (int u = 0; u < units && ok; ++u)
      for (int k = kb; k < ke; ++k, ++it) {
        ok = __all_sync(0xffffffffu, tm_wait(&ctl->empty_x[s], ph, ctl, OWL_ERR_WAIT_EPI));
        if (!ok) break;
        if (lane == 0) mbar_expect_tx(&ctl->full_x[s], xbytes + sbytes);
        __syncwarp();
        tm_bulk_warp(xb + s * xbytes, p.x + (size_t)k * xbytes, xbytes, &ctl->full_x[s]);
        tm_bulk_warp(sb + s * sbytes, p.xs + (size_t)k * sbytes, sbytes, &ctl->full_x[s]);
        if (++s == SX) { s = 0; ph ^= 1; }
      }
    if (lane == 0 && ctl->abort_flag) {
      for (int i = max(0, it - SX); i < it; ++i)      // copies in flight: a bounded wait for each
        for (uint32_t n = 0; n < 256u; ++n)
          if (mbar_try_wait(&ctl->full_x[i % SX], ((uint32_t)(i / SX)) & 1u)) break;
    }
    __syncwarp();
  } else if (warp == 1) {
    const uint32_t idesc = umma_idesc_f16(128, (p.M + 15) & ~15, F == TF_NV4 ? 0 : 1), xb = smem_u32(base);
    // free, x, a: this step's barriers, looked at before the last step's MMAs were issued
    uint32_t free = 0, x = 0, a = 0, phx = 0;
    int s = 0;
    for (int it = 0; it < total; ++it) {
      const int slot = it & (SLOTS - 1), as = it & (TM_AS - 1), n = it + 1;
      if (!__all_sync(0xffffffffu, free & x & a)) {
        if (!__all_sync(0xffffffffu, x) && !tm_wait_warp(&ctl->full_x[s], phx, ctl, OWL_ERR_WAIT_TMA)) break;
        if (!__all_sync(0xffffffffu, a) && !tm_wait_warp(&ctl->full_a[as], ((uint32_t)(it / TM_AS)) & 1u, ctl, OWL_ERR_WAIT_EPI)) break;
        if (!__all_sync(0xffffffffu, free) && !tm_wait_warp(&ctl->acc_free[slot], (((uint32_t)(it / SLOTS)) & 1u) ^ 1u, ctl, OWL_ERR_WAIT_EPI)) break;
      }
      tc_fence_after();
      uint64_t* done = &ctl->done[as];
      if (lane == 0) mbar_arrive(done);
      __syncwarp();
      const uint64_t db = tm_desc(xb + s * xbytes);
      const uint32_t ta = tmem + as * TM_A_COLS, d = tmem + TM_ACC + slot * (GPR * 32);
      if (++s == SX) { s = 0; phx ^= 1; }
      x = mbar_test(&ctl->full_x[s], phx);
      a = mbar_test(&ctl->full_a[n & (TM_AS - 1)], ((uint32_t)(n / TM_AS)) & 1u);
      free = mbar_test(&ctl->acc_free[n & (SLOTS - 1)], (((uint32_t)(n / SLOTS)) & 1u) ^ 1u);
#pragma unroll
      for (int i = 0; i < 8; ++i)        // word i / 2 of the record column, half i % 2 of its 32 k
        tc_mma_f16_ts_warp(d + (GPR == 4 ? (i >> 1) * 32 : 0), ta + i * 8, db + (uint64_t)((i >> 1) * 32 + (i & 1) * 2), idesc,
                           (GPR == 4 ? (i & 1) : i) ? 1u : 0u);
      tc_commit_warp(done);
    }
  } else if (!reader) {
    // this warp: rows 32 q .. 32 q + 31 of the row block (two tiles), every second step
    const int set = (warp - 2) >> 2;
    uint8_t* raw = raw_all + (warp - 2) * RAW * 2 * REC;
    // Fetch cursor: unit, record column, k slice (slice-major streams, see gemv.cu). A lane brings chunk t of row g: it is put
    // down at place (t + g / 2) % 4 of the row, so that eight rows' chunks t, which eight lanes read together, lie in eight banks.
    int fu = 0, fk = kb + set, sl = 0, k0 = 0, k1 = KT >> 3, ta = 0, tb = 0;
    const int cg = lane >> 2;
    const uint32_t raw_s = smem_u32(raw) + cg * 64 + ((((lane & 3) + (cg >> 1)) & 3) << 4);
    auto open_unit = [&]() {
      const int rb = cl + fu * n_cl;
      sl = k0 = 0; k1 = KT >> 3;
      ta = min(rb * 8 + q4 * 2, p.n_tiles - 1);
      tb = min(rb * 8 + q4 * 2 + 1, p.n_tiles - 1);
    };
    auto fetch = [&](int slot) {
      while (fk >= ke && fu < units) {     // past the unit's end: on to the one that holds the column
        fk -= len;
        if (++fu < units) open_unit();
      }
      if (fu < units) {
        const uint32_t d = raw_s + slot * 2 * REC;
        if (F == TF_NV4) {
          // rows of 64 code bytes (cg, cg + 8 of both tiles), then 8 scale bytes of each of the 32 rows
          const uint8_t* src = p.w + (size_t)(ta * 16 + cg) * (p.K >> 1) + (size_t)fk * 64 + (lane & 3) * 16;
          const uint8_t* src1 = src + (size_t)(tb - ta) * 8 * p.K;
          tm_cp16_ahead(d, src);
          tm_cp16_ahead(d + 512, src + (size_t)4 * p.K);
          tm_cp16_ahead(d + 1024, src1);
          tm_cp16_ahead(d + 1536, src1 + (size_t)4 * p.K);
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(raw) + slot * 2 * REC + 2048 + lane * 8),
                       "l"(p.sf + (size_t)((lane < 16 ? ta : tb) * 16 + (lane & 15)) * (p.K >> 4) + (size_t)fk * 8) : "memory");
        } else {
          while (k1 <= fk) { ++sl; k0 = k1; k1 = ((sl + 1) * KT) >> 3; }
          const int rpi = k1 - k0;
          const uint8_t* src = p.w + (size_t)(uint32_t)(p.n_tiles * k0 + ta * rpi + fk - k0) * REC;
          const uint8_t* src1 = src + (uint32_t)((tb - ta) * rpi) * (uint32_t)REC;
          tm_cp16(d, src + lane * 16);
          tm_cp16(d + 512, src + lane * 16 + 512);
          tm_cp16(d + 1024, src1 + lane * 16);
          tm_cp16(d + 1536, src1 + lane * 16 + 512);
          // the (scale, zero) pairs of both tiles behind the codes: [tile][group][16 rows]
          const uint32_t z = smem_u32(raw) + slot * 2 * REC + 2048 + lane * 16;
          if (GPR == 4) tm_cp16(z, (lane < 16 ? src : src1) + 1024 + (lane & 15) * 16);
          else if (lane < 8) tm_cp16(z, (lane < 4 ? src : src1) + 1024 + (lane & 3) * 16);
        }
        fk += TM_SETS;
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    open_unit();
#pragma unroll
    for (int i = 0; i < RAW - 1; ++i) fetch(i);
    pdl_launch_dependents();
    const int g = lane & 7;
    const uint32_t at0 = tmem + ((uint32_t)(q4 * 32) << 16);
    const uint8_t* row_q = raw + lane * 64;
    const uint8_t* row_z = raw + 2048 + (lane >> 4) * (GPR * 64) + (lane & 15) * 4;
    uint8_t* side = side_all + (q4 * 32 + lane) * 4;
    int slot = 0;
    for (int it = set; it < total; it += TM_SETS) {
      const int as = it & (TM_AS - 1);       // (stages of one parity: they belong to this set, which has seen each one's last step done)
      const uint32_t at = at0 + as * TM_A_COLS;
      asm volatile("cp.async.wait_group %0;" ::"n"(RAW - 2) : "memory");
      __syncwarp();                        // the column is here for all lanes, and all lanes left the slot refilled now
      fetch(slot == 0 ? RAW - 1 : slot - 1);
      uint4 v[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) v[t] = *reinterpret_cast<const uint4*>(row_q + slot * 2 * REC + (((t + (g >> 1)) & 3) << 4));
      uint2 e8 = make_uint2(0, 0);
      uint32_t sz[GPR];
      if (F == TF_NV4) e8 = *reinterpret_cast<const uint2*>(raw + slot * 2 * REC + 2048 + lane * 8);
      else {
#pragma unroll
        for (int q = 0; q < GPR; ++q) sz[q] = *reinterpret_cast<const uint32_t*>(row_z + slot * 2 * REC + q * 64);
      }
      slot = slot + 1 == RAW ? 0 : slot + 1;
      const bool ok = __all_sync(0xffffffffu, tm_wait(&ctl->done[as], (((uint32_t)(it / TM_AS)) & 1u) ^ 1u, ctl, OWL_ERR_WAIT_MMA));
      if (!ok) break;                      // (the lanes leave together)
      tc_fence_after();
      if (F != TF_NV4) {
        // (see tm_info)
#pragma unroll
        for (int q = 0; q < GPR; ++q) *reinterpret_cast<uint32_t*>(side + ((it & (INFO - 1)) * GPR + q) * 512) = sz[q];
      }
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        uint32_t o[16];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const uint32_t q = w == 0 ? v[t].x : w == 1 ? v[t].y : w == 2 ? v[t].z : v[t].w;
          if (F == TF_NV4) {
            // word w of chunk t: codes 32 t + 8 w.., block scale 2 t + w / 2
            const uint16_t b2 = (uint16_t)((t < 2 ? e8.x : e8.y) >> ((t & 1) * 16));
            const __half2 s2 = __half2(__nv_cvt_fp8x2_to_halfraw2(b2, __NV_E4M3));
            const __half2 s = w < 2 ? __low2half2(s2) : __high2half2(s2);
            uint32_t d[4];
            tm_e2m1x8(q, d);
#pragma unroll
            for (int i = 0; i < 4; ++i) o[t * 4 + i] = tm_mul2(d[i], *reinterpret_cast<const uint32_t*>(&s));
          } else {
            const uint32_t q8 = q >> 8;
            o[t * 4] = q & 0x000f000fu;
            o[t * 4 + 1] = q & 0x00f000f0u;
            o[t * 4 + 2] = q8 & 0x000f000fu;
            o[t * 4 + 3] = q8 & 0x00f000f0u;
          }
        }
        tm_st16(at + w * 16, o);
      }
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl->full_a[as]);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (h < rb_sets) {
    pdl_wait();                            // residual and output rows belong to the kernels before until here
    float y[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) y[i] = 0.f;
    const int r = q4 * 32 + lane, own = (((r >> 4) + 1) * KS - 1) >> 3;      // this lane's row of the block, and the part that owns it
    float* dst = in + ((size_t)rank * RM + ((r >> 4) - own * 8 / KS) * 16 + (r & 15)) * TM_LD + h * 16;
    int it = 0, sx = 0;
    const uint32_t sums_s = smem_u32(sums_all);
    bool ok = true;
    for (int u = 0; u < units; ++u) {
      for (int k = 0; k < len && ok; ++k, ++it) {
        const int slot = it & (SLOTS - 1), e = it & (INFO - 1);
        ok = __all_sync(0xffffffffu, tm_wait(&ctl->done[it & (TM_AS - 1)], ((uint32_t)(it / TM_AS)) & 1u, ctl, OWL_ERR_WAIT_MMA));
        if (!ok) break;
        tc_fence_after();
        // The slot of the step before goes back now, not at that step's end: a copy writes into it once all readers have arrived, and
        // nothing orders loads whose values have not been used yet before a copy (given back at the end of its step, a warp that was held
        // up there found the sums of six steps later in its last loads). The values of the step before have been used by now.
        if (it > 0) {
          __syncwarp();
          if (lane == 0) mbar_arrive(&ctl->empty_x[sx == 0 ? SX - 1 : sx - 1]);
        }
        const uint32_t a = tmem + ((uint32_t)(q4 * 32) << 16) + TM_ACC + slot * (GPR * 32) + h * 16;
        const uint32_t sums = sums_s + sx * sbytes + 2 * h * (GPR * 64);
        const uint8_t* side = side_all + e * GPR * 512 + r * 4;
        constexpr int GB = GPR == 4 ? 2 : 1;         // groups whose sums are fetched together
#pragma unroll
        for (int q0 = 0; q0 < GPR; q0 += GB) {
          uint32_t d[GB][16];
#pragma unroll
          for (int i = 0; i < GB; ++i) tmem_ld_32x32b_x16(a + (q0 + i) * 32, d[i]);
          float s[GB], nz[GB];
          float4 xs[GB][4];                // sums (NVFP4: scales) of the tokens: block i / 2 of 8 scales and 8 sums
#pragma unroll
          for (int i = 0; i < GB; ++i) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
              xs[i][j] = tm_ld4(sums + (j >> 1) * (GPR * 64) + (q0 + i) * 64 + ((j & 1) + (F == TF_NV4 ? 0 : 2)) * 16);
            const __half2 z = F == TF_NV4 ? __half2() : *reinterpret_cast<const __half2*>(side + (q0 + i) * 512);
            s[i] = __low2float(z);
            nz[i] = -__high2float(z);
          }
          tc_wait_ld();
          if (q0 + GB == GPR) {            // the accumulators are free for the step after the next
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&ctl->acc_free[slot]);
          }
#pragma unroll
          for (int g = 0; g < GB; ++g)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int j = i * 4;
              float d0 = __uint_as_float(d[g][j]), d1 = __uint_as_float(d[g][j + 1]), d2 = __uint_as_float(d[g][j + 2]), d3 = __uint_as_float(d[g][j + 3]);
              if (F == TF_NV4) {
                const float4 x = xs[g][i];
                tm_fma2(y[j], y[j + 1], d0, d1, x.x, x.y, y[j], y[j + 1]);
                tm_fma2(y[j + 2], y[j + 3], d2, d3, x.z, x.w, y[j + 2], y[j + 3]);
              } else {
                if (A8) {
                  const float4 x8 = tm_ld4(sums + (i >> 1) * (GPR * 64) + (q0 + g) * 64 + (i & 1) * 16);
                  d0 *= x8.x; d1 *= x8.y; d2 *= x8.z; d3 *= x8.w;
                }
                const float4 x = xs[g][i];
                tm_fma2(d0, d1, nz[g], nz[g], x.x, x.y, d0, d1);
                tm_fma2(d2, d3, nz[g], nz[g], x.z, x.w, d2, d3);
                tm_fma2(y[j], y[j + 1], s[g], s[g], d0, d1, y[j], y[j + 1]);
                tm_fma2(y[j + 2], y[j + 3], s[g], s[g], d2, d3, y[j + 2], y[j + 3]);
              }
            }
        }
        sx = sx + 1 == SX ? 0 : sx + 1;
      }
      if (KS > 1) {                        // (one unit)
        tm_cl_wait();
#pragma unroll
        for (int i = 0; i < 4; ++i) tm_push4(smem_u32(dst + i * 4), own, y[i * 4], y[i * 4 + 1], y[i * 4 + 2], y[i * 4 + 3]);
      } else {
        const int n = rb_sets * 128;
#pragma unroll
        for (int i = 0; i < 4; ++i) *reinterpret_cast<float4*>(dst + i * 4) = make_float4(y[i * 4], y[i * 4 + 1], y[i * 4 + 2], y[i * 4 + 3]);
#pragma unroll
        for (int i = 0; i < 16; ++i) y[i] = 0.f;
        asm volatile("bar.sync 1, %0;" ::"r"(n) : "memory");
        emit(cl + u * n_cl, threadIdx.x - TM_FIRST_RB * 32, n);
        if (u + 1 < units) asm volatile("bar.sync 1, %0;" ::"r"(n) : "memory");
      }
    }
  }
  if (KS > 1) {
    __syncwarp();
    if (!reader || h >= rb_sets) tm_cl_wait();
    tm_cl_arrive();                        // every part's sums have been pushed
    tm_cl_wait();
    emit(cl, threadIdx.x, TM_THREADS);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

template <int F, bool A8>
static int launch_tm(TmParams& p, int pdl, cudaStream_t st) {
  auto kernel = w4_tm_kernel<F, A8>;
  constexpr int smem = tm_smem<F>();
  static_assert(smem <= 227 * 1024, "shared memory");
  static SmemLimit limit;
  const int lrc = limit.raise(kernel, smem);
  if (lrc != OWL_OK) return lrc;
  p.n_tiles = p.N / 16;
  p.row_blocks = (p.n_tiles + 7) / 8;
  p.ab_blocks = (p.ab_rows + 15) / 16;
  // k parts: as many as the SMs hold beside each other, of at least two record columns each; independent of M
  const int sms = sm_count();
  int KS = 1;
  for (int ks : {2, 3, 4, 8})
    if ((p.row_blocks + p.ab_blocks) * ks <= sms && 2 * ks <= (p.K >> 7)) KS = ks;
  const int room = sms - p.ab_blocks, n_cl = KS > 1 || p.row_blocks < room ? p.row_blocks : room < 1 ? 1 : room;      // KS > 1: one unit a CTA
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(KS * (n_cl + p.ab_blocks));
  cfg.blockDim = dim3(TM_THREADS);
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
  cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, p, KS);
  if (e != cudaSuccess) return (int)OWL_ERR_LAUNCH * 1000 - (int)e;
  return OWL_OK;
}

static bool tm_args_ok(const void* x, const void* xs, const void* out, const void* residual, const void* ab_w, const void* ab_x,
                       const void* ab_out, int ab_rows, int ab_ld, int M, int N, int K, int ldo, int epi) {
  if (M < 1 || M > 32 || N < 16 || (N & 15) || K < 128 || (K & 127) || epi < 0 || epi > TEPI_SILU_MUL || !x || !xs || !out || (ldo & 1) ||
      ab_rows < 0 || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(xs)) & 15) || (reinterpret_cast<uintptr_t>(out) & 3))
    return false;
  if (epi == TEPI_RESIDUAL && (!residual || (reinterpret_cast<uintptr_t>(residual) & 3))) return false;
  if (ab_rows > 0 && (!ab_w || !ab_x || !ab_out || ab_ld < ab_rows || (reinterpret_cast<uintptr_t>(ab_w) & 15) ||
                      (reinterpret_cast<uintptr_t>(ab_x) & 15)))
    return false;
  return true;
}

}  // namespace owl
using namespace owl;

// Arguments as owl_w4_mma / owl_nvfp4_mma (gemv_mma.cu), the activations packed with ACT_TM for the same M.
OWL_API int owl_w4_tm(const void* records, const void* x, const void* xs, void* out, const void* residual, const void* ab_w,
                      const void* ab_x, void* ab_out, int ab_rows, int ab_ld, int M, int N, int K, int ldo, int group, int epi,
                      int a8, int pdl, cudaStream_t st) {
  if (!records || (group != 32 && group != 128) || (reinterpret_cast<uintptr_t>(records) & 15) ||
      !tm_args_ok(x, xs, out, residual, ab_w, ab_x, ab_out, ab_rows, ab_ld, M, N, K, ldo, epi))
    return OWL_ERR_BAD_ARG;
  TmParams p = {};
  p.w = (const uint8_t*)records; p.x = (const uint8_t*)x; p.xs = (const uint8_t*)xs; p.out = (__nv_bfloat16*)out;
  p.residual = (const __nv_bfloat16*)residual; p.ab_w = (const __nv_bfloat16*)ab_w; p.ab_x = (const __nv_bfloat16*)ab_x;
  p.ab_out = (__nv_bfloat16*)ab_out; p.ab_rows = ab_rows; p.ab_ld = ab_ld;
  p.out_scale = ACT_FRAG_UNIT; p.M = M; p.N = N; p.K = K; p.ldo = ldo; p.epi = epi;
  if (group == 128) return a8 ? launch_tm<TF_G128, true>(p, pdl, st) : launch_tm<TF_G128, false>(p, pdl, st);
  return a8 ? launch_tm<TF_G32, true>(p, pdl, st) : launch_tm<TF_G32, false>(p, pdl, st);
}

OWL_API int owl_nvfp4_tm(const void* codes, const void* sf, float alpha, const void* row_scale, const void* x, const void* xs, void* out,
                         const void* residual, const void* ab_w, const void* ab_x, void* ab_out, int ab_rows, int ab_ld, int M,
                         int N, int K, int ldo, int epi, int pdl, cudaStream_t st) {
  if (!codes || !sf || (reinterpret_cast<uintptr_t>(codes) & 15) || (reinterpret_cast<uintptr_t>(sf) & 7) ||
      !tm_args_ok(x, xs, out, residual, ab_w, ab_x, ab_out, ab_rows, ab_ld, M, N, K, ldo, epi))
    return OWL_ERR_BAD_ARG;
  TmParams p = {};
  p.w = (const uint8_t*)codes; p.sf = (const uint8_t*)sf; p.row_scale = (const float*)row_scale; p.x = (const uint8_t*)x;
  p.xs = (const uint8_t*)xs; p.out = (__nv_bfloat16*)out; p.residual = (const __nv_bfloat16*)residual;
  p.ab_w = (const __nv_bfloat16*)ab_w; p.ab_x = (const __nv_bfloat16*)ab_x; p.ab_out = (__nv_bfloat16*)ab_out;
  p.ab_rows = ab_rows; p.ab_ld = ab_ld; p.out_scale = alpha; p.M = M; p.N = N; p.K = K; p.ldo = ldo; p.epi = epi;
  return launch_tm<TF_NV4, false>(p, pdl, st);
}

// First bounded-wait failure of this kernel since the last call (0 = none); clears it.
OWL_API int owl_gemv_tm_status() {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_gemv_tm_status, sizeof(int)) != cudaSuccess) return -1;
  if (v != 0) cudaMemcpyToSymbol(g_gemv_tm_status, &zero, sizeof(int));
  return v;
}
