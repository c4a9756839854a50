// W4A16 GEMM on the 5th-generation tensor cores: out[M,N] = x[M,K] . dequant(qweight, scales), fp16 in and out, fp32
// accumulation in tensor memory; and the same with SwiGLU on the way out (weights gate | up, out[M, N/2]).
//
// Replaces the exported op of samples/05_llama2_7b_int4.py:135-144 for batches above the decode path (and the two
// projections and silu(gate) * up of :168-172 for a prompt); the weight fed to the tensor cores is
// w = RN_fp16(scale * fp16(q - 8)) (IR statement 2), the products accumulate in fp32.
//
// The weights take the M side of the MMA and the rows of x its N side: out^T[n, m] = sum_k w[k, n] x[m, k], M128 N<mt> K16
// with mt = the rows of a tile rounded up to 16, at most 256.  So the row tile follows the prompt (40 rows cost an MMA of
// N = 48, not a padded 128) and a weight is dequantised once per 256 rows.  A CTA takes two runs of 128 columns (two
// accumulators that share the x tile; neighbours, or the gate and up columns of the same 128 outputs) and a range of K in
// units of 64:
//   x        `cp.async.bulk.tensor.2d`, 64 k x mt rows, 128-byte swizzle, the K-major operand as it lands
//   weights  packed words (8 rows x 128 columns, twice) and the group's scales by TMA into their own deeper ring, so that
//            the HBM stream is not bound to registers.
// Where the dequantised weights go is the choice between two forms (the host's cost model takes it):
//   tensor memory (mt <= 192): a thread takes one column of a unit (8 words), turns it into 64 values in k order and stores
//            them with `tcgen05.st`; the MMA takes its A operand from there.  Accumulators 2 x mt columns, the rest two to
//            four stages of 2 x 32 columns.
//   shared memory (mt up to 256, when a round of wide tiles fits the SMs better): a thread takes one packed row of 8
//            columns, pairs the halves of neighbouring columns (`prmt`) and so gets (column, column + 1) pairs for each of
//            the 8 k: the operand is written MN-major (a 128-byte row = 64 columns of one k, 128-byte swizzle, no bank
//            conflicts), without reordering k; three stages of 32 KiB.
// What bounds them: with weights and x both in shared memory a unit moves 3 mt + 700 cycles' worth of it (128 bytes a
// cycle) for 4 mt cycles of MMA; with the weights in tensor memory it is the eight MMAs of a unit, which take 85 to 100
// cycles each however small mt is, 650 + 2 mt a unit in all.  Measured, us, K 4096 N 12288 / 22016: 128 rows 22 / 33, and
// 48 / 37 with the weights in shared memory; 2048 rows 161 / 298.  The kernel before this one (x as the M operand padded to
// 128, K split through global scratch): 43 / 43 and, in the same runs, 187 / 331.
// Roles: 2 x 8 dequantising warps (units alternate between the two halves), one thread each for the x copies and the
// packed copies, one warp for the MMAs; they meet through mbarriers.
// K split: the parts of a tile are the CTAs of one thread-block cluster (at most 8).  After the last MMA every CTA
// pushes its accumulators, 16 rows of x at a time, as fp32 into their owners' shared memory (distributed shared memory,
// 512 contiguous bytes per warp and store), and after one cluster barrier each CTA adds its own in rank order (bitwise
// repeatable).  The library owns no scratch for it: a recorded graph holds no pointer that a later call could move.
// Every mbarrier wait is bounded and reports through the status word (site 210).  In an early launch the rings fill while the
// kernel before still runs; no role starts a wait that x has a part in before that kernel is complete, so that the bound is on
// this kernel alone.
#include <atomic>

#include <cooperative_groups.h>
#include <cuda.h>  // CUtensorMap and its enums (types only)

#include "common.cuh"

namespace cg = cooperative_groups;

namespace ab200 {

constexpr int GS_BN = 256, GS_BK = 64, GS_MAX_MT = 256, GS_TMEM_MT = 192, GS_MAX_PARTS = 8;
constexpr int GS_DQ_WARPS = 16;                              // two groups of 8
constexpr int GS_X_WARP = 16, GS_MMA_WARP = 17, GS_P_WARP = 18;
constexpr int GS_THREADS = 19 * 32;
constexpr int GS_DQ_THREADS = GS_DQ_WARPS * 32;
constexpr int GS_W_COLS = 64;                                // a dequantised unit in tensor memory: 2 x 32 columns
constexpr int GS_PH_BYTES = (GS_BK / 8) * 128 * 4;            // packed words of one accumulator's columns
constexpr int GS_P_BYTES = 2 * GS_PH_BYTES + GS_BN * 2;       // packed unit + scales: 8704
constexpr int GS_W_BYTES = GS_BN * GS_BK * 2;                // the same in shared memory: 2 x [2 blocks of 64 columns][64 k][128 B]
constexpr int GS_MAX_DX = 6, GS_MAX_DW = 4, GS_MAX_DP = 12;  // ring depths: x, dequantised weights, packed weights (the deepest)
constexpr int GS_UNIT_BARS = 8;                              // more than any ring of x or weights is deep
constexpr int GS_ITEM_BYTES = 2 * 128 * 16 * 4;               // K split: 256 columns x 16 rows of x, fp32
constexpr int GS_ROWB = GS_BN * 2 + 16;                       // bytes per parked output row
constexpr int GS_SMEM_LIMIT = 227 * 1024 - 1024;             // 1 KiB for the static part
constexpr int GS_TILE_CYCLES = 6000, GS_SPLIT_CYCLES = 3000, GS_SPLIT_ROW_CYCLES = 30;  // see gemm_launch
constexpr unsigned GS_WAIT_POLLS = 1u << 22;

struct GemmParams {
  __half *out;
  int M, K, N, group;
  int mt;      // rows of x per tile, a multiple of 16
  int second;  // columns from an accumulator's run of 128 to the other's: 128, or N / 2 (gate | up)
  int n_out;   // columns of out
  int dx, dw, dp;  // ring depths
  int *status;
  int early;   // launched while the kernel before runs: weights and scales date from before it
};

__device__ __forceinline__ uint32_t gs_smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
// 128-byte-swizzled operand: atoms of 8 x 128 B, 1024 B apart; lead: bytes between blocks of 64 elements along MN of an
// MN-major operand (not used by a K-major one)
__device__ __forceinline__ uint64_t gs_desc(uint32_t addr, uint32_t lead) {
  return (uint64_t)((addr >> 4) & 0x3FFF) | (uint64_t)((lead >> 4) & 0x3FFF) << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)2 << 61;
}
// X: x has a part in what is waited for.  In an early launch the polls, which are counted, then begin when the kernel before is
// complete.
template <bool X>
__device__ __forceinline__ bool gs_wait(uint32_t bar, unsigned parity) {
  {  // non-blocking probe first: cheaper than try_wait when the phase completed long ago
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  if (X) pdl_wait();
  for (unsigned i = 0; i < GS_WAIT_POLLS; ++i) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}
__device__ __forceinline__ void gs_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void gs_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void gs_tma(uint32_t dst, const CUtensorMap *tm, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
               "l"(reinterpret_cast<uint64_t>(tm)), "r"(x), "r"(y), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void gs_commit(uint32_t bar) {  // by the thread that issues the MMAs
  asm volatile("{\n .reg .pred q;\n elect.sync _|q, 0xffffffff;\n @q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool gs_elect() {
  uint32_t e;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(e));
  return e != 0;
}
__device__ __forceinline__ void gs_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
        "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void gs_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};" ::"r"(r[0]), "r"(r[1]), "r"(r[2]),
               "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]),
               "r"(r[15]), "r"(taddr)
               : "memory");
}

__device__ __forceinline__ float gs_silu_mul(float g, float u) {  // of the fp16 results, as the separate kernel has them
  g = __half2float(__float2half_rn(g));
  return g / (1.0f + expf(-g)) * __half2float(__float2half_rn(u));
}

// SILU: the accumulators are gate and up of the same outputs, out = silu(gate) * up.  TMEM: where the dequantised weights are.
template <bool SILU, bool TMEM>
__global__ void __launch_bounds__(GS_THREADS, 1) w4a16_gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w,
                                                                         const __grid_constant__ CUtensorMap tm_s, GemmParams p) {
  extern __shared__ unsigned char gs_raw[];
  unsigned char *smem = gs_raw + ((1024u - (gs_smem_u32(gs_raw) & 1023u)) & 1023u);  // swizzle atoms need 1024-byte alignment
  // barriers of unit u (slot u % 8): operands there (eight dequantising warps and the x copy), MMAs complete; of the packed
  // ring: full, empty [12]; all MMAs complete
  __shared__ __align__(8) uint64_t bars[2 * GS_UNIT_BARS + 2 * GS_MAX_DP + 1];
  __shared__ uint32_t tmem_s;
  __shared__ int fail_s;
  cg::cluster_group cluster = cg::this_cluster();
  const int parts = (int)cluster.num_blocks(), part = (int)cluster.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n0 = ((int)blockIdx.x / parts) * (SILU ? GS_BN / 2 : GS_BN), mt = p.mt, m0 = (int)blockIdx.y * mt;
  const int units = p.K / GS_BK, u0 = (int)((long)units * part / parts), n_units = (int)((long)units * (part + 1) / parts) - u0;
  const int dx = p.dx, dw = p.dw, dp = p.dp;
  const uint32_t xb = (uint32_t)mt * (GS_BK * 2);
  const uint32_t b_full = gs_smem_u32(bars), b_used = b_full + 8 * GS_UNIT_BARS, b_pfull = b_used + 8 * GS_UNIT_BARS, b_pempty = b_pfull + 8 * GS_MAX_DP,
                 b_done = b_pempty + 8 * GS_MAX_DP;
  auto bar_of = [](uint32_t first, int u) { return first + 8 * (u & (GS_UNIT_BARS - 1)); };
  auto phase_of = [](int u) { return (unsigned)(u / GS_UNIT_BARS) & 1u; };
  const uint32_t s_w = gs_smem_u32(smem), s_x = s_w + (TMEM ? 0 : dw * GS_W_BYTES), s_p = s_x + dx * xb;

  if (tid == 0) {
    auto init = [](uint32_t bar, int count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count)); };
    for (int i = 0; i < GS_UNIT_BARS; ++i) init(b_full + 8 * i, GS_DQ_WARPS / 2 + 1), init(b_used + 8 * i, 1);
    for (int i = 0; i < GS_MAX_DP; ++i) init(b_pfull + 8 * i, 1), init(b_pempty + 8 * i, GS_DQ_WARPS / 2);
    init(b_done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fail_s = 0;
  }
  if (warp == GS_MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(gs_smem_u32(&tmem_s)), "n"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (p.early) pdl_launch_dependents();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_s, 0), acc1 = (mt + 31) & ~31, tmem_w = tmem + 2 * acc1;  // accumulators, then the weights
  bool good = true;

  if (warp == GS_P_WARP) {
    if (gs_elect()) {  // packed words and scales
      for (int u = 0, slot = 0, ph = 1; u < n_units; ++u) {
        if (u >= dp && !gs_wait<true>(b_pempty + 8 * slot, ph)) {
          good = false;
          break;
        }
        const uint32_t bar = b_pfull + 8 * slot, dst = s_p + slot * GS_P_BYTES;
        gs_expect(bar, GS_P_BYTES);
        const int row = (u0 + u) * (GS_BK / 8), srow = row * 8 / p.group;
        gs_tma(dst, &tm_w, n0, row, bar);
        gs_tma(dst + GS_PH_BYTES, &tm_w, n0 + p.second, row, bar);
        gs_tma(dst + 2 * GS_PH_BYTES, &tm_s, n0, srow, bar);
        gs_tma(dst + 2 * GS_PH_BYTES + 256, &tm_s, n0 + p.second, srow, bar);
        if (++slot == dp) slot = 0, ph ^= 1;
      }
      if (!good) fail_s = 1;
    }
    __syncwarp();
  } else if (warp == GS_X_WARP) {
    if (gs_elect()) {  // x tiles
      pdl_wait();      // x comes from the kernel before this one; weights and scales may be on their way already (p.early)
      for (int u = 0, slot = 0; u < n_units; ++u) {
        if (u >= dx && !gs_wait<true>(bar_of(b_used, u - dx), phase_of(u - dx))) {
          good = false;
          break;
        }
        gs_expect(bar_of(b_full, u), xb);
        gs_tma(s_x + slot * xb, &tm_x, (u0 + u) * GS_BK, m0, bar_of(b_full, u));
        if (++slot == dx) slot = 0;
      }
      if (!good) fail_s = 1;
    }
    __syncwarp();
  } else if (warp == GS_MMA_WARP) {
    // The whole warp runs the loop and only the MMAs and commits are one thread's: in a divergent branch every descriptor
    // would have to be moved into uniform registers on its own.
    // Instruction descriptor: D fp32, A/B fp16, B K-major, A K-major or (bit 15) MN-major, N = mt, M = 128
    const uint32_t idesc = (1u << 4) | (TMEM ? 0u : 1u << 15) | ((uint32_t)(mt >> 3) << 17) | (128u >> 4 << 24);
    // One wait and one commit per unit: at some hundred cycles each they, not the MMAs, are what this loop takes.
    for (int u = 0, xs = 0, ws = 0; u < n_units; ++u) {
      good = __all_sync(0xffffffffu, gs_wait<true>(bar_of(b_full, u), phase_of(u)));
      if (!good) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint64_t b0 = gs_desc(s_x + xs * xb, 16);
#pragma unroll
      for (int k = 0; k < GS_BK / 16; ++k)
#pragma unroll
        for (int a = 0; a < 2; ++a) {  // 16 k further: 32 B inside a row of x; 8 columns of tensor memory or two atoms of the weights
          const uint32_t accumulate = (u > 0 || k > 0) ? 1u : 0u;
          if constexpr (TMEM)
            asm volatile(
                "{\n .reg .pred p, q;\n elect.sync _|q, 0xffffffff;\n setp.ne.b32 p, %4, 0;\n @q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(
                    tmem + a * acc1),
                "r"(tmem_w + ws * GS_W_COLS + a * 32 + k * 8), "l"(b0 + (uint64_t)(k * 2)), "r"(idesc), "r"(accumulate)
                : "memory");
          else
            asm volatile(
                "{\n .reg .pred p, q;\n elect.sync _|q, 0xffffffff;\n setp.ne.b32 p, %4, 0;\n @q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(
                    tmem + a * acc1),
                "l"(gs_desc(s_w + ws * GS_W_BYTES, GS_BK * 128) + (uint64_t)((a * (GS_W_BYTES / 2) + k * 2048) >> 4)), "l"(b0 + (uint64_t)(k * 2)), "r"(idesc), "r"(accumulate)
                : "memory");
        }
      gs_commit(bar_of(b_used, u));
      if (++xs == dx) xs = 0;
      if (++ws == dw) ws = 0;
    }
    gs_commit(b_done);
    if (!good) fail_s = 1;
  } else {
    // ---- dequantise: half h takes units h, h + 2, ..
    // TMEM: a thread has one column, tensor-memory lane q * 32 + lane of accumulator a.
    // Otherwise: warp r of a half packed row r, lane c columns 8c .. 8c + 7.
    const int h = warp >> 3, a = TMEM ? (warp >> 2) & 1 : lane >> 4, q = warp & 3, r8 = warp & 7;
    const unsigned char *ring = smem + (s_p - s_w);
    const unsigned char *words = ring + a * GS_PH_BYTES + (TMEM ? (q * 32 + lane) * 4 : r8 * 512 + (lane & 15) * 32);
    const unsigned char *scale = ring + 2 * GS_PH_BYTES + (TMEM ? a * 256 + (q * 32 + lane) * 2 : lane * 16);
    constexpr uint32_t LO = 0x000F000Fu, HI = 0x00F000F0u, MAGIC = 0x64006400u;
    const __half2 c1032 = u2h2(0x64086408u), c16th = u2h2(0x2C002C00u), cm72 = u2h2(0xD480D480u);
    // RN(scale * (q - 8)) of the nibbles at bits 0 and 16 (l0), 4 and 20 (l1), 8 and 24 (l2), 12 and 28 (l3)
    auto dequant = [&](uint32_t v, __half2 sc, uint32_t &l0, uint32_t &l1, uint32_t &l2, uint32_t &l3) {
      const uint32_t v8 = v >> 8;
      l0 = h22u(__hmul2(__hsub2(u2h2(lop3<0xEA>(v, LO, MAGIC)), c1032), sc));
      l1 = h22u(__hmul2(__hfma2(u2h2(lop3<0xEA>(v, HI, MAGIC)), c16th, cm72), sc));
      l2 = h22u(__hmul2(__hsub2(u2h2(lop3<0xEA>(v8, LO, MAGIC)), c1032), sc));
      l3 = h22u(__hmul2(__hfma2(u2h2(lop3<0xEA>(v8, HI, MAGIC)), c16th, cm72), sc));
    };
    int ps = h, ws = h, pph = 0;  // ring slots of unit u, kept by counting: no divisions in the loop
    for (int u = h; u < n_units; u += 2) {
      // The stage first: once the MMAs of unit u - dw are complete, so is every packed unit up to there, and the packed
      // ring (at least as deep) cannot be two phases behind what this half, which sees every second unit, waits for.  (Nor
      // can the barrier waited on here: the MMAs of unit u - 2 - dw are known to be complete.)
      if (u >= dw) good = __all_sync(0xffffffffu, gs_wait<true>(bar_of(b_used, u - dw), phase_of(u - dw)));
      good = good && __all_sync(0xffffffffu, gs_wait<false>(b_pfull + 8 * ps, pph));
      if (!good) break;
      uint32_t w[8];
      uint4 sv = make_uint4(0, 0, 0, 0);
      if constexpr (TMEM) {
#pragma unroll
        for (int r = 0; r < 8; ++r) w[r] = *reinterpret_cast<const uint32_t *>(words + ps * GS_P_BYTES + r * 512);
        sv.x = h22u(__half2half2(*reinterpret_cast<const __half *>(scale + ps * GS_P_BYTES)));
      } else {
        const uint4 wa = *reinterpret_cast<const uint4 *>(words + ps * GS_P_BYTES), wb = *reinterpret_cast<const uint4 *>(words + ps * GS_P_BYTES + 16);
        w[0] = wa.x, w[1] = wa.y, w[2] = wa.z, w[3] = wa.w, w[4] = wb.x, w[5] = wb.y, w[6] = wb.z, w[7] = wb.w;
        sv = *reinterpret_cast<const uint4 *>(scale + ps * GS_P_BYTES);
      }
      __syncwarp();
      if (lane == 0) gs_arrive(b_pempty + 8 * ps);
      if constexpr (TMEM) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          uint32_t o[16];  // four words: 32 values in k order, two per column of tensor memory
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            uint32_t k04, k15, k26, k37;
            dequant(w[4 * half + r], u2h2(sv.x), k04, k15, k26, k37);
            o[4 * r] = __byte_perm(k04, k15, 0x5410);
            o[4 * r + 1] = __byte_perm(k26, k37, 0x5410);
            o[4 * r + 2] = __byte_perm(k04, k15, 0x7632);
            o[4 * r + 3] = __byte_perm(k26, k37, 0x7632);
          }
          gs_st16(tmem_w + a * 32 + ((uint32_t)(q * 32) << 16) + ws * GS_W_COLS + half * 16, o);
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      } else {
        uint32_t o[8][4];  // [k][column pair]
        const uint32_t sc[4] = {sv.x, sv.y, sv.z, sv.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {  // k 0..3 are the low halves of the words, k 4..7 the high ones
          dequant(__byte_perm(w[2 * j], w[2 * j + 1], 0x5410), u2h2(sc[j]), o[0][j], o[1][j], o[2][j], o[3][j]);
          dequant(__byte_perm(w[2 * j], w[2 * j + 1], 0x7632), u2h2(sc[j]), o[4][j], o[5][j], o[6][j], o[7][j]);
        }
        unsigned char *dst = smem + ws * GS_W_BYTES + (lane >> 3) * (GS_BK * 128) + r8 * 1024;  // block of 64 columns, atom of 8 k
#pragma unroll
        for (int k = 0; k < 8; ++k) *reinterpret_cast<uint4 *>(dst + k * 128 + (((lane & 7) ^ k) << 4)) = make_uint4(o[k][0], o[k][1], o[k][2], o[k][3]);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // generic-proxy writes -> visible to the tensor core
      }
      __syncwarp();
      if (lane == 0) gs_arrive(bar_of(b_full, u));
      ws += 2;
      if (ws >= dw) ws -= dw;
      ps += 2;
      if (ps >= dp) ps -= dp, pph ^= 1;
    }
    if (!good) fail_s = 1;
  }
  pdl_wait();  // (long satisfied) out may still have been in use
  // ---- all MMAs of this CTA are done, its shared memory is idle -----------------------------------------------------
  if (!gs_wait<true>(b_done, 0)) fail_s = 1;
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  __syncthreads();
  const bool failed = fail_s != 0;

  // Epilogue.  A warp reads the tensor-memory lanes of its quarter (warp % 4): lane = column of an accumulator's run; the
  // four warps of a quarter share the mt accumulator columns (= rows of x) in chunks of 16.
  const int q = warp & 3, sub = warp >> 2;
  const int chunks = mt / 16;
  const uint32_t lanes = (uint32_t)(q * 32) << 16;
  if (parts == 1) {
    // A thread holds a column: results are parked row by row in the idle operand memory and leave as whole 512-byte rows
    // (SILU: 256).  (Two bytes per lane straight to global memory were 5-10% of a large call.)
    constexpr int ROW_VECS = (SILU ? GS_BN / 2 : GS_BN) / 8;
    if (warp < GS_DQ_WARPS && !failed) {
      for (int i = sub; i < chunks; i += 4) {
        if (m0 + i * 16 >= p.M) break;
        float v[16], w[16];
        gs_ld16(tmem + i * 16 + lanes, v);
        gs_ld16(tmem + acc1 + i * 16 + lanes, w);
        __half *o = reinterpret_cast<__half *>(smem + (size_t)i * 16 * GS_ROWB) + q * 32 + lane;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          if (SILU) {
            o[j * (GS_ROWB / 2)] = __float2half_rn(gs_silu_mul(v[j], w[j]));
          } else {
            o[j * (GS_ROWB / 2)] = __float2half_rn(v[j]);
            o[j * (GS_ROWB / 2) + 128] = __float2half_rn(w[j]);
          }
        }
      }
      asm volatile("bar.sync 1, %0;" ::"n"(GS_DQ_THREADS) : "memory");
      const int piece = tid % ROW_VECS, n = n0 + piece * 8, rows = min(mt, p.M - m0);
      if (n < p.n_out)  // n_out is a multiple of 8: a piece is inside or outside as a whole
        for (int m = tid / ROW_VECS; m < rows; m += GS_DQ_THREADS / ROW_VECS)
          *reinterpret_cast<uint4 *>(p.out + (size_t)(m0 + m) * p.n_out + n) = *reinterpret_cast<const uint4 *>(smem + (size_t)m * GS_ROWB + piece * 16);
    }
  } else {
    // The chunks are owned by the ranks in consecutive runs.  Inbox of a CTA: [own chunk][source rank][accumulator][row
    // quad][column][4] fp32, 16 KiB per chunk and rank.  When they do not fit together, half of them go first.
    const int rounds = ((chunks + parts - 1) / parts) * parts * GS_ITEM_BYTES <= GS_SMEM_LIMIT - 1024 ? 1 : 2;
    for (int round = 0; round < rounds; ++round) {
      const int c0 = chunks * round / rounds, count = chunks * (round + 1) / rounds - c0;
      auto first = [&](int r) { return count * r / parts; };
      const int own0 = first(part), own = first(part + 1) - own0;
      cluster.sync();  // every CTA's shared memory is idle
      if (warp < GS_DQ_WARPS) {
        int owner = 0;
        for (int i = sub >> 1; i < count; i += 2) {  // two warps of a quarter per accumulator
          while (first(owner + 1) <= i) ++owner;
          const int a = sub & 1;
          float v[16];
          gs_ld16(tmem + a * acc1 + (c0 + i) * 16 + lanes, v);
          float4 *dst = reinterpret_cast<float4 *>(cluster.map_shared_rank(smem, owner) + ((i - first(owner)) * parts + part) * GS_ITEM_BYTES) + a * 512 + q * 32 + lane;
#pragma unroll
          for (int j = 0; j < 4; ++j) dst[j * 128] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        }
      }
      cluster.sync();
      if (warp < GS_DQ_WARPS && !failed) {
        for (int i = 0; i < own; ++i) {  // thread = row quad tid / 128 of a chunk, column tid % 128 of both accumulators
          const int m = m0 + (c0 + own0 + i) * 16 + (tid >> 7) * 4, n = n0 + (tid & 127);
          const float4 *src = reinterpret_cast<const float4 *>(smem + (size_t)i * parts * GS_ITEM_BYTES) + tid;
          float4 t = src[0], u = src[512];
          for (int r = 1; r < parts; ++r) {
            const float4 a = src[r * (GS_ITEM_BYTES / 16)], b = src[r * (GS_ITEM_BYTES / 16) + 512];
            t.x += a.x, t.y += a.y, t.z += a.z, t.w += a.w;
            u.x += b.x, u.y += b.y, u.z += b.z, u.w += b.w;
          }
          const float f[4] = {t.x, t.y, t.z, t.w}, g[4] = {u.x, u.y, u.z, u.w};
          __half *o = p.out + (size_t)m * p.n_out + n;
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (m + j < p.M) {
              if (SILU) {
                if (n < p.n_out) o[(size_t)j * p.n_out] = __float2half_rn(gs_silu_mul(f[j], g[j]));
              } else {
                if (n < p.n_out) o[(size_t)j * p.n_out] = __float2half_rn(f[j]);
                if (n + 128 < p.n_out) o[(size_t)j * p.n_out + 128] = __float2half_rn(g[j]);
              }
            }
        }
      }
    }
  }
  if (failed && tid == 0) atomicExch(p.status, 210);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == GS_MMA_WARP) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(512) : "memory");
}

// Clusters of `parts` CTAs of this kernel that are resident at once on the current device (asked once per device).
static int gs_clusters(int parts) {
  static std::atomic<int> known[64][GS_MAX_PARTS + 1];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  int n = known[dev][parts].load(std::memory_order_relaxed);
  if (n == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(parts, 1, 1);
    cfg.blockDim = dim3(GS_THREADS, 1, 1);
    cfg.dynamicSmemBytes = GS_SMEM_LIMIT;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = parts;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, w4a16_gemm_tcgen05_kernel<false, true>, &cfg) != cudaSuccess || n < 1) {
      (void)cudaGetLastError();
      n = -1;
    }
    known[dev][parts].store(n, std::memory_order_relaxed);
  }
  return n;
}

static int gemm_launch(const void *x, const int32_t *qweight, const void *scales, void *out, int M, int K, int N, int group, bool silu, bool early, cudaStream_t stream) {
  AB200_REQUIRE(x && qweight && scales && out, "w4a16_gemm: null pointer");
  AB200_REQUIRE(M > 0 && N > 0 && N % 8 == 0, "w4a16_gemm: M=%d must be positive, N=%d a positive multiple of 8", M, N);
  AB200_REQUIRE(K > 0 && K % GS_BK == 0, "w4a16_gemm: K=%d must be a positive multiple of %d", K, GS_BK);
  AB200_REQUIRE(group >= GS_BK && group % GS_BK == 0 && K % group == 0, "w4a16_gemm: group=%d must be a multiple of %d dividing K", group, GS_BK);
  AB200_REQUIRE(aligned16(x) && aligned16(qweight) && aligned16(scales) && aligned16(out), "w4a16_gemm: pointers must be 16-byte aligned");
  int *status = kernel_error_ptr();
  AB200_REQUIRE(status != nullptr, "w4a16_gemm: cannot resolve the status word");
  typedef CUresult (*EncodeFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                               const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  EncodeFn enc = reinterpret_cast<EncodeFn>(tensor_map_encoder());
  if (!enc) return fail(AB200_EUNSUPPORTED, "w4a16_gemm: this driver has no cuTensorMapEncodeTiled");
  AB200_CUDA(cudaFuncSetAttribute(w4a16_gemm_tcgen05_kernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, GS_SMEM_LIMIT));  // gs_clusters asks about it

  // Row tiles: at least M / 256; more and narrower ones when that fills the last round of CTAs better.  K split, when the
  // tiles leave SMs idle: as many parts as keep every tile's cluster resident at once (a cluster lies within one GPC, so
  // this is not SMs / parts), each of at least 4 units.  A unit costs about what was measured for the two
  // forms; a tile costs its start and epilogue, a split the exchange of its rows.  Unsplit, K = 4096, a round of all SMs takes
  // 33 / 35 / 37 us at 112 / 128 / 160 rows, 44 / 45 at 176 / 192 (tensor memory then has two stages of weights in place of
  // three) and 47.5 / 50 / 51.5 with the weights in shared memory at 208 / 240 / 256.  2048 rows of N 12288 / 22016 take 161 / 298 us
  // so (9 and 8 tiles), 183 / 343 with the former's costs taken for both (12 tiles of 176), 187 / 331 the kernel before this one.
  const int tiles_n = silu ? (N / 2 + GS_BN / 2 - 1) / (GS_BN / 2) : (N + GS_BN - 1) / GS_BN, units = K / GS_BK, sms = sm_count();
  auto rows_of = [&](int tiles_m) { return ((M + tiles_m - 1) / tiles_m + 15) / 16 * 16; };
  auto parts_of = [&](long tiles) {
    int parts = GS_MAX_PARTS;
    while (parts > 1 && (parts > units / 4 || tiles * parts > sms || tiles > gs_clusters(parts))) --parts;
    return parts;
  };
  auto cost = [&](int tiles_m) {
    const long tiles = (long)tiles_n * tiles_m, rounds = (tiles + sms - 1) / sms;
    const int rows = rows_of(tiles_m), parts = parts_of(tiles);
    const int unit = rows > GS_TMEM_MT ? (parts == 1 ? 770 + 5 * rows / 2 : 700 + 3 * rows) : 650 + 2 * rows + (parts == 1 && rows > 160 ? 170 : 0);
    return rounds * ((long)((units + parts - 1) / parts) * unit + GS_TILE_CYCLES + (parts > 1 ? GS_SPLIT_CYCLES + rows * GS_SPLIT_ROW_CYCLES : 0));
  };
  const int least = (M + GS_MAX_MT - 1) / GS_MAX_MT;
  int tiles_m = least;
  long best = cost(least);
  for (int t = least + 1; t <= least + 8 && t <= (M + 15) / 16; ++t)
    if (const long c = cost(t); c < best) best = c, tiles_m = t;
  const int mt = rows_of(tiles_m), parts = parts_of((long)tiles_n * tiles_m);

  auto encode = [&](CUtensorMap *tm, CUtensorMapDataType type, const void *base, int elt, cuuint64_t inner, cuuint64_t outer, int box_inner, int box_outer,
                    CUtensorMapSwizzle swizzle) {
    const cuuint64_t dims[2] = {inner, outer}, strides[1] = {inner * elt};
    const cuuint32_t box[2] = {(cuuint32_t)box_inner, (cuuint32_t)box_outer}, estr[2] = {1, 1};
    return enc(tm, type, 2, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  };
  CUtensorMap tm_x, tm_w, tm_s;
  CUresult r = encode(&tm_x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, x, 2, K, M, GS_BK, mt, CU_TENSOR_MAP_SWIZZLE_128B);
  if (r == CUDA_SUCCESS) r = encode(&tm_w, CU_TENSOR_MAP_DATA_TYPE_INT32, qweight, 4, N, K / 8, 128, GS_BK / 8, CU_TENSOR_MAP_SWIZZLE_NONE);
  if (r == CUDA_SUCCESS) r = encode(&tm_s, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, scales, 2, N, K / group, 128, 1, CU_TENSOR_MAP_SWIZZLE_NONE);
  if (r != CUDA_SUCCESS) return fail(AB200_ECUDA, "w4a16_gemm: cuTensorMapEncodeTiled failed with %d", (int)r);

  GemmParams p{(__half *)out, M, K, N, group, mt, silu ? N / 2 : 128, silu ? N / 2 : N, 0, 0, 0, status, early && pdl_enabled()};
  const bool in_tmem = mt <= GS_TMEM_MT;
  const int xb = mt * GS_BK * 2, w_cols = 512 - 2 * ((mt + 31) & ~31);
  p.dw = !in_tmem ? 3 : w_cols / GS_W_COLS < GS_MAX_DW ? w_cols / GS_W_COLS : GS_MAX_DW;
  p.dx = in_tmem ? GS_MAX_DX : 3;
  const int room = GS_SMEM_LIMIT - 1024 - p.dx * xb - (in_tmem ? 0 : p.dw * GS_W_BYTES);  // for at least 3 packed units (mt = 256), 9 in tensor memory's form
  p.dp = room / GS_P_BYTES < GS_MAX_DP ? room / GS_P_BYTES : GS_MAX_DP;
  auto kern = silu ? (in_tmem ? w4a16_gemm_tcgen05_kernel<true, true> : w4a16_gemm_tcgen05_kernel<true, false>) : (in_tmem ? w4a16_gemm_tcgen05_kernel<false, true> : w4a16_gemm_tcgen05_kernel<false, false>);
  AB200_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GS_SMEM_LIMIT));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(tiles_n * parts, tiles_m, 1);
  cfg.blockDim = dim3(GS_THREADS, 1, 1);
  cfg.dynamicSmemBytes = GS_SMEM_LIMIT;  // one CTA per SM; the inboxes of a K split use all of it
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = parts;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = p.early ? 2 : 1;
  AB200_CUDA(cudaLaunchKernelEx(&cfg, kern, tm_x, tm_w, tm_s, p));
  return AB200_OK;
}

}  // namespace ab200

using namespace ab200;

extern "C" int ab200_w4a16_gemm(const void *x, const int32_t *qweight, const void *scales, void *out, int M, int K, int N,
                                int group, int dtype, void *stream) {
  clear_error();
  AB200_REQUIRE(x && qweight && scales && out, "w4a16_gemm: null pointer");
  if (dtype != AB200_F16) return fail(AB200_EUNSUPPORTED, "w4a16_gemm: the tensor-core path is built for float16 (dtype %d given)", dtype);
  return gemm_launch(x, qweight, scales, out, M, K, N, group, false, false, (cudaStream_t)stream);
}

extern "C" int ab200_w4a16_gemm_early(const void *x, const int32_t *qweight, const void *scales, void *out, int M, int K, int N, int group, int silu, void *stream) {
  clear_error();
  AB200_REQUIRE(!silu || N % 16 == 0, "w4a16_gemm_early: N=%d must be twice a multiple of 8", N);
  return gemm_launch(x, qweight, scales, out, M, K, N, group, silu != 0, true, (cudaStream_t)stream);
}

extern "C" int ab200_w4a16_gemm_silu(const void *x, const int32_t *qweight, const void *scales, void *out, int M, int K, int N, int group, void *stream) {
  clear_error();
  AB200_REQUIRE(N % 16 == 0, "w4a16_gemm_silu: N=%d must be twice a multiple of 8", N);
  return gemm_launch(x, qweight, scales, out, M, K, N, group, true, false, (cudaStream_t)stream);
}
