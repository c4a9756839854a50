// Causal attention of a batch of prompt rows over an fp16 KV cache on the 5th-generation tensor cores
// (the batched form of samples/05_llama2_7b_int4.py:161-165): p = softmax_s(scale * q.K_s), out = sum_s p_s V_s,
// query row r (position pos0 + r) over the cache rows 0 .. pos0 + r.
//
// A CTA takes one head and 128 consecutive query rows and walks the cache in tiles of 64 rows:
//   S = Q K^T        8 `tcgen05.mma` M128 N64 K16, both operands in shared memory, S (fp32) in tensor memory
//   P = exp(S - max) four warps, one query row per thread; P goes back to tensor memory over S
//   O += P V         8 `tcgen05.mma` M128 N128 K16, P is the A operand straight from tensor memory
// P is stored as an fp16 pair hi + lo, 22 bits of an fp32 probability's 24, and both halves are multiplied with V into
// the same fp32 accumulator, so only q, K, V and the result are 16 bits wide.  P is scaled by 2^6 (the row sum with it),
// which keeps lo out of the subnormals where it matters.  The running maximum is only raised when a tile exceeds it by
// more than 2^8, as FlashAttention-4 does it (then O is rescaled in tensor memory): what the row is finally divided by
// contains the same factor.  Error of the fp16 result against 64 bits, 2000 rows: 1.95138e-4, the fp32 single-query
// kernel 1.95134e-4, the exact result rounded to fp16 1.95134e-4; the difference, 1e-6 of the result, is the tensor
// cores' accumulation (it grows with the number of MMAs a row has gone through).  The pair's own share is 5e-8 of the
// result, an fp32 probability's 2.4e-8, fp16 alone would be 2e-4.
//
// Roles: warps 0-3 softmax (warp w = tensor-memory lanes 32w..32w+31), warp 4 brings K tiles in and warps 5-6 V tiles
// (`cp.async`, 16 bytes per thread, into the 128-byte-swizzled layout both MMAs read: K-major for S, MN-major
// for O; a page table only changes the row address), warp 7 issues the MMAs.  S, K and V are
// double buffered; 97 KiB of shared memory and 256 tensor-memory columns, so two CTAs are
// resident per SM and one's MMAs run under the other's softmax.  Query tiles are issued last row first: the
// longest CTAs start first.
//
// What bounds it: the softmax warps.  A tile of a CTA takes 2200 cycles, 1250 of them exponentials, row sums and the split
// of P (two softmax warps share a scheduler's 4 exponentials a cycle: 1024 cycles); its 16 MMAs wait for that.
// 32 heads, 2000 rows: 78 us (4162 with the single-query kernel once per row); 128 rows: 12 us (33).
//
// Values of V that are not finite: a masked or underflowed probability is exactly 0 in the MMA, and 0 * inf
// would reach rows that never attend to that key.  The loading warps look at every V tile; a CTA that saw one
// recomputes its rows with fp32 code that touches only the keys a row attends to (attend_rows below).
#include <math_constants.h>

#include <type_traits>

#include "common.cuh"

namespace ab200 {

constexpr int AP_D = 128, AP_BM = 128, AP_BN = 64;
constexpr int AP_SOFT_WARPS = 4, AP_LOAD_WARPS = 3;  // one loads K, two load V and look at it
constexpr int AP_MMA_WARP = AP_SOFT_WARPS + AP_LOAD_WARPS;
constexpr int AP_THREADS = (AP_MMA_WARP + 1) * 32;
constexpr int AP_Q_BYTES = AP_BM * AP_D * 2;      // 32 KiB: two halves of 64 dims, [128 rows][128 B] each
constexpr int AP_STAGE_BYTES = AP_BN * AP_D * 2;  // 16 KiB: two halves of 64 dims, [64 rows][128 B] each
constexpr int AP_STAGES = 4;                      // two of K, two of V
constexpr int AP_SMEM = AP_Q_BYTES + AP_STAGES * AP_STAGE_BYTES + 1024;
constexpr int AP_TMEM_COLS = 256;                 // S0 | S1 (64 each, P overlays S), O (128)
constexpr int AP_ROWB = AP_D * 2 + 16;            // bytes per parked output row
constexpr unsigned AP_WAIT_POLLS = 1u << 22;
constexpr float AP_P_EXP = 6.f;                   // P is scaled by 2^6
constexpr float AP_RAISE = 8.f;                   // raise the running maximum when a tile exceeds it by 2^8

struct AttnPrefillParams {
  const __half *q;
  const __half *kc, *vc;
  __half *out;
  const int32_t *pos0;
  int rows, max_seq, H;
  long kv_stride;
  float scale;
  KvPages pages;
  int *status;
};

__device__ __forceinline__ uint32_t ap_smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// 128-byte-swizzled operand (rows of 128 B, atoms of 8 rows = 1024 B, stride between atoms 1024 B).  lead: bytes
// between blocks of 64 elements along MN for an MN-major operand (unused, 1 unit, for a K-major one).
__device__ __forceinline__ uint64_t ap_desc(uint32_t addr, uint32_t lead_bytes) {
  return (uint64_t)((addr >> 4) & 0x3FFF) | (uint64_t)((lead_bytes >> 4) & 0x3FFF) << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)2 << 61;
}

__device__ __forceinline__ bool ap_wait(uint32_t bar, unsigned parity) {
  for (unsigned i = 0; i < AP_WAIT_POLLS; ++i) {
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
__device__ __forceinline__ void ap_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
// The whole warp runs the issuing loop and only these instructions are one thread's: in a divergent branch every
// descriptor would have to be moved into uniform registers on its own.
__device__ __forceinline__ void ap_commit(uint32_t bar) {
  asm volatile("{\n .reg .pred q;\n elect.sync _|q, 0xffffffff;\n @q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(bar) : "memory");
}
// D (+)= A.B, A in shared memory (ss) or tensor memory (ts)
__device__ __forceinline__ void ap_mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p, q;\n elect.sync _|q, 0xffffffff;\n setp.ne.b32 p, %4, 0;\n @q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d), "l"(a), "l"(b),
      "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void ap_mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p, q;\n elect.sync _|q, 0xffffffff;\n setp.ne.b32 p, %4, 0;\n @q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d), "r"(a), "l"(b),
      "r"(idesc), "r"(accumulate)
      : "memory");
}
#define AP_R16(r, o) "=r"(r[o]), "=r"(r[o + 1]), "=r"(r[o + 2]), "=r"(r[o + 3]), "=r"(r[o + 4]), "=r"(r[o + 5]), "=r"(r[o + 6]), "=r"(r[o + 7]), \
    "=r"(r[o + 8]), "=r"(r[o + 9]), "=r"(r[o + 10]), "=r"(r[o + 11]), "=r"(r[o + 12]), "=r"(r[o + 13]), "=r"(r[o + 14]), "=r"(r[o + 15])
#define AP_I16(r) "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), \
    "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
// 32 columns of this warp's 32 lanes; the caller waits
__device__ __forceinline__ void ap_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : AP_R16(r, 0), AP_R16(r, 16)
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void ap_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};" ::AP_I16(r), "r"(taddr) : "memory");
}
__device__ __forceinline__ void ap_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void ap_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ float ap_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Four consecutive query rows by one warp in fp32, two passes over exactly the keys each attends to (lane = 4 dims).
// Four keys at a time: their rows are loaded once for the four queries, and the 16 dot products are summed over the warp
// together (16 shuffles), lane 2 i + (0, 1) ending with the score of key i / 4 and row i % 4.
// 32 heads with a value that is not finite, us: 70 / 128 / 512 / 2000 rows 83 / 147 / 639 / 4170; the single-query kernel once
// per row 24 / 42 / 306 / 4020; a warp with one row and one key at a time 2574 at 128 rows, 47242 at 2000.
__device__ __noinline__ void attend_rows(const AttnPrefillParams &p, int h, int row0, int pos0) {
  constexpr int R = 4, KEYS = 4;
  const int lane = threadIdx.x & 31, my_key = lane >> 3, my_row = (lane >> 1) & 3;
  auto wide4 = [](uint2 v, float (&f)[4]) {
    const float2 a = __half22float2(u2h2(v.x)), b = __half22float2(u2h2(v.y));
    f[0] = a.x, f[1] = a.y, f[2] = b.x, f[3] = b.y;
  };
  auto limit = [&](int r) {  // cache rows that row row0 + r attends to; not falling with r
    const long s = (long)pos0 + 1 + min(row0 + r, p.rows - 1);
    return (int)(s < 0 ? 0 : s > p.max_seq ? p.max_seq : s);
  };
  float qf[R][4], acc[R][4];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    wide4(*reinterpret_cast<const uint2 *>(p.q + ((size_t)min(row0 + r, p.rows - 1) * p.H + h) * AP_D + lane * 4), qf[r]);
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[r][j] = 0.f;
  }
  const int S = limit(R - 1), S_mine = limit(my_row);
  const size_t at = (size_t)h * AP_D + lane * 4;
  // the four keys from s0 on are asked for while the four before them are worked on; beyond the last one in use: that one again
  auto ask = [&](const __half *base, int s0, uint2 (&v)[KEYS]) {
#pragma unroll
    for (int k = 0; k < KEYS; ++k) v[k] = *reinterpret_cast<const uint2 *>(base + kv_row(p.pages, min(s0 + k, S - 1)) * p.kv_stride + at);
  };
  auto score = [&](const uint2 (&v)[KEYS]) {
    float f[KEYS][4], d[KEYS * R];
#pragma unroll
    for (int k = 0; k < KEYS; ++k) wide4(v[k], f[k]);
#pragma unroll
    for (int i = 0; i < KEYS * R; ++i) {
      const float(&x)[4] = qf[i % R];
      const float(&y)[4] = f[i / R];
      d[i] = x[0] * y[0] + x[1] * y[1] + x[2] * y[2] + x[3] * y[3];
    }
#pragma unroll
    for (int n = KEYS * R / 2, o = 16; n >= 1; n >>= 1, o >>= 1)
#pragma unroll
      for (int i = 0; i < n; ++i) {
        const float keep = lane & o ? d[i + n] : d[i], send = lane & o ? d[i] : d[i + n];
        d[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
    return (d[0] + __shfl_xor_sync(0xffffffffu, d[0], 1)) * p.scale;
  };
  float mx = -CUDART_INF_F, l = 0.f;
  uint2 k_now[KEYS], k_next[KEYS], v_now[KEYS], v_next[KEYS];
  if (S > 0) ask(p.kc, 0, k_next);
  for (int s0 = 0; s0 < S; s0 += KEYS) {
#pragma unroll
    for (int k = 0; k < KEYS; ++k) k_now[k] = k_next[k];
    ask(p.kc, s0 + KEYS, k_next);
    const float t = score(k_now);
    mx = s0 + my_key < S_mine ? fmaxf(mx, t) : mx;
  }
#pragma unroll
  for (int o = 8; o <= 16; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (S > 0) ask(p.kc, 0, k_next), ask(p.vc, 0, v_next);
  for (int s0 = 0; s0 < S; s0 += KEYS) {
#pragma unroll
    for (int k = 0; k < KEYS; ++k) k_now[k] = k_next[k], v_now[k] = v_next[k];
    ask(p.kc, s0 + KEYS, k_next);
    ask(p.vc, s0 + KEYS, v_next);
    const float e = expf(score(k_now) - mx);
    l += s0 + my_key < S_mine ? e : 0.f;
    float f[KEYS][4];
#pragma unroll
    for (int k = 0; k < KEYS; ++k) wide4(v_now[k], f[k]);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int S_r = __shfl_sync(0xffffffffu, S_mine, 2 * r);
#pragma unroll
      for (int k = 0; k < KEYS; ++k) {
        const float er = __shfl_sync(0xffffffffu, e, 8 * k + 2 * r);
        if (s0 + k < S_r) {
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[r][j] = fmaf(er, f[k][j], acc[r][j]);
        }
      }
    }
  }
#pragma unroll
  for (int o = 8; o <= 16; o <<= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const float lr = __shfl_sync(0xffffffffu, l, 2 * r);
    const int S_r = __shfl_sync(0xffffffffu, S_mine, 2 * r);
    if (row0 + r < p.rows) {
      __half *o = p.out + (size_t)(row0 + r) * p.H * AP_D + at;
#pragma unroll
      for (int j = 0; j < 4; ++j) o[j] = __float2half_rn(S_r > 0 ? acc[r][j] / lr : 0.f);
    }
  }
}

__global__ void __launch_bounds__(AP_THREADS, 2) attention_prefill_kernel(AttnPrefillParams p) {
  extern __shared__ unsigned char ap_smem_raw[];
  unsigned char *smem = ap_smem_raw + ((1024u - (ap_smem_u32(ap_smem_raw) & 1023u)) & 1023u);  // swizzle atoms need 1024-byte alignment
  // barriers: full[4], empty[4] (K, K, V, V), s_full[2], p_full[2], o_done
  __shared__ __align__(8) uint64_t bars[2 * AP_STAGES + 5];
  __shared__ uint32_t tmem_s;
  __shared__ int fail_s, bad_s;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int h = blockIdx.x, q0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * AP_BM;
  const int pos0 = *p.pos0;
  auto limit_of = [&](int row) {  // cache rows query row `row` attends to
    const long s = (long)pos0 + 1 + row;
    return (int)(s < 0 ? 0 : s > p.max_seq ? p.max_seq : s);
  };
  const int last_row = min(q0 + AP_BM, p.rows) - 1;
  const int S = limit_of(last_row);  // the most any row of this CTA attends to
  const int tiles = (S + AP_BN - 1) / AP_BN;
  const uint32_t b_full = ap_smem_u32(bars), b_empty = b_full + 8 * AP_STAGES, b_sfull = b_empty + 8 * AP_STAGES, b_pfull = b_sfull + 16, b_odone = b_pfull + 16;

  pdl_launch_dependents();  // the O projection may bring its weights in; it waits for this grid before it reads `out`
  if (tid == 0) {
    for (int i = 0; i < AP_STAGES; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(b_full + 8 * i), "r"(i < 2 ? 32 : 64));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b_empty + 8 * i));
    }
    for (int i = 0; i < 2; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b_sfull + 8 * i));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(b_pfull + 8 * i), "n"(AP_SOFT_WARPS * 32));
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b_odone));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fail_s = bad_s = 0;
  }
  if (warp == AP_MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ap_smem_u32(&tmem_s)), "n"(AP_TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  } else if (warp < AP_SOFT_WARPS) {
    // Q tile: 16-byte chunk c of row r to half c / 8, chunk position (c % 8) ^ (r % 8)
    const int c = tid & 15;
#pragma unroll 4
    for (int r = tid >> 4; r < AP_BM; r += AP_SOFT_WARPS * 32 / 16) {
      uint4 v = make_uint4(0, 0, 0, 0);
      if (q0 + r < p.rows) v = *reinterpret_cast<const uint4 *>(p.q + ((size_t)(q0 + r) * p.H + h) * AP_D + c * 8);
      *reinterpret_cast<uint4 *>(smem + (c >> 3) * (AP_Q_BYTES / 2) + r * 128 + (((c & 7) ^ (r & 7)) << 4)) = v;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_s, 0), tmem_o = tmem + 2 * AP_BN;
  const uint32_t ring = ap_smem_u32(smem) + AP_Q_BYTES;

  if (warp >= AP_SOFT_WARPS && warp < AP_MMA_WARP) {
    // ---- K tiles (one warp) and V tiles (two), two stages each.  A tile is announced once the next one has been
    // asked for, that is, once the MMAs of the tile before it are complete.
    auto load = [&](auto is_v) {
      constexpr bool V = decltype(is_v)::value;
      constexpr int STEP = V ? 4 : 2;  // rows per pass: 16 threads bring a row in
      const int t = tid - (AP_SOFT_WARPS + (V ? 1 : 0)) * 32, c = t & 15, r0 = t >> 4;
      const __half *src = (V ? p.vc : p.kc) + (size_t)h * AP_D + c * 8;
      const uint32_t dst0 = (uint32_t)((V ? 2 : 0) * AP_STAGE_BYTES + (c >> 3) * (AP_STAGE_BYTES / 2) + r0 * 128);
      const uint32_t full = b_full + (V ? 16 : 0), empty = b_empty + (V ? 16 : 0);
      const uint32_t sw = (uint32_t)(((c & 7) ^ r0) << 4);  // chunk position in row r0; that of row r0 + n is sw ^ (n % 8) * 16 for n a multiple of STEP
      bool good = true;
      auto landed = [&](int j) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        ap_arrive(full + 8 * (j & 1));
        if (V) {  // then look at what this thread brought in: nobody overwrites it before this thread does
          const unsigned char *sv = smem + AP_Q_BYTES + (j & 1) * AP_STAGE_BYTES + dst0;
          __half2 m = u2h2(0u);
#pragma unroll
          for (int n = 0; n < AP_BN; n += STEP) {
            const uint4 v = *reinterpret_cast<const uint4 *>(sv + n * 128 + (sw ^ ((n & 7) << 4)));
            m = __hmax2_nan(m, __hmax2_nan(__hmax2_nan(__habs2(u2h2(v.x)), __habs2(u2h2(v.y))), __hmax2_nan(__habs2(u2h2(v.z)), __habs2(u2h2(v.w)))));
          }
          const float2 f = __half22float2(m);
          if (!(f.x < CUDART_INF_F && f.y < CUDART_INF_F)) bad_s = 1;
        }
      };
      for (int j = 0; j < tiles; ++j) {
        if (j >= 2 && !__all_sync(0xffffffffu, ap_wait(empty + 8 * (j & 1), ((j >> 1) - 1) & 1))) {
          good = false;
          break;
        }
        const uint32_t dst = ring + (j & 1) * AP_STAGE_BYTES + dst0;
        const int s0 = j * AP_BN + r0;
        if (p.pages.table == nullptr && (j + 1) * AP_BN <= S) {  // a whole tile of consecutive rows
          const __half *g = src + (size_t)s0 * p.kv_stride;
#pragma unroll
          for (int n = 0; n < AP_BN; n += STEP, g += STEP * p.kv_stride)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + n * 128 + (sw ^ ((n & 7) << 4))), "l"(g) : "memory");
        } else {
#pragma unroll 4
          for (int n = 0; n < AP_BN; n += STEP) {
            const bool in = s0 + n < S;  // rows beyond the cache rows in use: zeros
            const __half *g = src + kv_row(p.pages, in ? s0 + n : 0) * p.kv_stride;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + n * 128 + (sw ^ ((n & 7) << 4))), "l"(g), "r"(in ? 16 : 0) : "memory");
          }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (j > 0) {
          asm volatile("cp.async.wait_group 1;" ::: "memory");
          landed(j - 1);
        }
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
      if (good && tiles > 0) landed(tiles - 1);
      if (!good) fail_s = 1;
    };
    if (warp == AP_SOFT_WARPS) load(std::false_type{});
    else load(std::true_type{});
  } else if (warp == AP_MMA_WARP) {
    // ---- MMA issue.  Order S0, S1, O0, S2, O1, ...: the scores of the next tile are ready while P of this one is made.
    // S of tile j + 1 overwrites P of tile j - 1.  Only MMAs of one shape are certain to execute in order, so S waits
    // until the MMAs that read that P are complete (which they are by the time the softmax of tile j is under way).
    constexpr uint32_t ID_S = (1u << 4) | ((uint32_t)(AP_BN >> 3) << 17) | ((uint32_t)(AP_BM >> 4) << 24);
    constexpr uint32_t ID_O = (1u << 4) | (1u << 16) | ((uint32_t)(AP_D >> 3) << 17) | ((uint32_t)(AP_BM >> 4) << 24);  // bit 16: B is MN-major
    const uint32_t q_s = ap_smem_u32(smem);
    bool good = true;
    auto scores = [&](int j) {
      const int slot = j & 1;
      good = __all_sync(0xffffffffu, ap_wait(b_full + 8 * slot, (j >> 1) & 1));
      if (!good) return;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint64_t a0 = ap_desc(q_s, 16), b0 = ap_desc(ring + slot * AP_STAGE_BYTES, 16);
#pragma unroll
      for (int k = 0; k < 8; ++k)  // 16 dims further: 32 B inside a swizzled row, four steps per 64-dim half
        ap_mma_ss(tmem + slot * AP_BN, a0 + (uint64_t)((k >> 2) * (AP_Q_BYTES / 2 / 16) + (k & 3) * 2), b0 + (uint64_t)((k >> 2) * (AP_STAGE_BYTES / 2 / 16) + (k & 3) * 2),
                  ID_S, k > 0);
      ap_commit(b_empty + 8 * slot);
      ap_commit(b_sfull + 8 * slot);
    };
    if (tiles > 0) scores(0);
    for (int j = 0; j < tiles && good; ++j) {
      if (j > 0) good = __all_sync(0xffffffffu, ap_wait(b_odone, (j - 1) & 1));
      if (good && j + 1 < tiles) scores(j + 1);
      const int slot = j & 1;
      good = good && __all_sync(0xffffffffu, ap_wait(b_full + 16 + 8 * slot, (j >> 1) & 1) && ap_wait(b_pfull + 8 * slot, (j >> 1) & 1));
      if (!good) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint64_t b0 = ap_desc(ring + (2 + slot) * AP_STAGE_BYTES, AP_STAGE_BYTES / 2);
      const uint32_t a0 = tmem + slot * AP_BN;
#pragma unroll
      for (int k = 0; k < 8; ++k)  // 4 steps of 16 keys (2 swizzle atoms of V) with P hi, the same with P lo
        ap_mma_ts(tmem_o, a0 + k * 8, b0 + (uint64_t)((k & 3) * (2048 / 16)), ID_O, (j > 0 || k > 0));
      ap_commit(b_empty + 16 + 8 * slot);
      ap_commit(b_odone);
    }
    if (!good) fail_s = 1;
  } else {
    // ---- softmax: thread = query row q0 + tid -----------------------------------------------------------------
    const uint32_t lanes = (uint32_t)(warp * 32) << 16;
    const int limit = min(limit_of(min(q0 + tid, last_row)), S);
    const float c = p.scale * 1.4426950408889634f;
    float m = -CUDART_INF_F, l = 0.f;
    bool good = true;
    for (int j = 0; j < tiles; ++j) {
      const uint32_t ts = tmem + (j & 1) * AP_BN + lanes;
      if (!__all_sync(0xffffffffu, ap_wait(b_sfull + 8 * (j & 1), (j >> 1) & 1))) {
        good = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      uint32_t r0[32], r1[32];
      ap_ld32(ts, r0);
      ap_ld32(ts + 32, r1);
      ap_wait_ld();
      float mx = -CUDART_INF_F;
      const int left = limit - j * AP_BN;  // keys of this tile the row attends to
      if (__all_sync(0xffffffffu, left >= AP_BN)) {
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const float a = __uint_as_float(r0[i]) * c, b = __uint_as_float(r1[i]) * c;
          mx = fmaxf(mx, fmaxf(a, b));
          r0[i] = __float_as_uint(a);
          r1[i] = __float_as_uint(b);
        }
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const float a = i < left ? __uint_as_float(r0[i]) * c : -CUDART_INF_F, b = i + 32 < left ? __uint_as_float(r1[i]) * c : -CUDART_INF_F;
          mx = fmaxf(mx, fmaxf(a, b));
          r0[i] = __float_as_uint(a);
          r1[i] = __float_as_uint(b);
        }
      }
      const bool raise = j == 0 || mx > m + AP_RAISE;
      float f = 1.f;
      if (raise) {
        f = j == 0 ? 0.f : ap_ex2(m - mx);
        m = mx;
        l *= f;
      }
      // rescale O: after the MMAs of the tile before (those of the tile before that are complete: these scores waited for them)
      if (j > 0 && __any_sync(0xffffffffu, raise)) {
        if (!__all_sync(0xffffffffu, ap_wait(b_odone, (j - 1) & 1))) {
          good = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
        for (int d = 0; d < AP_D; d += 16) {
          uint32_t o[16];
          asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                       : AP_R16(o, 0)
                       : "r"(tmem_o + lanes + d)
                       : "memory");
          ap_wait_ld();
#pragma unroll
          for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * f);
          ap_st16(tmem_o + lanes + d, o);
        }
      }
      const float shift = m == -CUDART_INF_F ? 0.f : m - AP_P_EXP;  // no finite score yet: every p is 0
      float l0 = 0.f, l1 = 0.f;
      auto put = [&](const uint32_t (&r)[32], int col) {  // 32 probabilities -> 16 registers of hi pairs, 16 of lo pairs
        uint32_t hi[16], lo[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float a = ap_ex2(__uint_as_float(r[2 * i]) - shift), b = ap_ex2(__uint_as_float(r[2 * i + 1]) - shift);
          l0 += a;
          l1 += b;
          const __half2 hh = __floats2half2_rn(a, b);
          const float2 hf = __half22float2(hh);
          hi[i] = h22u(hh);
          lo[i] = h22u(__floats2half2_rn(a - hf.x, b - hf.y));
        }
        ap_st16(ts + col, hi);
        ap_st16(ts + 32 + col, lo);
      };
      put(r0, 0);
      put(r1, 16);
      l += l0 + l1;
      ap_wait_st();
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      ap_arrive(b_pfull + 8 * (j & 1));
    }
    // ---- O / l, rounded, parked row by row in the idle Q and ring memory, then stored as whole 256-byte rows
    // the last tile but one first: its MMAs need not be complete yet, and a barrier two phases behind looks complete
    if (good && tiles > 1) good = __all_sync(0xffffffffu, ap_wait(b_odone, (tiles - 2) & 1));
    if (good && tiles > 0) good = __all_sync(0xffffffffu, ap_wait(b_odone, (tiles - 1) & 1));
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (!good) {
      fail_s = 1;
    } else {
      unsigned char *park = smem + (size_t)warp * 32 * AP_ROWB;
      if (tiles > 0) {
#pragma unroll 1
        for (int d = 0; d < AP_D; d += 32) {
          uint32_t o[32];
          ap_ld32(tmem_o + lanes + d, o);
          ap_wait_ld();
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            uint4 v;
            uint32_t u[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float a = __uint_as_float(o[8 * i + 2 * e]), b = __uint_as_float(o[8 * i + 2 * e + 1]);
              u[e] = limit > 0 ? h22u(__floats2half2_rn(a / l, b / l)) : 0u;
            }
            v = make_uint4(u[0], u[1], u[2], u[3]);
            *reinterpret_cast<uint4 *>(park + lane * AP_ROWB + (d + 8 * i) * 2) = v;
          }
        }
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) *reinterpret_cast<uint4 *>(park + lane * AP_ROWB + i * 16) = make_uint4(0, 0, 0, 0);
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == AP_MMA_WARP) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(AP_TMEM_COLS) : "memory");
  // Nothing is stored before it is known which of the two results it is: `out` may be `q`, which the other one reads again.
  if (fail_s) {
    if (tid == 0) atomicExch(p.status, 700);  // site 700: a wait of the prompt attention ran out
  } else if (bad_s) {
    for (int r = warp * 4; r < AP_BM && q0 + r < p.rows; r += AP_THREADS / 32 * 4) attend_rows(p, h, q0 + r, pos0);
  } else if (warp < AP_SOFT_WARPS) {
    const unsigned char *park = smem + (size_t)warp * 32 * AP_ROWB;
    const int piece = lane & 15;
#pragma unroll 4
    for (int rr = 0; rr < 32; rr += 2) {
      const int rl = rr + (lane >> 4), row = q0 + warp * 32 + rl;
      const uint4 v = *reinterpret_cast<const uint4 *>(park + rl * AP_ROWB + piece * 16);
      if (row < p.rows) *reinterpret_cast<uint4 *>(p.out + ((size_t)row * p.H + h) * AP_D + piece * 8) = v;
    }
  }
}

int attention_prefill_launch(const void *q, const void *kc, const void *vc, void *out, const int32_t *pos0_dev, int rows, int max_seq, int H, long kv_stride,
                             float scale, KvPages pages, cudaStream_t stream) {
  int *status = kernel_error_ptr();
  AB200_REQUIRE(status != nullptr, "attention_prefill: cannot resolve the status word");
  AttnPrefillParams p{(const __half *)q, (const __half *)kc, (const __half *)vc, (__half *)out, pos0_dev, rows, max_seq, H, kv_stride, scale, pages, status};
  AB200_CUDA(cudaFuncSetAttribute(attention_prefill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, AP_SMEM));
  attention_prefill_kernel<<<dim3(H, (rows + AP_BM - 1) / AP_BM), AP_THREADS, AP_SMEM, stream>>>(p);
  AB200_CHECK_LAUNCH("attention_prefill");
  return AB200_OK;
}

}  // namespace ab200
