// Row-reduction template for multi-statement Antares-IR programs outside the named operator family:
// a chain of row reductions followed by one map statement over the same [rows, cols] index space,
//   t0[N] >=! f0(x[N, C]);  t1[N] +=! f1(x[N, C], t0[N]);  out[N, C] = g(x[N, C], t0[N], t1[N])
// (softmax, AntaresIR.md:226; layernorm, AntaresIR.md:232).  The reference compiles each statement
// into its own generated kernel (lang/einstein_v2.py:297-578 -> antares/default_codegen.py); here one
// kernel runs all stages of a row back to back: every stage's expression is a small postfix program
// (the same operation set as the element-wise interpreter, plus "row value of an earlier stage",
// "column vector" and "number of columns"), run by the accumulator machine of vm_machine.cuh in fp32, eight
// elements of a thread at a time (one in small launches); a reduction stage folds the values of a row with + / max / min (warp shuffles,
// one shared-memory hop, fixed order, so results are bitwise repeatable), the final stage writes the output.  The
// row stays in L1/L2 between stages, so HBM sees each input once.  Instruction issue is what bounds it: layernorm with
// weight and bias over 2048 x 4096 fp16 takes 46 us (296 with one element per decode) for 5 us of traffic.  The block is as wide as the row needs (32 to 256
// threads), so short rows do not leave warps idle.
#include <math_constants.h>

#include "vm_machine.cuh"

namespace ab200 {

constexpr int RV_MAX_STAGES = 4, RV_MAX_MAT = 4, RV_MAX_COL = 4;
constexpr int RV_MAX_THREADS = 256;

enum { RV_MAP = 0, RV_SUM = 1, RV_RMAX = 2, RV_RMIN = 3 };

// All stages' instructions lie one after the other, a stage's temporaries (what it computes once per row) before its own:
// temporary i of stage s is code[begin[s][i]] .. code[begin[s][i + 1]), the stage itself the piece after the last of them.
constexpr int RV_MAX_CODE = RV_MAX_STAGES * 2 * VM_MAX_OPS;
struct RowProgram {
  int rows, cols;
  unsigned char n_stages, vec_ok, out_f16, reduce[RV_MAX_STAGES], n_temps[RV_MAX_STAGES];
  unsigned char mat_f16[RV_MAX_MAT], col_f16[RV_MAX_COL];
  unsigned short begin[RV_MAX_STAGES][VM_MAX_TEMPS + 2];
  const void *mat[RV_MAX_MAT];  // [rows, cols]
  const void *col[RV_MAX_COL];  // [cols]
  void *out;                    // [rows, cols]
  float cst[VM_MAX_CONSTS];
  VmCode code[RV_MAX_CODE];
};

// The instructions are read from the parameters: copied to shared memory first they were slower in every size (layernorm of
// 2048 x 4096 51.7 against 48.4 us), the copy being a start-up of a microsecond or more per block (4096 x 256: 22 against
// 10.8 us; with half-word instructions packed end to end 45.7 and 10.1).
template <int E>
__global__ void __launch_bounds__(RV_MAX_THREADS, 4) rowreduce_vm_kernel(const __grid_constant__ RowProgram p) {
  extern __shared__ float4 vm_stack[];
  // [row parity]: a warp that is a row ahead writes the other half (every row with a reduction has a barrier)
  __shared__ float part[2][RV_MAX_STAGES][RV_MAX_THREADS / 32];
  __shared__ float temp[RV_MAX_STAGES][VM_MAX_TEMPS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned threads = blockDim.x, step = p.vec_ok ? 1 : threads;
  const int per_pass = (int)threads * E;
  int parity = 0;
  for (int row = blockIdx.x; row < p.rows; row += gridDim.x, parity ^= 1) {
    const size_t base = (size_t)row * p.cols;
    float r0 = 0.f, r1 = 0.f, r2 = 0.f;  // results of the reduction stages
    for (int s = 0; s < p.n_stages; ++s) {
      const int kind = p.reduce[s], n_temps = p.n_temps[s];
      const unsigned short *begin = p.begin[s];
      auto scalar = [&](unsigned k, unsigned arg) {
        return k == VM_K_CONST ? p.cst[arg] : k == VM_K_COLLEN ? (float)p.cols : k == VM_K_TEMP ? temp[s][arg] : arg == 0 ? r0 : arg == 1 ? r1 : r2;
      };
      if (n_temps) {  // one warp's work; every warp on its own would spend a third of the row's instructions on it
        if (warp == 0) {
#pragma unroll 1
          for (int i = 0; i < n_temps; ++i) {
            float v[1];
            const float none[1] = {0.f};
            vm_run<1>(p.code + begin[i], begin[i + 1] - begin[i], vm_stack + threadIdx.x, threads, v, none, scalar, [](unsigned, unsigned, float(&)[1]) {});
            if (lane == 0) temp[s][i] = v[0];
          }
        }
        __syncthreads();  // (the reduction before this stage keeps the next row's temporaries away from this row's readers)
      }
      float acc = kind == RV_RMAX ? -CUDART_INF_F : kind == RV_RMIN ? CUDART_INF_F : 0.f;
      for (int c0 = 0; c0 < p.cols; c0 += per_pass) {
        const int c = c0 + (int)threadIdx.x * (p.vec_ok ? E : 1);
        const int left = c < p.cols ? (p.cols - c + (int)step - 1) / (int)step : 0;
        const int count = left < E ? left : E;
        const bool vec = p.vec_ok && count == E;
        float first[E], t[E];
        vm_load(p.mat[0], p.mat_f16[0], base + c, step, count, vec, first);
        vm_run<E>(p.code + begin[n_temps], begin[n_temps + 1] - begin[n_temps], vm_stack + threadIdx.x, threads, t, first, scalar, [&](unsigned k, unsigned arg, float(&b)[E]) {
          if (k == VM_K_COL) vm_load(p.col[arg], p.col_f16[arg], c, step, count, vec, b);
          else vm_load(p.mat[arg], p.mat_f16[arg], base + c, step, count, vec, b);
        });
        if (kind == RV_MAP) {
          vm_store(p.out, p.out_f16, base + c, step, count, vec, t);
        } else if (kind == RV_SUM) {
#pragma unroll
          for (int j = 0; j < E; ++j) acc += j < count ? t[j] : 0.f;
        } else if (kind == RV_RMAX) {
#pragma unroll
          for (int j = 0; j < E; ++j) acc = j < count ? fmaxf(acc, t[j]) : acc;
        } else {
#pragma unroll
          for (int j = 0; j < E; ++j) acc = j < count ? fminf(acc, t[j]) : acc;
        }
      }
      if (kind != RV_MAP) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const float other = __shfl_xor_sync(0xffffffffu, acc, o);
          acc = kind == RV_SUM ? acc + other : kind == RV_RMAX ? fmaxf(acc, other) : fminf(acc, other);
        }
        if (lane == 0) part[parity][s][warp] = acc;
        __syncthreads();
        float r = part[parity][s][0];
        for (int w = 1; w < (int)threads / 32; ++w) {
          const float other = part[parity][s][w];
          r = kind == RV_SUM ? r + other : kind == RV_RMAX ? fmaxf(r, other) : fminf(r, other);
        }
        if (s == 0) r0 = r;
        else if (s == 1) r1 = r;
        else r2 = r;
      }
    }
  }
}

}  // namespace ab200

using namespace ab200;

extern "C" int ab200_rowreduce_vm(const unsigned char *ops_host, const unsigned char *args_host, const int *stage_len_host,
                                  const int *stage_reduce_host, int n_stages, const float *consts_host, int n_consts,
                                  const void *const *mat_inputs_host, const int *mat_dtypes_host, int n_mat, const void *const *col_inputs_host,
                                  const int *col_dtypes_host, int n_col, void *out, int out_dtype, int rows, int cols, void *stream) {
  clear_error();
  AB200_REQUIRE(ops_host && args_host && stage_len_host && stage_reduce_host && out, "rowreduce_vm: null pointer");
  AB200_REQUIRE(n_stages >= 1 && n_stages <= RV_MAX_STAGES, "rowreduce_vm: %d stages (1..%d)", n_stages, RV_MAX_STAGES);
  AB200_REQUIRE(n_consts >= 0 && n_consts <= VM_MAX_CONSTS && (n_consts == 0 || consts_host), "rowreduce_vm: %d constants (at most %d)", n_consts, VM_MAX_CONSTS);
  AB200_REQUIRE(n_mat >= 1 && n_mat <= RV_MAX_MAT && mat_inputs_host && mat_dtypes_host, "rowreduce_vm: %d [rows, cols] inputs (1..%d)", n_mat, RV_MAX_MAT);
  AB200_REQUIRE(n_col >= 0 && n_col <= RV_MAX_COL && (n_col == 0 || (col_inputs_host && col_dtypes_host)), "rowreduce_vm: %d [cols] inputs (at most %d)", n_col, RV_MAX_COL);
  AB200_REQUIRE(rows > 0 && cols > 0, "rowreduce_vm: rows=%d cols=%d", rows, cols);
  AB200_REQUIRE(out_dtype == AB200_F16 || out_dtype == AB200_F32, "rowreduce_vm: output dtype %d", out_dtype);
  RowProgram p = {};
  for (int i = 0; i < n_mat; ++i) {
    AB200_REQUIRE(mat_inputs_host[i] && (mat_dtypes_host[i] == AB200_F16 || mat_dtypes_host[i] == AB200_F32), "rowreduce_vm: bad matrix input %d", i);
    p.mat[i] = mat_inputs_host[i];
    p.mat_f16[i] = mat_dtypes_host[i] == AB200_F16;
  }
  for (int i = 0; i < n_col; ++i) {
    AB200_REQUIRE(col_inputs_host[i] && (col_dtypes_host[i] == AB200_F16 || col_dtypes_host[i] == AB200_F32), "rowreduce_vm: bad column-vector input %d", i);
    p.col[i] = col_inputs_host[i];
    p.col_f16[i] = col_dtypes_host[i] == AB200_F16;
  }
  for (int i = 0; i < n_consts; ++i) p.cst[i] = consts_host[i];
  // validate every stage on the host: operand indices, stack discipline, stage order
  int off = 0, stack = 0, total = 0;
  for (int s = 0; s < n_stages; ++s) {
    const int len = stage_len_host[s], kind = stage_reduce_host[s];
    AB200_REQUIRE(len >= 1 && len <= VM_MAX_OPS, "rowreduce_vm: stage %d has %d operations (1..%d)", s, len, VM_MAX_OPS);
    AB200_REQUIRE(kind >= RV_MAP && kind <= RV_RMIN, "rowreduce_vm: stage %d has reduction kind %d", s, kind);
    AB200_REQUIRE((kind == RV_MAP) == (s == n_stages - 1), "rowreduce_vm: the last stage, and only the last, writes the output");
    int depth = 0;
    for (int k = 0; k < len; ++k) {
      const int op = ops_host[off + k], arg = args_host[off + k];
      AB200_REQUIRE(op <= VM_COLLEN, "rowreduce_vm: unknown operation %d", op);
      if (vm_is_leaf(op)) {
        AB200_REQUIRE(op != VM_IN || arg < n_mat, "rowreduce_vm: matrix input index %d out of range", arg);
        AB200_REQUIRE(op != VM_CONST || arg < n_consts, "rowreduce_vm: constant index %d out of range", arg);
        AB200_REQUIRE(op != VM_ROW || arg < s, "rowreduce_vm: stage %d reads the row value of stage %d, which is not earlier", s, arg);
        AB200_REQUIRE(op != VM_COL || arg < n_col, "rowreduce_vm: column-vector index %d out of range", arg);
        ++depth;
      } else if (vm_is_binary(op)) {
        AB200_REQUIRE(depth >= 2, "rowreduce_vm: stack underflow in stage %d", s);
        --depth;
      } else {
        AB200_REQUIRE(depth >= 1, "rowreduce_vm: stack underflow in stage %d", s);
      }
      AB200_REQUIRE(depth <= VM_MAX_STACK, "rowreduce_vm: stage %d needs a stack deeper than %d", s, VM_MAX_STACK);
    }
    AB200_REQUIRE(depth == 1, "rowreduce_vm: stage %d leaves %d values on the stack", s, depth);
    int depth_used = 0;
    VmTemps temps;
    VmCode code[VM_MAX_OPS];
    const int n = vm_translate(ops_host + off, args_host + off, len, code, &depth_used, &temps);
    p.n_temps[s] = temps.n;
    for (int i = 0; i <= temps.n; ++i) p.begin[s][i] = (unsigned short)(total + temps.start[i]);
    for (int i = 0; i < temps.start[temps.n]; ++i) p.code[total++] = temps.code[i];
    for (int i = 0; i < n; ++i) p.code[total++] = code[i];
    p.begin[s][temps.n + 1] = (unsigned short)total;
    if (depth_used > stack) stack = depth_used;
    p.reduce[s] = (unsigned char)kind;
    off += len;
  }
  p.out = out;
  p.n_stages = n_stages;
  p.out_f16 = out_dtype == AB200_F16;
  p.rows = rows;
  p.cols = cols;
  p.vec_ok = cols % VM_E == 0 && aligned16(out);
  for (int i = 0; i < n_mat; ++i) p.vec_ok = p.vec_ok && aligned16(mat_inputs_host[i]);
  for (int i = 0; i < n_col; ++i) p.vec_ok = p.vec_ok && aligned16(col_inputs_host[i]);
  // One element a thread where the whole launch then fits the SMs at once and a row is one pass: it is the latency of an
  // instruction over eight elements that such a launch would wait for.  Also for rows within a warp, which need no more warps
  // so.  us, layernorm, eight / one: 16 x 33 7.6 / 6.3, 1000 x 128 8.1 / 7.3, 400 x 256 7.0 / 7.0, 1000 x 256 7.2 / 13.4,
  // 2000 x 33 8.8 / 8.2, 4000 x 33 11.6 / 14.2, 20000 x 8 50 / 32.
  int threads = 32;
  while (threads < RV_MAX_THREADS && threads < cols) threads *= 2;
  const bool single = cols <= 32 || (cols <= RV_MAX_THREADS && (long)rows * (threads / 32) <= 28L * sm_count());
  if (!single)
    for (threads = 32; threads < RV_MAX_THREADS && threads * VM_E < cols;) threads *= 2;
  const int cap = sm_count() * (2048 / threads);
  const size_t smem = (size_t)stack * threads * VM_E * sizeof(float);
  // the limit that needs no opting in, 48 KiB, is on this and the static arrays together
  auto kern = single ? rowreduce_vm_kernel<1> : rowreduce_vm_kernel<VM_E>;
  if (smem > 46 * 1024) AB200_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kern<<<rows < cap ? rows : cap, threads, smem, (cudaStream_t)stream>>>(p);
  AB200_CHECK_LAUNCH("rowreduce_vm");
  return AB200_OK;
}
