// Interpreter for element-wise Antares-IR statements outside the named operator family
// (`out[axes] = expr` with every tensor indexed by the output's axes): the expression arrives as
// a small postfix program (antares_b200/ir.py::compile_elementwise), is turned into the accumulator machine's
// instructions (vm_machine.cuh) and travels in the kernel parameters; every thread evaluates it for
// eight elements at a time in fp32.  The reference generates a kernel per expression
// (lang/einstein_v2.py:297-578 -> antares/default_codegen.py); here one kernel serves them all, so no
// compiler is needed at run time.
//
// Inputs and output may be fp16 or fp32.  Where the pointers allow, a thread's eight elements are one aligned chunk
// (16-byte accesses); otherwise they lie THREADS apart, so that a warp's scalar accesses stay contiguous.
// Bound by instruction issue: tanh-GELU of 8.4 M fp16 values takes 29 us (51 with one element per decode), about half of it tanhf.
#include "vm_machine.cuh"

namespace ab200 {

constexpr int VM_MAX_INPUTS = 8;
constexpr int VM_THREADS = 128;

struct VmProgram {  // what every launch reads comes first: a small launch waits for each line of parameters it touches
  size_t n;
  int n_code;
  unsigned char out_f16, vec_ok, in_f16[VM_MAX_INPUTS];
  VmCode code[VM_MAX_OPS];
  void *out;
  const void *in[VM_MAX_INPUTS];
  float cst[VM_MAX_CONSTS];
};

__global__ void __launch_bounds__(VM_THREADS) eltwise_vm_kernel(const __grid_constant__ VmProgram p) {
  extern __shared__ float4 vm_stack[];
  const bool vec_ok = p.vec_ok;
  constexpr size_t BLOCK = (size_t)VM_THREADS * VM_E;
  for (size_t base = blockIdx.x * BLOCK; base < p.n; base += gridDim.x * BLOCK) {
    const size_t i = vec_ok ? base + threadIdx.x * VM_E : base + threadIdx.x;
    const unsigned step = vec_ok ? 1 : VM_THREADS;
    const size_t left = i < p.n ? (p.n - i + step - 1) / step : 0;
    const int count = left < VM_E ? (int)left : VM_E;
    const bool vec = vec_ok && count == VM_E;
    float first[VM_E], t[VM_E];
    vm_load(p.in[0], p.in_f16[0], i, step, count, vec, first);
    vm_run<VM_E>(p.code, p.n_code, vm_stack + threadIdx.x, VM_THREADS, t, first, [&](unsigned, unsigned arg) { return p.cst[arg]; },
                 [&](unsigned, unsigned arg, float(&b)[VM_E]) { vm_load(p.in[arg], p.in_f16[arg], i, step, count, vec, b); });
    vm_store(p.out, p.out_f16, i, step, count, vec, t);
  }
}

}  // namespace ab200

using namespace ab200;

// ops / args: the postfix program (n_ops entries, codes as in VmOp); consts: fp32 constants; inputs:
// device pointers with their dtypes (AB200_F16 / AB200_F32); every input and the output hold n elements.
extern "C" int ab200_eltwise_vm(const unsigned char *ops_host, const unsigned char *args_host, int n_ops, const float *consts_host, int n_consts,
                                const void *const *inputs_host, const int *in_dtypes_host, int n_inputs, void *out, int out_dtype, size_t n,
                                void *stream) {
  clear_error();
  AB200_REQUIRE(ops_host && args_host && inputs_host && in_dtypes_host && out, "eltwise_vm: null pointer");
  AB200_REQUIRE(n_ops >= 1 && n_ops <= VM_MAX_OPS && n_consts >= 0 && n_consts <= VM_MAX_CONSTS && n_inputs >= 1 && n_inputs <= VM_MAX_INPUTS,
                "eltwise_vm: program of %d ops, %d constants, %d inputs exceeds the interpreter (max %d / %d / %d)", n_ops, n_consts, n_inputs,
                VM_MAX_OPS, VM_MAX_CONSTS, VM_MAX_INPUTS);
  AB200_REQUIRE(n_consts == 0 || consts_host != nullptr, "eltwise_vm: constants missing");
  if (n == 0) return AB200_OK;
  VmProgram p{};
  int depth = 0, vec_ok = 1;
  for (int k = 0; k < n_ops; ++k) {  // validate on the host: the kernel trusts the program
    const int op = ops_host[k], arg = args_host[k];
    AB200_REQUIRE(op <= VM_SIGMOID, "eltwise_vm: unknown operation code %d", op);
    if (op == VM_IN) {
      AB200_REQUIRE(arg < n_inputs, "eltwise_vm: input index %d out of range", arg);
      ++depth;
    } else if (op == VM_CONST) {
      AB200_REQUIRE(arg < n_consts, "eltwise_vm: constant index %d out of range", arg);
      ++depth;
    } else if (op <= VM_DIV || (op >= VM_MAX && op <= VM_POW)) {
      AB200_REQUIRE(depth >= 2, "eltwise_vm: stack underflow at operation %d", k);
      --depth;
    } else {
      AB200_REQUIRE(depth >= 1, "eltwise_vm: stack underflow at operation %d", k);
    }
    AB200_REQUIRE(depth <= VM_MAX_STACK, "eltwise_vm: expression needs more than %d stack slots", VM_MAX_STACK);
  }
  AB200_REQUIRE(depth == 1, "eltwise_vm: the program leaves %d values on the stack", depth);
  for (int j = 0; j < n_consts; ++j) p.cst[j] = consts_host[j];
  for (int j = 0; j < n_inputs; ++j) {
    AB200_REQUIRE(inputs_host[j] != nullptr && (in_dtypes_host[j] == AB200_F16 || in_dtypes_host[j] == AB200_F32), "eltwise_vm: bad input %d", j);
    p.in[j] = inputs_host[j];
    p.in_f16[j] = in_dtypes_host[j] == AB200_F16;
    if (!aligned16(inputs_host[j])) vec_ok = 0;
  }
  AB200_REQUIRE(out_dtype == AB200_F16 || out_dtype == AB200_F32, "eltwise_vm: bad output dtype %d", out_dtype);
  if (!aligned16(out)) vec_ok = 0;
  p.vec_ok = (unsigned char)vec_ok;
  p.out = out;
  p.out_f16 = out_dtype == AB200_F16;
  p.n = n;
  int stack = 0;
  p.n_code = vm_translate(ops_host, args_host, n_ops, p.code, &stack);
  const size_t per_block = (size_t)VM_THREADS * VM_E;
  size_t blocks = (n + per_block - 1) / per_block;
  const size_t cap = (size_t)sm_count() * 64;
  if (blocks > cap) blocks = cap;
  eltwise_vm_kernel<<<(unsigned)blocks, VM_THREADS, stack * per_block * sizeof(float), (cudaStream_t)stream>>>(p);
  AB200_CHECK_LAUNCH("eltwise_vm");
  return AB200_OK;
}
