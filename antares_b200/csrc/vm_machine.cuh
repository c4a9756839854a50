// The machine that runs generic IR expressions (element-wise statements, row programs): a small accumulator
// machine, interpreted on the device for VM_E elements of a thread at a time.
//
// Expressions arrive as postfix programs (antares_b200/ir.py).  Interpreting those directly spends most of its
// instructions on moving operands and on decoding, so the host first turns a program into instructions with one
// operand: top = top OP operand, where the operand is a scalar (constant, row result, row length), a vector
// (an element of an input), or the value underneath.  Only a subexpression whose both sides are compound needs the
// stack; tanh-GELU's 20 postfix operations become 12 instructions with one push.  Every instruction is decoded once
// for VM_E elements, and the expression's first input stays in registers for the whole program.  In a row program the
// subexpressions that only read row results, constants and the row length (a mean, the reciprocal of a deviation) are
// taken out and run once per row.  The arithmetic is that of the postfix program, operation by operation, so results
// are bit for bit what a plain evaluation gives.
#pragma once
#include "common.cuh"

namespace ab200 {

constexpr int VM_MAX_OPS = 48, VM_MAX_CONSTS = 16, VM_MAX_STACK = 8;
constexpr int VM_E = 8;

// operation codes of the postfix programs; VM_ROW.. are operands that only row programs have
enum VmOp : unsigned {
  VM_IN = 0, VM_CONST, VM_ADD, VM_SUB, VM_MUL, VM_DIV, VM_NEG, VM_EXP, VM_LOG, VM_SQRT, VM_RSQRT, VM_TANH, VM_ERF, VM_SIN, VM_COS,
  VM_ABS, VM_FLOOR, VM_CEIL, VM_MAX, VM_MIN, VM_POW, VM_SIGMOID, VM_ROW, VM_COL, VM_COLLEN,
  VM_RSUB, VM_RDIV, VM_RPOW, VM_LOAD  // operand OP top; top = operand
};
__host__ __device__ constexpr bool vm_is_leaf(unsigned op) { return op <= VM_CONST || (op >= VM_ROW && op <= VM_COLLEN); }
__host__ __device__ constexpr bool vm_is_binary(unsigned op) { return (op >= VM_ADD && op <= VM_DIV) || (op >= VM_MAX && op <= VM_POW); }

// an instruction: operation | operand kind << 5 | operand index << 8 | push << 12.  Half words: a small launch waits for every
// line of its parameters that it touches.
typedef unsigned short VmCode;
enum { VM_K_NONE = 0, VM_K_POP, VM_K_CONST, VM_K_IN, VM_K_ROW, VM_K_COL, VM_K_COLLEN, VM_K_TEMP };
constexpr unsigned VM_PUSH = 1u << 12;

constexpr int VM_MAX_TEMPS = 4;
static_assert(VM_LOAD < 32 && VM_K_TEMP < 8 && VM_MAX_CONSTS <= 16 && VM_MAX_TEMPS <= 16, "an instruction's fields");

// Programs that run once per row: temp i is the value of pre[start[i]] .. pre[start[i + 1]).
struct VmTemps {
  VmCode code[VM_MAX_OPS];
  unsigned char start[VM_MAX_TEMPS + 1];
  unsigned char n;
};

// Host: a valid postfix program -> instructions; returns how many, and the deepest stack in *depth.  temps: where the
// subexpressions without vector operands go (nullptr: they stay).
inline int vm_translate(const unsigned char *op, const unsigned char *arg, int n, VmCode *code, int *depth, VmTemps *temps = nullptr) {
  int start[VM_MAX_OPS], temp[VM_MAX_OPS], top_of[VM_MAX_OPS], sp = 0;  // start[k]: first operation of the subexpression that k closes
  bool scalar[VM_MAX_OPS];
  for (int k = 0; k < n; ++k) {
    temp[k] = -1;
    if (vm_is_leaf(op[k])) {
      start[k] = k;
      scalar[k] = op[k] != VM_IN && op[k] != VM_COL;
      top_of[sp++] = k;
    } else if (vm_is_binary(op[k])) {
      start[k] = start[top_of[sp - 2]];
      scalar[k] = scalar[top_of[sp - 2]] && scalar[k - 1];
      top_of[--sp - 1] = k;
    } else {
      start[k] = start[top_of[sp - 1]];
      scalar[k] = scalar[k - 1];
      top_of[sp - 1] = k;
    }
  }
  struct Emit {
    const unsigned char *op, *arg;
    const int *start, *temp;
    VmCode *code;
    int n, live, deepest;
    bool simple(int k) const { return vm_is_leaf(op[k]) || temp[k] >= 0; }
    unsigned operand(int k) const {
      if (temp[k] >= 0) return VM_K_TEMP << 5 | (unsigned)temp[k] << 8;
      const unsigned kind = op[k] == VM_IN ? VM_K_IN : op[k] == VM_CONST ? VM_K_CONST : op[k] == VM_ROW ? VM_K_ROW : op[k] == VM_COL ? VM_K_COL : VM_K_COLLEN;
      return kind << 5 | (arg[k] & 15u) << 8;
    }
    static unsigned reversed(unsigned o) { return o == VM_SUB ? VM_RSUB : o == VM_DIV ? VM_RDIV : o == VM_POW ? VM_RPOW : o; }
    void eval(int k, bool push) {  // push: the value in `top` is needed later, save it before the first load
      if (simple(k)) {
        if (push && ++live > deepest) deepest = live;
        code[n++] = (VmCode)((unsigned)VM_LOAD | operand(k) | (push ? VM_PUSH : 0u));
      } else if (!vm_is_binary(op[k])) {
        eval(k - 1, push);
        code[n++] = op[k];
      } else {
        const int r = k - 1, l = start[r] - 1;
        if (simple(r)) {
          eval(l, push);
          code[n++] = (VmCode)(op[k] | operand(r));
        } else if (simple(l)) {
          eval(r, push);
          code[n++] = (VmCode)(reversed(op[k]) | operand(l));
        } else {
          eval(l, push);
          eval(r, true);
          --live;
          code[n++] = (VmCode)(reversed(op[k]) | (unsigned)VM_K_POP << 5);
        }
      }
    }
  };
  *depth = 0;
  if (temps) {
    temps->n = temps->start[0] = 0;
    for (int k = n - 1; k >= 0; --k) {  // from the end: a subexpression comes before its parts
      if (!scalar[k] || vm_is_leaf(op[k]) || temps->n == VM_MAX_TEMPS) continue;
      int same = -1;  // the same text computed already
      for (int t = n - 1; t > k && same < 0; --t)
        if (temp[t] >= 0 && t - start[t] == k - start[k]) {
          same = t;
          for (int i = 0; i <= k - start[k] && same >= 0; ++i)
            if (op[t - i] != op[k - i] || (vm_is_leaf(op[k - i]) && arg[t - i] != arg[k - i])) same = -1;
        }
      if (same >= 0) {
        temp[k] = temp[same];
      } else {
        Emit e{op, arg, start, temp, temps->code, temps->start[temps->n], 0, 0};
        e.eval(k, false);
        if (e.deepest > *depth) *depth = e.deepest;
        temp[k] = temps->n++;
        temps->start[temps->n] = (unsigned char)e.n;
      }
      k = start[k];  // its parts are done with
    }
  }
  Emit e{op, arg, start, temp, code, 0, 0, 0};
  e.eval(n - 1, false);
  if (e.deepest > *depth) *depth = e.deepest;
  return e.n;
}

// E elements (VM_E or 1) of an fp16 / fp32 tensor: element j is i + j * step.  vec: step is 1 and the elements are one
// aligned chunk; otherwise the first `count` elements exist and the others read as 0.
template <int E>
__device__ __forceinline__ void vm_load(const void *p, bool f16, size_t i, unsigned step, int count, bool vec, float (&v)[E]) {
  if (E == VM_E && vec) {
    if (f16) {
#pragma unroll
      for (int c = 0; c < E / 8; ++c) {
        const uint4 h = reinterpret_cast<const uint4 *>(reinterpret_cast<const __half *>(p) + i)[c];
        const uint32_t u[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = __half22float2(u2h2(u[j]));
          v[8 * c + 2 * j] = f.x;
          v[8 * c + 2 * j + 1] = f.y;
        }
      }
    } else {
#pragma unroll
      for (int c = 0; c < E / 4; ++c) {
        const float4 a = reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(p) + i)[c];
        v[4 * c] = a.x, v[4 * c + 1] = a.y, v[4 * c + 2] = a.z, v[4 * c + 3] = a.w;
      }
    }
  } else if (f16) {
#pragma unroll
    for (int j = 0; j < E; ++j) v[j] = j < count ? __half2float(reinterpret_cast<const __half *>(p)[i + (size_t)j * step]) : 0.f;
  } else {
#pragma unroll
    for (int j = 0; j < E; ++j) v[j] = j < count ? reinterpret_cast<const float *>(p)[i + (size_t)j * step] : 0.f;
  }
}
template <int E>
__device__ __forceinline__ void vm_store(void *p, bool f16, size_t i, unsigned step, int count, bool vec, const float (&v)[E]) {
  if (E == VM_E && vec) {
    if (f16) {
      uint4 *o = reinterpret_cast<uint4 *>(reinterpret_cast<__half *>(p) + i);
#pragma unroll
      for (int c = 0; c < E / 8; ++c) {
        const float *f = v + 8 * c;
        o[c] = make_uint4(h22u(__floats2half2_rn(f[0], f[1])), h22u(__floats2half2_rn(f[2], f[3])), h22u(__floats2half2_rn(f[4], f[5])), h22u(__floats2half2_rn(f[6], f[7])));
      }
    } else {
      float4 *o = reinterpret_cast<float4 *>(reinterpret_cast<float *>(p) + i);
#pragma unroll
      for (int c = 0; c < E / 4; ++c) o[c] = make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
    }
  } else {
#pragma unroll
    for (int j = 0; j < E; ++j)
      if (j < count) {
        if (f16) reinterpret_cast<__half *>(p)[i + (size_t)j * step] = __float2half_rn(v[j]);
        else reinterpret_cast<float *>(p)[i + (size_t)j * step] = v[j];
      }
  }
}

// Runs n instructions for EN elements; scalar(kind, index) and vector(kind, index, b) fetch operands, `first` is the
// first input.  stack: this thread's column of [slot][VM_E / 4][threads] float4.
// Decoding is a chain of dependent loads and branches, which is what a short program spends its time on: the next word is
// read ahead, and the commonest operations are tested before the jump table, with a scalar or the first input without a
// copy of the operand.
template <int EN, class Scalar, class Vector>
__device__ __forceinline__ void vm_run(const VmCode *code, int n, float4 *stack, unsigned threads, float (&t)[EN], const float (&first)[EN], Scalar scalar,
                                       Vector vector) {
  constexpr int QUADS = (EN + 3) / 4;
#define VM_EACH(expr)                             \
  {                                               \
    _Pragma("unroll") for (int j = 0; j < EN; ++j) { \
      const float x = t[j], y = b[j];             \
      (void)x, (void)y;                           \
      t[j] = (expr);                              \
    }                                             \
  }                                               \
  break
#define VM_COMMON(y)                                                        \
  if (o == VM_MUL) {                                                        \
    _Pragma("unroll") for (int j = 0; j < EN; ++j) t[j] = t[j] * (y);       \
    continue;                                                               \
  }                                                                         \
  if (o == VM_ADD) {                                                        \
    _Pragma("unroll") for (int j = 0; j < EN; ++j) t[j] = t[j] + (y);       \
    continue;                                                               \
  }                                                                         \
  if (o == VM_SUB) {                                                        \
    _Pragma("unroll") for (int j = 0; j < EN; ++j) t[j] = t[j] - (y);       \
    continue;                                                               \
  }                                                                         \
  if (o == VM_LOAD) {                                                       \
    _Pragma("unroll") for (int j = 0; j < EN; ++j) t[j] = (y);              \
    continue;                                                               \
  }
  unsigned ahead = code[0];
  for (int k = 0; k < n; ++k) {
    const unsigned w = ahead, o = w & 31u, kind = (w >> 5) & 7u, arg = (w >> 8) & 15u;
    if (k + 1 < n) ahead = code[k + 1];
    float b[EN];
    if (w & VM_PUSH) {
#pragma unroll
      for (int i = 0; i < QUADS; ++i) stack[i * threads] = EN == 1 ? make_float4(t[0], 0.f, 0.f, 0.f) : make_float4(t[4 * i], t[4 * i + 1], t[4 * i + 2], t[4 * i + 3]);
      stack += VM_E / 4 * threads;
    }
    if (kind == VM_K_IN && arg == 0) {
      VM_COMMON(first[j])
#pragma unroll
      for (int j = 0; j < EN; ++j) b[j] = first[j];
    } else if (kind >= VM_K_CONST && kind != VM_K_IN && kind != VM_K_COL) {
      const float c = scalar(kind, arg);
      VM_COMMON(c)
#pragma unroll
      for (int j = 0; j < EN; ++j) b[j] = c;
    } else if (kind == VM_K_POP) {
      stack -= VM_E / 4 * threads;
#pragma unroll
      for (int i = 0; i < QUADS; ++i) {
        const float4 v = stack[i * threads];
        if (EN == 1) b[0] = v.x;
        else b[4 * i] = v.x, b[4 * i + 1] = v.y, b[4 * i + 2] = v.z, b[4 * i + 3] = v.w;
      }
      VM_COMMON(b[j])
    } else if (kind != VM_K_NONE) {
      vector(kind, arg, b);
      VM_COMMON(b[j])
    } else {
#pragma unroll
      for (int j = 0; j < EN; ++j) b[j] = 0.f;
    }
    switch (o) {
      case VM_RSUB: VM_EACH(y - x);
      case VM_DIV: VM_EACH(x / y);
      case VM_RDIV: VM_EACH(y / x);
      case VM_MAX: VM_EACH(fmaxf(x, y));
      case VM_MIN: VM_EACH(fminf(x, y));
      case VM_POW: VM_EACH(powf(x, y));
      case VM_RPOW: VM_EACH(powf(y, x));
      case VM_NEG: VM_EACH(-x);
      case VM_EXP: VM_EACH(expf(x));
      case VM_LOG: VM_EACH(logf(x));
      case VM_SQRT: VM_EACH(sqrtf(x));
      case VM_RSQRT: VM_EACH(rsqrtf(x));
      case VM_TANH: VM_EACH(tanhf(x));
      case VM_ERF: VM_EACH(erff(x));
      case VM_SIN: VM_EACH(sinf(x));
      case VM_COS: VM_EACH(cosf(x));
      case VM_ABS: VM_EACH(fabsf(x));
      case VM_FLOOR: VM_EACH(floorf(x));
      case VM_CEIL: VM_EACH(ceilf(x));
      default: VM_EACH(1.0f / (1.0f + expf(-x)));  // VM_SIGMOID
    }
  }
#undef VM_EACH
#undef VM_COMMON
}

}  // namespace ab200
