// sr_notation.cu -- integer tape conversions of the grammar object:
//   * child table of left-packed postfix tapes   (reference get_postfix_children,
//     src/pcfg_cuda.cu:1228-1300, src/pcfg.cpp:957-986)
//   * postfix -> infix token ids with parentheses (reference postfix_to_infix,
//     src/pcfg_cuda.cu:502-701, src/pcfg.cpp:790-826)
//   * prefix -> postfix, postfix -> prefix, prefix -> infix and the parent table of
//     prefix rows (reference src/pcfg_cpu.cpp:637-1064, src/pcfg.cpp:827-955)
// All are bit-exact integer transformations with the reference's error codes and
// stack limits (128 entries, 3 x 128 output tokens).  One thread owns one tape.  Rows of up
// to 128 tokens go through shared memory, a token per byte; the kernels that read 8-byte
// tokens from L1 take longer rows and larger token ids, and the conversions of prefix rows
// that have no byte kernel.
#include <cstdint>

#include "sr_common.cuh"
#include "sr_ops.cuh"

namespace sr {

constexpr int kStackLimit = 128;  // the reference's HARD_MAX_LENGTH

enum NotationCode : int64_t {
  SYM_NEGATIVE = -1,  // a symbol < 0
  SYM_TOO_LARGE = -2, // a symbol >= n_operators
  PARSE_UNEXPECTED_TOKEN = 408,
  PARSE_UNARY_MISSING = 404,
  PARSE_BINARY_MISSING = 405,
  PARSE_STACK_OVERFLOW = 406,
  PARSE_MALFORMED = 407,
  CONV_TOO_LONG = 501,
  CONV_POSTFIX_TOO_LONG = 502,
  CONV_PREFIX_TOO_LONG = 503,
  CONV_STACK_OVERFLOW = 504,
  CONV_UNARY_MISSING = 505,
  CONV_BINARY_MISSING = 506,
  CONV_MULTIPLE_ROOTS = 508,
  CONV_UNEXPECTED_TOKEN = 509,
};

// Symbols must lie in [0, n_operators): -1 / -2 flag the two ways to fail.
__device__ __forceinline__ int64_t symbol_check(const int64_t* row, int64_t M, int64_t n_operators) {
  int64_t flag = 0;
  for (int64_t i = 0; i < M; ++i) {
    const int64_t t = row[i];
    if (t < 0) return SYM_NEGATIVE;
    if (t >= n_operators) flag = SYM_TOO_LARGE;
  }
  return flag;
}

// Unary operators written f(x); the others (^2, ^3, ^4, ^5, ^-1) are written (x)^k.
__device__ __forceinline__ bool functional_style(int64_t op) {
  return (op >= SIN && op <= LOG) || (op >= SQRT && op <= NEG);
}

__global__ void postfix_children_kernel(const int64_t* __restrict__ ops, int64_t B, int64_t M, int64_t n_operators,
                                        int64_t* __restrict__ ch, int64_t* __restrict__ err) {
  const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= B) return;
  const int64_t* row = ops + b * M;
  int64_t* out = ch + b * M * 2;
  for (int64_t i = 0; i < 2 * M; ++i) out[i] = -1;
  int64_t e = symbol_check(row, M, n_operators);
  if (e) {
    err[b] = e;
    return;
  }
  int stack[kStackLimit];
  int sp = 0;
  bool ended = false;
  for (int64_t i = 0; i < M; ++i) {
    const int64_t t = row[i];
    if (t == NO_OP) {
      ended = true;
      continue;
    }
    if (ended) { e = PARSE_UNEXPECTED_TOKEN; break; }
    const int ar = arity_of(t);
    if (ar == 1) {
      if (sp < 1) { e = PARSE_UNARY_MISSING; break; }
      out[i * 2] = stack[--sp];
    } else if (ar == 2) {
      if (sp < 2) { e = PARSE_BINARY_MISSING; break; }
      const int right = stack[--sp];
      const int left = stack[--sp];
      out[i * 2] = left;
      out[i * 2 + 1] = right;
    }
    if (sp >= kStackLimit) { e = PARSE_STACK_OVERFLOW; break; }
    stack[sp++] = (int)i;
  }
  if (!e && sp != 1) e = PARSE_MALFORMED;
  err[b] = e;
}

// The byte kernels: rows of 1..128 tokens with a byte per token, staged through shared memory.
// A CTA reads its 128 rows and writes its results with consecutive threads on consecutive
// elements; each thread then works on its own row in shared memory, where a row takes an odd
// number of words, so that threads at the same position meet no bank conflict.  The checks of
// a whole row go four tokens at a time, and only the tokens before the padding are walked.
// What bounds them: that walk, one thread's chain of shared-memory reads, over the warps that
// shared memory lets reside.
constexpr int kRowThreads = 128;
constexpr uint32_t kByteNegative = 0xff, kByteTooLarge = 0xfe;  // tokens that fail the check

__host__ __device__ __forceinline__ int row_stride(int bytes) { return ((bytes + 3) / 4 | 1) * 4; }

// Element j of a CTA's block of `rows` rows of `width` is element i of row r: f(j, r, i), with
// no division per element.
template <typename F>
__device__ __forceinline__ void each_element(int rows, int width, F f) {
  const int total = rows * width, dr = kRowThreads / width, di = kRowThreads % width;
  int r = threadIdx.x / width, i = threadIdx.x - r * width;
#pragma unroll 8
  for (int j = threadIdx.x; j < total; j += kRowThreads) {
    f(j, r, i);
    r += dr;
    i += di;
    if (i >= width) {
      i -= width;
      ++r;
    }
  }
}

// The CTA's rows as bytes.  kLeaves: only what a token is matters, and every leaf is staged as
// VAR, so that any number of variables fits a byte.
template <bool kLeaves>
__device__ __forceinline__ void stage_rows(const int64_t* __restrict__ src, int rows, int M, int64_t n_operators,
                                           unsigned char* dst) {
  const int stride = row_stride(M);
  if (threadIdx.x < rows) reinterpret_cast<uint32_t*>(dst + threadIdx.x * stride)[(M + 3) / 4 - 1] = 0u;
  __syncthreads();
  each_element(rows, M, [&](int j, int r, int i) {
    const int64_t tok = src[j];
    uint32_t v = (uint32_t)(kLeaves && tok > VAR ? VAR : tok);
    if (tok >= n_operators) v = kByteTooLarge;
    if (tok < 0) v = kByteNegative;
    dst[r * stride + i] = (unsigned char)v;
  });
  __syncthreads();
}

// Checks of a staged row: the symbol check's flag (0: passed), the tokens before the first
// NO_OP, whether a token follows it.
struct RowCheck {
  int64_t flag;
  int len;
  bool follows;
};
__device__ __forceinline__ RowCheck check_row(const unsigned char* row, int M) {
  RowCheck c{0, 0, false};
  const uint32_t* words = reinterpret_cast<const uint32_t*>(row);
  bool ended = false;
  for (int w = 0; w < (M + 3) / 4; ++w) {
    const uint32_t x = words[w];
    if (__vcmpeq4(x, 0xffffffffu)) c.flag = SYM_NEGATIVE;
    else if (__vcmpeq4(x, 0xfefefefeu) && c.flag == 0) c.flag = SYM_TOO_LARGE;
    if (ended) {
      c.follows |= x != 0;
      continue;
    }
    const uint32_t zero = __vcmpeq4(x, 0u);
    if (!zero) {
      c.len += 4;
    } else {
      const int at = (__ffs((int)zero) - 1) & ~7;  // first bit of the first NO_OP
      c.len += at >> 3;
      ended = true;
      c.follows |= (x >> at) != 0;
    }
  }
  return c;
}

// The child table.  A position's left child replaces its token, and its two children are
// written as one 16-byte store (kPairs: the table is aligned for it).  262144 rows of 64
// tokens: 87 us, where 16-bit tokens, checked and walked one by one over the whole row, took
// 235.
template <bool kPairs>
__global__ void __launch_bounds__(kRowThreads) postfix_children_bytes_kernel(
    const int64_t* __restrict__ ops, int64_t B, int M, int64_t n_operators, int64_t* __restrict__ ch,
    int64_t* __restrict__ err) {
  extern __shared__ __align__(16) unsigned char bsm[];
  __shared__ uint8_t reached[kRowThreads];  // positions of each row that the walk came past
  const int t = threadIdx.x, stride = row_stride(M);
  unsigned char* left = bsm + t * stride;  // tokens, then left children
  unsigned char* right = bsm + (kRowThreads + t) * stride;
  unsigned char* stk = bsm + (2 * kRowThreads + t) * stride;
  const int64_t b0 = (int64_t)blockIdx.x * kRowThreads;
  const int rows = (int)(B - b0 < kRowThreads ? B - b0 : kRowThreads);
  stage_rows<true>(ops + b0 * M, rows, M, n_operators, bsm);
  if (t < rows) {
    const RowCheck c = check_row(left, M);
    int64_t e = c.flag;
    int i = 0, sp = 0;
    if (!e) {
      for (; i < c.len; ++i) {
        const int ar = arity_of((int64_t)left[i]);
        unsigned char lc = 0xff, rc = 0xff;
        if (ar == 1) {
          if (sp < 1) { e = PARSE_UNARY_MISSING; break; }
          lc = stk[--sp];
        } else if (ar == 2) {
          if (sp < 2) { e = PARSE_BINARY_MISSING; break; }
          rc = stk[--sp];
          lc = stk[--sp];
        }
        stk[sp++] = (unsigned char)i;  // sp <= i + 1 <= M <= kStackLimit
        left[i] = lc;
        right[i] = rc;
      }
      // the walk goes on into the padding: a token there, or else no single tree
      if (!e && c.follows) e = PARSE_UNEXPECTED_TOKEN;
      if (!e && sp != 1) e = PARSE_MALFORMED;
    }
    reached[t] = (uint8_t)i;
    err[b0 + t] = e;
  }
  __syncthreads();
  int64_t* dst = ch + b0 * 2 * M;
  each_element(rows, M, [&](int j, int r, int i) {
    const unsigned char* p = bsm + r * stride + i;
    long long lc = -1, rc = -1;
    if (i < reached[r]) {
      lc = (signed char)p[0];  // a position is below 128; 0xff: none
      rc = (signed char)p[kRowThreads * stride];
    }
    if (kPairs) {
      reinterpret_cast<longlong2*>(dst)[j] = make_longlong2(lc, rc);
    } else {
      dst[2 * j] = lc;
      dst[2 * j + 1] = rc;
    }
  });
}

// Prefix <-> postfix in place, for token ids below kByteTooLarge.  Both directions emit a leaf at
// once and an operator when its last operand is complete (the stack's bit 7: one operand is
// left to come); from postfix the row is walked and refilled from its right end.  A token is
// emitted at or behind the position that was read, so the row holds both.
// 50001 prefix rows of 48 tokens: 21 us, where a thread per row in global memory took 54.
template <bool kFromPrefix>
__global__ void __launch_bounds__(kRowThreads) reorder_bytes_kernel(const int64_t* __restrict__ in, int64_t B, int M,
                                                                    int64_t n_operators, int64_t* __restrict__ outp,
                                                                    int64_t* __restrict__ err) {
  extern __shared__ __align__(16) unsigned char bsm[];
  __shared__ uint8_t counts[kRowThreads];  // tokens of each output row
  const int t = threadIdx.x, stride = row_stride(M);
  unsigned char* row = bsm + t * stride;
  unsigned char* stk = bsm + (kRowThreads + t) * stride;
  const int64_t b0 = (int64_t)blockIdx.x * kRowThreads;
  const int rows = (int)(B - b0 < kRowThreads ? B - b0 : kRowThreads);
  stage_rows<false>(in + b0 * M, rows, M, n_operators, bsm);
  if (t < rows) {
    const RowCheck c = check_row(row, M);
    int64_t e = c.flag;
    int n_out = 0;
    if (!e) {
      // from postfix a row with a token after a NO_OP is walked from its last token
      int end = c.len;
      if (!kFromPrefix && c.follows)
        for (end = M; row[end - 1] == NO_OP;) --end;
      int sp = 0, balance = 0, roots = 0;
      auto emit = [&](int v) {
        row[kFromPrefix ? n_out : end - 1 - n_out] = (unsigned char)v;
        ++n_out;
      };
      // A turn takes one token and completes at most one operator, so that the lanes of a
      // warp go through their rows side by side.  up: an operand was completed.
      bool up = false;
      for (int s = 0;;) {
        if (up) {
          up = sp > 0;
          if (up) {
            const int top = stk[sp - 1];
            if (top & 0x80) {
              emit(top & 0x7f);
              --sp;
            } else {
              stk[sp - 1] = (unsigned char)(top | 0x80);
              up = false;
            }
          }
        }
        if (!up) {
          if (s >= end) break;
          const int tok = row[kFromPrefix ? s : end - 1 - s];
          if (!kFromPrefix && tok == NO_OP) break;
          ++s;
          const int ar = arity_of((int64_t)tok);
          balance += ar - 1;
          if (balance == -1) ++roots;
          up = ar == 0;
          if (up) emit(tok);
          else stk[sp++] = (unsigned char)(tok | (ar == 1 ? 0x80 : 0));
        }
      }
      if (c.follows) {
        e = CONV_UNEXPECTED_TOKEN;  // what was emitted so far stays, in the order emitted
        if (!kFromPrefix) {
          for (int i = end - n_out, j = end - 1; i < j; ++i, --j) {
            const unsigned char x = row[i];
            row[i] = row[j];
            row[j] = x;
          }
          for (int i = 0; i < n_out; ++i) row[i] = row[end - n_out + i];
        }
      } else if (sp != 0) {
        e = arity_of((int64_t)(stk[sp - 1] & 0x7f)) == 1 ? CONV_UNARY_MISSING : CONV_BINARY_MISSING;
        n_out = 0;
      } else if (roots != 1 && n_out > 0) {
        e = CONV_MULTIPLE_ROOTS;
        n_out = 0;
      }
    }
    counts[t] = (uint8_t)n_out;
    err[b0 + t] = e;
  }
  __syncthreads();
  each_element(rows, M, [&](int j, int r, int i) {
    outp[b0 * M + j] = i < counts[r] ? (int64_t)bsm[r * stride + i] : (int64_t)NO_OP;
  });
}

// Right-to-left rendering: the output is built backwards from the end of a
// 3 x 128 buffer.  An operator first emits ")" (and, for (x)^k forms, its own
// token); once its right operand is complete a binary operator emits itself, once
// its left operand is complete it emits "(".  A unary f emits "( f" when its operand
// is complete, a (x)^k form emits "(".
__global__ void postfix_to_infix_kernel(const int64_t* __restrict__ ops, int64_t B, int64_t M, int64_t n_operators,
                                        int64_t lparen, int64_t rparen, int64_t* __restrict__ infix, int64_t M_out,
                                        int64_t* __restrict__ err) {
  const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= B) return;
  const int64_t* row = ops + b * M;
  int64_t* out = infix + b * M_out;
  for (int64_t i = 0; i < M_out; ++i) out[i] = NO_OP;
  int64_t e = symbol_check(row, M, n_operators);
  if (e) {
    err[b] = e;
    return;
  }
  // shape check from the right: padding only at the end, one root
  bool started = false;
  int len = 0, balance = 0, roots = 0;
  for (int64_t k = M - 1; k >= 0; --k) {
    const int64_t t = row[k];
    if (t == NO_OP) {
      if (started) { err[b] = CONV_UNEXPECTED_TOKEN; return; }
    } else {
      started = true;
      ++len;
      balance += arity_of(t) - 1;
      if (balance == -1) ++roots;
    }
  }
  if (len == 0) { err[b] = 0; return; }
  if (roots > 1) { err[b] = CONV_MULTIPLE_ROOTS; return; }

  constexpr int kBuf = 3 * kStackLimit;
  int32_t buf[kBuf];
  int32_t opst[kStackLimit];
  int8_t waiting_left[kStackLimit];
  int top = kBuf - 1;  // next free slot, filled downwards
  int sp = 0;
#define SR_EMIT(tok)                                \
  do {                                              \
    if (top < 0) { err[b] = CONV_STACK_OVERFLOW; return; } \
    buf[top--] = (int32_t)(tok);                    \
  } while (0)
  for (int k = len - 1; k >= 0; --k) {
    const int64_t t = row[k];
    const int ar = arity_of(t);
    if (ar == 0) {
      SR_EMIT(t);
      bool done = true;
      while (done && sp > 0) {
        const int32_t parent = opst[sp - 1];
        if (arity_of(parent) == 1) {
          if (functional_style(parent)) {
            if (top - 1 < 0) { err[b] = CONV_STACK_OVERFLOW; return; }
            buf[top--] = (int32_t)lparen;
            buf[top--] = parent;
          } else {
            SR_EMIT(lparen);
          }
          --sp;
        } else if (!waiting_left[sp - 1]) {
          SR_EMIT(parent);
          waiting_left[sp - 1] = 1;
          done = false;
        } else {
          SR_EMIT(lparen);
          --sp;
        }
      }
    } else {
      if (sp >= kStackLimit) { err[b] = CONV_STACK_OVERFLOW; return; }
      opst[sp] = (int32_t)t;
      waiting_left[sp] = 0;
      if (ar == 1 && !functional_style(t)) SR_EMIT(t);
      SR_EMIT(rparen);
      ++sp;
    }
  }
#undef SR_EMIT
  if (sp > 0) {
    err[b] = arity_of(opst[sp - 1]) == 1 ? CONV_UNARY_MISSING : CONV_BINARY_MISSING;
    return;
  }
  const int n = kBuf - 1 - top;
  if (n > M_out) { err[b] = CONV_TOO_LONG; return; }
  for (int i = 0; i < n; ++i) out[i] = buf[top + 1 + i];
  err[b] = 0;
}

// The same rendering for token ids whose parentheses fit a byte too.  A complete row renders
// to one token per leaf and three per operator, so the right end of the output is known, and
// a row that does not fit M_out tokens is walked for its error without being written.  The
// output buffer holds the smaller of M_out and 3 M tokens per row.
// 50001 rows of 48 tokens: 28 us, where buffers in local memory took 82.
__global__ void __launch_bounds__(kRowThreads) postfix_to_infix_bytes_kernel(
    const int64_t* __restrict__ ops, int64_t B, int M, int64_t n_operators, int64_t* __restrict__ infix, int64_t M_out,
    int cap, int64_t* __restrict__ err) {
  extern __shared__ __align__(16) unsigned char bsm[];
  __shared__ uint16_t counts[kRowThreads];  // tokens of each output row
  const int t = threadIdx.x, stride = row_stride(M), out_stride = row_stride(cap);
  unsigned char* row = bsm + t * stride;
  unsigned char* stk = bsm + (kRowThreads + t) * stride;
  unsigned char* bufs = bsm + 2 * kRowThreads * stride;
  unsigned char* buf = bufs + t * out_stride;
  const int lparen = (int)n_operators, rparen = lparen + 1;
  const int64_t b0 = (int64_t)blockIdx.x * kRowThreads;
  const int rows = (int)(B - b0 < kRowThreads ? B - b0 : kRowThreads);
  stage_rows<false>(ops + b0 * M, rows, M, n_operators, bsm);
  if (t < rows) {
    const RowCheck c = check_row(row, M);
    int64_t e = c.flag;
    int n = 0;
    if (!e && c.follows) e = CONV_UNEXPECTED_TOKEN;
    if (!e && c.len > 0) {
      int balance = 0, roots = 0;
      for (int k = c.len - 1; k >= 0; --k) {
        const int ar = arity_of((int64_t)row[k]);
        n += ar ? 3 : 1;
        balance += ar - 1;
        if (balance == -1) ++roots;
      }
      if (roots > 1) {
        e = CONV_MULTIPLE_ROOTS;
      } else {
        const bool fits = n <= M_out;
        int at = n, sp = 0;  // the output from its right end; fewer than n tokens if incomplete
        auto emit = [&](int v) {
          --at;
          if (fits) buf[at] = (unsigned char)v;
        };
        // turns as in reorder_bytes_kernel; the stack's bit 7: the operand that is being
        // rendered is the last one (the left one)
        bool up = false;
        for (int k = c.len - 1;;) {
          if (up) {
            up = sp > 0;
            if (up) {
              const int top = stk[sp - 1], parent = top & 0x7f;
              if (top & 0x80) {
                emit(lparen);
                if (arity_of((int64_t)parent) == 1 && functional_style(parent)) emit(parent);
                --sp;
              } else {
                emit(parent);
                stk[sp - 1] = (unsigned char)(top | 0x80);
                up = false;
              }
            }
          }
          if (!up) {
            if (k < 0) break;
            const int tok = row[k--];
            const int ar = arity_of((int64_t)tok);
            up = ar == 0;
            if (!up) stk[sp++] = (unsigned char)(tok | (ar == 1 ? 0x80 : 0));
            if (up || (ar == 1 && !functional_style(tok))) emit(tok);
            if (!up) emit(rparen);
          }
        }
        if (sp > 0) e = arity_of((int64_t)(stk[sp - 1] & 0x7f)) == 1 ? CONV_UNARY_MISSING : CONV_BINARY_MISSING;
        else if (!fits) e = CONV_TOO_LONG;
      }
    }
    counts[t] = (uint16_t)(e ? 0 : n);
    err[b0 + t] = e;
  }
  __syncthreads();
  if (M_out > 0)
    each_element(rows, (int)M_out, [&](int j, int r, int i) {
      infix[b0 * M_out + j] = i < counts[r] ? (int64_t)bufs[r * out_stride + i] : (int64_t)NO_OP;
    });
}

// ---- prefix conversions ---------------------------------------------------------
// prefix <-> postfix (src/pcfg_cpu.cpp:812-993): a stack of (node, children still
// missing); a node is emitted once all its children are.  postfix -> prefix walks the
// row from the right and reverses what it emits.  Rows with an error are all NO_OP.
template <bool kFromPrefix>
__global__ void reorder_kernel(const int64_t* __restrict__ in, int64_t B, int64_t M, int64_t n_operators,
                               int64_t* __restrict__ outp, int64_t* __restrict__ err) {
  const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= B) return;
  const int64_t* row = in + b * M;
  int64_t* out = outp + b * M;
  for (int64_t i = 0; i < M; ++i) out[i] = NO_OP;
  int64_t e = symbol_check(row, M, n_operators);
  if (e) {
    err[b] = e;
    return;
  }
  int32_t node[kStackLimit];
  int8_t missing[kStackLimit];
  int sp = 0, n_out = 0, balance = 0, roots = 0;
  bool seen = false;  // prefix: past the end; postfix: the expression has started
  for (int64_t s = 0; s < M; ++s) {
    const int64_t i = kFromPrefix ? s : M - 1 - s;
    const int64_t t = row[i];
    if (t == NO_OP) {
      if (kFromPrefix) seen = true;
      else if (seen) { err[b] = CONV_UNEXPECTED_TOKEN; return; }
      continue;
    }
    if (kFromPrefix && seen) { err[b] = CONV_UNEXPECTED_TOKEN; return; }
    if (!kFromPrefix) seen = true;
    const int ar = arity_of(t);
    balance += ar - 1;
    if (balance == -1) ++roots;
    if (sp >= kStackLimit) { err[b] = CONV_STACK_OVERFLOW; return; }
    node[sp] = (int32_t)i;
    missing[sp++] = (int8_t)ar;
    while (sp > 0 && missing[sp - 1] == 0) {
      --sp;
      if (n_out >= M) { err[b] = kFromPrefix ? CONV_POSTFIX_TOO_LONG : CONV_PREFIX_TOO_LONG; return; }
      out[n_out++] = row[node[sp]];
      if (sp > 0) --missing[sp - 1];
    }
  }
  if (sp != 0) {
    for (int64_t i = 0; i < M; ++i) out[i] = NO_OP;
    err[b] = arity_of(row[node[sp - 1]]) == 1 ? CONV_UNARY_MISSING : CONV_BINARY_MISSING;
    return;
  }
  if (roots != 1 && n_out > 0) {
    for (int64_t i = 0; i < M; ++i) out[i] = NO_OP;
    err[b] = CONV_MULTIPLE_ROOTS;
    return;
  }
  if (!kFromPrefix) {  // emitted from the right: reverse into prefix order
    for (int i = 0, j = n_out - 1; i < j; ++i, --j) {
      const int64_t x = out[i];
      out[i] = out[j];
      out[j] = x;
    }
  }
  err[b] = 0;
}

// Parent of every node of a prefix row (src/pcfg_cpu.cpp:995-1064): from the right,
// a stack of finished subtrees; an operator adopts the top one or two.  Roots and
// padding keep -1.
__global__ void prefix_parent_kernel(const int64_t* __restrict__ in, int64_t B, int64_t M, int64_t n_operators,
                                     int64_t* __restrict__ parent, int64_t* __restrict__ err) {
  const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= B) return;
  const int64_t* row = in + b * M;
  int64_t* par = parent + b * M;
  for (int64_t i = 0; i < M; ++i) par[i] = -1;
  int64_t e = symbol_check(row, M, n_operators);
  if (e) {
    err[b] = e;
    return;
  }
  int32_t st[kStackLimit];
  int sp = 0;
  bool started = false;
  for (int64_t i = M - 1; i >= 0; --i) {
    const int64_t t = row[i];
    if (t == NO_OP) {
      if (started) { err[b] = PARSE_UNEXPECTED_TOKEN; return; }
      continue;
    }
    started = true;
    const int ar = arity_of(t);
    if (ar == 1) {
      if (sp < 1) { err[b] = PARSE_UNARY_MISSING; return; }
      par[st[--sp]] = i;
    } else if (ar == 2) {
      if (sp < 2) { err[b] = PARSE_BINARY_MISSING; return; }
      par[st[--sp]] = i;
      par[st[--sp]] = i;
    }
    if (sp >= kStackLimit) { err[b] = PARSE_STACK_OVERFLOW; return; }
    st[sp++] = (int32_t)i;
  }
  err[b] = (started && sp != 1) ? PARSE_MALFORMED : 0;
}

// Prefix -> infix token ids with parentheses (src/pcfg_cpu.cpp:637-811): the same
// rendering as postfix -> infix, produced left to right by a stack of operators that
// wait for their left or right operand.
__global__ void prefix_to_infix_kernel(const int64_t* __restrict__ in, int64_t B, int64_t M, int64_t n_operators,
                                       int64_t lparen, int64_t rparen, int64_t* __restrict__ infix, int64_t M_out,
                                       int64_t* __restrict__ err) {
  const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= B) return;
  const int64_t* row = in + b * M;
  int64_t* out = infix + b * M_out;
  for (int64_t i = 0; i < M_out; ++i) out[i] = NO_OP;
  int64_t e = symbol_check(row, M, n_operators);
  if (e) {
    err[b] = e;
    return;
  }
  int len = 0, balance = 0, roots = 0;
  bool ended = false;
  for (int64_t i = 0; i < M; ++i) {
    if (row[i] == NO_OP) {
      ended = true;
    } else {
      if (ended) { err[b] = CONV_UNEXPECTED_TOKEN; return; }
      ++len;
      balance += arity_of(row[i]) - 1;
      if (balance == -1) ++roots;
    }
  }
  if (len == 0) { err[b] = 0; return; }
  if (roots > 1) { err[b] = CONV_MULTIPLE_ROOTS; return; }
  int32_t opst[kStackLimit];
  int8_t waiting_right[kStackLimit];
  int sp = 0;
  int64_t n = 0;
#define SR_PUT(tok)                                            \
  do {                                                         \
    if (n >= M_out) { err[b] = CONV_TOO_LONG; goto fail; }     \
    out[n++] = (tok);                                          \
  } while (0)
  for (int k = 0; k < len; ++k) {
    const int64_t t = row[k];
    const int ar = arity_of(t);
    if (ar == 0) {
      SR_PUT(t);
      bool done = true;
      while (done && sp > 0) {
        const int32_t parent = opst[sp - 1];
        if (arity_of(parent) == 1) {
          SR_PUT(rparen);
          if (!functional_style(parent)) SR_PUT(parent);
          --sp;
        } else if (!waiting_right[sp - 1]) {
          SR_PUT(parent);
          waiting_right[sp - 1] = 1;
          done = false;
        } else {
          SR_PUT(rparen);
          --sp;
        }
      }
    } else {
      if (sp >= kStackLimit) { err[b] = CONV_STACK_OVERFLOW; goto fail; }
      opst[sp] = (int32_t)t;
      waiting_right[sp] = 0;
      if (ar == 1 && functional_style(t)) {
        if (n + 2 > M_out) { err[b] = CONV_TOO_LONG; goto fail; }
        out[n++] = t;
        out[n++] = lparen;
      } else {
        SR_PUT(lparen);
      }
      ++sp;
    }
  }
#undef SR_PUT
  if (sp != 0) {
    err[b] = arity_of(opst[sp - 1]) == 1 ? CONV_UNARY_MISSING : CONV_BINARY_MISSING;
    goto fail;
  }
  err[b] = 0;
  return;
fail:
  for (int64_t i = 0; i < M_out; ++i) out[i] = NO_OP;
}

}  // namespace sr

static unsigned row_blocks(int64_t B) { return (unsigned)((B + sr::kRowThreads - 1) / sr::kRowThreads); }

// Rows whose tokens, the ids up to `last` included, fit the byte kernels.
static bool byte_rows(int64_t M, int64_t last) { return M >= 1 && M <= sr::kStackLimit && last <= 255; }

extern "C" {

int sr_postfix_children(const int64_t* ops, int64_t B, int64_t M, int32_t n_vars, int64_t* ch, int64_t* err,
                        void* stream) {
  using namespace sr;
  if (B < 0 || M < 0 || n_vars < 0 || (B > 0 && (!ops || !ch || !err))) {
    set_error("invalid arguments");
    return SR_ERR_INVALID_ARGUMENT;
  }
  if (B == 0) return SR_OK;
  const int64_t n_operators = (int64_t)VAR + n_vars;
  if (M >= 1 && M <= kStackLimit) {
    const size_t smem = (size_t)3 * kRowThreads * row_stride((int)M);
    auto kern = reinterpret_cast<uintptr_t>(ch) % 16 ? postfix_children_bytes_kernel<false>
                                                     : postfix_children_bytes_kernel<true>;
    if (const int rc = sr::allow_dynamic_smem(reinterpret_cast<const void*>(kern), smem)) return rc;
    kern<<<row_blocks(B), kRowThreads, smem, as_stream(stream)>>>(ops, B, (int)M, n_operators, ch, err);
    return launch_check("postfix_children_bytes_kernel");
  }
  const int threads = 128;
  postfix_children_kernel<<<(unsigned)((B + threads - 1) / threads), threads, 0, as_stream(stream)>>>(
      ops, B, M, n_operators, ch, err);
  return launch_check("postfix_children_kernel");
}

int sr_postfix_to_infix(const int64_t* ops, int64_t B, int64_t M, int32_t n_vars, int64_t* infix, int64_t M_out,
                        int64_t* err, void* stream) {
  using namespace sr;
  if (B < 0 || M < 0 || M_out < 0 || n_vars < 0 || (B > 0 && (!ops || !err || (M_out > 0 && !infix)))) {
    set_error("invalid arguments");
    return SR_ERR_INVALID_ARGUMENT;
  }
  if (B == 0) return SR_OK;
  const int64_t n_operators = (int64_t)VAR + n_vars;
  if (byte_rows(M, n_operators + 1) && M_out <= INT32_MAX / kRowThreads) {
    const int cap = (int)(M_out < 3 * M ? M_out : 3 * M);
    const size_t smem = (size_t)kRowThreads * (2 * row_stride((int)M) + row_stride(cap));
    if (const int rc = sr::allow_dynamic_smem(reinterpret_cast<const void*>(postfix_to_infix_bytes_kernel), smem)) return rc;
    postfix_to_infix_bytes_kernel<<<row_blocks(B), kRowThreads, smem, as_stream(stream)>>>(ops, B, (int)M, n_operators,
                                                                                        infix, M_out, cap, err);
    return launch_check("postfix_to_infix_bytes_kernel");
  }
  const int threads = 128;
  const int64_t lparen = (int64_t)VAR + n_vars, rparen = lparen + 1;
  postfix_to_infix_kernel<<<(unsigned)((B + threads - 1) / threads), threads, 0, as_stream(stream)>>>(
      ops, B, M, (int64_t)VAR + n_vars, lparen, rparen, infix, M_out, err);
  return launch_check("postfix_to_infix_kernel");
}

}  // extern "C"

template <bool kFromPrefix>
static int launch_reorder(const int64_t* in, int64_t B, int64_t M, int32_t n_vars, int64_t* out, int64_t* err,
                          void* stream) {
  using namespace sr;
  const size_t smem = (size_t)2 * kRowThreads * row_stride((int)M);
  auto kern = reorder_bytes_kernel<kFromPrefix>;
  if (const int rc = sr::allow_dynamic_smem(reinterpret_cast<const void*>(kern), smem)) return rc;
  kern<<<row_blocks(B), kRowThreads, smem, as_stream(stream)>>>(in, B, (int)M, (int64_t)VAR + n_vars, out, err);
  return launch_check(kFromPrefix ? "reorder_bytes_kernel<prefix>" : "reorder_bytes_kernel<postfix>");
}

extern "C" {

static int notation_args_ok(const int64_t* in, int64_t B, int64_t M, int32_t n_vars, const void* out,
                            const int64_t* err) {
  if (B < 0 || M < 0 || n_vars < 0 || (B > 0 && (!in || !out || !err))) {
    sr::set_error("invalid arguments");
    return 0;
  }
  return 1;
}

int sr_prefix_to_postfix(const int64_t* prefix, int64_t B, int64_t M, int32_t n_vars, int64_t* postfix, int64_t* err,
                         void* stream) {
  using namespace sr;
  if (!notation_args_ok(prefix, B, M, n_vars, postfix, err)) return SR_ERR_INVALID_ARGUMENT;
  if (B == 0) return SR_OK;
  if (byte_rows(M, (int64_t)VAR + n_vars + 1)) return launch_reorder<true>(prefix, B, M, n_vars, postfix, err, stream);
  reorder_kernel<true><<<(unsigned)((B + 127) / 128), 128, 0, as_stream(stream)>>>(prefix, B, M, (int64_t)VAR + n_vars,
                                                                                postfix, err);
  return launch_check("reorder_kernel<prefix>");
}

int sr_postfix_to_prefix(const int64_t* postfix, int64_t B, int64_t M, int32_t n_vars, int64_t* prefix, int64_t* err,
                         void* stream) {
  using namespace sr;
  if (!notation_args_ok(postfix, B, M, n_vars, prefix, err)) return SR_ERR_INVALID_ARGUMENT;
  if (B == 0) return SR_OK;
  if (byte_rows(M, (int64_t)VAR + n_vars + 1)) return launch_reorder<false>(postfix, B, M, n_vars, prefix, err, stream);
  reorder_kernel<false><<<(unsigned)((B + 127) / 128), 128, 0, as_stream(stream)>>>(postfix, B, M,
                                                                                 (int64_t)VAR + n_vars, prefix, err);
  return launch_check("reorder_kernel<postfix>");
}

int sr_prefix_parent(const int64_t* prefix, int64_t B, int64_t M, int32_t n_vars, int64_t* parent, int64_t* err,
                     void* stream) {
  using namespace sr;
  if (!notation_args_ok(prefix, B, M, n_vars, parent, err)) return SR_ERR_INVALID_ARGUMENT;
  if (B == 0) return SR_OK;
  prefix_parent_kernel<<<(unsigned)((B + 127) / 128), 128, 0, as_stream(stream)>>>(prefix, B, M, (int64_t)VAR + n_vars,
                                                                                 parent, err);
  return launch_check("prefix_parent_kernel");
}

int sr_prefix_to_infix(const int64_t* prefix, int64_t B, int64_t M, int32_t n_vars, int64_t* infix, int64_t M_out,
                       int64_t* err, void* stream) {
  using namespace sr;
  if (!notation_args_ok(prefix, B, M, n_vars, M_out > 0 ? (const void*)infix : (const void*)err, err) || M_out < 0)
    return SR_ERR_INVALID_ARGUMENT;
  if (B == 0) return SR_OK;
  const int64_t lparen = (int64_t)VAR + n_vars, rparen = lparen + 1;
  prefix_to_infix_kernel<<<(unsigned)((B + 127) / 128), 128, 0, as_stream(stream)>>>(
      prefix, B, M, (int64_t)VAR + n_vars, lparen, rparen, infix, M_out, err);
  return launch_check("prefix_to_infix_kernel");
}

}  // extern "C"
