// sr_pcfg.cu -- grammar sampling and infix parsing on the GPU.
//
// The sampler draws expressions from a probabilistic context-free grammar given as
// the reference's CSR tables (src/pcfg.cpp:364-451): rules sorted by left-hand
// side, nt_rule_ptr[s] .. nt_rule_ptr[s + 1] the rules of symbol s, their cumulative
// probabilities, and the concatenated right-hand sides.  A lane derives one expression
// at a time (the derivation is sequential; persistent CTAs hand a finished lane the
// next expression), leftmost first with an explicit stack,
// exactly as the reference's sample_infix_kernel (src/pcfg_cuda.cu:10-118) does: a
// try restarts when the stack would exceed 128 symbols or the output would exceed
// the padded length, and after max_tries failed tries the expression reports 303.
// The random numbers come from a counter-based SplitMix64 stream per expression
// (Steele, Lea and Flood, "Fast splittable pseudorandom number generators", OOPSLA
// 2014), seeded from the caller's seed, so a seed fixes every expression; the
// oracle restates the same stream, so samples are checked token for token.
//
// The parser is the reference's shunting-yard (src/pcfg_cpu.cpp:121-448, the CUDA
// kernels at src/pcfg_cuda.cu:150-480 are the same): precedence 1 for + -, 2 for
// * /, 3 for ^, 4 for functions and parentheses, 0 (an operand) for everything
// else; ^ and the functions associate to the right.  To postfix it then checks
// that every operator has its operands and exactly one tree remains; to prefix it
// runs the mirrored algorithm from the right end.  One thread per expression; the
// stacks and the CTA's rows sit in shared memory, and rows are read and written by
// the whole CTA in coalesced order; token ids below 254 take a byte there.
#include <cstdint>

#include "sr_common.cuh"
#include "sr_ops.cuh"

namespace sr {
namespace pcfg {

constexpr int kHardMax = 128;  // the reference's HARD_MAX_LENGTH (include/pcfg_kernels.h:4)
constexpr int kThreads = 128;  // expressions per CTA

enum : int {
  GEN_MAX_TRIES = 303,
  GEN_NO_RULE = 304,
  PARSE_QUEUE_OVERFLOW = 401,
  PARSE_STACK_OVERFLOW = 402,
  PARSE_PAREN = 403,
  PARSE_UNARY_MISSING = 404,
  PARSE_BINARY_MISSING = 405,
  PARSE_MALFORMED = 407,
  PARSE_UNEXPECTED = 408,
  BAD_NEGATIVE = -1,  // a token below 0
  BAD_RANGE = -2,     // a token at or above the grammar's terminal limit
};

// SplitMix64 finaliser and stream (see the file comment).
__host__ __device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

struct Stream {
  uint64_t s;
  __device__ Stream(uint64_t seed, uint64_t index) : s(mix64(seed ^ mix64(index + 0x9E3779B97F4A7C15ull))) {}
  // uniform in (0, 1], 24 bits: the range the reference's curand_uniform draws from
  __device__ float uniform() {
    s += 0x9E3779B97F4A7C15ull;
    return (float)((uint32_t)(mix64(s) >> 40) + 1u) * (1.0f / 16777216.0f);
  }
};

__host__ __device__ __forceinline__ int odd_stride(int bytes) { return ((bytes + 3) / 4 | 1) * 4; }

// The grammar as the caller gave it.  rules() gives a symbol's first rule and how many it has
// (0: a terminal; an id outside [0, n_symbols) reads no table), choose() the first rule whose
// cumulative probability reaches u (-1: none), length() a rule's symbols.
struct WideGrammar {
  const int32_t *nt_ptr, *rhs_ptr, *rhs;
  const float* cum;
  int n_symbols;
  __device__ __forceinline__ int rules(int sym, int& r0) const {
    if ((unsigned)sym >= (unsigned)n_symbols) return 0;
    r0 = nt_ptr[sym];
    return nt_ptr[sym + 1] - r0;
  }
  __device__ __forceinline__ int choose(int r0, int n, float u) const {
    for (int r = r0; r < r0 + n; ++r)
      if (u <= cum[r]) return r;
    return -1;
  }
  __device__ __forceinline__ int length(int rule) const {
    const int n = rhs_ptr[rule + 1] - rhs_ptr[rule];
    return n > 0 ? n : 0;
  }
  // pushes all but the first symbol, last first; returns the first
  template <typename Tok>
  __device__ __forceinline__ int push(int rule, int n, Tok* stack, int& sp) const {
    const int32_t* p = rhs + rhs_ptr[rule];
    for (int i = n - 1; i >= 1; --i) stack[sp++] = (Tok)p[i];
    return n > 0 ? (int)(Tok)p[0] : 0;
  }
};

// A grammar with symbols below 256 whose tables take kTableBytes at most, in shared memory:
// one word per symbol and three per rule (its cumulative probability, its first four symbols,
// and where all of them are).  A symbol's rules start at a multiple of four and are filled up
// with NaN, which no number reaches, so a step waits for three reads, one after the other:
// the symbol's word, four probabilities at once, the rule.
constexpr int kTableBytes = 5120, kTableRules = 208, kTableSymbols = kTableBytes - 1024 - 12 * kTableRules;
struct SmallGrammar {
  const uint32_t* nt;    // [256] first rule | rules << 16
  const float* cum;      // [kTableRules]
  const uint2* rule;     // [kTableRules] first four symbols, offset | symbols << 16
  const uint8_t* rhs;
  __device__ __forceinline__ int rules(int sym, int& r0) const {
    const uint32_t e = nt[sym];
    r0 = (int)(e & 0xffffu);
    return (int)(e >> 16);
  }
  __device__ __forceinline__ int choose(int r0, int n, float u) const {
    for (int r = r0; r < r0 + n; r += 4) {
      const float4 c = *reinterpret_cast<const float4*>(cum + r);
      int at = -1;  // the first of the four, without branches that the lanes would part at
      if (u <= c.w) at = r + 3;
      if (u <= c.z) at = r + 2;
      if (u <= c.y) at = r + 1;
      if (u <= c.x) at = r;
      if (at >= 0) return at;
    }
    return -1;
  }
  __device__ __forceinline__ int length(int r) const { return (int)(rule[r].y >> 16); }
  template <typename Tok>
  __device__ __forceinline__ int push(int r, int n, Tok* stack, int& sp) const {
    const uint2 e = rule[r];
    for (int i = n - 1; i >= 4; --i) stack[sp++] = (Tok)rhs[(e.y & 0xffffu) + i];
    if (n > 3) stack[sp++] = (Tok)(e.x >> 24);
    if (n > 2) stack[sp++] = (Tok)((e.x >> 16) & 0xffu);
    if (n > 1) stack[sp++] = (Tok)((e.x >> 8) & 0xffu);
    return (int)(e.x & 0xffu);
  }
};

// The CTA's copy of a small grammar at `at`; false (in every thread) if it is not one.
__device__ __forceinline__ bool stage_grammar(const WideGrammar& W, int start, unsigned char* at, SmallGrammar& G) {
  const int t = threadIdx.x;
  if (W.n_symbols > 256 || start > 255) return false;
  const int rules = W.nt_ptr[W.n_symbols];
  if (rules < 0 || rules > kTableRules) return false;
  const int total = W.rhs_ptr[rules];
  if (total < 0 || total > kTableSymbols) return false;
  uint32_t* nt = reinterpret_cast<uint32_t*>(at);
  float* cum = reinterpret_cast<float*>(at + 1024);
  uint2* rule = reinterpret_cast<uint2*>(at + 1024 + 4 * kTableRules);
  uint8_t* rhs = at + 1024 + 12 * kTableRules;
  bool ok = true;
  for (int i = t; i < total; i += blockDim.x) {
    const int v = W.rhs[i];
    ok &= v >= 0 && v < 256;
    rhs[i] = (uint8_t)v;
  }
  if (t < 32) {  // a lane per symbol: its rules' place is a sum over the symbols before it
    int placed = 0;
    for (int s0 = 0; s0 < 256; s0 += 32) {
      const int s = s0 + t;
      int from = 0, n = 0;
      if (s < W.n_symbols) {
        from = W.nt_ptr[s];
        n = W.nt_ptr[s + 1] - from;
        const bool in = from >= 0 && n >= 0 && from <= rules - n;
        ok &= in;
        if (!in) n = 0;
      }
      const int room = (n + 3) & ~3;
      int upto = room;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, upto, o);
        if (t >= o) upto += x;
      }
      const int r0 = placed + upto - room;
      placed += __shfl_sync(0xffffffffu, upto, 31);
      const bool fits = placed <= kTableRules;
      ok &= fits;
      nt[s] = (uint32_t)(n > 0 ? r0 : 0) | (uint32_t)n << 16;
      for (int j = 0; fits && j < room; ++j) {
        const bool real = j < n;
        const int lo = real ? W.rhs_ptr[from + j] : 0, k = real ? W.rhs_ptr[from + j + 1] - lo : 0;
        const bool in = lo >= 0 && k >= 0 && lo <= total - k;
        ok &= in;
        uint32_t first = 0;
        for (int i = 0; in && i < k && i < 4; ++i) first |= (uint32_t)(W.rhs[lo + i] & 0xff) << (8 * i);
        rule[r0 + j] = make_uint2(first, (uint32_t)lo | (uint32_t)k << 16);
        cum[r0 + j] = real ? W.cum[from + j] : __int_as_float(0x7fffffff);
      }
    }
  }
  G = SmallGrammar{nt, cum, rule, rhs};
  return __syncthreads_and(ok);
}

// Whether every symbol id that a derivation can meet fits a byte; the same in every thread.
__device__ __forceinline__ bool byte_symbols(const WideGrammar& W, int start) {
  if (W.n_symbols > 256 || start > 255) return false;
  const int rules = W.nt_ptr[W.n_symbols];
  if (rules < 0) return false;
  const int total = W.rhs_ptr[rules];
  bool ok = total >= 0;
  for (int s = threadIdx.x; s < W.n_symbols; s += blockDim.x) {
    const int from = W.nt_ptr[s], to = W.nt_ptr[s + 1];
    ok &= from >= 0 && from <= to && to <= rules;
  }
  for (int j = threadIdx.x; j < rules; j += blockDim.x) {
    const int lo = W.rhs_ptr[j], hi = W.rhs_ptr[j + 1];
    ok &= lo >= 0 && hi <= total;
  }
  for (int i = threadIdx.x; i < total; i += blockDim.x) ok &= (unsigned)W.rhs[i] < 256u;
  return __syncthreads_and(ok);
}

// The CTA's warps derive the expressions [beg, beg + count).  Every lane works on one
// expression; a turn of the loop emits at most one terminal and expands at most one
// non-terminal of it, with the next symbol in a register and the next random number drawn
// ahead.  A lane whose expression is finished takes the CTA's next one (`queue`), so that a
// warp does not wait for its longest derivation before it goes on.  The draws of expression b
// come from its own stream, so the assignment of expressions to lanes changes no output.
template <typename Tok, typename G>
__device__ __forceinline__ void derive(const G& g, int start, int64_t beg, int64_t count, int* queue, int max_len,
                                       int max_tries, uint64_t seed, unsigned char* stacks, unsigned char* bufs,
                                       int64_t* __restrict__ out, int64_t* __restrict__ errors) {
  const int t = threadIdx.x, lane = t & 31;
  const int buf_bytes = odd_stride(max_len * (int)sizeof(Tok));
  Tok* stack = reinterpret_cast<Tok*>(stacks + t * odd_stride(kHardMax * (int)sizeof(Tok)));
  Tok* buf = reinterpret_cast<Tok*>(bufs + t * buf_bytes);
  const unsigned below = (1u << lane) - 1u;
  int64_t b = t;  // within the CTA's expressions
  bool active = b < count;
  Stream rng(seed, 0);
  float u = 0.0f;
  // cur: the symbol to work on; the stack holds the sp symbols after it
  int cur = start, tries = 0, sp = 0, len = 0, err = 0;
  // a new expression: its first try
  auto begin = [&]() {
    rng = Stream(seed, (uint64_t)(beg + b));
    u = rng.uniform();
    cur = start;
    tries = sp = len = err = 0;
  };
  if (active) begin();
  while (__any_sync(0xffffffffu, active)) {
    bool done = false;
    if (active) {
      enum { kGoOn, kEnded, kRestart, kNoRule };
      int state = kGoOn;
      int r0 = 0, n = g.rules(cur, r0);
      if (n == 0) {  // a terminal: emit it and take the next symbol
        if (len >= max_len) {  // past the padded length
          state = kRestart;
        } else {
          buf[len++] = (Tok)cur;
          if (sp == 0) {
            state = kEnded;
          } else {
            cur = stack[--sp];
            n = g.rules(cur, r0);
          }
        }
      }
      if (n != 0) {  // a non-terminal: choose a rule, leftmost symbol next
        const int chosen = g.choose(r0, n, u);
        u = rng.uniform();
        if (chosen < 0) {
          state = kNoRule;
        } else {
          const int k = g.length(chosen);
          if (sp + k > kHardMax) {
            state = kRestart;
          } else {
            cur = g.push(chosen, k, stack, sp);
            if (k == 0) {  // an empty right-hand side
              if (sp == 0) state = kEnded;
              else cur = stack[--sp];
            }
          }
        }
      }
      // a try ends: without a rule, restarted, or derived completely (an empty derivation
      // fails too)
      if (state != kGoOn) {
        done = true;
        if (state == kNoRule) {
          err = GEN_NO_RULE;
          len = 0;
        } else if (state == kRestart || len == 0) {
          len = 0;
          if (++tries >= max_tries) {
            err = GEN_MAX_TRIES;
          } else {
            cur = start;
            sp = 0;
            done = false;
          }
        }
      }
    }
    const unsigned m = __ballot_sync(0xffffffffu, done);
    if (m == 0) continue;
    // the warp writes the rows finished in this turn together, one row at a time, its
    // lanes on consecutive tokens (coalesced), while no lane waits on another's row
    int first = 0;
    if (lane == 0) first = atomicAdd(queue, __popc(m));
    first = __shfl_sync(0xffffffffu, first, 0);
    __syncwarp();  // the finished rows' tokens, written by their lanes
    for (unsigned mm = m; mm; mm &= mm - 1) {
      const int src = __ffs(mm) - 1;
      const int64_t bs = beg + __shfl_sync(0xffffffffu, b, src);
      const int ls = __shfl_sync(0xffffffffu, len, src);
      const int es = __shfl_sync(0xffffffffu, err, src);
      const Tok* row = reinterpret_cast<const Tok*>(bufs + ((t & ~31) + src) * buf_bytes);
      for (int i = lane; i < max_len; i += 32) out[bs * max_len + i] = i < ls ? (int64_t)row[i] : NO_OP;
      if (lane == 0) errors[bs] = es;
    }
    __syncwarp();  // read before their lanes start the next expressions
    if (done) {
      b = (int64_t)first + __popc(m & below);
      active = b < count;
      if (active) begin();
    }
  }
}

// Persistent CTAs, each with an equal share of the expressions.  What bounds it: the longest
// derivations of a CTA's share (a few hundred steps where the mean is 33), so the latency of
// a step: the symbol at hand in a register, the tables in shared memory and packed
// (SmallGrammar), rows of an odd number of words per thread (no bank conflicts when a warp
// writes a finished row), and symbols in a byte, which put 28 warps on an SM instead of 16.
// 262144 expressions of up to 64 tokens take 283 us where one symbol per turn, the tables
// read from L1 and 16-bit symbols took 513; 1000 take 132 us (before: 226), 1000000 take 501
// (1051).  With the probabilities read one by one (indexes clamped to the symbol's last) the
// first took 320 us; with two CTAs per SM, each with a longer queue, 425; with the streams of
// 32 expressions seeded ahead by all lanes, 343.
// Grammars with larger tables keep them in global memory, with symbols in a byte where all ids
// fit (400 rules, 262144 expressions of up to 64 tokens: 308 us, with 16-bit symbols and half
// the threads 401, with all 369).  Other ids keep 16 bits; `wide_threads`
// threads of the CTA then work (all of them, or the half that shared memory sized for bytes
// holds).
__global__ void __launch_bounds__(kThreads) sample_infix_kernel(
    const int32_t* __restrict__ nt_ptr, const float* __restrict__ cum, const int32_t* __restrict__ rhs_ptr,
    const int32_t* __restrict__ rhs, int32_t n_symbols, int32_t start, int64_t B, int32_t max_len,
    int32_t max_tries, uint64_t seed, int wide_threads, int64_t* __restrict__ out, int64_t* __restrict__ errors) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int queue;
  const int64_t per = (B + gridDim.x - 1) / gridDim.x, beg = per * blockIdx.x;
  const int64_t count = B - beg < per ? (B - beg > 0 ? B - beg : 0) : per;
  if (max_tries <= 0) {  // no try is allowed
    for (int64_t j = threadIdx.x; j < count * max_len; j += kThreads) out[beg * max_len + j] = NO_OP;
    for (int64_t j = threadIdx.x; j < count; j += kThreads) errors[beg + j] = GEN_MAX_TRIES;
    return;
  }
  const WideGrammar W{nt_ptr, rhs_ptr, rhs, cum, n_symbols};
  SmallGrammar S;
  const bool small = stage_grammar(W, start, smem, S);
  const bool narrow = small || byte_symbols(W, start);
  if (threadIdx.x == 0) queue = narrow ? kThreads : wide_threads;
  __syncthreads();
  if (small) {
    derive<uint8_t>(S, start, beg, count, &queue, max_len, max_tries, seed, smem + kTableBytes,
                    smem + kTableBytes + kThreads * odd_stride(kHardMax), out, errors);
  } else if (narrow) {
    derive<uint8_t>(W, start, beg, count, &queue, max_len, max_tries, seed, smem,
                    smem + kThreads * odd_stride(kHardMax), out, errors);
  } else if ((int)threadIdx.x < wide_threads) {
    derive<int16_t>(W, start, beg, count, &queue, max_len, max_tries, seed, smem,
                    smem + wide_threads * odd_stride(kHardMax * (int)sizeof(int16_t)), out, errors);
  }
}

__device__ __forceinline__ int precedence(int64_t tok, int64_t lp, int64_t rp) {
  if (tok == ADD || tok == SUB) return 1;
  if (tok == MUL || tok == DIV) return 2;
  if (tok == POW) return 3;
  if ((tok >= SIN && tok <= FIFTH) || tok == lp || tok == rp) return 4;
  return 0;
}

__device__ __forceinline__ bool right_assoc(int tok) { return tok == POW || (tok >= SIN && tok <= FIFTH); }

// kPrefix: infix -> prefix (src/pcfg_cpu.cpp:121-259); else infix -> postfix with the
// tree check (src/pcfg_cpu.cpp:261-448).
template <bool kPrefix>
__global__ void __launch_bounds__(kThreads) infix_parse_kernel(const int64_t* __restrict__ infix, int64_t B,
                                                               int64_t M, int32_t n_vars,
                                                               int64_t* __restrict__ outp,
                                                               int64_t* __restrict__ errors) {
  // An M-token row never holds more than M operators on the stack or M tokens in the
  // queue, so both are sized by M (the reference's 128-entry limits cannot be reached
  // for M <= 128; their checks stay).
  extern __shared__ int16_t sm[];
  const int cap = (int)M;
  int16_t* row = sm;                    // [M][kThreads]: the input, then the output
  int16_t* ops = sm + M * kThreads;     // [M][kThreads] operator stack
  // [M][kThreads] output queue.  To postfix the queue lives in the row itself: every
  // queued token was read before (operands when read, operators after, parentheses
  // never), so the queue never holds more tokens than the scan has read and each write
  // lands on a token already consumed.  To prefix the scan runs from the right end and
  // the queue from the left, so it has its own array.
  int16_t* queue = kPrefix ? ops + M * kThreads : row;
  const int t = threadIdx.x;
  const int64_t b0 = (int64_t)blockIdx.x * kThreads;
  const int64_t rows = B - b0 < kThreads ? B - b0 : kThreads;
  const int64_t lp = VAR + n_vars, rp = lp + 1, limit = rp + 1;
  // tokens outside [0, limit) are staged as -1 (negative) or -2 (too large).  Element j
  // of the CTA's block is token i = j % M of row r = j / M; j advances by kThreads, so
  // (r, i) advance by (kThreads / M, kThreads % M) with a carry (no division per token).
  int bad = 0;
  const int Mi = M > 0 ? (int)M : 1, total = (int)(rows * M);  // M = 0: no element
  const int dr = kThreads / Mi, di = kThreads % Mi;
  int r = t / Mi, i = t - (t / Mi) * Mi;
#pragma unroll 4
  for (int j = t; j < total; j += kThreads) {
    const int64_t tok = infix[b0 * M + j];
    int16_t v = (int16_t)tok;
    if (tok < 0 || tok >= limit) v = (int16_t)(tok < 0 ? -1 : -2);
    row[i * kThreads + r] = v;
    r += dr;
    i += di;
    if (i >= Mi) {
      i -= Mi;
      ++r;
    }
  }
  __syncthreads();
  const int64_t b = b0 + t;
  int n_out = 0;
  int err = 0;
  if (b < B) {
    for (int i = 0; i < M; ++i) {
      const int v = row[i * kThreads + t];
      if (v == -1) bad = BAD_NEGATIVE;  // reported before an out-of-range token, as the reference checks
      else if (v == -2 && bad == 0) bad = BAD_RANGE;
    }
    // a token after the first NO_OP
    int len = 0;
    bool ended = false;
    for (int i = 0; i < M && !err; ++i) {
      if (row[i * kThreads + t] == NO_OP) {
        ended = true;
      } else if (ended) {
        err = PARSE_UNEXPECTED;
      } else {
        ++len;
      }
    }
    int sp = 0;
    for (int step = 0; step < len && !err && !bad; ++step) {
      const int tok = row[(kPrefix ? len - 1 - step : step) * kThreads + t];
      const int open = (int)(kPrefix ? rp : lp), close = (int)(kPrefix ? lp : rp);
      const int pt = precedence(tok, lp, rp);
      if (pt == 0) {
        if (n_out >= cap) { err = PARSE_QUEUE_OVERFLOW; break; }
        queue[(n_out++) * kThreads + t] = (int16_t)tok;
      } else if (tok == open) {
        if (sp >= cap) { err = PARSE_STACK_OVERFLOW; break; }
        ops[(sp++) * kThreads + t] = (int16_t)tok;
      } else if (tok == close) {
        while (sp > 0 && ops[(sp - 1) * kThreads + t] != open) {
          if (n_out >= cap) { err = PARSE_QUEUE_OVERFLOW; break; }
          queue[(n_out++) * kThreads + t] = ops[(--sp) * kThreads + t];
        }
        if (err) break;
        if (sp == 0) { err = PARSE_PAREN; break; }
        --sp;
      } else {
        const bool ra = right_assoc(tok);
        while (sp > 0) {
          const int top = ops[(sp - 1) * kThreads + t];
          if (top == open) break;
          const int ptop = precedence(top, lp, rp);
          // to postfix: pop while the top binds at least as tightly (left-assoc) or
          // more tightly (right-assoc); to prefix the two conditions swap
          const bool pop = kPrefix ? (ra ? ptop >= pt : ptop > pt) : (ra ? ptop > pt : ptop >= pt);
          if (!pop) break;
          if (n_out >= cap) { err = PARSE_QUEUE_OVERFLOW; break; }
          queue[(n_out++) * kThreads + t] = (int16_t)top;
          --sp;
        }
        if (err) break;
        if (sp >= cap) { err = PARSE_STACK_OVERFLOW; break; }
        ops[(sp++) * kThreads + t] = (int16_t)tok;
      }
    }
    while (!err && !bad && sp > 0) {
      const int top = ops[(sp - 1) * kThreads + t];
      if (top == (int)(kPrefix ? rp : lp)) { err = PARSE_PAREN; break; }
      if (n_out >= cap) { err = PARSE_QUEUE_OVERFLOW; break; }
      queue[(n_out++) * kThreads + t] = (int16_t)top;
      --sp;
    }
    if (!kPrefix && !err && !bad && n_out > 0) {
      int depth = 0;
      for (int i = 0; i < n_out && !err; ++i) {
        const int tok = queue[i * kThreads + t];
        if (precedence(tok, lp, rp) == 0) {
          ++depth;
        } else {
          const int ar = arity_of(tok);
          if (depth < ar) err = ar == 1 ? PARSE_UNARY_MISSING : PARSE_BINARY_MISSING;
          depth = depth - ar + 1;
        }
      }
      if (!err && depth != 1) err = PARSE_MALFORMED;
    }
    if (err || bad) n_out = 0;
    errors[b] = bad ? bad : err;
  }
  __syncthreads();  // every thread is done with the staged rows
  if (b < B) {
    for (int i = 0; i < M; ++i) {
      int16_t v = (int16_t)NO_OP;
      if (i < n_out) v = queue[(kPrefix ? n_out - 1 - i : i) * kThreads + t];
      row[i * kThreads + t] = v;
    }
  }
  __syncthreads();
  r = t / Mi;
  i = t - r * Mi;
#pragma unroll 4
  for (int j = t; j < total; j += kThreads) {
    outp[b0 * M + j] = row[i * kThreads + r];
    r += dr;
    i += di;
    if (i >= Mi) {
      i -= Mi;
      ++r;
    }
  }
}

// The same parsers for rows of up to 128 tokens and token ids below 254, a token per byte.
// What bounds them: the passes of one thread over its row, over the warps that shared memory
// lets reside.  Each thread's row, stack and queue are rows of an odd number of words (no bank
// conflicts between the threads of a warp), the checks of the whole row go word by word, a
// table says what a token does, and only the tokens before the padding are parsed: 243 us for 262144 rows of 64 tokens with 16-bit tokens and six
// token-by-token passes, 90 us this way.
constexpr uint32_t kByteNegative = 0xff, kByteRange = 0xfe;  // tokens that fail the checks
constexpr int kByteLimit = 0xfe;

// Tokens of rows r < rows of the CTA's block into bytes, consecutive threads on consecutive tokens.
__device__ __forceinline__ void stage_bytes(const int64_t* __restrict__ src, int rows, int M, int stride, int64_t limit,
                                            unsigned char* dst) {
  const int total = rows * M, dr = kThreads / M, di = kThreads % M;
  int r = threadIdx.x / M, i = threadIdx.x - r * M;
#pragma unroll 8
  for (int j = threadIdx.x; j < total; j += kThreads) {
    const int64_t tok = src[j];
    dst[r * stride + i] = (unsigned char)(tok < 0 ? kByteNegative : (tok >= limit ? kByteRange : (uint32_t)tok));
    r += dr;
    i += di;
    if (i >= M) {
      i -= M;
      ++r;
    }
  }
}

// Row checks, four tokens at a time: a token that failed (BAD_*), the tokens before the first
// NO_OP (len), whether a token follows it.
__device__ __forceinline__ void check_row(const uint32_t* words, int n_words, int& bad, int& len, bool& follows) {
  bad = 0;
  len = 0;
  follows = false;
  bool ended = false;
  for (int w = 0; w < n_words; ++w) {
    const uint32_t x = words[w];
    if (__vcmpeq4(x, 0xffffffffu)) bad = BAD_NEGATIVE;
    else if (__vcmpeq4(x, 0xfefefefeu) && bad == 0) bad = BAD_RANGE;
    if (ended) {
      follows |= x != 0;
      continue;
    }
    const uint32_t zero = __vcmpeq4(x, 0u);
    if (!zero) {
      len += 4;
    } else {
      const int at = (__ffs((int)zero) - 1) & ~7;  // bit of the first NO_OP
      len += at >> 3;
      ended = true;
      follows |= (x >> at) != 0;
    }
  }
}

template <bool kPrefix>
__global__ void __launch_bounds__(kThreads) infix_parse_bytes_kernel(const int64_t* __restrict__ infix, int64_t B,
                                                                     int M, int32_t n_vars, int64_t* __restrict__ outp,
                                                                     int64_t* __restrict__ errors) {
  extern __shared__ __align__(16) unsigned char smem[];
  // What the parser needs to know of a token: its precedence on the stack (an opening
  // parenthesis 0), from which precedence on the stack's operators go to the queue before it
  // is taken, and what is then done with it.
  constexpr int kOperand = 0, kPush = 1, kClose = 2, kNever = 7;
  __shared__ uint8_t table[256];  // precedence | threshold << 3 | kind << 6
  __shared__ uint8_t counts[kThreads];  // tokens of each output row
  const int t = threadIdx.x, stride = odd_stride(M), n_words = (M + 3) / 4;
  unsigned char* row = smem + t * stride;
  unsigned char* ops = smem + (kThreads + t) * stride;  // operator stack
  // The output queue.  To postfix it lives in the row itself (see infix_parse_kernel); to
  // prefix, which scans from the right end, it fills an array of its own from the right end.
  unsigned char* queues = kPrefix ? smem + 2 * kThreads * stride : smem;
  unsigned char* queue = queues + t * stride;
  const int64_t b0 = (int64_t)blockIdx.x * kThreads;
  const int rows = (int)(B - b0 < kThreads ? B - b0 : kThreads);
  const int lp = VAR + n_vars, rp = lp + 1;
  const int open = kPrefix ? rp : lp, close = kPrefix ? lp : rp;
  for (int k = t; k < 256; k += kThreads) {
    // to postfix: an operator takes off those that bind at least as tightly (left-assoc) or
    // more tightly (right-assoc); to prefix the two conditions swap
    const int p = precedence(k, lp, rp);
    int e = p | (p + (right_assoc(k) != kPrefix ? 1 : 0)) << 3 | kPush << 6;
    if (p == 0) e = kNever << 3 | kOperand << 6;
    if (k == open) e = kNever << 3 | kPush << 6;
    if (k == close) e = 1 << 3 | kClose << 6;
    table[k] = (uint8_t)e;
  }
  reinterpret_cast<uint32_t*>(row)[n_words - 1] = 0u;  // bytes past the last token
  __syncthreads();
  stage_bytes(infix + b0 * M, rows, M, stride, rp + 1, smem);
  __syncthreads();
  if (t < rows) {
    int bad, len, n_out = 0, err = 0;
    bool follows;
    check_row(reinterpret_cast<const uint32_t*>(row), n_words, bad, len, follows);
    if (follows) err = PARSE_UNEXPECTED;
    int sp = 0, depth = 0;
    int missing = 0;  // first operator of the postfix row without its operands
    auto enqueue = [&](int tok, int p) {
      queue[kPrefix ? M - 1 - n_out : n_out] = (unsigned char)tok;
      ++n_out;
      if (!kPrefix) {
        const int ar = p == 0 ? 0 : (p == 4 ? 1 : 2);
        if (depth < ar && !missing) missing = ar == 1 ? PARSE_UNARY_MISSING : PARSE_BINARY_MISSING;
        depth = depth - ar + 1;
      }
    };
    // A turn either queues the top of the stack or takes the next token, so that the lanes of
    // a warp go through their rows side by side, whatever each row needs.  The end of the row
    // empties the stack as a closing parenthesis does.
    const int end = 1 << 3 | kClose << 6;
    int step = 0, top = 0, ptop = 0;
    auto next = [&](int& tok) {
      tok = step < len ? (int)row[kPrefix ? len - 1 - step : step] : -1;
      return step < len ? (int)table[tok] : end;
    };
    auto look = [&]() {  // the stack's new top
      top = sp > 0 ? (int)ops[sp - 1] : 0;
      ptop = sp > 0 ? table[top] & 7 : 0;
    };
    int tok, e = next(tok);
    while (!err && !bad) {
      const int kind = e >> 6;
      if (ptop >= ((e >> 3) & 7)) {
        enqueue(top, ptop);
        --sp;
        look();
        continue;
      }
      if (kind == kOperand) {
        enqueue(tok, 0);
      } else if (kind == kPush) {
        ops[sp++] = (unsigned char)tok;
        top = tok;
        ptop = e & 7;
      } else {
        // the stack is empty or an opening parenthesis is on top
        if (tok < 0 && sp == 0) break;
        if (tok < 0 || sp == 0) {
          err = PARSE_PAREN;
          break;
        }
        --sp;
        look();
      }
      ++step;
      e = next(tok);
    }
    if (!kPrefix && !err && !bad && n_out > 0) err = missing ? missing : (depth != 1 ? PARSE_MALFORMED : 0);
    if (err || bad) n_out = 0;
    errors[b0 + t] = bad ? bad : err;
    counts[t] = (uint8_t)n_out;
  }
  __syncthreads();
  const int total = rows * M, dr = kThreads / M, di = kThreads % M;
  int r = t / M, i = t - r * M;
#pragma unroll 8
  for (int j = t; j < total; j += kThreads) {
    const int n = counts[r];
    outp[b0 * M + j] = i < n ? (int64_t)queues[r * stride + (kPrefix ? M - n + i : i)] : (int64_t)NO_OP;
    r += dr;
    i += di;
    if (i >= M) {
      i -= M;
      ++r;
    }
  }
}

template <bool kPrefix>
static int launch_parse(const int64_t* infix, int64_t B, int64_t M, int32_t n_vars, int64_t* outp, int64_t* errors,
                        void* stream) {
  if (B < 0 || M < 0) { set_error("negative size"); return SR_ERR_INVALID_ARGUMENT; }
  if (M > kHardMax) {
    set_error("M must be less than or equal to HARD_MAX_LENGTH, but got %lld > %d.", (long long)M, kHardMax);
    return SR_ERR_UNSUPPORTED;
  }
  if (n_vars < 0 || n_vars > SR_MAX_VARS) { set_error("n_vars out of range (%d)", n_vars); return SR_ERR_UNSUPPORTED; }
  if (B == 0) return SR_OK;
  if (!errors || (M > 0 && (!infix || !outp))) { set_error("null pointer argument"); return SR_ERR_INVALID_ARGUMENT; }
  const int64_t arrays = kPrefix ? 3 : 2;  // row, operator stack (, queue)
  if (M >= 1 && VAR + n_vars + 2 <= kByteLimit) {
    const size_t bytes = (size_t)arrays * kThreads * odd_stride((int)M);
    auto kern = infix_parse_bytes_kernel<kPrefix>;
    const int rc = allow_dynamic_smem(reinterpret_cast<const void*>(kern), bytes);
    if (rc) return rc;
    kern<<<(unsigned)((B + kThreads - 1) / kThreads), kThreads, bytes, as_stream(stream)>>>(infix, B, (int)M, n_vars, outp,
                                                                                           errors);
    return launch_check(kPrefix ? "infix_parse_bytes_kernel<prefix>" : "infix_parse_bytes_kernel<postfix>");
  }
  const size_t smem = (size_t)(arrays * M > 0 ? arrays * M : 1) * kThreads * sizeof(int16_t);
  auto kern = infix_parse_kernel<kPrefix>;
  int rc = allow_dynamic_smem(reinterpret_cast<const void*>(kern), smem);
  if (rc) return rc;
  const int64_t blocks = (B + kThreads - 1) / kThreads;
  kern<<<(unsigned)blocks, kThreads, smem, as_stream(stream)>>>(infix, B, M, n_vars, outp, errors);
  return launch_check(kPrefix ? "infix_parse_kernel<prefix>" : "infix_parse_kernel<postfix>");
}

}  // namespace pcfg
}  // namespace sr

extern "C" {

int sr_pcfg_sample_infix(const int32_t* nt_rule_ptr, const float* nt_rule_cum_probs, const int32_t* rhs_ptr,
                         const int32_t* rhs_concat, int32_t n_symbols, int32_t start_symbol, int64_t B,
                         int32_t max_length, int32_t max_tries, uint64_t seed, int64_t* out, int64_t* errors,
                         void* stream) {
  using namespace sr;
  using namespace sr::pcfg;
  if (B < 0 || max_length < 1 || max_length > kHardMax || max_tries < 0) {
    set_error("bad sampling request: B=%lld max_length=%d max_tries=%d", (long long)B, max_length, max_tries);
    return SR_ERR_INVALID_ARGUMENT;
  }
  if (n_symbols < 1 || n_symbols >= 32768 || start_symbol < 0 || start_symbol >= 32768) {
    set_error("grammar symbol ids must lie in [0, 32768) (n_symbols=%d, start=%d)", n_symbols, start_symbol);
    return SR_ERR_UNSUPPORTED;
  }
  if (B == 0) return SR_OK;
  if (!nt_rule_ptr || !nt_rule_cum_probs || !rhs_ptr || !rhs_concat || !out || !errors) {
    set_error("null pointer argument");
    return SR_ERR_INVALID_ARGUMENT;
  }
  // Grammars that may have symbols below 256 get shared memory for those (and for half as
  // many threads with 16-bit symbols, should an id or the tables turn out larger).
  const bool bytes = n_symbols <= 256 && start_symbol < 256;
  const int wide_threads = bytes ? kThreads / 2 : kThreads;
  size_t smem = (size_t)wide_threads * (odd_stride(2 * kHardMax) + odd_stride(2 * max_length));
  const size_t narrow = (size_t)kTableBytes + (size_t)kThreads * (odd_stride(kHardMax) + odd_stride(max_length));
  if (bytes && narrow > smem) smem = narrow;
  if (smem > (size_t)max_dyn_smem()) { set_error("sampling tables do not fit in shared memory"); return SR_ERR_UNSUPPORTED; }
  int rc = allow_dynamic_smem(reinterpret_cast<const void*>(sample_infix_kernel), smem);
  if (rc) return rc;
  // persistent grid: the CTAs that fit at once, or fewer when B is small
  int dev = 0, sms = 0, per_sm = 0;
  rc = cuda_check(cudaGetDevice(&dev), "cudaGetDevice");
  if (!rc) rc = cuda_check(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "SM count");
  if (rc) return rc;
  per_sm = resident_ctas(reinterpret_cast<const void*>(sample_infix_kernel), kThreads, smem);
  int64_t blocks = (int64_t)sms * (per_sm > 0 ? per_sm : 1);
  const int64_t need = (B + wide_threads - 1) / wide_threads;
  if (blocks > need) blocks = need;
  sample_infix_kernel<<<(unsigned)blocks, kThreads, smem, as_stream(stream)>>>(
      nt_rule_ptr, nt_rule_cum_probs, rhs_ptr, rhs_concat, n_symbols, start_symbol, B, max_length, max_tries, seed,
      wide_threads, out, errors);
  return launch_check("sample_infix_kernel");
}

int sr_infix_to_postfix(const int64_t* infix, int64_t B, int64_t M, int32_t n_vars, int64_t* postfix,
                        int64_t* errors, void* stream) {
  return sr::pcfg::launch_parse<false>(infix, B, M, n_vars, postfix, errors, stream);
}

int sr_infix_to_prefix(const int64_t* infix, int64_t B, int64_t M, int32_t n_vars, int64_t* prefix, int64_t* errors,
                       void* stream) {
  return sr::pcfg::launch_parse<true>(infix, B, M, n_vars, prefix, errors, stream);
}

}  // extern "C"
