// sr_eval.cu -- tape validation/staging and forward evaluation kernels (the adjoint is in
// sr_adjoint.cu).
//
// Design (sm_103a): one warp interprets one tape; its lanes cover data points, so
// opcode dispatch is warp-uniform and every cache row segment a warp writes is a
// contiguous run of 128-byte lines.  The tape words of a warp and the node values of the
// points it is working on live in shared memory; children are read from there,
// never from HBM.  The forward pass writes each (node, point) value once with a
// streaming store, which makes it bound by HBM write bandwidth.
#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <type_traits>

#include <cooperative_groups.h>

#include "sr_eval.cuh"

namespace sr {

static thread_local char g_err[512];

void set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
}

// ------------------------------------------------------------------------------------
// Validation + staging.  One warp per tape row; lanes over nodes.
// Validation follows the reference (src/evaluation_kernels_cuda.cu:13-49): a child
// that is not NULL_CHILD counts towards the arity and must be below its parent
// (101); the count must equal the arity (102).  Inputs the reference accepts but
// then reads out of bounds (a counted child < 0, or a unary node whose only child
// sits in the second slot) are reported as 101 here.
// The batch summary is one maximum per CTA, by warps that each take several tapes: with an
// atomic per tape the 65536 atomics on four words bound the kernel (16384 tapes of 64 nodes:
// 46 us; 10 us so).
// ------------------------------------------------------------------------------------
template <bool kStage>
__global__ void __launch_bounds__(256) tape_compile_kernel(const int64_t* __restrict__ ops,
                                                           const int64_t* __restrict__ ch, int64_t B,
                                                           int64_t M, int64_t ops_sb, int64_t ops_sm,
                                                           int64_t ch_sb, int64_t ch_sm, int64_t ch_si,
                                                           int32_t n_vars, uint32_t* __restrict__ desc,
                                                           int32_t* __restrict__ meta,
                                                           int32_t* __restrict__ status) {
  const int lane = threadIdx.x & 31;
  const int64_t warps_total = (int64_t)gridDim.x * (blockDim.x >> 5);
  int max_len = 0, max_root = 0, max_kroot = 0, max_ops = 0;  // of this warp's tapes
  for (int64_t b = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); b < B; b += warps_total) {
    int count = 0, last = -1;
    int err = 0;
    for (int64_t m0 = 0; m0 < M; m0 += 32) {
      const int64_t m = m0 + lane;
      const bool in = m < M;
      int64_t op = 0;
      if (in) {
        op = ops[b * ops_sb + m * ops_sm];
        const int64_t c0 = ch[b * ch_sb + m * ch_sm];
        const int64_t c1 = ch[b * ch_sb + m * ch_sm + ch_si];
        const int ar = arity_of(op);
        int actual = 0;
        int e = 0;
        if (c0 != -1) { actual++; if (c0 >= m) e = ERR_CHILD_GEQ_PARENT; }
        if (!e && c1 != -1) { actual++; if (c1 >= m) e = ERR_CHILD_GEQ_PARENT; }
        if (!e && actual != ar) e = ERR_ARITY;
        if (!e && ar >= 1 && c0 < 0) e = ERR_CHILD_GEQ_PARENT;
        if (!e && ar == 2 && c1 < 0) e = ERR_CHILD_GEQ_PARENT;
        err = err ? err : e;
        if (kStage) {
          int code;
          uint32_t f0 = 0, f1 = 0;
          if (op == NO_OP || (op >= LEARNABLE && op <= E_) || (op >= SIN && op <= FIFTH) ||
              (op >= ADD && op <= POW)) {
            code = (int)op;
            if (ar >= 1 && !e) f0 = (uint32_t)c0;
            if (ar == 2 && !e) f1 = (uint32_t)c1;
          } else if (op >= VAR && op < VAR + (int64_t)n_vars) {
            code = VAR;
            f0 = (uint32_t)(op - VAR);
          } else {
            code = ZERO;
          }
          desc[b * M + m] = pack(code, f0, f1);
        }
      }
      const unsigned real = __ballot_sync(0xffffffffu, in && op != NO_OP);
      count += __popc(real);
      if (real) last = (int)m0 + 31 - __clz((int)real);
    }
    if (err) report(status, err);
    if (kStage) {
      const int root = count > 0 ? count - 1 : 0;
      int kroot = 0, kall = 0, nops = 0;
      for (int64_t m0 = 0; m0 < M; m0 += 32) {
        const int64_t m = m0 + lane;
        const int64_t op = m < M ? ops[b * ops_sb + m * ops_sm] : -1;
        const bool lc = op == LEARNABLE;
        kall += __popc(__ballot_sync(0xffffffffu, lc));
        kroot += __popc(__ballot_sync(0xffffffffu, lc && m <= root));
        nops += __popc(__ballot_sync(0xffffffffu, m <= root && (op == NO_OP || arity_of(op) >= 1)));
      }
      if (lane == 0) {
        meta[b * 4 + 0] = last + 1;
        meta[b * 4 + 1] = root;
        meta[b * 4 + 2] = kroot;
        meta[b * 4 + 3] = kall;
      }
      max_len = max(max_len, last + 1);
      max_root = max(max_root, root + 1);
      max_kroot = max(max_kroot, kroot);
      max_ops = max(max_ops, nops);
    }
  }
  if (kStage) {
    // batch summary: stats[1] = max L_eff, stats[2] = max root + 1, stats[3] = max constants
    // to the root, stats[4] = max operator nodes
    __shared__ int cta_max[4];
    if (threadIdx.x < 4) cta_max[threadIdx.x] = 0;
    __syncthreads();
    if (lane < 4) {
      const int mine = lane == 0 ? max_len : lane == 1 ? max_root : lane == 2 ? max_kroot : max_ops;
      atomicMax(&cta_max[lane], mine);
    }
    __syncthreads();
    if (threadIdx.x < 4) atomicMax(status + 1 + threadIdx.x, cta_max[threadIdx.x]);
  }
}

// Rows L..M-1 of every tape's cache block are NaN.  They form one contiguous range per
// tape, written on a side stream, concurrently with the forward kernel, which writes only
// the real rows.  One warp per SM sends them with bulk copies from a block of NaNs in shared
// memory: the copy engine moves the bytes, so the fill takes next to none of the issue slots
// and warp places that the forward needs (as a kernel of vector stores it held 64 warps of
// every SM, and the forward grids waited for it: 16384 tapes of mean length 20, M = 64,
// N = 1024: 925 us with it, 697 us with the copies, for 4.3 GB).  Short ranges go 32 at a time, a
// lane each: one after the other they were what 5000 short tapes waited for.
// A tape longer than the max_len the call was given is evaluated by no class grid: its
// whole block is NaN, so no row keeps what the buffer held before.
constexpr int kFillBytes = 4096;          // one bulk copy
constexpr size_t kFillReserve = kFillBytes + 1024;  // shared memory of an SM that its CTA takes

template <typename T>
__global__ void __launch_bounds__(32) pad_fill_kernel(const int32_t* __restrict__ meta, int64_t B, int64_t M,
                                                      int64_t NK, int Lmax, T* __restrict__ cache) {
  __shared__ __align__(128) T block[kFillBytes / sizeof(T)];
  const int lane = threadIdx.x;
  const T qnan = M_<T>::nan();
  for (int i = lane; i < kFillBytes / (int)sizeof(T); i += 32) block[i] = qnan;
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncwarp();
  const uint32_t src = static_cast<uint32_t>(__cvta_generic_to_shared(block));
  // 32 tapes at a time: a lane for each while their ranges take one copy (or none), else the warp
  // for one after the other
  auto range = [&](int64_t b, int64_t L, T*& p, size_t& count, size_t& head) -> size_t {
    p = cache + (size_t)b * M * NK + (size_t)L * NK;
    count = (size_t)(M - L) * NK;
    // bulk copies start and end on 16-byte boundaries
    head = ((16 - (reinterpret_cast<uintptr_t>(p) & 15)) & 15) / sizeof(T);
    if (head > count) head = count;
    return (count - head) * sizeof(T) & ~size_t(15);
  };
  auto copy = [&](void* to, size_t bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(to), "r"(src), "r"((uint32_t)bytes)
                 : "memory");
  };
  for (int64_t b0 = blockIdx.x; b0 < B; b0 += 32 * (int64_t)gridDim.x) {
    const int64_t mine = b0 + (int64_t)lane * gridDim.x;
    int L = mine < B ? meta[mine * 4] : 0;
    if (L > Lmax) L = 0;
    T* p;
    size_t count = 0, head = 0, body = 0;
    if (mine < B) body = range(mine, L, p, count, head);
    if (!__any_sync(0xffffffffu, body > (size_t)kFillBytes)) {
      for (size_t i = 0; i < head; ++i) __stcs(p + i, qnan);
      if (body) copy(p + head, body);
      for (size_t i = head + body / sizeof(T); i < count; ++i) __stcs(p + i, qnan);
    } else {
      for (int t = 0; t < 32 && b0 + (int64_t)t * gridDim.x < B; ++t) {
        body = range(b0 + (int64_t)t * gridDim.x, __shfl_sync(0xffffffffu, L, t), p, count, head);
        const size_t tail = head + body / sizeof(T);
        if ((size_t)lane < head) __stcs(p + lane, qnan);
        for (size_t off = (size_t)lane * kFillBytes; off < body; off += 32 * (size_t)kFillBytes)
          copy(reinterpret_cast<unsigned char*>(p + head) + off, body - off < (size_t)kFillBytes ? body - off : (size_t)kFillBytes);
        if (tail + lane < count) __stcs(p + tail + lane, qnan);
      }
    }
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  }
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// Work order: the tapes by falling meta[column], by one cluster of CTAs (each counts the values of
// its share of the tapes, all add up the counts through each other's shared memory, then each
// places its share).  The order decides only which warp takes which tape, so tapes of one length
// come in any order.  What bounds it: two passes over meta, so a thread reads kOrderLoads tapes at
// once and counts with plain shared-memory atomics; with the lanes of a warp grouped by value
// first one CTA took 31 us for 16384 tapes instead of 13.5.  A large batch is shared among
// kOrderCtas CTAs (with the call, 1000000 tapes 637 to 97 us, 65536 61 to 27; 1000 24 with one CTA, 27
// with eight); a
// library sort's five launches took the host longer than the forward of a small batch.
constexpr int kOrderLoads = 8, kOrderCtas = 8;
constexpr int64_t kOrderOneCta = 8192;  // tapes that one CTA reads in one go

__global__ void __launch_bounds__(1024) tape_order_kernel(const int32_t* __restrict__ meta, int64_t B, int column,
                                                          int add, int bins, int32_t* __restrict__ order) {
  namespace cg = cooperative_groups;
  extern __shared__ int count[];  // per value: the count of this CTA's tapes
  int* at = count + bins;         // the next place
  __shared__ int warp_sum_[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const cg::cluster_group cluster = cg::this_cluster();
  const int ctas = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int64_t share = (B + ctas - 1) / ctas, from = share * rank, to = from + share < B ? from + share : B;
  for (int i = tid; i < bins; i += blockDim.x) count[i] = 0;
  __syncthreads();
  // f(b, key) for every tape of the share, the lanes of a warp together; key 0 for the largest
  // value, -1 past the last tape
  auto each_tape = [&](auto f) {
    for (int64_t b0 = from; b0 < to; b0 += (int64_t)kOrderLoads * blockDim.x) {
      int k[kOrderLoads];
#pragma unroll
      for (int j = 0; j < kOrderLoads; ++j) {
        const int64_t b = b0 + j * (int)blockDim.x + tid;
        k[j] = b < to ? bins - 1 - min(max(meta[b * 4 + column] + add, 0), bins - 1) : -1;
      }
#pragma unroll
      for (int j = 0; j < kOrderLoads; ++j)
        if (b0 + j * (int)blockDim.x < to) f(b0 + j * (int)blockDim.x + tid, k[j]);
    }
  };
  each_tape([&](int64_t, int k) {
    if (k >= 0) atomicAdd(&count[k], 1);
  });
  cluster.sync();
  // exclusive running sums over the bins, a run of consecutive bins per thread; within a bin the
  // shares in their order
  const int per = (bins + (int)blockDim.x - 1) / (int)blockDim.x, lo = min(bins, tid * per), hi = min(bins, lo + per);
  int sum = 0;
  for (int i = lo; i < hi; ++i) {
    int before = 0;
    for (int c = 0; c < ctas; ++c) {
      if (c == rank) at[i] = before;
      before += *cluster.map_shared_rank(count + i, c);
    }
    sum += before;
  }
  int incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_sum_[warp] = incl;
  __syncthreads();
  int before = incl - sum;
  for (int w = 0; w < warp; ++w) before += warp_sum_[w];
  for (int i = lo; i < hi; ++i) {
    at[i] += before;
    for (int c = 0; c < ctas; ++c) before += *cluster.map_shared_rank(count + i, c);
  }
  cluster.sync();  // also: no CTA leaves while another reads its counts
  each_tape([&](int64_t b, int k) {
    if (k >= 0) order[atomicAdd(&at[k], 1)] = (int32_t)b;
  });
}

// Whether any of n words is not zero.
__global__ void __launch_bounds__(256) any_nonzero_kernel(const int64_t* __restrict__ words, int64_t n,
                                                          int32_t* __restrict__ out) {
  bool nz = false;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    nz |= words[i] != 0;
  if (__any_sync(0xffffffffu, nz) && (threadIdx.x & 31) == 0) atomicOr(out, 1);
}

// ------------------------------------------------------------------------------------
// Forward.  Work unit = (tape, slice of its points); units are taken in grid-stride order
// over the tapes sorted longest first, so every warp of the persistent grid gets a similar
// mix of long and short tapes.
//
// Per unit the warp compiles its tape into an operator program whose operands are
// precomputed addresses, then passes over its points 32 V at a time (V = 4 float32 or 2
// float64 points per lane, see Pack): leaves are loads and stores, and only operator nodes
// are dispatched.  What bounds it: the instructions per node and point.  One point per lane
// paid a node's decode, address arithmetic and dispatch (about 25 of 35 instructions for an
// addition) for every 32 values; V points pay them once, and the operand, result and output
// accesses are 16 bytes wide.  That needs V times the shared memory per row, which the stack
// rows (stack_rows) give back: a 64-node tape holds 16 rows of 512 bytes instead of 64 of
// 128.  Measured with the fill kernel above: 16384 tapes of mean length 20 at N = 1024, 914 to
// 697 us (6.2 TB/s); 65536 tapes 3500 to 2770 us; 1003 tapes at N = 777, 135 to 72 us.
//
// Tapes out of stack order take a row per operator, and as many values per lane (V, V / 2 or 1)
// as the table then holds: with one value and a row per node 4096 tapes with shared subtrees took
// 302 us where this takes 239, deep tapes (20 results waiting) 568 and 355; where every tape
// has 30 operators out of order (422 us) the kernel of one point per lane, with more warps, took
// 382.  Variables beyond the rows are numbered by the tape's distinct ones (17 variables: 394 to
// 270 us).  Few points skip the search for the stack's order, as a pass of V values per lane
// would be half empty: 20000 tapes at N = 16, 72 to 43 us with the fill's change.
//
// With K constant sets the cache is (B, M, N, K): node k's values are the N K consecutive
// elements p = n K + kk, and the lanes run over them as over points (coalesced stores for
// any K; stores K elements apart took 537 us for 1000 tapes at N = 256, K = 8, where this takes
// 63); a constant's value then depends on the element, and is read from its K entries at
// kk = p mod K.  More sets than the table of constants holds are taken one by one, as units
// (tape, set, slice) whose values lie K elements apart (kStrided).
// ------------------------------------------------------------------------------------

// Shared-memory layout of one warp: the tape words (offset 0); the program, from the front
// 16 bytes per operator (dense code | node << 8, own row, two operand words) and from the
// back 4 bytes per leaf (node | variable flag << 12 | variable or constant index << 13); the
// constants' values (K entries for each learnable or fixed leaf), the rows of the variables,
// and the rows of the operator results.
struct FwdLayout {
  size_t prog, cval, xvar, xrow, rows, bytes;
};


constexpr int kMaxVarRows = 16;  // variables held in rows

template <typename T>
__host__ __device__ __forceinline__ FwdLayout forward_layout(int Lmax, int nx_rows, int64_t K) {
  FwdLayout l;
  l.prog = align16((size_t)Lmax * 4);
  l.cval = l.prog + 16 * (size_t)Lmax;
  l.xvar = l.cval + align16((size_t)Lmax * (size_t)K * sizeof(T));
  l.xrow = l.xvar + (nx_rows > 0 ? kMaxVarRows * 4 : 0);
  l.rows = l.xrow + (size_t)nx_rows * kRowBytes;
  l.bytes = l.rows + (size_t)table_rows<T>(Lmax) * kRowBytes;
  return l;
}

// Operand word: a row (offset of the row; the lane's part follows from the path), or the
// entries of a constant (bit 31).
constexpr uint32_t kConstOperand = 0x80000000u;

template <typename T, int kMode, bool kVec>
__global__ void __launch_bounds__(256) eval_forward_kernel(const T* __restrict__ X, int64_t N, int64_t n_x,
                                                           const uint32_t* __restrict__ desc,
                                                           const int32_t* __restrict__ meta,
                                                           const int32_t* __restrict__ order, int64_t B,
                                                           int64_t M, int Llo, int Lhi, int nx_rows,
                                                           const T* __restrict__ C, int64_t c_sb, int64_t c_sm,
                                                           int64_t c_sk, int64_t K_, int64_t slice, int64_t nslices,
                                                           T* __restrict__ cache) {
  constexpr int V = Pack<T>::V;
  constexpr int G = V / 2;  // values per lane where the rows do not hold V
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr bool kMulti = kMode == kFlat;
  const int64_t K = kMulti ? K_ : 1;            // sets in one pass (one: the index arithmetic folds)
  const int64_t es = kMode == kStrided ? K_ : 1;  // elements between the values of a unit
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const FwdLayout fl = forward_layout<T>(Lhi, nx_rows, K);
  const struct { uint32_t prog, cval, xvar, xrow, rows; } ly{(uint32_t)fl.prog, (uint32_t)fl.cval, (uint32_t)fl.xvar,
                                                             (uint32_t)fl.xrow, (uint32_t)fl.rows};
  const int R = table_rows<T>(Lhi);
  unsigned char* wb = smem + (size_t)warp * fl.bytes;
  uint32_t* tape = reinterpret_cast<uint32_t*>(wb);
  uint4* prog = reinterpret_cast<uint4*>(wb + ly.prog);
  uint32_t* leaf = reinterpret_cast<uint32_t*>(wb + ly.cval) - 1;  // leaf j at leaf[-j]
  T* cval = reinterpret_cast<T*>(wb + ly.cval);
  const unsigned below = (1u << lane) - 1u;
  const int64_t total = N * K, rs = total * es;  // values per node of a unit, elements per node
  const int64_t sets = kMode == kStrided ? K_ : 1, units = B * sets * nslices;
  for (int64_t u = (int64_t)blockIdx.x * nwarp + warp; u < units; u += (int64_t)gridDim.x * nwarp) {
    const int64_t ts = u / nslices, sl = u - ts * nslices;
    const int64_t ti = kMode == kStrided ? ts / sets : ts, set = ts - ti * sets;
    const int64_t b = order ? (int64_t)order[ti] : ti;
    const int L = meta[b * 4];
    if (L <= Llo || L > Lhi) continue;  // another class's grid takes it (warp-uniform)
    __syncwarp();                       // every lane is done with the previous unit's tables
    for (int k = lane; k < L; k += 32) tape[k] = desc[b * M + k];
    __syncwarp();
    // the rows: while the program is built their place holds the scratch of stack_rows
    int* row = reinterpret_cast<int*>(wb + ly.rows);
    int* xvar = reinterpret_cast<int*>(wb + ly.xvar);  // variable of each row, where not the row's number
    // few points: no pass of 32 V values, so rows are not short and stack order is not looked for
    const bool few = total <= 16 * V;
    int need = few ? -1 : stack_rows(tape, L, lane, row + L, row);
    // variables of the tape in rows: row v for variable v, or the distinct ones in the order found
    const bool by_number = n_x <= nx_rows;
    unsigned used = 0;
    int nvr = 0;  // rows taken
    for (int k0 = 0; k0 < L; k0 += 32) {
      const int k = k0 + lane;
      const bool isvar = k < L && code_of(tape[k]) == VAR;
      const int var = isvar ? child0(tape[k]) : 0;
      if (by_number) {
        used |= __reduce_or_sync(0xffffffffu, isvar ? 1u << (var & 31) : 0u);
        nvr = max(nvr, __reduce_max_sync(0xffffffffu, isvar ? var + 1 : 0));
      } else if (nvr <= nx_rows) {
        int at = -1;  // its row
        for (int r = 0; r < nvr; ++r) at = isvar && xvar[r] == var ? r : at;
        const unsigned same = __match_any_sync(0xffffffffu, isvar ? var : -1 - lane);
        const bool fresh = isvar && at < 0 && (same & below) == 0;
        const unsigned mf = __ballot_sync(0xffffffffu, fresh);
        if (fresh) {
          at = nvr + __popc(mf & below);
          if (at < nx_rows) xvar[at] = var;
        }
        at = __shfl_sync(0xffffffffu, at, __ffs((int)same) - 1);
        if (isvar) row[k] = at;
        nvr += __popc(mf);
        __syncwarp();
      }
    }
    // more variables than rows: every variable leaf takes a row of its own among the operators'
    const bool own_rows = nvr > nx_rows;
    const uint32_t vrow = own_rows ? ly.rows : ly.xrow;
    if (own_rows) {
      need = -1;
      used = 0;
      nvr = 0;
    }
    if (need < 0) {  // a row for each operator (and such leaf)
      need = 0;
      for (int k0 = 0; k0 < L; k0 += 32) {
        const int k = k0 + lane;
        const int code = k < L ? code_of(tape[k]) : ZERO;
        const bool has = is_op_code(code) || (own_rows && code == VAR);
        const unsigned mh = __ballot_sync(0xffffffffu, has);
        if (has) row[k] = need + __popc(mh & below);
        need += __popc(mh);
      }
      __syncwarp();
    }
    // values per lane: as many as the rows hold
    const int VV = need <= R && !few ? V : G > 1 && need * G <= R * V && total > 32 ? G : 1;
    const uint32_t row_bytes = 32u * (uint32_t)VV * (uint32_t)sizeof(T);
    // a leaf's constant index is its position among the broadcast leaves (written first: the
    // program's operand words need it)
    int nleaf = 0, nbc = 0;
    for (int k0 = 0; k0 < L; k0 += 32) {
      const int k = k0 + lane;
      const int code = k < L ? code_of(tape[k]) : NO_OP;
      const bool isleaf = !is_op_code(code), isvar = code == VAR;
      const unsigned ml = __ballot_sync(0xffffffffu, isleaf), mb = __ballot_sync(0xffffffffu, isleaf && !isvar);
      const int j = nbc + __popc(mb & below);
      if (isleaf) {
        int xr = 0;  // a variable's row
        if (isvar) {
          xr = by_number && !own_rows ? child0(tape[k]) : row[k];
          row[k] = xr;
        }
        const uint32_t idx = isvar ? (uint32_t)xr : (uint32_t)j;
        leaf[-(nleaf + __popc(ml & below))] = (uint32_t)k | (isvar ? 1u << 12 : 0u) | (idx << 13);
        if (!isvar) {
          row[k] = j;  // a broadcast leaf has no row: its place holds the constant index
          const T fixed = code == LEARNABLE ? T(0) : node_value<T>(code, T(0), T(0), T(0), T(0));
          for (int64_t kk = 0; kk < K; ++kk)
            cval[(int64_t)j * K + kk] =
                code == LEARNABLE ? __ldg(C + b * c_sb + (int64_t)k * c_sm + (set + kk) * c_sk) : fixed;
        }
      }
      nleaf += __popc(ml);
      nbc += __popc(mb);
    }
    __syncwarp();
    auto operand = [&](int c) -> uint32_t {
      const int cc = code_of(tape[c]);
      if (is_op_code(cc)) return ly.rows + (uint32_t)row[c] * row_bytes;
      if (cc == VAR) return vrow + (uint32_t)row[c] * row_bytes;
      return kConstOperand | (ly.cval + (uint32_t)row[c] * (uint32_t)K * (uint32_t)sizeof(T));
    };
    int nop = 0;
    for (int k0 = 0; k0 < L; k0 += 32) {
      const int k = k0 + lane;
      const uint32_t d = k < L ? tape[k] : 0u;
      const int code = code_of(d), ar = arity_of(code);
      const bool isop = k < L && is_op_code(code);
      const unsigned mo = __ballot_sync(0xffffffffu, isop);
      if (isop) {
        // an operand that is not there reads the node's own row (its value is not used)
        const uint32_t own = ly.rows + (uint32_t)row[k] * row_bytes;
        prog[nop + __popc(mo & below)] = make_uint4((uint32_t)dense_op(code) | ((uint32_t)k << 8), own,
                                                    ar >= 1 ? operand(child0(d)) : own, ar == 2 ? operand(child1(d)) : own);
      }
      nop += __popc(mo);
    }
    __syncwarp();
    T* out = cache + (size_t)b * M * rs + set;
    const int64_t e0 = sl * slice, e1 = min(total, e0 + slice);
    auto passes = [&](auto width) {
      constexpr int W = decltype(width)::value;  // values per lane
      for (int64_t base = e0; base < e1; base += 32 * W) {
        // element, point and constant-set index of each of the lane's values
        int64_t p[W];
        uint32_t kko[W];
        bool valid[W];
        int64_t n[W];
#pragma unroll
        for (int v = 0; v < W; ++v) {
          p[v] = base + (kVec ? lane * W + v : 32 * v + lane);
          valid[v] = p[v] < e1;
          const int64_t q = valid[v] ? p[v] : e1 - 1;
          n[v] = !kMulti ? q : total <= (int64_t)0xffffffff ? (int64_t)((uint32_t)q / (uint32_t)K) : q / K;
          kko[v] = kMulti ? (uint32_t)(q - n[v] * K) * (uint32_t)sizeof(T) : 0u;
        }
        unsigned char* const mine = wb + lane * (W * (int)sizeof(T));
        auto put = [&](int64_t k, const T (&x)[W]) {
          T* o = out + k * rs;
          if (kVec) {  // the row's elements come in whole packs
            if (valid[0]) stream_part<T, W>(o + p[0], x);
          } else {
#pragma unroll
            for (int v = 0; v < W; ++v)
              if (valid[v]) __stcs(o + p[v] * es, x[v]);
          }
        };
        auto constant = [&](uint32_t off, T (&x)[W]) {
#pragma unroll
          for (int v = 0; v < W; ++v) x[v] = *reinterpret_cast<const T*>(wb + off + kko[v]);
        };
        auto fetch = [&](uint32_t w, T (&x)[W]) {
          if (w & kConstOperand) constant(w & ~kConstOperand, x);
          else load_part<T, W>(mine + w, x);
        };
        auto variable = [&](int var, T (&x)[W]) {
#pragma unroll
          for (int v = 0; v < W; ++v) x[v] = __ldg(X + n[v] * n_x + var);
        };
        if (by_number) {
          for (unsigned m = used; m; m &= m - 1) {
            const int var = __ffs((int)m) - 1;
            T x[W];
            variable(var, x);
            store_part<T, W>(mine + vrow + (uint32_t)var * row_bytes, x);
          }
        } else {
          for (int r = 0; r < nvr; ++r) {
            T x[W];
            variable(xvar[r], x);
            store_part<T, W>(mine + vrow + (uint32_t)r * row_bytes, x);
          }
        }
        if (own_rows) {
          for (int j = 0; j < nleaf; ++j) {
            const uint32_t w = leaf[-j];
            T x[W];
            if (!(w & (1u << 12))) continue;
            variable(child0(tape[w & 0xfffu]), x);
            store_part<T, W>(mine + vrow + (w >> 13) * row_bytes, x);
          }
        }
        for (int j = 0; j < nleaf; ++j) {
          const uint32_t w = leaf[-j];
          T x[W];
          if (w & (1u << 12)) load_part<T, W>(mine + vrow + (w >> 13) * row_bytes, x);
          else constant(ly.cval + (w >> 13) * (uint32_t)K * (uint32_t)sizeof(T), x);
          put(w & 0xfffu, x);
        }
        for (int i = 0; i < nop; ++i) {
          const uint4 w = prog[i];
          T a[W], c[W], r[W];
          fetch(w.z, a);
          fetch(w.w, c);
          op_value_v<T, W>((int)(w.x & 0xffu), a, c, r);
          store_part<T, W>(mine + w.y, r);
          put(w.x >> 8, r);
        }
      }
    };
    if (VV == V) passes(std::integral_constant<int, V>{});
    else if (G > 1 && VV == G) passes(std::integral_constant<int, G>{});
    else passes(std::integral_constant<int, 1>{});
    // rows after the last real node are filled with NaN by pad_fill_kernel
  }
}

// ------------------------------------------------------------------------------------
// Host launchers
// ------------------------------------------------------------------------------------
int device_sm_count() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 148;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 148;
  return sms;
}

int max_dyn_smem() {
  int dev = 0, v = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 48 * 1024;
  if (cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) return 48 * 1024;
  return v;
}

int max_sm_smem() {
  int dev = 0, v = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 48 * 1024;
  if (cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) != cudaSuccess) return 48 * 1024;
  return v;
}

int resident_ctas(const void* kern, int threads, size_t smem) {
  struct Entry {
    const void* kern;
    int dev, threads, ctas;
    size_t smem;
  };
  constexpr size_t kEntries = 256;  // direct-mapped: a shape that collides is asked for again
  static Entry table[kEntries] = {};
  static std::mutex mu;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  const size_t h = ((reinterpret_cast<uintptr_t>(kern) >> 4) * 31 + (size_t)dev * 17 + (size_t)threads + smem / 16 * 7) % kEntries;
  {
    std::lock_guard<std::mutex> hold(mu);
    const Entry& e = table[h];
    if (e.kern == kern && e.dev == dev && e.threads == threads && e.smem == smem) return e.ctas;
  }
  int ctas = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ctas, kern, threads, smem) != cudaSuccess) return 0;
  std::lock_guard<std::mutex> hold(mu);
  table[h] = Entry{kern, dev, threads, ctas, smem};
  return ctas;
}

int check_tape_args(int64_t B, int64_t M) {
  if (B < 0 || M < 0) { set_error("negative size"); return SR_ERR_INVALID_ARGUMENT; }
  if (M > kMaxNodes) {
    set_error("tapes longer than %d nodes are not supported (M=%lld)", kMaxNodes, (long long)M);
    return SR_ERR_UNSUPPORTED;
  }
  return SR_OK;
}

Aux* aux_for_current_device() {
  constexpr int kMaxDevices = 64;
  static Aux aux[kMaxDevices];
  static std::mutex create_mu;
  int dev = 0;
  if (cuda_check(cudaGetDevice(&dev), "cudaGetDevice")) return nullptr;
  if (dev < 0 || dev >= kMaxDevices) {
    set_error("device index %d out of range", dev);
    return nullptr;
  }
  std::lock_guard<std::mutex> hold(create_mu);
  Aux& a = aux[dev];
  if (!a.stream) {
    // created into locals and published together, so a failure leaves nothing behind
    cudaStream_t s = nullptr;
    cudaEvent_t f = nullptr, j = nullptr;
    int rc = cuda_check(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking), "side stream");
    if (!rc) rc = cuda_check(cudaEventCreateWithFlags(&f, cudaEventDisableTiming), "fork event");
    if (!rc) rc = cuda_check(cudaEventCreateWithFlags(&j, cudaEventDisableTiming), "join event");
    if (rc) {
      if (j) cudaEventDestroy(j);
      if (f) cudaEventDestroy(f);
      if (s) cudaStreamDestroy(s);
      return nullptr;
    }
    a.fork = f;
    a.join = j;
    a.stream = s;
  }
  return &a;
}

template <bool kStage>
static int launch_compile(const int64_t* ops, const int64_t* ch, int64_t B, int64_t M, int64_t ops_sb,
                          int64_t ops_sm, int64_t ch_sb, int64_t ch_sm, int64_t ch_si, int32_t n_vars,
                          uint32_t* desc, int32_t* meta, int32_t* status, void* stream) {
  int rc = check_tape_args(B, M);
  if (rc) return rc;
  if (!status || (B > 0 && M > 0 && (!ops || !ch)) || (kStage && B > 0 && (!meta || (M > 0 && !desc)))) {
    set_error("null pointer argument");
    return SR_ERR_INVALID_ARGUMENT;
  }
  if (n_vars < 0 || n_vars > SR_MAX_VARS) {
    set_error("n_vars out of range (%d)", n_vars);
    return SR_ERR_UNSUPPORTED;
  }
  cudaStream_t st = as_stream(stream);
  rc = cuda_check(cudaMemsetAsync(status, 0, (kStage ? 8 : 1) * sizeof(int32_t), st), "status reset");
  if (rc || B == 0) return rc;
  const int threads = 256;
  int64_t blocks = (B + 7) / 8;
  const int64_t cap = (int64_t)device_sm_count() * 8;
  if (blocks > cap) blocks = cap;
  tape_compile_kernel<kStage><<<(unsigned)blocks, threads, 0, st>>>(ops, ch, B, M, ops_sb, ops_sm, ch_sb, ch_sm,
                                                                    ch_si, n_vars, desc, meta, status);
  return launch_check("tape_compile_kernel");
}

bool pick_shape(const void* kern, size_t per_warp, int64_t work_items, Shape& sh, size_t reserve) {
  const int limit = max_dyn_smem();
  const int sm_bytes = max_sm_smem();
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, limit) != cudaSuccess) return false;
  if (reserve && cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                                      cudaSharedmemCarveoutMaxShared) != cudaSuccess)
    return false;
  // the CTA size (8, 4, 2 or 1 warps) that keeps the most warps resident per SM
  int w = 0, per_sm = 0, best = 0;
  for (int cand = 8; cand >= 1; cand >>= 1) {
    if (per_warp * cand > (size_t)limit) continue;
    int blocks = resident_ctas(kern, cand * 32, per_warp * cand);
    // every CTA takes 1 KB of its SM's shared memory besides its own
    const int room = (int)(((size_t)sm_bytes - reserve) / (per_warp * cand + 1024));
    if (reserve && blocks > room && room > 0) blocks = room;
    if (blocks * cand > best) {
      best = blocks * cand;
      w = cand;
      per_sm = blocks;
    }
  }
  if (w == 0) return false;
  sh.warps = w;
  sh.smem = per_warp * w;
  int64_t blocks = (int64_t)device_sm_count() * per_sm;
  const int64_t need = (work_items + w - 1) / w;
  sh.blocks = blocks < need ? blocks : need;
  if (sh.blocks < 1) sh.blocks = 1;
  return true;
}

// Points a forward unit covers: whole tapes while the batch alone gives every resident warp
// several units (the program is compiled once per unit), else as few passes as it takes.
template <typename T>
static int64_t forward_slice(int64_t B, int64_t total) {
  constexpr int64_t pass = 32 * Pack<T>::V;
  const int64_t passes = (total + pass - 1) / pass, want = (int64_t)device_sm_count() * 20 * 4;
  int64_t per = passes * B / want;
  if (per < 1) per = 1;
  if (per > passes) per = passes;
  return per * pass;
}

template <typename T>
static int launch_forward(const T* X, int64_t N, int64_t n_x, const uint32_t* desc, const int32_t* meta,
                          const int32_t* order, int64_t B, int64_t M, int32_t max_len, const T* C, int64_t c_sb,
                          int64_t c_sm, int64_t c_sk, int64_t K, T* cache, void* stream) {
  int rc = check_tape_args(B, M);
  if (rc) return rc;
  if (N < 0 || n_x < 0 || K < 0) { set_error("negative size"); return SR_ERR_INVALID_ARGUMENT; }
  if (B == 0 || M == 0 || N == 0 || K == 0) return SR_OK;
  if (!X && n_x > 0) { set_error("null X"); return SR_ERR_INVALID_ARGUMENT; }
  if (!desc || !meta || !C || !cache) { set_error("null pointer argument"); return SR_ERR_INVALID_ARGUMENT; }
  const int Lmax = (max_len > 0 && max_len < M) ? max_len : (int)M;
  const bool aligned = reinterpret_cast<uintptr_t>(cache) % 16 == 0;
  cudaStream_t st = as_stream(stream);
  // a small output is filled on the caller's stream: the fork and join take longer (8 MB are
  // written in a few microseconds)
  const bool fork = (double)B * M * N * K * sizeof(T) > (double)(8 << 20);
  SideStream side(fork, st);
  rc = side.begin();
  if (rc) return rc;
  {
    // one warp per SM, placed before the forward grids, which leave its shared memory free
    int64_t fblocks = device_sm_count();
    if (fblocks > B) fblocks = B;
    // an SM cannot change its split of L1 and shared memory while a CTA is on it: both kernels
    // ask for the largest shared memory, or whichever comes first locks the other out
    rc = cuda_check(cudaFuncSetAttribute(pad_fill_kernel<T>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                         cudaSharedmemCarveoutMaxShared), "fill carveout");
    pad_fill_kernel<T><<<(unsigned)fblocks, 32, 0, side.stream()>>>(meta, B, M, N * K, Lmax, cache);
    if (!rc) rc = launch_check("pad_fill_kernel");
  }
  // one persistent grid per class of tape lengths, as in launch_backward
  int cls[3][2], nc = 0;
  if (Lmax > 32) { cls[nc][0] = 32; cls[nc][1] = Lmax; ++nc; }
  if (Lmax > 16) { cls[nc][0] = 16; cls[nc][1] = Lmax < 32 ? Lmax : 32; ++nc; }
  cls[nc][0] = -1; cls[nc][1] = Lmax < 16 ? Lmax : 16; ++nc;
  for (int ci = 0; ci < nc && !rc; ++ci) {
    const int Lhi = cls[ci][1];
    // rows for the variables unless a long tape needs their place (its tapes then take the
    // general path); all sets in one pass while their constants take little of the table
    int nx_rows = (int)(n_x < kMaxVarRows ? n_x : kMaxVarRows);
    if (forward_layout<T>(Lhi, nx_rows, 1).bytes > (size_t)max_dyn_smem()) nx_rows = 0;
    const int mode = K == 1 ? kSingle : (K <= 64 && forward_layout<T>(Lhi, nx_rows, K).bytes <= (56u << 10) ? kFlat : kStrided);
    const int64_t flat = mode == kFlat ? K : 1, sets = mode == kStrided ? K : 1, total = N * flat;
    const int64_t slice = forward_slice<T>(B * sets, total), nslices = (total + slice - 1) / slice;
    const bool vec = mode != kStrided && aligned && total % Pack<T>::V == 0;
    auto kern = mode == kStrided ? eval_forward_kernel<T, kStrided, false>
                : mode == kFlat  ? (vec ? eval_forward_kernel<T, kFlat, true> : eval_forward_kernel<T, kFlat, false>)
                                 : (vec ? eval_forward_kernel<T, kSingle, true> : eval_forward_kernel<T, kSingle, false>);
    Shape sh;
    if (!pick_shape(reinterpret_cast<const void*>(kern), forward_layout<T>(Lhi, nx_rows, flat).bytes,
                    B * sets * nslices, sh, kFillReserve)) {
      set_error("tape of %d nodes does not fit in shared memory", Lhi);
      rc = SR_ERR_UNSUPPORTED;
      break;
    }
    kern<<<(unsigned)sh.blocks, sh.warps * 32, sh.smem, st>>>(X, N, n_x, desc, meta, order, B, M, cls[ci][0], Lhi,
                                                             nx_rows, C, c_sb, c_sm, c_sk, K, slice, nslices, cache);
    rc = launch_check("eval_forward_kernel");
  }
  const int rj = side.end();
  return rc ? rc : rj;
}

}  // namespace sr

// ------------------------------------------------------------------------------------
// C ABI
// ------------------------------------------------------------------------------------
extern "C" {

const char* sr_last_error(void) { return sr::g_err; }

const char* sr_version(void) { return "sr_gb300 0.1 (sm_103a)"; }

int sr_validate(const int64_t* ops, const int64_t* ch, int64_t B, int64_t M, int64_t ops_sb, int64_t ops_sm,
                int64_t ch_sb, int64_t ch_sm, int64_t ch_si, int32_t* status, void* stream) {
  return sr::launch_compile<false>(ops, ch, B, M, ops_sb, ops_sm, ch_sb, ch_sm, ch_si, 0, nullptr, nullptr, status,
                                   stream);
}

int sr_tape_compile(const int64_t* ops, const int64_t* ch, int64_t B, int64_t M, int64_t ops_sb, int64_t ops_sm,
                    int64_t ch_sb, int64_t ch_sm, int64_t ch_si, int32_t n_vars, uint32_t* desc, int32_t* meta,
                    int32_t* stats, void* stream) {
  return sr::launch_compile<true>(ops, ch, B, M, ops_sb, ops_sm, ch_sb, ch_sm, ch_si, n_vars, desc, meta, stats,
                                  stream);
}

int sr_tape_order(const int32_t* meta, int64_t B, int64_t M, int32_t column, int32_t* order, void* stream) {
  using namespace sr;
  int rc = check_tape_args(B, M);
  if (rc) return rc;
  if (column < 0 || column > 1 || B > INT32_MAX) { set_error("invalid column or too many tapes"); return SR_ERR_INVALID_ARGUMENT; }
  if (B == 0) return SR_OK;
  if (!meta || !order) { set_error("null pointer argument"); return SR_ERR_INVALID_ARGUMENT; }
  const int bins = (int)M + 1;
  cudaLaunchAttribute cluster;
  cluster.id = cudaLaunchAttributeClusterDimension;
  cluster.val.clusterDim.x = B > kOrderOneCta ? kOrderCtas : 1;
  cluster.val.clusterDim.y = cluster.val.clusterDim.z = 1;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(cluster.val.clusterDim.x);
  config.blockDim = dim3(1024);
  config.dynamicSmemBytes = 2 * bins * sizeof(int);
  config.stream = as_stream(stream);
  config.attrs = &cluster;
  config.numAttrs = 1;
  return cuda_check(cudaLaunchKernelEx(&config, tape_order_kernel, meta, B, (int)column, (int)column, bins, order),
                    "tape_order_kernel");
}

int sr_any_nonzero(const int64_t* words, int64_t n, int32_t* out, void* stream) {
  using namespace sr;
  if (n < 0 || !out || (n > 0 && !words)) { set_error("invalid arguments"); return SR_ERR_INVALID_ARGUMENT; }
  const int rc = cuda_check(cudaMemsetAsync(out, 0, sizeof(int32_t), as_stream(stream)), "flag reset");
  if (rc || n == 0) return rc;
  int64_t blocks = (n + 2047) / 2048;
  const int64_t cap = (int64_t)device_sm_count() * 8;
  if (blocks > cap) blocks = cap;
  any_nonzero_kernel<<<(unsigned)blocks, 256, 0, as_stream(stream)>>>(words, n, out);
  return launch_check("any_nonzero_kernel");
}

int sr_eval_forward_f32(const float* X, int64_t N, int64_t n_x, const uint32_t* desc, const int32_t* meta,
                        const int32_t* order, int64_t B, int64_t M, int32_t max_len, const float* C, int64_t c_sb,
                        int64_t c_sm, float* cache, void* stream) {
  return sr::launch_forward<float>(X, N, n_x, desc, meta, order, B, M, max_len, C, c_sb, c_sm, 0, 1, cache, stream);
}

int sr_eval_forward_f64(const double* X, int64_t N, int64_t n_x, const uint32_t* desc, const int32_t* meta,
                        const int32_t* order, int64_t B, int64_t M, int32_t max_len, const double* C, int64_t c_sb,
                        int64_t c_sm, double* cache, void* stream) {
  return sr::launch_forward<double>(X, N, n_x, desc, meta, order, B, M, max_len, C, c_sb, c_sm, 0, 1, cache, stream);
}

int sr_eval_forward_multi_f32(const float* X, int64_t N, int64_t n_x, const uint32_t* desc, const int32_t* meta,
                              const int32_t* order, int64_t B, int64_t M, int32_t max_len, const float* C,
                              int64_t c_sb, int64_t c_sm, int64_t c_sk, int64_t K, float* cache, void* stream) {
  return sr::launch_forward<float>(X, N, n_x, desc, meta, order, B, M, max_len, C, c_sb, c_sm, c_sk, K, cache, stream);
}

int sr_eval_forward_multi_f64(const double* X, int64_t N, int64_t n_x, const uint32_t* desc, const int32_t* meta,
                              const int32_t* order, int64_t B, int64_t M, int32_t max_len, const double* C,
                              int64_t c_sb, int64_t c_sm, int64_t c_sk, int64_t K, double* cache, void* stream) {
  return sr::launch_forward<double>(X, N, n_x, desc, meta, order, B, M, max_len, C, c_sb, c_sm, c_sk, K, cache,
                                    stream);
}

}  // extern "C"
