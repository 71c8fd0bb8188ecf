// sr_adjoint.cu -- adjoint of the forward evaluation for a dense output gradient: the
// padding-row check and the adjoint proper.
#include "sr_eval.cuh"

namespace sr {

// ------------------------------------------------------------------------------------
// Adjoint for a dense grad_out: the padding-row check and the adjoint proper, run
// concurrently (the check streams the padding rows from HBM, the adjoint is bound by
// instruction latency).
// ------------------------------------------------------------------------------------

// Error precedence of the adjoint: a gradient on a NO_OP row (201) is reported over a
// zero denominator (204) whichever kernel finds it first, as in the reference, whose
// reverse loop meets the padding rows first.
__device__ __forceinline__ void report_adjoint(int* status, int code) {
  if (!code) return;
  const int prev = atomicCAS(status, 0, code);
  if (code == ERR_GRAD_ON_NO_OP && prev == ERR_DIV_BY_ZERO) atomicCAS(status, ERR_DIV_BY_ZERO, code);
}

// ---- padding rows: any nonzero output gradient on a NO_OP row is error 201 ----------
// Rows L..M-1 of a tape's (M, N) gradient block are one contiguous range.  One CTA per SM
// takes every gridDim-th tape: its last warp streams the ranges into a ring in shared memory
// with bulk copies, and the others look for a nonzero word (a float or double is nonzero when
// any bit but its sign is).  What bounds it: HBM reads, together with the adjoint's own.  The
// copies keep 32 KB of every SM in flight from one warp; the vector loads before it held
// 16 warps and a quarter of the registers that the adjoint beside it needs (65536 tapes: the
// two together 5.48 ms with them, 4.5 to 4.9 ms with the copies; 16384 tapes with 3 stages
// 1160 us, 4 stages 1046, 6 stages 1081).  Two adjoint CTAs leave an SM 4096 registers, too few
// for this CTA, so where it comes first one of them waits for it.  Three readers of 32 registers
// fit beside both: 4.08 ms, but 5.9 ms instead of 5.6 where every tape has a gradient, so they
// are not used.  Every wait gives up after about a second (status 601).
// A tape longer than the max_len the call was given is adjoined by no class grid: it
// is reported (status 602) instead of being skipped silently.
constexpr int kCheckWarps = 4;          // readers
constexpr int kCheckStages = 4;
constexpr int kCheckBytes = 8192;       // one bulk copy
constexpr size_t kCheckReserve = kCheckStages * kCheckBytes + 2048;  // shared memory of an SM its CTA takes
constexpr long long kCheckWaitCycles = 2000000000LL;  // about one second

__device__ __forceinline__ bool check_wait(uint32_t bar, uint32_t parity) {
  const long long t0 = clock64();
  while (true) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
    if (clock64() - t0 > kCheckWaitCycles) return false;
  }
}

template <typename T>
__global__ void __launch_bounds__((kCheckWarps + 1) * 32) padding_check_kernel(const T* __restrict__ gout,
                                                                              const int32_t* __restrict__ meta,
                                                                              int64_t B, int64_t M, int64_t N,
                                                                              int Lmax, int32_t* __restrict__ status) {
  __shared__ __align__(128) unsigned char ring[kCheckStages][kCheckBytes];
  __shared__ __align__(8) unsigned long long full[kCheckStages], empty[kCheckStages];
  __shared__ int bytes_of[kCheckStages];  // of the copy in each stage, 0: no more
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto addr = [](const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); };
  if (threadIdx.x == 0) {
    for (int i = 0; i < kCheckStages; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(addr(&full[i])), "r"(1) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(addr(&empty[i])), "r"(kCheckWarps) : "memory");
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  bool nz = false, stuck = false;
  if (warp == kCheckWarps) {
    // the range of a tape: elements before and after its 16-byte-aligned part are read here
    int64_t turn = 0;
    auto put = [&](const unsigned char* src, int bytes) {  // lane 0: one copy, or the end (bytes 0)
      const int st = (int)(turn % kCheckStages);
      if (turn >= kCheckStages && !check_wait(addr(&empty[st]), (uint32_t)((turn / kCheckStages - 1) & 1))) return false;
      bytes_of[st] = bytes;
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(addr(&full[st])), "r"(bytes) : "memory");
      if (bytes)
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                addr(ring[st])),
            "l"(src), "r"(bytes), "r"(addr(&full[st]))
            : "memory");
      ++turn;
      return true;
    };
    for (int64_t b = blockIdx.x; b < B && !stuck; b += gridDim.x) {
      const int64_t L = meta[b * 4];
      if (L > Lmax) {
        if (lane == 0) report(status, SR_TAPE_EXCEEDS_LAUNCH);
        continue;
      }
      // nothing more to find once a 201 is recorded
      if (__shfl_sync(0xffffffffu, *reinterpret_cast<volatile int32_t*>(status), 0) == ERR_GRAD_ON_NO_OP) break;
      const T* p = gout + (size_t)b * M * N + (size_t)L * N;
      const size_t count = (size_t)(M - L) * N;
      size_t head = ((16 - (reinterpret_cast<uintptr_t>(p) & 15)) & 15) / sizeof(T);
      if (head > count) head = count;
      const size_t body = (count - head) * sizeof(T) & ~size_t(15), tail = head + body / sizeof(T);
      if ((size_t)lane < head) nz |= __ldg(p + lane) != T(0);
      if (tail + lane < count) nz |= __ldg(p + tail + lane) != T(0);
      if (lane == 0) {
        const unsigned char* q = reinterpret_cast<const unsigned char*>(p + head);
        for (size_t off = 0; off < body && !stuck; off += kCheckBytes)
          stuck = !put(q + off, (int)(body - off < (size_t)kCheckBytes ? body - off : (size_t)kCheckBytes));
      }
      stuck = __any_sync(0xffffffffu, stuck);
    }
    // the end, and none of this CTA's copies in flight when it leaves
    if (lane == 0) {
      if (!stuck) stuck = !put(nullptr, 0);
      for (int64_t i = turn < kCheckStages ? 0 : turn - kCheckStages; i < turn; ++i)
        if (!check_wait(addr(&full[i % kCheckStages]), (uint32_t)((i / kCheckStages) & 1))) stuck = true;
    }
  } else {
    unsigned any = 0;
    for (int64_t turn = 0;; ++turn) {
      const int st = (int)(turn % kCheckStages);
      if (!check_wait(addr(&full[st]), (uint32_t)((turn / kCheckStages) & 1))) {
        stuck = true;
        break;
      }
      const int bytes = bytes_of[st];
      if (!bytes) break;
#pragma unroll 4
      for (int i = (warp * 32 + lane) * 16; i < bytes; i += kCheckWarps * 32 * 16) {
        const uint4 v = *reinterpret_cast<const uint4*>(ring[st] + i);
        // the word that holds the sign: every one of a float, the upper one of a double
        any |= sizeof(T) == 4 ? (v.x | v.y | v.z | v.w) & 0x7fffffffu : v.x | v.z | ((v.y | v.w) & 0x7fffffffu);
      }
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(addr(&empty[st])) : "memory");
    }
    nz = any != 0;
  }
  if (__any_sync(0xffffffffu, nz) && lane == 0) report_adjoint(status, ERR_GRAD_ON_NO_OP);
  if (__any_sync(0xffffffffu, stuck) && lane == 0) report(status, SR_MLP_TIMEOUT);
}

// ------------------------------------------------------------------------------------
// Adjoint.  Work unit = (tape, all or one of its constant sets), one warp or,
// for small batches, several warps of a CTA.  The unit's values per node (points, or points x
// sets, see SetMode) are cut into chunks of 32 consecutive ones; a warp sweeps V chunks at a
// time, V values per lane, so one decode and dispatch of a node serves all of them.
//
// Nothing is staged: the sweep visits the operator nodes from the last to the first, and
// for each it needs the values of its children (if its rule uses them) and the output
// gradients of its children, rows of the cache and of grad_out that a warp reads in full
// 128-byte lines.  They are loaded into registers one node ahead, so a node's arithmetic
// covers the latency of the next node's loads.  Only the adjoints of operator nodes between
// their parent's step and their own wait in shared memory, in the stack rows of stack_rows.
// What bounds it: the instructions of the sweep and the bytes of the real rows (read once
// each).  The kernel before it staged every grad_out and value row of a chunk in shared
// memory (256 bytes per node and warp: 12 warps per SM for 64 nodes) and swept one point per
// lane.  Measured with the check above: 16384 tapes of mean length 20 at N = 1024, 1390 to
// 1060 us; 1003 tapes at N = 777, 834 to 96 us; 512 float64 tapes at N = 1000, 1850 to 172 us;
// 1000 tapes at N = 256, K = 8, 1214 to 166 us.  (One warp per tape left most of the GPU idle
// in the last three.)  At 65536 tapes it is no faster: 4.3 ms became 4.5 to 4.9 with a gradient
// on the tapes of moderate values only, 4.9 became 5.7 with one on every tape.  A launch bound
// of three CTAs per SM (80 registers instead of 118) undoes the loads ahead: 1450 us.
//
// Sums keep one order whatever the split.  A child's adjoint is its output gradient plus its
// parent's contribution.  A constant's gradient is summed per residue of the point index mod
// 32 over the chunks in order, then by a lane butterfly.  With one set a chunk's lanes are the
// residues, and when several warps share a unit they write the chunks' terms to shared memory
// and add them in chunk order behind a barrier.  With K sets value p = n K + kk belongs to
// residue p mod 32 K, that is to lane p mod 32 of the chunks s with s mod K = class: a warp
// takes whole classes, so their sums are its own, and the set of a lane is fixed in a class.
//
// grad_X is an atomic sum over the tapes, constant sets and leaves.  A lane first adds up
// the leaves of a variable at its value, so that there is one atomic for all of them (and the
// sum over a tape's leaves has one order); more than 16 variables go straight to the atomics.
//
// Tapes whose child table is not that of a stack, or that need more rows than the table has,
// take one adjoint row per node, set to its output gradient before the sweep, and one value
// per lane.  So do calls without a cache, which recompute the node values into rows first.
// ------------------------------------------------------------------------------------

// Shared memory of a CTA: the tape words (offset 0); the program, from the front 16 bytes per
// operator and from the back 4 bytes per leaf without a parent; per node its row or constant
// index; the nodes of the learnable constants; the constants' values (learnable j at j, fixed
// f at L - 1 - f, one entry per set); the sums of ncap constants (32 K lanes each); the first
// error of each point residue; then per warp the adjoint rows, without a cache a value row
// per node, with several warps the terms of one pass, and with grad_X the sums of one pass
// for each variable.
struct AdjLayout {
  size_t prog, cidx, lcon, cval, acc, errs, warps, warp_bytes, vals, crow, xacc, bytes;
  int ncap;
};

template <typename T>
__host__ __device__ __forceinline__ AdjLayout adjoint_layout(int Lmax, int64_t K, int nwarp, bool recompute, int xrows) {
  AdjLayout l;
  // constants summed in one sweep: half the nodes of a tree are leaves, few of them
  // constants; a tape with more is swept again for the rest
  int cap = (Lmax + 1) / 2;
  if (cap > 12) cap = 12;
  const int64_t room = (int64_t)(24 << 10) / (K * 32 * (int64_t)sizeof(T));
  if (cap > room) cap = room < 1 ? 1 : (int)room;
  if (nwarp > 1 && cap > 8) cap = 8;
  l.ncap = cap;
  l.prog = align16((size_t)Lmax * 4);
  l.cidx = l.prog + 16 * (size_t)Lmax;
  l.lcon = l.cidx + align16((size_t)Lmax * 4);
  l.cval = l.lcon + align16((size_t)Lmax * 4);
  l.acc = l.cval + align16((size_t)Lmax * (size_t)K * sizeof(T));
  l.errs = l.acc + (size_t)cap * (size_t)K * 32 * sizeof(T);
  l.warps = l.errs + 32 * 8 + 32;
  l.vals = (size_t)table_rows<T>(Lmax) * kRowBytes;
  l.crow = l.vals + (recompute ? (size_t)Lmax * 32 * sizeof(T) : 0);
  l.xacc = l.crow + (nwarp > 1 ? (size_t)cap * kRowBytes : 0);
  l.warp_bytes = l.xacc + (size_t)xrows * kRowBytes;
  l.bytes = l.warps + (size_t)nwarp * l.warp_bytes;
  return l;
}

// Variables whose sums over the leaves are kept in rows.
__host__ __device__ __forceinline__ int x_sum_rows(int64_t n_x) { return n_x <= 16 ? (int)n_x : 0; }

// Program words of operator node k:
//   x: dense code (bits 0..4) | no parent (bit 5) | k << 8 | adjoint row << 20
//   y, z: for child 0 and 1: where its value comes from (bits 0..1: nowhere, its cache row,
//      a constant entry, the node's own cache row), the constant index (bits 2..13), where
//      its adjoint goes (bits 16..17: nowhere, a row, a constant's sum, grad_X), the row,
//      constant or variable index (bits 18..29)
//   w: child 0 | child 1 << 12
enum ValueFrom : uint32_t { kNoValue = 0, kChildRow = 1, kConstant = 2, kOwnRow = 3 };
enum AdjointTo : uint32_t { kNowhere = 0, kRow = 1, kSum = 2, kGradX = 3 };

// Whether the adjoint rule of an operator reads its operands' values (node_adjoint).
__device__ __forceinline__ bool reads_operands(int code) {
  return !(code == NO_OP || code == ADD || code == SUB || code == NEG || code == FLOOR || code == CEIL);
}

// The rule of an operator for V values at once, its contributions added to the children's
// output gradients s0 and s1 inside the operator's case, so that nothing but those values
// leaves the dispatch.  ep takes the first error of each value (two bits: 1 = 201, 2 = 204).
template <typename T, int V>
__device__ __forceinline__ void op_adjoint_onto(int d, const T (&g)[V], const T (&a)[V], const T (&b)[V], T (&s0)[V],
                                                T (&s1)[V], uint32_t& ep) {
  switch (d) {
#define SR_ADJOINT_ONTO_CASE(i)                                                                         \
  case i:                                                                                               \
    _Pragma("unroll") for (int q = 0; q < V; ++q) {                                                     \
      bool a0, a1;                                                                                      \
      T o0, o1;                                                                                         \
      const int e = node_adjoint<T>(op_of_dense(i), g[q], a[q], b[q], a[q], a0, o0, a1, o1);            \
      if (e && !(ep >> (2 * q) & 3u)) ep |= (e == ERR_DIV_BY_ZERO ? 2u : 1u) << (2 * q);                \
      if (a0) s0[q] = M_<T>::add(s0[q], o0);                                                            \
      if (a1) s1[q] = M_<T>::add(s1[q], o1);                                                            \
    }                                                                                                   \
    break;
    SR_DENSE_CASES(SR_ADJOINT_ONTO_CASE)
#undef SR_ADJOINT_ONTO_CASE
    default: break;
  }
}

// The general path over one class of a unit's chunks: one adjoint row per node and one value
// per lane.  Kept out of line: its code and registers would otherwise weigh on the sweep that
// nearly every tape takes (1050 us became 1486 for 16384 tapes, M = 64, N = 1024).
template <typename T>
struct GeneralSweep {
  const T *X, *Cc, *G;  // Cc: null without a cache
  T* gX;
  int64_t N, n_x, rs, es, total, K, set, cl, nq, rounds;
  const uint32_t* tape;
  const uint4* prog;
  const uint32_t* orphan;
  const int *cidx, *lcon;
  const T* cv;           // the lane's constant entries
  T *accl, *adj, *vals;  // the lane's sums, adjoint rows and value rows
  T* xs;                 // the lane's sums per variable, kRowBytes apart
  unsigned xused;
  T* crow;
  const unsigned char* crows;
  size_t warp_bytes;
  unsigned long long* errs;
  int L, nop, norph, g0, ng, lane, rank, ranks;
};

template <typename T, int kMode>
__device__ __noinline__ void general_sweep(const GeneralSweep<T>& q) {
  constexpr int V = Pack<T>::V;  // the stride of crow
  for (int64_t round = 0; round < q.rounds; ++round) {
    const int64_t p = 32 * (q.cl + q.K * (round * q.ranks + q.rank)) + q.lane;
    const bool valid = p < q.total;
    const int64_t pv = valid ? p : q.total - 1, n = kMode == kFlat ? pv / q.K : pv;
    for (int k = 0; k < q.L; ++k) q.adj[k * 32] = valid ? __ldg(q.G + (int64_t)k * q.rs + p * q.es) : T(0);
    // a node's value: a constant's entry, its cache row, or what is recomputed here
    auto node = [&](int k) -> T {
      const int code = code_of(q.tape[k]);
      if (!is_op_code(code) && code != VAR) return q.cv[(int64_t)q.cidx[k] * q.K];
      return q.Cc ? __ldg(q.Cc + (int64_t)k * q.rs + pv * q.es) : q.vals[k * 32];
    };
    if (!q.Cc) {
      for (int k = 0; k < q.L; ++k) {
        const uint32_t d = q.tape[k];
        const int code = code_of(d), ar = arity_of(code);
        if (code == VAR) q.vals[k * 32] = __ldg(q.X + n * q.n_x + child0(d));
        else if (is_op_code(code))
          q.vals[k * 32] =
              op_value<T>(dense_op(code), ar >= 1 ? node(child0(d)) : T(0), ar == 2 ? node(child1(d)) : T(0));
      }
    }
    int err = 0;
    for (int i = q.nop - 1; i >= 0; --i) {
      const uint4 w = q.prog[i];
      const int own = (int)(w.x >> 8 & 0xfffu), c0 = (int)(w.w & 0xfffu), c1 = (int)(w.w >> 12);
      const T a = (w.y & 3u) == kNoValue ? T(0) : node((w.y & 3u) == kOwnRow ? own : c0);
      const T b = (w.z & 3u) == kNoValue ? T(0) : node(c1);
      T o0, o1;
      bool a0, a1;
      const int e = op_adjoint<T>((int)(w.x & 31u), q.adj[own * 32], a, b, a, a0, o0, a1, o1);
      if (e && !err) err = e;
      if (a0 && (w.y >> 16 & 3u)) q.adj[c0 * 32] = M_<T>::add(q.adj[c0 * 32], o0);
      if (a1 && (w.z >> 16 & 3u)) q.adj[c1 * 32] = M_<T>::add(q.adj[c1 * 32], o1);
    }
    for (int j = 0; j < q.ng; ++j) {
      const T g = valid ? q.adj[q.lcon[q.g0 + j] * 32] : T(0);
      if (q.ranks > 1) q.crow[j * V * 32 + q.lane] = g;
      else if (g != T(0)) q.accl[j * 32] = M_<T>::add(q.accl[j * 32], g);
    }
    if (q.gX && valid) {  // in the order of the sweep, each variable leaf once
      auto leaf = [&](int k) {
        if (code_of(q.tape[k]) != VAR) return;
        const T g = q.adj[k * 32];
        q.adj[k * 32] = T(0);
        if (g == T(0)) return;
        const int var = child0(q.tape[k]);
        if (!q.xused) {
          atomicAdd(q.gX + n * q.n_x + var, g);
        } else {
          T* t = q.xs + var * (int)(kRowBytes / sizeof(T));
          *t = M_<T>::add(*t, g);
        }
      };
      for (int i = q.nop - 1; i >= 0; --i) {
        const uint4 w = q.prog[i];
        if (w.y >> 16 & 3u) leaf((int)(w.w & 0xfffu));
        if (w.z >> 16 & 3u) leaf((int)(w.w >> 12));
      }
      for (int j = 0; j < q.norph; ++j) leaf((int)(q.orphan[-j] & 0xfffu));
      for (unsigned m = q.xused; m; m &= m - 1) {
        const int var = __ffs((int)m) - 1;
        T* t = q.xs + var * (int)(kRowBytes / sizeof(T));
        if (*t != T(0)) atomicAdd(q.gX + n * q.n_x + var, *t);
        *t = T(0);
      }
    }
    if (err && valid) {
      const int64_t kk = kMode == kFlat ? p - n * q.K : q.set, pchunks = (q.N + 31) / 32;
      atomicMin(&q.errs[n & 31],
                ((unsigned long long)(kk * pchunks + n / 32) << 16) | (unsigned long long)err);
    }
    if (q.ranks > 1) {
      __syncthreads();
      for (int j = q.rank; j < q.ng; j += q.ranks) {
        T t = q.accl[j * 32];
        for (int r = 0; r < q.ranks && round * q.ranks + r < q.nq; ++r) {
          const T x = reinterpret_cast<const T*>(q.crows + (size_t)r * q.warp_bytes)[j * V * 32 + q.lane];
          if (x != T(0)) t = M_<T>::add(t, x);
        }
        q.accl[j * 32] = t;
      }
      __syncthreads();
    }
  }
}

template <typename T, int kMode>
__global__ void __launch_bounds__(256, 2) eval_adjoint_kernel(
    const T* __restrict__ X, const T* __restrict__ cache, int64_t N, int64_t n_x, const uint32_t* __restrict__ desc,
    const int32_t* __restrict__ meta, const int32_t* __restrict__ order, int64_t B, int64_t M, int Llo, int Lhi,
    const T* __restrict__ C, int64_t c_sb, int64_t c_sm, int64_t c_sk, int64_t Ktot, const T* __restrict__ gout,
    T* __restrict__ gC, T* __restrict__ gX, int32_t* __restrict__ status) {
  constexpr int V = Pack<T>::V;
  extern __shared__ __align__(16) unsigned char smem[];
  const int64_t K = kMode == kFlat ? Ktot : 1;       // sets of a unit
  const int64_t es = kMode == kStrided ? Ktot : 1;   // elements between its values
  const int64_t sets = kMode == kStrided ? Ktot : 1;
  const int64_t total = N * K, rs = total * es;      // values per node, elements per node
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const unsigned below = (1u << lane) - 1u;
  const int xrows = gX ? x_sum_rows(n_x) : 0;
  const AdjLayout ly = adjoint_layout<T>(Lhi, K, nwarp, !cache, xrows);
  const int ncap = ly.ncap;
  uint32_t* tape = reinterpret_cast<uint32_t*>(smem);
  uint4* prog = reinterpret_cast<uint4*>(smem + ly.prog);
  uint32_t* orphan = reinterpret_cast<uint32_t*>(smem + ly.cidx) - 1;  // leaf j without a parent at orphan[-j]
  int* cidx = reinterpret_cast<int*>(smem + ly.cidx);
  int* lcon = reinterpret_cast<int*>(smem + ly.lcon);
  T* cval = reinterpret_cast<T*>(smem + ly.cval);
  T* acc = reinterpret_cast<T*>(smem + ly.acc);
  unsigned long long* errs = reinterpret_cast<unsigned long long*>(smem + ly.errs);
  int* info = reinterpret_cast<int*>(smem + ly.errs + 32 * 8);  // operators, constants, orphans, stack order
  unsigned char* wb = smem + ly.warps + (size_t)warp * ly.warp_bytes;
  T* crow = reinterpret_cast<T*>(wb + ly.crow);
  // with one set the warps of a unit take turns over its passes (ranks), else whole classes
  const int ranks = kMode == kFlat ? 1 : nwarp, rank = kMode == kFlat ? 0 : warp;
  const int64_t nchunks = (total + 31) / 32, pchunks = (N + 31) / 32;

  // The units come longest first: a CTA takes them there and back (i, 2 G - 1 - i, 2 G + i, ...),
  // so that the ones with the longest first unit get the shortest next.
  const int64_t units = B * sets;
  for (int64_t turn = 0; turn * gridDim.x < units; ++turn) {
    const int64_t u = turn * gridDim.x + (turn & 1 ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
    if (u >= units) continue;
    const int64_t ti = kMode == kStrided ? u / sets : u, set = u - ti * sets;
    const int64_t b = order ? (int64_t)order[ti] : ti;
    const int L = meta[b * 4];
    if (L <= Llo || L > Lhi) continue;  // another class's grid takes it (the same in every thread)
    __syncthreads();                    // every warp is done with the previous unit's tables
    for (int k = threadIdx.x; k < L; k += blockDim.x) tape[k] = desc[b * M + k];
    if (threadIdx.x < 32) errs[threadIdx.x] = ~0ull;
    __syncthreads();
    if (warp == 0) {
      int* last = reinterpret_cast<int*>(wb);  // scratch in the rows' place
      int* parent = last + L + 1;
      const int need = stack_rows(tape, L, lane, last, cidx);
      // the general path also takes a tape of leaves alone, a call without a cache, and rows
      // of 4 GB or more (the sweep's row offsets have 32 bits)
      const bool stack = need >= 1 && need <= table_rows<T>(Lhi) && cache && rs <= (int64_t)0xffffffff / (int64_t)sizeof(T);
      for (int k = lane; k < L; k += 32) parent[k] = 0;
      __syncwarp();
      for (int k = lane; k < L; k += 32) {
        const uint32_t d = tape[k];
        const int ar = arity_of(code_of(d));
        if (ar >= 1) parent[child0(d)] = 1;
        if (ar == 2) parent[child1(d)] = 1;
      }
      __syncwarp();
      int ncon = 0, nfix = 0, norph = 0;
      unsigned used = 0;  // variables of the tape
      for (int k0 = 0; k0 < L; k0 += 32) {
        const int k = k0 + lane;
        const int code = k < L ? code_of(tape[k]) : NO_OP;
        const bool con = code == LEARNABLE, var = code == VAR, fix = !is_op_code(code) && !con && !var;
        const unsigned mc = __ballot_sync(0xffffffffu, con), mf = __ballot_sync(0xffffffffu, fix);
        const bool orph = (con || (var && gX)) && !parent[k];
        const unsigned mo = __ballot_sync(0xffffffffu, orph);
        used |= __reduce_or_sync(0xffffffffu, var ? 1u << (child0(tape[k]) & 31) : 0u);
        const int j = ncon + __popc(mc & below);
        if (con) {
          cidx[k] = j;
          lcon[j] = k;
        }
        if (fix) {
          const int f = L - 1 - (nfix + __popc(mf & below));
          cidx[k] = f;
          const T x = node_value<T>(code, T(0), T(0), T(0), T(0));
          for (int64_t kk = 0; kk < K; ++kk) cval[(int64_t)f * K + kk] = x;
        }
        if (orph)
          orphan[-(norph + __popc(mo & below))] =
              (uint32_t)k | (var ? 1u << 12 : 0u) | ((uint32_t)(var ? child0(tape[k]) : j) << 13);
        ncon += __popc(mc);
        nfix += __popc(mf);
        norph += __popc(mo);
      }
      __syncwarp();
      auto operand = [&](int code, int k, int c) -> uint32_t {
        const int cc = code_of(tape[c]);
        const bool op = is_op_code(cc), con = cc == LEARNABLE, var = cc == VAR;
        uint32_t w = 0;
        if (reads_operands(code)) {
          if (code == EXP) w = kOwnRow;  // its rule uses the node's own value
          else if (op || var) w = kChildRow;
          else w = kConstant | ((uint32_t)cidx[c] << 2);
        }
        if (!stack) {
          if (op || con || var) w |= (kRow << 16) | ((uint32_t)c << 18);
        } else if (op) {
          w |= (kRow << 16) | ((uint32_t)cidx[c] << 18);
        } else if (con) {
          w |= (kSum << 16) | ((uint32_t)cidx[c] << 18);
        } else if (var && gX) {
          w |= (kGradX << 16) | ((uint32_t)child0(tape[c]) << 18);
        }
        return w;
      };
      int nop = 0;
      for (int k0 = 0; k0 < L; k0 += 32) {
        const int k = k0 + lane;
        const uint32_t d = k < L ? tape[k] : 0u;
        const int code = code_of(d), ar = arity_of(code);
        const bool op = k < L && is_op_code(code);
        const unsigned mo = __ballot_sync(0xffffffffu, op);
        if (op) {
          uint4 w = make_uint4((uint32_t)dense_op(code) | ((uint32_t)k << 8) | ((uint32_t)(stack ? cidx[k] : k) << 20),
                               0u, 0u, 0u);
          if (!parent[k]) w.x |= 1u << 5;
          if (ar >= 1) {
            w.y = operand(code, k, child0(d));
            w.w = (uint32_t)child0(d);
          }
          if (ar == 2) {
            w.z = operand(code, k, child1(d));
            w.w |= (uint32_t)child1(d) << 12;
          }
          prog[nop + __popc(mo & below)] = w;
        }
        nop += __popc(mo);
      }
      if (lane == 0) {
        info[0] = nop;
        info[1] = ncon;
        info[2] = norph;
        info[3] = stack ? 1 : 0;
        info[4] = (int)used;
      }
    }
    __syncthreads();
    const int nop = info[0], ncon = info[1], norph = info[2];
    const bool stack = info[3] != 0;
    const unsigned xused = xrows ? (unsigned)info[4] : 0u;
    for (int64_t i = threadIdx.x; i < (int64_t)ncon * K; i += blockDim.x) {
      const int64_t j = i / K, kk = i - j * K;
      cval[i] = __ldg(C + b * c_sb + (int64_t)lcon[j] * c_sm + (set + kk) * c_sk);
    }
    // every other node's gradient is zero
    for (int64_t i = threadIdx.x; i < M * K; i += blockDim.x) {
      const int64_t k = i / K, kk = i - k * K;
      if (!(k < L && code_of(tape[k]) == LEARNABLE)) gC[(b * M + k) * Ktot + set + kk] = T(0);
    }
    const T* G = gout + (size_t)b * M * rs + set;
    const T* Cc = cache ? cache + (size_t)b * M * rs + set : nullptr;
    const int64_t vs = 32 * K * es;  // elements from one of a lane's values to the next
    const uint32_t row_bytes = (uint32_t)(rs * (int64_t)sizeof(T));
    const int Vp = stack ? V : 1;    // chunks in a pass

    // sweeps of ncap constants each: one, but for tapes with more of them
    for (int g0 = 0; g0 == 0 || g0 < ncon; g0 += ncap) {
      const int ng = min(ncap, ncon - g0);
      for (int i = threadIdx.x; i < ncap * (int)K * 32; i += blockDim.x) acc[i] = T(0);
      __syncthreads();
      T* const gXg = g0 == 0 ? gX : nullptr;
      for (int64_t cl = kMode == kFlat ? warp : 0; cl < K; cl += kMode == kFlat ? nwarp : 1) {
        const int64_t nq = cl < nchunks ? (nchunks - cl + K - 1) / K : 0;  // chunks of this class
        const int64_t rounds = (nq + (int64_t)ranks * Vp - 1) / ((int64_t)ranks * Vp);
        const int64_t kkl = kMode == kFlat ? (32 * cl + lane) % K : 0;
        const T* const cv = cval + kkl;
        T* const accl = acc + cl * ncap * 32 + lane;
        int64_t p0 = 0;    // value index of the lane's first value in this pass
        unsigned vm = 0;   // which of its values exist
        uint32_t ep = 0;   // first error of each value: two bits (1 = 201, 2 = 204)
        // a value's term of constant j
        auto add_constant = [&](uint32_t idx, const T (&val)[V]) {
          const int j = (int)idx - g0;
          if (j < 0 || j >= ng) return;
          if (ranks == 1) {
            T t = accl[j * 32];
#pragma unroll
            for (int v = 0; v < V; ++v)
              if ((vm >> v & 1u) && val[v] != T(0)) t = M_<T>::add(t, val[v]);
            accl[j * 32] = t;
          } else {
#pragma unroll
            for (int v = 0; v < V; ++v)
              if (v < Vp) crow[(j * V + v) * 32 + lane] = (vm >> v & 1u) ? val[v] : T(0);
          }
        };
        auto to_grad_x = [&](uint32_t var, const T (&val)[V]) {
#pragma unroll
          for (int v = 0; v < V; ++v) {
            if ((vm >> v & 1u) && val[v] != T(0)) {
              const int64_t p = p0 + v * 32 * K;
              atomicAdd(gXg + (kMode == kFlat ? p / K : p) * n_x + var, val[v]);
            }
          }
        };
        unsigned char* const xs = wb + ly.xacc + lane * 16;  // the lane's sums per variable
        auto add_variable = [&](uint32_t var, const T (&val)[V]) {
          if (!gXg) return;
          if (!xrows) return to_grad_x(var, val);
          T t[V];
          load16(xs + var * kRowBytes, t);
#pragma unroll
          for (int v = 0; v < V; ++v)
            if (val[v] != T(0)) t[v] = M_<T>::add(t[v], val[v]);
          store16(xs + var * kRowBytes, t);
        };
        auto clear_variables = [&]() {
          T zero[V];
#pragma unroll
          for (int v = 0; v < V; ++v) zero[v] = T(0);
          for (unsigned m = xused; m; m &= m - 1) store16(xs + (__ffs((int)m) - 1) * kRowBytes, zero);
        };
        if (gXg) clear_variables();
        auto place = [&](int64_t round, int64_t& p, unsigned& m) {
          const int64_t q0 = (round * ranks + rank) * Vp;
          p = 32 * (cl + K * q0) + lane;
          m = 0;
#pragma unroll
          for (int v = 0; v < V; ++v)
            if (v < Vp && p + v * 32 * K < total) m |= 1u << v;
        };
        auto row = [&](const T* at, uint32_t k, unsigned m, T (&x)[V]) {  // at: the lane's first value of node 0
          const T* r = reinterpret_cast<const T*>(reinterpret_cast<const char*>(at) + (uint64_t)k * row_bytes);
#pragma unroll
          for (int v = 0; v < V; ++v) x[v] = (m >> v & 1u) ? __ldg(r + v * vs) : T(0);
        };
        if (stack) {
          // next: the loads of the node to come (operand values, children's output gradients,
          // and its own for a node without a parent); cur: the node at hand
          struct Loads {
            uint4 w;
            T a[V], b[V], s0[V], s1[V], g[V];
          } next, cur;
          next.w = make_uint4(0u, 0u, 0u, 0u);
          auto value = [&](uint32_t w, uint32_t child, uint32_t own, const T* cp, unsigned m, T (&x)[V]) {
            const uint32_t from = w & 3u;
            if (from == kConstant) {
              const T t = cv[(int64_t)(w >> 2 & 0xfffu) * K];
#pragma unroll
              for (int v = 0; v < V; ++v) x[v] = t;
            } else if (from != kNoValue) {
              row(cp, from == kOwnRow ? own : child, m, x);
            }
          };
          // a child's adjoint: its output gradient plus the contribution
          auto give = [&](uint32_t w, const T (&val)[V]) {
            const uint32_t to = w >> 16 & 3u, idx = w >> 18 & 0xfffu;
            if (to == kRow) store16(wb + idx * kRowBytes + lane * 16, val);
            else if (to == kSum) add_constant(idx, val);
            else if (to == kGradX) add_variable(idx, val);
          };
          int64_t pl = 0;      // first value, and which exist, of the pass that is being loaded
          unsigned ml = 0;
          int64_t round = 0, rcur = 0;  // the pass that is being loaded, the pass at hand
          int in = nop - 1, icur = -1;  // the node to load next, the node at hand
          if (rounds > 0) place(0, pl, ml);
          while (true) {
            const bool more = round < rounds;
            cur = next;
            if (more) {
              next.w = prog[in];
              const uint32_t own = next.w.x >> 8 & 0xfffu, c0 = next.w.w & 0xfffu, c1 = next.w.w >> 12;
              const T *cp = Cc + pl * es, *gp = G + pl * es;
              value(next.w.y, c0, own, cp, ml, next.a);
              value(next.w.z, c1, own, cp, ml, next.b);
              if (next.w.y >> 16 & 3u) row(gp, c0, ml, next.s0);
              if (next.w.z >> 16 & 3u) row(gp, c1, ml, next.s1);
              if (next.w.x & 32u) row(gp, own, ml, next.g);
            }
            if (icur >= 0) {
              if (!(cur.w.x & 32u)) load16(wb + (cur.w.x >> 20) * kRowBytes + lane * 16, cur.g);
              op_adjoint_onto<T, V>((int)(cur.w.x & 31u), cur.g, cur.a, cur.b, cur.s0, cur.s1, ep);
              give(cur.w.y, cur.s0);
              give(cur.w.z, cur.s1);
              if (icur == 0) {  // the pass ends
                for (int j = 0; j < norph; ++j) {  // leaves without a parent: their output gradient alone
                  const uint32_t w = orphan[-j];
                  T val[V];
                  row(G + p0 * es, w & 0xfffu, vm, val);
                  if (w & (1u << 12)) add_variable(w >> 13, val);
                  else add_constant(w >> 13, val);
                }
                if (gXg && xused) {
                  for (unsigned m = xused; m; m &= m - 1) {
                    T t[V];
                    load16(xs + (__ffs((int)m) - 1) * kRowBytes, t);
                    to_grad_x((uint32_t)(__ffs((int)m) - 1), t);
                  }
                  clear_variables();
                }
                if (__any_sync(0xffffffffu, ep != 0)) {
#pragma unroll
                  for (int v = 0; v < V; ++v) {
                    const uint32_t e = ep >> (2 * v) & 3u;
                    if (e && (vm >> v & 1u)) {
                      const int64_t p = p0 + v * 32 * K, n = kMode == kFlat ? p / K : p;
                      const int64_t kk = kMode == kFlat ? p - n * K : set;
                      atomicMin(&errs[n & 31], ((unsigned long long)(kk * pchunks + n / 32) << 16) |
                                                   (unsigned long long)(e == 2 ? ERR_DIV_BY_ZERO : ERR_GRAD_ON_NO_OP));
                    }
                  }
                  ep = 0;
                }
                if (ranks > 1) {
                  __syncthreads();
                  for (int j = rank; j < ng; j += ranks) {
                    T t = accl[j * 32];
                    for (int r = 0; r < ranks; ++r) {
                      const T* cr = reinterpret_cast<const T*>(smem + ly.warps + (size_t)r * ly.warp_bytes + ly.crow);
                      const int64_t q0 = (rcur * ranks + r) * V;
#pragma unroll
                      for (int v = 0; v < V; ++v) {
                        if (q0 + v < nq) {
                          const T x = cr[(j * V + v) * 32 + lane];
                          if (x != T(0)) t = M_<T>::add(t, x);
                        }
                      }
                    }
                    accl[j * 32] = t;
                  }
                  __syncthreads();
                }
              }
            }
            if (!more) break;
            if (in == nop - 1) {  // the first node of a pass is loaded: the pass begins
              p0 = pl;
              vm = ml;
              rcur = round;
            }
            icur = in;
            if (--in < 0) {
              in = nop - 1;
              if (++round < rounds) place(round, pl, ml);
            }
          }
        } else {
          GeneralSweep<T> q;
          q.X = X; q.Cc = Cc; q.G = G; q.gX = gXg;
          q.N = N; q.n_x = n_x; q.rs = rs; q.es = es; q.total = total; q.K = K; q.set = set; q.cl = cl;
          q.nq = nq; q.rounds = rounds;
          q.tape = tape; q.prog = prog; q.orphan = orphan; q.cidx = cidx; q.lcon = lcon; q.cv = cv; q.accl = accl;
          q.adj = reinterpret_cast<T*>(wb) + lane; q.vals = reinterpret_cast<T*>(wb + ly.vals) + lane;
          q.xs = reinterpret_cast<T*>(xs); q.xused = xused;
          q.crow = crow; q.crows = smem + ly.warps + ly.crow; q.warp_bytes = ly.warp_bytes; q.errs = errs;
          q.L = L; q.nop = nop; q.norph = norph; q.g0 = g0; q.ng = ng; q.lane = lane; q.rank = rank; q.ranks = ranks;
          general_sweep<T, kMode>(q);
        }
      }
      __syncthreads();  // every class's sums are complete
      for (int i = warp; i < ng * (int)K; i += nwarp) {
        const int j = i / (int)K, kk = i - j * (int)K;
        const int pos = lane * (int)K + kk;
        const T s = warp_sum(acc[((pos >> 5) * ncap + j) * 32 + (pos & 31)]);
        if (lane == 0) gC[(b * M + lcon[g0 + j]) * Ktot + set + kk] = s;
      }
      __syncthreads();
    }
    if (warp == 0) {
      int err = errs[lane] == ~0ull ? 0 : (int)(errs[lane] & 0xffffu);
      err = __reduce_max_sync(0xffffffffu, err);
      if (err && lane == 0) report_adjoint(status, err);
    }
  }
}

// ------------------------------------------------------------------------------------
// Host launchers
// ------------------------------------------------------------------------------------
// One class of tape lengths (Llo, Lhi]: how many constant sets a unit
// takes, and how many warps share it.
//   sets:  all in one pass while their constants and sums take little shared memory, else
//          one by one (see SetMode);
//   warps: the power of two that puts the most warps on the GPU at once, as far as the points
//          reach: one when the batch alone fills it (1003 tapes at N = 777: 97 us with 4 warps,
//          167 us with 2).
template <typename T, int kMode>
static int launch_adjoint_mode(const T* X, const T* cache, int64_t N, int64_t n_x, const uint32_t* desc, const int32_t* meta,
                               const int32_t* order, int64_t B, int64_t M, int Llo, int Lhi, const T* C, int64_t c_sb,
                               int64_t c_sm, int64_t c_sk, int64_t K, const T* gout, T* gC, T* gX, int32_t* status,
                               cudaStream_t st) {
  auto kern = eval_adjoint_kernel<T, kMode>;
  const void* kp = reinterpret_cast<const void*>(kern);
  const int xrows = gX ? x_sum_rows(n_x) : 0;
  const int64_t flat = kMode == kFlat ? K : 1, units = kMode == kStrided ? B * K : B;
  const int64_t chunks = (N * flat + 31) / 32;
  const int limit = max_dyn_smem(), sms = device_sm_count(), sm_bytes = max_sm_smem();
  int rc = cuda_check(cudaFuncSetAttribute(kp, cudaFuncAttributeMaxDynamicSharedMemorySize, limit), "adjoint smem");
  if (!rc)
    rc = cuda_check(cudaFuncSetAttribute(kp, cudaFuncAttributePreferredSharedMemoryCarveout,
                                         cudaSharedmemCarveoutMaxShared), "adjoint carveout");
  if (rc) return rc;
  const int64_t most = kMode == kFlat ? flat : (chunks + Pack<T>::V - 1) / Pack<T>::V;
  int best_w = 0, per_sm = 0;
  int64_t most_warps = 0;
  for (int w = 1; w <= 8; w *= 2) {
    const size_t bytes = adjoint_layout<T>(Lhi, flat, w, !cache, xrows).bytes;
    if (bytes > (size_t)limit) break;
    int blocks = resident_ctas(kp, w * 32, bytes);
    if (blocks < 1) break;
    if (w == 1 && units > (int64_t)sms * blocks) {
      // several waves: leave room for the padding check's CTA on every SM, its shared memory
      // (every CTA takes 1 KB besides its own) and the registers of its warps, as those of two
      const int room = (int)(((size_t)sm_bytes - kCheckReserve) / (bytes + 1024));
      blocks = blocks - 2 < room ? blocks - 2 : room;
      best_w = 1;
      per_sm = blocks < 1 ? 1 : blocks;
      break;
    }
    const int64_t ctas = (int64_t)sms * blocks, warps = (units < ctas ? units : ctas) * w;
    if (warps > most_warps) {
      most_warps = warps;
      best_w = w;
      per_sm = blocks;
    }
    if (w >= most) break;
  }
  if (!best_w) {
    set_error("tape of %d nodes does not fit in shared memory", Lhi);
    return SR_ERR_UNSUPPORTED;
  }
  int64_t blocks = (int64_t)sms * per_sm;
  if (blocks > units) blocks = units;
  kern<<<(unsigned)blocks, best_w * 32, adjoint_layout<T>(Lhi, flat, best_w, !cache, xrows).bytes, st>>>(
      X, cache, N, n_x, desc, meta, order, B, M, Llo, Lhi, C, c_sb, c_sm, c_sk, K, gout, gC, gX, status);
  return launch_check("eval_adjoint_kernel");
}

template <typename T>
static int launch_backward_class(const T* X, int64_t N, int64_t n_x, const uint32_t* desc, const int32_t* meta,
                                 const int32_t* order, int64_t B, int64_t M, int Llo, int Lhi, const T* C,
                                 int64_t c_sb, int64_t c_sm, int64_t c_sk, int64_t K, const T* cache, const T* gout,
                                 T* gC, T* gX, int32_t* status, cudaStream_t st) {
#define SR_ADJ_ARGS X, cache, N, n_x, desc, meta, order, B, M, Llo, Lhi, C, c_sb, c_sm, c_sk, K, gout, gC, gX, status, st
  const int xrows = gX ? x_sum_rows(n_x) : 0;
  if (K == 1) return launch_adjoint_mode<T, kSingle>(SR_ADJ_ARGS);
  if (K <= 64 && adjoint_layout<T>(Lhi, K, 1, !cache, xrows).bytes <= (56u << 10)) return launch_adjoint_mode<T, kFlat>(SR_ADJ_ARGS);
  return launch_adjoint_mode<T, kStrided>(SR_ADJ_ARGS);
#undef SR_ADJ_ARGS
}

template <typename T>
static int launch_backward(const T* X, int64_t N, int64_t n_x, const uint32_t* desc, const int32_t* meta,
                           const int32_t* order, int64_t B, int64_t M, int32_t max_len, const T* C, int64_t c_sb,
                           int64_t c_sm, int64_t c_sk, int64_t K, const T* cache, const T* gout, T* gC, T* gX,
                           int32_t* status, void* stream) {
  int rc = check_tape_args(B, M);
  if (rc) return rc;
  if (N < 0 || n_x < 0 || K < 0) { set_error("negative size"); return SR_ERR_INVALID_ARGUMENT; }
  if (!status) { set_error("null status"); return SR_ERR_INVALID_ARGUMENT; }
  cudaStream_t st = as_stream(stream);
  rc = cuda_check(cudaMemsetAsync(status, 0, sizeof(int32_t), st), "status reset");
  if (rc) return rc;
  if (B == 0 || M == 0 || K == 0) return SR_OK;
  if (!desc || !meta || !C || !gC || (N > 0 && !gout)) { set_error("null pointer argument"); return SR_ERR_INVALID_ARGUMENT; }
  if (N == 0) return cuda_check(cudaMemsetAsync(gC, 0, sizeof(T) * B * M * K, st), "grad_C reset");
  const int Lmax = (max_len > 0 && max_len < M) ? max_len : (int)M;
  // the padding check runs on a side stream, forked from and joined back into the
  // caller's stream (a CUDA graph capture records the same fork and join)
  // (on the caller's stream when there is little to check, as in launch_forward)
  SideStream side((double)B * M * N * K * sizeof(T) > (double)(8 << 20), st);
  rc = side.begin();
  if (rc) return rc;
  // one persistent grid per class of tape lengths (Llo, Lhi], each with the tables its class
  // needs; a batch too small to fill the GPU class by class runs as one grid
  const int bound[3] = {64, 32, 16};
  int cls[4][2], nc = 0, hi = Lmax;
  const bool split = B * K >= (int64_t)device_sm_count() * 32;
  for (int j = 0; j < 3; ++j) {
    if (hi > bound[j] && (split || bound[j] == 64)) {
      cls[nc][0] = bound[j];
      cls[nc][1] = hi;
      ++nc;
      hi = bound[j];
    }
  }
  cls[nc][0] = -1;
  cls[nc][1] = hi;
  ++nc;
  {
    // one CTA per SM, placed before the adjoint's grids, which leave it its shared memory.  An
    // SM cannot change its split of L1 and shared memory while a CTA is on it, so both ask for
    // the largest shared memory, or whichever comes first locks the other out
    int64_t pblocks = device_sm_count();
    if (pblocks > B) pblocks = B;
    rc = cuda_check(cudaFuncSetAttribute(padding_check_kernel<T>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                         cudaSharedmemCarveoutMaxShared), "check carveout");
    if (!rc) {
      padding_check_kernel<T><<<(unsigned)pblocks, (kCheckWarps + 1) * 32, 0, side.stream()>>>(gout, meta, B, M, N * K,
                                                                                            Lmax, status);
      rc = launch_check("padding_check_kernel");
    }
  }
  for (int ci = 0; ci < nc && !rc; ++ci) {
    rc = launch_backward_class<T>(X, N, n_x, desc, meta, order, B, M, cls[ci][0], cls[ci][1], C, c_sb, c_sm, c_sk, K,
                                  cache, gout, gC, gX, status, st);
  }
  const int rj = side.end();
  return rc ? rc : rj;
}

}  // namespace sr

extern "C" {

int sr_eval_backward_f32(const float* X, int64_t N, int64_t n_x, const uint32_t* desc, const int32_t* meta,
                         const int32_t* order, int64_t B, int64_t M, int32_t max_len, const float* C, int64_t c_sb,
                         int64_t c_sm, const float* cache, const float* gout, float* gC, float* gX, int32_t* status,
                         void* stream) {
  return sr::launch_backward<float>(X, N, n_x, desc, meta, order, B, M, max_len, C, c_sb, c_sm, 0, 1, cache, gout, gC,
                                    gX, status, stream);
}

int sr_eval_backward_f64(const double* X, int64_t N, int64_t n_x, const uint32_t* desc, const int32_t* meta,
                         const int32_t* order, int64_t B, int64_t M, int32_t max_len, const double* C, int64_t c_sb,
                         int64_t c_sm, const double* cache, const double* gout, double* gC, double* gX,
                         int32_t* status, void* stream) {
  return sr::launch_backward<double>(X, N, n_x, desc, meta, order, B, M, max_len, C, c_sb, c_sm, 0, 1, cache, gout, gC,
                                     gX, status, stream);
}

int sr_eval_backward_multi_f32(const float* X, int64_t N, int64_t n_x, const uint32_t* desc, const int32_t* meta,
                               const int32_t* order, int64_t B, int64_t M, int32_t max_len, const float* C,
                               int64_t c_sb, int64_t c_sm, int64_t c_sk, int64_t K, const float* cache,
                               const float* gout, float* gC, float* gX, int32_t* status, void* stream) {
  return sr::launch_backward<float>(X, N, n_x, desc, meta, order, B, M, max_len, C, c_sb, c_sm, c_sk, K, cache, gout,
                                    gC, gX, status, stream);
}

int sr_eval_backward_multi_f64(const double* X, int64_t N, int64_t n_x, const uint32_t* desc, const int32_t* meta,
                               const int32_t* order, int64_t B, int64_t M, int32_t max_len, const double* C,
                               int64_t c_sb, int64_t c_sm, int64_t c_sk, int64_t K, const double* cache,
                               const double* gout, double* gC, double* gX, int32_t* status, void* stream) {
  return sr::launch_backward<double>(X, N, n_x, desc, meta, order, B, M, max_len, C, c_sb, c_sm, c_sk, K, cache, gout,
                                     gC, gX, status, stream);
}

}  // extern "C"
