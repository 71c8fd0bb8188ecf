// sr_adjoint.cu -- adjoint of the forward evaluation for a dense output gradient: the
// padding-row check and the adjoint proper.
#include <type_traits>

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
// 16 warps and a quarter of the registers that the adjoint beside it needs (16384 tapes with 3 stages
// 1160 us, 4 stages 1046, 6 stages 1081).  Every wait gives up after about a second (status 601).
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
    // the lengths of its next 32 tapes at once, and as often a look at whether there is anything
    // left to find
    int lens = 0;
    int64_t seen = 0;
    for (int64_t b = blockIdx.x; b < B && !stuck; b += gridDim.x, ++seen) {
      if ((seen & 31) == 0) {
        const int64_t mine = b + (int64_t)lane * gridDim.x;
        lens = mine < B ? meta[mine * 4] : 0;
        if (__shfl_sync(0xffffffffu, *reinterpret_cast<volatile int32_t*>(status), 0) == ERR_GRAD_ON_NO_OP) break;
      }
      const int64_t L = __shfl_sync(0xffffffffu, lens, (int)(seen & 31));
      if (L > Lmax) {
        if (lane == 0) report(status, SR_TAPE_EXCEEDS_LAUNCH);
        continue;
      }
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

// The check beside the staged kernel, which takes the shared memory that the ring needs: one CTA
// per tape (grid-stride), 16-byte streaming loads, four in flight per thread.
template <typename T>
__global__ void __launch_bounds__(256) padding_check_direct_kernel(const T* __restrict__ gout,
                                                                   const int32_t* __restrict__ meta, int64_t B,
                                                                   int64_t M, int64_t N, int Lmax,
                                                                   int32_t* __restrict__ status) {
  constexpr int kVec = 16 / sizeof(T);
  for (int64_t b = blockIdx.x; b < B; b += gridDim.x) {
    // the whole CTA stops once a 201 is recorded (uniform decision)
    if (__syncthreads_or(threadIdx.x == 0 && *reinterpret_cast<volatile int32_t*>(status) == ERR_GRAD_ON_NO_OP))
      return;
    const int64_t L = meta[b * 4];
    if (L > Lmax) {
      if (threadIdx.x == 0) report(status, SR_TAPE_EXCEEDS_LAUNCH);
      continue;
    }
    const T* p = gout + (size_t)b * M * N + (size_t)L * N;
    const size_t count = (size_t)(M - L) * N;
    size_t head = (size_t)((16 - (reinterpret_cast<uintptr_t>(p) & 15)) & 15) / sizeof(T);
    if (reinterpret_cast<uintptr_t>(p) % sizeof(T)) head = count;  // unaligned elements: one by one
    if (head > count) head = count;
    bool nz = false;
    for (size_t i = threadIdx.x; i < head; i += blockDim.x) nz |= __ldcs(p + i) != T(0);
    const size_t nvec = (count - head) / kVec;
    const float4* q = reinterpret_cast<const float4*>(p + head);
    size_t i = threadIdx.x;
    for (; i + 3 * blockDim.x < nvec; i += 4 * blockDim.x) {
      float4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = __ldcs(q + i + u * blockDim.x);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (sizeof(T) == 4) {
          nz |= (v[u].x != 0.f) | (v[u].y != 0.f) | (v[u].z != 0.f) | (v[u].w != 0.f);
        } else {
          const double* d = reinterpret_cast<const double*>(&v[u]);
          nz |= (d[0] != 0.0) | (d[1] != 0.0);
        }
      }
    }
    for (; i < nvec; i += blockDim.x) {
      const float4 v = __ldcs(q + i);
      if (sizeof(T) == 4) {
        nz |= (v.x != 0.f) | (v.y != 0.f) | (v.z != 0.f) | (v.w != 0.f);
      } else {
        const double* d = reinterpret_cast<const double*>(&v);
        nz |= (d[0] != 0.0) | (d[1] != 0.0);
      }
    }
    for (size_t j = head + nvec * kVec + threadIdx.x; j < count; j += blockDim.x) nz |= __ldcs(p + j) != T(0);
    if (__syncthreads_or(nz) && threadIdx.x == 0) report_adjoint(status, ERR_GRAD_ON_NO_OP);
  }
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
// in the last three.)  It issues as many instructions per value as the kernel before it did, so
// large batches, which fill the GPU either way, go to that one (see eval_adjoint_staged_kernel).  A
// launch bound of three CTAs per SM (80 registers) undoes the loads ahead: 1450 us; prefetching
// the next pass's rows into L2 adds instructions and gains nothing (5.9 to 7.4 ms at 65536).
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
// Tapes whose child table is not that of a stack, or that need more rows than the table has, take
// a general sweep: one adjoint row per operator, and per leaf with several parents, of one or two
// values per lane, as many as the table then holds.  A node's first parent in the sweep starts
// from its output gradient, the others add to the row, and a leaf's last one hands the sum on.
// Calls without a cache take it with one value per lane and recompute the node values into rows.
// ------------------------------------------------------------------------------------

// Shared memory of a CTA: the tape words (offset 0); the program, from the front 16 bytes per
// operator and from the back 4 bytes per leaf without a parent; per node its row or constant
// index; the nodes of the learnable constants (and from the back those of the variables); the
// constants' values (learnable j at j, fixed
// f at L - 1 - f, one entry per set); the sums of ncap constants (32 K lanes each); the first
// error of each point residue; then per warp the adjoint rows, without a cache a value row
// per node, with several warps the terms of one pass, and with grad_X the sums of one pass
// for each variable.
struct AdjLayout {
  size_t prog, cidx, lcon, cval, acc, errs, warps, warp_bytes, vals, crow, xacc, bytes;
};

template <typename T>
__host__ __device__ __forceinline__ AdjLayout adjoint_layout(int Lmax, int64_t K, int nwarp, bool recompute, int xrows,
                                                             int ncap) {
  AdjLayout l;
  l.prog = align16((size_t)Lmax * 4);
  l.cidx = l.prog + 16 * (size_t)Lmax;
  l.lcon = l.cidx + align16((size_t)Lmax * 4);
  l.cval = l.lcon + align16((size_t)Lmax * 4);
  l.acc = l.cval + align16((size_t)Lmax * (size_t)K * sizeof(T));
  l.errs = l.acc + (size_t)ncap * (size_t)K * 32 * sizeof(T);
  l.warps = l.errs + 32 * 8 + 32;
  l.vals = (size_t)table_rows<T>(Lmax) * kRowBytes;
  l.crow = l.vals + (recompute ? (size_t)Lmax * 32 * sizeof(T) : 0);
  l.xacc = l.crow + (nwarp > 1 ? (size_t)ncap * kRowBytes : 0);
  l.warp_bytes = l.xacc + (size_t)xrows * kRowBytes;
  l.bytes = l.warps + (size_t)nwarp * l.warp_bytes;
  return l;
}

// Constants summed in one sweep: half the nodes of a tree are leaves, few of them constants; a
// tape with more is swept again for the rest.  Long tapes get more, beside rows that are larger
// anyway (256 tapes of 200 to 400 nodes, N = 256: 979 us with 8, 343 with an eighth of the
// nodes).
template <typename T>
static int sum_capacity(int Lmax, int64_t K, int nwarp) {
  int cap = nwarp > 1 ? 8 : 12;
  if (cap < Lmax / 8) cap = Lmax / 8;
  if (cap > (Lmax + 1) / 2) cap = (Lmax + 1) / 2;
  const int64_t room = (int64_t)(24 << 10) / (K * 32 * (int64_t)sizeof(T));
  return cap > room ? (room < 1 ? 1 : (int)room) : cap;
}

// Variables whose sums over the leaves are kept in rows.
__host__ __device__ __forceinline__ int x_sum_rows(int64_t n_x) { return n_x <= 16 ? (int)n_x : 0; }

// Program words of operator node k:
//   x: dense code (bits 0..4) | no parent (bit 5) | one child twice (bit 6) | k << 8 |
//      adjoint row << 20
//   y, z: for child 0 and 1: where its value comes from (bits 0..1: nowhere, its cache row,
//      a constant entry, the node's own cache row), the constant index (bits 2..13), where
//      its adjoint goes (bits 16..17: nowhere, a row, a constant's sum, grad_X), the row,
//      constant or variable index (bits 18..29); for a node with several parents whether an
//      earlier parent has left its adjoint in the row (bit 30), and for such a leaf at its last
//      parent (bit 31) that bits 18..29 are the row and bits 2..13 the constant or variable
//   w: child 0 | child 1 << 12
enum ValueFrom : uint32_t { kNoValue = 0, kChildRow = 1, kConstant = 2, kOwnRow = 3 };
enum AdjointTo : uint32_t { kNowhere = 0, kRow = 1, kSum = 2, kGradX = 3 };
constexpr uint32_t kNoParent = 1u << 5, kSameChild = 1u << 6, kEdgeAdd = 1u << 30, kEdgeLeaf = 1u << 31;
constexpr uint32_t kNothing = 31u;  // the code of the one entry of a tape without operators

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

// Whether a tape of the class takes the sweep over stack rows: its rows fit the table, and rows of
// the cache have less than 4 GB (that sweep's offsets have 32 bits).
template <typename T>
__device__ __forceinline__ bool in_stack_order(int need, int Lhi, int64_t rs) {
  return need >= 0 && need <= table_rows<T>(Lhi) && rs <= (int64_t)0xffffffff / (int64_t)sizeof(T);
}

// What a warp sweeps: one class of a unit's chunks.
template <typename T>
struct Sweep {
  const T *X, *Cc, *G;  // Cc: null without a cache
  T* gX;
  int64_t N, n_x, rs, es, total, K, set, cl, nq;
  const uint32_t* tape;
  const uint4* prog;
  const uint32_t* orphan;  // leaf j without a parent at orphan[-j]
  const int *vars, *cidx;  // variable leaf j at vars[-j]
  const T* cv;             // the lane's constant entries
  T* accl;                 // the lane's sums
  unsigned char* wb;       // the warp's rows
  const unsigned char* rows0;  // the first warp's rows
  uint32_t vals, crow, xacc;   // in the warp's rows: values, terms of a pass, sums per variable
  size_t warp_bytes;
  unsigned long long* errs;
  unsigned xused;
  int xrows, L, nop, norph, nvar, g0, ng, lane, rank, ranks;
};

// The sweep, VV values per lane.  kShared: nodes may have several parents.  Not kCached: the node
// values are recomputed into rows at the start of a pass (VV is 1).
template <typename T, int kMode, int VV, bool kShared, bool kCached>
__device__ __forceinline__ void sweep(const Sweep<T>& q) {
  constexpr uint32_t RB = 32u * VV * (uint32_t)sizeof(T);  // bytes of an adjoint row
  constexpr bool kFold = kMode != kFlat;
  const int64_t K = kFold ? 1 : q.K, es = kMode == kStrided ? q.es : 1;
  const int lane = q.lane, ranks = kFold ? q.ranks : 1, rank = kFold ? q.rank : 0;
  const int64_t rounds = (q.nq + (int64_t)ranks * VV - 1) / ((int64_t)ranks * VV);
  const int64_t vs = 32 * K * es;  // elements from one of a lane's values to the next
  using RowBytes = std::conditional_t<kShared, uint64_t, uint32_t>;
  const RowBytes row_bytes = (RowBytes)(q.rs * (int64_t)sizeof(T));
  T* const gX = q.gX;
  T* const accl = q.accl;
  T* const crow = reinterpret_cast<T*>(q.wb + q.crow);
  unsigned char* const rows = q.wb + lane * (VV * (int)sizeof(T));
  unsigned char* const xs = q.wb + q.xacc + lane * 16;  // the lane's sums per variable
  T* const vals = reinterpret_cast<T*>(q.wb + q.vals) + lane;
  int64_t p0 = 0;   // value index of the lane's first value in this pass
  unsigned vm = 0;  // which of its values exist
  uint32_t ep = 0;  // first error of each value: two bits (1 = 201, 2 = 204)
  auto point = [&](int64_t p) -> int64_t {  // the point of a value
    if (kMode != kFlat) return p;
    return q.total <= (int64_t)0xffffffff ? (int64_t)((uint32_t)p / (uint32_t)K) : p / K;
  };
  // a value's term of constant j
  auto add_constant = [&](uint32_t idx, const T (&val)[VV]) {
    const int j = (int)idx - q.g0;
    if (j < 0 || j >= q.ng) return;
    if (ranks == 1) {
      T t = accl[j * 32];
#pragma unroll
      for (int v = 0; v < VV; ++v)
        if ((vm >> v & 1u) && val[v] != T(0)) t = M_<T>::add(t, val[v]);
      accl[j * 32] = t;
    } else {
#pragma unroll
      for (int v = 0; v < VV; ++v) crow[(j * VV + v) * 32 + lane] = (vm >> v & 1u) ? val[v] : T(0);
    }
  };
  auto to_grad_x = [&](uint32_t var, const T (&val)[VV]) {
#pragma unroll
    for (int v = 0; v < VV; ++v)
      if ((vm >> v & 1u) && val[v] != T(0)) atomicAdd(gX + point(p0 + v * 32 * K) * q.n_x + var, val[v]);
  };
  auto add_variable = [&](uint32_t var, const T (&val)[VV]) {
    if (!gX) return;
    if (!q.xrows) return to_grad_x(var, val);
    T t[VV];
    load_part<T, VV>(xs + var * kRowBytes, t);
#pragma unroll
    for (int v = 0; v < VV; ++v)
      if (val[v] != T(0)) t[v] = M_<T>::add(t[v], val[v]);
    store_part<T, VV>(xs + var * kRowBytes, t);
  };
  auto clear_variables = [&]() {
    T zero[VV];
#pragma unroll
    for (int v = 0; v < VV; ++v) zero[v] = T(0);
    for (unsigned m = q.xused; m; m &= m - 1) store_part<T, VV>(xs + (__ffs((int)m) - 1) * kRowBytes, zero);
  };
  if (gX) clear_variables();
  auto place = [&](int64_t round, int64_t& p, unsigned& m) {
    const int64_t q0 = (round * ranks + rank) * VV;
    p = 32 * (q.cl + K * q0) + lane;
    m = 0;
#pragma unroll
    for (int v = 0; v < VV; ++v)
      if (p + v * 32 * K < q.total) m |= 1u << v;
  };
  auto row = [&](const T* at, uint32_t k, unsigned m, T (&x)[VV]) {  // at: the lane's first value of node 0
    const T* r = reinterpret_cast<const T*>(reinterpret_cast<const char*>(at) + (uint64_t)k * row_bytes);
#pragma unroll
    for (int v = 0; v < VV; ++v) x[v] = (m >> v & 1u) ? __ldg(r + v * vs) : T(0);
  };
  // next: the loads of the node to come (operand values, children's output gradients,
  // and its own for a node without a parent); cur: the node at hand
  struct Loads {
    uint4 w;
    T a[VV], b[VV], s0[VV], s1[VV], g[VV];
  } next, cur;
  next.w = make_uint4(0u, 0u, 0u, 0u);
  auto value = [&](uint32_t w, uint32_t child, uint32_t own, const T* cp, unsigned m, T (&x)[VV]) {
    const uint32_t from = w & 3u;
    if (!kCached) {
      if (from != kNoValue) x[0] = vals[(from == kOwnRow ? own : child) * 32];
    } else if (from == kConstant) {
      const T t = q.cv[(int64_t)(w >> 2 & 0xfffu) * K];
#pragma unroll
      for (int v = 0; v < VV; ++v) x[v] = t;
    } else if (from != kNoValue) {
      row(cp, from == kOwnRow ? own : child, m, x);
    }
  };
  // a child's adjoint: its output gradient plus the contributions
  auto give = [&](uint32_t w, const T (&val)[VV]) {
    const uint32_t to = w >> 16 & 3u;
    const uint32_t idx = kShared && (w & kEdgeLeaf) ? w >> 2 & 0xfffu : w >> 18 & 0xfffu;
    if (to == kRow) store_part<T, VV>(rows + idx * RB, val);
    else if (to == kSum) add_constant(idx, val);
    else if (to == kGradX) add_variable(idx, val);
  };
  auto from_gout = [&](uint32_t w) { return (w >> 16 & 3u) && !(kShared && (w & kEdgeAdd)); };
  if constexpr (!kCached) {
    for (int k = 0; k < q.L; ++k) {
      const int code = code_of(q.tape[k]);
      if (!is_op_code(code) && code != VAR) vals[k * 32] = q.cv[(int64_t)q.cidx[k] * K];
    }
  }
  auto recompute = [&]() {
    const int64_t n = point(p0 < q.total ? p0 : q.total - 1);
    for (int j = 0; j < q.nvar; ++j) {
      const int k = q.vars[-j];
      vals[k * 32] = __ldg(q.X + n * q.n_x + child0(q.tape[k]));
    }
    for (int i = 0; i < q.nop; ++i) {
      const uint4 w = q.prog[i];
      vals[(w.x >> 8 & 0xfffu) * 32] = op_value<T>((int)(w.x & 31u), vals[(w.w & 0xfffu) * 32], vals[(w.w >> 12) * 32]);
    }
  };
  int64_t pl = 0;  // first value, and which exist, of the pass that is being loaded
  unsigned ml = 0;
  int64_t round = 0, rcur = 0;         // the pass that is being loaded, the pass at hand
  int in = q.nop - 1, icur = -1;       // the node to load next, the node at hand
  if (rounds > 0) place(0, pl, ml);
  while (true) {
    const bool more = round < rounds;
    cur = next;
    if (more) {
      next.w = q.prog[in];
      const uint32_t own = next.w.x >> 8 & 0xfffu, c0 = next.w.w & 0xfffu, c1 = next.w.w >> 12;
      const T* gp = q.G + pl * es;
      if constexpr (kCached) {
        const T* cp = q.Cc + pl * es;
        value(next.w.y, c0, own, cp, ml, next.a);
        value(next.w.z, c1, own, cp, ml, next.b);
      }
      if (from_gout(next.w.y)) row(gp, c0, ml, next.s0);
      if (from_gout(next.w.z)) row(gp, c1, ml, next.s1);
      if (next.w.x & kNoParent) row(gp, own, ml, next.g);
    }
    if (icur >= 0) {
      if constexpr (!kCached) {
        if (icur == q.nop - 1) recompute();
        const uint32_t own = cur.w.x >> 8 & 0xfffu;
        value(cur.w.y, cur.w.w & 0xfffu, own, nullptr, vm, cur.a);
        value(cur.w.z, cur.w.w >> 12, own, nullptr, vm, cur.b);
      }
      if (!(cur.w.x & kNoParent)) load_part<T, VV>(rows + (cur.w.x >> 20) * RB, cur.g);
      if constexpr (kShared) {
        if (cur.w.y & kEdgeAdd) load_part<T, VV>(rows + (cur.w.y >> 18 & 0xfffu) * RB, cur.s0);
        if (cur.w.z & kEdgeAdd) load_part<T, VV>(rows + (cur.w.z >> 18 & 0xfffu) * RB, cur.s1);
        if (cur.w.x & kSameChild) {
#pragma unroll
          for (int v = 0; v < VV; ++v) cur.s1[v] = T(0);
        }
      }
      op_adjoint_onto<T, VV>((int)(cur.w.x & 31u), cur.g, cur.a, cur.b, cur.s0, cur.s1, ep);
      if constexpr (kShared) {
        if (cur.w.x & kSameChild) {  // (its second edge goes nowhere)
#pragma unroll
          for (int v = 0; v < VV; ++v) cur.s0[v] = M_<T>::add(cur.s0[v], cur.s1[v]);
        }
      }
      give(cur.w.y, cur.s0);
      give(cur.w.z, cur.s1);
      if (icur == 0) {  // the pass ends
        for (int j = 0; j < q.norph; ++j) {  // leaves without a parent: their output gradient alone
          const uint32_t w = q.orphan[-j];
          T val[VV];
          row(q.G + p0 * es, w & 0xfffu, vm, val);
          if (w & (1u << 12)) add_variable(w >> 13, val);
          else add_constant(w >> 13, val);
        }
        if (gX && q.xused) {
          for (unsigned m = q.xused; m; m &= m - 1) {
            T t[VV];
            load_part<T, VV>(xs + (__ffs((int)m) - 1) * kRowBytes, t);
            to_grad_x((uint32_t)(__ffs((int)m) - 1), t);
          }
          clear_variables();
        }
        if (__any_sync(0xffffffffu, ep != 0)) {
          const int64_t pchunks = (q.N + 31) / 32;
#pragma unroll
          for (int v = 0; v < VV; ++v) {
            const uint32_t e = ep >> (2 * v) & 3u;
            if (e && (vm >> v & 1u)) {
              const int64_t p = p0 + v * 32 * K, n = point(p);
              const int64_t kk = kMode == kFlat ? p - n * K : q.set;
              atomicMin(&q.errs[n & 31], ((unsigned long long)(kk * pchunks + n / 32) << 16) |
                                             (unsigned long long)(e == 2 ? ERR_DIV_BY_ZERO : ERR_GRAD_ON_NO_OP));
            }
          }
          ep = 0;
        }
        if (ranks > 1) {
          __syncthreads();
          for (int j = rank; j < q.ng; j += ranks) {
            T t = accl[j * 32];
            for (int r = 0; r < ranks; ++r) {
              const T* cr = reinterpret_cast<const T*>(q.rows0 + (size_t)r * q.warp_bytes + q.crow);
              const int64_t q0 = (rcur * ranks + r) * VV;
#pragma unroll
              for (int v = 0; v < VV; ++v) {
                if (q0 + v < q.nq) {
                  const T x = cr[(j * VV + v) * 32 + lane];
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
    if (in == q.nop - 1) {  // the first node of a pass is loaded: the pass begins
      p0 = pl;
      vm = ml;
      rcur = round;
    }
    icur = in;
    if (--in < 0) {
      in = q.nop - 1;
      if (++round < rounds) place(round, pl, ml);
    }
  }
}

// The arguments of the kernel below.
template <typename T>
struct AdjArgs {
  const T *X, *cache;
  int64_t N, n_x;
  const uint32_t* desc;
  const int32_t *meta, *order;
  int64_t B, M;
  int Llo, Lhi, xrows, ncap;
  const T* C;
  int64_t c_sb, c_sm, c_sk, Ktot;
  const T* gout;
  T *gC, *gX;
  int32_t* status;
};

// A CTA's view of its unit: sizes and the tables in shared memory.
template <typename T, int kMode, bool kCached>
struct UnitView {
  int64_t K, es, total, rs, nchunks;  // sets; elements between values; values per node; elements per node
  int lane, warp, nwarp, ranks, rank;
  AdjLayout ly;
  uint32_t* tape;
  uint4* prog;
  uint32_t* orphan;  // leaf j without a parent at orphan[-j]
  int *cidx, *lcon, *vars;  // variable leaf j at vars[-j] (without a cache)
  T *cval, *acc;
  unsigned long long* errs;
  int* info;  // operators, constants, orphans, variable leaves, variables, values per lane
  unsigned char* wb;
  __device__ __forceinline__ UnitView(const AdjArgs<T>& A, unsigned char* smem) {
    K = kMode == kFlat ? A.Ktot : 1;
    es = kMode == kStrided ? A.Ktot : 1;
    total = A.N * K;
    rs = total * es;
    nchunks = (total + 31) / 32;
    lane = threadIdx.x & 31;
    warp = threadIdx.x >> 5;
    nwarp = blockDim.x >> 5;
    // with one set the warps of a unit take turns over its passes (ranks), else whole classes
    ranks = kMode == kFlat ? 1 : nwarp;
    rank = kMode == kFlat ? 0 : warp;
    ly = adjoint_layout<T>(A.Lhi, K, nwarp, !kCached, A.xrows, A.ncap);
    tape = reinterpret_cast<uint32_t*>(smem);
    prog = reinterpret_cast<uint4*>(smem + ly.prog);
    orphan = reinterpret_cast<uint32_t*>(smem + ly.cidx) - 1;
    cidx = reinterpret_cast<int*>(smem + ly.cidx);
    lcon = reinterpret_cast<int*>(smem + ly.lcon);
    vars = lcon + A.Lhi - 1;
    cval = reinterpret_cast<T*>(smem + ly.cval);
    acc = reinterpret_cast<T*>(smem + ly.acc);
    errs = reinterpret_cast<unsigned long long*>(smem + ly.errs);
    info = reinterpret_cast<int*>(smem + ly.errs + 32 * 8);
    wb = smem + ly.warps + (size_t)warp * ly.warp_bytes;
  }
};

// The sweeps of one unit, once its program stands, and its gradients of the constants.
template <typename T, int kMode, int VV, bool kShared, bool kCached>
__device__ __forceinline__ void sweep_unit(const AdjArgs<T>& A, const UnitView<T, kMode, kCached>& u, unsigned char* smem,
                                           int64_t b, int64_t set, int L) {
  const int K = (int)u.K, ncap = A.ncap, ncon = u.info[1];
  // sweeps of ncap constants each: one, but for tapes with more of them
  for (int g0 = 0; g0 == 0 || g0 < ncon; g0 += ncap) {
    const int ng = min(ncap, ncon - g0);
    for (int i = threadIdx.x; i < ncap * K * 32; i += blockDim.x) u.acc[i] = T(0);
    __syncthreads();
    for (int cl = kMode == kFlat ? u.warp : 0; cl < K; cl += kMode == kFlat ? u.nwarp : 1) {
      Sweep<T> q;
      q.X = A.X;
      q.Cc = kCached ? A.cache + (size_t)b * A.M * u.rs + set : nullptr;
      q.G = A.gout + (size_t)b * A.M * u.rs + set;
      q.gX = g0 == 0 ? A.gX : nullptr;
      q.N = A.N; q.n_x = A.n_x; q.rs = u.rs; q.es = u.es; q.total = u.total; q.K = K; q.set = set;
      q.cl = cl;
      q.nq = cl < u.nchunks ? (u.nchunks - cl + K - 1) / K : 0;  // chunks of this class
      q.tape = u.tape; q.prog = u.prog; q.orphan = u.orphan; q.vars = u.vars; q.cidx = u.cidx;
      q.cv = u.cval + (kMode == kFlat ? (32 * cl + u.lane) % K : 0);
      q.accl = u.acc + (int64_t)cl * ncap * 32 + u.lane;
      q.wb = u.wb; q.rows0 = smem + u.ly.warps; q.vals = (uint32_t)u.ly.vals; q.crow = (uint32_t)u.ly.crow;
      q.xacc = (uint32_t)u.ly.xacc; q.warp_bytes = u.ly.warp_bytes; q.errs = u.errs;
      q.xused = A.xrows ? (unsigned)u.info[4] : 0u;
      q.xrows = A.xrows;
      q.L = L; q.nop = u.info[0]; q.norph = u.info[2]; q.nvar = u.info[3]; q.g0 = g0; q.ng = ng;
      q.lane = u.lane; q.rank = u.rank; q.ranks = u.ranks;
      sweep<T, kMode, VV, kShared, kCached>(q);
    }
    __syncthreads();  // every class's sums are complete
    for (int i = u.warp; i < ng * K; i += u.nwarp) {
      const int j = i / K, kk = i - j * K, pos = u.lane * K + kk;
      const T s = warp_sum(u.acc[((pos >> 5) * ncap + j) * 32 + (pos & 31)]);
      if (u.lane == 0) A.gC[(b * A.M + u.lcon[g0 + j]) * A.Ktot + set + kk] = s;
    }
    __syncthreads();
  }
}

// The same for the tapes that the sweep over stack rows does not take, out of line: its code and
// registers would otherwise weigh on that sweep (1050 us became 1486 for 16384 tapes, M = 64,
// N = 1024), and so would values that the caller keeps across it.
template <typename T, int kMode, int VV>
__device__ __noinline__ void general_unit(const AdjArgs<T>& A, int64_t b, int64_t set, int L) {
  extern __shared__ __align__(16) unsigned char smem[];
  const UnitView<T, kMode, true> u(A, smem);
  sweep_unit<T, kMode, VV, true, true>(A, u, smem, b, set, L);
}

// Not kGeneral: the tapes that are not in stack order are left to the staged kernel below (118
// registers, where the call of the general sweeps makes it 128 and 17 resident warps 16).
template <typename T, int kMode, bool kCached, bool kGeneral>
__global__ void __launch_bounds__(256, 2) eval_adjoint_kernel(const __grid_constant__ AdjArgs<T> A) {
  constexpr int V = Pack<T>::V;
  constexpr int G = V / 2;  // values per lane of the wider of the two general sweeps
  extern __shared__ __align__(16) unsigned char smem[];
  const UnitView<T, kMode, kCached> v(A, smem);
  const int64_t K = v.K, rs = v.rs, sets = kMode == kStrided ? A.Ktot : 1;
  const int64_t N = A.N, M = A.M;
  const int lane = v.lane, warp = v.warp, Lhi = A.Lhi;
  const unsigned below = (1u << lane) - 1u;
  T* const gX = A.gX;
  uint32_t *tape = v.tape, *orphan = v.orphan;
  uint4* prog = v.prog;
  int *cidx = v.cidx, *lcon = v.lcon, *vars = v.vars, *info = v.info;
  T* cval = v.cval;
  unsigned char* wb = v.wb;

  // The units come longest first: a CTA takes them there and back (i, 2 G - 1 - i, 2 G + i, ...),
  // so that the ones with the longest first unit get the shortest next.
  const int64_t units = A.B * sets;
  for (int64_t turn = 0; turn * gridDim.x < units; ++turn) {
    const int64_t u = turn * gridDim.x + (turn & 1 ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
    if (u >= units) continue;
    const int64_t ti = kMode == kStrided ? u / sets : u, set = u - ti * sets;
    const int64_t b = A.order ? (int64_t)A.order[ti] : ti;
    const int L = A.meta[b * 4];
    if (L <= A.Llo || L > Lhi) continue;  // another class's grid takes it (the same in every thread)
    __syncthreads();                    // every warp is done with the previous unit's tables
    for (int k = threadIdx.x; k < L; k += blockDim.x) tape[k] = A.desc[b * M + k];
    if (threadIdx.x < 32) v.errs[threadIdx.x] = ~0ull;
    __syncthreads();
    if (warp == 0) {
      int* scratch = reinterpret_cast<int*>(wb);  // in the rows' place
      int need = -1;
      if (kCached) need = stack_rows(tape, L, lane, scratch, cidx);
      const int R = table_rows<T>(Lhi);
      const bool stack = in_stack_order<T>(need, Lhi, rs);
      if (!kGeneral && !stack) {
        if (lane == 0) info[5] = 0;
      } else {
        int *first = scratch, *final = scratch + L, *rowof = scratch + 2 * L;  // parents that the sweep meets first and last
        for (int k = lane; k < L; k += 32) {
          first[k] = -1;
          final[k] = L;
        }
        __syncwarp();
        for (int k = lane; k < L; k += 32) {
          const uint32_t d = tape[k];
          const int ar = arity_of(code_of(d));
          if (stack) {
            if (ar >= 1) first[child0(d)] = k;
            if (ar == 2) first[child1(d)] = k;
          } else {
            for (int j = 0; j < ar; ++j) {
              const int c = j == 0 ? child0(d) : child1(d);
              atomicMax(&first[c], k);
              atomicMin(&final[c], k);
            }
          }
        }
        __syncwarp();
        // a leaf whose adjoint has to wait for further parents in a row
        auto waits = [&](int c, bool leaf) { return leaf && first[c] >= 0 && first[c] != final[c]; };
        int ncon = 0, nfix = 0, norph = 0, nvar = 0, nrow = 0;
        unsigned used = 0;  // variables of the tape
        for (int k0 = 0; k0 < L; k0 += 32) {
          const int k = k0 + lane;
          const bool in = k < L;
          const int code = in ? code_of(tape[k]) : NO_OP;
          const bool con = code == LEARNABLE, var = code == VAR, fix = !is_op_code(code) && !con && !var;
          const unsigned mc = __ballot_sync(0xffffffffu, con), mf = __ballot_sync(0xffffffffu, fix);
          const bool orph = (con || (var && gX)) && first[k] < 0;
          const unsigned mo = __ballot_sync(0xffffffffu, orph);
          used |= __reduce_or_sync(0xffffffffu, var ? 1u << (child0(tape[k]) & 31) : 0u);
          const int j = ncon + __popc(mc & below);
          if (!stack) {
            const bool has = in && (is_op_code(code) || waits(k, con || (var && gX)));
            const unsigned mr = __ballot_sync(0xffffffffu, has);
            if (in) rowof[k] = need >= 0 ? cidx[k] : nrow + __popc(mr & below);
            nrow += __popc(mr);
          }
          if (!kCached) {
            const unsigned mv = __ballot_sync(0xffffffffu, var);
            if (var) vars[-(nvar + __popc(mv & below))] = k;
            nvar += __popc(mv);
          }
          if (con) {
            cidx[k] = j;
            lcon[j] = k;
          }
          if (fix) {
            const int f = L - 1 - (nfix + __popc(mf & below));
            cidx[k] = f;
            const T x = node_value<T>(code, T(0), T(0), T(0), T(0));
            for (int kk = 0; kk < (int)K; ++kk) cval[(int64_t)f * K + kk] = x;
          }
          if (orph)
            orphan[-(norph + __popc(mo & below))] =
                (uint32_t)k | (var ? 1u << 12 : 0u) | ((uint32_t)(var ? child0(tape[k]) : j) << 13);
          ncon += __popc(mc);
          nfix += __popc(mf);
          norph += __popc(mo);
        }
        if (need >= 0) nrow = need;
        __syncwarp();
        auto operand = [&](int code, int k, int c, bool merged) -> uint32_t {
          const int cc = code_of(tape[c]);
          const bool op = is_op_code(cc), con = cc == LEARNABLE, var = cc == VAR;
          uint32_t w = 0;
          if (reads_operands(code)) {
            if (code == EXP) w = kOwnRow;  // its rule uses the node's own value
            else if (op || var) w = kChildRow;
            else w = kConstant | ((uint32_t)cidx[c] << 2);
          }
          const bool leaf = con || (var && gX);
          if (merged || !(op || leaf)) return w;
          const uint32_t kind = con ? kSum : kGradX, at = con ? (uint32_t)cidx[c] : (uint32_t)child0(tape[c]);
          if (stack) return w | (op ? (kRow << 16) | ((uint32_t)cidx[c] << 18) : (kind << 16) | (at << 18));
          const bool wait = waits(c, leaf);
          if (!op && !wait) return w | (kind << 16) | (at << 18);
          w |= ((uint32_t)rowof[c] << 18) | (k == first[c] ? 0u : kEdgeAdd);
          if (op || k != final[c]) return w | (kRow << 16);
          return w | (kind << 16) | (at << 2) | kEdgeLeaf;
        };
        int nop = 0;
        for (int k0 = 0; k0 < L; k0 += 32) {
          const int k = k0 + lane;
          const uint32_t d = k < L ? tape[k] : 0u;
          const int code = code_of(d), ar = arity_of(code);
          const bool op = k < L && is_op_code(code);
          const unsigned mo = __ballot_sync(0xffffffffu, op);
          if (op) {
            uint4 w = make_uint4((uint32_t)dense_op(code) | ((uint32_t)k << 8) |
                                     ((uint32_t)(stack ? cidx[k] : rowof[k]) << 20), 0u, 0u, 0u);
            if (first[k] < 0) w.x |= kNoParent;
            if (ar >= 1) {
              w.y = operand(code, k, child0(d), false);
              w.w = (uint32_t)child0(d);
            }
            if (ar == 2) {
              const bool same = child0(d) == child1(d);
              if (same) w.x |= kSameChild;
              w.z = operand(code, k, child1(d), same);
              w.w |= (uint32_t)child1(d) << 12;
            }
            prog[nop + __popc(mo & below)] = w;
          }
          nop += __popc(mo);
        }
        if (lane == 0) {
          if (nop == 0) prog[nop++] = make_uint4(kNothing, 0u, 0u, 0u);
          info[0] = nop;
          info[1] = ncon;
          info[2] = norph;
          info[3] = nvar;
          info[4] = (int)used;
          // values per lane: G where the rows hold them and a warp has more than one chunk
          info[5] = stack ? V : nrow * G <= R * V && N > 32 * v.ranks ? G : 1;
        }
      }
    }
    __syncthreads();
    const int ncon = info[1], VV = info[5];
    if (!kGeneral && VV != V) continue;
    for (int i = threadIdx.x; i < ncon * (int)K; i += blockDim.x) {
      const int j = i / (int)K, kk = i - j * (int)K;
      cval[i] = __ldg(A.C + b * A.c_sb + (int64_t)lcon[j] * A.c_sm + (set + kk) * A.c_sk);
    }
    // every other node's gradient is zero
    for (int i = threadIdx.x; i < (int)M * (int)K; i += blockDim.x) {
      const int k = i / (int)K, kk = i - k * (int)K;
      if (!(k < L && code_of(tape[k]) == LEARNABLE)) A.gC[(b * M + k) * A.Ktot + set + kk] = T(0);
    }
    if constexpr (!kCached) {
      sweep_unit<T, kMode, 1, true, false>(A, v, smem, b, set, L);
    } else {
      if (VV == V) sweep_unit<T, kMode, V, false, true>(A, v, smem, b, set, L);
      else if (kGeneral && G > 1 && VV == G) general_unit<T, kMode, G>(A, b, set, L);
      else if (kGeneral) general_unit<T, kMode, 1>(A, b, set, L);
    }
    if (warp == 0) {
      int err = v.errs[lane] == ~0ull ? 0 : (int)(v.errs[lane] & 0xffffu);
      err = __reduce_max_sync(0xffffffffu, err);
      if (err && lane == 0) report_adjoint(A.status, err);
    }
  }
}

// ------------------------------------------------------------------------------------
// Adjoint with staged rows.  One warp per tape, one value per lane.  A chunk's output gradients
// and node values are copied into shared memory at once (16 bytes per lane where the rows are
// aligned), then swept from there through precomputed byte offsets: half the
// instructions per value of the sweep above with one value per lane, and level with its four values
// per lane, but 256 bytes per node and warp, and nothing to split a tape over.  It takes
//   - tapes that the sweep above would give one or two values per lane, where the batch alone
//     fills the GPU, in grids of their own after those of the tapes in stack order (4096 tapes of
//     50 nodes with shared subtrees, N = 1024: 735 us, 2020 in the general sweep);
//   - calls of such batches without a cache (65536 tapes, N = 1024: 6.6 ms, 14 by the sweep);
//   - batches of one set from 192 tapes per SM on (65536 tapes, N = 1024, a gradient on every root:
//     4.6 ms, 5.1 by the sweep; with quotients, so with infinite and huge arguments, 5.0 and 6.5;
//     at 24576 tapes the sweep is still ahead, 2.48 and 2.60 ms);
//   - few points, where a pass of the sweep would be mostly empty (5000 tapes at N = 7: 64 us, 99;
//     20000 at N = 64, K = 3: 317 and 530).
// Sums and orders are the same, grad_X's within a tape included.
// ------------------------------------------------------------------------------------
template <int kBytes>
__device__ __forceinline__ void cp_async(void* dst_smem, const void* src, int src_bytes) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst_smem));
  if (kBytes == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(src_bytes) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %3, %2;" ::"r"(d), "l"(src), "r"(src_bytes), "n"(kBytes) : "memory");
}

// Copies 32 values from p on of rows node(0), ..., node(n - 1) of a block into rows of 32 of buf
// (zero past the last value).  vec16: every row's start is 16-byte aligned.
template <typename T, typename Node>
__device__ __forceinline__ void stage_rows(T* buf, const T* block, int n, Node node, int64_t total, int64_t rs, int64_t es,
                                           int64_t p, int lane, bool vec16) {
  if (vec16) {
    constexpr int E = 16 / sizeof(T), kLanes = 32 / E, kRows = 32 / kLanes;
    const int e = (lane % kLanes) * E;
    const int64_t left = total - (p + e);
    const int bytes = left >= E ? 16 : (left > 0 ? (int)left * (int)sizeof(T) : 0);
    for (int r = lane / kLanes; r < n; r += kRows) {
      const int k = node(r);
      cp_async<16>(buf + k * 32 + e, bytes ? block + (size_t)k * rs + p + e : block, bytes);
    }
  } else {
    const int bytes = p + lane < total ? (int)sizeof(T) : 0;
    for (int r = 0; r < n; ++r) {
      const int k = node(r);
      cp_async<(int)sizeof(T)>(buf + k * 32 + lane, bytes ? block + (size_t)k * rs + (p + lane) * es : block, bytes);
    }
  }
}

// Shared memory of a warp: the tape words (offset 0); per operator its code, the operands' source
// words (byte offset, bits 0..23, lane stride, bits 24..31), its value row and the operands'
// adjoint rows; the learnable and the variable leaves; the broadcast entries; a value and an adjoint row
// per node.  A learnable constant's value row holds its lanes' sums.
struct StagedLayout {
  uint32_t code, sa, sb, own, da, db, lcon, lvar, bc, vals, adj, bytes;
};
template <typename T>
__host__ __device__ __forceinline__ StagedLayout staged_layout(int Lmax) {
  const uint32_t lb = (uint32_t)align16((size_t)Lmax * 4), rows = (uint32_t)Lmax * 32u * (uint32_t)sizeof(T);
  StagedLayout l;
  l.code = lb;
  l.sa = 2 * lb;
  l.sb = 3 * lb;
  l.own = 4 * lb;
  l.da = 5 * lb;
  l.db = 6 * lb;
  l.lcon = 7 * lb;
  l.lvar = 8 * lb;
  l.bc = 9 * lb;
  l.vals = l.bc + (uint32_t)align16((size_t)(Lmax + 1) * sizeof(T));
  l.adj = l.vals + rows;
  l.bytes = l.adj + rows;
  return l;
}

template <typename T, bool kMulti, bool kCached>
__global__ void __launch_bounds__(256, 4) eval_adjoint_staged_kernel(
    const T* __restrict__ X, const T* __restrict__ cache, int64_t N, int64_t n_x, const uint32_t* __restrict__ desc,
    const int32_t* __restrict__ meta, const int32_t* __restrict__ order, int64_t B, int64_t M, int Llo, int Lhi,
    bool general_only, const T* __restrict__ C, int64_t c_sb, int64_t c_sm, int64_t c_sk, int64_t K_,
    const T* __restrict__ gout, T* __restrict__ gC, T* __restrict__ gX, int32_t* __restrict__ status, bool vec16) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int64_t K = kMulti ? K_ : 1, rs = N * K;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  constexpr uint32_t RB = 32u * (uint32_t)sizeof(T), kRowStride = (uint32_t)sizeof(T) << 24;
  const StagedLayout ly = staged_layout<T>(Lhi);
  unsigned char* wb = smem + (size_t)warp * ly.bytes;
  uint32_t* tape = reinterpret_cast<uint32_t*>(wb);
  auto table = [&](uint32_t at) { return reinterpret_cast<uint32_t*>(wb + at); };
  uint32_t *code_ = table(ly.code), *psa = table(ly.sa), *psb = table(ly.sb), *pown = table(ly.own), *pda = table(ly.da),
           *pdb = table(ly.db), *lcon = table(ly.lcon), *lvar = table(ly.lvar);
  T* bc = reinterpret_cast<T*>(wb + ly.bc);
  T* vals = reinterpret_cast<T*>(wb + ly.vals);
  T* adj = reinterpret_cast<T*>(wb + ly.adj);
  const uint32_t adj_delta = ly.adj - ly.vals;
  const unsigned below = (1u << lane) - 1u;
  auto at = [&](uint32_t off) -> T& { return reinterpret_cast<T*>(wb + off)[lane]; };
  auto operand = [&](uint32_t w) { return *reinterpret_cast<const T*>(wb + (w & 0xffffffu) + (uint32_t)lane * (w >> 24)); };
  for (int64_t ti = (int64_t)blockIdx.x * nwarp + warp; ti < B; ti += (int64_t)gridDim.x * nwarp) {
    const int64_t b = order ? (int64_t)order[ti] : ti;
    const int L = meta[b * 4];
    if (L <= Llo || L > Lhi) continue;  // another class's grid takes it (warp-uniform)
    for (int k = lane; k < L; k += 32) tape[k] = desc[b * M + k];
    if (lane == 0) bc[0] = T(0);
    __syncwarp();
    if (general_only) {
      int* scratch = reinterpret_cast<int*>(adj);
      const int need = stack_rows(tape, L, lane, scratch, scratch + L + 1);
      __syncwarp();
      if (in_stack_order<T>(need, Lhi, rs)) continue;  // eval_adjoint_kernel takes it
    }
    // the operators, learnable and variable leaves; the broadcast entries of fixed leaves (and of
    // codes that evaluate to 0) now
    int nop = 0, ncon = 0, nvar = 0;
    for (int k0 = 0; k0 < L; k0 += 32) {
      const int k = k0 + lane;
      const uint32_t d = k < L ? tape[k] : 0u;
      const int code = k < L ? code_of(d) : -1;
      const bool op = k < L && is_op_code(code), con = code == LEARNABLE, var = code == VAR;
      const unsigned mo = __ballot_sync(0xffffffffu, op), mc = __ballot_sync(0xffffffffu, con),
                     mv = __ballot_sync(0xffffffffu, var);
      // source word of operand node c: its value row, or its broadcast entry
      auto src = [&](int c) -> uint32_t {
        const int cc = code_of(tape[c]);
        if (is_op_code(cc) || cc == VAR) return (ly.vals + (uint32_t)c * RB) | kRowStride;
        return ly.bc + (uint32_t)(1 + c) * (uint32_t)sizeof(T);
      };
      if (op) {
        const int ar = arity_of(code), i = nop + __popc(mo & below);
        const uint32_t none = ly.adj + (uint32_t)k * RB;  // never written through (arity < 2)
        code_[i] = (uint32_t)dense_op(code);
        pown[i] = ly.vals + (uint32_t)k * RB;
        psa[i] = ar >= 1 ? src(child0(d)) : ly.bc;
        pda[i] = ar >= 1 ? ly.adj + (uint32_t)child0(d) * RB : none;
        psb[i] = ar == 2 ? src(child1(d)) : ly.bc;
        pdb[i] = ar == 2 ? ly.adj + (uint32_t)child1(d) * RB : none;
      } else if (k < L && !con && !var) {
        bc[1 + k] = node_value<T>(code, T(0), T(0), T(0), T(0));
      }
      if (con) lcon[ncon + __popc(mc & below)] = (uint32_t)k;
      if (var) lvar[nvar + __popc(mv & below)] = (uint32_t)k;
      nop += __popc(mo);
      ncon += __popc(mc);
      nvar += __popc(mv);
    }
    __syncwarp();
    if (gX && nvar > 0) {
      // the variable leaves in the order in which the sweep meets their last parents (leaves without
      // one at the end), each with the first of its variable in bits 12..23: that one's
      // adjoint row takes the sum
      int* key = reinterpret_cast<int*>(adj);
      uint32_t* sorted = reinterpret_cast<uint32_t*>(adj) + L;
      for (int k = lane; k < L; k += 32) key[k] = 0x7fffffff;
      __syncwarp();
      for (int k = lane; k < L; k += 32) {
        const uint32_t d = tape[k];
        const int ar = arity_of(code_of(d));
        if (ar >= 1) atomicMin(&key[child0(d)], 2 * k);
        if (ar == 2) atomicMin(&key[child1(d)], 2 * k + 1);
      }
      __syncwarp();
      auto later = [&](int c) { return key[c] == 0x7fffffff ? -1 - c : (key[c] ^ 1) + 1; };  // falls along the sweep
      for (int j = lane; j < nvar; j += 32) {
        const int mine = later((int)lvar[j]);
        int place = 0;
        for (int i = 0; i < nvar; ++i) place += later((int)lvar[i]) > mine ? 1 : 0;
        sorted[place] = lvar[j];
      }
      __syncwarp();
      for (int j = lane; j < nvar; j += 32) {
        const int var = child0(tape[sorted[j]]);
        int i = 0;
        while (child0(tape[sorted[i]]) != var) ++i;
        lvar[j] = sorted[j] | sorted[i] << 12;
      }
      __syncwarp();
    }
    int err = 0;
    const int64_t nchunks = (N + 31) / 32;
    // the sets one after the other: set kk of node k, point n is at ((b M + k) N + n) K + kk
    for (int64_t kk = 0; kk < K; ++kk) {
      const T* Crow = C + b * c_sb + kk * c_sk;
      for (int j = lane; j < ncon; j += 32) bc[1 + lcon[j]] = __ldg(Crow + (int64_t)lcon[j] * c_sm);
      for (int j = 0; j < ncon; ++j) vals[lcon[j] * 32 + lane] = T(0);
      const T* G = gout + (size_t)b * M * rs + kk;
      const T* Cc = kCached ? cache + (size_t)b * M * rs + kk : nullptr;
      __syncwarp();
      for (int64_t c = 0; c < nchunks; ++c) {
        const int64_t n = c * 32 + lane, nn = n < N ? n : N - 1;
        const bool valid = n < N;
        // the adjoints start as the output gradients
        stage_rows(adj, G, L, [](int r) { return r; }, N, rs, K, c * 32, lane, vec16);
        if constexpr (kCached) {
          auto node = [&](int r) { return r < nop ? (int)((pown[r] - ly.vals) / RB) : (int)(lvar[r - nop] & 0xfffu); };
          stage_rows(vals, Cc, nop + nvar, node, N, rs, K, c * 32, lane, vec16);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        if constexpr (!kCached) {
          for (int j = 0; j < nvar; ++j) {
            const int k = (int)(lvar[j] & 0xfffu);
            vals[k * 32 + lane] = __ldg(X + nn * n_x + child0(tape[k]));
          }
          for (int i = 0; i < nop; ++i) {
            const int code = (int)code_[i];
            const uint32_t sa = psa[i], sb = psb[i], own = pown[i];
            at(own) = op_value<T>(code, operand(sa), operand(sb));
          }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncwarp();
        for (int i = nop - 1; i >= 0; --i) {
          const int code = (int)code_[i];
          const uint32_t sa = psa[i], sb = psb[i], own = pown[i], da = pda[i], db = pdb[i];
          T g[1], a[1], c1[1], v[1], o0[1], o1[1];
          bool a0[1], a1[1];
          int e[1];
          g[0] = at(own + adj_delta);
          a[0] = operand(sa);
          c1[0] = operand(sb);
          v[0] = at(own);
          op_adjoint_v<T, 1>(code, g, a, c1, v, a0, o0, a1, o1, e);
          if (valid) {
            if (e[0] && !err) err = e[0];
            if (a0[0]) { T& x = at(da); x = M_<T>::add(x, o0[0]); }
            if (a1[0]) { T& x = at(db); x = M_<T>::add(x, o1[0]); }
          }
        }
        // leaves: every contribution from the parents has arrived
        for (int j = 0; j < ncon; ++j) {
          const T g = adj[lcon[j] * 32 + lane];
          T& x = vals[lcon[j] * 32 + lane];
          if (valid && g != T(0)) x = M_<T>::add(x, g);
        }
        if (gX) {
          for (int j = 1; j < nvar; ++j) {
            const uint32_t k = lvar[j] & 0xfffu, first = lvar[j] >> 12;
            const T g = adj[k * 32 + lane];
            T& x = adj[first * 32 + lane];
            if (k != first && g != T(0)) x = M_<T>::add(x, g);
          }
          for (int j = 0; j < nvar; ++j) {
            const uint32_t k = lvar[j] & 0xfffu;
            const T g = adj[k * 32 + lane];
            if (k == lvar[j] >> 12 && valid && g != T(0)) atomicAdd(gX + nn * n_x + child0(tape[k]), g);
          }
        }
        __syncwarp();  // every lane is done with the rows before the next chunk's land
      }
      // the constants' sums (lane partials in chunk order, then a butterfly) replace
      // their values in the broadcast entries
      for (int j = 0; j < ncon; ++j) {
        const T part = warp_sum(vals[lcon[j] * 32 + lane]);
        if (lane == 0) bc[1 + lcon[j]] = part;
      }
      __syncwarp();
      for (int64_t k = lane; k < M; k += 32)
        gC[(b * M + k) * K + kk] = k < L && code_of(tape[k]) == LEARNABLE ? bc[1 + k] : T(0);
      __syncwarp();
    }
    err = __reduce_max_sync(0xffffffffu, err);
    if (err && lane == 0) report_adjoint(status, err);
    __syncwarp();
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
template <typename T, int kMode, bool kCached, bool kGeneral>
static int launch_adjoint_mode(const T* X, const T* cache, int64_t N, int64_t n_x, const uint32_t* desc, const int32_t* meta,
                               const int32_t* order, int64_t B, int64_t M, int Llo, int Lhi, const T* C, int64_t c_sb,
                               int64_t c_sm, int64_t c_sk, int64_t K, const T* gout, T* gC, T* gX, int32_t* status,
                               cudaStream_t st) {
  auto kern = eval_adjoint_kernel<T, kMode, kCached, kGeneral>;
  constexpr int V = kCached ? Pack<T>::V / 2 : 1;  // as few points per warp as a general sweep can use
  const void* kp = reinterpret_cast<const void*>(kern);
  const int64_t flat = kMode == kFlat ? K : 1, units = kMode == kStrided ? B * K : B;
  const int64_t chunks = (N * flat + 31) / 32;
  const int limit = max_dyn_smem(), sms = device_sm_count(), sm_bytes = max_sm_smem();
  int rc = cuda_check(cudaFuncSetAttribute(kp, cudaFuncAttributeMaxDynamicSharedMemorySize, limit), "adjoint smem");
  if (!rc)
    rc = cuda_check(cudaFuncSetAttribute(kp, cudaFuncAttributePreferredSharedMemoryCarveout,
                                         cudaSharedmemCarveoutMaxShared), "adjoint carveout");
  if (rc) return rc;
  // a tape that only just fits gets one constant at a time and no sums per variable
  int xrows = gX ? x_sum_rows(n_x) : 0;
  auto bytes_of = [&](int w, int cap) { return adjoint_layout<T>(Lhi, flat, w, !kCached, xrows, cap).bytes; };
  const bool tight = bytes_of(1, sum_capacity<T>(Lhi, flat, 1)) > (size_t)limit;
  if (tight) xrows = 0;
  auto capacity = [&](int w) { return tight ? 1 : sum_capacity<T>(Lhi, flat, w); };
  const int64_t most = kMode == kFlat ? flat : (chunks + V - 1) / V;
  int best_w = 0, per_sm = 0;
  int64_t most_warps = 0;
  for (int w = 1; w <= 8; w *= 2) {
    const size_t bytes = bytes_of(w, capacity(w));
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
  const AdjArgs<T> args{X, cache, N, n_x, desc, meta, order, B, M, Llo, Lhi, xrows, capacity(best_w), C, c_sb, c_sm, c_sk, K, gout, gC, gX, status};
  kern<<<(unsigned)blocks, best_w * 32, bytes_of(best_w, capacity(best_w)), st>>>(args);
  return launch_check("eval_adjoint_kernel");
}

template <typename T, bool kCached>
static int launch_streaming(const T* X, const T* cache, int64_t N, int64_t n_x, const uint32_t* desc, const int32_t* meta,
                            const int32_t* order, int64_t B, int64_t M, int Llo, int Lhi, const T* C, int64_t c_sb,
                            int64_t c_sm, int64_t c_sk, int64_t K, const T* gout, T* gC, T* gX, int32_t* status,
                            bool stack_only, cudaStream_t st) {
#define SR_ADJ_ARGS \
  X, cache, N, n_x, desc, meta, order, B, M, Llo, Lhi, C, c_sb, c_sm, c_sk, K, gout, gC, gX, status, st
  const int xrows = gX ? x_sum_rows(n_x) : 0;
  if (K == 1)
    return stack_only ? launch_adjoint_mode<T, kSingle, true, false>(SR_ADJ_ARGS)
                      : launch_adjoint_mode<T, kSingle, kCached, true>(SR_ADJ_ARGS);
  if (K <= 64 && adjoint_layout<T>(Lhi, K, 1, !kCached, xrows, sum_capacity<T>(Lhi, K, 1)).bytes <= (56u << 10))
    return launch_adjoint_mode<T, kFlat, kCached, true>(SR_ADJ_ARGS);
  return launch_adjoint_mode<T, kStrided, kCached, true>(SR_ADJ_ARGS);
#undef SR_ADJ_ARGS
}

template <typename T, bool kCached>
static int launch_staged(const T* X, const T* cache, int64_t N, int64_t n_x, const uint32_t* desc, const int32_t* meta,
                         const int32_t* order, int64_t B, int64_t M, int Llo, int Lhi, const T* C, int64_t c_sb,
                         int64_t c_sm, int64_t c_sk, int64_t K, const T* gout, T* gC, T* gX, int32_t* status,
                         bool general_only, cudaStream_t st) {
  auto kern = K == 1 ? eval_adjoint_staged_kernel<T, false, kCached> : eval_adjoint_staged_kernel<T, true, kCached>;
  Shape sh;
  // beside the padding check's ring, which a large batch keeps busy meanwhile (16384 tapes with
  // shared subtrees 1.98 to 1.85 ms; 4096 of them 743 to 910 us)
  const size_t reserve = general_only && B >= (int64_t)device_sm_count() * 32 ? kCheckReserve : 0;
  if (!pick_shape(reinterpret_cast<const void*>(kern), staged_layout<T>(Lhi).bytes, B, sh, reserve)) {
    set_error("tape of %d nodes does not fit in shared memory", Lhi);
    return SR_ERR_UNSUPPORTED;
  }
  auto aligned = [&](const T* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
  const bool vec16 = K == 1 && aligned(gout) && aligned(cache) && N % Pack<T>::V == 0;
  kern<<<(unsigned)sh.blocks, sh.warps * 32, sh.smem, st>>>(X, cache, N, n_x, desc, meta, order, B, M, Llo, Lhi,
                                                           general_only, C, c_sb, c_sm, c_sk, K, gout, gC, gX, status,
                                                           vec16);
  return launch_check("eval_adjoint_staged_kernel");
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
  // which kernel takes what (see eval_adjoint_staged_kernel, whose tables hold fewer nodes).  A batch
  // fills the GPU when at least half of that kernel's warps that fit get a tape.
  const int64_t sms = device_sm_count();
  const size_t staged_bytes = staged_layout<T>(Lmax).bytes;
  const int64_t per_sm = (int64_t)(max_sm_smem() / staged_bytes) < 32 ? (int64_t)(max_sm_smem() / staged_bytes) : 32;
  const bool holds = staged_bytes <= (size_t)max_dyn_smem(), fills = holds && K <= 4 && 2 * B >= sms * per_sm;
  const bool few = holds && N <= 16 * Pack<T>::V && K <= 4;
  const bool all_staged = few || (fills && (!cache || (K == 1 && B >= sms * 192)));
  const bool general_staged = fills && K == 1 && !all_staged;
  // one persistent grid per class of tape lengths (Llo, Lhi], each with the tables its class
  // needs; a batch too small to fill the GPU class by class runs as one grid.  The staged kernel's
  // tables are the larger: its longest class is split at 48 rather than 64.
  const int bound[3] = {all_staged ? 48 : 64, 32, 16};
  int cls[4][2], nc = 0, hi = Lmax;
  const bool split = B * K >= sms * 32;
  for (int j = 0; j < 3; ++j) {
    if (hi > bound[j] && (split || hi > 64)) {
      cls[nc][0] = bound[j];
      cls[nc][1] = hi;
      ++nc;
      hi = bound[j];
    }
  }
  cls[nc][0] = -1;
  cls[nc][1] = hi;
  ++nc;
  auto check = [&]() -> int {
    if (all_staged) {
      const int64_t pblocks = sms * 2 < B ? sms * 2 : B;
      padding_check_direct_kernel<T><<<(unsigned)pblocks, 256, 0, side.stream()>>>(gout, meta, B, M, N * K, Lmax, status);
      return launch_check("padding_check_direct_kernel");
    }
    // one CTA per SM, placed before the adjoint's grids, which leave it its shared memory.  An
    // SM cannot change its split of L1 and shared memory while a CTA is on it, so both ask for
    // the largest shared memory, or whichever comes first locks the other out
    const int64_t pblocks = sms < B ? sms : B;
    const int e = cuda_check(cudaFuncSetAttribute(padding_check_kernel<T>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                                  cudaSharedmemCarveoutMaxShared), "check carveout");
    if (e) return e;
    padding_check_kernel<T><<<(unsigned)pblocks, (kCheckWarps + 1) * 32, 0, side.stream()>>>(gout, meta, B, M, N * K,
                                                                                          Lmax, status);
    return launch_check("padding_check_kernel");
  };
  if (!all_staged) rc = check();
  for (int ci = 0; ci < nc && !rc; ++ci) {
    const int Llo = cls[ci][0], Lhi = cls[ci][1];
    auto streaming = cache ? launch_streaming<T, true> : launch_streaming<T, false>;
    auto staged = cache ? launch_staged<T, true> : launch_staged<T, false>;
    if (!all_staged)
      rc = streaming(X, cache, N, n_x, desc, meta, order, B, M, Llo, Lhi, C, c_sb, c_sm, c_sk, K, gout, gC, gX, status,
                     general_staged, st);
    if (!rc && (all_staged || general_staged))
      rc = staged(X, cache, N, n_x, desc, meta, order, B, M, Llo, Lhi, C, c_sb, c_sm, c_sk, K, gout, gC, gX, status,
                  general_staged, st);
    // enqueued after the first grid, whose CTAs are placed first: the check's CTAs take the
    // registers and warp slots they leave
    if (!rc && all_staged && ci == 0) rc = check();
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
