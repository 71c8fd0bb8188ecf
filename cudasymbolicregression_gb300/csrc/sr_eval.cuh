// sr_eval.cuh -- what the forward (sr_eval.cu) and the adjoint (sr_adjoint.cu) share:
// 16-byte lane packs, the stack rows of a tape, launch shapes and the side stream.
#pragma once
#include <cstdint>
#include <mutex>

#include "sr_common.cuh"
#include "sr_ops.cuh"

namespace sr {

__host__ __device__ __forceinline__ size_t align16(size_t x) { return (x + 15) & ~size_t(15); }

// The points a lane works on at once: as many as fill 16 bytes, so that a lane's part of a
// value row is one 16-byte shared-memory access and one decode and dispatch of a node
// serves all of them.  A row is 32 lanes x 16 bytes; a lane touches only its own part.
template <typename T>
struct Pack {
  static constexpr int V = 16 / (int)sizeof(T);
};
constexpr uint32_t kRowBytes = 512;

__device__ __forceinline__ void load16(const void* p, float (&r)[4]) {
  const float4 t = *reinterpret_cast<const float4*>(p);
  r[0] = t.x; r[1] = t.y; r[2] = t.z; r[3] = t.w;
}
__device__ __forceinline__ void load16(const void* p, double (&r)[2]) {
  const double2 t = *reinterpret_cast<const double2*>(p);
  r[0] = t.x; r[1] = t.y;
}
__device__ __forceinline__ void store16(void* p, const float (&r)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(r[0], r[1], r[2], r[3]);
}
__device__ __forceinline__ void store16(void* p, const double (&r)[2]) {
  *reinterpret_cast<double2*>(p) = make_double2(r[0], r[1]);
}
__device__ __forceinline__ void stream16(void* p, const float (&r)[4]) {
  __stcs(reinterpret_cast<float4*>(p), make_float4(r[0], r[1], r[2], r[3]));
}
__device__ __forceinline__ void stream16(void* p, const double (&r)[2]) {
  __stcs(reinterpret_cast<double2*>(p), make_double2(r[0], r[1]));
}

// A lane's part of a row: VV values.
template <typename T, int VV>
__device__ __forceinline__ void load_part(const void* p, T (&r)[VV]) {
  if constexpr (VV * sizeof(T) == 16) {
    load16(p, r);
  } else if constexpr (VV == 2) {
    const float2 t = *reinterpret_cast<const float2*>(p);
    r[0] = t.x; r[1] = t.y;
  } else {
    r[0] = *reinterpret_cast<const T*>(p);
  }
}
template <typename T, int VV>
__device__ __forceinline__ void store_part(void* p, const T (&r)[VV]) {
  if constexpr (VV * sizeof(T) == 16) store16(p, r);
  else if constexpr (VV == 2) *reinterpret_cast<float2*>(p) = make_float2(r[0], r[1]);
  else *reinterpret_cast<T*>(p) = r[0];
}
template <typename T, int VV>
__device__ __forceinline__ void stream_part(void* p, const T (&r)[VV]) {
  if constexpr (VV * sizeof(T) == 16) stream16(p, r);
  else if constexpr (VV == 2) __stcs(reinterpret_cast<float2*>(p), make_float2(r[0], r[1]));
  else __stcs(reinterpret_cast<T*>(p), r[0]);
}

// How a unit takes the K constant sets of its tape: one set (K = 1), all of them as N K
// consecutive values per node, or one set whose values lie K elements apart.
enum SetMode : int { kSingle = 0, kFlat = 1, kStrided = 2 };

// NO_OP nodes count as operators: their value (NaN) and their adjoint check matter.
__device__ __forceinline__ bool is_op_code(int code) { return code == NO_OP || arity_of(code) >= 1; }

// Rows of the operator nodes of a tape in stack order, by one warp.  A postfix tape whose
// operators take the top entries of an evaluation stack (what the child table of every
// postfix expression says) needs a row only for the operator results that wait on that
// stack: node k's row is the number of operator results below its own, a prefix sum over
// the nodes, so no serial assignment is needed.  The reverse sweep visits the same tree the
// other way round, and the adjoints that wait there are the same sets.  Writes row[k] for the
// operator nodes and returns how many rows the tape takes, or -1 if its child table is not
// that of a stack (a shared or a skipped subtree): such tapes take one row per node.
// The check: the (right) child of k is k - 1, and a left child is the last node before k
// whose result sits at the depth of k's own result.  last (L + 1 entries) is scratch.
__device__ __forceinline__ int stack_rows(const uint32_t* tape, int L, int lane, int* last, int* row,
                                          int* depth = nullptr) {
  const unsigned below = (1u << lane) - 1u, upto = below | (1u << lane);
  for (int d = lane; d <= L; d += 32) last[d] = -1;
  __syncwarp();
  int S = 0, D = 0, most = 0;
  bool ok = true;
  for (int k0 = 0; k0 < L; k0 += 32) {
    const int k = k0 + lane;
    const bool in = k < L;
    const uint32_t d = in ? tape[k] : 0u;
    const int code = code_of(d);
    const int ar = in ? arity_of(code) : 0;
    const unsigned push = __ballot_sync(0xffffffffu, in && ar == 0), pop = __ballot_sync(0xffffffffu, ar == 2);
    const int s = S + __popc(push & upto) - __popc(pop & upto);  // stack depth after k
    int delta = in && is_op_code(code) ? 1 : 0;
    if (ar >= 1 && is_op_code(code_of(tape[child0(d)]))) --delta;
    if (ar == 2 && is_op_code(code_of(tape[child1(d)]))) --delta;
    const unsigned up = __ballot_sync(0xffffffffu, delta > 0), down = __ballot_sync(0xffffffffu, delta < 0);
    const int r = D + __popc(up & upto) - __popc(down & upto);  // operator results on the stack after k
    const unsigned same = __match_any_sync(0xffffffffu, in ? s : -1 - lane);
    const unsigned lower = same & below;
    const int prev = lower ? k0 + 31 - __clz((int)lower) : (in && s >= 1 && s <= L ? last[s] : -1);
    const bool good = !in || (s >= 1 && (ar == 0 || (ar == 1 ? child0(d) == k - 1
                                                             : child1(d) == k - 1 && child0(d) == prev)));
    ok = __all_sync(0xffffffffu, good) && ok;
    most = max(most, __reduce_max_sync(0xffffffffu, in ? r : 0));
    if (in) row[k] = r - 1;
    __syncwarp();
    if (in && s >= 1 && s <= L && (same & ~upto) == 0) last[s] = k;
    __syncwarp();
    const int end = min(31, L - 1 - k0);
    S = __shfl_sync(0xffffffffu, s, end);
    D = __shfl_sync(0xffffffffu, r, end);
  }
  if (depth) *depth = S;  // entries that are left (1: a single tree)
  return ok ? most : -1;
}

// Rows a kernel's table gets for tapes of up to Lmax nodes.  A stack-ordered tape of L
// nodes never has more than (L + 1) / 3 operator results waiting (each but the last waits
// beside a binary parent and has a leaf of its own), and 12 hold every tape of the
// evaluation and fit workloads (64 nodes; 99.9% of them take 9).  The other tapes use the
// same table as one row of 32 values per node, which is what the second bound is for.
template <typename T>
__host__ __device__ __forceinline__ int table_rows(int Lmax) {
  const int tree = (Lmax + 1) / 3 + 1, need = tree < 12 ? tree : 12;
  const int per_node = (Lmax + Pack<T>::V - 1) / Pack<T>::V;
  return need > per_node ? need : per_node;
}

int device_sm_count();
int max_sm_smem();  // shared memory of an SM
int check_tape_args(int64_t B, int64_t M);

// Side stream and fork/join events per device, created on first use and kept for the
// life of the process.
struct Aux {
  std::mutex mu;
  cudaStream_t stream = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr;
};
Aux* aux_for_current_device();

// The side stream of one call, forked from the caller's stream and joined back into it (a CUDA
// graph capture of the caller's stream records both); without a fork, the caller's stream.
class SideStream {
 public:
  SideStream(bool fork, cudaStream_t st) : fork_(fork), st_(st) {}
  int begin() {
    if (!fork_) return SR_OK;
    aux_ = aux_for_current_device();
    if (!aux_) return SR_ERR_CUDA;
    hold_ = std::unique_lock<std::mutex>(aux_->mu);
    const int rc = cuda_check(cudaEventRecord(aux_->fork, st_), "fork event");
    return rc ? rc : cuda_check(cudaStreamWaitEvent(aux_->stream, aux_->fork, 0), "fork wait");
  }
  cudaStream_t stream() const { return fork_ ? aux_->stream : st_; }
  // also after a failed launch: the side stream must not outlive the call
  int end() {
    if (!fork_) return SR_OK;
    const int rc = cuda_check(cudaEventRecord(aux_->join, aux_->stream), "join event");
    return rc ? rc : cuda_check(cudaStreamWaitEvent(st_, aux_->join, 0), "join wait");
  }

 private:
  bool fork_;
  cudaStream_t st_;
  Aux* aux_ = nullptr;
  std::unique_lock<std::mutex> hold_;
};

// Persistent grid for an interpreter kernel: warps per CTA and CTAs from the
// per-warp shared memory and the occupancy the kernel reaches.
struct Shape {
  int warps;
  size_t smem;
  int64_t blocks;
};
// reserve: shared memory of every SM to leave to a kernel that runs beside the grid.
bool pick_shape(const void* kern, size_t per_warp, int64_t work_items, Shape& sh, size_t reserve = 0);

}  // namespace sr
