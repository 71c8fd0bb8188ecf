// sr_adjoint.cu -- adjoint of the forward evaluation for a dense output gradient.
#include "sr_eval.cuh"
namespace sr {
template <typename T>
__device__ __forceinline__ T lds_operand(const unsigned char* wb, uint32_t w, int li) {
  return *reinterpret_cast<const T*>(wb + (w & 0xffffffu) + (uint32_t)li * (w >> 24));
}

template <typename T>
__device__ __forceinline__ T* row_at(unsigned char* wb, uint32_t off, int li) {
  return reinterpret_cast<T*>(wb + off) + li;
}

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
// One CTA per tape (grid-stride): rows L..M-1 of its (M, N) gradient block are one
// contiguous range, read with 16-byte streaming loads, four in flight per thread.
// A tape longer than the max_len the call was given is adjoined by no class grid: it
// is reported (status 602) instead of being skipped silently.
template <typename T>
__global__ void __launch_bounds__(256) padding_check_kernel(const T* __restrict__ gout,
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
    if (reinterpret_cast<uintptr_t>(p) % sizeof(T)) head = count;  // unaligned element type: scalar path
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

// ---- asynchronous staging of output-gradient rows -----------------------------------

__device__ __forceinline__ void cp_async(void* dst_smem, const void* src, int cp_bytes, int src_bytes) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst_smem));
  if (cp_bytes == 16) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(src_bytes) : "memory");
  } else if (cp_bytes == 8) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(src_bytes) : "memory");
  } else {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(src_bytes) : "memory");
  }
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int kPending>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(kPending) : "memory"); }

// Copies rows 0..L-1, points base..base+32V-1 of the gradient block G (node k, point
// n at G[k * rs + n * es]) into buf[k][32 V] (zero beyond N).  vec16 (es == 1, rows
// 16-byte aligned): each lane moves 16 bytes (E = 16 / sizeof(T) points), 32 E / (32 V)
// rows per instruction; otherwise one element per lane, point and row.
template <typename T, int V>
__device__ __forceinline__ void stage_rows(T* buf, const T* G, int L, int64_t N, int64_t rs, int64_t es,
                                           int64_t base, int lane, bool vec16) {
  constexpr int RW = 32 * V;
  if (vec16) {
    constexpr int E = 16 / sizeof(T);
    constexpr int kLanesPerRow = RW / E;
    static_assert(kLanesPerRow <= 32 && 32 % kLanesPerRow == 0, "row width");
    constexpr int kRowsPerStep = 32 / kLanesPerRow;
    const int r0 = lane / kLanesPerRow, p = (lane % kLanesPerRow) * E;
    const int64_t left = N - (base + p);
    const int bytes = left >= E ? 16 : (left > 0 ? (int)left * (int)sizeof(T) : 0);
    for (int k = r0; k < L; k += kRowsPerStep) {
      const T* src = bytes ? G + (size_t)k * rs + base + p : G;
      cp_async(buf + k * RW + p, src, 16, bytes);
    }
  } else {
#pragma unroll
    for (int v = 0; v < V; ++v) {
      const int64_t n = base + v * 32 + lane;
      const int bytes = n < N ? (int)sizeof(T) : 0;
      for (int k = 0; k < L; ++k) {
        const T* src = bytes ? G + (size_t)k * rs + n * es : G;
        cp_async(buf + k * RW + v * 32 + lane, src, (int)sizeof(T), bytes);
      }
    }
  }
  cp_async_commit();
}

// Copies the value rows of this chunk from the forward cache Cc (node k, point n at
// Cc[k * rs + n * es]) into vals[k][32 V] for the operator nodes (rows at byte offsets
// prow[0..nop) from vals_off) and the variable leaves lvar[0..nvar); the rows of the
// learnable leaves hold their gradient partial sums and are not touched.  Same copy
// shapes as stage_rows.
template <typename T, int V>
__device__ __forceinline__ void stage_value_rows(T* vals, const T* Cc, const uint32_t* prow, uint32_t vals_off,
                                                 int nop, const int* lvar, int nvar, int64_t N, int64_t rs,
                                                 int64_t es, int64_t base, int lane, bool vec16) {
  constexpr int RW = 32 * V;
  constexpr uint32_t RB = RW * (uint32_t)sizeof(T);
  const int nrows = nop + nvar;
  auto node_of = [&](int r) -> int { return r < nop ? (int)((prow[r] - vals_off) / RB) : lvar[r - nop]; };
  if (vec16) {
    constexpr int E = 16 / sizeof(T);
    constexpr int kLanesPerRow = RW / E;
    constexpr int kRowsPerStep = 32 / kLanesPerRow;
    const int r0 = lane / kLanesPerRow, p = (lane % kLanesPerRow) * E;
    const int64_t left = N - (base + p);
    const int bytes = left >= E ? 16 : (left > 0 ? (int)left * (int)sizeof(T) : 0);
    for (int r = r0; r < nrows; r += kRowsPerStep) {
      const int k = node_of(r);
      const T* src = bytes ? Cc + (size_t)k * rs + base + p : Cc;
      cp_async(vals + k * RW + p, src, 16, bytes);
    }
  } else {
#pragma unroll
    for (int v = 0; v < V; ++v) {
      const int64_t n = base + v * 32 + lane;
      const int bytes = n < N ? (int)sizeof(T) : 0;
      for (int r = 0; r < nrows; ++r) {
        const int k = node_of(r);
        const T* src = bytes ? Cc + (size_t)k * rs + n * es : Cc;
        cp_async(vals + k * RW + v * 32 + lane, src, (int)sizeof(T), bytes);
      }
    }
  }
  cp_async_commit();
}

// ------------------------------------------------------------------------------------
// Adjoint.  One warp per tape, 32 V points per chunk (V points per lane: the per-node
// decode and dispatch serve V points).  The host launches one persistent grid per
// class of tape lengths (Llo, Lhi], each sized for its class's shared memory, so short
// tapes run at the occupancy their size allows; every grid scans the whole work order
// and takes the tapes of its class.  Per tape the warp compiles its nodes into an
// operator program (NO_OP nodes included: their value NaN and their adjoint check
// matter) whose operands are precomputed addresses in the warp's shared memory:
//   source word = byte offset (bits 0..23) | lane stride in bytes (bits 24..31): the
//                 value row of an operator node or a variable leaf (stride sizeof(T))
//                 or the broadcast entry of any other leaf (stride 0);
//   adjoint destination = byte offset of the child's adjoint row.
// Every node has an adjoint row.  Per chunk the output-gradient rows are staged into
// them with cp.async.  With the forward cache (kCached: the reference's backward reads
// it too) the value rows of the operator nodes and variables are staged from it in the
// same way, the cache holding exactly the values the forward kernel computed; without
// it the operator nodes are recomputed while the copies are in flight.  The reverse
// sweep then adds the contributions into the children's rows in the
// reference's order (parents from the last to the first, child 0 before child 1), and
// the leaves are reduced afterwards.  A learnable constant's operand is a broadcast
// entry, so its value row is free and holds its per-lane gradient sums over the
// chunks; one butterfly per constant and set ends the sum (a fixed order: grad_C is
// deterministic).
// ------------------------------------------------------------------------------------
struct BwdLayout {
  uint32_t pcode, psa, psb, prow, pda, pdb, lcon, lvar, bc, vals, adj, bytes;
};

template <typename T, int V>
__host__ __device__ __forceinline__ BwdLayout backward_layout(int Lmax) {
  const uint32_t lb = (uint32_t)align16((size_t)Lmax * 4);
  BwdLayout l;
  l.pcode = lb;  // the tape words sit at offset 0
  l.psa = 2 * lb;
  l.psb = 3 * lb;
  l.prow = 4 * lb;
  l.pda = 5 * lb;
  l.pdb = 6 * lb;
  l.lcon = 7 * lb;
  l.lvar = 8 * lb;
  l.bc = 9 * lb;
  l.vals = l.bc + (uint32_t)align16((size_t)(Lmax + 1) * sizeof(T));
  const uint32_t rows = (uint32_t)Lmax * 32u * V * (uint32_t)sizeof(T);
  l.adj = l.vals + rows;
  l.bytes = l.adj + rows;
  return l;
}

template <typename T, bool kMulti, int V, bool kCached>
__global__ void __launch_bounds__(256, 4) eval_backward_kernel(
    const T* __restrict__ X, int64_t N, int64_t n_x, const uint32_t* __restrict__ desc,
    const int32_t* __restrict__ meta, const int32_t* __restrict__ order, int64_t B, int64_t M, int Llo, int Lhi,
    const T* __restrict__ C, int64_t c_sb, int64_t c_sm, int64_t c_sk, int64_t K_, const T* __restrict__ cache,
    const T* __restrict__ gout, T* __restrict__ gC, T* __restrict__ gX, int32_t* __restrict__ status, bool vec16,
    bool cvec16) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int64_t K = kMulti ? K_ : 1;  // one constant set: the strides fold at compile time
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  constexpr uint32_t RW = 32u * V;                       // elements per row
  constexpr uint32_t RB = RW * (uint32_t)sizeof(T);      // bytes per row
  constexpr uint32_t kRowStride = (uint32_t)sizeof(T) << 24;
  const BwdLayout ly = backward_layout<T, V>(Lhi);
  unsigned char* wb = smem + (size_t)warp * ly.bytes;
  uint32_t* tape = reinterpret_cast<uint32_t*>(wb);
  uint32_t* pcode = reinterpret_cast<uint32_t*>(wb + ly.pcode);
  uint32_t* psa = reinterpret_cast<uint32_t*>(wb + ly.psa);
  uint32_t* psb = reinterpret_cast<uint32_t*>(wb + ly.psb);
  uint32_t* prow = reinterpret_cast<uint32_t*>(wb + ly.prow);
  uint32_t* pda = reinterpret_cast<uint32_t*>(wb + ly.pda);
  uint32_t* pdb = reinterpret_cast<uint32_t*>(wb + ly.pdb);
  int* lcon = reinterpret_cast<int*>(wb + ly.lcon);
  int* lvar = reinterpret_cast<int*>(wb + ly.lvar);
  T* bc = reinterpret_cast<T*>(wb + ly.bc);
  T* vals = reinterpret_cast<T*>(wb + ly.vals);
  T* adj = reinterpret_cast<T*>(wb + ly.adj);
  const uint32_t adj_delta = ly.adj - ly.vals;
  const unsigned below = (1u << lane) - 1u;
  for (int64_t ti = (int64_t)blockIdx.x * nwarp + warp; ti < B; ti += (int64_t)gridDim.x * nwarp) {
    const int64_t b = order ? (int64_t)order[ti] : ti;
    const int L = meta[b * 4];
    if (L <= Llo || L > Lhi) continue;  // another class's grid takes it (warp-uniform)
    for (int k = lane; k < L; k += 32) tape[k] = desc[b * M + k];
    if (lane == 0) bc[0] = T(0);
    __syncwarp();
    // source word of operand node c: its value row, or its broadcast entry
    auto src_word = [&](int c) -> uint32_t {
      const int cc = code_of(tape[c]);
      if (cc == NO_OP || cc == VAR || arity_of(cc) >= 1) return (ly.vals + (uint32_t)c * RB) | kRowStride;
      return ly.bc + (uint32_t)(1 + c) * (uint32_t)sizeof(T);
    };
    // compaction: operator nodes, learnable and variable leaves; the broadcast
    // entries of fixed leaves (and of codes that evaluate to 0) now
    int nop = 0, ncon = 0, nvar = 0;
    for (int k0 = 0; k0 < L; k0 += 32) {
      const int k = k0 + lane;
      const uint32_t d = k < L ? tape[k] : 0u;
      const int code = k < L ? code_of(d) : -1;
      const bool isop = k < L && (code == NO_OP || arity_of(code) >= 1);
      const bool iscon = code == LEARNABLE, isvar = code == VAR;
      const unsigned mo = __ballot_sync(0xffffffffu, isop);
      const unsigned mc = __ballot_sync(0xffffffffu, iscon);
      const unsigned mv = __ballot_sync(0xffffffffu, isvar);
      if (isop) {
        const int ar = arity_of(code);
        const int pos = nop + __popc(mo & below);
        const uint32_t own = ly.adj + (uint32_t)k * RB;  // never written through (arity < 2)
        uint32_t sa = ly.bc, sb = ly.bc, da = own, db = own;
        if (ar >= 1) {
          sa = src_word(child0(d));
          da = ly.adj + (uint32_t)child0(d) * RB;
        }
        if (ar == 2) {
          sb = src_word(child1(d));
          db = ly.adj + (uint32_t)child1(d) * RB;
        }
        pcode[pos] = (uint32_t)dense_op(code);
        psa[pos] = sa;
        psb[pos] = sb;
        prow[pos] = ly.vals + (uint32_t)k * RB;
        pda[pos] = da;
        pdb[pos] = db;
      } else if (k < L && !iscon && !isvar) {
        bc[1 + k] = node_value<T>(code, T(0), T(0), T(0), T(0));
      }
      if (iscon) lcon[ncon + __popc(mc & below)] = k;
      if (isvar) lvar[nvar + __popc(mv & below)] = k;
      nop += __popc(mo);
      ncon += __popc(mc);
      nvar += __popc(mv);
    }
    int err = 0;
    const int64_t nchunks = (N + RW - 1) / RW;
    // K constant sets, one after the other: grad_out is (B, M, N, K), set kk of
    // node k, point n at ((b M + k) N + n) K + kk
    for (int64_t kk = 0; kk < K; ++kk) {
      const T* Crow = C + b * c_sb + kk * c_sk;
      for (int j = lane; j < ncon; j += 32) bc[1 + lcon[j]] = __ldg(Crow + (int64_t)lcon[j] * c_sm);
      for (int j = 0; j < ncon; ++j) {
#pragma unroll
        for (int v = 0; v < V; ++v) vals[lcon[j] * RW + v * 32 + lane] = T(0);
      }
      const T* G = gout + (size_t)b * M * N * K + kk;
      const T* Cc = kCached ? cache + (size_t)b * M * N * K + kk : nullptr;
      const int64_t rs = N * K;
      __syncwarp();
      for (int64_t c = 0; c < nchunks; ++c) {
        const int64_t base = c * RW;
        int64_t nn[V];
        bool valid[V];
#pragma unroll
        for (int v = 0; v < V; ++v) {
          const int64_t n = base + v * 32 + lane;
          valid[v] = n < N;
          nn[v] = valid[v] ? n : N - 1;
        }
        // the adjoint seeds (grad_out rows of this chunk) are in flight while the node
        // values are recomputed.  Seeding with the raw values instead of 0 + grad_out
        // (the reference's zeros_like(cache).add_(grad_output)) can only flip the sign
        // of a zero seed, which no output can see: a zero adjoint contributes nothing
        stage_rows<T, V>(adj, G, L, N, rs, K, base, lane, vec16);
        if constexpr (kCached) {
          stage_value_rows<T, V>(vals, Cc, prow, ly.vals, nop, lvar, nvar, N, rs, K, base, lane, cvec16);
        } else {
          for (int j = 0; j < nvar; ++j) {
            const int k = lvar[j];
            const int var = child0(tape[k]);
#pragma unroll
            for (int v = 0; v < V; ++v) vals[k * RW + v * 32 + lane] = __ldg(X + nn[v] * n_x + var);
          }
          __syncwarp();
          for (int i = 0; i < nop; ++i) {
            const int code = (int)pcode[i];
            const uint32_t sa = psa[i], sb = psb[i], pr = prow[i];
            T a[V], bb[V], r[V];
#pragma unroll
            for (int v = 0; v < V; ++v) {
              a[v] = lds_operand<T>(wb, sa, v * 32 + lane);
              bb[v] = lds_operand<T>(wb, sb, v * 32 + lane);
            }
            op_value_v<T, V>(code, a, bb, r);
#pragma unroll
            for (int v = 0; v < V; ++v) *row_at<T>(wb, pr, v * 32 + lane) = r[v];
          }
        }
        cp_async_wait<0>();
        __syncwarp();
        for (int i = nop - 1; i >= 0; --i) {
          const int code = (int)pcode[i];
          const uint32_t sa = psa[i], sb = psb[i], pr = prow[i], da = pda[i], db = pdb[i];
          T g[V], a[V], bb[V], vv[V], o0[V], o1[V];
          bool a0[V], a1[V];
          int e[V];
#pragma unroll
          for (int v = 0; v < V; ++v) {
            const int li = v * 32 + lane;
            g[v] = *row_at<T>(wb, pr + adj_delta, li);
            a[v] = lds_operand<T>(wb, sa, li);
            bb[v] = lds_operand<T>(wb, sb, li);
            vv[v] = *row_at<T>(wb, pr, li);
          }
          op_adjoint_v<T, V>(code, g, a, bb, vv, a0, o0, a1, o1, e);
#pragma unroll
          for (int v = 0; v < V; ++v) {
            if (valid[v]) {
              const int li = v * 32 + lane;
              if (e[v] && !err) err = e[v];
              if (a0[v]) { T* d = row_at<T>(wb, da, li); *d = M_<T>::add(*d, o0[v]); }
              if (a1[v]) { T* d = row_at<T>(wb, db, li); *d = M_<T>::add(*d, o1[v]); }
            }
          }
        }
        // leaves: every contribution from the parents has arrived
        for (int j = 0; j < ncon; ++j) {
          const int k = lcon[j];
#pragma unroll
          for (int v = 0; v < V; ++v) {
            const T g = adj[k * RW + v * 32 + lane];
            if (valid[v] && g != T(0)) vals[k * RW + v * 32 + lane] = M_<T>::add(vals[k * RW + v * 32 + lane], g);
          }
        }
        if (gX) {
          for (int j = 0; j < nvar; ++j) {
            const int k = lvar[j];
            const int var = child0(tape[k]);
#pragma unroll
            for (int v = 0; v < V; ++v) {
              const T g = adj[k * RW + v * 32 + lane];
              if (valid[v] && g != T(0)) atomicAdd(gX + nn[v] * n_x + var, g);
            }
          }
        }
        __syncwarp();  // every lane is done with the seeds before the next chunk's land
      }
      // the constants' sums (lane partials in point order, then a butterfly) replace
      // their values in the broadcast entries
      for (int j = 0; j < ncon; ++j) {
        const int k = lcon[j];
        T part = vals[k * RW + lane];
#pragma unroll
        for (int v = 1; v < V; ++v) part = M_<T>::add(part, vals[k * RW + v * 32 + lane]);
        part = warp_sum(part);
        if (lane == 0) bc[1 + k] = part;
      }
      __syncwarp();
      // gradient row of this set: constant nodes get their sums, everything else 0
      T* gCrow = gC + (size_t)b * M * K + kk;
      for (int64_t k = lane; k < M; k += 32) {
        T val = T(0);
        if (k < L && code_of(tape[k]) == LEARNABLE) val = bc[1 + k];
        gCrow[k * K] = val;
      }
      __syncwarp();
    }  // sets
    err = __reduce_max_sync(0xffffffffu, err);
    if (err && lane == 0) report_adjoint(status, err);
    __syncwarp();
  }
}

template <typename T, bool kMulti, int V, bool kCached>
static int launch_backward_v(const T* X, int64_t N, int64_t n_x, const uint32_t* desc, const int32_t* meta,
                             const int32_t* order, int64_t B, int64_t M, int Llo, int Lhi, const T* C, int64_t c_sb,
                             int64_t c_sm, int64_t c_sk, int64_t K, const T* cache, const T* gout, T* gC, T* gX,
                             int32_t* status, bool vec16, bool cvec16, cudaStream_t st) {
  const size_t per_warp = backward_layout<T, V>(Lhi).bytes;
  Shape sh;
  auto kern = eval_backward_kernel<T, kMulti, V, kCached>;
  if (!pick_shape(reinterpret_cast<const void*>(kern), per_warp, B, sh)) {
    set_error("tape of %d nodes does not fit in shared memory", Lhi);
    return SR_ERR_UNSUPPORTED;
  }
  kern<<<(unsigned)sh.blocks, sh.warps * 32, sh.smem, st>>>(X, N, n_x, desc, meta, order, B, M, Llo, Lhi, C, c_sb,
                                                           c_sm, c_sk, K, cache, gout, gC, gX, status, vec16, cvec16);
  return launch_check("eval_backward_kernel");
}

// One point per lane: two points per lane (one dispatch for both, their chains
// interleaved in registers) ran at half the resident warps, and the adjoint took 1.4x as
// long on a GB300 (10.3 ms against 7.1 ms for 65536 tapes of mean length 20, N = 1024),
// so only the one-point kernels are instantiated.
template <typename T>
static int launch_backward_class(const T* X, int64_t N, int64_t n_x, const uint32_t* desc, const int32_t* meta,
                                 const int32_t* order, int64_t B, int64_t M, int Llo, int Lhi, const T* C,
                                 int64_t c_sb, int64_t c_sm, int64_t c_sk, int64_t K, const T* cache, const T* gout,
                                 T* gC, T* gX, int32_t* status, bool vec16, bool cvec16, cudaStream_t st) {
#define SR_BWD_ARGS X, N, n_x, desc, meta, order, B, M, Llo, Lhi, C, c_sb, c_sm, c_sk, K, cache, gout, gC, gX, status, \
                    vec16, cvec16, st
  if (K == 1)
    return cache ? launch_backward_v<T, false, 1, true>(SR_BWD_ARGS) : launch_backward_v<T, false, 1, false>(SR_BWD_ARGS);
  return cache ? launch_backward_v<T, true, 1, true>(SR_BWD_ARGS) : launch_backward_v<T, true, 1, false>(SR_BWD_ARGS);
#undef SR_BWD_ARGS
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
  Aux* aux = aux_for_current_device();
  if (!aux) return SR_ERR_CUDA;
  std::lock_guard<std::mutex> hold(aux->mu);
  rc = cuda_check(cudaEventRecord(aux->fork, st), "fork event");
  if (!rc) rc = cuda_check(cudaStreamWaitEvent(aux->stream, aux->fork, 0), "fork wait");
  if (rc) return rc;
  // 16-byte staging needs every (tape, row, chunk) start 16-byte aligned
  const bool vec16 =
      K == 1 && (reinterpret_cast<uintptr_t>(gout) % 16 == 0) && (N % (16 / (int64_t)sizeof(T)) == 0);
  const bool cvec16 =
      K == 1 && (reinterpret_cast<uintptr_t>(cache) % 16 == 0) && (N % (16 / (int64_t)sizeof(T)) == 0);
  // one persistent grid per class of tape lengths (Llo, Lhi]: (48, Lmax], (32, 48],
  // (16, 32], [0, 16], as far as Lmax reaches.  The longest class is bound by the
  // warps its shared memory lets reside (1.5x its tables cost 23% of the adjoint's time
  // on a GB300, the same for the middle class 5%, the shortest nothing): splitting it at
  // 48 gained 2%, further splits at 40, 56 or 24 lost more to the extra grids' tails.
  const int bound[3] = {48, 32, 16};
  int cls[4][2], nc = 0, hi = Lmax;
  for (int j = 0; j < 3; ++j) {
    if (hi > bound[j]) {
      cls[nc][0] = bound[j];
      cls[nc][1] = hi;
      ++nc;
      hi = bound[j];
    }
  }
  cls[nc][0] = -1;
  cls[nc][1] = hi;
  ++nc;
  for (int ci = 0; ci < nc; ++ci) {
    rc = launch_backward_class<T>(X, N, n_x, desc, meta, order, B, M, cls[ci][0], cls[ci][1], C, c_sb, c_sm, c_sk, K,
                                  cache, gout, gC, gX, status, vec16, cvec16, st);
    if (rc) break;
    if (ci == 0) {
      // enqueued after the first adjoint grid, so that grid's CTAs are placed first and
      // the check's CTAs take the registers and warp slots they leave
      int64_t pblocks = (int64_t)device_sm_count() * 2;
      if (pblocks > B) pblocks = B;
      padding_check_kernel<T><<<(unsigned)pblocks, 256, 0, aux->stream>>>(gout, meta, B, M, N * K, Lmax, status);
      rc = launch_check("padding_check_kernel");
      if (rc) break;
    }
  }
  // join (also after a failed launch: the side stream must not outlive the call)
  const int rj = cuda_check(cudaEventRecord(aux->join, aux->stream), "join event");
  const int rw = rj ? rj : cuda_check(cudaStreamWaitEvent(st, aux->join, 0), "join wait");
  return rc ? rc : rw;
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
