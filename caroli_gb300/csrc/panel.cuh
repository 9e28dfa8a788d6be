// Panel sweeps of large fronts and roots spread over a cluster of CTAs, and the kernel that brings
// the rest of the matrix up to date with a panel.
//
// A 32-column panel is a chain of 32 pivot steps over its candidate rows. FP64 runs at about two
// multiply-adds per clock and SM here, so one CTA per matrix is bound by its own SM's FP64 pipe as
// soon as there are fewer matrices than SMs: the chain itself is short. Two kernels replace it:
//   panel_sweep_kernel  the candidate rows split over the CTAs of a cluster, an exchange per
//                       pivot step; each CTA publishes its best candidate row, already scaled by the
//                       reciprocal of its pivot, into every CTA's shared memory, so a step costs one
//                       exchange and no CTA computes a reciprocal or a pivot search twice;
//   panel_rest_kernel   what is independent per row (the rows outside the candidates replay the
//                       steps) and per column (the pivot rows of the other columns), over as many
//                       CTAs as there are pieces of 4 to 16 rows and columns; trail::rest_kernel
//                       (trail.cuh) in its place in the trailing form.
//
// Two forms (InvTask::trail):
//   full   Gauss-Jordan, as inv_panel_kernel: the swept panel holds [P^-1; -a P^-1] and every other
//          row and column is updated (roots, and fronts whose factors are kept);
//   trail  LU: only the rows and columns after the panel are updated, which is all a front that
//          hands up its Schur complement needs (FP64 fronts below the root: nothing reads their
//          F11^-1, X or W). The panel holds the columns of L below the pivots (the multipliers
//          of the scaled pivot rows); L11 with the reciprocals of the pivots on its diagonal.
// Measured with ozaki.cuh against the former FP64 path (one CTA per matrix and panel, rank-32 updates on
// the FP64 pipe, every row and column updated): panels + updates of two 48 x 24 x 24 cubic wires (fronts
// up to 1 728, root 1 152) 337 -> 27 ms, of 16 BHZ 200 x 64 solves (fronts up to 384) 88 -> 16 ms, of one
// 32 x 32 square (fronts up to 94) 1.57 -> 0.40 ms (24, 13 and 0.39 before outputs far below the largest were computed
// again, see oz::far_below).
//
// The pivots (largest modulus among the candidate rows, ties to the smaller row) and the test
// |pivot| > tol max|F11| are those of inv_panel_kernel.
#pragma once
#include <cooperative_groups.h>

#include "dense.cuh"
#include "ozaki.cuh"

namespace caroli {

constexpr int PS_THREADS = 256;
constexpr int PS_PERM = 3 * GJ_KB + 4;  // ints of InvTask::perm: source rows, displaced rows, their sources, count

// Candidate rows per CTA of a cluster of c for m candidates (a multiple of 8: a warp takes 8 x 4 entries).
__host__ __device__ inline int panel_rows(int m, int c) { return ((m + c - 1) / c + 7) / 8 * 8; }
// Dynamic shared memory: the rows (r x kb), the column buffer (2 r), the published rows of every
// CTA (2 x c x kb), row k (2 x kb), keys with their rows (2 x c).
__host__ __device__ inline size_t panel_sweep_bytes(int r, int c, size_t vbytes) {
  return ((size_t)r * GJ_KB + 2 * (size_t)r + 2 * (size_t)c * GJ_KB + 2 * GJ_KB) * vbytes + 2 * (size_t)c * 16 + 16;
}

// The lane holding the largest key of the warp, ties to the smallest index; -1 when every key is 0. The
// upper words mostly decide it: one warp reduction and a vote.
__device__ __forceinline__ int key_argmax(unsigned long long key, int idx) {
  const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
  const unsigned th = __reduce_max_sync(0xffffffffu, hi);
  unsigned in = __ballot_sync(0xffffffffu, hi == th);
  if (__popc(in) > 1) {
    const unsigned tl = __reduce_max_sync(0xffffffffu, hi == th ? lo : 0u);
    const bool top = hi == th && lo == tl;
    const int first = __reduce_min_sync(0xffffffffu, top ? idx : 0x7fffffff);
    in = __ballot_sync(0xffffffffu, top && idx == first && key != 0ull);
  }
  return __ffs(in) - 1;
}
// Shared-memory address of the same location in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t cluster_addr(const void* p, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(tc::smem_addr(p)), "r"(rank));
  return r;
}
// 16 bytes into a CTA of the cluster, counted on its barrier when they have arrived.
__device__ __forceinline__ void store_remote(uint32_t addr, uint4 v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr),
               "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void store_remote(uint32_t addr, double2 v, uint32_t bar) {
  store_remote(addr, *reinterpret_cast<const uint4*>(&v), bar);
}
// Waits (bounded) for a phase completed by other CTAs of the cluster.
__device__ __forceinline__ bool cluster_wait(uint64_t* bar, uint32_t parity, uint32_t limit) {
  for (uint32_t i = 0; i < limit; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, "
        "p;\n}\n"
        : "=r"(ok)
        : "r"(tc::smem_addr(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// max |a_ij|^2 over the leading npiv rows and columns of every matrix, into *scale2 (zeroed before;
// non-negative doubles order as integers). grid (matrices, column chunks).
template <typename T>
__global__ void __launch_bounds__(256) panel_scale_kernel(const InvTask* __restrict__ tasks) {
  using V = typename Cx<T>::V;
  const InvTask t = tasks[blockIdx.x];
  const V* A = static_cast<const V*>(t.a);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  NormKey<T> mt = 0;
  for (int j = blockIdx.y * 8 + w; j < t.npiv; j += gridDim.y * 8)
    for (int i = lane; i < t.npiv; i += 32) mt = max(mt, norm_key(cnorm(A[i + (int64_t)j * t.ld])));
  int first = 0;
  mt = warp_top(mt, first);
  if (lane == 0 && mt)
    atomicMax(reinterpret_cast<unsigned long long*>(t.scale2), (unsigned long long)__double_as_longlong(key_norm<T>(mt)));
}

// grid: matrices x cluster (clusters along x), PS_THREADS threads. R: rows per CTA.
//
// Per step: every warp waits for the C candidates and row k and picks the winner; the warp in turn
// updates the four columns around column k + 1 and searches it (and takes the reciprocal) while the
// others update the rest; a block barrier; four warps scale the CTA's candidate row and store it into every
// CTA, four store row k + 1. The stores are asynchronous and counted in bytes on the receiver's mbarrier
// (a cluster barrier per step, with its release of the stores, cost 2 400 of a step's 4 400 clocks; the
// stores' flight still takes about 1 500 of 3 900 with 8 rows per CTA). Two
// sets of slots suffice: a CTA stores step k + 2's rows only after it has received every CTA's for step
// k + 1, which those sent after reading step k's.
// An FP64 instruction holds its scheduler for 64 clocks whatever its active lanes, so what is repeated per
// warp is kept to integers, and entries are taken 8 rows x 4 columns at a time to leave few idle lanes.
template <typename T>
__global__ void __launch_bounds__(PS_THREADS) panel_sweep_kernel(const InvTask* __restrict__ tasks, int k0, double tol,
                                                                 int R, const JobDesc* __restrict__ jobs,
                                                                 int32_t* __restrict__ status, uint32_t wait_limit) {
  using V = typename Cx<T>::V;
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_piv[GJ_KB];
  __shared__ unsigned long long s_key;
  __shared__ int s_loc;
  __shared__ V s_inv;
  __shared__ __align__(8) uint64_t arrived[2];
  cg::cluster_group cluster = cg::this_cluster();
  const int C = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const InvTask t = tasks[blockIdx.x / C];
  const int np = t.npiv;
  if (k0 >= np || *t.bad) return;  // uniform in the cluster: *bad is only set after its first barrier
  const int kb = min(GJ_KB, np - k0), m = np - k0;
  const bool trail = t.trail != 0;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int r8 = lane & 7, c4 = lane >> 3;
  const int r0 = rank * R, rows = max(0, min(R, m - r0));
  V* F = reinterpret_cast<V*>(smem_raw);
  V* cb = F + (size_t)R * GJ_KB;            // 2 x R: column k of the own rows
  V* prow = cb + 2 * (size_t)R;             // 2 x C x kb: scaled candidate rows of every CTA
  V* krow = prow + 2 * (size_t)C * GJ_KB;   // 2 x kb: row k before step k
  uint4* cand = reinterpret_cast<uint4*>(krow + 2 * GJ_KB);  // 2 x C: key, row (bit 30: refused)
  const uint32_t tx = (uint32_t)(C * (kb * sizeof(V) + 16) + kb * sizeof(V));  // bytes of a step
  if (tid == 0) {
    tc::mbar_init(&arrived[0], 1);
    tc::mbar_init(&arrived[1], 1);
    tc::mbar_arrive_expect_tx(&arrived[0], tx);
    if (kb > 1) tc::mbar_arrive_expect_tx(&arrived[1], tx);
  }
  V* A = static_cast<V*>(t.a) + k0 + (int64_t)k0 * t.ld;
  for (int j = w; j < kb; j += PS_THREADS / 32)
    for (int i = lane; i < rows; i += 32) {
      const V v = A[(r0 + i) + (int64_t)j * t.ld];
      F[i + (size_t)j * R] = v;
      if (j == 0) cb[i] = v;
    }
  __syncthreads();
  const unsigned long long refuse = refuse_key<T>(tol * tol * *t.scale2);
  // The CTA's best candidate of column k among its rows at or past k: key, local row and the
  // reciprocal of the pivot. One warp, the candidates' entries in `col`.
  auto search = [&](int k, const V* col) {
    unsigned long long key = 0;
    int loc = 0x7fffffff;
    for (int i = lane; i < rows; i += 32)
      if (r0 + i >= k) {
        const unsigned long long q = norm_key(cnorm(col[i]));
        if (q > key) { key = q; loc = i; }
      }
    const int win = key_argmax(key, loc);
    if (win < 0 || !__shfl_sync(0xffffffffu, key != 0ull, win)) {
      if (lane == 0) s_key = 0;
      return;
    }
    if (lane != win) return;
    s_inv = cinv(col[loc]);
    s_key = key;
    s_loc = key > refuse ? loc : loc | 1 << 30;
  };
  // Publishes the candidate found by `search`, scaled (warps 0-3: eight columns each, the CTAs split four
  // ways over the lanes), and row k if it is here (warps 4-7).
  auto publish = [&](int k) {
    const int par = k & 1, col = 8 * (w & 3) + r8;
    const unsigned long long key = s_key;
    if (w < 4) {
      if (col < kb) {
        V v = cx<V>(0.0, 0.0);
        if (key) {
          const V raw = F[(s_loc & ~(1 << 30)) + (size_t)col * R], inv = s_inv;
          v = col == k ? inv : ((trail && col < k) ? raw : cmul(raw, inv));
        }
        for (int c = c4; c < C; c += 4)
          store_remote(cluster_addr(prow + ((size_t)par * C + rank) * GJ_KB + col, c), v, cluster_addr(&arrived[par], c));
      }
    } else {
      if (k >= r0 && k < r0 + rows && col < kb) {
        const V v = F[(k - r0) + (size_t)col * R];
        for (int c = c4; c < C; c += 4)
          store_remote(cluster_addr(krow + par * GJ_KB + col, c), v, cluster_addr(&arrived[par], c));
      }
      if (w == 4 && lane < C) {
        const int loc = key ? s_loc : 0;
        store_remote(cluster_addr(cand + par * C + rank, lane),
                     make_uint4((uint32_t)key, (uint32_t)(key >> 32), (uint32_t)((r0 + (loc & ~(1 << 30))) | (loc & (1 << 30))), 0u),
                     cluster_addr(&arrived[par], lane));
      }
    }
    __syncwarp();
  };
  if (w == 0) search(0, cb);
  __syncwarp();
  cluster_sync_all();  // every CTA of the cluster runs, its barriers armed, before its shared memory is written
  publish(0);
  const int quads = (kb + 3) / 4, groups = (rows + 7) / 8;
  bool bad = false, late = false;
  for (int k = 0; k < kb; ++k) {
    const int par = k & 1;
    // A wait that runs out marks the solve, then waits for the same stores once more with a bound of its own: no CTA
    // may leave while they are in flight. They mostly arrive, and the sweep goes on; else it ends here.
    bool here = cluster_wait(&arrived[par], (uint32_t)((k >> 1) & 1), wait_limit);
    late |= !here;
    if (!here) here = cluster_wait(&arrived[par], (uint32_t)((k >> 1) & 1), TCU_WAIT);
    const bool lost = !__all_sync(0xffffffffu, here);
    const uint4 cd = lane < C ? cand[par * C + lane] : make_uint4(0u, 0u, 0x3fffffffu, 0u);
    const unsigned long long key = ((unsigned long long)cd.y << 32) | cd.x;
    const int id = (int)cd.z;
    const int win = key_argmax(key, id & ~(1 << 30));
    const int wid = __shfl_sync(0xffffffffu, id, max(win, 0));
    // A refused pivot (the same decision in every CTA) or stores that never came end the sweep at the block
    // barrier below; what the step computes until then is dropped.
    const bool refused = win < 0 || (wid & (1 << 30));
    if (tid == 0 && k + 2 < kb) tc::mbar_arrive_expect_tx(&arrived[par], tx);
    const int p = wid;
    const V* pr = prow + ((size_t)par * C + max(win, 0)) * GJ_KB;
    const V* kr = krow + par * GJ_KB;
    const V* ck = cb + (size_t)par * R;
    V* cn = cb + (size_t)(par ^ 1) * R;
    const int lk = k - r0, lp = p - r0;  // rows k and p among the own rows
    // Columns 4 q .. 4 q + 3 of the row groups g and gb (gb < 0: one): two groups' loads and chains in flight.
    // Without branches: column k (full form) is updated from zero, row k takes the pivot row afterwards.
    auto block = [&](int q, int g, int gb) {
      const int j = 4 * q + c4;
      const V prj = pr[j];
      V c[2], v[2];
      bool on[2];
      int il[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        il[u] = 8 * (u ? gb : g) + r8;
        on[u] = (u == 0 || gb >= 0) && j < kb && il[u] < rows && !(trail && (j <= k || il[u] <= lk));
        c[u] = v[u] = cx<V>(0.0, 0.0);
        if (on[u]) {
          c[u] = il[u] == lp ? kr[k] : ck[il[u]];
          v[u] = il[u] == lp ? kr[j] : F[il[u] + (size_t)j * R];
        }
        if (j == k) v[u] = cx<V>(0.0, 0.0);
      }
#pragma unroll
      for (int u = 0; u < 2; ++u)
        if (u == 0 || gb >= 0) v[u] = cfms_pk(v[u], c[u], prj);
#pragma unroll
      for (int u = 0; u < 2; ++u)
        if (on[u]) {
          if (il[u] == lk) v[u] = prj;
          F[il[u] + (size_t)j * R] = v[u];
          if (j == k + 1) cn[il[u]] = v[u];
        }
    };
    // The four columns around column k + 1 first, over all warps (one group of rows: by the warp in turn);
    // then the warp in turn searches column k + 1 while the others take the remaining columns.
    const int g0 = trail ? min(groups, max(0, lk + 1) >> 3) : 0;
    const int q1 = (k + 1) >> 2, turn = k & 7;
    if (groups > 1 && q1 < quads) {
      for (int g = g0 + ((w - turn) & 7); g < groups; g += 16) block(q1, g, g + 8 < groups ? g + 8 : -1);
      __syncthreads();
    }
    if (w == turn) {
      if (groups <= 1 && q1 < quads) {
        if (g0 < groups) block(q1, g0, -1);
        __syncwarp();
      }
      if (k + 1 < kb) search(k + 1, cn);
      __syncwarp();
    } else {
      const int me = (w - turn - 1) & 7;  // 0 .. 6
      const int others = trail ? quads - q1 - 1 : (q1 < quads ? quads - 1 : quads), ng = groups - g0;
      const int qs = q1 < quads ? q1 + 1 : 0;
      if (ng == 1) {
        for (int x = me; x < others; x += 7) block(qs + x < quads ? qs + x : qs + x - quads, g0, -1);
      } else if (ng > 1) {
        const int pairs = (ng + 1) >> 1;
        int gp = me % pairs;  // seven warps walk the pairs of groups of one quad after another
        for (int x = me / pairs; x < others;) {
          const int g = g0 + 2 * gp;
          block(qs + x < quads ? qs + x : qs + x - quads, g, g + 1 < groups ? g + 1 : -1);
          gp += 7;
          while (gp >= pairs) { gp -= pairs; ++x; }
        }
      }
      if (me == 6) {
        if (rank == 0) {
          if (lane == 0) s_piv[k] = p;
          if (lane < kb) static_cast<V*>(t.prows)[k * GJ_KB + lane] = pr[lane];
        }
        if (trail && lane <= k) {  // the interchange of the columns done: row k takes the pivot row's, row p row k's
          if (lk >= 0 && lk < rows) F[lk + (size_t)lane * R] = pr[lane];
          if (p != k && lp >= 0 && lp < rows) F[lp + (size_t)lane * R] = kr[lane];
        }
      }
    }
    if (__syncthreads_or(refused || lost)) {
      if (lost && lane == 0) {
        *t.bad = 1;
      } else if (rank == 0 && tid == 0) {
        *t.bad = 1;
        if (trail && t.front >= 0) jobs[t.job].fail[t.front] = 1;
      }
      bad = true;
      break;
    }
    if (k + 1 < kb) publish(k + 1);
  }
  if (__any_sync(0xffffffffu, late) && lane == 0) status[t.job] = ST_TIMEOUT;
  __syncwarp();
  cluster_sync_all();  // no CTA leaves while another may still store into it
  if (bad) return;
  for (int j = w; j < kb; j += PS_THREADS / 32)
    for (int i = lane; i < rows; i += 32) A[(r0 + i) + (int64_t)j * t.ld] = F[i + (size_t)j * R];
  if (rank == 0 && w == 0) {
    if (lane < kb) t.piv[k0 + lane] = k0 + s_piv[lane];
    panel_permutation(s_piv, kb, t.perm);
  }
}

// The recorded steps replayed on a row of the panel held by LPR lanes, lane h the entries LPR i + h:
// step k subtracts entry k times row k of `pk` (stride GJ_KB) from all others, entry k becoming -a pk[k].
template <int LPR, typename V>
__device__ __forceinline__ void replay_row(V (&b)[GJ_KB / LPR], const V* pk, int kb, int h) {
  constexpr int Q = GJ_KB / LPR;
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < GJ_KB; ++k) {
    if (k >= kb) break;
    const V own = b[k / LPR];
    const int src = (lane & ~(LPR - 1)) | (k % LPR);
    const V ak = cx<V>(__shfl_sync(0xffffffffu, own.x, src), __shfl_sync(0xffffffffu, own.y, src));
    if (h == k % LPR) b[k / LPR] = cx<V>(0.0, 0.0);  // entry k: 0 - a pk[k]
#pragma unroll
    for (int i = 0; i < Q; ++i) b[i] = cfms_pk(b[i], ak, pk[k * GJ_KB + LPR * i + h]);
  }
}

// After a panel's sweep in the full form (the trailing form: trail.cuh): grid (matrices, row pieces then
// column pieces), NT threads, LPR lanes per row or column (a piece has NT / LPR of them).
// Row piece: rows outside the candidates replay the recorded steps. With oa set (FP64), every row the
// update reads also becomes an operand row.
// Column piece: the pivot rows of the columns outside the panel into Y (or B', or the FP64 operand), the
// displaced rows into place.
// LPR: 16 while the pieces of 4 do not fill the GPU (a piece is then a chain of 256 FP64
// instructions per warp instead of 1 024), 4 past that (fewer shuffles per entry).
template <typename T, int LPR, int NT>
__global__ void __launch_bounds__(NT) panel_rest_kernel(const InvTask* __restrict__ tasks, int k0,
                                                                int row_pieces) {
  using V = typename Cx<T>::V;
  constexpr int Q = GJ_KB / LPR, PIECE = NT / LPR;
  __shared__ V sm[GJ_KB * GJ_KB];
  const InvTask t = tasks[blockIdx.x];
  const int n = t.n, np = t.npiv;
  if (k0 >= np || *t.bad) return;
  const int kb = min(GJ_KB, np - k0);
  const int h = threadIdx.x % LPR;
  V* A = static_cast<V*>(t.a);
  const int64_t ld = t.ld;
  if ((int)blockIdx.y < row_pieces) {
    const int row0 = blockIdx.y * PIECE;
    if (row0 >= n) return;
    const int row = row0 + threadIdx.x / LPR;
    const bool act = row < n;
    const bool out = act && (row < k0 || row >= np);
    const bool any = __syncthreads_or(out);
    if (any) {
      const V* pg = static_cast<const V*>(t.prows);
      for (int e = threadIdx.x; e < kb * GJ_KB; e += NT) sm[e] = (e & (GJ_KB - 1)) < kb ? pg[e] : cx<V>(0.0, 0.0);
    } else if (sizeof(T) == 4) {
      return;
    }
    __syncthreads();
    V* Ar = A + row + (int64_t)k0 * ld;
    V a[Q];
#pragma unroll
    for (int i = 0; i < Q; ++i) a[i] = (act && LPR * i + h < kb) ? Ar[(int64_t)(LPR * i + h) * ld] : cx<V>(0.0, 0.0);
    if (any) {
      V b[Q];
#pragma unroll
      for (int i = 0; i < Q; ++i) b[i] = a[i];
      replay_row<LPR>(b, sm, kb, h);
      if (out)
#pragma unroll
        for (int i = 0; i < Q; ++i)
          if (LPR * i + h < kb) {
            a[i] = b[i];
            Ar[(int64_t)(LPR * i + h) * ld] = b[i];
          }
    }
    if constexpr (sizeof(T) == 8) {
      const uint32_t mask = oz::row_mask<LPR>(a, h);
      if (act && h == 0) t.ma[row] = mask;
      oz::write_a<LPR>(t.oa, t.ea, row, h, act, a);
    }
    return;
  }
  const int total = t.ncol - kb;
  const int c0 = ((int)blockIdx.y - row_pieces) * PIECE;
  if (c0 >= total) return;
  const int* perm = t.perm;
  const int nd = perm[3 * GJ_KB];
  const int r = c0 + threadIdx.x / LPR;
  const bool act = r < total;
  const int j = r < k0 ? r : r + kb;
  V* Aj = A + (int64_t)j * ld;
  V y[Q], dv[Q];
#pragma unroll
  for (int i = 0; i < Q; ++i) {
    const int c = LPR * i + h;
    y[i] = (act && c < kb) ? Aj[k0 + perm[c]] : cx<V>(0.0, 0.0);
    dv[i] = (act && c < nd) ? Aj[k0 + perm[2 * GJ_KB + c]] : cx<V>(0.0, 0.0);
  }
  __syncwarp();  // a displaced row's place may be another lane's source
#pragma unroll
  for (int i = 0; i < Q; ++i) {
    const int c = LPR * i + h;
    if (act && c < nd) Aj[k0 + perm[GJ_KB + c]] = dv[i];
  }
  if constexpr (sizeof(T) == 8) {
    const uint32_t mask = oz::row_mask<LPR>(y, h);
    if (act) {
      if (h == 0) t.mb[r] = mask;
#pragma unroll
      for (int i = 0; i < Q; ++i) static_cast<double2*>(t.y)[(int64_t)r * GJ_KB + LPR * i + h] = y[i];
    }
    oz::write_b<LPR>(t.ob, t.eb, r, h, act, y);
    return;
  }
  if (!act) return;
  V* Y = static_cast<V*>(t.y);
#pragma unroll
  for (int i = 0; i < Q; ++i) {
    const int c = LPR * i + h;
    if (c < kb) Y[c + (int64_t)j * kb] = y[i];
    if (sizeof(T) == 4 && t.bt) {
      unsigned char* tile = static_cast<unsigned char*>(t.bt) + (size_t)(r / TCU_COLS) * 2 * TCU_B_BYTES;
      const uint32_t off = tc::kmajor_offset(r % TCU_COLS, 2 * c, TCU_COLS);
      const float2 v = make_float2((float)y[i].x, (float)y[i].y);
      const float2 hi = make_float2(tc::to_tf32(v.x), tc::to_tf32(v.y));
      *reinterpret_cast<float2*>(tile + off) = hi;
      *reinterpret_cast<float2*>(tile + TCU_B_BYTES + off) =
          make_float2(tc::to_tf32(v.x - hi.x), tc::to_tf32(v.y - hi.y));
    }
  }
}

}  // namespace caroli
