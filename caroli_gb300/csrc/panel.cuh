// Panel sweeps of large fronts and roots spread over a cluster of CTAs, and the kernel that brings
// the rest of the matrix up to date with a panel.
//
// A 32-column panel is a chain of 32 pivot steps over its candidate rows. FP64 runs at about two
// multiply-adds per clock and SM here, so one CTA per matrix is bound by its own SM's FP64 pipe as
// soon as there are fewer matrices than SMs: the chain itself is short. Two kernels replace it:
//   panel_sweep_kernel  the candidate rows split over the CTAs of a cluster, a cluster barrier per
//                       pivot step; each CTA publishes its best candidate row, already scaled by the
//                       reciprocal of its pivot, into every CTA's shared memory, so a step costs one
//                       exchange and no CTA computes a reciprocal or a pivot search twice;
//   panel_rest_kernel   what is independent per row (the rows outside the candidates replay the
//                       steps) and per column (the pivot rows of the other columns), over as many
//                       CTAs as there are 16-row and 8-column pieces.
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
// up to 1 728, root 1 152) 337 -> 41 ms, of 16 BHZ 200 x 64 solves (fronts up to 384) 88 -> 26 ms, of one
// 32 x 32 square (fronts up to 94) 1.57 -> 0.66 ms.
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

// Candidate rows per CTA of a cluster of c for m candidates (a multiple of 16: a half warp's rows).
__host__ __device__ inline int panel_rows(int m, int c) { return ((m + c - 1) / c + 15) / 16 * 16; }
// Dynamic shared memory: the rows (r x kb), the column buffer (2 r), the published rows of every
// CTA (2 x c x kb), row k (2 x kb), keys and indices (2 x c).
__host__ __device__ inline size_t panel_sweep_bytes(int r, int c, size_t vbytes) {
  return ((size_t)r * GJ_KB + 2 * (size_t)r + 2 * (size_t)c * GJ_KB + 2 * GJ_KB) * vbytes + 2 * (size_t)c * 12 + 16;
}

// Orders squared moduli as unsigned integers; 0: no candidate (also NaN).
__device__ __forceinline__ unsigned long long norm_key(double m) {
  return m >= 0.0 ? (unsigned long long)__double_as_longlong(m) + 1ull : 0ull;
}
__device__ __forceinline__ unsigned long long norm_key(float m) {
  return m >= 0.f ? (unsigned long long)__float_as_uint(m) + 1ull : 0ull;
}
// Largest key of the warp and the smallest index holding it: three warp reductions on 32-bit words.
__device__ __forceinline__ void key_argmax(unsigned long long& key, int& idx) {
  const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
  const unsigned th = __reduce_max_sync(0xffffffffu, hi);
  const unsigned tl = __reduce_max_sync(0xffffffffu, hi == th ? lo : 0u);
  idx = __reduce_min_sync(0xffffffffu, (hi == th && lo == tl) ? idx : 0x7fffffff);
  key = ((unsigned long long)th << 32) | tl;
}
template <typename T> __device__ __forceinline__ double key_norm(unsigned long long key) {
  if constexpr (sizeof(T) == 8) return __longlong_as_double((long long)(key - 1ull));
  else return (double)__uint_as_float((unsigned)(key - 1ull));
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
  T mt = 0;
  for (int j = blockIdx.y * 8 + w; j < t.npiv; j += gridDim.y * 8)
    for (int i = lane; i < t.npiv; i += 32) mt = fmax(mt, cnorm(A[i + (int64_t)j * t.ld]));
  unsigned long long key = (unsigned long long)__double_as_longlong((double)mt);
  int idx = 0;
  key_argmax(key, idx);
  if (lane == 0 && key) atomicMax(reinterpret_cast<unsigned long long*>(t.scale2), key);
}

// grid: matrices x cluster (clusters along x), PS_THREADS threads. R: rows per CTA.
template <typename T>
__global__ void __launch_bounds__(PS_THREADS) panel_sweep_kernel(const InvTask* __restrict__ tasks, int k0, double tol,
                                                                 int perturb, int R, const JobDesc* __restrict__ jobs) {
  using V = typename Cx<T>::V;
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_piv[GJ_KB];
  __shared__ unsigned long long s_key;
  __shared__ int s_loc;
  __shared__ V s_inv;
  cg::cluster_group cluster = cg::this_cluster();
  const int C = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const InvTask t = tasks[blockIdx.x / C];
  const int np = t.npiv;
  if (k0 >= np || *t.bad) return;  // uniform in the cluster: *bad is only set after its first barrier
  const int kb = min(GJ_KB, np - k0), m = np - k0;
  const bool trail = t.trail != 0;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int l16 = lane & 15, half = lane >> 4;
  const int r0 = rank * R, rows = max(0, min(R, m - r0));
  V* F = reinterpret_cast<V*>(smem_raw);
  V* cb = F + (size_t)R * GJ_KB;            // 2 x R: column k of the own rows
  V* prow = cb + 2 * (size_t)R;             // 2 x C x kb: scaled candidate rows of every CTA
  V* krow = prow + 2 * (size_t)C * GJ_KB;   // 2 x kb: row k before step k
  unsigned long long* keys = reinterpret_cast<unsigned long long*>(krow + 2 * GJ_KB);  // 2 x C
  int* idxs = reinterpret_cast<int*>(keys + 2 * C);                                    // 2 x C: row, bit 30 refused
  V* A = static_cast<V*>(t.a) + k0 + (int64_t)k0 * t.ld;
  for (int j = w; j < kb; j += PS_THREADS / 32)
    for (int i = lane; i < rows; i += 32) {
      const V v = A[(r0 + i) + (int64_t)j * t.ld];
      F[i + (size_t)j * R] = v;
      if (j == 0) cb[i] = v;
    }
  __syncthreads();
  const double scale2 = *t.scale2;
  const double thresh = tol * tol * scale2;
  // The CTA's best candidate of column k among its rows at or past k: key, local row and the
  // reciprocal of the (possibly perturbed) pivot. One warp, the candidates' entries in `col`.
  auto search = [&](int k, const V* col) {
    unsigned long long key = 0;
    int loc = 0x7fffffff;
    for (int i = lane; i < rows; i += 32)
      if (r0 + i >= k) {
        const unsigned long long q = norm_key(cnorm(col[i]));
        if (q > key) { key = q; loc = i; }
      }
    key_argmax(key, loc);
    V inv = cx<V>(0.0, 0.0);
    int refused = 0;
    if (key) {
      V d = col[loc];
      const double big = key_norm<T>(key);
      if (!(big > thresh)) {
        if (perturb && scale2 > 0.0) {  // static pivoting (see gj_sweep)
          const double mag = sqrt(big), target = tol * sqrt(scale2);
          if (mag > 0.0) { d.x = (T)(d.x / mag * target); d.y = (T)(d.y / mag * target); }
          else { d.x = (T)target; d.y = (T)0; }
        } else {
          refused = 1 << 30;
        }
      }
      inv = cinv(d);
    }
    if (lane == 0) {
      s_key = key;
      s_loc = key ? (loc | refused) : 0;
      s_inv = inv;
    }
  };
  // Publishes the candidate found by `search` (warp 0) and row k if it is here (warp 1).
  auto publish = [&](int k) {
    const int par = k & 1;
    if (w == 0) {
      const unsigned long long key = s_key;
      const int loc = s_loc & ~(1 << 30), refused = s_loc & (1 << 30);
      V v = cx<V>(0.0, 0.0);
      if (key && lane < kb) {
        const V raw = F[loc + (size_t)lane * R];
        v = lane == k ? s_inv : ((trail && lane < k) ? raw : cmul(raw, s_inv));
      }
      for (int c = 0; c < C; ++c) {
        if (key && lane < kb) cluster.map_shared_rank(prow, c)[((size_t)par * C + rank) * GJ_KB + lane] = v;
        if (lane == 0) {
          cluster.map_shared_rank(keys, c)[par * C + rank] = key;
          cluster.map_shared_rank(idxs, c)[par * C + rank] = (r0 + loc) | refused;
        }
      }
    } else if (w == 1 && k >= r0 && k < r0 + rows) {
      if (lane < kb) {
        const V v = F[(k - r0) + (size_t)lane * R];
        for (int c = 0; c < C; ++c) cluster.map_shared_rank(krow, c)[par * GJ_KB + lane] = v;
      }
    }
    __syncwarp();
  };
  if (w == 0) search(0, cb);
  cluster_sync_all();  // every CTA of the cluster runs before its shared memory is written
  publish(0);
  for (int k = 0; k < kb; ++k) {
    cluster_sync_all();  // step k's candidates and row k are here; everyone has finished step k - 1
    const int par = k & 1;
    unsigned long long key = lane < C ? keys[par * C + lane] : 0ull;
    int p = lane < C && key ? idxs[par * C + lane] : 0x7fffffff;
    const unsigned long long mine = key;
    const int mp = p;
    p &= ~(1 << 30);
    key_argmax(key, p);
    const unsigned win = __ballot_sync(0xffffffffu, mine == key && key && (mp & ~(1 << 30)) == p);
    if (!win || (__shfl_sync(0xffffffffu, mp, __ffs(win) - 1) & (1 << 30))) {  // the same decision in every CTA
      if (rank == 0 && tid == 0) {
        *t.bad = 1;
        if (trail && t.front >= 0) jobs[t.job].fail[t.front] = 1;
      }
      return;
    }
    const V* pr = prow + ((size_t)par * C + (__ffs(win) - 1)) * GJ_KB;
    const V* kr = krow + par * GJ_KB;
    const V* ck = cb + (size_t)par * R;
    V* cn = cb + (size_t)(par ^ 1) * R;
    if (rank == 0) {
      if (tid == 0) s_piv[k] = p;
      if (w == 2 && lane < kb) static_cast<V*>(t.prows)[k * GJ_KB + lane] = pr[lane];
    }
    const V krk = kr[k];
    // A warp takes pairs of columns (a half warp each, 16 rows at a time), the pair of column k + 1
    // first: its warp then searches that column while the others go on.
    const int first = ((k + 1) >> 1) & 7;
    for (int u = 0; u < GJ_KB / 16; ++u) {
      const int q = w == first ? ((u == 0) == (((k + 1) >> 1) < 8) ? w : w + 8) : w + 8 * u;
      const int j = 2 * q + half;
      const bool live = j < kb;
      const bool moves = trail && j <= k;  // columns done: only the interchange reaches them
      if (!moves || 2 * q <= k) {
        const V prj = live ? pr[j] : cx<V>(0.0, 0.0), krj = live ? kr[j] : cx<V>(0.0, 0.0);
        V* Fj = F + (size_t)j * R;
        for (int il = l16; il < rows; il += 16) {
          const int i = r0 + il;
          if (!live) continue;
          if (i == k) {
            Fj[il] = prj;
            if (j == k + 1) cn[il] = prj;
            continue;
          }
          const bool sw = i == p;
          if (moves) {
            if (sw) Fj[il] = krj;
            continue;
          }
          if (trail && i < k) continue;
          const V c = sw ? krk : ck[il];
          V nv;
          if (j == k) nv = cmul(cx<V>(-c.x, -c.y), prj);
          else nv = cfms_pk(sw ? krj : Fj[il], c, prj);
          Fj[il] = nv;
          if (j == k + 1) cn[il] = nv;
        }
      }
      if (w == first && u == 0 && k + 1 < kb) {
        __syncwarp();
        search(k + 1, cn);
      }
    }
    __syncthreads();
    if (k + 1 < kb) publish(k + 1);
  }
  for (int j = w; j < kb; j += PS_THREADS / 32)
    for (int i = lane; i < rows; i += 32) A[(r0 + i) + (int64_t)j * t.ld] = F[i + (size_t)j * R];
  if (rank == 0 && w == 0) {
    // Where the row now at position x came from: the interchanges undone last first.
    auto origin = [&](int x) {
      for (int k = kb - 1; k >= 0; --k) {
        const int p = s_piv[k];
        x = x == k ? p : (x == p ? k : x);
      }
      return x;
    };
    int* perm = t.perm;
    if (lane < kb) {
      t.piv[k0 + lane] = k0 + s_piv[lane];
      perm[lane] = origin(lane);
    }
    // Positions at or past kb that hold another row now: each is some piv[k], listed once.
    const int p = lane < kb ? s_piv[lane] : -1;
    const int from = lane < kb && p >= kb ? origin(p) : p;
    const bool moved = lane < kb && p >= kb && from != p;
    const unsigned same = __match_any_sync(0xffffffffu, moved ? p : -1 - lane);
    const bool leader = moved && (__ffs(same) - 1 == lane);
    const unsigned bal = __ballot_sync(0xffffffffu, leader);
    if (leader) {
      const int at = __popc(bal & ((1u << lane) - 1u));
      perm[GJ_KB + at] = p;
      perm[2 * GJ_KB + at] = from;
    }
    if (lane == 0) perm[3 * GJ_KB] = __popc(bal);
  }
}

constexpr int PR_THREADS = 64, PR_ROWS = 16, PR_COLS = 8;

// After panel_sweep_kernel: grid (matrices, row pieces then column pieces), PR_THREADS threads.
// Row piece: four lanes per row, eight panel columns each; rows outside the candidates replay the
// recorded steps. With oa set (FP64), every row the update reads also becomes an operand row.
// Column piece: a warp per column; the pivot rows of a column outside the panel into Y (or B', or the
// FP64 operand), the displaced rows into place. In the trail form the column is first solved with L11
// (a lane per pivot row).
template <typename T>
__global__ void __launch_bounds__(PR_THREADS) panel_rest_kernel(const InvTask* __restrict__ tasks, int k0,
                                                                int row_pieces) {
  using V = typename Cx<T>::V;
  __shared__ V sm[GJ_KB * GJ_KB];
  const InvTask t = tasks[blockIdx.x];
  const int n = t.n, np = t.npiv;
  if (k0 >= np || *t.bad) return;
  const int kb = min(GJ_KB, np - k0);
  const bool trail = t.trail != 0;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  V* A = static_cast<V*>(t.a);
  const int64_t ld = t.ld;
  const int base = trail ? k0 + kb : 0;  // first row (and, for trail, column) of the update
  if ((int)blockIdx.y < row_pieces) {
    const int total = n - base;
    const int q0 = blockIdx.y * PR_ROWS;
    if (q0 >= total) return;
    const int q = q0 + (threadIdx.x >> 2), h = threadIdx.x & 3;
    const int row = base + q;
    const bool act = q < total;
    const bool out = act && (row < k0 || row >= np);
    if (__syncthreads_or(out)) {
      const V* pg = static_cast<const V*>(t.prows);
      for (int e = threadIdx.x; e < kb * GJ_KB; e += PR_THREADS) sm[e] = pg[e];
    } else if (sizeof(T) == 4) {
      return;
    }
    __syncthreads();
    V* Ar = A + row + (int64_t)(k0 + 8 * h) * ld;
    V a[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) a[c] = (act && 8 * h + c < kb) ? Ar[(int64_t)c * ld] : cx<V>(0.0, 0.0);
    if (__any_sync(0xffffffffu, out)) {
      V b[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) b[c] = a[c];
#pragma unroll
      for (int k = 0; k < GJ_KB; ++k) {
        if (k >= kb) break;
        const V* pk = sm + k * GJ_KB + 8 * h;
        const int src = (lane & ~3) | (k >> 3);
        const V own = b[k & 7];
        const V ak = cx<V>(__shfl_sync(0xffffffffu, own.x, src), __shfl_sync(0xffffffffu, own.y, src));
        const int rel = k - 8 * h;  // the step's column among this lane's
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          if (trail && c <= rel) continue;
          if (c == rel) b[c] = cmul(cx<V>(-ak.x, -ak.y), pk[c]);
          else b[c] = cfms_pk(b[c], ak, pk[c]);
        }
      }
      if (out)
#pragma unroll
        for (int c = 0; c < 8; ++c)
          if (8 * h + c < kb) {
            a[c] = b[c];
            Ar[(int64_t)c * ld] = b[c];
          }
    }
    if constexpr (sizeof(T) == 8) {
      if (t.oa) oz::write_a(t.oa, t.ea, q, h, act, a);
    }
    return;
  }
  const int total = (trail ? n : t.ncol) - (trail ? base : kb);
  const int c0 = ((int)blockIdx.y - row_pieces) * PR_COLS;
  if (c0 >= total) return;
  const int* perm = t.perm;
  const int nd = perm[3 * GJ_KB];
  if (trail) {
    // L11 with each column scaled by its pivot's reciprocal (the column steps then use the raw
    // pivot-row entries), the reciprocals on the diagonal.
    for (int e = threadIdx.x; e < kb * GJ_KB; e += PR_THREADS) {
      const int c = e & (GJ_KB - 1), k = e / GJ_KB;
      V v = cx<V>(0.0, 0.0);
      if (c < kb && c >= k) {
        v = A[(k0 + c) + (int64_t)(k0 + k) * ld];
        if (c > k) v = cmul(v, A[(k0 + k) + (int64_t)(k0 + k) * ld]);
      }
      sm[e] = v;
    }
    __syncthreads();
  }
  const int src = k0 + (lane < kb ? perm[lane] : 0);
  const int dto = k0 + (lane < nd ? perm[GJ_KB + lane] : 0), dfrom = k0 + (lane < nd ? perm[2 * GJ_KB + lane] : 0);
  V* Y = static_cast<V*>(t.y);
#pragma unroll 2
  for (int u = 0; u < PR_COLS / 2; ++u) {
    const int r = c0 + w + 2 * u;
    if (r >= total) continue;
    const int j = trail ? base + r : (r < k0 ? r : r + kb);
    V* Aj = A + (int64_t)j * ld;
    V y = cx<V>(0.0, 0.0), dv = cx<V>(0.0, 0.0);
    if (lane < kb) y = Aj[src];
    if (lane < nd) dv = Aj[dfrom];
    __syncwarp();
    if (lane < nd) Aj[dto] = dv;
    if (trail) {
      for (int k = 0; k < kb - 1; ++k) {
        const V yk = cx<V>(__shfl_sync(0xffffffffu, y.x, k), __shfl_sync(0xffffffffu, y.y, k));
        if (lane > k) y = cfms(y, sm[lane + k * GJ_KB], yk);
      }
      if (lane < kb) y = cmul(y, sm[lane + lane * GJ_KB]);
    }
    if constexpr (sizeof(T) == 8) {
      if (t.ob) {
        oz::write_b(t.ob, t.eb, r, lane, y);
        continue;
      }
    }
    if (lane < kb) Y[lane + (int64_t)j * kb] = y;
    if (sizeof(T) == 4 && t.bt) {
      unsigned char* tile = static_cast<unsigned char*>(t.bt) + (size_t)(r / TCU_COLS) * 2 * TCU_B_BYTES;
      const uint32_t off = tc::kmajor_offset(r % TCU_COLS, 2 * lane, TCU_COLS);
      const float2 v = make_float2((float)y.x, (float)y.y);
      const float2 hi = make_float2(tc::to_tf32(v.x), tc::to_tf32(v.y));
      *reinterpret_cast<float2*>(tile + off) = hi;
      *reinterpret_cast<float2*>(tile + TCU_B_BYTES + off) =
          make_float2(tc::to_tf32(v.x - hi.x), tc::to_tf32(v.y - hi.y));
    }
  }
}

}  // namespace caroli
