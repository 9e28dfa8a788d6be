// Complex FP64 GEMMs on the tcgen05 tensor cores, from digit products as the rank-32 updates of
// ozaki.cuh: C = (C +) sign A B. Operands are first written as digits (oz_pack_kernel), 32 entries of the
// inner dimension at a time, each 32 with its own power-of-two scale per row of A and column of B; the
// chunks' products, rounded each, are summed in FP64 registers.
//
// They carry the dense FP64 products of the framework: the slices' Σ and Γ against the refinement's
// right-hand sides, the Caroli traces Tr[Γ_p G_pq Γ_q G_pq^†], and the lead self-energies Y diag(λ) Y^†.
// On the FP64 pipe (1.7 multiply-adds per clock and SM) these were 14 of 42 ms of two 48 x 24 x 24 cubic
// wires, 4.9 of 16 ms of a four-terminal square cross, 7.8 of 23 ms of a refined BHZ cross.
#pragma once
#include "ozaki.cuh"
#include "refine.cuh"

namespace caroli {
namespace oz {

// One operand to write as digits. Element (r, k) of the operand is p[(r0 + rmap(r)) + (k0 + kmap(k)) ld], or
// with `trans` p[(k0 + kmap(k)) + (r0 + rmap(r)) ld], conjugated with `conj`, times kscale[k]. A row of A is
// a row r; a column of B is written as "row" r with the inner dimension as k.
struct PackTask {
  const void* p;
  int64_t ld;
  const int32_t *rmap, *kmap;  // null: the index itself
  const double2* kscale;       // null: 1
  unsigned char* dig;
  int32_t* exp;                // chunk-major: exp[chunk * rows + r]
  const RefineDesc* rd;        // a refinement vector instead of p: see `src`
  int32_t r0, k0, rows, k;
  int32_t trans, conj, b;      // b: written as B'
  int32_t src;                 // 0: p; 1: Z_step (f32; skipped once the inner solve is done); 2: x
};

struct GemmTask {
  const unsigned char *a, *b;
  const int32_t *ea, *eb;
  double2* c;
  int64_t ldc;
  const int32_t* crow;  // row i goes to row crow[i] of C (null: i)
  const RefineDesc* rd; // a refinement vector instead of c: see `dst`
  const PackTask *pa, *pb;  // outputs far below the largest entries' product: again from these (null: as they are)
  int32_t* status;      // set to ST_TIMEOUT by a wait that runs out (null: the solve of rd is marked late)
  int32_t m, n, chunks;
  int32_t dst;          // 0: c; 1: V_{step + 1} (accumulated); 2: r (accumulated); 3: gx
  int32_t far;          // how many bits far below (with pa)
  double sign;
};

__host__ __device__ inline int chunks_of(int k) { return (k + GJ_KB - 1) / GJ_KB; }
__host__ __device__ inline size_t pack_a_bytes(int m, int k) {
  return (size_t)((m + ROWS - 1) / ROWS) * chunks_of(k) * A_TILE;
}
__host__ __device__ inline size_t pack_b_bytes(int n, int k) {
  return (size_t)((n + COLS - 1) / COLS) * chunks_of(k) * B_TILE;
}
__host__ __device__ inline size_t pack_e_bytes(int rows, int k) { return ((size_t)rows * chunks_of(k) * 4 + 255) / 256 * 256; }

__device__ __forceinline__ bool pack_idle(const RefineDesc* rd, bool inner) {
  return rd && (rd->done || (inner && rd->inner_done));
}

// Entry k of row r of an operand.
__device__ __forceinline__ double2 pack_entry(const PackTask& t, int r, int k, int step) {
  const int64_t row = t.r0 + (t.rmap ? t.rmap[r] : r), kk = t.k0 + (t.kmap ? t.kmap[k] : k);
  const int64_t at = t.trans ? kk + row * t.ld : row + kk * t.ld;
  double2 v;
  if (t.src == 1) {
    const float2 f = t.rd->Z[(int64_t)step * t.rd->nblk * t.rd->c + at];
    v = make_double2((double)f.x, (double)f.y);
  } else {
    v = t.src == 2 ? t.rd->x[at] : static_cast<const double2*>(t.p)[at];
  }
  if (t.conj) v.y = -v.y;
  return t.kscale ? cmul(v, t.kscale[k]) : v;
}

// Four lanes per (row, chunk). grid (pieces of 64 (row, chunk) pairs, tasks); with a job list, task
// jl[y / per] * per + y % per (`per` tasks per job).
__global__ void __launch_bounds__(256) pack_kernel(const PackTask* __restrict__ tasks, const int32_t* __restrict__ jl, int per,
                                                   int step) {
  const PackTask t = tasks[jl ? jl[blockIdx.y / per] * per + blockIdx.y % per : blockIdx.y];
  if (pack_idle(t.rd, t.src == 1)) return;
  const int nch = chunks_of(t.k);
  const int64_t pair = (int64_t)blockIdx.x * 64 + (threadIdx.x >> 2);
  if ((int64_t)blockIdx.x * 64 >= (int64_t)t.rows * nch) return;
  const int h = threadIdx.x & 3;
  const bool act = pair < (int64_t)t.rows * nch;
  const int r = act ? (int)(pair % t.rows) : 0, ch = act ? (int)(pair / t.rows) : 0;
  double2 a[GJ_KB / 4];
#pragma unroll
  for (int i = 0; i < GJ_KB / 4; ++i) {
    const int k = ch * GJ_KB + 4 * i + h;
    a[i] = act && k < t.k ? pack_entry(t, r, k, step) : make_double2(0.0, 0.0);
  }
  if (t.b) write_b<4>(t.dig + (size_t)ch * B_TILE, t.exp + (size_t)ch * t.rows, r, h, act, a, (size_t)nch * B_TILE);
  else write_a<4>(t.dig + (size_t)ch * A_TILE, t.exp + (size_t)ch * t.rows, r, h, act, a, (size_t)nch * A_TILE);
}

// A CTA computes a 128 x 16 complex tile of one task: per chunk, one thread copies the digits of A (single
// buffer: 112 KB) and B (two), one issues 28 MMAs into one of two accumulator sets, sixteen warps add the
// other set's chunk to FP64 sums in registers, while the next chunk's digits arrive. Waits are bounded.
// grid (row tiles, column tiles, tasks), tasks as pack_kernel; `side` >= 0: only task `side` of every job.
constexpr int GEMM_STAGES = 2;
constexpr int GEMM_SMEM = A_TILE + GEMM_STAGES * B_TILE + 1024;

__global__ void __launch_bounds__(THREADS, 1) gemm_kernel(const GemmTask* __restrict__ tasks, const int32_t* __restrict__ jl,
                                                          int per, int step, int side, uint32_t wait_limit) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint32_t tslot;
  __shared__ __align__(8) uint64_t afull, aempty, bfull[GEMM_STAGES], bempty[GEMM_STAGES], tfull[2], tempty[2];
  __shared__ int abort_flag;
  const GemmTask t = tasks[!jl ? blockIdx.z : side < 0 ? jl[blockIdx.z / per] * per + blockIdx.z % per : jl[blockIdx.z] * per + side];
  const int i0 = blockIdx.x * ROWS, j0 = blockIdx.y * COLS;
  if (i0 >= t.m || j0 >= t.n || pack_idle(t.rd, t.dst == 1)) return;
  const int nch = t.chunks;
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  unsigned char* sa = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* sb = sa + A_TILE;
  if (w == 0) tc::tmem_alloc(&tslot, 2 * ACC);
  if (tid == 0) {
    tc::mbar_init(&afull, 1);
    tc::mbar_init(&aempty, 1);
    for (int i = 0; i < GEMM_STAGES; ++i) {
      tc::mbar_init(&bfull[i], 1);
      tc::mbar_init(&bempty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&tfull[i], 1);
      tc::mbar_init(&tempty[i], EPI_WARPS);
    }
    abort_flag = 0;
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tbase = tslot;
  volatile int* abort_v = &abort_flag;
  auto fail = [&]() {
    *abort_v = 1;
    if (t.status) *t.status = ST_TIMEOUT;
    else if (t.rd) const_cast<RefineDesc*>(t.rd)->late = 1;
  };
  int copies = 0, mmas = 0;
  if (w == 0) {
    if (lane == 0) {
      const unsigned char* ga = t.a + (size_t)blockIdx.x * nch * A_TILE;
      const unsigned char* gb = t.b + (size_t)blockIdx.y * nch * B_TILE;
      for (int ch = 0; ch < nch && !*abort_v; ++ch) {
        const int st = ch % GEMM_STAGES;
        if (ch >= GEMM_STAGES && !tc::mbar_wait(&bempty[st], (uint32_t)((ch / GEMM_STAGES - 1) & 1), wait_limit)) { fail(); break; }
        if (ch >= 1 && !tc::mbar_wait(&aempty, (uint32_t)((ch - 1) & 1), wait_limit)) { fail(); break; }
        tc::mbar_arrive_expect_tx(&bfull[st], B_TILE);
        tc::bulk_copy_g2s(sb + st * B_TILE, gb + (size_t)ch * B_TILE, B_TILE, &bfull[st]);
        tc::mbar_arrive_expect_tx(&afull, A_TILE);
        for (int s = 0; s < S; ++s)
          tc::bulk_copy_g2s(sa + s * A_SLICE, ga + (size_t)ch * A_TILE + s * A_SLICE, A_SLICE, &afull);
        ++copies;
      }
    }
  } else if (w == 1) {
    if (lane == 0) {
      for (int ch = 0; ch < nch && !*abort_v; ++ch) {
        const int st = ch % GEMM_STAGES, a = ch & 1;
        if (!tc::mbar_wait(&bfull[st], (uint32_t)((ch / GEMM_STAGES) & 1), wait_limit)) { fail(); break; }
        if (!tc::mbar_wait(&afull, (uint32_t)(ch & 1), wait_limit)) { fail(); break; }
        if (ch >= 2 && !tc::mbar_wait(&tempty[a], (uint32_t)(((ch >> 1) - 1) & 1), wait_limit)) { fail(); break; }
        tc::fence_after_sync();
        mma_tile(tbase + (uint32_t)(a * ACC), sa, sb + st * B_TILE);
        tc::mma_commit(&aempty);
        tc::mma_commit(&bempty[st]);
        tc::mma_commit(&tfull[a]);
        ++mmas;
      }
    }
  } else {
    const int q = w & 3, part = (w - 2) >> 2;
    const int r = i0 + 32 * q + lane, c0 = j0 + part * 4;
    const bool row_in = r < t.m;
    double2 sum[4];
    int top[4];  // largest exponent of a product of the chunks' largest entries
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      sum[j] = make_double2(0.0, 0.0);
      top[j] = 0;
    }
    bool ok = true;
    for (int ch = 0; ch < nch; ++ch) {
      const int a = ch & 1;
      const int er = row_in ? t.ea[(size_t)ch * t.m + r] : 1;
      int ec[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) ec[j] = c0 + j < t.n ? er + t.eb[(size_t)ch * t.n + c0 + j] : 2;
      ok = !*abort_v && tc::mbar_wait(&tfull[a], (uint32_t)((ch >> 1) & 1), wait_limit);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) {
        if (lane == 0) fail();
        break;
      }
      tc::fence_after_sync();
      float v[S][8];
#pragma unroll
      for (int l = 0; l < S; ++l)
        tmem_ld8(tbase + ((uint32_t)(32 * q) << 16) + (uint32_t)(a * ACC + l * 2 * COLS + part * 8), v[l]);
      tc::tmem_ld_wait();
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&tempty[a]);
      if (c0 >= t.n) continue;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float x[S], y[S];
#pragma unroll
        for (int l = 0; l < S; ++l) {
          x[l] = v[l][2 * j];
          y[l] = v[l][2 * j + 1];
        }
        sum[j].x += combine(x, ec[j]);
        sum[j].y += combine(y, ec[j]);
        top[j] = max(top[j], ec[j]);
      }
    }
    if (ok && row_in) {
      double2* C = t.c;
      int64_t ldc = t.ldc;
      const bool add = t.dst == 1 || t.dst == 2;
      if (t.dst == 1) { C = t.rd->V + (int64_t)(step + 1) * t.rd->nblk * t.rd->c; ldc = t.rd->nblk; }
      else if (t.dst == 2) { C = t.rd->r; ldc = t.rd->nblk; }
      else if (t.dst == 3) { C = t.rd->gx; ldc = t.rd->nl; }
      C += (t.crow ? t.crow[r] : r) + (int64_t)c0 * ldc;
      if (t.pa) {  // see far_below
        uint32_t far = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (c0 + j < t.n && far_below(top[j], 1u, sum[j], add ? C[j * ldc] : sum[j], t.far)) far |= 1u << j;
        if (far) {
          const PackTask pa = *t.pa, pb = *t.pb;
#pragma unroll 1
          for (int j = 0; j < 4; ++j) {
            if (!(far >> j & 1u)) continue;
            double2 s = make_double2(0.0, 0.0);
            for (int ch = 0; ch < nch; ++ch) {
              if (t.ea[(size_t)ch * t.m + r] <= 1 || t.eb[(size_t)ch * t.n + c0 + j] <= 1) continue;  // zeros
#pragma unroll 4
              for (int k = ch * GJ_KB; k < min(pa.k, (ch + 1) * GJ_KB); ++k)
                s = cfma(s, pack_entry(pa, r, k, step), pack_entry(pb, c0 + j, k, step));
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (i == j) sum[i] = s;
          }
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (c0 + j >= t.n) break;
        double2& o = C[j * ldc];
        const double2 v = make_double2(t.sign * sum[j].x, t.sign * sum[j].y);
        o = add ? make_double2(o.x + v.x, o.y + v.y) : v;
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (abort_flag) {  // a wait ran out: drain (see tc_update_kernel)
    if (w == 0 && lane == 0 && copies > 0) {
      for (int ch = max(0, copies - GEMM_STAGES); ch < copies; ++ch)
        tc::mbar_wait(&bfull[ch % GEMM_STAGES], (uint32_t)((ch / GEMM_STAGES) & 1), TCU_WAIT);
      tc::mbar_wait(&afull, (uint32_t)((copies - 1) & 1), TCU_WAIT);
    }
    if (w == 1 && lane == 0 && mmas > 0) tc::mbar_wait(&aempty, (uint32_t)((mmas - 1) & 1), TCU_WAIT);
    tc::fence_before_sync();
    __syncthreads();
  }
  if (w == 0) tc::tmem_dealloc(tbase, 2 * ACC);
}

// Σ_ij Re(X_ij conj(Y_ij)) of dense m x n blocks, added to the task's DOT_PARTS partial sums. grid (tasks, DOT_PARTS).
struct DotTask {
  const double2 *x, *y;
  int64_t count;
  double* part;
};
constexpr int DOT_PARTS = 16;
__global__ void __launch_bounds__(256) dot_kernel(const DotTask* __restrict__ tasks) {
  __shared__ double red[32];
  const DotTask t = tasks[blockIdx.x];
  double s = 0.0;
  for (int64_t e = blockIdx.y * (int64_t)blockDim.x + threadIdx.x; e < t.count; e += (int64_t)gridDim.y * blockDim.x) {
    const double2 a = t.x[e], b = t.y[e];
    s += a.x * b.x + a.y * b.y;
  }
  s = block_sum(s, red);
  if (threadIdx.x == 0) t.part[blockIdx.y] += s;
}

}  // namespace oz
}  // namespace caroli
