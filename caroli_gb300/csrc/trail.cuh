// What follows a panel's sweep in the trailing form: the rows below the candidates are solved with the
// panel's U11 (L21 = A21 U11^-1), the pivot rows of the later columns with L11 (U12 = L11^-1 A12), both by
// replaying the panel's steps on a vector of 32 entries, and the results become the operands of
// oz::update_kernel.
//
// The replay is a triangular recursion of 496 complex multiply-adds per vector, bound by the FP64 pipe (two
// multiply-adds per clock and SM: 127 000 clocks for 128 vectors). Here only its four diagonal blocks of
// 8 x 8 stay there (112 multiply-adds); the blocks between them, 8 -> 8 columns twice and 16 -> 16 once, are
// products of 128 vectors with a small matrix, taken as digit products on the tensor cores (ozaki.cuh:
// same digits, levels, rounding and entries computed again). Blocks of 16 would leave 240 multiply-adds,
// blocks of 4 would leave 48 but need seven products, with 48 outputs per vector to put together in place of
// 32, and their eight operand columns are half of an MMA's K.
//
// Digits are cut relative to the largest entry of a row of L and of a column of U, and the pivot rows are scaled
// by the pivots' reciprocals: behind a small pivot p, row k of U (of size 1 / p) would take its place in the
// digits of every column, also for rows of L that are zero in column k. So the digits are taken of L D^-1 and
// D U, D_kk the power of two next to |p_k|^(1/2): the same product, and neither side exceeds its other
// entries by more than p^(-1/2). (U11 likewise; L11's columns are at most 1 against their pivots.)
//
// Measured against the whole replay on the FP64 pipe: 3 584 fronts of 16 BHZ 200 x 64 solves (first panel)
// 1.47 -> 0.83 ms, all panels of these solves 9.0 -> 5.5 ms; the panels (with their sweeps) of two
// 48 x 24 x 24 cubic wires 11.1 -> 10.6 ms (0.78, 5.3 and 9.9 before oz::far_below had entries kept and computed
// again). The FP64 pipe is then busy half of the time, one or two warps per scheduler being all that 32 FP64
// entries per thread leave room for.
#pragma once
#include "ozaki.cuh"

namespace caroli {
namespace trail {

constexpr int B = 8;                            // columns of a diagonal block
constexpr int A_BYTES = oz::S * 128 * 32 * 2;   // digits of 128 vectors x 16 complex entries
constexpr int B8_BYTES = oz::S * 16 * 16 * 2;   // digits of 8 complex columns x 8 entries
constexpr int B16_BYTES = oz::S * 32 * 32 * 2;  // digits of 16 complex columns x 16 entries
constexpr int SIDE = A_BYTES + 2 * B8_BYTES + B16_BYTES + GJ_KB * GJ_KB * 16;  // shared memory of the rows or the columns
constexpr int COARSE_SMEM = 2 * SIDE + 128, FINE_SMEM = SIDE + 128;

// Biased exponent of an entry times 2^shift.
constexpr int LEAST = -4096;
__device__ __forceinline__ int exponent(double2 v, int shift) {
  const int e = max(1, max(oz::biased_exponent(v.x), oz::biased_exponent(v.y)));
  return e == 0x7ff ? 2 * oz::NOT_FINITE : e + shift;
}

// Column r of the digits of a W x W block T[c0 .. c0 + W)[c0 + W ..) (row stride GJ_KB), W / 8 entries per
// lane of eight, entry k times 2^(mul half[k]); returns the column's exponent, and in `mask` its nonzero entries.
template <int W>
__device__ __forceinline__ int put_block(unsigned char* dst, const double2* T, int c0, int r, int h, const int* half, int mul,
                                         uint32_t& mask) {
  double2 y[W / 8];
  int e = LEAST;
  mask = 0;
#pragma unroll
  for (int i = 0; i < W / 8; ++i) {
    y[i] = T[(c0 + 8 * i + h) * GJ_KB + c0 + W + r];
    e = max(e, exponent(y[i], mul * half[c0 + 8 * i + h]));
    mask |= (oz::is_zero(y[i]) ? 0u : 1u) << (8 * i + h);
  }
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) {
    e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
    mask |= __shfl_xor_sync(0xffffffffu, mask, o);
  }
#pragma unroll
  for (int i = 0; i < W / 8; ++i) {
    uint32_t d[oz::S];
    oz::digit_pairs(y[i], e - mul * half[c0 + 8 * i + h], d);
    const int k = 2 * (8 * i + h);
#pragma unroll
    for (int s = 0; s < oz::S; ++s) {
      *reinterpret_cast<uint32_t*>(dst + oz::offset(2 * W * s + 2 * r, k, oz::S * 2 * W)) = d[s] ^ 0x80000000u;
      *reinterpret_cast<uint32_t*>(dst + oz::offset(2 * W * s + 2 * r + 1, k, oz::S * 2 * W)) = __funnelshift_l(d[s], d[s], 16);
    }
  }
  return e;
}

// Steps 8 b .. 8 b + 7 replayed on the columns up to 8 b + 7; returns the largest exponent
// of those columns (times 2^(mul half[k])).
template <int LPR, int b>
__device__ __forceinline__ int replay_block(double2 (&v)[GJ_KB / LPR], const double2* T, int h, bool any, const int* half, int mul) {
  constexpr int C0 = B * b;
  const int lane = threadIdx.x & 31;
  if (any) {
#pragma unroll
    for (int k = C0; k < C0 + B; ++k) {
      double2 ak = v[k / LPR];
      if (LPR > 1) {
        const int src = (lane & ~(LPR - 1)) | (k % LPR);
        ak = make_double2(__shfl_sync(0xffffffffu, ak.x, src), __shfl_sync(0xffffffffu, ak.y, src));
        if (h > k % LPR) v[k / LPR] = cfms(v[k / LPR], ak, T[k * GJ_KB + k / LPR * LPR + h]);
      }
#pragma unroll
      for (int i = k / LPR + 1; i < (C0 + B) / LPR; ++i) v[i] = cfms(v[i], ak, T[k * GJ_KB + LPR * i + h]);
    }
  }
  int e = LEAST;
#pragma unroll
  for (int i = C0 / LPR; i < (C0 + B) / LPR; ++i) e = max(e, exponent(v[i], mul * half[LPR * i + h]));
#pragma unroll
  for (int o = 1; o < LPR; o <<= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
  return e;
}

// grid (matrices, tiles of 128 vectors), 256 threads: threads 0-127 the rows, the others the columns of a tile, a
// vector per thread (LPR = 1, for many matrices); or grid (matrices, pieces of 32 vectors, rows | columns),
// 128 threads, four lanes per vector (LPR = 4), which leaves each SM a quarter of the chain. The same
// operations in the same order on every entry: the results do not depend on the choice.
// A warp's vectors are the tensor-memory lanes it can read. The rows fill a tile from its first warp and the
// columns from its last, so that the schedulers share a tile of few vectors. The rows and
// the columns synchronise apart (named barriers); 255 registers: 16 complex products of eight digit sums
// are put together beside the 32 entries.
template <int LPR>
__global__ void __launch_bounds__(LPR == 1 ? 256 : 128, LPR == 1 ? 1 : 2)
rest_kernel(const InvTask* __restrict__ tasks, int k0, int32_t* __restrict__ status, uint32_t wait_limit) {
  constexpr int Q = GJ_KB / LPR, VECS = 128 / LPR;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint32_t tslot;
  __shared__ __align__(8) uint64_t done[2];
  __shared__ int s_eb[2][GJ_KB];
  __shared__ uint32_t s_mb[2][GJ_KB];
  __shared__ __align__(16) int s_half[GJ_KB];
  const InvTask t = tasks[blockIdx.x];
  const int n = t.n, np = t.npiv;
  if (k0 >= np || *t.bad) return;
  const int kb = min(GJ_KB, np - k0), base = k0 + kb, total = n - base;
  const int first = blockIdx.y * VECS, cnt = min(VECS, total - first);
  if (cnt <= 0) return;
  const int slot = LPR == 1 ? (int)(threadIdx.x >> 7) : 0;
  const bool columns = LPR == 1 ? slot == 1 : blockIdx.z == 1;
  const int tid = threadIdx.x & 127, w = tid >> 5, lane = tid & 31, h = lane & (LPR - 1);
  const int m = LPR == 1 ? tid : 32 * w + (lane >> 2);  // row of A' and tensor-memory lane
  const int x = LPR == 1 ? tid - (columns ? 32 * (4 - (cnt + 31) / 32) : 0) : 8 * w + (lane >> 2);
  const bool act = x >= 0 && x < cnt;
  const int q = first + x;                                  // row or column of the update
  const bool solve = columns || base + first + cnt > np;    // the candidates are solved already
  const bool out = act && (columns || base + q >= np);
  unsigned char* sa = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 127) & ~(uintptr_t)127) + slot * SIDE;
  unsigned char* sb8 = sa + A_BYTES;
  unsigned char* sb16 = sb8 + 2 * B8_BYTES;
  double2* T = reinterpret_cast<double2*>(sb16 + B16_BYTES);
  double2* A = static_cast<double2*>(t.a);
  const int64_t ld = t.ld;
  auto side_sync = [&]() { asm volatile("bar.sync %0, 128;" ::"r"(1 + slot) : "memory"); };

  double2 v[Q];
  double2* Ar = A + base + q + (int64_t)k0 * ld;  // row q of the panel
  double2* Ac = A + (int64_t)(base + q) * ld + k0;
  if (columns) {
    const int* perm = t.perm;
#pragma unroll
    for (int i = 0; i < Q; ++i) {
      const int c = LPR * i + h;
      v[i] = act && c < kb ? Ac[perm[c]] : make_double2(0.0, 0.0);
    }
  } else {
#pragma unroll
    for (int i = 0; i < Q; ++i) {
      const int c = LPR * i + h;
      v[i] = act && c < kb ? Ar[(int64_t)c * ld] : make_double2(0.0, 0.0);
    }
  }
  if (threadIdx.x < 32) tc::tmem_alloc(&tslot, LPR == 1 ? 512 : 256);
  if (threadIdx.x == 0) {
    tc::mbar_init(&done[0], 1);
    tc::mbar_init(&done[1], 1);
  }
  if (threadIdx.x < GJ_KB) {  // half of the pivot's exponent
    const double2 inv = static_cast<const double2*>(t.prows)[threadIdx.x * (GJ_KB + 1)];
    s_half[threadIdx.x] = (int)threadIdx.x < kb ? (1023 - exponent(inv, 0)) >> 1 : 0;
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tacc = tslot + (uint32_t)(slot * 256);

  // Entry k of a row times 2^-half[k], row k of U11 and entry k of a column times 2^half[k]: see above.
  const int inner = columns ? 0 : -1;
  bool late = false;
  uint32_t phase = 0, issued = 0;
  constexpr int NE = 4 / LPR;  // entries per lane of a group of four columns
  constexpr int UNROLL = LPR == 1 ? 1 : 4;
  // A group's entries, or a change to them: a uniform jump in place of eight copies of the code around it. (Fully
  // unrolled, 190 KB of instructions run once each: the warps waited for instructions 40 % of the time.)
  auto fetch = [&](int g, double2 (&o)[NE]) {
    switch (g) {
#define CAROLI_GROUP(G) \
  case G: \
    _Pragma("unroll") for (int i = 0; i < NE; ++i) o[i] = v[NE * G + i]; \
    break;
      CAROLI_GROUP(0) CAROLI_GROUP(1) CAROLI_GROUP(2) CAROLI_GROUP(3)
      CAROLI_GROUP(4) CAROLI_GROUP(5) CAROLI_GROUP(6) CAROLI_GROUP(7)
#undef CAROLI_GROUP
    }
  };
  auto subtract = [&](int g, const double2 (&o)[NE]) {
    switch (g) {
#define CAROLI_GROUP(G) \
  case G: \
    _Pragma("unroll") for (int i = 0; i < NE; ++i) { \
      v[NE * G + i].x -= o[i].x; \
      v[NE * G + i].y -= o[i].y; \
    } \
    break;
      CAROLI_GROUP(2) CAROLI_GROUP(3) CAROLI_GROUP(4) CAROLI_GROUP(5) CAROLI_GROUP(6) CAROLI_GROUP(7)
#undef CAROLI_GROUP
    }
  };
  // Digits of the groups g0 .. g0 + ng - 1 as row `row` of an operand: digit s at dst + s slice, 16 bytes (four entries)
  // per store where a thread holds them.
  auto put = [&](unsigned char* dst, uint32_t slice, int row, int rows, int g0, int ng, int e, int mul) {
    uint32_t mask = 0;  // the vector's nonzero entries
#pragma unroll UNROLL
    for (int g = 0; g < ng; ++g) {
      double2 o[NE];
      fetch(g0 + g, o);
      uint32_t d[NE][oz::S];
#pragma unroll
      for (int i = 0; i < NE; ++i) {
        oz::digit_pairs(o[i], e - mul * s_half[4 * (g0 + g) + LPR * i + h], d[i]);
        mask |= (oz::is_zero(o[i]) ? 0u : 1u) << (4 * g + LPR * i + h);
      }
      unsigned char* at = dst + oz::offset(row, 8 * g + 2 * h, rows);
#pragma unroll
      for (int s = 0; s < oz::S; ++s) {
        if constexpr (LPR == 1) *reinterpret_cast<uint4*>(at + s * slice) = make_uint4(d[0][s], d[1][s], d[2][s], d[3][s]);
        else *reinterpret_cast<uint32_t*>(at + s * slice) = d[0][s];
      }
    }
    return mask;
  };
  // v[c0 + W .. c0 + 2 W) -= v[c0 .. c0 + W) x the block `sb`: digits of the own entries (largest exponent e) into
  // A', the MMAs of a digit of A' with all digits of B' it still meets (level sums of 2 W columns), the sums put
  // together.
  auto product = [&](int c0, int W, const unsigned char* sb, const int* eb, const uint32_t* mb, int e) {
    uint32_t mask = put(sa, 128 * 4 * W, m, 128, c0 / 4, W / 4, e, inner);
    tc::fence_smem_async();
    tc::fence_before_sync();
    side_sync();
    if (tid == 0 && !late) {
      tc::fence_after_sync();
      const uint32_t pa = tc::smem_addr(sa), pb = tc::smem_addr(sb);
#pragma unroll
      for (int i = 0; i < oz::S; ++i)
        for (int ks = 0; ks < W / 8; ++ks)
          oz::mma_f16(tacc + (uint32_t)(i * 2 * W), tc::smem_desc(pa + i * 128 * 4 * W + ks * 128 * 32, 128, 256),
                      tc::smem_desc(pb + ks * oz::S * 2 * W * 32, 128, 256), oz::idesc_f16(128, 2 * W * (oz::S - i)),
                      i > 0 || ks > 0);
      tc::mma_commit(&done[slot]);
      ++issued;
    }
    __syncwarp();
    late = !__all_sync(0xffffffffu, !late && tc::mbar_wait(&done[slot], phase & 1u, wait_limit));
    ++phase;
    tc::fence_after_sync();
#pragma unroll
    for (int o = 1; o < LPR; o <<= 1) mask |= __shfl_xor_sync(0xffffffffu, mask, o);
    const int er = LPR == 1 ? e : __shfl_sync(0xffffffffu, e, 4 * (lane & 7));
#pragma unroll LPR == 1 ? 1 : 2
    for (int g = 0; g < W / 4; ++g) {
      float a[oz::S][8];
#pragma unroll
      for (int l = 0; l < oz::S; ++l) oz::tmem_ld8(tacc + ((uint32_t)(32 * w) << 16) + (uint32_t)(l * 2 * W + 8 * g), a[l]);
      tc::tmem_ld_wait();
      double2 o[NE];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float re[oz::S], im[oz::S];
#pragma unroll
        for (int l = 0; l < oz::S; ++l) {
          re[l] = a[l][2 * j];
          im[l] = a[l][2 * j + 1];
        }
        const int ec = er + eb[4 * g + j];
        double2 d = make_double2(oz::combine(re, ec), oz::combine(im, ec));
        if constexpr (LPR == 1) {
          o[j] = d;
        } else {  // lanes 0 .. 7 hold the eight vectors' sums, lane 4 x + j wants column j
          d = make_double2(__shfl_sync(0xffffffffu, d.x, lane >> 2), __shfl_sync(0xffffffffu, d.y, lane >> 2));
          if (j == 0 || h == j) o[0] = d;
        }
      }
      // Entries far below the operands' largest: again from the vector and T (see oz::far_below).
      double2 old[NE];
      fetch((c0 + W) / 4 + g, old);
      uint32_t far = 0;
#pragma unroll
      for (int i = 0; i < NE; ++i) {
        const int j = 4 * g + LPR * i + h;
        const double2 out = make_double2(old[i].x - o[i].x, old[i].y - o[i].y);
        if (oz::far_below(e + eb[j], mask & mb[j], old[i], out)) far |= 1u << i;
      }
      if (__any_sync(0xffffffffu, far)) {
        double2 sum[NE];
#pragma unroll
        for (int i = 0; i < NE; ++i) sum[i] = make_double2(0.0, 0.0);
#pragma unroll 1
        for (int kg = 0; kg < W / 4; ++kg) {
          double2 a4[NE];
          fetch(c0 / 4 + kg, a4);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            double2 ak = a4[k % NE];
            if (LPR > 1)
              ak = make_double2(__shfl_sync(0xffffffffu, ak.x, (lane & ~3) | k), __shfl_sync(0xffffffffu, ak.y, (lane & ~3) | k));
#pragma unroll
            for (int i = 0; i < NE; ++i) sum[i] = cfma(sum[i], ak, T[(c0 + 4 * kg + k) * GJ_KB + c0 + W + 4 * g + LPR * i + h]);
          }
        }
#pragma unroll
        for (int i = 0; i < NE; ++i)
          if (far >> i & 1u) o[i] = sum[i];
      }
      subtract((c0 + W) / 4 + g, o);
    }
  };
  if (solve) {
    // T: the scaled pivot rows; or L11^T with each column of L11 scaled by its pivot's reciprocal (the steps then
    // use the raw pivot-row entries), the reciprocals on the diagonal. Zero past kb.
    if (columns) {
      for (int e = tid; e < GJ_KB * GJ_KB; e += 128) {
        const int c = e & (GJ_KB - 1), k = e / GJ_KB;
        double2 u = make_double2(0.0, 0.0);
        if (c < kb && c >= k) {
          u = A[(k0 + c) + (int64_t)(k0 + k) * ld];
          if (c > k) u = cmul(u, A[(k0 + k) + (int64_t)(k0 + k) * ld]);
        }
        T[e] = u;
      }
    } else {
      const double2* pg = static_cast<const double2*>(t.prows);
      for (int e = tid; e < GJ_KB * GJ_KB; e += 128) {
        const int c = e & (GJ_KB - 1), k = e / GJ_KB;
        T[e] = c < kb && k < kb && c > k ? pg[e] : make_double2(0.0, 0.0);
      }
    }
    side_sync();
    int* eb = s_eb[slot];
    uint32_t* mb = s_mb[slot];
    {
      uint32_t m16, m8;
      const int r = tid >> 3, h8 = tid & 7;
      const int e16 = put_block<16>(sb16, T, 0, r, h8, s_half, -inner, m16);
      const int e8 = put_block<8>(sb8 + (tid >> 6) * B8_BYTES, T, 16 * (tid >> 6), r & 7, h8, s_half, -inner, m8);
      if (h8 == 0) {
        eb[r] = e16;
        eb[16 + r] = e8;
        mb[r] = m16;
        mb[16 + r] = m8;
      }
    }
    // A warp without vectors to solve only takes part in the barriers.
    const bool any = __any_sync(0xffffffffu, out);
    int e0 = LEAST;  // largest exponent of the block solved last
#pragma unroll 1
    for (int b = 0; b < GJ_KB / B && B * b < kb; ++b) {
      if (b > 0) {
        const bool wide = b == 2;
        product(b == 3 ? 16 : 0, wide ? 16 : 8, wide ? sb16 : sb8 + (b >> 1) * B8_BYTES, eb + (wide ? 0 : 16 + 8 * (b >> 1)),
                mb + (wide ? 0 : 16 + 8 * (b >> 1)), e0);
      }
      switch (b) {
        case 0: e0 = replay_block<LPR, 0>(v, T, h, any, s_half, inner); break;
        case 1: e0 = max(e0, replay_block<LPR, 1>(v, T, h, any, s_half, inner)); break;
        case 2: e0 = replay_block<LPR, 2>(v, T, h, any, s_half, inner); break;
        default: e0 = replay_block<LPR, 3>(v, T, h, any, s_half, inner); break;
      }
    }
    if (late && lane == 0) status[t.job] = ST_TIMEOUT;
  }
  if (columns) {
#pragma unroll
    for (int i = 0; i < Q; ++i) {
      const int c = LPR * i + h;
      if (c < kb) v[i] = cmul(v[i], T[c + c * GJ_KB]);
    }
    // Displaced rows into place (their places lie past the panel, their sources in it).
    const int* perm = t.perm;
    const int nd = perm[3 * GJ_KB];
    if (act)
#pragma unroll 4
      for (int c = h; c < nd; c += LPR) Ac[perm[GJ_KB + c]] = Ac[perm[2 * GJ_KB + c]];
  } else if (solve && act && !out) {  // a candidate: as the sweep left it
#pragma unroll
    for (int i = 0; i < Q; ++i) {
      const int c = LPR * i + h;
      v[i] = c < kb ? Ar[(int64_t)c * ld] : make_double2(0.0, 0.0);
    }
  }
  const int outer = columns ? 1 : -1;
  int e = LEAST;
#pragma unroll
  for (int i = 0; i < Q; ++i) e = max(e, exponent(v[i], outer * s_half[LPR * i + h]));
#pragma unroll
  for (int o = 1; o < LPR; o <<= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
  if (act && h == 0) (columns ? t.eb : t.ea)[q] = e;
  // The entries themselves for what oz::update_kernel computes again: solved rows in the panel, columns in t.y.
  if (out && !columns && solve) {
#pragma unroll
    for (int i = 0; i < Q; ++i) {
      const int c = LPR * i + h;
      if (c < kb) Ar[(int64_t)c * ld] = v[i];
    }
  }
  if (act && columns) {
    double2* Y = static_cast<double2*>(t.y) + (int64_t)q * GJ_KB;
#pragma unroll
    for (int i = 0; i < Q; ++i) Y[LPR * i + h] = v[i];
  }
  uint32_t mask = 0;
  if (act && !columns) {
    mask = put(t.oa + (size_t)(q / oz::ROWS) * oz::A_TILE, oz::A_SLICE, q % oz::ROWS, oz::ROWS, 0, GJ_KB / 4, e, outer);
  } else if (act) {  // rows (re, -im) and (im, re) of every digit (oz::write_b)
    unsigned char* tile = t.ob + (size_t)(q / oz::COLS) * oz::B_TILE;
#pragma unroll UNROLL
    for (int g = 0; g < GJ_KB / 4; ++g) {
      double2 o[NE];
      fetch(g, o);
      uint32_t d[NE][oz::S];
#pragma unroll
      for (int i = 0; i < NE; ++i) {
        oz::digit_pairs(o[i], e - s_half[4 * g + LPR * i + h], d[i]);
        mask |= (oz::is_zero(o[i]) ? 0u : 1u) << (4 * g + LPR * i + h);
      }
#pragma unroll
      for (int s = 0; s < oz::S; ++s)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          unsigned char* at = tile + oz::offset(2 * oz::COLS * s + 2 * (q % oz::COLS) + r, 8 * g + 2 * h, oz::B_ROWS);
          uint32_t p[NE];
#pragma unroll
          for (int i = 0; i < NE; ++i) p[i] = r ? __funnelshift_l(d[i][s], d[i][s], 16) : d[i][s] ^ 0x80000000u;
          if constexpr (LPR == 1) *reinterpret_cast<uint4*>(at) = make_uint4(p[0], p[1], p[2], p[3]);
          else *reinterpret_cast<uint32_t*>(at) = p[0];
        }
    }
  }
#pragma unroll
  for (int o = 1; o < LPR; o <<= 1) mask |= __shfl_xor_sync(0xffffffffu, mask, o);
  if (act && h == 0) (columns ? t.mb : t.ma)[q] = mask;
  // An MMA whose wait ran out is waited for once more before its memory goes away.
  if (late && tid == 0 && issued) tc::mbar_wait(&done[slot], (issued - 1) & 1u, TCU_WAIT);
  tc::fence_before_sync();
  __syncthreads();
  if (threadIdx.x < 32) tc::tmem_dealloc(tslot, LPR == 1 ? 512 : 256);
}

}  // namespace trail
}  // namespace caroli
