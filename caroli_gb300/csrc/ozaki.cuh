// FP64 rank-32 updates on the tcgen05 tensor cores: the products of inv_update_kernel<double> from
// exact integer products of operand digits (the Ozaki scheme, K. Ozaki, T. Ogita, S. Oishi, S. M. Rump,
// "Error-free transformations of matrix multiplication by using fast routines of matrix
// multiplication and its applications", Numer. Algorithms 59, 2012; with f16 inputs and f32
// accumulation as D. Mukunoki, K. Ozaki, T. Ogita, T. Imamura, ISC High Performance 2020).
//
// GB300's FP64 pipe does about two multiply-adds per clock and SM; the f16 tensor cores do 4 096. A
// row of the left factor (32 complex entries, K = 64 real) is scaled by the power of two above its
// largest component and written as seven signed base-512 digits (62 bits, so an entry keeps 53 bits
// down to 2^-9 of the row's largest); a column of the right factor likewise. Digits are at most 256 in
// modulus, exact in f16; a product of digits is at most 2^16 and a sum of 64 of them 2^22, so the
// f32 accumulators hold exact integers while fewer than five digit pairs share one (levels i + j <= 3)
// and, past that, unless nearly every digit has its largest value: then a rounding of 2^-24 of a level
// that itself weighs 2^-36 or less. Levels i + j <= 6 are kept (28 pairs); what is left out, with what the digits
// cut off, weighs 2^-59 of (row's largest) x (column's largest) per term at most. The levels are put together in
// 64-bit integers and rounded to FP64 (integer arithmetic: the FP64 pipe only does the final add).
//
// A 128 x 16 complex tile takes 15 Mflop on the f16 cores in place of 0.52 Mflop on the FP64 pipe (80 us
// on one SM). Measured: the updates of two 48 x 24 x 24 cubic wires' fronts 121 -> 9.2 ms
// (a factor 1.4 of it from the trailing form), of 16 BHZ 200 x 64 solves 58.8 -> 6.2 ms (6.9 and 3.9 without what
// far_below has computed again); T against 64 bits equal to the FP64 pipe's within its scatter (1e-15 to 5e-12 on
// these devices).
//
// The complex product is a real GEMM D = A' B'^T with the row's 32 complex entries as K = 64 and
// two columns of D per complex column:
//     A'[i][2c] = Re P[i, c], A'[i][2c+1] = Im P[i, c]
//     B'[2j][2c] = Re Y[c, j], B'[2j][2c+1] = -Im Y[c, j], B'[2j+1][2c] = Im Y, B'[2j+1][2c+1] = Re Y
// so a lane of tensor memory is a complex row and 32 lanes read and write 512 consecutive bytes of a
// column of the matrix.
#pragma once
#include <cuda_fp16.h>

#include "dense.cuh"

namespace caroli {
namespace oz {

constexpr int S = 7;                             // digits per operand
constexpr int ROWS = 128;                        // complex rows per tile (the MMA's M)
constexpr int COLS = 16;                         // complex columns per tile (N = 32)
constexpr int A_SLICE = ROWS * 2 * GJ_KB * 2;    // bytes of one digit of A': 128 x 64 f16
constexpr int A_TILE = S * A_SLICE;
// B' of a tile stacks its digits along N (row 32 s + j: digit s of B' row j), so that one MMA multiplies
// a digit i of A' with the digits 0 .. 6 - i of B' into the accumulators of the levels i .. 6.
constexpr int B_ROWS = S * 2 * COLS;
constexpr int B_TILE = B_ROWS * 2 * GJ_KB * 2;
constexpr int STAGES = 3;                        // B' tiles in shared memory
constexpr int SMEM = A_TILE + STAGES * B_TILE + 1024;
constexpr int ACC = 256;                         // tensor-memory columns of one of two accumulator sets (S x 32 used)
constexpr int EPI_WARPS = 16;
constexpr int THREADS = 32 * (2 + EPI_WARPS);
constexpr int NOT_FINITE = 1 << 20;              // exponent of a row or column holding Inf or NaN

// Operand bytes of a matrix of n rows and columns: A' and B' tiles, row and column exponents and masks, and the columns'
// entries in FP64 (the rows' are in the panel).
__host__ __device__ inline size_t a_bytes(int n) { return (size_t)((n + ROWS - 1) / ROWS) * A_TILE; }
__host__ __device__ inline size_t b_bytes(int n) { return (size_t)((n + COLS - 1) / COLS) * B_TILE; }
__host__ __device__ inline size_t e_bytes(int n) { return ((size_t)n * 4 + 255) / 256 * 256; }
__host__ __device__ inline size_t y_bytes(int n) { return (size_t)n * GJ_KB * sizeof(double2); }
__host__ __device__ inline size_t bytes(int n) { return a_bytes(n) + b_bytes(n) + 4 * e_bytes(n) + y_bytes(n); }

// Byte offset of element (row, k) of an f16 operand: K-slices of 16 elements (one kind::f16 MMA) in the
// core-matrix layout of tc.cuh (8 rows x 16 bytes; leading offset 128, stride offset 256).
__device__ __forceinline__ uint32_t offset(int row, int k, int rows) {
  return (uint32_t)((k >> 4) * rows * 32 + (row >> 3) * 256 + ((k >> 3) & 1) * 128 + (row & 7) * 16 + (k & 7) * 2);
}

__device__ __forceinline__ int biased_exponent(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }

// Digits are cut relative to the largest entries, so an output's error is relative to their product M, whatever its own
// size: 2^-57 of it or so. Where the large entries of a row meet small ones of a column and the other way round, as in
// the fronts of a device whose couplings decay over the pivots of a panel, the output is far below M; at 2^-62 M
// nothing is left of it. An output whose old and new values are both below 2^-FAR M is therefore computed again on the
// FP64 pipe. (Without, T of a 60 x 30 square with Anderson disorder 16, 2.5e-31, was off by 7e-5, and by decades at 30.)
// Rows and columns that share no nonzero entry (masks) give an exact zero and stay out.
// FAR = 12: with 8, two 48 x 24 x 24 cubic wires take 42.3 ms in place of 28.9, with 16 28.1 and with none computed again
// 27.6; devices whose rows and columns are scaled over six decades either way come out 1.0e-13 (geometric mean)
// off with 12, 1.1e-12 with 16 and 8e-14 on the FP64 pipe alone.
// Where most outputs are computed again (four solves of a 24 x 14 x 14 cubic wire, disorder 60) a solve takes 10.0 ms in
// place of 5.8 (disorder 16.5) and of 36.5 with rank-32 updates on the FP64 pipe.
constexpr int FAR = 12;
__device__ __forceinline__ bool is_zero(double2 v) {
  return ((unsigned)(__double2hiint(v.x) | __double2hiint(v.y)) << 1 | (unsigned)(__double2loint(v.x) | __double2loint(v.y))) == 0u;
}
__device__ __forceinline__ int top_exponent(double2 v) { return max(biased_exponent(v.x), biased_exponent(v.y)); }
// ec: sum of the row's and the column's biased exponents; common: their common nonzero entries.
__device__ __forceinline__ bool far_below(int ec, uint32_t common, double2 old, double2 out, int far = FAR) {
  return common && max(top_exponent(old), top_exponent(out)) < ec - 1023 - far;
}

// x as a 62-bit fixed-point number, x 2^(1084 - e) rounded toward zero (e the biased exponent of the largest
// entry, at least 1), plus 256 in the place of each base-512 digit: the digits of the sum, less 256, are the signed digits of x.
__device__ __forceinline__ unsigned long long biased_digits(double x, int e) {
  const int hi = __double2hiint(x);
  const int ex = (hi >> 20) & 0x7ff;
  const unsigned mh = (unsigned)(hi & 0xfffff) | (ex ? 0x100000u : 0u), ml = (unsigned)__double2loint(x);
  const unsigned long long m = ((unsigned long long)mh << 32 | ml) << 9;
  const unsigned long long v = m >> min(e - max(ex, 1), 63);
  constexpr unsigned long long BIAS = 0x4020100804020100ull;  // 256 x (1 + 512 + ... + 512^6)
  return hi < 0 ? BIAS - v : BIAS + v;
}
// The seven signed digits of a complex entry, most significant first, each in [-256, 256], as pairs (re, im) of
// f16: 0x6400 + u is 1024 + u in f16's binade [1024, 2048), from which 1280 is taken.
__device__ __forceinline__ void digit_pairs(double2 x, int e, uint32_t (&d)[S]) {
  const unsigned long long re = biased_digits(x.x, e), im = biased_digits(x.y, e);
#pragma unroll
  for (int s = 0; s < S; ++s) {
    const int at = 9 * (S - 1 - s);
    const unsigned mask = s ? 511u : 1023u;
    const uint32_t b = ((uint32_t)(re >> at) & mask) | ((((uint32_t)(im >> at) & mask) | 0x6400u) << 16) | 0x6400u;
    const __half2 v = __hsub2(*reinterpret_cast<const __half2*>(&b), __half2half2(__ushort_as_half(0x6500)));
    d[s] = *reinterpret_cast<const uint32_t*>(&v);
  }
}

// The largest exponent of the entries LPR lanes hold (at least 1).
template <int LPR> __device__ __forceinline__ int row_exponent(const double2 (&a)[GJ_KB / LPR]) {
  int e = 1;
#pragma unroll
  for (int i = 0; i < GJ_KB / LPR; ++i) e = max(e, max(biased_exponent(a[i].x), biased_exponent(a[i].y)));
#pragma unroll
  for (int o = 1; o < LPR; o <<= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
  return e;
}

// The nonzero entries of LPR lanes, lane h holding LPR i + h.
template <int LPR> __device__ __forceinline__ uint32_t row_mask(const double2 (&a)[GJ_KB / LPR], int h) {
  uint32_t m = 0;
#pragma unroll
  for (int i = 0; i < GJ_KB / LPR; ++i) m |= (is_zero(a[i]) ? 0u : 1u) << (LPR * i + h);
#pragma unroll
  for (int o = 1; o < LPR; o <<= 1) m |= __shfl_xor_sync(0xffffffffu, m, o);
  return m;
}

// Row q of A' from LPR lanes, lane h holding the entries LPR i + h: four lanes' 4-byte pairs (re, im) fill
// a 16-byte core-matrix row.
template <int LPR>
__device__ __forceinline__ void write_a(unsigned char* oa, int32_t* ea, int q, int h, bool act,
                                        const double2 (&a)[GJ_KB / LPR], size_t tile_stride = A_TILE) {
  const int e = row_exponent<LPR>(a);
  if (!act) return;
  if (h == 0) ea[q] = e == 0x7ff ? NOT_FINITE : e;
  unsigned char* tile = oa + (size_t)(q / ROWS) * tile_stride;
#pragma unroll
  for (int i = 0; i < GJ_KB / LPR; ++i) {
    uint32_t d[S];
    digit_pairs(a[i], e, d);
    const uint32_t off = offset(q % ROWS, 2 * (LPR * i + h), ROWS);
#pragma unroll
    for (int s = 0; s < S; ++s) *reinterpret_cast<uint32_t*>(tile + s * A_SLICE + off) = d[s];
  }
}

// Column r of B' (rows 2r and 2r + 1) from LPR lanes, laid out over the lanes as in write_a.
template <int LPR>
__device__ __forceinline__ void write_b(unsigned char* ob, int32_t* eb, int r, int h, bool act,
                                        const double2 (&y)[GJ_KB / LPR], size_t tile_stride = B_TILE) {
  const int e = row_exponent<LPR>(y);
  if (!act) return;
  if (h == 0) eb[r] = e == 0x7ff ? NOT_FINITE : e;
  unsigned char* tile = ob + (size_t)(r / COLS) * tile_stride;
  const int row = 2 * (r % COLS);
#pragma unroll
  for (int i = 0; i < GJ_KB / LPR; ++i) {
    uint32_t d[S];
    digit_pairs(y[i], e, d);
    const int k = 2 * (LPR * i + h);
#pragma unroll
    for (int s = 0; s < S; ++s) {
      *reinterpret_cast<uint32_t*>(tile + offset(2 * COLS * s + row, k, B_ROWS)) = d[s] ^ 0x80000000u;
      *reinterpret_cast<uint32_t*>(tile + offset(2 * COLS * s + row + 1, k, B_ROWS)) = __funnelshift_l(d[s], d[s], 16);
    }
  }
}

// The seven level sums of one output as FP64: 2^(e - 2114) Σ_l a_l 512^(6 - l), an integer of at most 77 bits. e: sum of
// the row's and the column's biased exponents. Taken as 64 bits, 5 or 14 of them left out (rounded) where it is below or
// past 2^-10 of the product of the largest entries, then rounded to FP64: off by less than one last place. (14 left
// out everywhere, rounded toward minus infinity, was up to 2^-54 of that product, the larger error of small outputs.)
__device__ __forceinline__ double combine(const float (&a)[S], int e) {
  int v[S];
#pragma unroll
  for (int l = 0; l < S; ++l) v[l] = __float2int_rn(a[l]);
  const long long hi = ((long long)v[0] << 18) + ((long long)v[1] << 9) + v[2];
  const long long lo = ((long long)v[3] << 27) + ((long long)v[4] << 18) + ((long long)v[5] << 9) + v[6];
  const bool small = hi == (long long)(int)hi;
  const long long w = small ? (hi << 31) + ((lo + 16) >> 5) : (hi << 22) + ((lo + 8192) >> 14);
  if (e >= NOT_FINITE) return __longlong_as_double(0x7ff8000000000000ll);
  if (w == 0) return 0.0;
  const unsigned long long u = w < 0 ? (unsigned long long)(-w) : (unsigned long long)w;
  const int lz = __clzll((long long)u);
  const unsigned long long norm = u << lz;
  const int ex = 1023 + 63 - lz + e - (small ? 2109 : 2100);
  // 53 bits rounded to nearest (ties up); the carry of the rounding moves the exponent.
  unsigned long long bits;
  if (ex > 0) bits = ex > 2046 ? 0x7ff0000000000000ull : ((unsigned long long)(ex - 1) << 52) + (norm >> 11) + ((norm >> 10) & 1ull);
  else bits = ex > -52 ? (norm >> (12 - ex)) + ((norm >> (11 - ex)) & 1ull) : 0ull;  // below the normal numbers
  return __longlong_as_double((long long)(bits | (w < 0 ? 1ull << 63 : 0ull)));
}

__host__ __device__ constexpr uint32_t idesc_f16(int m, int n) {
  return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);  // D: f32; A, B: f16, K-major
}
__device__ __forceinline__ void mma_f16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, bool accumulate) {
  const uint32_t acc = accumulate ? 1u : 0u;
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.u32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8]) {
  uint32_t r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

// The products of a tile's digits (one thread): one MMA per digit i of A' and K-slice, N = 32 (7 - i).
__device__ __forceinline__ void mma_tile(uint32_t acc, const unsigned char* sa, const unsigned char* sb) {
  const uint32_t pb = tc::smem_addr(sb);
#pragma unroll
  for (int i = 0; i < S; ++i) {
    const uint32_t pa = tc::smem_addr(sa + i * A_SLICE);
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
      mma_f16(acc + (uint32_t)(i * 2 * COLS), tc::smem_desc(pa + ks * ROWS * 32, 128, 256),
              tc::smem_desc(pb + ks * B_ROWS * 32, 128, 256), idesc_f16(ROWS, 2 * COLS * (S - i)), i > 0 || ks > 0);
  }
}

// The update of one panel (operands written by panel_rest_kernel). A CTA takes 128 rows of a matrix and
// `group` tiles of 16 columns: warp 0 (one thread) bulk-copies A' once and the B' tiles into a ring of
// three, warp 1 (one thread) issues 7 x 4 MMAs per tile (N = 224, 192, ... 32: 1 792 clocks at the full f16
// rate; a 128 x 32 x 16 MMA per digit pair took 53 clocks, 6 000 per tile) into one of two sets of seven
// 32-column accumulators, warps 2-17 (four per lane quarter, four complex columns each) add the other set's
// tile to the old values (zero on the pivot rows of the full form) and compute again what is far below (far_below):
// with their FP64 adds that keeps the pipe 37 % busy on BHZ fronts, the integer pipe as much. Two sets of 32-column
// tiles would not fit in tensor memory. Waits are bounded as in tc_update_kernel. grid (row tiles, matrices,
// column groups).
__global__ void __launch_bounds__(THREADS, 1) update_kernel(const InvTask* __restrict__ tasks, int k0, int group,
                                                            int32_t* __restrict__ status, uint32_t wait_limit) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint32_t tslot;
  __shared__ __align__(8) uint64_t afull, bfull[STAGES], bempty[STAGES], tfull[2], tempty[2];
  __shared__ int abort_flag;
  const InvTask t = tasks[blockIdx.y];
  const int n = t.n;
  if (k0 >= t.npiv || *t.bad) return;
  const int kb = min(GJ_KB, t.npiv - k0);
  const bool trail = t.trail != 0;
  const int base = trail ? k0 + kb : 0;
  const int rows = n - base, rest = trail ? rows : n - kb;
  const int i0 = blockIdx.x * ROWS;
  const int tile0 = blockIdx.z * group;
  const int tiles = min((rest + COLS - 1) / COLS - tile0, group);
  if (i0 >= rows || tiles <= 0) return;
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  unsigned char* sa = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* sb = sa + A_TILE;
  if (w == 0) tc::tmem_alloc(&tslot, 2 * ACC);
  if (tid == 0) {
    tc::mbar_init(&afull, 1);
    for (int i = 0; i < STAGES; ++i) {
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
    status[t.job] = ST_TIMEOUT;
  };
  int copies = 0, mma_tiles = 0;
  if (w == 0) {
    if (lane == 0) {
      tc::mbar_arrive_expect_tx(&afull, A_TILE);
      for (int s = 0; s < S; ++s)
        tc::bulk_copy_g2s(sa + s * A_SLICE, t.oa + (size_t)blockIdx.x * A_TILE + s * A_SLICE, A_SLICE, &afull);
      for (int ct = 0; ct < tiles && !*abort_v; ++ct) {
        const int st = ct % STAGES;
        if (ct >= STAGES && !tc::mbar_wait(&bempty[st], (uint32_t)((ct / STAGES - 1) & 1), wait_limit)) { fail(); break; }
        tc::mbar_arrive_expect_tx(&bfull[st], B_TILE);
        tc::bulk_copy_g2s(sb + st * B_TILE, t.ob + (size_t)(tile0 + ct) * B_TILE, B_TILE, &bfull[st]);
        ++copies;
      }
    }
  } else if (w == 1) {
    if (lane == 0) {
      if (!tc::mbar_wait(&afull, 0, wait_limit)) fail();
      for (int ct = 0; ct < tiles && !*abort_v; ++ct) {
        const int st = ct % STAGES, a = ct & 1;
        if (!tc::mbar_wait(&bfull[st], (uint32_t)((ct / STAGES) & 1), wait_limit)) { fail(); break; }
        if (ct >= 2 && !tc::mbar_wait(&tempty[a], (uint32_t)(((ct >> 1) - 1) & 1), wait_limit)) { fail(); break; }
        tc::fence_after_sync();
        mma_tile(tbase + (uint32_t)(a * ACC), sa, sb + st * B_TILE);
        tc::mma_commit(&bempty[st]);
        tc::mma_commit(&tfull[a]);
        ++mma_tiles;
      }
    }
  } else {
    // The warp's lane quarter of tensor memory (rows) and four of the tile's complex columns; their old
    // values are requested while the tile is multiplied.
    const int q = w & 3, part = (w - 2) >> 2;
    const int r = i0 + 32 * q + lane, gi = base + r;
    const bool row_in = r < rows;
    const bool keep_old = row_in && (trail || gi < k0 || gi >= k0 + kb);
    const int er = row_in ? t.ea[r] : 1;
    const uint32_t mr = row_in ? t.ma[r] : 0u;
    const double2* Y = static_cast<const double2*>(t.y);
    double2* Ai = static_cast<double2*>(t.a) + gi;
    const int64_t ld = t.ld;
    constexpr int CW = 4 * COLS / EPI_WARPS;  // complex columns per warp and tile
    static_assert(CW == 4, "eight accumulator columns per load");
    auto col_of = [&](int c) { return trail ? base + c : (c < k0 ? c : c + kb); };
    for (int ct = 0; ct < tiles; ++ct) {
      const int c0 = (tile0 + ct) * COLS + part * CW, a = ct & 1;
      double2 old[CW];
      int ec[CW];
#pragma unroll
      for (int j = 0; j < CW; ++j) {
        const bool in = c0 + j < rest;
        old[j] = (keep_old && in) ? Ai[(int64_t)col_of(c0 + j) * ld] : make_double2(0.0, 0.0);
        ec[j] = in ? er + t.eb[c0 + j] : 2;
      }
      bool ok = !*abort_v && tc::mbar_wait(&tfull[a], (uint32_t)((ct >> 1) & 1), wait_limit);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) {
        if (lane == 0) fail();
        break;
      }
      tc::fence_after_sync();
      float v[S][2 * CW];
#pragma unroll
      for (int l = 0; l < S; ++l)
        tmem_ld8(tbase + ((uint32_t)(32 * q) << 16) + (uint32_t)(a * ACC + l * 2 * COLS + part * 2 * CW), v[l]);
      tc::tmem_ld_wait();
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&tempty[a]);
      uint32_t far = 0;
#pragma unroll
      for (int j = 0; j < CW; ++j) {
        float x[S], y[S];
#pragma unroll
        for (int l = 0; l < S; ++l) {
          x[l] = v[l][2 * j];
          y[l] = v[l][2 * j + 1];
        }
        // trail: old - L Y; full: old + (swept panel) Y.
        const double re = combine(x, ec[j]), im = combine(y, ec[j]);
        const double2 out = trail ? make_double2(old[j].x - re, old[j].y - im) : make_double2(old[j].x + re, old[j].y + im);
        const bool in = row_in && c0 + j < rest;
        if (in) Ai[(int64_t)col_of(c0 + j) * ld] = out;
        if (in && far_below(ec[j], mr & t.mb[c0 + j], old[j], out)) far |= 1u << j;
      }
      if (__any_sync(0xffffffffu, far)) {
        // Few rows of a column: the lanes share the sum of a row; many: a row per lane.
        const double2* P = static_cast<const double2*>(t.a) + (int64_t)k0 * ld;  // the panel
#pragma unroll
        for (int j = 0; j < CW; ++j) {
          uint32_t rows_far = __ballot_sync(0xffffffffu, far >> j & 1u);
          const double2* Yj = Y + (int64_t)(c0 + j) * GJ_KB;
          double2 sum = make_double2(0.0, 0.0);
          if (__popc(rows_far) > 8) {
            if (far >> j & 1u)
#pragma unroll 4
              for (int k = 0; k < kb; ++k) sum = cfma(sum, P[gi + k * ld], Yj[k]);
          } else {
            while (rows_far) {
              const int src = __ffs(rows_far) - 1, i = __shfl_sync(0xffffffffu, gi, src);
              rows_far &= rows_far - 1;
              double2 p = lane < kb ? cmul(P[i + lane * ld], Yj[lane]) : make_double2(0.0, 0.0);
#pragma unroll
              for (int o = 16; o > 0; o >>= 1) {
                p.x += __shfl_xor_sync(0xffffffffu, p.x, o);
                p.y += __shfl_xor_sync(0xffffffffu, p.y, o);
              }
              if (lane == src) sum = p;
            }
          }
          if (far >> j & 1u)
            Ai[(int64_t)col_of(c0 + j) * ld] =
                trail ? make_double2(old[j].x - sum.x, old[j].y - sum.y) : make_double2(old[j].x + sum.x, old[j].y + sum.y);
        }
      }
    }
  }
  // Where a wait ran out, drain what was issued (see tc_update_kernel).
  tc::fence_before_sync();
  __syncthreads();
  if (abort_flag) {
    if (w == 0 && lane == 0) {
      tc::mbar_wait(&afull, 0, TCU_WAIT);
      for (int ct = max(0, copies - STAGES); ct < copies; ++ct)
        tc::mbar_wait(&bfull[ct % STAGES], (uint32_t)((ct / STAGES) & 1), TCU_WAIT);
    }
    if (w == 1 && lane == 0 && mma_tiles > 0)
      tc::mbar_wait(&bempty[(mma_tiles - 1) % STAGES], (uint32_t)(((mma_tiles - 1) / STAGES) & 1), TCU_WAIT);
    tc::fence_before_sync();
    __syncthreads();
  }
  if (w == 0) tc::tmem_dealloc(tbase, 2 * ACC);
}

}  // namespace oz
}  // namespace caroli
