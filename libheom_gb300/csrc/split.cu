// FP64 stage kernel with the commutator on the tensor cores: site-local baths,
// real symmetric H, 4 to 32 levels.  Same operator and stage epilogues as
// k_rhs_diag<double> (heom_hilb.h:96-215 with the fused rk4 / lsrk4 / rkdp
// stages).
//
// The FP64 pipe executes two operations per clock per SM, and 4 n of an
// element's operations are the commutator.  Here rho and H are cut into eight
// signed digits of nine bits each (fixed point, 70 bits below the largest value
// of a row of rho's operand, or of a column of H); the digits are integers of at
// most 256, exact in FP16, and a product of two digit matrices summed over
// n <= 32 and over the eight pairs of one order i + j is at most 2^24, so the
// FP32 accumulators of the tensor cores hold it exactly.  The orders 0 to 7 are
// combined with integer operations and rounded to FP64 once per value; what is
// left out (orders above 7 and bits of the values below 2^-70 of their row's
// largest) is below n 2^-66.8 of the scale, the product of the row's and the
// column's power of two (the error-free splitting of matrix products of Ozaki,
// Ogita, Oishi and Rump, Numer. Algorithms 59, 2012).
//
// Element by element the result is as good as FP64 sums, whose error is n 2^-53
// of an element's own terms at worst: a component whose larger product reaches
// 2^-13 of the scale has an error of n 2^-53.8 of it at worst (2^-55 in the mean),
// and the others (2 in 10000 for 24 coupled sites, nearly all for a state
// localised on a chain), rows whose largest value lies outside 2^-800 .. 2^900,
// infinities and NaNs take FP64 sums in pass 5.  One scale for an ADO and seven
// digits were faster (0.59 ms where this takes 0.78) and lost the small elements of
// graded states.  Measured against 64 bits, 24 sites, mean of eight states: 8.1e-17
// of the norm after four steps (FP64 sums 9.7e-17), 3.0e-16 after 40 (3.4e-16).  A
// stage of the 24-site model at depth 3 (12M elements) takes 0.78 ms, 2.95 with
// k_rhs_diag<double>, whose FP64 pipe alone needs 2.58 (16 sites: 0.115 and 0.287).
//
// Per tile of T = 128 / (4 n) ADOs, the first group of a CTA (256 threads):
//   1. the stage input (copied with cp.async a tile ahead), the largest exponent
//      of each row of R, I, R^T and I^T (rho = R + iI);
//   2. the rows' digits (4 n rows per ADO, K = n padded to 16) into the A
//      operand, K-major without swizzle;
//   3. MMAs (M = 128, one thread): digit i of rho against the digits 0..7-i of
//      H at once (N = 8 - i blocks of n padded to 16), into the tensor-memory
//      columns of the orders i..7, so 8 MMAs per 16 of K cover all 36 pairs;
//   4. read-back: rows of R H, I H (rho H) and R^T H, I^T H (H rho,
//      transposed) in FP64 to shared memory;
// and the second group (192 threads), a tile behind it:
//   5. one element per thread: the difference of the two products, or FP64 sums
//      (a few elements of a warp by the whole warp one after another, many lane
//      by lane); damping and +1 terms (ADOs below the deepest tier);
//   6. the -1 terms, one thread per element that a mode touches (an FP64
//      instruction takes the pipe's 64 cycles whatever lanes it has: inside
//      pass 5 these terms' few lanes made every warp pay, 0.44 of 1.22 ms);
//   7. the stage epilogue, one element per thread.
// The groups meet on named barriers: products full (first to second) and free
// (second to first).  Two CTAs per SM, by tensor memory (256 of 512 columns)
// and registers.  What bounds it: the first group's chain of integer work (digits,
// read-back), then the second's FP64 issue and shared memory latency.  Measured at 24
// sites, ms a stage: threads of the groups 128 and 320 0.89, 256 and 192 0.82, 256
// and 224 0.84, 256 and 160 0.85, 384 and 128 1.07; the digits written four at a
// time by row 0.79; pass 1 with two threads a row 0.78.  Without any FP64 sums
// in pass 5 it would take 0.76, without pass 1 0.73.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "heomgb_impl.cuh"
#include "stage.cuh"
#include "tcore.cuh"

namespace heomgb {

namespace {

constexpr int kDigits = 8, kBits = 9;
constexpr int kSplitX = 256, kSplitY = 192;  // threads of the two groups
constexpr int kSplitThreads = kSplitX + kSplitY;
constexpr int kBarX = 1, kBarY = 2, kBarFull = 3, kBarFree = 4;  // named barriers
constexpr int kSplitCols = 256;  // tensor-memory columns of a CTA: eight orders of at most 32
// the bias of four digits: sum of 256 * 2^(9 k), k = 0..3
constexpr unsigned long long kBias = 0x804020100ull;
constexpr unsigned long long kLow = (1ull << 36) - 1;
// A row's exponent field (s_exp): 0 for a row of zeros, kRowOut for one that the digits do not hold
constexpr int kRowMin = 223, kRowMax = 1922, kRowOut = 3000;
// A commutator's component whose larger product is below 2^-kTrust of its scale takes FP64 sums
constexpr int kTrust = 13;
constexpr int kNoColumn = -20000;  // the exponent of a column of zeros

struct SplitGeom {
  int tile, rows, kp, np;  // ADOs; rows 4 n tile; K and N padded to 16
  int sbo, dstride;        // bytes of an 8-row group, of a digit
};
__host__ __device__ __forceinline__ SplitGeom split_geom(int n) {
  SplitGeom g;
  g.tile = 128 / (4 * n);
  g.rows = 4 * n * g.tile;
  g.kp = g.np = (n + 15) & ~15;
  g.sbo = g.kp / 8 * 128;
  g.dstride = (g.rows + 7) / 8 * g.sbo;
  return g;
}
// the A operand (the last digit's MMA reads 128 rows), then the products
__host__ __device__ __forceinline__ size_t split_a_bytes(int n) {
  const SplitGeom g = split_geom(n);
  return (static_cast<size_t>(kDigits - 1) * g.dstride + 16 * static_cast<size_t>(g.sbo) + 127) & ~size_t(127);
}
__host__ __device__ __forceinline__ size_t split_p_bytes(int n) {
  return (static_cast<size_t>(split_geom(n).rows) * (n + 1) * 8 + 127) & ~size_t(127);
}
__host__ __device__ __forceinline__ size_t split_b_bytes(int n) {
  const SplitGeom g = split_geom(n);
  return static_cast<size_t>(kDigits) * g.np / 8 * g.sbo;
}
__host__ __device__ __forceinline__ size_t split_y_bytes(int n, int w) {
  const SplitGeom g = split_geom(n);
  return static_cast<size_t>(g.tile) * (n * n * sizeof(double2) + (1 + w) * sizeof(int4));
}

// |x| truncated to 70 bits at the scale of the biased exponent es (at least x's), plus
// the digits' bias: digits 0..3 in the low 36 bits of lo, 4..7 of hi
struct Fixed {
  unsigned long long lo, hi;
  uint32_t sign;  // 0x8000 for a negative x
};
__device__ __forceinline__ Fixed to_fixed(double x, int es) {
  const unsigned long long u = static_cast<unsigned long long>(__double_as_longlong(x));
  const int ex = static_cast<int>(u >> 52) & 0x7ff;
  const unsigned long long m = ex ? (u << 11) | (1ull << 63) : 0ull;  // the leading bit at 63: bit 69 of the 70
  const int sh = min(es - ex, 97);
  const unsigned long long hi = sh < 34 ? m >> (30 + sh) : 0ull;
  const unsigned long long lo = (sh < 34 ? m << (34 - sh) : m >> (sh - 34)) >> 28;
  Fixed f;
  f.lo = lo + kBias;
  f.hi = hi + kBias + (f.lo >> 36);
  f.sign = static_cast<uint32_t>(u >> 48) & 0x8000u;
  return f;
}

__device__ __forceinline__ uint32_t digit(unsigned long long y, int k) {  // the biased digit of weight 2^(9 k)
  return static_cast<uint32_t>(y >> (kBits * k)) & 0x1ffu;
}
// two biased digits as a pair of FP16 integers: 1024 + u from the bits, minus 1024 + 256 (exact)
__device__ __forceinline__ uint32_t digit_pair(uint32_t a, uint32_t b) {
  const uint32_t w = (a | (b << 16)) | 0x64006400u;
  const __half2 h = __hsub2(*reinterpret_cast<const __half2*>(&w), __floats2half2_rn(1280.f, 1280.f));
  return *reinterpret_cast<const uint32_t*>(&h);
}

__device__ __forceinline__ long long mad_wide(int a, int b, long long c) {
  long long r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
}

// x != 0 on the bit patterns (a comparison takes the FP64 pipe)
__device__ __forceinline__ bool nonzero_bits(double x) { return (__double_as_longlong(x) << 1) != 0; }

// v 2^e as the nearest double (ties to even), |v| < 2^63 and the result normal:
// about 20 integer instructions, where a conversion and a multiplication take
// the FP64 pipe for 128 cycles a warp
__device__ __forceinline__ double from_fixed(long long v, int e) {
  const unsigned long long s = static_cast<unsigned long long>(v) & (1ull << 63);
  unsigned long long m = static_cast<unsigned long long>(v < 0 ? -v : v);
  if (m == 0ull) return 0.0;
  const int lz = __clzll(static_cast<long long>(m)) - 1;  // the leading bit to position 62
  m <<= lz;
  m = (m + 0x1ffull + ((m >> 10) & 1ull)) >> 10;  // 53 bits; a carry into bit 53 raises the exponent below
  const unsigned long long ex = static_cast<unsigned long long>(1023 + 62 - lz + e - 1);
  return __longlong_as_double(static_cast<long long>(s | ((ex << 52) + m)));
}

// sum of o[s] 2^(9 (7 - s)) over the eight orders, times 2^e, to the nearest double (|o| <= 2^24)
__device__ __forceinline__ double from_orders(const int (&o)[kDigits], int e) {
  const long long hi = mad_wide(o[0], 1 << 27, mad_wide(o[1], 1 << 18, mad_wide(o[2], 1 << 9, o[3])));
  const long long lo = mad_wide(o[4], 1 << 27, mad_wide(o[5], 1 << 18, mad_wide(o[6], 1 << 9, o[7])));
  // hi 2^36 + lo in the 62 bits from its leading one on
  const int s = min(36, __clzll(hi < 0 ? -hi : hi) - 2);
  return from_fixed((hi << s) + (lo >> (36 - s)), e + 36 - s);
}

// four columns of one order at taddr, without the wait
__device__ __forceinline__ void ld4_issue(uint32_t taddr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
}

template <int ID, int COUNT>
__device__ __forceinline__ void bar_sync() {
  asm volatile("bar.sync %0, %1;\n" ::"n"(ID), "n"(COUNT) : "memory");
}
template <int ID, int COUNT>
__device__ __forceinline__ void bar_arrive() {
  asm volatile("bar.arrive %0, %1;\n" ::"n"(ID), "n"(COUNT) : "memory");
}

__device__ __forceinline__ void split_cp(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s_addr(dst)), "l"(src) : "memory");
}
// Issues the copies of a tile's stage input and records (first group).
__device__ __forceinline__ void split_stage(const DiagInst* __restrict__ I, const DiagTile& td,
                                            const double2* __restrict__ y, unsigned char* raw) {
  const int n2 = I->n2, w1 = 1 + I->site_w;
  double2* ys = reinterpret_cast<double2*>(raw);
  int4* rec = reinterpret_cast<int4*>(ys + static_cast<size_t>(I->tile) * n2);
  const double2* ysrc = y + I->elem_off + static_cast<size_t>(td.l0) * n2;
  const int4* rsrc = I->site_rec + static_cast<size_t>(td.l0) * w1;
  for (int i = threadIdx.x; i < td.nt * n2; i += kSplitX) split_cp(ys + i, ysrc + i);
  for (int i = threadIdx.x; i < td.nt * w1; i += kSplitX) split_cp(rec + i, rsrc + i);
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}

template <int KIND>
__global__ void __launch_bounds__(kSplitThreads, 2) k_rhs_split(const DiagSet ds, const Stage st) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t mbar;
  __shared__ uint32_t tslot;
  __shared__ short s_exp2[2][128];  // the exponent of every row of A, two tiles in turn
  __shared__ volatile int s_fail;  // 1 + the tile whose MMAs did not complete
  double dt;
  int cur;
  // one verdict per CTA (k_rhs_diag_tc)
  if (!__syncthreads_and(stage_prologue<KIND>(st, dt, cur))) return;
  const double2* __restrict__ y = stage_input<double2>(st, cur);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned char* As = smem_raw;
  double* P = reinterpret_cast<double*>(smem_raw + ds.split_p);
  unsigned char* Bs = smem_raw + ds.split_b;
  if (warp == 0) tmem_alloc(&tslot, kSplitCols);
  if (tid == 0) {
    mbar_init(&mbar);
    mbar_init_fence();
  }
  if (tid == 0) s_fail = 0;
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = tslot;
  double local = 0.0;
  const int step = gridDim.x;
  if (tid < kSplitX) {
    // ---------------------------------------------------------------- first group: passes 1 to 4
    uint32_t parity = 0;
    int b_inst = -1, buf = 0, eb = 0;
    DiagTile td{}, tdn{};
    if (blockIdx.x < ds.n_tiles) {
      tdn = ds.tiles[blockIdx.x];
      split_stage(ds.inst + tdn.inst, tdn, y, smem_raw + ds.split_y);
    }
    for (int t = blockIdx.x; t < ds.n_tiles; t += step, buf = buf == 2 ? 0 : buf + 1, eb ^= 1) {
      td = tdn;
      const DiagInst* __restrict__ I = ds.inst + td.inst;
      const int n = I->n, n2 = n * n;
      const SplitGeom g = split_geom(n);
      const int nt = td.nt;
      const double2* ys = reinterpret_cast<const double2*>(smem_raw + ds.split_y + buf * ds.split_ybuf);
      short* s_exp = s_exp2[eb];
      // pass 1: the tile (in flight since the last one) has landed
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
      bar_sync<kBarX, kSplitX>();
      {  // two threads: a row of A, that is a row or a column of one component of an ADO
        static_assert(kSplitX >= 256, "two threads for each of 128 rows");
        const int row = tid >> 1;
        unsigned int top = 0u, any = 0u;
        if (row < nt * 4 * n) {
          const float r_n = 1.0f / n;
          const int q = small_div(row, r_n), lt = q >> 2, x = row - q * n;
          const double* src = reinterpret_cast<const double*>(ys + lt * n2) + (q & 1);
          const int ld = q & 2 ? n : 1, at = q & 2 ? x : x * n;
          int c = x + (tid & 1);  // rows start at different columns: fewer bank conflicts
          if (c >= n) c -= n;
#pragma unroll 4
          for (int i = 0; i < (n + 1) >> 1; ++i) {
            const double v = src[2 * (at + c * ld)];
            top = max(top, static_cast<unsigned int>(__double2hiint(v)) & 0x7fffffffu);
            any |= static_cast<unsigned int>(__double2loint(v));
            c += 2;
            if (c >= n) c -= n;
          }
        }
        top = max(top, __shfl_xor_sync(0xffffffffu, top, 1));
        any |= __shfl_xor_sync(0xffffffffu, any, 1);
        const int ex = static_cast<int>(top >> 20);
        if ((tid & 1) == 0 && row < 128)
          s_exp[row] = static_cast<short>((top | any) == 0u ? 0 : ex < kRowMin || ex > kRowMax ? kRowOut : ex);
      }
      const int n8 = (n + 7) & ~7;
      if (td.inst != b_inst) {  // H's digits, and the K padding of A
        const int nb = static_cast<int>(split_b_bytes(n) / 16);
        for (int i = tid; i < nb; i += kSplitX) reinterpret_cast<uint4*>(Bs)[i] = __ldg(I->h_digits + i);
        if (g.kp > n8) {  // one core matrix: K is n padded to 16
          const int m = tid & 127;
          if (m < g.rows)
            for (int d = tid >> 7; d < kDigits; d += kSplitX / 128)
              *reinterpret_cast<uint4*>(As + d * g.dstride + (m >> 3) * g.sbo + (n8 >> 3) * 128 + (m & 7) * 16) =
                  make_uint4(0u, 0u, 0u, 0u);
        }
        b_inst = td.inst;
      }
      bar_sync<kBarX, kSplitX>();
      // pass 2: four neighbours in K of a row of A per thread
      {
        const int rows = 4 * n, per = rows * (n8 >> 2);
        const float r_per = 1.0f / per, r_rows = 1.0f / rows, r_n = 1.0f / n;
        for (int q = tid; q < nt * per; q += kSplitX) {
          const int lt = small_div(q, r_per), r = q - lt * per, k4 = small_div(r, r_rows), row = r - k4 * rows;
          const int m = lt * rows + row, part = small_div(row, r_n), x = row - part * n;
          const double* src = reinterpret_cast<const double*>(ys + lt * n2) + (part & 1);
          const int ld = part & 2 ? n : 1, at = part & 2 ? x : x * n;
          const int es = min(static_cast<int>(s_exp[m]), 2047);
          Fixed v[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int k = 4 * k4 + j;
            v[j] = to_fixed(k < n ? src[2 * (at + k * ld)] : 0.0, es);
          }
          const uint32_t s0 = v[0].sign | (v[1].sign << 16), s1 = v[2].sign | (v[3].sign << 16);
          unsigned char* to = As + (m >> 3) * g.sbo + (k4 >> 1) * 128 + (m & 7) * 16 + (k4 & 1) * 8;
#pragma unroll
          for (int d = 0; d < kDigits; ++d) {
            const int w = kDigits - 1 - d;
            auto dig = [&](const Fixed& f) { return w > 3 ? digit(f.hi, w - 4) : digit(f.lo, w); };
            *reinterpret_cast<uint2*>(to + d * g.dstride) =
                make_uint2(digit_pair(dig(v[0]), dig(v[1])) ^ s0, digit_pair(dig(v[2]), dig(v[3])) ^ s1);
          }
        }
      }
      fence_async();
      fence_before();
      bar_sync<kBarX, kSplitX>();
      fence_after();
      // pass 3
      if (warp == 0) {
        if (elect_one()) {
          const uint32_t a0 = s_addr(As), b0 = s_addr(Bs);
          for (int d = 0; d < kDigits; ++d) {
            const int nn = (kDigits - d) * g.np;
            // D FP32, A and B FP16, both K-major, M = 128
            const uint32_t idesc = (1u << 4) | (static_cast<uint32_t>(nn >> 3) << 17) | (8u << 24);
            for (int s = 0; s < g.kp / 16; ++s)
              g_mma(tmem + d * g.np, g_desc(a0 + d * g.dstride + s * 256, 128, g.sbo), g_desc(b0 + s * 256, 128, g.sbo),
                    idesc, d > 0 || s > 0 ? 1 : 0);
          }
          g_commit(&mbar);
        }
        __syncwarp();
      }
      if (!g_wait(&mbar, parity)) s_fail = t + 1;  // the tensor-core wait gave up
      parity ^= 1u;
      if (t != blockIdx.x) bar_sync<kBarFree, kSplitThreads>();  // the second group has read the last products
      // the second group is past the tile before the last one, whose buffer takes the next input
      const int nb = buf == 2 ? 0 : buf + 1;
      bar_sync<kBarX, kSplitX>();
      if (s_fail == t + 1) {
        bar_arrive<kBarFull, kSplitThreads>();  // the second group leaves too
        g_wait(&mbar, parity ^ 1u);             // what is in flight drains (bounded) before the tensor memory goes
        break;
      }
      fence_after();
      if (t + step < ds.n_tiles) {
        tdn = ds.tiles[t + step];
        split_stage(ds.inst + tdn.inst, tdn, y, smem_raw + ds.split_y + nb * ds.split_ybuf);
      }
      // pass 4: warp w reads the lanes of sub-partition w % 4, in blocks of four columns
      if ((warp & 3) * 32 < nt * 4 * n) {
        const int m = (warp & 3) * 32 + lane;
        // products of a row that the digits do not hold are not used
        const int er = m < nt * 4 * n ? min(static_cast<int>(s_exp[m]), kRowMax) - 1022 - 77 : 0;
        for (int cb = warp >> 2; 4 * cb < n; cb += kSplitX / 128) {
          uint32_t f[kDigits][4];
#pragma unroll
          for (int d = 0; d < kDigits; ++d)
            ld4_issue(tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + static_cast<uint32_t>(d * g.np + cb * 4), f[d]);
          asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (m >= nt * 4 * n || cb * 4 + j >= n) continue;
            int o[kDigits];
#pragma unroll
            for (int d = 0; d < kDigits; ++d) o[d] = __float2int_rn(__uint_as_float(f[d][j]));
            P[m * (n + 1) + cb * 4 + j] = from_orders(o, er + max(__ldg(I->h_exp + cb * 4 + j), -100));
          }
        }
      }
      fence_before();
      bar_arrive<kBarFull, kSplitThreads>();
    }
  } else {
    // ---------------------------------------------------------------- second group: passes 5 to 7
    const int ty = tid - kSplitX;
    int buf = 0, eb = 0;
    for (int t = blockIdx.x; t < ds.n_tiles; t += step, buf = buf == 2 ? 0 : buf + 1, eb ^= 1) {
      const DiagTile td = ds.tiles[t];
      const DiagInst* __restrict__ I = ds.inst + td.inst;
      const int n = I->n, n2 = n * n, K = I->K, w = I->site_w, w1 = 1 + w, void_idx = I->nh, tile = I->tile;
      const int l0 = td.l0, nt = td.nt, ne = nt * n2;
      const double2* __restrict__ yi = y + I->elem_off;
      double2* ys = reinterpret_cast<double2*>(smem_raw + ds.split_y + buf * ds.split_ybuf);
      const int4* rec = reinterpret_cast<const int4*>(ys + static_cast<size_t>(tile) * n2);
      const float r_n2 = 1.0f / n2, r_n = 1.0f / n;
      const short* s_exp = s_exp2[eb];
      bar_sync<kBarFull, kSplitThreads>();
      if (s_fail == t + 1) break;  // a later tile's failure does not concern this one
      // pass 5
      const bool sqn = I->sqrt_norm != 0;
      const size_t g0 = static_cast<size_t>(I->elem_off) + static_cast<size_t>(l0) * n2;
      // the neighbour value of the thread's first -1 term is in flight during pass 5
      // task q of pass 6: mode m of ADO lt (the q-th of w * 2 n places), element e; -1: none
      const float r_task = 1.0f / (w * 2 * n);
      auto task = [&](int q, int& lt, int& m) {
        lt = small_div(q, r_task);
        const int r = q - lt * (w * 2 * n);
        m = small_div(r, 0.5f * r_n);
        const int4* rl = rec + lt * w1;
        if (lt >= nt || m >= rl->x) return -1;
        const int j = r - m * 2 * n, s = rl[1 + m].w, a = j < n ? s : j - n, b = j < n ? j : s;
        if (j >= n && a == s) return -1;
        for (int p = 0; p < m; ++p)
          if (rl[1 + p].w == a || rl[1 + p].w == b) return -1;
        return a * n + b;
      };
      auto minus_coef = [&](const int4& r, int a, int b) {
        return __ldg(I->site_cmn_d + (3 * r.x + (r.w == a ? (r.w == b ? 2 : 0) : 1)) * I->occ_rows + r.z);
      };
      int lt_q = 0, m_q = 0;
      const int e_q = task(ty, lt_q, m_q);
      double2 v_q = make_double2(0.0, 0.0);
      if (e_q >= 0) v_q = __ldg(yi + static_cast<size_t>(rec[lt_q * w1 + 1 + m_q].y) * n2 + e_q);
      for (int ib = ty - lane; ib < ne; ib += kSplitY) {
        const int i = min(ib + lane, ne - 1);
        const int lt = small_div(i, r_n2), e = i - lt * n2, a = small_div(e, r_n), b = e - a * n, l = l0 + lt;
        double2 acc;
        bool ok;
        {
          const int r0 = lt * 4 * n, ra = r0 + a, rb = r0 + 2 * n + b;
          const double x2 = P[rb * (n + 1) + a], x1 = P[ra * (n + 1) + b];
          const double y2 = P[(rb + n) * (n + 1) + a], y1 = P[(ra + n) * (n + 1) + b];
          acc = make_double2(x2 - x1, y2 - y1);
          const int ha = __ldg(I->h_exp + a), hb = __ldg(I->h_exp + b);
          auto scale = [](int f) { return f == 0 ? kNoColumn : f == kRowOut ? 50000 : f - 1022; };
          auto trusted = [&](double p2, double p1, int f2, int f1) {
            const unsigned int top = max(static_cast<unsigned int>(__double2hiint(p2)) & 0x7fffffffu,
                                         static_cast<unsigned int>(__double2hiint(p1)) & 0x7fffffffu);
            return static_cast<int>(top >> 20) - 1023 + kTrust >= max(scale(f2) + ha, scale(f1) + hb);
          };
          ok = trusted(x2, x1, s_exp[rb], s_exp[ra]) && trusted(y2, y1, s_exp[rb + n], s_exp[ra + n]);
        }
        // FP64 sums of the others: lane by lane where there are many, else the warp on one after another
        unsigned int rest = __ballot_sync(0xffffffffu, !ok && ib + lane < ne);
        if (__popc(rest) * 4 > n) {
          if (!ok) {
            acc = make_double2(0.0, 0.0);
            const double2* __restrict__ yl = yi + static_cast<size_t>(l) * n2;  // ys is being replaced
            for (int c = 0; c < n; ++c) {
              const double hac = I->H[a * n + c].x, hcb = I->H[c * n + b].x;
              const double2 ycb = __ldg(yl + c * n + b), yac = __ldg(yl + a * n + c);
              acc.x = fma(hac, ycb.x, acc.x);
              acc.x = fma(-hcb, yac.x, acc.x);
              acc.y = fma(hac, ycb.y, acc.y);
              acc.y = fma(-hcb, yac.y, acc.y);
            }
          }
        } else {
          for (; rest; rest &= rest - 1) {
            const int j = __ffs(rest) - 1, lj = small_div(ib + j, r_n2), ej = ib + j - lj * n2, aj = small_div(ej, r_n),
                      bj = ej - aj * n;
            double2 v = make_double2(0.0, 0.0);
            if (lane < n) {
              const double2* __restrict__ yl = yi + static_cast<size_t>(l0 + lj) * n2;
              const double hac = I->H[aj * n + lane].x, hcb = I->H[lane * n + bj].x;
              const double2 ycb = __ldg(yl + lane * n + bj), yac = __ldg(yl + aj * n + lane);
              v.x = fma(-hcb, yac.x, hac * ycb.x);
              v.y = fma(-hcb, yac.y, hac * ycb.y);
            }
            for (int o = 16; o > 0; o >>= 1) {
              v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
              v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
            }
            if (lane == j) acc = v;
          }
        }
        if (ib + lane >= ne) continue;
        double2 D = make_double2(-acc.y, acc.x);
        // damping
        const double2 d0 = __ldg(I->ngd + l), d1 = __ldg(I->c_sd + e), yv = ys[i];
        cfma(D, make_double2(d0.x + d1.x, d0.y + d1.y), yv);
        if (rec[lt * w1].y && a != b) {  // +1 terms, the two sites' modes in increasing k
          const int* p1r = I->p1 + static_cast<size_t>(l) * K;
          int pa = __ldg(I->site_ptr + a), pb = __ldg(I->site_ptr + b);
          const int pa1 = __ldg(I->site_ptr + a + 1), pb1 = __ldg(I->site_ptr + b + 1);
          while (pa < pa1 || pb < pb1) {
            const int ka = pa < pa1 ? __ldg(I->site_modes + pa) : 0x7fffffff;
            const int kb = pb < pb1 ? __ldg(I->site_modes + pb) : 0x7fffffff;
            const bool row = ka < kb;
            const int k = row ? ka : kb;
            pa += row ? 1 : 0;
            pb += row ? 0 : 1;
            const int lp = __ldg(p1r + k);
            double2 c = __ldg(I->site_cp2_d + 2 * k + (row ? 0 : 1));
            if (lp != void_idx && (nonzero_bits(c.x) || nonzero_bits(c.y))) {
              if (sqn) {
                const double f = sqrt(static_cast<double>(__ldg(I->nidx + static_cast<size_t>(l) * K + k) + 1));
                c = make_double2(f * c.x, f * c.y);
              }
              cfma(D, c, __ldg(yi + static_cast<size_t>(lp) * n2 + e));
            }
          }
        }
        ys[i] = D;  // the element's input is spent
      }
      bar_sync<kBarY, kSplitY>();
      if (t + step < ds.n_tiles) bar_arrive<kBarFree, kSplitThreads>();  // the products are read
      // pass 6: the -1 terms of the occupied modes.  A mode touches 2 n - 1 elements of its ADO;
      // the thread of an element's first mode adds the terms of all
      for (int q = ty; q < nt * w * 2 * n; q += kSplitY) {
        int lt = lt_q, m = m_q, e = e_q;
        double2 v = v_q;
        if (q != ty) {
          e = task(q, lt, m);
          if (e >= 0) v = __ldg(yi + static_cast<size_t>(rec[lt * w1 + 1 + m].y) * n2 + e);
        }
        if (e < 0) continue;
        const int4* rl = rec + lt * w1;
        const int a = small_div(e, r_n), b = e - a * n, nm = rl->x;
        double2 D = ys[lt * n2 + e];
        for (int p = m; p < nm; ++p) {
          const int4 r = rl[1 + p];  // k, ptr_m1, n_k, site
          if (r.w == a || r.w == b) {
            const double2 c = minus_coef(r, a, b);
            if (p > m) v = __ldg(yi + static_cast<size_t>(r.y) * n2 + e);
            if (nonzero_bits(c.x) || nonzero_bits(c.y)) cfma(D, c, v);
          }
        }
        ys[lt * n2 + e] = D;
      }
      bar_sync<kBarY, kSplitY>();
      // pass 7: stage epilogue
      for (int i = ty; i < ne; i += kSplitY) {
        const EpiPre p = epi_pre<double, KIND>(st, g0 + i, cur);
        local += epi_post<double, KIND>(st, g0 + i, ys[i], dt, cur, p);
      }
    }
  }
  fence_before();
  __syncthreads();
  fence_after();
  if (s_fail && tid == 0 && st.ctl) st.ctl->status = 2;
  if (warp == 0) tmem_free(tmem, kSplitCols);
  if (KIND == EPI_DP7) dp7_finish(st, local, ds.total);
}

using SplitKernel = void (*)(const DiagSet, const Stage);
SplitKernel split_kernel(int kind) {
  switch (kind) {
    case EPI_RK4_1: return k_rhs_split<EPI_RK4_1>;
    case EPI_RK4_2: return k_rhs_split<EPI_RK4_2>;
    case EPI_RK4_3: return k_rhs_split<EPI_RK4_3>;
    case EPI_RK4_4: return k_rhs_split<EPI_RK4_4>;
    case EPI_LS: return k_rhs_split<EPI_LS>;
    case EPI_DP: return k_rhs_split<EPI_DP>;
    case EPI_DP7: return k_rhs_split<EPI_DP7>;
    default: return nullptr;  // calc_diff keeps k_rhs_diag
  }
}

}  // namespace

std::vector<unsigned short> split_h_digits(const double* H, int n, std::vector<int>& exponent) {
  std::vector<double> top(n, 0.0);
  double all = 0.0;
  for (int i = 0; i < n * n; ++i) {
    if (!std::isfinite(H[i])) return {};
    top[i % n] = std::max(top[i % n], std::fabs(H[i]));
    all = std::max(all, std::fabs(H[i]));
  }
  int eh = 0;
  if (all > 0.0) std::frexp(all, &eh);  // all < 2^eh
  if (eh < -100 || eh > 100) return {};
  exponent.assign(n, kNoColumn);
  for (int b = 0; b < n; ++b)
    if (top[b] > 0.0) {
      std::frexp(top[b], &exponent[b]);
      exponent[b] = std::max(exponent[b], -100);
    }
  const SplitGeom g = split_geom(n);
  std::vector<unsigned short> out(split_b_bytes(n) / 2, 0);
  for (int b = 0; b < n; ++b)
    for (int c = 0; c < n; ++c) {
      // |H| truncated to 70 bits below the column's power of two, as to_fixed does
      int ex = 0;
      const double frac = std::frexp(std::fabs(H[c * n + b]), &ex);
      if (frac == 0.0) continue;
      const unsigned long long man = static_cast<unsigned long long>(std::ldexp(frac, 53));
      const int sh = 17 + ex - exponent[b];  // at most 17
      unsigned long long hi = 0, lo = 0;
      if (sh > 0) {
        hi = man >> (36 - sh);
        lo = (man << sh) & kLow;
      } else if (sh > -53) {
        hi = (man >> -sh) >> 36;
        lo = (man >> -sh) & kLow;
      }
      lo += kBias;
      hi += kBias + (lo >> 36);
      for (int d = 0; d < kDigits; ++d) {
        const int w = kDigits - 1 - d;
        int dig = static_cast<int>((w > 3 ? hi >> (kBits * (w - 4)) : lo >> (kBits * w)) & 0x1ff) - 256;
        if (H[c * n + b] < 0.0) dig = -dig;
        // the digit's FP16 bits: sign, exponent, ten fraction bits
        unsigned short h = 0;
        if (dig != 0) {
          const int mag = dig < 0 ? -dig : dig;
          int p = 0;
          while ((mag >> (p + 1)) != 0) ++p;
          h = static_cast<unsigned short>((dig < 0 ? 0x8000 : 0) | ((p + 15) << 10) | ((mag << (10 - p)) & 0x3ff));
        }
        const int row = d * g.np + b;
        out[(static_cast<size_t>(row >> 3) * g.sbo + (c >> 3) * 128 + (row & 7) * 16 + (c & 7) * 2) / 2] = h;
      }
    }
  return out;
}

bool split_eligible(const DiagInst& I, bool mixed) {
  return !mixed && I.site_local && I.site_rec && I.h_digits && I.h_sym && I.n >= 4 && I.n <= 32 && !I.term_p &&
         I.max_terms <= 4;
}

// Where the kernel beats k_rhs_diag<double>: the commutator's share of an element
// grows with n, and a tile's chain of passes has to be hidden behind other tiles.
// Measured, us a stage of k_rhs_diag<double> and of this, LSRK4 (RK4 alike): 8
// levels, 310k elements 47 and 49; 10, 23k 10 and 17, 177k 34 and 26; 12, 47k 19 and 18
// (Dormand-Prince 25 and 26), 421k 73 and 45; 13, 64k 19 and 19; 16, 144k 35 and 24; 24, 28k
// 32 and 26, 12M 2944 and 783; 32, 67k 55 and 37.
bool split_pays(const std::vector<DiagInst>& insts) {
  long long elems = 0, work = 0;
  int n = 32;
  for (const DiagInst& I : insts) {
    const long long e = static_cast<long long>(I.n2) * I.nh;
    elems += e;
    work += e * I.n;
    n = std::min(n, I.n);
  }
  return n >= 10 && elems >= 25000 && work >= (n >= 16 ? 600000 : 1500000);
}

int split_tile(int n) { return split_geom(n).tile; }

void split_smem(const DiagInst& I, size_t* a, size_t* p, size_t* b, size_t* y) {
  *a = split_a_bytes(I.n);
  *p = split_p_bytes(I.n);
  *b = split_b_bytes(I.n);
  *y = split_y_bytes(I.n, I.site_w);
}

int split_threads() { return kSplitThreads; }

cudaError_t launch_split(const DiagSet& ds, const Stage& st, int grid, cudaStream_t s) {
  SplitKernel kern = split_kernel(st.kind);
  if (!kern) return cudaErrorInvalidValue;
  cudaError_t e = allow_smem(reinterpret_cast<const void*>(kern));
  if (e != cudaSuccess) return e;
  kern<<<grid, kSplitThreads, ds.smem, s>>>(ds, st);
  ++g_launches;
  return cudaGetLastError();
}

}  // namespace heomgb
