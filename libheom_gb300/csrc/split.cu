// FP64 stage kernel with the commutator on the tensor cores: site-local baths,
// real symmetric H, 4 to 32 levels.  Same operator and stage epilogues as
// k_rhs_diag<double> (heom_hilb.h:96-215 with the fused rk4 / lsrk4 / rkdp
// stages).
//
// The FP64 pipe executes two operations per clock per SM, and 4 n of an
// element's operations are the commutator.  Here rho and H are cut into seven
// signed digits of nine bits each (fixed point, 62 bits below the largest
// element of the ADO, or of H); the digits are integers of at most 256, exact
// in FP16, and a product of two digit matrices summed over n <= 32 and over
// the seven pairs of one order i + j stays below 2^24, so the FP32
// accumulators of the tensor cores hold it exactly.  The orders 0 to 6 are
// combined with integer operations and rounded to FP64 once per value; what is
// left out (orders above 6 and bits of rho below 2^-62 of the ADO's largest)
// is below 2^-57 of the largest product (the error-free splitting of matrix
// products of Ozaki, Ogita, Oishi and Rump, Numer. Algorithms 59, 2012).
// Measured on the 24-site aggregate at depth 3: a state's error against
// extended precision is 7.0e-17 after 4 steps, 7.6e-17 with the FP64 sums; a
// stage of 12M elements takes 1.22 ms, 2.95 with k_rhs_diag<double>, whose FP64
// pipe alone needs 2.58.
//
// Per tile of T = 128 / (4 n) ADOs:
//   1. the stage input to shared memory, each ADO's largest exponent;
//   2. digits of R, I, R^T and I^T (rho = R + iI; rows 4 n per ADO, K = n
//      padded to 16) into the A operand, K-major without swizzle;
//   3. MMAs (M = 128, one thread): digit i of rho against the digits 0..6-i of
//      H at once (N = 7 - i blocks of n padded to 16), into the tensor-memory
//      columns of the orders i..6, so 7 MMAs per 16 of K cover all 28 pairs;
//   4. read-back: rows of R H, I H (rho H) and R^T H, I^T H (H rho,
//      transposed) as 128-bit integers in shared memory, over the A operand;
//   5. one element per thread: the difference of the two products in integers,
//      one rounding to FP64 (three FP64 additions per component), damping,
//      bath terms, stage epilogue.
// An ADO with elements beyond 2^900, infinities or NaNs takes FP64 sums in
// pass 5.  Two CTAs per SM overlap each other's passes.
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

constexpr int kDigits = 7, kBits = 9;
constexpr int kSplitThreads = 320;
constexpr int kSplitCols = 256;  // tensor-memory columns of a CTA: seven orders of at most 32
// the digits' bias: sum of 256 * 2^(9 k)
constexpr unsigned long long kBias = 0x4020100804020100ull;

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
// the A operand (the last digit's MMA reads 128 rows), later the products
__host__ __device__ __forceinline__ size_t split_a_bytes(int n) {
  const SplitGeom g = split_geom(n);
  const size_t a = static_cast<size_t>(kDigits - 1) * g.dstride + 16 * static_cast<size_t>(g.sbo);
  const size_t p = static_cast<size_t>(g.rows) * (n + 1) * 16;
  return ((a > p ? a : p) + 127) & ~size_t(127);
}
__host__ __device__ __forceinline__ size_t split_b_bytes(int n) {
  const SplitGeom g = split_geom(n);
  return static_cast<size_t>(kDigits) * g.np / 8 * g.sbo;
}
__host__ __device__ __forceinline__ size_t split_y_bytes(int n, int w) {
  const SplitGeom g = split_geom(n);
  return static_cast<size_t>(g.tile) * (n * n * sizeof(double2) + (1 + w) * sizeof(int4));
}

// |x| as a 62-bit fixed-point number below 2^61 at the scale of exponent es
// (es >= the exponent field of x), with its sign
__device__ __forceinline__ long long to_fixed(double x, int es) {
  const unsigned long long u = static_cast<unsigned long long>(__double_as_longlong(x));
  const int hi = static_cast<int>(u >> 32), ex = (hi >> 20) & 0x7ff;
  const unsigned long long man = ex ? ((u & 0xfffffffffffffull) | (1ull << 52)) << 8 : 0ull;
  const long long v = static_cast<long long>(man >> min(es - ex, 63));
  const long long s = static_cast<long long>(hi >> 31);
  return (v ^ s) - s;
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

// the eight columns of one order at taddr, without the wait
__device__ __forceinline__ void ld8_issue(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}

template <int KIND>
__global__ void __launch_bounds__(kSplitThreads, 2) k_rhs_split(const DiagSet ds, const Stage st) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t mbar;
  __shared__ uint32_t tslot;
  __shared__ unsigned int s_max[8];
  double dt;
  int cur;
  // one verdict per CTA (k_rhs_diag_tc)
  if (!__syncthreads_and(stage_prologue<KIND>(st, dt, cur))) return;
  const double2* __restrict__ y = stage_input<double2>(st, cur);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned char* As = smem_raw;
  longlong2* P = reinterpret_cast<longlong2*>(smem_raw);
  unsigned char* Bs = smem_raw + ds.split_b;
  if (warp == 0) tmem_alloc(&tslot, kSplitCols);
  if (tid == 0) {
    mbar_init(&mbar);
    mbar_init_fence();
  }
  if (tid < 8) s_max[tid] = 0u;
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = tslot;
  uint32_t parity = 0;
  int b_inst = -1;
  bool fail = false;
  double local = 0.0;
  for (int t = blockIdx.x; t < ds.n_tiles; t += gridDim.x) {
    const DiagTile td = ds.tiles[t];
    const DiagInst* __restrict__ I = ds.inst + td.inst;
    const int n = I->n, n2 = n * n, K = I->K, w1 = 1 + I->site_w, void_idx = I->nh;
    const SplitGeom g = split_geom(n);
    const int l0 = td.l0, nt = td.nt, ne = nt * n2;
    const double2* __restrict__ yi = y + I->elem_off;
    double2* ys = reinterpret_cast<double2*>(smem_raw + ds.split_y);
    int4* rec = reinterpret_cast<int4*>(ys + static_cast<size_t>(g.tile) * n2);
    // pass 1
    const double2* ysrc = yi + static_cast<size_t>(l0) * n2;
    for (int i = tid; i < ne; i += kSplitThreads) ys[i] = __ldg(ysrc + i);
    for (int i = tid; i < nt * w1; i += kSplitThreads) rec[i] = __ldg(I->site_rec + static_cast<size_t>(l0) * w1 + i);
    if (td.inst != b_inst) {
      const int nb = static_cast<int>(split_b_bytes(n) / 16);
      for (int i = tid; i < nb; i += kSplitThreads) reinterpret_cast<uint4*>(Bs)[i] = __ldg(I->h_digits + i);
      b_inst = td.inst;
    }
    const int n8 = (n + 7) & ~7, cores = (g.kp - n8) >> 3;  // whole core matrices of K padding
    for (int q = tid; q < kDigits * nt * 4 * n * cores; q += kSplitThreads) {
      const int m = q % (nt * 4 * n), r = q / (nt * 4 * n), c = r % cores, d = r / cores;
      *reinterpret_cast<uint4*>(As + d * g.dstride + (m >> 3) * g.sbo + ((n8 >> 3) + c) * 128 + (m & 7) * 16) =
          make_uint4(0u, 0u, 0u, 0u);
    }
    __syncthreads();
    for (int lt = 0; lt < nt; ++lt) {
      unsigned int top = 0u;
      for (int e = tid; e < n2; e += kSplitThreads) {
        const double2 v = ys[lt * n2 + e];
        top = max(top, max(static_cast<unsigned int>(__double2hiint(v.x)) & 0x7fffffffu,
                                 static_cast<unsigned int>(__double2hiint(v.y)) & 0x7fffffffu));
      }
      top = __reduce_max_sync(0xffffffffu, top);
      if (lane == 0) atomicMax(&s_max[lt], top);
    }
    __syncthreads();
    // pass 2: 2 x 2 blocks of one component, 16 of them an 8 x 8 block
    {
      const int nb8 = n8 >> 3, per = 2 * nb8 * nb8 * 16;
      for (int q = tid; q < nt * per; q += kSplitThreads) {
        const int lt = q / per, r = q - lt * per, s16 = r & 15, sb = r >> 4;
        const int comp = sb & 1, b8 = sb >> 1, A8 = b8 / nb8, C8 = b8 - A8 * nb8;
        const int a = A8 * 8 + (s16 >> 2) * 2, c = C8 * 8 + (s16 & 3) * 2;
        if (a >= n && c >= n) continue;
        const int es = max(static_cast<int>(s_max[lt] >> 20), 223);
        const double* src = reinterpret_cast<const double*>(ys + lt * n2) + comp;
        unsigned long long v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int aj = a + (j >> 1), cj = c + (j & 1);
          const double x = aj < n && cj < n ? src[2 * (aj * n + cj)] : 0.0;
          v[j] = static_cast<unsigned long long>(to_fixed(x, es)) + kBias;
        }
        const int m = lt * 4 * n + comp * n, mt = m + 2 * n;
        auto at = [&](int row, int k) { return As + (row >> 3) * g.sbo + (k >> 3) * 128 + (row & 7) * 16 + (k & 7) * 2; };
        unsigned char *r0 = at(m + a, c), *r1 = at(m + a + 1, c), *t0 = at(mt + c, a), *t1 = at(mt + c + 1, a);
#pragma unroll
        for (int d = 0; d < kDigits; ++d) {
          const int k = kDigits - 1 - d;
          const uint32_t h0 = digit_pair(digit(v[0], k), digit(v[1], k)), h1 = digit_pair(digit(v[2], k), digit(v[3], k));
          const int o = d * g.dstride;
          if (a < n) *reinterpret_cast<uint32_t*>(r0 + o) = h0;
          if (a + 1 < n) *reinterpret_cast<uint32_t*>(r1 + o) = h1;
          if (c < n) *reinterpret_cast<uint32_t*>(t0 + o) = __byte_perm(h0, h1, 0x5410);
          if (c + 1 < n) *reinterpret_cast<uint32_t*>(t1 + o) = __byte_perm(h0, h1, 0x7632);
        }
      }
    }
    fence_async();
    fence_before();
    __syncthreads();
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
    const uint32_t done = g_wait(&mbar, parity);
    parity ^= 1u;
    if (!__syncthreads_and(done)) {
      if (tid == 0 && st.ctl) st.ctl->status = 2;  // tensor-core wait gave up
      fail = true;
      break;
    }
    fence_after();
    // pass 4: warps w and w + 4 read the lanes of sub-partition w, every other block of eight columns
    if (warp < 8 && (warp & 3) * 32 < nt * 4 * n) {
      const int m = (warp & 3) * 32 + lane;
      for (int cb = warp >> 2; cb < n8 >> 3; cb += 2) {
        uint32_t f[kDigits][8];
#pragma unroll
        for (int d = 0; d < kDigits; ++d)
          ld8_issue(tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + static_cast<uint32_t>(d * g.np + cb * 8), f[d]);
        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          long long o[kDigits];
#pragma unroll
          for (int d = 0; d < kDigits; ++d) o[d] = __float2int_rn(__uint_as_float(f[d][j]));
          const long long hi = (o[0] << 18) + (o[1] << 9) + o[2];
          const long long lo = (o[3] << 27) + (o[4] << 18) + (o[5] << 9) + o[6];
          if (m < nt * 4 * n && cb * 8 + j < n) P[m * (n + 1) + cb * 8 + j] = make_longlong2(hi, lo);
        }
      }
    }
    fence_before();
    __syncthreads();
    // pass 5
    const bool sqn = I->sqrt_norm != 0;
    const size_t g0 = static_cast<size_t>(I->elem_off) + static_cast<size_t>(l0) * n2;
    const float r_n2 = 1.0f / n2, r_n = 1.0f / n;
    for (int i = tid; i < ne; i += kSplitThreads) {
      const int lt = small_div(i, r_n2), e = i - lt * n2, a = small_div(e, r_n), b = e - a * n, l = l0 + lt;
      const EpiPre pre = epi_pre<double, KIND>(st, g0 + i, cur);
      const int ex = static_cast<int>(s_max[lt] >> 20), es = max(ex, 223);
      double2 acc;
      if (ex <= 1922) {
        const longlong2* Pl = P + lt * 4 * n * (n + 1);
        const longlong2 rx = Pl[a * (n + 1) + b], ry = Pl[(n + a) * (n + 1) + b];
        const longlong2 tx = Pl[(2 * n + b) * (n + 1) + a], ty = Pl[(3 * n + b) * (n + 1) + a];
        // units of lo: 2^u; a 64-bit integer v with |v| < 2^51 times 2^u is (1.5 2^(52+u) + v 2^u) - 1.5 2^(52+u)
        const int u = es - 1022 + I->h_exp - 68;
        const long long ml = (static_cast<long long>(1075 + u) << 52) | (1ll << 51);
        const long long mh = ml + (36ll << 52);
        const double cl = __longlong_as_double(ml), ch = __longlong_as_double(mh);
        acc.x = (__longlong_as_double(mh + (tx.x - rx.x)) - ch) + (__longlong_as_double(ml + (tx.y - rx.y)) - cl);
        acc.y = (__longlong_as_double(mh + (ty.x - ry.x)) - ch) + (__longlong_as_double(ml + (ty.y - ry.y)) - cl);
      } else {  // out of the fixed-point range
        acc = make_double2(0.0, 0.0);
        const double2* yl = ys + lt * n2;
        for (int c = 0; c < n; ++c) {
          const double hac = I->H[a * n + c].x, hcb = I->H[c * n + b].x;
          const double2 ycb = yl[c * n + b], yac = yl[a * n + c];
          acc.x = fma(hac, ycb.x, acc.x);
          acc.x = fma(-hcb, yac.x, acc.x);
          acc.y = fma(hac, ycb.y, acc.y);
          acc.y = fma(-hcb, yac.y, acc.y);
        }
      }
      double2 D = make_double2(-acc.y, acc.x);
      const double2 d0 = __ldg(I->ngd + l), d1 = __ldg(I->c_sd + e);
      cfma(D, make_double2(d0.x + d1.x, d0.y + d1.y), ys[i]);
      const int4* rl = rec + lt * w1;
      const int4 hdr = *rl;
      if (hdr.y && a != b) {  // +1 terms, the two sites' modes in increasing k
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
          if (lp != void_idx && (c.x != 0.0 || c.y != 0.0)) {
            if (sqn) {
              const double f = sqrt(static_cast<double>(__ldg(I->nidx + static_cast<size_t>(l) * K + k) + 1));
              c = make_double2(f * c.x, f * c.y);
            }
            cfma(D, c, __ldg(yi + static_cast<size_t>(lp) * n2 + e));
          }
        }
      }
      for (int q = 1; q <= hdr.x; ++q) {  // -1 terms: the ADO's occupied modes
        const int4 r = rl[q];              // k, ptr_m1, n_k, site
        if (r.w == a || r.w == b) {
          const double2 c = __ldg(I->site_cm3_d + 3 * r.x + (r.w == a ? (r.w == b ? 2 : 0) : 1));
          if (c.x != 0.0 || c.y != 0.0) {
            const double f = sqn ? sqrt(static_cast<double>(r.z)) : occ<double>(r.z);
            cfma(D, make_double2(f * c.x, f * c.y), __ldg(yi + static_cast<size_t>(r.y) * n2 + e));
          }
        }
      }
      local += epi_post<double, KIND>(st, g0 + i, D, dt, cur, pre);
    }
    __syncthreads();  // the products, the input and the maxima are free
    if (tid < 8) s_max[tid] = 0u;
  }
  if (fail) {
    g_wait(&mbar, parity ^ 1u);  // what is in flight drains (bounded) before the tensor memory goes
    __syncthreads();
  }
  fence_before();
  __syncthreads();
  fence_after();
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

std::vector<unsigned short> split_h_digits(const double* H, int n, int* exponent) {
  double top = 0.0;
  for (int i = 0; i < n * n; ++i) {
    if (!std::isfinite(H[i])) return {};
    top = std::max(top, std::fabs(H[i]));
  }
  int eh = 0;
  if (top > 0.0) std::frexp(top, &eh);  // top < 2^eh
  if (eh < -100 || eh > 100) return {};
  *exponent = eh;
  const SplitGeom g = split_geom(n);
  std::vector<unsigned short> out(split_b_bytes(n) / 2, 0);
  for (int b = 0; b < n; ++b)
    for (int c = 0; c < n; ++c) {
      unsigned long long v =
          static_cast<unsigned long long>(static_cast<long long>(std::ldexp(H[c * n + b], 61 - eh))) + kBias;
      for (int d = 0; d < kDigits; ++d) {
        const int dig = static_cast<int>((v >> (kBits * (kDigits - 1 - d))) & 0x1ff) - 256;
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

int split_tile(int n) { return split_geom(n).tile; }

void split_smem(const DiagInst& I, size_t* a, size_t* b, size_t* y) {
  *a = split_a_bytes(I.n);
  *b = split_b_bytes(I.n);
  *y = split_y_bytes(I.n, I.site_w);
}

int split_threads() { return kSplitThreads; }

cudaError_t launch_split(const DiagSet& ds, const Stage& st, int grid, cudaStream_t s) {
  SplitKernel kern = split_kernel(st.kind);
  if (!kern) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(ds.smem));
  if (e != cudaSuccess) return e;
  kern<<<grid, kSplitThreads, ds.smem, s>>>(ds, st);
  ++g_launches;
  return cudaGetLastError();
}

}  // namespace heomgb
