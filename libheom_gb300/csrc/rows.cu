// Stage kernel for batches and mid-size models of site-local baths (every V_u
// diagonal with a single nonzero entry), at most 32 levels, real H, mixed
// form (FP32 stage input, FP64 state).  Same operator and stage epilogues as
// k_rhs_diag (heom_hilb.h:96-215 with the fused rk4 / lsrk4 / rkdp stages).
//
// A warp works for itself: it takes a group of consecutive ADOs of the CTA's
// instance (as many as their rows fill its lanes, or fewer where the model is
// small), keeps their stage input, records and right-hand sides in its part of
// shared memory, and meets the other warps only where the CTA changes its
// instance, whose tables they share.  Nothing waits on a CTA barrier, so the
// phases of the SM's warps overlap; the next group's input is copied with
// cp.async meanwhile.  Per group:
//
// 1. Commutator and damping: a lane owns one row of an ADO (up to eight levels,
//    N a template argument: the row's accumulators and every address are fixed
//    at compile time) or four columns of a row (N = 0).  Every H and rho value
//    read from shared memory feeds a whole row, with paired FP32 FMAs
//    (__ffma2_rn); H is stored with each value doubled, so that a pair is one
//    load.  The right-hand sides go to shared memory.
// 2. Bath terms: mode k (site s) touches row s and column s of an ADO, 2 n - 1
//    elements; 16 lanes (n <= 8; else 32) take an ADO's modes one after another
//    in increasing k, each lane its element of the mode's row or column in
//    shared memory (a later mode of another site reaches some of the same
//    elements through other lanes: __syncwarp between them), with the gathers
//    of four modes in flight.  First the +1 terms, on ADOs below the deepest
//    tier or with a closure, then the -1 terms of the occupied modes.
// 3. Stage epilogue, one element per lane (coalesced state accesses), two
//    elements' loads in flight.
//
// What bounds it: the instructions it issues (about 2200 a group of four 7-level
// ADOs, a third of them the bath terms) and, with 24 warps a SM, their latency;
// the state's traffic alone would take 15 us of the 48 (16 instances of 7 sites,
// depth 4, 2.4M elements; k_rhs_diag takes 74).  Measured there: CTAs of 256
// threads with barriers between the passes 58 us, one warp per group 48; four
// elements in the epilogue at a time, or eight gathers, spill: 64.
//
// Every element's arithmetic and its order are k_rhs_diag's (commutator over
// c, the damping, up to four +1 terms, up to four -1 terms; rows_eligible
// refuses more), so the two kernels give the same values.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "heomgb_impl.cuh"
#include "stage.cuh"

namespace heomgb {

namespace {

__device__ __forceinline__ uint32_t r_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
template <int BYTES>
__device__ __forceinline__ void r_cp(void* dst_smem, const void* src_gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(r_addr(dst_smem)), "l"(src_gmem), "n"(BYTES)
               : "memory");
}

// The instance's tables, shared by the CTA: H doubled (n rows of rows_ld(n)
// float2), damping differences, -1 and +1 coefficients per mode and case, the
// site of every mode.
__host__ __device__ __forceinline__ int rows_ld(int n) { return (n + 3) & ~3; }
struct RowsTab {
  float2 *H, *csd, *cm3, *cp2;
  int* msite;
};
__host__ __device__ __forceinline__ size_t rows_tab_bytes(int n, int K) {
  const size_t n2 = static_cast<size_t>(n) * n;
  return (sizeof(float2) * (n * rows_ld(n) + n2 + 5 * static_cast<size_t>(K)) + sizeof(int) * static_cast<size_t>(K) +
          15) & ~size_t(15);
}
__device__ __forceinline__ RowsTab rows_tab(unsigned char* raw, int n, int K) {
  RowsTab T;
  T.H = reinterpret_cast<float2*>(raw);
  T.csd = T.H + n * rows_ld(n);
  T.cm3 = T.csd + n * n;
  T.cp2 = T.cm3 + 3 * K;
  T.msite = reinterpret_cast<int*>(T.cp2 + 2 * K);
  return T;
}
// A warp's buffer for a group of `ados`: their records, stage input (four
// values of padding: the last row's four-column reads), ptr_p1 and occupation
// rows.
struct RowsBuf {
  int4* rec;
  float2* y;
  int *p1, *nk;
};
__host__ __device__ __forceinline__ size_t rows_buf_bytes(int n2, int K, int w, int ados) {
  return (sizeof(int4) * static_cast<size_t>(ados) * (1 + w) + sizeof(float2) * (static_cast<size_t>(ados) * n2 + 4) +
          2 * sizeof(int) * static_cast<size_t>(ados) * K + 15) & ~size_t(15);
}
__device__ __forceinline__ RowsBuf rows_layout(unsigned char* raw, int n2, int K, int w, int ados) {
  RowsBuf L;
  L.rec = reinterpret_cast<int4*>(raw);
  L.y = reinterpret_cast<float2*>(L.rec + ados * (1 + w));
  L.p1 = reinterpret_cast<int*>(L.y + ados * n2 + 4);
  L.nk = L.p1 + ados * K;
  return L;
}

// Issues the copies of a group (ADOs l0 .. l0+nt-1) into a buffer.
__device__ __forceinline__ void rows_stage(const DiagInst* __restrict__ I, const float2* __restrict__ yi, int n2,
                                           int l0, int nt, const RowsBuf& L, int lane) {
  const int K = I->K, w1 = 1 + I->site_w;
  const float2* ysrc = yi + static_cast<size_t>(l0) * n2;
#pragma unroll 1
  for (int i = lane; i < nt * n2; i += 32) r_cp<8>(L.y + i, ysrc + i);
  const int4* rsrc = I->rows_rec + static_cast<size_t>(l0) * w1;
#pragma unroll 1
  for (int i = lane; i < nt * w1; i += 32) r_cp<16>(L.rec + i, rsrc + i);
  const int* psrc = I->p1 + static_cast<size_t>(l0) * K;
#pragma unroll 1
  for (int i = lane; i < nt * K; i += 32) r_cp<4>(L.p1 + i, psrc + i);
  if (I->sqrt_norm) {
    const int* nsrc = I->nidx + static_cast<size_t>(l0) * K;
#pragma unroll 1
    for (int i = lane; i < nt * K; i += 32) r_cp<4>(L.nk + i, nsrc + i);
  }
}

__device__ __forceinline__ bool r_nonzero(float2 c) { return c.x != 0.f || c.y != 0.f; }

// Pass 1 for the CW columns from b0 on of row a of an ADO (its rho at yl);
// ad: the damping of the ADO; out: its right-hand sides.
template <int N, int CW>
__device__ __forceinline__ void rows_commutator(const RowsTab& L, const float2* yl, int n_rt, int a, int b0, float2 gl,
                                                float2* out) {
  const int n = N > 0 ? N : n_rt, ld = rows_ld(n);
  float2 acc[CW];
#pragma unroll
  for (int j = 0; j < CW; ++j) acc[j] = make_float2(0.f, 0.f);
  auto step = [&](int c) {
    const float2 hac = L.H[a * ld + c], yac = yl[a * n + c];
    const float2 m = make_float2(-yac.x, -yac.y);  // -h y = h (-y), to the bit
    float2 hb[(CW + 1) & ~1];
#pragma unroll
    for (int j = 0; j < CW; j += 2) {
      const float4 h = *reinterpret_cast<const float4*>(L.H + c * ld + b0 + j);
      hb[j] = make_float2(h.x, h.y);
      hb[j + 1] = make_float2(h.z, h.w);
    }
#pragma unroll
    for (int j = 0; j < CW; ++j) {
      acc[j] = __ffma2_rn(hac, yl[c * n + b0 + j], acc[j]);
      acc[j] = __ffma2_rn(hb[j], m, acc[j]);
    }
  };
  if (N > 0) {
#pragma unroll
    for (int c = 0; c < (N > 0 ? N : 1); ++c) step(c);
  } else {
#pragma unroll 2
    for (int c = 0; c < n; ++c) step(c);
  }
#pragma unroll
  for (int j = 0; j < CW; ++j) {
    if (N == 0 && b0 + j >= n) break;
    const int e = a * n + b0 + j;
    const float2 sd = L.csd[e];
    float2 D = make_float2(-acc[j].y, acc[j].x);
    cfma(D, make_float2(gl.x + sd.x, gl.y + sd.y), yl[e]);
    out[e] = D;
  }
}

// The stage epilogues in three groups, each a kernel of its own: the registers
// that Dormand-Prince's takes would leave the others spilling.
enum { ROWS_RK4 = 0, ROWS_LS = 1, ROWS_DP = 2 };
// The stage epilogue of a group's `ne` elements, two at a time.
template <int KIND>
__device__ __forceinline__ double rows_epilogue(const Stage& st, const float2* Ds, size_t g0, int ne, double dt,
                                                int cur, int lane) {
  double local = 0.0;
#pragma unroll 1
  for (int i = lane; i < ne; i += 64) {
    const int i1 = i + 32;
    const EpiPre p0 = epi_pre<float, KIND>(st, g0 + i, cur);
    EpiPre p1;
    if (i1 < ne) p1 = epi_pre<float, KIND>(st, g0 + i1, cur);
    local += epi_post<float, KIND>(st, g0 + i, Ds[i], dt, cur, p0);
    if (i1 < ne) local += epi_post<float, KIND>(st, g0 + i1, Ds[i1], dt, cur, p1);
  }
  return local;
}

template <int N, int G>
__global__ void __launch_bounds__(256, 3) k_rhs_rows(const DiagSet ds, const Stage st) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int ticket;
  double dt;
  int cur;
  if (!stage_prologue(st, dt, cur)) return;
  const float2* __restrict__ y = stage_input<float2>(st, cur);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned char* mine = smem_raw + ds.rows_tab + warp * ds.rows_warp;
  double local = 0.0;
  for (int t = blockIdx.x; t < ds.n_tiles; t += gridDim.x) {
    // the CTA's share of an instance: groups td.l0, td.l0 + td.nt, ...
    const DiagTile td = ds.tiles[t];
    const DiagInst* __restrict__ I = ds.inst + td.inst;
    const int n = N > 0 ? N : I->n, n2 = n * n, K = I->K, w1 = 1 + I->site_w, void_idx = I->nh, ados = I->tile;
    const RowsTab T = rows_tab(smem_raw, n, K);
    __syncthreads();  // the last instance's tables and ticket are free
    {
      const int ld = rows_ld(n);
      for (int i = threadIdx.x; i < n * ld; i += blockDim.x) {
        const int a = i / ld, c = i - a * ld;
        const float h = c < n ? __ldg(&I->H_f[a * n + c].x) : 0.f;
        T.H[i] = make_float2(h, h);
      }
      for (int i = threadIdx.x; i < n2; i += blockDim.x) T.csd[i] = __ldg(I->c_sd_f + i);
      for (int i = threadIdx.x; i < 3 * K; i += blockDim.x) T.cm3[i] = __ldg(I->site_cm3 + i);
      for (int i = threadIdx.x; i < 2 * K; i += blockDim.x) T.cp2[i] = __ldg(I->site_cp2 + i);
      for (int s = threadIdx.x; s < n; s += blockDim.x)
        for (int p = I->site_ptr[s]; p < I->site_ptr[s + 1]; ++p) T.msite[I->site_modes[p]] = s;
      if (threadIdx.x == 0) ticket = 0;
    }
    __syncthreads();
    const float2* __restrict__ yi = y + I->elem_off;
    const float2* __restrict__ term_p = I->term_p;
    const bool sqn = I->sqrt_norm != 0;
    const int groups = (I->nh + ados - 1) / ados;
    const size_t bsz = rows_buf_bytes(n2, K, w1 - 1, ados);
    float2* Ds = reinterpret_cast<float2*>(mine + 2 * bsz);
    // the warps draw the CTA's groups (the low tiers' take longer); Dormand-Prince's
    // keep a fixed order, in which the error norm is summed
    int turn = warp;
    auto take = [&]() {
      int k = turn;
      if (G != ROWS_DP) {
        if (lane == 0) k = atomicAdd(&ticket, 1);
        k = __shfl_sync(0xffffffffu, k, 0);
      }
      turn += blockDim.x >> 5;
      return td.l0 + td.nt * k;
    };
    int g = take(), bsel = 0;
    if (g < groups)
      rows_stage(I, yi, n2, g * ados, min(ados, I->nh - g * ados), rows_layout(mine, n2, K, w1 - 1, ados), lane);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    while (g < groups) {
      const int gn = take();
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
      __syncwarp();  // the group has landed; the other buffer and Ds are free
      if (gn < groups)
        rows_stage(I, yi, n2, gn * ados, min(ados, I->nh - gn * ados),
                   rows_layout(mine + (bsel ^ 1) * bsz, n2, K, w1 - 1, ados), lane);
      asm volatile("cp.async.commit_group;\n" ::: "memory");
      const int l0 = g * ados, nt = min(ados, I->nh - l0), ne = nt * n2;
      const RowsBuf L = rows_layout(mine + bsel * bsz, n2, K, w1 - 1, ados);
      // pass 1
      if (N > 0) {
        if (lane < nt * n) {  // the host takes at most 32 / n ADOs
          const int lt = lane / n, a = lane - lt * n;
          const int4 hdr = L.rec[lt * w1];
          rows_commutator<N, (N > 0 ? N : 1)>(T, L.y + lt * n2, n, a, 0,
                                              make_float2(__int_as_float(hdr.z), __int_as_float(hdr.w)), Ds + lt * n2);
        }
      } else {
        const int nc = (n + 3) >> 2, per = n * nc;
        for (int q = lane; q < nt * per; q += 32) {
          const int lt = q / per, r = q - lt * per, a = r / nc, b0 = (r - a * nc) << 2;
          const int4 hdr = L.rec[lt * w1];
          rows_commutator<0, 4>(T, L.y + lt * n2, n, a, b0, make_float2(__int_as_float(hdr.z), __int_as_float(hdr.w)),
                                Ds + lt * n2);
        }
      }
      __syncwarp();
      // pass 2
      constexpr int G16 = N > 0 ? 16 : 32, R = N > 0 ? 1 : 2;  // lanes of an ADO; elements of a lane
      {
        // the lane's place in the row of a mode of site s (col 0: element s n + x) or
        // in its column (col 1: x n + s, without the diagonal)
        const int sub = lane & (G16 - 1);
        int x[R], col[R], mul[R], add[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int j = sub + r * G16;
          col[r] = j >= n ? 1 : 0;
          x[r] = j < 2 * n ? j - col[r] * n : -1;
          mul[r] = col[r] ? 1 : n;
          add[r] = col[r] ? x[r] * n : x[r];
        }
        for (int lt0 = 0; lt0 < nt; lt0 += 32 / G16) {
          const int lt = lt0 + lane / G16;
          const int4* rec = L.rec + min(lt, nt - 1) * w1;
          float2* dl = Ds + lt * n2;
          const int pad = (ados - lt) * n2 + (lane & 15);  // an element of its own behind the group's
          const int4 hdr = *rec;
          const int nm = lt < nt ? hdr.x : 0;
          const bool plus = lt < nt && (hdr.y || term_p);
          // A lane's terms are gathered together, then added in order.  No
          // branches: a lane without a term works on the padding element.
          auto add_term = [&](int el, float2 c, float2 v) {
            float2 D = dl[el];
            cfma(D, c, v);
            dl[el] = D;
          };
          if (__any_sync(0xffffffffu, plus)) {  // +1 terms (they vanish on the diagonal)
            const int ltc = min(lt, nt - 1);
            const int* p1r = L.p1 + ltc * K;
            const float2* tp = yi;
            if (term_p && plus) tp = term_p + static_cast<ptrdiff_t>(l0 + lt - I->term_first) * K * n2;
            constexpr int B = 4;
#pragma unroll 1
            for (int k0 = 0; k0 < K; k0 += B) {
              float2 v[B][R];
              unsigned hits = 0;
#pragma unroll
              for (int u = 0; u < B; ++u) {
                const int k = min(k0 + u, K - 1), s = T.msite[k], lp = p1r[k];
                const bool real = lp != void_idx, on = plus && k0 + u < K && (real || term_p);
                const float2* src = yi + (real ? lp * n2 : 0);
                if (!real) src = tp + k * n2;
#pragma unroll
                for (int r = 0; r < R; ++r) {
                  const bool hit = on && x[r] >= 0 && x[r] != s;
                  v[u][r] = hit ? __ldg(src + add[r] + mul[r] * s) : make_float2(0.f, 0.f);
                  hits |= (hit ? 1u : 0u) << (u * R + r);
                }
              }
#pragma unroll
              for (int u = 0; u < B; ++u) {
                const int k = min(k0 + u, K - 1), s = T.msite[k];
                float f = 1.f;
                if (sqn && p1r[k] != void_idx) f = sqrtf(static_cast<float>(L.nk[ltc * K + k] + 1));
#pragma unroll
                for (int r = 0; r < R; ++r) {
                  float2 c = T.cp2[2 * k + col[r]];
                  const bool hit = ((hits >> (u * R + r)) & 1u) && r_nonzero(c);
                  if (sqn) c = make_float2(f * c.x, f * c.y);
                  add_term(hit ? add[r] + mul[r] * s : pad, c, v[u][r]);
                }
                __syncwarp();
              }
            }
          }
          // -1 terms: the ADO's occupied modes
#pragma unroll 1
          for (int m0 = 1; __any_sync(0xffffffffu, m0 <= nm); m0 += 4) {
            float2 v[4][R], cf[4][R];
            int e[4][R];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const int4 q = rec[max(min(m0 + u, nm), 1)];  // the -1 neighbour's offset, site, 3 k, factor
              const float f = __int_as_float(q.w);
#pragma unroll
              for (int r = 0; r < R; ++r) {
                const bool dg = x[r] == q.y;
                const float2 c = T.cm3[q.z + (dg ? 2 : col[r])];
                const bool hit = m0 + u <= nm && x[r] >= 0 && !(col[r] && dg) && r_nonzero(c);
                const int el = add[r] + mul[r] * q.y;
                v[u][r] = hit ? __ldg(yi + q.x + el) : make_float2(0.f, 0.f);
                cf[u][r] = make_float2(f * c.x, f * c.y);
                e[u][r] = hit ? el : pad;
              }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
#pragma unroll
              for (int r = 0; r < R; ++r) add_term(e[u][r], cf[u][r], v[u][r]);
              __syncwarp();
            }
          }
        }
      }
      __syncwarp();
      // pass 3
      const size_t g0 = static_cast<size_t>(I->elem_off) + static_cast<size_t>(l0) * n2;
      if (G == ROWS_LS)
        local += rows_epilogue<EPI_LS>(st, Ds, g0, ne, dt, cur, lane);
      else if (G == ROWS_DP)
        local += st.kind == EPI_DP7 ? rows_epilogue<EPI_DP7>(st, Ds, g0, ne, dt, cur, lane)
                                    : rows_epilogue<EPI_DP>(st, Ds, g0, ne, dt, cur, lane);
      else if (st.kind == EPI_RK4_1)
        rows_epilogue<EPI_RK4_1>(st, Ds, g0, ne, dt, cur, lane);
      else if (st.kind == EPI_RK4_2)
        rows_epilogue<EPI_RK4_2>(st, Ds, g0, ne, dt, cur, lane);
      else if (st.kind == EPI_RK4_3)
        rows_epilogue<EPI_RK4_3>(st, Ds, g0, ne, dt, cur, lane);
      else
        rows_epilogue<EPI_RK4_4>(st, Ds, g0, ne, dt, cur, lane);
      bsel ^= 1;
      g = gn;
    }
  }
  if (G == ROWS_DP && st.kind == EPI_DP7) dp7_finish(st, local, ds.total);
}

// The kernel's own records: per ADO the header of site_rec, then per occupied
// mode the -1 neighbour's element offset, the site, 3 k and the factor (n_k, or
// its root) that scales the mode's coefficients.
__global__ void k_rows_records(const DiagInst I, int4* rec) {
  const int w1 = 1 + I.site_w, i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= I.nh * w1) return;
  const int4 r = I.site_rec[i];
  if (i % w1 == 0) {
    rec[i] = r;
    return;
  }
  const float nk = static_cast<float>(r.z);
  rec[i] = make_int4(r.y * I.n2, r.w, 3 * r.x, __float_as_int(I.sqrt_norm ? sqrtf(nk) : nk));
}

using RowsKernel = void (*)(const DiagSet, const Stage);
template <int N>
RowsKernel rows_variant(int kind) {
  if (kind == EPI_DP || kind == EPI_DP7) return k_rhs_rows<N, ROWS_DP>;
  return kind == EPI_LS ? k_rhs_rows<N, ROWS_LS> : k_rhs_rows<N, ROWS_RK4>;
}
RowsKernel rows_kernel(const DiagSet& ds, int kind) {
  switch (ds.rows_n) {
    case 2: return rows_variant<2>(kind);
    case 3: return rows_variant<3>(kind);
    case 4: return rows_variant<4>(kind);
    case 5: return rows_variant<5>(kind);
    case 6: return rows_variant<6>(kind);
    case 7: return rows_variant<7>(kind);
    case 8: return rows_variant<8>(kind);
    default: return rows_variant<0>(kind);
  }
}

}  // namespace

bool rows_eligible(const DiagInst& I, bool mixed) {
  return mixed && I.site_local && I.site_rec && I.h_real && I.max_terms <= 4 && I.n >= 2 && I.n <= 32 &&
         static_cast<long long>(I.nh) * std::max(I.n2, 1 + I.site_w) < (1ll << 31);
}

cudaError_t launch_rows_records(const DiagInst& I, int4* rec, cudaStream_t s) {
  const int count = I.nh * (1 + I.site_w);
  if (count <= 0) return cudaSuccess;
  k_rows_records<<<(count + 255) / 256, 256, 0, s>>>(I, rec);
  ++g_launches;
  return cudaGetLastError();
}

size_t rows_tables(const DiagInst& I) { return rows_tab_bytes(I.n, I.K); }

size_t rows_warp(const DiagInst& I, int ados) {
  return (2 * rows_buf_bytes(I.n2, I.K, I.site_w, ados) + sizeof(float2) * (static_cast<size_t>(ados) * I.n2 + 16) + 15) &
         ~size_t(15);
}

int rows_resident(const DiagSet& ds, int kind, int block) {
  RowsKernel kern = rows_kernel(ds, kind);
  if (ds.smem > 48 * 1024 &&
      allow_smem(reinterpret_cast<const void*>(kern)) != cudaSuccess)
    return 0;
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, block, ds.smem) != cudaSuccess) return 0;
  return per_sm;
}

cudaError_t launch_rows(const DiagSet& ds, const Stage& st, int grid, int block, cudaStream_t s) {
  if (st.kind == EPI_DIFF) return cudaErrorInvalidValue;  // calc_diff keeps k_rhs_diag
  RowsKernel kern = rows_kernel(ds, st.kind);
  if (ds.smem > 48 * 1024) {
    cudaError_t e = allow_smem(reinterpret_cast<const void*>(kern));
    if (e != cudaSuccess) return e;
  }
  kern<<<grid, block, ds.smem, s>>>(ds, st);
  ++g_launches;
  return cudaGetLastError();
}

}  // namespace heomgb
