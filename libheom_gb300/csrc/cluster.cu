// Cluster-resident fixed steps: one output interval (RK4 or LSRK4) of one or
// many small models in one launch, a thread-block cluster per bin of whole
// instances.  Fixed-step part of rk4.h:40-65 and lsrk4.h:32-47 over
// heom_hilb::calc_diff_impl (heom_hilb.h:70-215) with diagonal couplings.
//
// The ADOs of a bin's instances are dealt out to the cluster's CTAs in turn.
// Every CTA keeps the stage input of its ADOs in shared memory (two copies)
// and reads a neighbour ADO's elements from the shared memory of the CTA that
// owns it; a thread keeps the state, the accumulator and the damping of its
// elements in registers.  Stages are separated by the hardware's cluster
// barrier: its arrival follows the stage's writes, the commutators (own ADOs
// only) run behind it, and the wait stands before the neighbour reads.  Nothing
// goes through global memory between the interval's first load and its last
// store, and nothing spins.
//
// What bounds it: a stage is a chain of barrier, neighbour read, bath terms
// and epilogue.  In the FP64 form a warp instruction holds its sub-partition's
// FP64 pipe for 64 cycles however many lanes are active, so the two components
// of an element go to two neighbouring lanes (half the chain of one lane per
// element; the sums keep their order, component by component).
//
// Measured per stage, before (grid barriers through L2, or graphs of stage
// launches) and now: spin-boson depth 10 FP64 3.23 -> 2.03 us (16 CTAs; per
// stage about 440 cycles to arrive, 900 commutator and damping, 2500 neighbour
// reads and up to six bath terms, 290 epilogue: the dependent FP64 FMAs are
// the chain), mixed 1.75 -> 1.28 us; 128 uneven sweep instances (42 FP64, 86
// mixed, concurrently) 12.6 -> 6.3 us.
//
// The arithmetic per element is the stage kernels' (k_rhs_diag with the fused
// epilogues), in their order, so the results are their bits.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "heomgb_impl.cuh"
#include "stage.cuh"

namespace heomgb {

namespace {

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_size() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;\n" : "=r"(r));
  return r;
}
// (both want a converged warp)
__device__ __forceinline__ void cluster_arrive() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// the address, in the cluster's shared window, of this CTA's address `a` in CTA `rank`
__device__ __forceinline__ uint32_t cluster_addr(uint32_t a, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_load(uint32_t a, double2& v) {
  asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];\n" : "=d"(v.x), "=d"(v.y) : "r"(a) : "memory");
}
__device__ __forceinline__ void cluster_load(uint32_t a, float2& v) {
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];\n" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
}

// What a lane computes: an element (mixed form) or one component of it (FP64 form).
template <typename TC>
struct Part;
template <>
struct Part<float> {
  using V = float2;
  static constexpr int kLanes = 1;
};
template <>
struct Part<double> {
  using V = double;
  static constexpr int kLanes = 2;
};
__device__ __forceinline__ double sel(double2 v, int p) { return p ? v.y : v.x; }

// i[H, rho] + damping of element (a, b); Xl: the ADO's stage input.  FP64:
// component p of the result, which the commutator's other component feeds.
__device__ __forceinline__ float2 own_part(const float2* H, const float2* Xl, int n, int a, int b, bool hreal,
                                           float2 g, int) {
  float2 acc = make_float2(0.f, 0.f);
  if (hreal) {
#pragma unroll 2
    for (int c = 0; c < n; ++c) {
      const float hac = H[a * n + c].x, hcb = H[c * n + b].x;
      const float2 ycb = Xl[c * n + b], yac = Xl[a * n + c];
      acc.x = fmaf(hac, ycb.x, acc.x);
      acc.x = fmaf(-hcb, yac.x, acc.x);
      acc.y = fmaf(hac, ycb.y, acc.y);
      acc.y = fmaf(-hcb, yac.y, acc.y);
    }
  } else {
    float2 neg = make_float2(0.f, 0.f);
    for (int c = 0; c < n; ++c) {
      cfma(acc, H[a * n + c], Xl[c * n + b]);
      cfma(neg, Xl[a * n + c], H[c * n + b]);
    }
    acc.x -= neg.x;
    acc.y -= neg.y;
  }
  float2 D = make_float2(-acc.y, acc.x);
  cfma(D, g, Xl[a * n + b]);
  return D;
}
__device__ __forceinline__ double own_part(const double2* H, const double2* Xl, int n, int a, int b, bool hreal,
                                           double2 g, int p) {
  const int q = 1 - p;
  double acc = 0.0;
  if (hreal) {
    const double* X = reinterpret_cast<const double*>(Xl) + q;
#pragma unroll 2
    for (int c = 0; c < n; ++c) {
      const double hac = H[a * n + c].x, hcb = H[c * n + b].x;
      acc = fma(hac, X[2 * (c * n + b)], acc);
      acc = fma(-hcb, X[2 * (a * n + c)], acc);
    }
  } else {
    double neg = 0.0;
    for (int c = 0; c < n; ++c) {
      const double2 h1 = H[a * n + c], h2 = H[c * n + b], y1 = Xl[c * n + b], y2 = Xl[a * n + c];
      acc = fma(h1.x, sel(y1, q), acc);
      acc = fma(q ? h1.y : -h1.y, sel(y1, p), acc);
      neg = fma(y2.x, sel(h2, q), neg);
      neg = fma(q ? y2.y : -y2.y, sel(h2, p), neg);
    }
    acc -= neg;
  }
  double D = p ? acc : -acc;
  const double2 y = Xl[a * n + b];
  D = fma(g.x, sel(y, p), D);
  return fma(p ? g.y : -g.y, sel(y, 1 - p), D);
}
__device__ __forceinline__ void add_term(float2& D, float2 c, float2 v, int) { cfma(D, c, v); }
__device__ __forceinline__ void add_term(double& D, double2 c, double2 v, int p) {
  D = fma(c.x, sel(v, p), D);
  D = fma(p ? c.y : -c.y, sel(v, 1 - p), D);
}

// What a lane keeps of its element between stages: state, RK4 accumulator or
// LSRK4 buffer and (mixed form) the state's FP32 copy; `stage` takes D and
// gives the next stage's input.
// COMP (FP64): the state's additions carry their rounding errors along (quick
// two-sums), for models that run in another basis than the caller's: two more
// roundings, into the basis and out of it, must not cost accuracy (two levels, V =
// sigma_x, 200 steps, mean of six models against 80 bits: 1.0e-15 in the caller's basis,
// 1.2e-15 in the other without this, 1.8e-16 with it; a step takes 4 % longer).
template <typename TC, int SCHEME, bool COMP = false>
struct Keep;
template <int SCHEME>
struct Keep<double, SCHEME, true> {
  double S, A, C;  // state, RK4's increment or LSRK4's buffer, what S's rounding left out
  __device__ __forceinline__ double start(double2 v, int p) {
    S = sel(v, p);
    A = C = 0.0;
    return S;
  }
  __device__ __forceinline__ void add(double inc) {
    const double s = __dadd_rn(S, inc);
    C = __dsub_rn(inc, __dsub_rn(s, S));
    S = s;
  }
  __device__ __forceinline__ double stage(int s, double dt, double D) {
    const double k = __dmul_rn(-dt, D);
    if constexpr (SCHEME == kResidentLs) {
      const double B = s == 0 ? 1.0 / 3.0 : s == 1 ? 3.0 / 4.0 : s == 2 ? 2.0 / 3.0 : 1.0 / 4.0;
      A = s == 0 ? k : __dadd_rn(-A, k);
      add(fma(B, A, C));
      return S;
    } else {
      if (s < 3) {
        A = s == 0 ? fma(1.0 / 6.0, k, C) : fma(2.0 / 6.0, k, A);
        return fma(s == 2 ? 1.0 : 0.5, k, S);
      }
      add(fma(1.0 / 6.0, k, A));
      return S;
    }
  }
  __device__ __forceinline__ void finish(double2* out, int p) const { reinterpret_cast<double*>(out)[p] = S; }
};
template <int SCHEME>
struct Keep<double, SCHEME, false> {
  double S, A;
  __device__ __forceinline__ double start(double2 v, int p) {
    S = sel(v, p);
    A = 0.0;
    return S;
  }
  __device__ __forceinline__ double stage(int s, double dt, double D) {
    const double k = __dmul_rn(-dt, D);
    if constexpr (SCHEME == kResidentLs) {
      const double B = s == 0 ? 1.0 / 3.0 : s == 1 ? 3.0 / 4.0 : s == 2 ? 2.0 / 3.0 : 1.0 / 4.0;
      A = s == 0 ? k : __dadd_rn(-A, k);
      S = fma(B, A, S);
      return S;
    } else {
      if (s < 3) {
        const double y = fma(s == 2 ? 1.0 : 0.5, k, S);
        A = fma(s == 0 ? (1.0 / 6.0) : (2.0 / 6.0), k, s == 0 ? S : A);
        return y;
      }
      S = fma(1.0 / 6.0, k, A);
      return S;
    }
  }
  __device__ __forceinline__ void finish(double2* out, int p) const { reinterpret_cast<double*>(out)[p] = S; }
};
template <int SCHEME>
struct Keep<float, SCHEME, false> {
  double2 S, A;
  float2 B, F;  // LSRK4 buffer; RK4: the state's FP32 copy
  __device__ __forceinline__ float2 start(double2 v, int) {
    S = v;
    A = v;
    B = make_float2(0.f, 0.f);
    F = to_f(v);
    return F;
  }
  __device__ __forceinline__ float2 stage(int s, double dt, float2 D) {
    const float fdt = static_cast<float>(dt);
    if constexpr (SCHEME == kResidentLs) {
      const double w = s == 0 ? 1.0 / 3.0 : s == 1 ? 3.0 / 4.0 : s == 2 ? 2.0 / 3.0 : 1.0 / 4.0;
      B = s == 0 ? make_float2(__fmul_rn(-fdt, D.x), __fmul_rn(-fdt, D.y))
                 : make_float2(fmaf(-fdt, D.x, -B.x), fmaf(-fdt, D.y, -B.y));
      const double2 bd = to_d(B);
      S = make_double2(fma(w, bd.x, S.x), fma(w, bd.y, S.y));
      return to_f(S);
    } else {
      const float2 k = make_float2(__fmul_rn(-fdt, D.x), __fmul_rn(-fdt, D.y));
      if (s < 3) {
        const float c = s == 2 ? 1.0f : 0.5f;
        const float w = static_cast<float>(s == 0 ? (1.0 / 6.0) : (2.0 / 6.0));
        const double2 kw = to_d(make_float2(__fmul_rn(w, k.x), __fmul_rn(w, k.y)));
        if (s == 0) A = S;
        A.x += kw.x;
        A.y += kw.y;
        return make_float2(fmaf(c, k.x, F.x), fmaf(c, k.y, F.y));
      }
      const double2 k6 = to_d(make_float2(__fmul_rn(1.0f / 6.0f, k.x), __fmul_rn(1.0f / 6.0f, k.y)));
      S = make_double2(A.x + k6.x, A.y + k6.y);
      F = to_f(S);
      return F;
    }
  }
  __device__ __forceinline__ void finish(double2* out, int) const { *out = S; }
};

// The ADOs of a bin's instances are dealt out to the cluster's CTAs in turn:
// ADO l of an instance that starts at the bin's ADO `base` goes to CTA
// (base + l) % cs.  (Stretches of consecutive ADOs per CTA, whose neighbour
// reads go to fewer CTAs, were no faster for two levels and 17 % slower for the
// 7-site depth-2 hierarchy: the tiers below the deepest have twice the terms.)
__host__ __device__ __forceinline__ int first_ado(int base, int r, int cs) { return (r - base % cs + cs) % cs; }
__host__ __device__ __forceinline__ int count_ados(int base, int nh, int r, int cs) {
  const int f = first_ado(base, r, cs);
  return f < nh ? (nh - 1 - f) / cs + 1 : 0;
}

// Shared memory: H of the bin's instances | two stage-input copies (ecap
// elements) | the bath terms' coefficients, then addresses (terms x ecap).
// Up to two elements per thread the kernel keeps to 72 registers, so that a CTA
// of an FP64 and one of a mixed sub-batch share an SM.
template <typename TC, int SCHEME, int EPT, bool COMP>
__global__ void __launch_bounds__(EPT > 2 ? 512 : kClusterMaxBlock, EPT > 2 ? 1 : 2) k_cluster(const ClusterArgs A) {
  using C = cx_t<TC>;
  using V = typename Part<TC>::V;
  constexpr int L = Part<TC>::kLanes;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ DiagInst s_inst[kClusterMaxInst];
  __shared__ int s_h[kClusterMaxInst + 1], s_base[kClusterMaxInst + 1];  // an instance's H, its first ADO in the bin
  __shared__ int s_off[kClusterMaxInst + 1][kClusterMaxSize];  // an instance's first element in each CTA
  const int cs = static_cast<int>(cluster_size()), rank = static_cast<int>(cluster_rank());
  const int bin = blockIdx.x / cs;
  const int i0 = A.bin_ptr[bin], ni = A.bin_ptr[bin + 1] - i0;
  for (int i = threadIdx.x; i < ni; i += blockDim.x) s_inst[i] = A.inst[A.bin_inst[i0 + i]];
  __syncthreads();
  for (int r = threadIdx.x; r < cs; r += blockDim.x) {
    int e = 0, h = 0, base = 0;
    for (int i = 0; i < ni; ++i) {
      s_off[i][r] = e;
      if (r == 0) {
        s_h[i] = h;
        s_base[i] = base;
      }
      e += count_ados(base, s_inst[i].nh, r, cs) * s_inst[i].n2;
      h += s_inst[i].n2;
      base += s_inst[i].nh;
    }
    s_off[ni][r] = e;
    if (r == 0) s_h[ni] = h;
  }
  __syncthreads();
  const int E = s_off[ni][rank], ecap = A.ecap;
  C* Hs = reinterpret_cast<C*>(smem_raw);
  C* X = Hs + ((s_h[ni] + 1) & ~1);
  C* Tc = X + 2 * static_cast<size_t>(ecap);
  uint32_t* Ta = reinterpret_cast<uint32_t*>(Tc + static_cast<size_t>(A.terms) * ecap);
  for (int i = 0; i < ni; ++i) {
    const C* Hg = pick<TC>(s_inst[i].H, s_inst[i].H_f);
    for (int j = threadIdx.x; j < s_inst[i].n2; j += blockDim.x) Hs[s_h[i] + j] = Hg[j];
  }
  const uint32_t x_addr = static_cast<uint32_t>(__cvta_generic_to_shared(X));
  const uint32_t x_bytes = static_cast<uint32_t>(ecap) * sizeof(C);
  const int p = L == 2 ? static_cast<int>(threadIdx.x & 1) : 0;
  const int per = blockDim.x / L;  // elements per round
  // the lane's elements
  Keep<TC, SCHEME, COMP> keep[EPT];
  C damp[EPT];
  int ii[EPT], cnt[EPT], ab[EPT], pos[EPT];  // instance, bath terms, (a, b), place in X
  long long gi[EPT];
#pragma unroll
  for (int q = 0; q < EPT; ++q) {
    const int le = static_cast<int>(threadIdx.x) / L + q * per;
    ii[q] = cnt[q] = ab[q] = pos[q] = 0;
    gi[q] = 0;
    damp[q] = cx<TC>(0, 0);
    if (le >= E) {
      keep[q].start(make_double2(0.0, 0.0), p);
      continue;
    }
    int i = 0;
    while (s_off[i + 1][rank] <= le) ++i;
    const DiagInst& I = s_inst[i];
    const int n = I.n, n2 = I.n2, K = I.K, base = s_base[i];
    // FP64: the elements with the most bath terms first, ADO by ADO for each, so
    // that the warps of elements with few terms skip the others' FP64 work
    const int loc = le - s_off[i][rank], na = (s_off[i + 1][rank] - s_off[i][rank]) / n2;
    const int slot = L == 2 ? loc % na : loc / n2, e = L == 2 ? __ldg(I.e_order + loc / na) : loc - slot * n2;
    const int a = e / n, at = s_off[i][rank] + slot * n2 + e;
    const int l = first_ado(base, rank, cs) + slot * cs;
    pos[q] = at;
    ii[q] = i;
    ab[q] = a << 16 | (e - a * n);
    gi[q] = I.elem_off + static_cast<long long>(l) * n2 + e;
    const C g0 = pick<TC>(I.ngd, I.ngd_f)[l], g1 = pick<TC>(I.c_sd, I.c_sd_f)[e];
    damp[q] = cx<TC>(g0.x + g1.x, g0.y + g1.y);
    const V x = keep[q].start(A.S[gi[q]], p);
    if constexpr (L == 2)
      reinterpret_cast<double*>(X + at)[p] = x;
    else
      X[at] = x;
    // the terms that have a neighbour, k_rhs_diag's order
    auto put = [&](int k_ado, C cf) {
      if (p == 0) {
        const int r = (base + k_ado) % cs;
        const int to = s_off[i][r] + (k_ado - first_ado(base, r, cs)) / cs * n2 + e;
        Ta[static_cast<size_t>(cnt[q]) * ecap + le] = cluster_addr(x_addr + static_cast<uint32_t>(to) * sizeof(C), r);
        Tc[static_cast<size_t>(cnt[q]) * ecap + le] = cf;
      }
      ++cnt[q];
    };
    const bool sqn = I.sqrt_norm != 0;
    const int* __restrict__ nrow = I.nidx + static_cast<size_t>(l) * K;
    for (int t = __ldg(I.plus_ptr + e); t < __ldg(I.plus_ptr + e + 1); ++t) {
      const int k = __ldg(I.plus_mode + t), lp = __ldg(I.p1 + static_cast<size_t>(l) * K + k);
      if (lp == I.nh) continue;
      C cf = pick<TC>(I.c_plus, I.c_plus_f)[t];
      if (sqn) {
        if constexpr (L == 2) {
          cf = I.c_plus_n[static_cast<size_t>(t) * I.occ_rows + __ldg(nrow + k)];
        } else {
          const float f = sqrtf(static_cast<float>(__ldg(nrow + k) + 1));
          cf = make_float2(f * cf.x, f * cf.y);
        }
      }
      put(lp, cf);
    }
    for (int t = __ldg(I.minus_ptr + e); t < __ldg(I.minus_ptr + e + 1); ++t) {
      const int k = __ldg(I.minus_mode + t), lm = __ldg(I.m1 + static_cast<size_t>(l) * K + k);
      if (lm == I.nh) continue;
      const int nk_i = __ldg(nrow + k);
      if constexpr (L == 2) {
        put(lm, I.c_minus_n[static_cast<size_t>(t) * I.occ_rows + nk_i]);
      } else {
        const float nk = sqn ? sqrtf(static_cast<float>(nk_i)) : static_cast<float>(nk_i);
        const float2 cm = I.c_minus_f[t];
        put(lm, make_float2(nk * cm.x, nk * cm.y));
      }
    }
  }
  for (long long step = 0; step <= A.n_steps; ++step) {
    const double dt = step < A.n_steps ? A.dt_step : A.dt_last;
#pragma unroll 1
    for (int s = 0; s < 4; ++s) {
      // the stage's input is complete in this CTA; the others' is behind the wait
      cluster_arrive();
      __syncthreads();
      const C* Xs = X + static_cast<size_t>(s & 1) * ecap;
      C* Xn = X + static_cast<size_t>((s + 1) & 1) * ecap;
      V D[EPT];
#pragma unroll
      for (int q = 0; q < EPT; ++q) {
        const int le = static_cast<int>(threadIdx.x) / L + q * per;
        if (le >= E) continue;
        const DiagInst& I = s_inst[ii[q]];
        const int n = I.n, a = ab[q] >> 16, b = ab[q] & 0xffff;
        D[q] = own_part(Hs + s_h[ii[q]], Xs + (pos[q] - a * n - b), n, a, b, I.h_real != 0, damp[q], p);
      }
      cluster_wait();
      const uint32_t xo = static_cast<uint32_t>(s & 1) * x_bytes;
#pragma unroll
      for (int q = 0; q < EPT; ++q) {
        const int le = static_cast<int>(threadIdx.x) / L + q * per;
        if (le >= E) continue;
        for (int t0 = 0; t0 < cnt[q]; t0 += 4) {  // four neighbour reads in flight
          C v[4];
#pragma unroll
          for (int t = 0; t < 4; ++t)
            if (t0 + t < cnt[q]) cluster_load(Ta[static_cast<size_t>(t0 + t) * ecap + le] + xo, v[t]);
#pragma unroll
          for (int t = 0; t < 4; ++t)
            if (t0 + t < cnt[q]) add_term(D[q], Tc[static_cast<size_t>(t0 + t) * ecap + le], v[t], p);
        }
        const V x = keep[q].stage(s, dt, D[q]);
        if constexpr (L == 2)
          reinterpret_cast<double*>(Xn + pos[q])[p] = x;
        else
          Xn[pos[q]] = x;
      }
    }
  }
#pragma unroll
  for (int q = 0; q < EPT; ++q)
    if (static_cast<int>(threadIdx.x) / L + q * per < E) keep[q].finish(A.S + gi[q], p);
  // no CTA leaves while another may still read its shared memory
  cluster_arrive();
  cluster_wait();
}

template <typename TC, int SCHEME, bool COMP = false>
const void* kernel_ept(int ept) {
  switch (ept) {
    case 1: return reinterpret_cast<const void*>(k_cluster<TC, SCHEME, 1, COMP>);
    case 2: return reinterpret_cast<const void*>(k_cluster<TC, SCHEME, 2, COMP>);
    case 4: return reinterpret_cast<const void*>(k_cluster<TC, SCHEME, 4, COMP>);
    default: return nullptr;
  }
}
template <int SCHEME>
const void* kernel_form(ClusterForm f, int ept) {
  return f == kClusterMixed ? kernel_ept<float, SCHEME>(ept)
         : f == kClusterFp64 ? kernel_ept<double, SCHEME>(ept)
                             : kernel_ept<double, SCHEME, true>(ept);
}
const void* cluster_kernel(ClusterForm f, int scheme, int ept) {
  return scheme == kResidentLs ? kernel_form<kResidentLs>(f, ept) : kernel_form<kResidentRk4>(f, ept);
}

cudaError_t configure(const void* kern, int size, size_t smem, int grid, int block, cudaStream_t s,
                      cudaLaunchConfig_t& cfg, cudaLaunchAttribute& attr) {
  // the largest shared-memory split, so that the launches of two sub-batches can share an SM
  const cudaError_t e = allow_smem(kern, true, true);
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = size;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg = cudaLaunchConfig_t{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return e;
}

}  // namespace

int cluster_lanes(bool mixed) { return mixed ? 1 : 2; }

int cluster_elements(const int* n2, const int* nh, int count, int size) {
  int most = 0;
  for (int r = 0; r < size; ++r) {
    int e = 0, base = 0;
    for (int i = 0; i < count; ++i) {
      e += count_ados(base, nh[i], r, size) * n2[i];
      base += nh[i];
    }
    most = std::max(most, e);
  }
  return most;
}

size_t cluster_smem(int h_elems, int ecap, int terms, bool mixed) {
  const size_t c = mixed ? sizeof(float2) : sizeof(double2);
  return c * (((h_elems + 1) & ~1) + static_cast<size_t>(ecap) * (2 + terms)) +
         sizeof(uint32_t) * static_cast<size_t>(ecap) * terms;
}

int cluster_active(ClusterForm form, int scheme, int ept, int size, int block, size_t smem) {
  const void* kern = cluster_kernel(form, scheme, ept);
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr;
  int n = 0;
  if (!kern || configure(kern, size, smem, size, block, nullptr, cfg, attr) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

cudaError_t launch_cluster(const ClusterArgs& args, ClusterForm form, int scheme, int ept, int size, int bins, int block,
                           size_t smem, cudaStream_t s) {
  const void* kern = cluster_kernel(form, scheme, ept);
  if (!kern) return cudaErrorInvalidValue;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr;
  cudaError_t e = configure(kern, size, smem, bins * size, block, s, cfg, attr);
  if (e != cudaSuccess) return e;
  ClusterArgs a = args;
  void* params[] = {&a};
  e = cudaLaunchKernelExC(&cfg, kern, params);
  ++g_launches;
  return e;
}

}  // namespace heomgb
