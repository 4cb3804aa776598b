// The learned closure's fused tensor-core kernels: the inference of one stage
// (k_term_mlp) and the training pass over a minibatch (k_train, k_dw, k_adam).
//
// A CTA keeps the activations of its tile of rows in shared memory as BF16
// core matrices and the accumulators in tensor memory.  The weights come
// packed as the core-matrix chunks that the MMAs read (tcore.cuh), so a chunk
// is one bulk copy and no thread converts or moves a weight.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "heomgb_impl.cuh"
#include "tcore.cuh"

namespace heomgb {

namespace {

constexpr int kThr = 512;   // 16 warps of work: warp w reads tensor-memory lanes 32 (w % 4) ..
constexpr int kWarps = kThr / 32;
constexpr int kThrAll = kThr + 32;  // and the producer's warp
constexpr size_t kMaxSmem = 232448;

// barrier of the working warps (the producer's warp takes no part)
__device__ __forceinline__ void sync_work() { asm volatile("bar.sync 1, 512;\n" ::: "memory"); }
__device__ __forceinline__ bool and_work(bool p) {
  int r;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.b32 p, %1, 0;\n bar.red.and.pred q, 1, 512, p;\n selp.b32 %0, 1, 0, q;\n}\n"
      : "=r"(r)
      : "r"(static_cast<int>(p))
      : "memory");
  return r != 0;
}

__device__ __forceinline__ uint4 pack8(const float* f) {
  uint32_t w[4];
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(f[2 * t], f[2 * t + 1]);  // the first in the low half
    w[t] = *reinterpret_cast<const uint32_t*>(&h);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// the warps' writes to shared memory become visible to the MMAs
__device__ __forceinline__ void publish() {
  fence_async();
  fence_before();
  sync_work();
  fence_after();
}

// One layer: a thread of warp 0 issues its MMAs and waits for them (bounded)
// while the other warps sleep in the barrier; the verdict is theirs too.
template <int SLOTS>
__device__ __forceinline__ bool run_layer(const WeightRing<SLOTS>& W, unsigned char* act, int n, int m_tiles,
                                          int n_chunks, uint32_t tmem, uint64_t* done, uint32_t& parity, int& taken) {
  bool mine = true;
  if (threadIdx.x < 32) {
    if (elect_one()) {
      mine = W.layer(s_addr(act), n, m_tiles, n_chunks, tmem, taken);
      g_commit(done);
      mine = g_wait(done, parity) && mine;  // on failure: what is in flight ends, bounded
    }
    __syncwarp();
  }
  taken += n_chunks;
  parity ^= 1u;
  const bool ok = and_work(mine);
  fence_after();
  return ok;
}

// byte offset of (column c, rows 8 g ..) in an activation tile of `rows` rows
__device__ __forceinline__ int act_off(int c, int g, int rows) {
  return ((c >> 3) * (rows >> 3) + g) * 128 + (c & 7) * 16;
}

// ------------------------------------------------------------------ inference
// One launch per stage evaluates the closure for every row (tier-N ADO j,
// mode k): CTA t takes the rows of ADOs [t * apt, (t + 1) * apt), builds their
// input features in shared memory, runs the three layers and applies the gain
// head: P[(j K + k) n2 + e] = C_e rho_l[e] / sigma_k, C_e = y_e - i sg_e softplus(z_e).
//
// Bound: the instructions of the two GELU passes (about 40 each for 256 values
// per row) and the latency of one tile's chain, so the tile is the smallest
// that fills the SMs in one wave (the 7-site depth-3 model: 4 ADOs, 56 rows,
// 140 CTAs).  The weights run ahead of the MMAs through a ring of eight 16 KB
// slots: the first layer's are in flight while the features are built.
// Measured there (7840 rows, 210-256-256-98): 106.6 us in 126-row tiles with
// weights and features staged element by element; 46.5 us with bulk-copied
// weights; 39.8 us in 56-row tiles; 15-17 us in this form (the MMAs issued by an
// elected thread, the row factors from set-up tables): 34 k cycles, of which
// the GELU passes 10 k, the MMAs 10 k, set-up and features 9 k, gain head 5 k.
constexpr int kTermSlots = 8;

__host__ __device__ __forceinline__ int term_rows(int apt, int K) { return (apt * K + 15) / 16 * 16; }
__host__ __device__ __forceinline__ size_t term_smem_bytes(int apt, int K, int n2) {
  return static_cast<size_t>(256) * term_rows(apt, K) * 2 + kTermSlots * 16384 + 8 * (2 * kTermSlots + 2) +
         sizeof(float) * (640 + 128 + 128) + sizeof(float2) * (256 + static_cast<size_t>(apt) * n2);
}

template <typename TB>
__global__ void __launch_bounds__(kThrAll, 1) k_term_mlp(const TermMlpArgs A) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const TermModel& tm = A.tm;
  const int n = tm.n, n2 = n * n, K = tm.K, din = A.din, h = A.h, dout = A.dout;
  const int NR = term_rows(A.apt, K), ng = NR >> 3;
  unsigned char* act = smem_raw;                               // 256 x NR BF16: features, then the hidden activations
  unsigned char* ring = act + static_cast<size_t>(256) * NR * 2;  // after the last layer NR x dout FP32 outputs
  uint64_t* bar = reinterpret_cast<uint64_t*>(ring + kTermSlots * 16384);  // full[8], empty[8], done
  uint64_t* done = bar + 2 * kTermSlots;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(done + 1);
  float* bias = reinterpret_cast<float*>(bar + 2 * kTermSlots + 2);  // b1, b2 (256 each), b3 (128)
  float* inv_s = bias + 640;                              // per ADO: 1 / s
  int* jk = reinterpret_cast<int*>(inv_s + 128);          // per row: its ADO and mode (j << 16 | k), -1 past the last
  float2* rowf = reinterpret_cast<float2*>(jk + 128);     // per row: (n_k + 1) / (ngamma_l + gamma_kk)
  float2* isig = rowf + 128;                              // per mode: 1 / sigma_k
  float2* rho_s = isig + 128;                             // apt * n2: the tile's ADOs
  float* ys = reinterpret_cast<float*>(ring);
  const int kp1 = pack_k(din), ht = pack_rows(h) / 128;
  const int j0 = blockIdx.x * A.apt, na = min(A.apt, A.n_tier - j0), rows = na * K;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t cols = 32;
  while (cols < static_cast<uint32_t>(2 * NR)) cols <<= 1;
  const WeightRing<kTermSlots> W(ring, bar);
  if (threadIdx.x == kThr) {
    W.init();
    mbar_init(done);
    mbar_init_fence();
  }
  if (threadIdx.x < 32) tmem_alloc(tslot, cols);
  fence_before();
  __syncthreads();
  fence_after();
  if (warp == kWarps) {  // the producer
    if (lane == 0) {
      int nc = 0;
      if (W.copy(A.W1, pack_rows(h), kp1, nc) && W.copy(A.W2, pack_rows(h), h, nc))
        W.copy(A.W3, pack_rows(dout), h, nc);
      W.drain(nc);
    }
    return;
  }
  const uint32_t tmem = *tslot;
  const int cur = A.in.ctl ? A.in.ctl->cur : 0;
  const void* ysel = A.in.y_sel == 1 ? A.in.yb[cur] : (A.in.y_sel == 2 ? A.in.yb[1 - cur] : A.in.y_fixed);
  const TB* y = static_cast<const TB*>(ysel);
  // the tile's ADOs, and the scale s of each: sqrt(max_e |rho_l[e]|^2) (a warp per ADO)
  for (int j = warp; j < na; j += kWarps) {
    const TB* yl = y + static_cast<size_t>(A.first + j0 + j) * n2;
    float mx = 0.f;
    for (int e = lane; e < n2; e += 32) {
      const float re = static_cast<float>(yl[e].x), im = static_cast<float>(yl[e].y);
      rho_s[j * n2 + e] = make_float2(re, im);
      mx = fmaxf(mx, re * re + im * im);
    }
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) inv_s[j] = 1.0f / (sqrtf(mx) + 1e-30f);
  }
  for (int i = threadIdx.x; i < h; i += kThr) {
    bias[i] = __ldg(A.b1 + i);
    bias[256 + i] = __ldg(A.b2 + i);
  }
  for (int i = threadIdx.x; i < dout; i += kThr) bias[512 + i] = __ldg(A.b3 + i);
  for (int k = threadIdx.x; k < K; k += kThr) isig[k] = __ldg(tm.isig + k);
  for (int r = threadIdx.x; r < NR; r += kThr) {
    const int j = r / K, k = r - j * K;
    jk[r] = r < rows ? j << 16 | k : -1;
    rowf[r] = r < rows ? __ldg(tm.rowf + static_cast<size_t>(j0) * K + r) : make_float2(0.f, 0.f);
  }
  sync_work();
  // input features: a unit is 8 rows of one element e (its four features: Re
  // and Im of rho / s and of the adiabatic estimate) or of one mode's one-hot
  // column, or of a padding column; a warp's lanes take consecutive columns
  const int nc = n2 + K + kp1 - din;
  for (int u = threadIdx.x; u < nc * ng; u += kThr) {
    const int g = u / nc, c = u - g * nc;
    if (c >= n2) {
      const int k1 = c - n2;  // one-hot column of mode k1, or (k1 >= K) a padding column
      float f[8];
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        const int q = jk[g * 8 + t];
        f[t] = (k1 < K && q >= 0 && (q & 0xffff) == k1) ? 1.f : 0.f;
      }
      const int col = k1 < K ? 2 * n2 + k1 : din + k1 - K;
      *reinterpret_cast<uint4*>(act + act_off(col, g, NR)) = pack8(f);
      continue;
    }
    const int e = c;
    float f0[8], f1[8], f2[8], f3[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const int q = jk[g * 8 + t];
      f0[t] = f1[t] = f2[t] = f3[t] = 0.f;
      if (q >= 0) {
        const int j = q >> 16, k = q & 0xffff;
        const float2 yl = rho_s[j * n2 + e];
        const float inv = inv_s[j];
        const float2 fr = rowf[g * 8 + t];
        f0[t] = yl.x * inv;
        f1[t] = yl.y * inv;
        // the adiabatic estimate (n_k + 1) c_ke rho_e / (ngamma_l + gamma_kk), in FP32
        const float2 cc = __ldg(tm.cke + static_cast<size_t>(k) * n2 + e);
        const float2 cf = make_float2(cc.x * fr.x - cc.y * fr.y, cc.x * fr.y + cc.y * fr.x);
        f2[t] = (cf.x * yl.x - cf.y * yl.y) * inv;
        f3[t] = (cf.x * yl.y + cf.y * yl.x) * inv;
      }
    }
    *reinterpret_cast<uint4*>(act + act_off(e, g, NR)) = pack8(f0);
    *reinterpret_cast<uint4*>(act + act_off(n2 + e, g, NR)) = pack8(f1);
    *reinterpret_cast<uint4*>(act + act_off(2 * n2 + K + e, g, NR)) = pack8(f2);
    *reinterpret_cast<uint4*>(act + act_off(3 * n2 + K + e, g, NR)) = pack8(f3);
  }
  publish();
  uint32_t parity = 0u;
  int taken = 0;
  bool ok = true;
  const int sp = warp & 3;
  for (int layer = 0; layer < 3 && ok; ++layer) {
    const int kp = layer == 0 ? kp1 : h;
    ok = run_layer(W, act, NR, layer < 2 ? ht : 1, kp / kChunkK, tmem, done, parity, taken);
    if (ok && layer < 2) {  // hidden layer: act = GELU(D + bias), 8 rows per step
      for (int i = warp >> 2; i < ht * ng; i += kWarps / 4) {
        const int m = i / ng, g = i - m * ng, o = m * 128 + sp * 32 + lane;
        float v[8];
        g_ld8(tmem + (static_cast<uint32_t>(sp * 32) << 16) + static_cast<uint32_t>(m * NR + g * 8), v);
        if (o < h) {
          const float b = bias[256 * layer + o];
#pragma unroll
          for (int j = 0; j < 8; ++j) v[j] = gelu_f(v[j] + b);
          *reinterpret_cast<uint4*>(act + act_off(o, g, NR)) = pack8(v);
        }
      }
      publish();
    }
  }
  if (ok) {  // the outputs into shared memory (every weight chunk has been read)
    const int o = sp * 32 + lane;
    for (int g = warp >> 2; g < ng; g += kWarps / 4) {
      float v[8];
      g_ld8(tmem + (static_cast<uint32_t>(sp * 32) << 16) + static_cast<uint32_t>(g * 8), v);
      if (o < dout) {
#pragma unroll
        for (int j = 0; j < 8; ++j) ys[(g * 8 + j) * dout + o] = v[j] + bias[512 + o];
      }
    }
  }
  fence_before();
  sync_work();
  fence_after();
  if (threadIdx.x < 32) tmem_free(tmem, cols);
  if (!ok) {
    if (threadIdx.x == 0) atomicExch(A.err, 1);
    return;
  }
  // gain head: the prediction of rho_{n+1_k} for every (row, element)
  const float r_n2 = 1.0f / static_cast<float>(n2);
  for (int i = threadIdx.x; i < rows * n2; i += kThr) {
    // i / n2: i < 2^16, n2 <= 2^12; (i + 0.5) / n2 lies further from an integer than the rounding moves it
    const int r = __float2int_rz(__fmul_rn(static_cast<float>(i) + 0.5f, r_n2)), e = i - r * n2;
    const int j = jk[r] >> 16, k = jk[r] & 0xffff;
    const float sg = __ldg(tm.sgn + static_cast<size_t>(k) * n2 + e);  // sign(Re(v_a - v_b))
    float2 out = make_float2(0.f, 0.f);
    if (sg != 0.f) {
      const float* yr = ys + r * dout;
      const float cr = yr[e], zz = yr[n2 + e];
      const float ci = -sg * (fmaxf(zz, 0.f) + log1pf(expf(-fabsf(zz))));
      const float2 rho = rho_s[j * n2 + e];
      const float rr = rho.x, ri = rho.y;
      const float pr = cr * rr - ci * ri, pi = cr * ri + ci * rr;  // C rho
      const float2 is = isig[k];  // 1 / sigma_k
      out = make_float2(pr * is.x - pi * is.y, pr * is.y + pi * is.x);
    }
    A.P[static_cast<size_t>(j0) * K * n2 + i] = out;
  }
}

// Set-up tables of the inference: rowf[(l - first) K + k] = (n_k + 1) /
// (ngamma_l + gamma_kk) and isig[k] = 1 / sigma_k, formed in FP64.
__global__ void k_term_tables(const TermModel tm, int first, int n_tier, float2* rowf, float2* isig) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n_tier * tm.K) {
    const int j = i / tm.K, k = i - j * tm.K, l = first + j;
    const double2 gk = tm.gdiag[k], gl = tm.ngd[l];
    const double nk1 = static_cast<double>(tm.nidx[static_cast<size_t>(l) * tm.K + k]) + 1.0;
    const double dr = gl.x + gk.x, di = gl.y + gk.y, dd = dr * dr + di * di;
    rowf[i] = dd > 0.0 ? make_float2(static_cast<float>(nk1 * dr / dd), static_cast<float>(-nk1 * di / dd))
                       : make_float2(0.f, 0.f);
  }
  if (i < tm.K) {
    const double2 sk = tm.sigma[i];
    const double sd = sk.x * sk.x + sk.y * sk.y;
    isig[i] = make_float2(static_cast<float>(sk.x / sd), static_cast<float>(-sk.y / sd));
  }
}

// ------------------------------------------------------------------ training
// k_train: a CTA takes 32 rows of the minibatch through forward, loss and the
// backward products over the layers, everything on the chip (pre-activations
// in shared memory in FP32), and writes its operands of the weight gradients
// (the inputs and the gradients of every layer, BF16 core matrices) and its
// rows' bias-gradient sums.  k_dw: a CTA takes a 128 x 64 tile of one layer's
// weight gradient D^T = X^T dZ (inputs along the tensor-memory lanes, so a
// warp stores 32 consecutive entries of a row of dW) and runs through the
// rows in order in one accumulator: the summation order of the GEMM over the
// whole batch, whatever the number of tiles.  k_adam: Adam.
//
// BF16 rounding happens where the operands are written instead of where a
// GEMM reads them: the same values, and every sum (MMAs over the rows in
// steps of 16, bias sums row by row in FP32) keeps the order of the GEMM form,
// so both forms give the same gradients bit for bit.  Bounds: k_train the
// latency of a tile's chain of phases (32 rows, so that a batch of 4096 fills
// 128 SMs); k_dw its serial chain of MMAs (49 cycles each, the operand reads;
// two per 32 rows) and the copies of 12 KB per 32 rows into each SM.
// Measured for the 7-site closure (210-256-256-98, batch 4096): 3360 us a step
// with one GEMM launch per product (three weight-gradient GEMMs on 1 or 2 CTAs
// 1410-1490 us each, three bias sums 230 us each, the others 93 us each); now
// 27.7 us (k_train) + 19.4 us (k_dw) + 4.8 us (k_adam), 75 us a step with the host.
constexpr int kTR = 32;  // rows per CTA of k_train
constexpr int kTrainSlots = 4;

// The operand image in global memory: per field, blocks of columns (128 for
// the layers' inputs, the M operands of k_dw; 64 for the gradients, its N
// operands), each block [tile][columns of the block x 32 rows], so that
// consecutive tiles of a block are one stretch for a bulk copy; then the
// gradients in FP32 for the bias sums, blocks of 32 columns [tile][8][32] of
// four rows each (columns: dz1, dz2, dy).
struct TrainImage {
  unsigned char* base;
  int din, h, dout, tiles;
  __host__ __device__ __forceinline__ size_t a_block() const { return static_cast<size_t>(tiles) * 128 * 2 * kTR; }
  __host__ __device__ __forceinline__ int x_blocks() const { return (pack_k(din) + 127) / 128; }
  // first byte of input field l (0: X, 1: a1, 2: a2) and gradient field l (0: dz1, 1: dz2, 2: dy)
  __host__ __device__ __forceinline__ size_t in_field(int l) const {
    return a_block() * (l == 0 ? 0 : x_blocks() + (l - 1) * (h / 128));
  }
  __host__ __device__ __forceinline__ size_t grad_field(int l) const {
    return in_field(2) + a_block() * (h / 128) + a_block() / 2 * (l * (h / 64));
  }
  __host__ __device__ __forceinline__ size_t f32_field() const { return grad_field(2) + a_block(); }
  __host__ __device__ __forceinline__ int f32_blocks() const { return (2 * h + dout + 31) / 32; }
  __host__ __device__ __forceinline__ size_t f32_block() const { return static_cast<size_t>(tiles) * 4096; }
  __host__ __device__ __forceinline__ size_t bytes() const { return f32_field() + f32_block() * f32_blocks(); }
  // rows 8 g .. of column c, in a tile
  __device__ __forceinline__ uint4* in(int l, int c, int tile, int g) const {
    return reinterpret_cast<uint4*>(base + in_field(l) + a_block() * (c >> 7) + static_cast<size_t>(tile) * 8192 +
                                    act_off(c & 127, g, kTR));
  }
  __device__ __forceinline__ uint4* grad(int l, int c, int tile, int g) const {
    return reinterpret_cast<uint4*>(base + grad_field(l) + a_block() / 2 * (c >> 6) + static_cast<size_t>(tile) * 4096 +
                                    act_off(c & 63, g, kTR));
  }
  // rows 4 r4 .. of gradient column c
  __device__ __forceinline__ float4* f32(int c, int tile, int r4) const {
    return reinterpret_cast<float4*>(base + f32_field() + f32_block() * (c >> 5) + static_cast<size_t>(tile) * 4096) +
           r4 * 32 + (c & 31);
  }
};
// shared memory of k_train: x | a1 | a2 | dz2 | dy | ring | z1 | z2 (FP32) | barriers | y (FP32, kTR x dout) | row terms
__host__ __device__ __forceinline__ size_t train_smem_bytes(int din, int h, int dout) {
  return static_cast<size_t>(2 * kTR) * (pack_k(din) + 3 * h + 128) + kTrainSlots * 16384 +
         sizeof(float) * (2 * static_cast<size_t>(kTR) * h + static_cast<size_t>(kTR) * dout +
                          static_cast<size_t>(kTR) * 65 + kTR + 4) +
         8 * (2 * kTrainSlots + 2) + 16;
}

// z = D + bias (kept in FP32) and act = GELU(z): thread = (output o, half of
// the rows); the activation goes to shared memory and to the operand image.
__device__ __forceinline__ void train_hidden(uint32_t tmem, const float* __restrict__ bias, int h, float4* z,
                                             unsigned char* act, const TrainImage& I, int l, int tile) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sp = warp & 3;
  for (int i = warp >> 2; i < (h >> 7) * 2; i += kWarps / 4) {
    const int m = i >> 1, half = i & 1, o = m * 128 + sp * 32 + lane;
    float v[16];
    g_ld16(tmem + (static_cast<uint32_t>(sp * 32) << 16) + static_cast<uint32_t>(m * kTR + half * 16), v);
    const float b = __ldg(bias + o);
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] += b;
#pragma unroll
    for (int j = 0; j < 4; ++j) z[(half * 4 + j) * h + o] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = gelu_f(v[j]);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const uint4 w = pack8(v + 8 * j);
      *reinterpret_cast<uint4*>(act + act_off(o, half * 2 + j, kTR)) = w;
      *I.in(l, o, tile, half * 2 + j) = w;
    }
  }
}

// dz = D * GELU'(z), to the image in both precisions.
__device__ __forceinline__ void train_dhidden(uint32_t tmem, int h, const float4* z, unsigned char* act,
                                              const TrainImage& I, int l, int tile) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sp = warp & 3;
  for (int i = warp >> 2; i < (h >> 7) * 2; i += kWarps / 4) {
    const int m = i >> 1, half = i & 1, o = m * 128 + sp * 32 + lane;
    float v[16];
    g_ld16(tmem + (static_cast<uint32_t>(sp * 32) << 16) + static_cast<uint32_t>(m * kTR + half * 16), v);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float4 zz = z[(half * 4 + j) * h + o];
      v[4 * j] *= gelu_grad_f(zz.x);
      v[4 * j + 1] *= gelu_grad_f(zz.y);
      v[4 * j + 2] *= gelu_grad_f(zz.z);
      v[4 * j + 3] *= gelu_grad_f(zz.w);
      *I.f32(l * h + o, tile, half * 4 + j) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const uint4 w = pack8(v + 8 * j);
      if (act) *reinterpret_cast<uint4*>(act + act_off(o, half * 2 + j, kTR)) = w;
      *I.grad(l, o, tile, half * 2 + j) = w;
    }
  }
}

__device__ __forceinline__ float softplus_f(float z) { return fmaxf(z, 0.f) + log1pf(expf(-fabsf(z))); }
__device__ __forceinline__ float sigmoid_f(float z) { return 1.f / (1.f + expf(-z)); }

// Loss of the tile's rows and its gradient, in place of the outputs ys (row
// stride dout): a warp takes two rows.  Kind 1: the closure loss (mlp.cu)
// over target rows [Re t, Im t, Re r, Im r, sg]; the sum of a row's weight runs
// over the elements in order (one lane per row), because the BF16 rounding
// downstream turns a last-bit difference there into a visible one.  Kind 0:
// the mean squared error.  rowloss[r] receives the row's loss.
struct TrainTargets {
  float v[2][2][5];  // [row of the warp][element lane + 32 i]: Re t, Im t, Re r, Im r, sg
};
__device__ __forceinline__ void load_targets(TrainTargets& t, const float* __restrict__ T, int r0, int B, int n2) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int q = 0; q < 2; ++q)
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 5; ++j) {
        const int r = r0 + warp * 2 + q, e = lane + 32 * i;
        t.v[q][i][j] = (r < B && e < n2) ? __ldg(T + static_cast<size_t>(r) * 5 * n2 + j * n2 + e) : 0.f;
      }
}
__device__ __forceinline__ float sum_lanes(float v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ void closure_loss(float* ys, const TrainTargets& T, int r0, int B, int dout, int n2,
                                             float* inner, float* rowloss) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int q = 0; q < 2; ++q)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float t0 = T.v[q][i][0], t1 = T.v[q][i][1], t2 = T.v[q][i][2], t3 = T.v[q][i][3];
      const float m = fabsf(T.v[q][i][4]);
      if (lane + 32 * i < n2)
        inner[(warp * 2 + q) * 65 + lane + 32 * i] =
            m * fmaf(1e-2f, fmaf(t2, t2, __fmul_rn(t3, t3)), fmaf(t0, t0, __fmul_rn(t1, t1)));
    }
  __syncwarp();
  float den = 1e-6f;
  if (lane < 2) {
    const float* p = inner + (warp * 2 + lane) * 65;
#pragma unroll 8
    for (int e = 0; e < n2; ++e) den += p[e];
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int r = warp * 2 + q;
    const float dq = __shfl_sync(0xffffffffu, den, q);
    const bool live = r0 + r < B;
    const float w = 2.f / (static_cast<float>(B) * dq);
    float* y = ys + r * dout;
    float num = 0.f;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int e = lane + 32 * i;
      if (e >= n2) continue;
      const float sg = T.v[q][i][4], m = fabsf(sg);
      const float zz = y[n2 + e];
      const float cr = y[e], ci = -sg * softplus_f(zz);
      const float rr = T.v[q][i][2], ri = T.v[q][i][3];
      const float dr = cr * rr - ci * ri - T.v[q][i][0], di = cr * ri + ci * rr - T.v[q][i][1];
      num += m * (dr * dr + di * di);
      // conj(d) r = (dr rr + di ri) + i (dr ri - di rr)
      const float re = dr * rr + di * ri, im = dr * ri - di * rr;
      y[e] = live ? w * m * re : 0.f;
      y[n2 + e] = live ? w * m * sg * sigmoid_f(zz) * im : 0.f;
    }
    num = sum_lanes(num);
    if (lane == 0) rowloss[r] = live ? num / dq : 0.f;
  }
}
__device__ __forceinline__ void mse_loss(float* ys, const float* __restrict__ T, int r0, int B, int dout,
                                         float* rowloss) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float scale = 2.0f / static_cast<float>(static_cast<long long>(B) * dout);
  for (int q = 0; q < 2; ++q) {
    const int r = warp * 2 + q;
    const bool live = r0 + r < B;
    float* y = ys + r * dout;
    float num = 0.f;
    for (int c = lane; c < dout; c += 32) {
      const float d = live ? y[c] - __ldg(T + static_cast<size_t>(r0 + r) * dout + c) : 0.f;
      num += d * d;
      y[c] = scale * d;
    }
    num = sum_lanes(num);
    if (lane == 0) rowloss[r] = num;
  }
}

__global__ void __launch_bounds__(kThrAll, 1) k_train(const TrainArgs A) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int din = A.din, h = A.h, dout = A.dout, B = A.B;
  const int kp1 = pack_k(din), kp3 = pack_k(dout);
  unsigned char* xb = smem_raw;
  unsigned char* a1 = xb + static_cast<size_t>(2 * kTR) * kp1;
  unsigned char* a2 = a1 + static_cast<size_t>(2 * kTR) * h;
  unsigned char* dz2 = a2 + static_cast<size_t>(2 * kTR) * h;
  unsigned char* dy = dz2 + static_cast<size_t>(2 * kTR) * h;
  unsigned char* ring = dy + 2 * kTR * 128;
  float4* z1 = reinterpret_cast<float4*>(ring + kTrainSlots * 16384);
  float4* z2 = z1 + static_cast<size_t>(kTR) * h / 4;
  uint64_t* bar = reinterpret_cast<uint64_t*>(z2 + static_cast<size_t>(kTR) * h / 4);
  uint64_t* done = bar + 2 * kTrainSlots;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(done + 1);
  float* ys = reinterpret_cast<float*>(done + 2);  // kTR x dout
  float* inner = ys + kTR * dout;                  // kTR x 65
  float* rowloss = inner + kTR * 65;               // kTR
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sp = warp & 3, ht = h >> 7;
  const int tile = blockIdx.x, r0 = tile * kTR;
  const WeightRing<kTrainSlots> W(ring, bar);
  if (threadIdx.x == kThr) {
    W.init();
    mbar_init(done);
    mbar_init_fence();
  }
  if (threadIdx.x < 32) tmem_alloc(tslot, 64u);
  fence_before();
  __syncthreads();
  fence_after();
  if (warp == kWarps) {  // the producer
    if (lane == 0) {
      int n = 0;
      if (W.copy(A.W1, h, kp1, n) && W.copy(A.W2, h, h, n) && W.copy(A.W3, 128, h, n) && W.copy(A.W3t, h, kp3, n))
        W.copy(A.W2t, h, h, n);
      W.drain(n);
    }
    return;
  }
  const uint32_t tmem = *tslot;
  const TrainImage I{A.img, din, h, dout, static_cast<int>(gridDim.x)};
  // the rows' inputs: 8 rows of one column per step, lanes along the columns
  for (int u = threadIdx.x; u < kp1 * (kTR / 8); u += kThr) {
    const int g = u / kp1, c = u - g * kp1;
    float f[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const int r = r0 + g * 8 + t;
      f[t] = (r < B && c < din) ? __ldg(A.X + static_cast<size_t>(r) * din + c) : 0.f;
    }
    const uint4 w = pack8(f);
    *reinterpret_cast<uint4*>(xb + act_off(c, g, kTR)) = w;
    *I.in(0, c, tile, g) = w;
  }
  publish();
  uint32_t parity = 0u;
  int taken = 0;
  bool ok = run_layer(W, xb, kTR, ht, kp1 / kChunkK, tmem, done, parity, taken);
  if (ok) {
    train_hidden(tmem, A.b1, h, z1, a1, I, 1, tile);
    publish();
    ok = run_layer(W, a1, kTR, ht, h / kChunkK, tmem, done, parity, taken);
  }
  if (ok) {
    train_hidden(tmem, A.b2, h, z2, a2, I, 2, tile);
    publish();
    TrainTargets T;
    if (A.kind == 1) load_targets(T, A.T, r0, B, A.n2);
    ok = run_layer(W, a2, kTR, 1, h / kChunkK, tmem, done, parity, taken);
    if (ok) {
      const int o = sp * 32 + lane;
      if (warp < 8) {
        float v[16];
        const int half = warp >> 2;
        g_ld16(tmem + (static_cast<uint32_t>(sp * 32) << 16) + static_cast<uint32_t>(half * 16), v);
        if (o < dout) {
          const float b = __ldg(A.b3 + o);
#pragma unroll
          for (int j = 0; j < 16; ++j) ys[(half * 16 + j) * dout + o] = v[j] + b;
        }
      }
      fence_before();
      sync_work();
      if (A.kind == 1)
        closure_loss(ys, T, r0, B, dout, A.n2, inner, rowloss);
      else
        mse_loss(ys, A.T, r0, B, dout, rowloss);
      sync_work();
      {  // the gradient as an operand (columns past dout are zero)
        const int c = threadIdx.x & 127, g = threadIdx.x >> 7;
        float f[8];
#pragma unroll
        for (int t = 0; t < 8; ++t) f[t] = c < dout ? ys[(g * 8 + t) * dout + c] : 0.f;
        const uint4 w = pack8(f);
        *reinterpret_cast<uint4*>(dy + act_off(c, g, kTR)) = w;
        *I.grad(2, c, tile, g) = w;
        if (2 * h + c < 32 * I.f32_blocks()) {
          *I.f32(2 * h + c, tile, 2 * g) = make_float4(f[0], f[1], f[2], f[3]);
          *I.f32(2 * h + c, tile, 2 * g + 1) = make_float4(f[4], f[5], f[6], f[7]);
        }
      }
      if (warp == kWarps - 1) {
        const float s = sum_lanes(rowloss[lane]);
        if (lane == 0) A.loss[tile] = s;
      }
      publish();
      ok = run_layer(W, dy, kTR, ht, kp3 / kChunkK, tmem, done, parity, taken);
    }
  }
  if (ok) {
    train_dhidden(tmem, h, z2, dz2, I, 1, tile);
    publish();
    ok = run_layer(W, dz2, kTR, ht, h / kChunkK, tmem, done, parity, taken);
  }
  if (ok)
    train_dhidden(tmem, h, z1, nullptr, I, 0, tile);
  else if (threadIdx.x == 0)
    atomicExch(A.err, 1);
  fence_before();
  sync_work();
  fence_after();
  if (threadIdx.x < 32) tmem_free(tmem, 64u);
}

// Weight and bias gradients into A.g.  A slot of the ring holds four tiles
// (128 rows): 32 KB of the M operand and 16 KB of the N operand.
constexpr int kDwSlots = 4, kDwTiles = 4, kDwThr = 256, kDwN = 64;
constexpr int kDwA = kDwTiles * 8192, kDwSlot = kDwA + kDwTiles * 4096;
constexpr size_t kDwSmem = static_cast<size_t>(kDwSlots) * kDwSlot + 8 * (2 * kDwSlots + 1);
struct DwTile {
  int l, i0, o0, n, n_i, n_o;  // layer, first input and output, columns of the MMA, the layer's sizes
};
// tile `id` of the three layers' weight gradients (128 inputs x kDwN outputs); false past the last
__host__ __device__ __forceinline__ bool dw_tile(int id, int din, int h, int dout, DwTile& t) {
  for (int l = 0; l < 3; ++l) {
    t.l = l;
    t.n_i = l == 0 ? din : h;
    t.n_o = l == 2 ? dout : h;
    const int mt = (t.n_i + 127) / 128, nt = (t.n_o + kDwN - 1) / kDwN;
    if (id < mt * nt) {
      t.i0 = id / nt * 128;
      t.o0 = id % nt * kDwN;
      t.n = ((t.n_o - t.o0 < kDwN ? t.n_o - t.o0 : kDwN) + 15) / 16 * 16;
      return true;
    }
    id -= mt * nt;
  }
  return false;
}

__global__ void __launch_bounds__(kDwThr, 1) k_dw(const TrainArgs A, int n_tiles, int n_dw) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ uint32_t tslot;
  const bool bias = static_cast<int>(blockIdx.x) >= n_dw;  // a CTA of the bias sums: 32 columns
  DwTile t{};
  if (!bias) dw_tile(blockIdx.x, A.din, A.h, A.dout, t);
  const TrainImage I{A.img, A.din, A.h, A.dout, n_tiles};
  uint64_t* full = reinterpret_cast<uint64_t*>(smem_raw + kDwSlots * kDwSlot);
  uint64_t* empty = full + kDwSlots;
  uint64_t* done = empty + kDwSlots;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == 0) tmem_alloc(&tslot, kDwN);
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2 * kDwSlots + 1; ++i) mbar_init(full + i);
    mbar_init_fence();
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = tslot;
  const int nb = (n_tiles + kDwTiles - 1) / kDwTiles;
  bool mine = true;
  if (threadIdx.x == 0) {  // the copies
    const unsigned char* pa = bias ? I.base + I.f32_field() + I.f32_block() * (blockIdx.x - n_dw)
                                   : I.base + I.in_field(t.l) + I.a_block() * (t.i0 >> 7);
    const unsigned char* pb = I.base + I.grad_field(t.l) + I.a_block() / 2 * (t.o0 >> 6);
    int i = 0;
    for (; i < nb; ++i) {
      const int s = i & (kDwSlots - 1), nt = min(kDwTiles, n_tiles - i * kDwTiles);
      if (i >= kDwSlots && !g_wait(empty + s, static_cast<uint32_t>(i / kDwSlots - 1) & 1u)) {
        mine = false;
        break;
      }
      unsigned char* slot = smem_raw + s * kDwSlot;
      const uint32_t ab = static_cast<uint32_t>(nt) * (bias ? 4096u : 8192u), bb = bias ? 0u : nt * 4096u;
      expect_bytes(full + s, ab + bb);
      bulk_load(slot, pa, ab, full + s);
      pa += ab;
      if (bb) bulk_load(slot + kDwA, pb, bb, full + s);
      pb += bb;
    }
    for (int c = max(0, i - kDwSlots); c < i; ++c)  // the copies in flight land before the CTA leaves
      g_wait(full + (c & (kDwSlots - 1)), static_cast<uint32_t>(c / kDwSlots) & 1u);
  } else if (warp == 1 && bias) {  // a lane: a column; its rows in order, in FP32
    float sum = 0.f;
    for (int i = 0; i < nb && mine; ++i) {
      const int s = i & (kDwSlots - 1), nt = min(kDwTiles, n_tiles - i * kDwTiles);
      mine = __all_sync(0xffffffffu, g_wait(full + s, static_cast<uint32_t>(i / kDwSlots) & 1u) != 0);
      if (!mine) break;
      const float4* v = reinterpret_cast<const float4*>(smem_raw + s * kDwSlot) + lane;
#pragma unroll 8
      for (int r = 0; r < nt * 8; ++r) {
        const float4 x = v[r * 32];
        sum += x.x;
        sum += x.y;
        sum += x.z;
        sum += x.w;
      }
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(s_addr(empty + s)) : "memory");
    }
    const int c = (blockIdx.x - n_dw) * 32 + lane;
    if (mine && c < 2 * A.h + A.dout)
      A.g[c < A.h ? A.off[1] + c : c < 2 * A.h ? A.off[3] + c - A.h : A.off[5] + c - 2 * A.h] = sum;
  } else if (warp == 1) {  // the MMAs
    if (elect_one()) {
      const uint32_t idesc = g_idesc(t.n, 0, 0);
      const uint64_t d0 = g_desc(s_addr(smem_raw), 128, 512);
      for (int i = 0; i < nb && mine; ++i) {
        const int s = i & (kDwSlots - 1), nt = min(kDwTiles, n_tiles - i * kDwTiles);
        mine = g_wait(full + s, static_cast<uint32_t>(i / kDwSlots) & 1u) != 0;
        if (!mine) break;
        const uint64_t da = d0 + s * (kDwSlot >> 4), db = da + (kDwA >> 4);
        for (int q = 0; q < nt; ++q) {
          g_mma(tmem, da + q * (8192 >> 4), db + q * (4096 >> 4), idesc, (i > 0 || q > 0) ? 1 : 0);
          g_mma(tmem, da + q * (8192 >> 4) + 16, db + q * (4096 >> 4) + 16, idesc, 1);
        }
        g_commit(empty + s);
      }
      g_commit(done);
      mine = g_wait(done, 0u) && mine;  // on failure: what is in flight ends, bounded
    }
    __syncwarp();
  }
  const bool ok = __syncthreads_and(mine) != 0;
  fence_after();
  if (ok && !bias) {
    const int sp = warp & 3, i = t.i0 + sp * 32 + lane;
    float* g = A.g + A.off[2 * t.l];
    for (int q = (warp >> 2) * 8; q < t.n; q += 8 * (kDwThr / 128)) {
      float v[8];
      g_ld8(tmem + (static_cast<uint32_t>(sp * 32) << 16) + static_cast<uint32_t>(q), v);
      if (i < t.n_i) {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (t.o0 + q + j < t.n_o) g[static_cast<long long>(t.o0 + q + j) * t.n_i + i] = v[j];
      }
    }
  } else if (!ok && threadIdx.x == 0) {
    atomicExch(A.err, 1);
  }
  fence_before();
  __syncthreads();
  fence_after();
  if (warp == 0) tmem_free(tmem, kDwN);
}

// parameter i takes the value v in every BF16 copy
__device__ __forceinline__ void store_weight(const WeightStore& W, long long i, float v) {
  const __nv_bfloat16 b = __float2bfloat16(v);
  W.wb[i] = b;
  if (!W.f[0]) return;
  if (i < W.off[1]) {
    const int o = static_cast<int>(i / W.din), k = static_cast<int>(i - static_cast<long long>(o) * W.din);
    W.f[0][pack_index(pack_rows(W.h), o, k)] = b;
  } else if (i >= W.off[2] && i < W.off[3]) {
    const int x = static_cast<int>(i - W.off[2]), o = x / W.h, k = x - o * W.h;
    W.f[1][pack_index(pack_rows(W.h), o, k)] = b;
    W.t[0][pack_index(pack_rows(W.h), k, o)] = b;
  } else if (i >= W.off[4] && i < W.off[5]) {
    const int x = static_cast<int>(i - W.off[4]), o = x / W.h, k = x - o * W.h;
    W.f[2][pack_index(pack_rows(W.dout), o, k)] = b;
    W.t[1][pack_index(pack_rows(W.h), k, o)] = b;
  }
}

// Adam on the FP32 masters and every BF16 copy.
__global__ void __launch_bounds__(256) k_adam(const AdamArgs A) {
  if (*A.err) return;  // a wait ran out: the weights stay
  const long long i = blockIdx.x * 256ll + threadIdx.x;
  if (i >= A.n_params) return;
  const float gi = A.g[i];
  const float mi = fmaf(1.f - A.b1, gi, __fmul_rn(A.b1, A.m[i]));
  const float vi = fmaf(__fmul_rn(1.f - A.b2, gi), gi, __fmul_rn(A.b2, A.v[i]));
  A.m[i] = mi;
  A.v[i] = vi;
  const float wi = A.w[i] - A.lr * (mi / A.c1) / (sqrtf(vi / A.c2) + A.eps);
  A.w[i] = wi;
  store_weight(A.wt, i, wi);
}

__global__ void k_weights(const float* __restrict__ w, const WeightStore wt, long long n) {
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x)
    store_weight(wt, i, w[i]);
}

}  // namespace

bool closure_sizes_ok(int din, int h, int dout) { return din <= 256 && h % 64 == 0 && h >= 64 && h <= 256 && dout <= 128; }

size_t closure_pack_elems(int which, int din, int h, int dout) {
  const int rows = which == 2 ? dout : h, k = which == 0 ? din : which == 4 ? dout : h;
  return static_cast<size_t>(pack_rows(rows)) * pack_k(k);
}

bool term_fused_ok(int din, int h, int dout, int K, int n2) {
  return closure_sizes_ok(din, h, dout) && K >= 1 && K <= 128 && term_smem_bytes(1, K, n2) <= kMaxSmem;
}

bool train_fused_ok(int din, int h, int dout, int kind, int n2) {
  return closure_sizes_ok(din, h, dout) && h % 128 == 0 && (kind == 0 || (n2 <= 64 && dout == 2 * n2)) &&
         train_smem_bytes(din, h, dout) <= kMaxSmem;
}

cudaError_t launch_term_tables(const TermModel& tm, int first, int n_tier, float2* rowf, float2* isig, cudaStream_t s) {
  const int total = std::max(n_tier * tm.K, tm.K);
  if (total <= 0) return cudaSuccess;
  k_term_tables<<<(total + 127) / 128, 128, 0, s>>>(tm, first, n_tier, rowf, isig);
  ++g_launches;
  return cudaGetLastError();
}

cudaError_t launch_term_fused(TermMlpArgs a, int n_sm, bool y_float, cudaStream_t s) {
  if (a.n_tier <= 0) return cudaSuccess;
  // as few ADOs per CTA as one wave takes (at most 128 rows)
  const int n2 = a.tm.n * a.tm.n, K = a.tm.K;
  a.apt = std::max(1, std::min(128 / K, (a.n_tier + n_sm - 1) / n_sm));
  while (a.apt > 1 && term_smem_bytes(a.apt, K, n2) > kMaxSmem) --a.apt;
  const size_t smem = term_smem_bytes(a.apt, K, n2);
  const int grid = (a.n_tier + a.apt - 1) / a.apt;
  const void* kern = y_float ? reinterpret_cast<const void*>(k_term_mlp<float2>)
                             : reinterpret_cast<const void*>(k_term_mlp<double2>);
  cudaError_t e = allow_smem(kern);
  if (e != cudaSuccess) return e;
  if (y_float)
    k_term_mlp<float2><<<grid, kThrAll, smem, s>>>(a);
  else
    k_term_mlp<double2><<<grid, kThrAll, smem, s>>>(a);
  ++g_launches;
  return cudaGetLastError();
}

int train_tiles(int batch) { return (batch + kTR - 1) / kTR; }
size_t train_image_bytes(int din, int h, int dout, int tiles) { return TrainImage{nullptr, din, h, dout, tiles}.bytes(); }

cudaError_t launch_train(const TrainArgs& a, cudaStream_t s) {
  const size_t smem = train_smem_bytes(a.din, a.h, a.dout);
  const int tiles = train_tiles(a.B);
  cudaError_t e = allow_smem(reinterpret_cast<const void*>(k_train));
  if (e != cudaSuccess) return e;
  e = allow_smem(reinterpret_cast<const void*>(k_dw));
  if (e != cudaSuccess) return e;
  k_train<<<tiles, kThrAll, smem, s>>>(a);
  int n = 0;
  DwTile t;
  while (dw_tile(n, a.din, a.h, a.dout, t)) ++n;
  k_dw<<<n + TrainImage{nullptr, a.din, a.h, a.dout, tiles}.f32_blocks(), kDwThr, kDwSmem, s>>>(a, tiles, n);
  g_launches += 2;
  return cudaGetLastError();
}

cudaError_t launch_adam(const AdamArgs& a, cudaStream_t s) {
  k_adam<<<static_cast<unsigned>((a.n_params + 255) / 256), 256, 0, s>>>(a);
  ++g_launches;
  return cudaGetLastError();
}

cudaError_t launch_weights(const float* w, const WeightStore& wt, long long n, cudaStream_t s) {
  const int grid = static_cast<int>(std::max<long long>(1, std::min<long long>((n + 255) / 256, 1024)));
  k_weights<<<grid, 256, 0, s>>>(w, wt, n);
  ++g_launches;
  return cudaGetLastError();
}

}  // namespace heomgb
