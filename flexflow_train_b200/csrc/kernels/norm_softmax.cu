// norm_softmax.cu -- row-wise kernels: LayerNorm fwd/bwd (with the dX pass the
// reference defines but never launches, lib/kernels/src/cuda/ops/layer_norm_kernels.cu:163),
// softmax fwd/bwd (replaces cudnnSoftmaxForward, softmax_kernels.cu:57), fused
// softmax + sparse categorical cross-entropy, and the loss-gradient kernels of
// lib/kernels/src/cuda/loss_function_kernels.cu:21-51.
//
// All kernels take bf16 or fp32 activations (dt: 0 = fp32, 1 = bf16) and keep
// statistics in fp32.
#include "common.cuh"
#include "rowwise_vec.cuh"
#include "tcgen05.cuh"

namespace {

template <typename T> __device__ __forceinline__ float ldf(const T *p);
template <> __device__ __forceinline__ float ldf<float>(const float *p) { return *p; }
template <> __device__ __forceinline__ float ldf<bf16>(const bf16 *p) { return bf2f(*p); }
template <typename T> __device__ __forceinline__ void stf(T *p, float v);
template <> __device__ __forceinline__ void stf<float>(float *p, float v) { *p = v; }
template <> __device__ __forceinline__ void stf<bf16>(bf16 *p, float v) { *p = f2bf(v); }

// ------------------------------------------------------------------ LayerNorm
// y = LN(a + b) * gamma + beta ; b optional (fused residual add); when b is
// given and xsum is non-null the sum a + b is written too (backward needs it).
template <typename T>
__global__ void layernorm_fwd_kernel(const T *a, const T *b, const T *gamma,
                                     const T *beta, T *__restrict__ xsum, T *__restrict__ y,
                                     float *__restrict__ mean, float *__restrict__ rstd, int rows, int cols,
                                     float eps) {
  pdl_entry();
  __shared__ float red[32];
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const T *pa = a + (long long)row * cols;
    const T *pb = b ? b + (long long)row * cols : nullptr;
    float s = 0.f, ss = 0.f;
    for (int c = threadIdx.x; c < cols; c += blockDim.x) {
      float v = ldf(pa + c) + (pb ? ldf(pb + c) : 0.f);
      if (pb && xsum) {
        stf(xsum + (long long)row * cols + c, v);
        v = ldf(xsum + (long long)row * cols + c);  // statistics of the rounded value backward will see
      }
      s += v;
      ss += v * v;
    }
    s = block_sum(s, red);
    ss = block_sum(ss, red);
    float mu = s / cols;
    float var = fmaxf(ss / cols - mu * mu, 0.f);
    float rs = rsqrtf(var + eps);
    if (threadIdx.x == 0) {
      if (mean) mean[row] = mu;
      if (rstd) rstd[row] = rs;
    }
    const T *px = (pb && xsum) ? xsum + (long long)row * cols : pa;
    for (int c = threadIdx.x; c < cols; c += blockDim.x) {
      float v = (pb && !xsum) ? ldf(pa + c) + ldf(pb + c) : ldf(px + c);
      float o = (v - mu) * rs;
      if (gamma) o = o * ldf(gamma + c) + (beta ? ldf(beta + c) : 0.f);
      stf(y + (long long)row * cols + c, o);
    }
  }
}

// One pass over (dy, x): writes dx and per-block partial column sums of
// dgamma / dbeta into scratch `partial` laid out [2][gridDim.x][cols].
// Thread t owns columns t, t+blockDim, ... (at most KMAX of them).
template <typename T, int KMAX>
__global__ void layernorm_bwd_kernel(const T *dy, const T *x, const T *gamma,
                                     const float *mean, const float *rstd,
                                     T *__restrict__ dx, T *__restrict__ dx2, float *__restrict__ partial, int rows,
                                     int cols, int accumulate_dx, int accumulate_dx2) {
  pdl_entry(dx, dx2);
  __shared__ float red[32];
  float dg[KMAX], db[KMAX];
#pragma unroll
  for (int k = 0; k < KMAX; ++k) { dg[k] = 0.f; db[k] = 0.f; }
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const T *pdy = dy + (long long)row * cols;
    const T *px = x + (long long)row * cols;
    float mu = mean[row], rs = rstd[row];
    float s1 = 0.f, s2 = 0.f;
    float vg[KMAX], vx[KMAX];
#pragma unroll
    for (int k = 0; k < KMAX; ++k) {
      int c = threadIdx.x + k * blockDim.x;
      if (c < cols) {
        float g = ldf(pdy + c);
        float xh = (ldf(px + c) - mu) * rs;
        dg[k] += g * xh;
        db[k] += g;
        float gg = gamma ? g * ldf(gamma + c) : g;
        vg[k] = gg;
        vx[k] = xh;
        s1 += gg;
        s2 += gg * xh;
      }
    }
    s1 = block_sum(s1, red);
    s2 = block_sum(s2, red);
    float m1 = s1 / cols, m2 = s2 / cols;
#pragma unroll
    for (int k = 0; k < KMAX; ++k) {
      int c = threadIdx.x + k * blockDim.x;
      if (c < cols) {
        float o = rs * (vg[k] - m1 - vx[k] * m2);
        T *pdx = dx + (long long)row * cols + c;
        stf(pdx, accumulate_dx ? ldf(pdx) + o : o);
        if (dx2) {  // second consumer of the same gradient (the other operand of a fused residual add)
          T *pdx2 = dx2 + (long long)row * cols + c;
          stf(pdx2, accumulate_dx2 ? ldf(pdx2) + o : o);
        }
      }
    }
  }
  if (partial) {
#pragma unroll
    for (int k = 0; k < KMAX; ++k) {
      int c = threadIdx.x + k * blockDim.x;
      if (c < cols) {
        partial[(long long)blockIdx.x * cols + c] = dg[k];
        partial[((long long)gridDim.x + blockIdx.x) * cols + c] = db[k];
      }
    }
  }
}
// ------------------------------------------------------------------ Softmax
// y = softmax(scale * x) over the last dim.  causal_q > 0: row r is query
// position (r % causal_q) and keys past it are masked out.
template <typename T>
__global__ void softmax_fwd_kernel(const T *x, T *__restrict__ y, int rows, int cols, float scale,
                                   int causal_q) {
  pdl_entry();
  __shared__ float red[32];
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const T *px = x + (long long)row * cols;
    int limit = causal_q > 0 ? min(cols, (row % causal_q) + 1) : cols;
    float mx = -INFINITY;
    for (int c = threadIdx.x; c < limit; c += blockDim.x) mx = fmaxf(mx, ldf(px + c) * scale);
    mx = block_max(mx, red);
    float s = 0.f;
    for (int c = threadIdx.x; c < limit; c += blockDim.x) s += __expf(ldf(px + c) * scale - mx);
    s = block_sum(s, red);
    float inv = 1.f / s;
    T *py = y + (long long)row * cols;
    for (int c = threadIdx.x; c < cols; c += blockDim.x)
      stf(py + c, c < limit ? __expf(ldf(px + c) * scale - mx) * inv : 0.f);
  }
}
// dx = scale * y * (dy - sum(dy * y))
template <typename T>
__global__ void softmax_bwd_kernel(const T *dy, const T *y, T *__restrict__ dx, int rows,
                                   int cols, float scale) {
  pdl_entry();
  __shared__ float red[32];
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const T *pdy = dy + (long long)row * cols;
    const T *py = y + (long long)row * cols;
    float s = 0.f;
    for (int c = threadIdx.x; c < cols; c += blockDim.x) s += ldf(pdy + c) * ldf(py + c);
    s = block_sum(s, red);
    T *pdx = dx + (long long)row * cols;
    for (int c = threadIdx.x; c < cols; c += blockDim.x) stf(pdx + c, scale * ldf(py + c) * (ldf(pdy + c) - s));
  }
}

// Fused softmax + sparse categorical cross-entropy: per-row loss, optional
// probabilities, and dlogits = (p - onehot(label)) * grad_scale.  Rows whose
// label is negative contribute no loss and no gradient.
template <typename T, typename L>
__global__ void softmax_ce_kernel(const T *logits, const L *labels, T *__restrict__ probs,
                                  T *__restrict__ dlogits, float *__restrict__ loss, int rows, int cols,
                                  float grad_scale) {
  pdl_entry();
  __shared__ float red[32];
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const T *px = logits + (long long)row * cols;
    long long label = (long long)labels[row];
    float mx = -INFINITY;
    for (int c = threadIdx.x; c < cols; c += blockDim.x) mx = fmaxf(mx, ldf(px + c));
    mx = block_max(mx, red);
    float s = 0.f;
    for (int c = threadIdx.x; c < cols; c += blockDim.x) s += __expf(ldf(px + c) - mx);
    s = block_sum(s, red);
    float inv = 1.f / s;
    bool valid = label >= 0 && label < cols;
    if (threadIdx.x == 0 && loss) loss[row] = valid ? (__logf(s) + mx - ldf(px + label)) : 0.f;
    for (int c = threadIdx.x; c < cols; c += blockDim.x) {
      float p = __expf(ldf(px + c) - mx) * inv;
      if (probs) stf(probs + (long long)row * cols + c, p);
      if (dlogits) stf(dlogits + (long long)row * cols + c, valid ? (p - (c == label ? 1.f : 0.f)) * grad_scale : 0.f);
    }
  }
}

// bf16 rows of up to 4096 with cols % 8 == 0: the row stays in registers between the loss and the gradient (one block per row,
// see rowwise_vec.cuh).
constexpr int ROW_THREADS = 128;
template <int VPT, typename L>
__global__ void __launch_bounds__(ROW_THREADS) softmax_ce_row_kernel(const bf16 *logits, const L *labels,
                                                                bf16 *__restrict__ probs, bf16 *__restrict__ dlogits,
                                                                float *__restrict__ loss, int cols, float grad_scale) {
  pdl_entry();
  __shared__ float red[64];
  const int nvec = cols >> 3;
  const long long base = (long long)blockIdx.x * cols;
  uint4 u[VPT];
  vec::row_load<VPT>(logits + base, nvec, u);
  const long long label = (long long)labels[blockIdx.x];
  const bool valid = label >= 0 && label < cols;
  const float at_label = valid ? bf2f(logits[base + label]) : 0.f;  // before dlogits is written: it may be the same buffer
  float m, s;
  vec::row_max_sum<VPT>(u, nvec, red, m, s);
  const float inv = 1.f / s;
  if (threadIdx.x == 0 && loss) loss[blockIdx.x] = valid ? (__logf(s) + m - at_label) : 0.f;
  if (!probs && !dlogits) return;
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int c = i * blockDim.x + threadIdx.x;
    if (c < nvec) {
      float v[8];
      vec::unpack8(u[i], v);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = __expf(v[j] - m) * inv;
      if (probs) vec::st8(probs + base + c * 8, v);
      if (dlogits) {
        const int hit = valid ? (int)label - c * 8 : -1;
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = valid ? (v[j] - (j == hit ? 1.f : 0.f)) * grad_scale : 0.f;
        vec::st8(dlogits + base + c * 8, v);
      }
    }
  }
}

// Wide rows (4096 < cols <= 32768, a vocabulary): persistent blocks whose next rows travel into a ring in shared memory by bulk
// copies while the current one is reduced and written.  Bound by HBM (one read, one write per element).  Holding the row in
// registers alone leaves nothing in flight between a block's phases (cross-entropy of 8192 x 30528: 294 us; a running maximum with
// the row read twice: 254 us; softmax of 4004 x 32000: 144 us, three passes of 2-byte loads: 549 us), and forming each
// exponential twice makes the special-function unit (16 a clock and SM) as slow as the memory.  Here each is formed once, in
// fp32 registers: four 16-byte pieces per thread, 1024 threads per SM in blocks of 256, 512 or 1024 (113 us for the softmax).
constexpr int WIDE_VPT = 4;
constexpr int WIDE_SMEM = 220 * 1024;   // of one SM, shared by its blocks
__device__ int g_rows_err = 0;
template <bool CE, typename L>
__global__ void __launch_bounds__(1024, 1) softmax_wide_kernel(const bf16 *x, const L *labels, bf16 *__restrict__ probs,
                                                               bf16 *__restrict__ dlogits, float *__restrict__ loss, int rows, int cols,
                                                               float scale, float grad_scale, int depth, unsigned long long wait_ns) {
  pdl_entry();
  extern __shared__ __align__(128) uint8_t wide_smem[];
  __shared__ float red[64];
  __shared__ uint64_t full[4];
  __shared__ int abort_flag;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int nvec = cols >> 3;
  const uint32_t row_bytes = (uint32_t)cols * 2u;
  auto fetch = [&](int row, int stage) {   // one thread; row_bytes and both addresses are multiples of 16
    mbar_expect_tx(&full[stage], row_bytes);
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(wide_smem) + (uint32_t)stage * row_bytes),
                 "l"(x + (long long)row * cols), "r"(row_bytes), "r"(smem_u32(&full[stage]))
                 : "memory");
  };
  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int s = 0; s < depth; ++s) mbar_init(&full[s], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (int s = 0; s < depth; ++s)
      if ((long long)blockIdx.x + (long long)s * gridDim.x < rows) fetch(blockIdx.x + s * gridDim.x, s);
  }
  __syncthreads();
  int stage = 0;
  uint32_t phase = 0;
  for (long long row = blockIdx.x; row < rows; row += gridDim.x) {
    const long long label = CE ? (long long)labels[row] : -1;  // asked for before the wait, which no load passes
    const bool ok = mbar_wait(&full[stage], phase, &abort_flag, &g_rows_err, FFK_ERR_TIMEOUT_PRODUCER, wait_ns);
    const uint4 *src = reinterpret_cast<const uint4 *>(wide_smem + (size_t)stage * row_bytes);
    float v[WIDE_VPT][8];
    float m = -INFINITY;
#pragma unroll
    for (int i = 0; i < WIDE_VPT; ++i) {
      const int c = i * blockDim.x + threadIdx.x;
      if (c < nvec) {
        vec::unpack8(src[c], v[i]);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          v[i][j] *= scale;
          m = fmaxf(m, v[i][j]);
        }
      }
    }
    bool valid = false;
    float at_label = 0.f;
    if (CE) {
      valid = label >= 0 && label < cols;
      if (valid && threadIdx.x == 0) at_label = bf2f(reinterpret_cast<const bf16 *>(src)[label]);
    }
    m = warp_max(m);
    if (lane == 0) red[wid] = m;
    // past this barrier the row's stage is free; a copy that did not come (ok is false) ends the block here
    if (__syncthreads_or(!ok)) {
      if (threadIdx.x == 0)   // the copies in flight land, or a second limit runs out, before the shared memory goes away
        for (int a = 0; a < depth && row + (long long)a * gridDim.x < rows; ++a) {
          const int k = stage + a < depth ? stage + a : stage + a - depth;
          const uint64_t t0 = ffk_globaltimer();
          while (!mbar_try_wait(&full[k], k >= stage ? phase : phase ^ 1) && ffk_globaltimer() - t0 < WAIT_LIMIT_NS) {}
        }
      __syncthreads();
      // the rows this block leaves undone are no numbers, so that what an earlier call left there does not pass for results
      const uint4 nan8 = make_uint4(0x7FFF7FFFu, 0x7FFF7FFFu, 0x7FFF7FFFu, 0x7FFF7FFFu);
      for (long long r = row; r < rows; r += gridDim.x) {
        if (CE && threadIdx.x == 0 && loss) loss[r] = __int_as_float(0x7FFFFFFF);
        for (int c = threadIdx.x; c < nvec; c += blockDim.x) {
          if (probs) reinterpret_cast<uint4 *>(probs + r * cols)[c] = nan8;
          if (CE && dlogits) reinterpret_cast<uint4 *>(dlogits + r * cols)[c] = nan8;
        }
      }
      return;
    }
    if (threadIdx.x == 0 && row + (long long)depth * gridDim.x < rows) fetch((int)(row + (long long)depth * gridDim.x), stage);
    m = warp_max(red[lane < nw ? lane : 0]);
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < WIDE_VPT; ++i)
      if (i * blockDim.x + threadIdx.x < nvec) {
        float a = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          v[i][j] = __expf(v[i][j] - m);
          a += v[i][j];
        }
        s += a;
      }
    s = warp_sum(s);
    if (lane == 0) red[32 + wid] = s;
    __syncthreads();
    s = warp_sum(lane < nw ? red[32 + lane] : 0.f);
    const float inv = 1.f / s;
    if (CE && threadIdx.x == 0 && loss) loss[row] = valid ? (__logf(s) + m - at_label) : 0.f;
    const long long base = row * cols;
#pragma unroll
    for (int i = 0; i < WIDE_VPT; ++i) {
      const int c = i * blockDim.x + threadIdx.x;
      if (c < nvec) {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[i][j] *= inv;
        if (probs) vec::st8(probs + base + c * 8, v[i]);
        if (CE && dlogits) {
          const int hit = valid ? (int)label - c * 8 : -1;
#pragma unroll
          for (int j = 0; j < 8; ++j) v[i][j] = valid ? (v[i][j] - (j == hit ? 1.f : 0.f)) * grad_scale : 0.f;
          vec::st8(dlogits + base + c * 8, v[i]);
        }
      }
    }
    if (++stage == depth) { stage = 0; phase ^= 1; }
  }
}

// Rows that the ring does not hold twice (more than 32768, cols % 8 == 0), and those above 16384 of which only the loss is wanted: one
// pass finds the row's maximum and the sum of exponentials together, a second one over the row, which L2 still holds, writes the
// results; 16-byte accesses.  Softmax (labels null; SCALED: scale is not 1) or its cross-entropy.  Bound by HBM and the second
// exponential: 1024 x 128256 takes 139 us for gradient and loss, 50 for the loss alone, 135 for the softmax; the scalar kernels take
// 550, 331 and 740, the row in registers (64 of them for 16 pieces alone, so it spills) 365 for 2048 x 50304, this one 111.
template <typename L, bool SCALED>
__global__ void __launch_bounds__(512) softmax_long_kernel(const bf16 *x, const L *labels, bf16 *__restrict__ probs,
                                                           bf16 *__restrict__ dlogits, float *__restrict__ loss, int rows, int cols, float scale,
                                                           float grad_scale) {
  pdl_entry();
  __shared__ float2 red[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int nvec = cols >> 3;
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const bf16 *px = x + (long long)row * cols;
    const long long label = labels ? (long long)labels[row] : -1;
    const bool valid = label >= 0 && label < cols;
    float m = -INFINITY, s = 0.f;
    for (int i = threadIdx.x; i < nvec; i += blockDim.x) {
      float v[8];
      vec::ld8(px + (long long)i * 8, v);
      float nm = m;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (SCALED) v[j] *= scale;
        nm = fmaxf(nm, v[j]);
      }
      const float sub = nm == -INFINITY ? 0.f : nm;  // nothing but masked elements so far: their exponentials are 0
      float acc = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) acc += __expf(v[j] - sub);
      s = s * __expf(m - sub) + acc;
      m = nm;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float om = __shfl_xor_sync(0xffffffffu, m, o), os = __shfl_xor_sync(0xffffffffu, s, o);
      const float nm = fmaxf(m, om), sub = nm == -INFINITY ? 0.f : nm;
      s = s * __expf(m - sub) + os * __expf(om - sub);
      m = nm;
    }
    const float at_label = valid && threadIdx.x == 0 ? bf2f(px[label]) : 0.f;  // dlogits may be the same buffer
    __syncthreads();  // the previous row's readers are done with `red`
    if (lane == 0) red[wid] = make_float2(m, s);
    __syncthreads();
    float M = -INFINITY, S = 0.f;
    for (int k = 0; k < nw; ++k) M = fmaxf(M, red[k].x);
    for (int k = 0; k < nw; ++k) S += (red[k].x == -INFINITY && red[k].y == 0.f) ? 0.f : red[k].y * __expf(red[k].x - M);
    const float inv = 1.f / S;
    if (threadIdx.x == 0 && loss) loss[row] = valid ? (__logf(S) + M - at_label) : 0.f;
    if (!probs && !dlogits) continue;
    for (int i = threadIdx.x; i < nvec; i += blockDim.x) {
      const long long at = (long long)row * cols + (long long)i * 8;
      float v[8];
      vec::ld8(px + (long long)i * 8, v);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = __expf((SCALED ? v[j] * scale : v[j]) - M) * inv;
      if (probs) vec::st8(probs + at, v);
      if (dlogits) {
        const int hit = valid ? (int)label - i * 8 : -1;
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = valid ? (v[j] - (j == hit ? 1.f : 0.f)) * grad_scale : 0.f;
        vec::st8(dlogits + at, v);
      }
    }
  }
}

// ------------------------------------------------------------------ loss gradients
enum { LOSS_SPARSE_CCE = 0, LOSS_CCE = 1, LOSS_MSE_AVG = 2, LOSS_IDENTITY = 3, LOSS_MSE_SUM = 4 };
// dlogit for losses whose input is already a probability / prediction tensor.
template <typename T, typename L>
__global__ void loss_bwd_kernel(int kind, const T *pred, const void *target,
                                T *__restrict__ dpred, long long rows, int cols, float scale) {
  pdl_entry();
  long long n = rows * cols;
  long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    float p = ldf(pred + i), g;
    if (kind == LOSS_SPARSE_CCE) {
      long long lab = (long long)((const L *)target)[i / cols];
      g = p - ((i % cols) == lab ? 1.f : 0.f);
    } else if (kind == LOSS_CCE) {
      g = p - ldf((const T *)target + i);
    } else if (kind == LOSS_MSE_AVG || kind == LOSS_MSE_SUM) {
      g = 2.f * (p - ldf((const T *)target + i));
    } else {
      g = 1.f;
    }
    stf(dpred + i, g * scale);
  }
}
// per-row loss values for reporting
template <typename T, typename L>
__global__ void loss_fwd_kernel(int kind, const T *pred, const void *target,
                                float *__restrict__ loss, int rows, int cols) {
  pdl_entry();
  __shared__ float red[32];
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const T *pp = pred + (long long)row * cols;
    float acc = 0.f;
    if (kind == LOSS_SPARSE_CCE) {
      long long lab = (long long)((const L *)target)[row];
      if (threadIdx.x == 0 && lab >= 0 && lab < cols) acc = -__logf(fmaxf(ldf(pp + lab), 1e-30f));
    } else {
      const T *pt = (const T *)target + (long long)row * cols;
      for (int c = threadIdx.x; c < cols; c += blockDim.x) {
        float p = ldf(pp + c);
        if (kind == LOSS_CCE) acc += -ldf(pt + c) * __logf(fmaxf(p, 1e-30f));
        else if (kind == LOSS_IDENTITY) acc += p;
        else { float d = p - ldf(pt + c); acc += d * d; }
      }
    }
    acc = block_sum(acc, red);
    if (threadIdx.x == 0) loss[row] = acc;
  }
}

}  // namespace

#define DISPATCH_FLOAT(dt, ...)                                   \
  if ((dt) == 0) { typedef float T; __VA_ARGS__; }                \
  else if ((dt) == 1) { typedef bf16 T; __VA_ARGS__; }            \
  else return -2;

static int rows_grid(int rows) { return rows < 148 * 8 ? rows : 148 * 8; }
static bool aligned16(const void *p) { return (((uintptr_t)p) & 15) == 0; }
// vectors per thread for the vectorised LayerNorm kernels: the smallest of 1/2/4 that gives a block of
// whole warps with at most 512 threads; 0 = not expressible
static int ln_vpt(int cols) {
  if (cols % 8) return 0;
  int nv = cols / 8;
  for (int v = 1; v <= 4; v *= 2)
    if (nv % v == 0 && (nv / v) % 32 == 0 && nv / v <= 512) return v;
  return 0;
}
static bool ln_vec_ok(int cols, const void *a, const void *b, const void *c, const void *d, const void *e, const void *f) {
  return ln_vpt(cols) > 0 && aligned16(a) && aligned16(b) && aligned16(c) && aligned16(d) && aligned16(e) && aligned16(f);
}

FFK_API int ffk_layernorm_fwd(const void *a, const void *b, const void *gamma, const void *beta, void *xsum, void *y,
                              float *mean, float *rstd, int rows, int cols, float eps, int dt, cudaStream_t st) {
  if (rows <= 0) return 0;
  FfkTraffic traffic((long long)rows * cols * (dt == 1 ? 2 : 4) * (b ? 4 : 2));
  if (dt == 1 && ln_vec_ok(cols, a, b, gamma, beta, xsum, y)) {
    int vpt = ln_vpt(cols), threads = cols / 8 / vpt;
    const bf16 *A = (const bf16 *)a, *B = (const bf16 *)b, *G = (const bf16 *)gamma, *Bt = (const bf16 *)beta;
    // rows of up to 2048 elements in steps of 256: one warp per row, no block-wide barriers in the row loop
    if (cols % 256 == 0 && cols <= 2048 && rows >= 8) {
      const int wv = cols / 256;
      long long want = ((long long)rows + 7) / 8;
      const int grid = (int)(want < 148 * 2 ? want : 148 * 2);
#define LN_WARP(V) ffk_launch(vec::layernorm_fwd_warp_kernel<V>, grid, 256, 0, st, A, B, G, Bt, (bf16 *)xsum, (bf16 *)y, mean, rstd, rows, eps)
      switch (wv) {
        case 1: LN_WARP(1); break;
        case 2: LN_WARP(2); break;
        case 3: LN_WARP(3); break;
        case 4: LN_WARP(4); break;
        case 5: LN_WARP(5); break;
        case 6: LN_WARP(6); break;
        case 7: LN_WARP(7); break;
        default: LN_WARP(8); break;
      }
#undef LN_WARP
      return (int)cudaGetLastError();
    }
    if (vpt == 1) ffk_launch(vec::layernorm_fwd_vec_kernel<1>, rows_grid(rows), threads, 0, st, A, B, G, Bt, (bf16 *)xsum, (bf16 *)y, mean, rstd, rows, cols, eps);
    else if (vpt == 2) ffk_launch(vec::layernorm_fwd_vec_kernel<2>, rows_grid(rows), threads, 0, st, A, B, G, Bt, (bf16 *)xsum, (bf16 *)y, mean, rstd, rows, cols, eps);
    else ffk_launch(vec::layernorm_fwd_vec_kernel<4>, rows_grid(rows), threads, 0, st, A, B, G, Bt, (bf16 *)xsum, (bf16 *)y, mean, rstd, rows, cols, eps);
    return (int)cudaGetLastError();
  }
  int threads = cols >= 2048 ? 512 : 256;
  DISPATCH_FLOAT(dt, (ffk_launch(layernorm_fwd_kernel<T>, rows_grid(rows), threads, 0, st, 
                         (const T *)a, (const T *)b, (const T *)gamma, (const T *)beta, (T *)xsum, (T *)y, mean, rstd,
                         rows, cols, eps)));
  return (int)cudaGetLastError();
}

// Persistent blocks of the backward kernel: as many per SM as its registers allow for the block size in use (narrow
// rows mean small blocks, of which two per SM left most of the SM idle); each block writes one partial row of
// dgamma / dbeta, which the fold kernel sums.
static int ln_bwd_grid(int rows, int cols, bool vec) {
  int per_sm = 2;
  if (vec && ln_vpt(cols) > 0) {
    const int threads = cols / 8 / ln_vpt(cols);
    per_sm = 768 / threads;
    if (per_sm < 2) per_sm = 2;
    if (per_sm > 8) per_sm = 8;
  }
  const int g = 148 * per_sm;
  return rows < g ? rows : g;
}
// The one-warp-per-row backward kernel takes rows of 256, 512, 768 or 1024; from 64 rows on its blocks of 8 warps are filled.
static bool ln_bwd_warp_ok(int rows, int cols) { return cols % 256 == 0 && cols <= 1024 && rows >= 64; }
static int ln_bwd_warp_grid(int rows, int cols) {
  const int most = cols <= 512 ? 148 * 2 : 148, want = (rows + 7) / 8;
  return want < most ? want : most;
}
// floats of scratch needed by ffk_layernorm_bwd (the larger of the kernel forms' needs)
FFK_API long long ffk_layernorm_bwd_scratch(int rows, int cols) {
  const int a = ln_bwd_grid(rows, cols, true), b = ln_bwd_grid(rows, cols, false);
  return 2ll * (a > b ? a : b) * cols;
}

// dx (+)= LN backward; dgamma/dbeta (+)= column sums.  `partial` is scratch of
// ffk_layernorm_bwd_scratch(rows, cols) floats.  cols <= 16384.
FFK_API int ffk_layernorm_bwd(const void *dy, const void *x, const void *gamma, const float *mean, const float *rstd,
                              void *dx, void *dx2, void *dgamma, void *dbeta, float *partial, int rows, int cols, int dt,
                              int accumulate_dx, int accumulate_dx2, int accumulate_params, cudaStream_t st) {
  if (rows <= 0) return 0;
  FfkTraffic traffic((long long)rows * cols * (dt == 1 ? 2 : 4) * (dx2 ? 4 : 3));
  if (cols > 16384) return -2;
  const bool vec = dt == 1 && ln_vec_ok(cols, dy, x, gamma, dx, dx2, nullptr);
  int grid = ln_bwd_grid(rows, cols, vec);
  float *part = (dgamma || dbeta) ? partial : nullptr;
  if (vec) {
    int vpt = ln_vpt(cols), threads = cols / 8 / vpt;
    const bf16 *DY = (const bf16 *)dy, *X = (const bf16 *)x, *G = (const bf16 *)gamma;
    if (ln_bwd_warp_ok(rows, cols)) {
      grid = ln_bwd_warp_grid(rows, cols);
#define LN_BWD(V)                                                                                                                            \
  ffk_launch(vec::layernorm_bwd_warp_kernel<V>, grid, 256, 0, st, DY, X, G, mean, rstd, (bf16 *)dx, (bf16 *)dx2, part, rows, accumulate_dx, \
             accumulate_dx2)
      switch (cols / 256) {
        case 1: LN_BWD(1); break;
        case 2: LN_BWD(2); break;
        case 3: LN_BWD(3); break;
        default: LN_BWD(4); break;
      }
#undef LN_BWD
    } else if (vpt == 1) ffk_launch(vec::layernorm_bwd_vec_kernel<1>, grid, threads, 0, st, DY, X, G, mean, rstd, (bf16 *)dx, (bf16 *)dx2, part, rows, cols, accumulate_dx, accumulate_dx2);
    else if (vpt == 2) ffk_launch(vec::layernorm_bwd_vec_kernel<2>, grid, threads, 0, st, DY, X, G, mean, rstd, (bf16 *)dx, (bf16 *)dx2, part, rows, cols, accumulate_dx, accumulate_dx2);
    else ffk_launch(vec::layernorm_bwd_vec_kernel<4>, grid, threads, 0, st, DY, X, G, mean, rstd, (bf16 *)dx, (bf16 *)dx2, part, rows, cols, accumulate_dx, accumulate_dx2);
    traffic.done();
    if (part)
      ffk_launch(vec::fold_partials_kernel<bf16>, (cols + 31) / 32, dim3(32, 32), 0, st, part, grid, cols, (bf16 *)dgamma, (bf16 *)dbeta, accumulate_params);
    return (int)cudaGetLastError();
  }
  DISPATCH_FLOAT(dt, {
    if (cols <= 512 * 4)
      ffk_launch(layernorm_bwd_kernel<T, 4>, grid, 512, 0, st, (const T *)dy, (const T *)x, (const T *)gamma, mean, rstd,
                                                        (T *)dx, (T *)dx2, part, rows, cols, accumulate_dx, accumulate_dx2);
    else if (cols <= 512 * 16)
      ffk_launch(layernorm_bwd_kernel<T, 16>, grid, 512, 0, st, (const T *)dy, (const T *)x, (const T *)gamma, mean, rstd,
                                                         (T *)dx, (T *)dx2, part, rows, cols, accumulate_dx, accumulate_dx2);
    else
      ffk_launch(layernorm_bwd_kernel<T, 32>, grid, 512, 0, st, (const T *)dy, (const T *)x, (const T *)gamma, mean, rstd,
                                                         (T *)dx, (T *)dx2, part, rows, cols, accumulate_dx, accumulate_dx2);
    traffic.done();
    if (part)
      ffk_launch(vec::fold_partials_kernel<T>, (cols + 31) / 32, dim3(32, 32), 0, st, part, grid, cols, (T *)dgamma, (T *)dbeta, accumulate_params);
  });
  return (int)cudaGetLastError();
}

// Rows of up to 4096 bf16 elements at a pitch of whole 16-byte pieces: one warp per row.
static bool softmax_warp_ok(int cols, int ld, int dt, const void *a, const void *b, const void *c) {
  return dt == 1 && cols > 0 && cols <= 4096 && ld >= cols && ld % 8 == 0 && aligned16(a) && aligned16(b) && aligned16(c);
}
// It pays up to `most` elements and where the row fills the lanes' registers; a longer row that leaves a part of them empty costs as
// much as the full one (2048 x 2056: forward 14.7 us, backward 16.7), and the block-per-row kernel is faster (11.7 and 9.6).
static bool softmax_warp_pays(int cols, int most) { return cols <= most || cols == 2048 || cols == 4096; }
constexpr int WARP_FWD_MOST = 2048, WARP_BWD_MOST = 1536;
static int softmax_scalar_fwd(const void *x, void *y, int rows, int cols, float scale, int causal_q, int dt, cudaStream_t st) {
  const int threads = cols >= 1024 ? 256 : 128;
  DISPATCH_FLOAT(dt, (ffk_launch(softmax_fwd_kernel<T>, rows < 148 * 16 ? rows : 148 * 16, threads, 0, st, (const T *)x, (T *)y, rows, cols, scale,
                                 causal_q)));
  return (int)cudaGetLastError();
}
static int softmax_scalar_bwd(const void *dy, const void *y, void *dx, int rows, int cols, float scale, int dt, cudaStream_t st) {
  const int threads = cols >= 1024 ? 256 : 128;
  DISPATCH_FLOAT(dt, (ffk_launch(softmax_bwd_kernel<T>, rows < 148 * 16 ? rows : 148 * 16, threads, 0, st, (const T *)dy, (const T *)y, (T *)dx, rows,
                                 cols, scale)));
  return (int)cudaGetLastError();
}
// vectors of 8 per lane that hold a row: the next of 1, 2, 3, 4, 6, 8, 16
static int softmax_vpt(int cols) {
  const int v = (cols + 255) / 256;
  return v <= 4 ? v : v <= 6 ? 6 : v <= 8 ? 8 : 16;
}
// y = softmax(scale * x) over rows of `cols` at pitch `ld`; yd (optional) = dropout(y, p) with the mask
// hash(salt, *seed_ptr, row * cols + column).  Returns -3 for rows the one-warp-per-row kernel cannot take.
FFK_API int ffk_softmax_dropout_fwd(const void *x, void *y, void *yd, int rows, int cols, int ld, float scale, int causal_q, float p,
                                    unsigned long long salt, const unsigned long long *seed_ptr, int dt, cudaStream_t st) {
  if (rows <= 0) return 0;
  FfkTraffic traffic((long long)rows * cols * 2 * (yd ? 3 : 2));
  if (!softmax_warp_ok(cols, ld, dt, x, y, yd)) return -3;
  if (!yd && ld == cols && !softmax_warp_pays(cols, WARP_FWD_MOST)) return softmax_scalar_fwd(x, y, rows, cols, scale, causal_q, dt, st);
  const int grid = ffk_blocks(rows, 8);
#define SM_FWD(V)                                                                                                                        \
  case V:                                                                                                                                \
    if (cols == 256 * V && ld == cols)                                                                                                   \
      ffk_launch(vec::softmax_fwd_warp_kernel<V, true>, grid, 256, 0, st, (const bf16 *)x, (bf16 *)y, (bf16 *)yd, rows, cols, ld, scale, causal_q, \
                                                                  p, salt, seed_ptr);                                                    \
    else                                                                                                                                 \
      ffk_launch(vec::softmax_fwd_warp_kernel<V, false>, grid, 256, 0, st, (const bf16 *)x, (bf16 *)y, (bf16 *)yd, rows, cols, ld, scale, causal_q, \
                                                                   p, salt, seed_ptr);                                                   \
    break;
  switch (softmax_vpt(cols)) { SM_FWD(1) SM_FWD(2) SM_FWD(3) SM_FWD(4) SM_FWD(6) SM_FWD(8) SM_FWD(16) }
#undef SM_FWD
  return (int)cudaGetLastError();
}
// dx = scale * y * (g - sum(g*y)) with g = dropout_backward(dy) (p = 0: g = dy).  Same rows as above.
FFK_API int ffk_softmax_dropout_bwd(const void *dy, const void *y, void *dx, int rows, int cols, int ld, float scale, float p,
                                    unsigned long long salt, const unsigned long long *seed_ptr, int dt, cudaStream_t st) {
  if (rows <= 0) return 0;
  FfkTraffic traffic((long long)rows * cols * 2 * 3);
  if (!softmax_warp_ok(cols, ld, dt, dy, y, dx)) return -3;
  if (!(p > 0.f) && ld == cols && !softmax_warp_pays(cols, WARP_BWD_MOST)) return softmax_scalar_bwd(dy, y, dx, rows, cols, scale, dt, st);
  const int grid = ffk_blocks(rows, 8);
#define SM_BWD(V)                                                                                                                       \
  case V:                                                                                                                               \
    if (cols == 256 * V && ld == cols)                                                                                                  \
      ffk_launch(vec::softmax_bwd_warp_kernel<V, true>, grid, 256, 0, st, (const bf16 *)dy, (const bf16 *)y, (bf16 *)dx, rows, cols, ld, scale, p, \
                                                                  salt, seed_ptr);                                                      \
    else                                                                                                                                \
      ffk_launch(vec::softmax_bwd_warp_kernel<V, false>, grid, 256, 0, st, (const bf16 *)dy, (const bf16 *)y, (bf16 *)dx, rows, cols, ld, scale, p, \
                                                                   salt, seed_ptr);                                                     \
    break;
  switch (softmax_vpt(cols)) { SM_BWD(1) SM_BWD(2) SM_BWD(3) SM_BWD(4) SM_BWD(6) SM_BWD(8) SM_BWD(16) }
#undef SM_BWD
  return (int)cudaGetLastError();
}
// y = dropout(x) over bf16 rows of `cols` at pitch `ld`: the dropped copy ffk_softmax_dropout_fwd would write.
FFK_API int ffk_dropout_rows(const void *x, void *y, long long rows, int cols, int ld, float p, unsigned long long salt,
                             const unsigned long long *seed_ptr, cudaStream_t st) {
  if (rows <= 0) return 0;
  if (!softmax_warp_ok(cols, ld, 1, x, y, nullptr)) return -3;
  ffk_launch(vec::dropout_rows_kernel, ffk_blocks(rows * (ld / 8), 256), 256, 0, st, (const bf16 *)x, (bf16 *)y, rows, cols, ld, p, salt, seed_ptr);
  return (int)cudaGetLastError();
}

// The wide-row kernel takes rows of whole 16-byte pieces that fill its threads at least to half and its ring at least twice.
static bool softmax_wide_ok(int cols, int dt) { return dt == 1 && cols % 8 == 0 && cols > 4096 && cols <= 32768; }
static bool softmax_long_ok(int cols, int dt) { return dt == 1 && cols % 8 == 0 && cols > 32768; }
static int long_grid(int rows) { return rows < 148 * 8 ? rows : 148 * 8; }
template <bool CE, typename L>
static int launch_softmax_wide(const void *x, const void *labels, void *probs, void *dlogits, float *loss, int rows, int cols, float scale,
                               float grad_scale, cudaStream_t st, unsigned long long wait_ns = WAIT_LIMIT_NS) {
  auto kern = softmax_wide_kernel<CE, L>;
  static unsigned long long done = 0;
  if (cudaError_t e = ffk_allow_smem(kern, WIDE_SMEM, done)) return (int)e;
  const int threads = cols <= 8192 ? 256 : cols <= 16384 ? 512 : 1024;   // at most four pieces of 8 per thread
  const int per_sm = 1024 / threads;
  int depth = WIDE_SMEM / per_sm / (cols * 2);
  if (depth > 4) depth = 4;
  const int grid = rows < 148 * per_sm ? rows : 148 * per_sm;
  ffk_launch(kern, grid, threads, (size_t)depth * cols * 2, st, (const bf16 *)x, (const L *)labels, (bf16 *)probs, (bf16 *)dlogits, loss, rows, cols,
                                                        scale, grad_scale, depth, wait_ns);
  return (int)cudaGetLastError();
}
// Error word of the wide-row kernel's bounded waits (read and cleared; synchronises the device).
FFK_API int ffk_softmax_last_error() {
  int v = 0, z = 0;
  if (cudaDeviceSynchronize() != cudaSuccess) return -1;
  cudaMemcpyFromSymbol(&v, g_rows_err, sizeof(int));
  cudaMemcpyToSymbol(g_rows_err, &z, sizeof(int));
  return v;
}

FFK_API int ffk_softmax_fwd(const void *x, void *y, int rows, int cols, float scale, int causal_q, int dt,
                            cudaStream_t st) {
  if (rows <= 0) return 0;
  FfkTraffic traffic((long long)rows * cols * (dt == 1 ? 2 : 4) * 2);
  if (softmax_warp_ok(cols, cols, dt, x, y, nullptr))
    return ffk_softmax_dropout_fwd(x, y, nullptr, rows, cols, cols, scale, causal_q, 0.f, 0, nullptr, dt, st);
  if (softmax_wide_ok(cols, dt) && causal_q <= 0 && aligned16(x) && aligned16(y))
    return launch_softmax_wide<false, int>(x, nullptr, y, nullptr, nullptr, rows, cols, scale, 1.f, st);
  if (softmax_long_ok(cols, dt) && causal_q <= 0 && aligned16(x) && aligned16(y)) {
    if (scale == 1.f)
      ffk_launch(softmax_long_kernel<int, false>, long_grid(rows), 512, 0, st, (const bf16 *)x, nullptr, (bf16 *)y, nullptr, nullptr, rows, cols, 1.f, 1.f);
    else
      ffk_launch(softmax_long_kernel<int, true>, long_grid(rows), 512, 0, st, (const bf16 *)x, nullptr, (bf16 *)y, nullptr, nullptr, rows, cols, scale, 1.f);
    return (int)cudaGetLastError();
  }
  return softmax_scalar_fwd(x, y, rows, cols, scale, causal_q, dt, st);
}
FFK_API int ffk_softmax_bwd(const void *dy, const void *y, void *dx, int rows, int cols, float scale, int dt,
                            cudaStream_t st) {
  if (rows <= 0) return 0;
  FfkTraffic traffic((long long)rows * cols * (dt == 1 ? 2 : 4) * 3);
  if (softmax_warp_ok(cols, cols, dt, dy, y, dx))
    return ffk_softmax_dropout_bwd(dy, y, dx, rows, cols, cols, scale, 0.f, 0, nullptr, dt, st);
  return softmax_scalar_bwd(dy, y, dx, rows, cols, scale, dt, st);
}
template <int VPT, typename L>
static void launch_softmax_ce_row(const void *logits, const void *labels, void *probs, void *dlogits, float *loss, int rows, int cols,
                                  float grad_scale, cudaStream_t st) {
  ffk_launch(softmax_ce_row_kernel<VPT, L>, rows, ROW_THREADS, 0, st, (const bf16 *)logits, (const L *)labels, (bf16 *)probs, (bf16 *)dlogits, loss,
             cols, grad_scale);
}
// bf16 rows of whole 16-byte pieces: in registers up to 4096, through the ring up to 32768, in two passes beyond
template <typename L>
static int launch_softmax_ce(const void *logits, const void *labels, void *probs, void *dlogits, float *loss, int rows, int cols, float grad_scale,
                             cudaStream_t st) {
  // The ring pays where rows are written too, and up to 16384 also for a loss alone (300 x 8192: 4.0 us, in one pass without it 6.5); beyond,
  // where it is one block per SM, a loss alone is the faster without (8192 x 30528: 160 us through the ring, 132).
  const bool ring = softmax_wide_ok(cols, 1) && (probs || dlogits || cols <= 16384);
  if (ring) return launch_softmax_wide<true, L>(logits, labels, probs, dlogits, loss, rows, cols, 1.f, grad_scale, st);
  if (softmax_long_ok(cols, 1) || softmax_wide_ok(cols, 1))
    ffk_launch(softmax_long_kernel<L, false>, long_grid(rows), 512, 0, st, (const bf16 *)logits, (const L *)labels, (bf16 *)probs, (bf16 *)dlogits, loss, rows,
               cols, 1.f, grad_scale);
  else if (cols <= 8 * ROW_THREADS) launch_softmax_ce_row<1, L>(logits, labels, probs, dlogits, loss, rows, cols, grad_scale, st);
  else if (cols <= 16 * ROW_THREADS) launch_softmax_ce_row<2, L>(logits, labels, probs, dlogits, loss, rows, cols, grad_scale, st);
  else launch_softmax_ce_row<4, L>(logits, labels, probs, dlogits, loss, rows, cols, grad_scale, st);
  return (int)cudaGetLastError();
}
// label_dt: 2 = int32, 3 = int64
FFK_API int ffk_softmax_ce(const void *logits, const void *labels, void *probs, void *dlogits, float *loss, int rows,
                           int cols, float grad_scale, int dt, int label_dt, cudaStream_t st) {
  if (rows <= 0) return 0;
  FfkTraffic traffic((long long)rows * cols * (dt == 1 ? 2 : 4) * 2);
  if (dt == 1 && cols % 8 == 0 && aligned16(logits) && aligned16(probs) && aligned16(dlogits))
    return label_dt == 3 ? launch_softmax_ce<long long>(logits, labels, probs, dlogits, loss, rows, cols, grad_scale, st)
                         : launch_softmax_ce<int>(logits, labels, probs, dlogits, loss, rows, cols, grad_scale, st);
  const int threads = cols >= 4096 ? 1024 : 256;
  const int grid = rows < 148 * 4 ? rows : 148 * 4;
  DISPATCH_FLOAT(dt, {
    if (label_dt == 3)
      ffk_launch(softmax_ce_kernel<T, long long>, grid, threads, 0, st, (const T *)logits, (const long long *)labels,
                                                                 (T *)probs, (T *)dlogits, loss, rows, cols, grad_scale);
    else
      ffk_launch(softmax_ce_kernel<T, int>, grid, threads, 0, st, (const T *)logits, (const int *)labels, (T *)probs,
                                                           (T *)dlogits, loss, rows, cols, grad_scale);
  });
  return (int)cudaGetLastError();
}
// The wide-row cross-entropy with another limit of its waits: 0 lets the first one run out, so that a test sees what then comes back.
FFK_API int ffk_softmax_ce_wait(const void *logits, const int *labels, void *probs, void *dlogits, float *loss, int rows, int cols,
                                unsigned long long wait_ns, cudaStream_t st) {
  if (rows <= 0 || !softmax_wide_ok(cols, 1) || !aligned16(logits) || !aligned16(probs) || !aligned16(dlogits)) return -2;
  return launch_softmax_wide<true, int>(logits, labels, probs, dlogits, loss, rows, cols, 1.f, 1.f, st, wait_ns);
}
FFK_API int ffk_loss_bwd(int kind, const void *pred, const void *target, void *dpred, long long rows, int cols,
                         float scale, int dt, int label_dt, cudaStream_t st) {
  if (rows <= 0) return 0;
  DISPATCH_FLOAT(dt, {
    if (label_dt == 3)
      ffk_launch(loss_bwd_kernel<T, long long>, ffk_blocks(rows * cols, 256), 256, 0, st, kind, (const T *)pred, target,
                                                                                   (T *)dpred, rows, cols, scale);
    else
      ffk_launch(loss_bwd_kernel<T, int>, ffk_blocks(rows * cols, 256), 256, 0, st, kind, (const T *)pred, target, (T *)dpred,
                                                                             rows, cols, scale);
  });
  return (int)cudaGetLastError();
}
FFK_API int ffk_loss_fwd(int kind, const void *pred, const void *target, float *loss, int rows, int cols, int dt,
                         int label_dt, cudaStream_t st) {
  if (rows <= 0) return 0;
  DISPATCH_FLOAT(dt, {
    if (label_dt == 3)
      ffk_launch(loss_fwd_kernel<T, long long>, rows < 2368 ? rows : 2368, 128, 0, st, kind, (const T *)pred, target, loss,
                                                                                rows, cols);
    else
      ffk_launch(loss_fwd_kernel<T, int>, rows < 2368 ? rows : 2368, 128, 0, st, kind, (const T *)pred, target, loss, rows,
                                                                          cols);
  });
  return (int)cudaGetLastError();
}
