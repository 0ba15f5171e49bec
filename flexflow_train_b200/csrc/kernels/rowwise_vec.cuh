// rowwise_vec.cuh -- 128-bit vectorised fast paths of the row-wise kernels: softmax fwd/bwd (optionally fused
// with dropout of the probabilities; bf16 rows of any length at a pitch of a multiple of 8), LayerNorm fwd/bwd
// (fused residual add; bf16) and the bias/activation backward with its column
// reduction (bf16 rows whose length is a multiple of 8).
//
// Each thread owns whole 8-element vectors of a row and keeps them in registers, so a row is read once
// and written once; HBM traffic is the algorithmic minimum.  The scalar kernels in norm_softmax.cu and
// elementwise.cu remain the general path (fp32, odd lengths).
#pragma once
#include "common.cuh"

namespace vec {

__device__ __forceinline__ void ld8(const bf16 *p, float *v) {
  uint4 u = *reinterpret_cast<const uint4 *>(p);
  float2 a = unpack_bf162(u.x), b = unpack_bf162(u.y), c = unpack_bf162(u.z), d = unpack_bf162(u.w);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y; v[6] = d.x; v[7] = d.y;
}
__device__ __forceinline__ void unpack8(const uint4 &u, float *v) {
  float2 a = unpack_bf162(u.x), b = unpack_bf162(u.y), c = unpack_bf162(u.z), d = unpack_bf162(u.w);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y; v[6] = d.x; v[7] = d.y;
}
__device__ __forceinline__ void st8(bf16 *p, const float *v) {
  *reinterpret_cast<uint4 *>(p) = make_uint4(pack_bf162(v[0], v[1]), pack_bf162(v[2], v[3]), pack_bf162(v[4], v[5]), pack_bf162(v[6], v[7]));
}

// ---------------------------------------------------------------- softmax: one warp per row
// Keep flags of the 8 elements from flat index e on (two group words where the row length is a multiple of 4, and e with it;
// otherwise element by element, the same function of (seed, flat index) as the stand-alone dropout kernel).
__device__ __forceinline__ uint32_t keep8(unsigned long long seed, unsigned long long e, bool grouped, uint32_t thr) {
  if (grouped) return ffk_keep4(seed, e >> 2, thr) | (ffk_keep4(seed, (e >> 2) + 1, thr) << 4);
  uint32_t k = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) k |= (ffk_keep(seed, e + j, thr) ? 1u : 0u) << j;
  return k;
}
// Rows of `cols` elements at a pitch of `ld` (a multiple of 8, at least cols); 256 * (VPT - 1) < cols <= 256 * VPT; FULL: cols
// fills the vectors and ld == cols.  y = softmax(scale * x); yd (optional) = dropout(y) with keep mask hash(seed, row * cols +
// column); the pitch's tail columns of y / yd are written as zeros.  Bound by HBM: the row is read once into registers.  Rows
// that are no multiple of 256 (sequence 500, 128 x 500 x 500 scores) used to take the block-per-row scalar kernel, which reads
// the row three times in 2-byte pieces and left the dropped copy to a second kernel: 104 + 28 us.
template <int VPT, bool FULL>
__global__ void softmax_fwd_warp_kernel(const bf16 *x, bf16 *__restrict__ y, bf16 *__restrict__ yd, int rows, int cols, int ld,
                                        float scale, int causal_q, float p_drop, unsigned long long salt, const unsigned long long *seed_ptr) {
  pdl_entry();
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  unsigned long long seed = salt;
  if (seed_ptr) seed = salt * 0x9E3779B97F4A7C15ull + *seed_ptr;
  const float keep_scale = p_drop < 1.f ? 1.f / (1.f - p_drop) : 0.f;
  const uint32_t thr = ffk_drop_threshold(p_drop);
  const bool grouped = FULL || (cols & 3) == 0;
  for (long long row = (long long)blockIdx.x * wpb + wib; row < rows; row += (long long)gridDim.x * wpb) {
    const bf16 *px = x + row * ld;
    float v[VPT][8];
    const int limit = causal_q > 0 ? min(cols, (int)(row % causal_q) + 1) : cols;
    float mx = -INFINITY;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      int c0 = (i * 32 + lane) * 8;
      if (FULL || c0 < cols) ld8(px + c0, v[i]);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        v[i][j] = (c0 + j < limit) ? v[i][j] * scale : -INFINITY;
        mx = fmaxf(mx, v[i][j]);
      }
    }
    mx = warp_max(mx);
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        v[i][j] = __expf(v[i][j] - mx);
        if (!FULL && (i * 32 + lane) * 8 + j >= cols) v[i][j] = 0.f;  // also when the row's maximum is -inf
        s += v[i][j];
      }
    s = warp_sum(s);
    const float inv = 1.f / s;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      int c0 = (i * 32 + lane) * 8;
      if (!FULL && c0 >= cols) continue;
#pragma unroll
      for (int j = 0; j < 8; ++j) v[i][j] = (FULL || c0 + j < cols) ? v[i][j] * inv : 0.f;
      st8(y + row * ld + c0, v[i]);
      if (yd) {
        float d[8];
        const uint32_t keep = keep8(seed, (unsigned long long)(row * cols + c0), grouped, thr);
#pragma unroll
        for (int j = 0; j < 8; ++j) d[j] = (keep >> j) & 1u ? v[i][j] * keep_scale : 0.f;
        st8(yd + row * ld + c0, d);
      }
    }
  }
}
// dx = scale * y * (g - sum(g * y)), g = dy (optionally first passed back through the dropout mask); rows as above
template <int VPT, bool FULL>
__global__ void softmax_bwd_warp_kernel(const bf16 *dy, const bf16 *y, bf16 *__restrict__ dx, int rows, int cols,
                                        int ld, float scale, float p_drop, unsigned long long salt, const unsigned long long *seed_ptr) {
  pdl_entry();
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  unsigned long long seed = salt;
  if (seed_ptr) seed = salt * 0x9E3779B97F4A7C15ull + *seed_ptr;
  const float keep_scale = p_drop < 1.f ? 1.f / (1.f - p_drop) : 0.f;
  const uint32_t thr = ffk_drop_threshold(p_drop);
  const bool grouped = FULL || (cols & 3) == 0;
  for (long long row = (long long)blockIdx.x * wpb + wib; row < rows; row += (long long)gridDim.x * wpb) {
    float g[VPT][8], p[VPT][8];
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      int c0 = (i * 32 + lane) * 8;
      if (FULL || c0 < cols) {
        ld8(dy + row * ld + c0, g[i]);
        ld8(y + row * ld + c0, p[i]);
      }
    }
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      int c0 = (i * 32 + lane) * 8;
      uint32_t keep = 0xFFu;
      if (p_drop > 0.f && (FULL || c0 < cols)) keep = keep8(seed, (unsigned long long)(row * cols + c0), grouped, thr);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (!FULL && c0 + j >= cols) { g[i][j] = 0.f; p[i][j] = 0.f; }
        if (p_drop > 0.f) g[i][j] = (keep >> j) & 1u ? g[i][j] * keep_scale : 0.f;
        s += g[i][j] * p[i][j];
      }
    }
    s = warp_sum(s);
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      int c0 = (i * 32 + lane) * 8;
      if (!FULL && c0 >= cols) continue;
#pragma unroll
      for (int j = 0; j < 8; ++j) g[i][j] = (FULL || c0 + j < cols) ? scale * p[i][j] * (g[i][j] - s) : 0.f;
      st8(dx + row * ld + c0, g[i]);
    }
  }
}
// y = dropout(x) over rows of `cols` at pitch `ld`, the mask of softmax_fwd_warp_kernel's yd; a thread per 8 elements
static __global__ void dropout_rows_kernel(const bf16 *x, bf16 *__restrict__ y, long long rows, int cols, int ld, float p_drop,
                                           unsigned long long salt, const unsigned long long *seed_ptr) {
  pdl_entry();
  const unsigned long long seed = seed_ptr ? salt * 0x9E3779B97F4A7C15ull + *seed_ptr : salt;
  const float keep_scale = p_drop < 1.f ? 1.f / (1.f - p_drop) : 0.f;
  const uint32_t thr = ffk_drop_threshold(p_drop);
  const int nv = ld >> 3;
  const long long total = rows * nv;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total; t += (long long)gridDim.x * blockDim.x) {
    const long long row = t / nv;
    const int c0 = (int)(t - row * nv) * 8;
    float v[8];
    ld8(x + t * 8, v);
    const uint32_t keep = keep8(seed, (unsigned long long)(row * cols + c0), (cols & 3) == 0, thr);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = ((keep >> j) & 1u) && c0 + j < cols ? v[j] * keep_scale : 0.f;
    st8(y + t * 8, v);
  }
}

// ---------------------------------------------------------------- rows of one block each
// The row (cols % 8 == 0, up to 8 * VPT * blockDim.x) stays packed in registers between the maximum, the sum and the result, so
// HBM sees one read and one write.
template <int VPT>
__device__ __forceinline__ void row_load(const bf16 *p, int nvec, uint4 (&u)[VPT]) {
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int c = i * blockDim.x + threadIdx.x;
    if (c < nvec) u[i] = reinterpret_cast<const uint4 *>(p)[c];
  }
}
// maximum of the row's values and the sum of exp(value - maximum); `red`: 64 floats of shared memory
template <int VPT>
__device__ __forceinline__ void row_max_sum(const uint4 (&u)[VPT], int nvec, float *red, float &mx, float &sum) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  float m = -INFINITY;
#pragma unroll
  for (int i = 0; i < VPT; ++i)
    if (i * blockDim.x + threadIdx.x < nvec) {
      float v[8];
      unpack8(u[i], v);
#pragma unroll
      for (int j = 0; j < 8; ++j) m = fmaxf(m, v[j]);
    }
  m = warp_max(m);
  if (lane == 0) red[wid] = m;
  __syncthreads();
  m = red[0];
  for (int k = 1; k < nw; ++k) m = fmaxf(m, red[k]);
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < VPT; ++i)
    if (i * blockDim.x + threadIdx.x < nvec) {
      float v[8];
      unpack8(u[i], v);
      float a = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) a += __expf(v[j] - m);
      s += a;
    }
  s = warp_sum(s);
  if (lane == 0) red[32 + wid] = s;
  __syncthreads();
  s = 0.f;
  for (int k = 0; k < nw; ++k) s += red[32 + k];
  mx = m;
  sum = s;
}
// ---------------------------------------------------------------- LayerNorm: one block per row
// cols = 8 * blockDim.x * VPT.  y = LN(a + b) * gamma + beta, xsum = a + b (when b is given).
template <int VPT>
__global__ void layernorm_fwd_vec_kernel(const bf16 *a, const bf16 *b, const bf16 *gamma,
                                         const bf16 *beta, bf16 *__restrict__ xsum, bf16 *__restrict__ y,
                                         float *__restrict__ mean, float *__restrict__ rstd, int rows, int cols, float eps) {
  pdl_entry();
  // two block reductions per row (mean, then centred variance), each through its own double-buffered slot so
  // that one barrier per reduction suffices
  __shared__ float red_a[2][32], red_b[2][32];
  int parity = 0;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  float gm[VPT][8], bt[VPT][8];
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    int c0 = (i * blockDim.x + threadIdx.x) * 8;
    if (gamma) ld8(gamma + c0, gm[i]);
    if (beta) ld8(beta + c0, bt[i]);
  }
  // the next row's 16-byte pieces are fetched into registers before this row's two reductions, so that every
  // thread keeps loads in flight across the barriers
  uint4 na[VPT], nb[VPT];
  if ((int)blockIdx.x < rows) {
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      long long off = (long long)blockIdx.x * cols + (i * blockDim.x + threadIdx.x) * 8;
      na[i] = *reinterpret_cast<const uint4 *>(a + off);
      if (b) nb[i] = *reinterpret_cast<const uint4 *>(b + off);
    }
  }
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    float v[VPT][8];
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      long long off = (long long)row * cols + (i * blockDim.x + threadIdx.x) * 8;
      unpack8(na[i], v[i]);
      if (b) {
        float w[8];
        unpack8(nb[i], w);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[i][j] += w[j];
        if (xsum) {
          st8(xsum + off, v[i]);
#pragma unroll
          for (int j = 0; j < 8; ++j) v[i][j] = bf2f(f2bf(v[i][j]));  // statistics of the value backward will read
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) s += v[i][j];
    }
    const int next = row + gridDim.x;
    if (next < rows) {
#pragma unroll
      for (int i = 0; i < VPT; ++i) {
        long long off = (long long)next * cols + (i * blockDim.x + threadIdx.x) * 8;
        na[i] = *reinterpret_cast<const uint4 *>(a + off);
        if (b) nb[i] = *reinterpret_cast<const uint4 *>(b + off);
      }
    }
    s = warp_sum(s);
    if (lane == 0) red_a[parity][wid] = s;
    __syncthreads();
    float tot = 0.f;
    for (int k = 0; k < nw; ++k) tot += red_a[parity][k];
    const float mu = tot / cols;
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) { float d = v[i][j] - mu; ss += d * d; }
    ss = warp_sum(ss);
    if (lane == 0) red_b[parity][wid] = ss;
    __syncthreads();
    float tot2 = 0.f;
    for (int k = 0; k < nw; ++k) tot2 += red_b[parity][k];
    parity ^= 1;
    const float rs = rsqrtf(tot2 / cols + eps);
    if (threadIdx.x == 0) {
      if (mean) mean[row] = mu;
      if (rstd) rstd[row] = rs;
    }
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      long long off = (long long)row * cols + (i * blockDim.x + threadIdx.x) * 8;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float o = (v[i][j] - mu) * rs;
        v[i][j] = gamma ? o * gm[i][j] + (beta ? bt[i][j] : 0.f) : o;
      }
      st8(y + off, v[i]);
    }
  }
}
// LayerNorm forward, one warp per row: cols = 256 * VPT (up to 2048).  A lane holds VPT 16-byte pieces of the row
// (piece i of lane l = elements [(i * 32 + l) * 8, +8): coalesced), all loaded before anything is computed, so a
// warp has VPT (2 VPT with a fused add) loads in flight and the two row reductions are warp shuffles: no
// block-wide barrier after the one that stages gamma / beta in shared memory.
template <int VPT>
__global__ void __launch_bounds__(256, 2) layernorm_fwd_warp_kernel(const bf16 *a, const bf16 *b,
                                                                    const bf16 *gamma, const bf16 *beta,
                                                                    bf16 *__restrict__ xsum, bf16 *__restrict__ y, float *__restrict__ mean,
                                                                    float *__restrict__ rstd, int rows, float eps) {
  pdl_entry();
  constexpr int COLS = 256 * VPT, NV = 32 * VPT;
  __shared__ uint4 g_s[NV], b_s[NV];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  for (int i = threadIdx.x; i < NV; i += blockDim.x) {
    if (gamma) g_s[i] = reinterpret_cast<const uint4 *>(gamma)[i];
    if (beta) b_s[i] = reinterpret_cast<const uint4 *>(beta)[i];
  }
  __syncthreads();
  for (int row = blockIdx.x * wpb + wid; row < rows; row += gridDim.x * wpb) {
    const long long base = (long long)row * COLS;
    const uint4 *ar = reinterpret_cast<const uint4 *>(a + base);
    uint4 ua[VPT], ub[VPT];
#pragma unroll
    for (int i = 0; i < VPT; ++i) ua[i] = ar[i * 32 + lane];
    if (b) {
      const uint4 *br = reinterpret_cast<const uint4 *>(b + base);
#pragma unroll
      for (int i = 0; i < VPT; ++i) ub[i] = br[i * 32 + lane];
    }
    float v[VPT][8];
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      unpack8(ua[i], v[i]);
      if (b) {
        float w[8];
        unpack8(ub[i], w);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[i][j] += w[j];
        if (xsum) {
          st8(xsum + base + (i * 32 + lane) * 8, v[i]);
#pragma unroll
          for (int j = 0; j < 8; ++j) v[i][j] = bf2f(f2bf(v[i][j]));  // statistics of the value backward will read
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) s += v[i][j];
    }
    const float mu = warp_sum(s) * (1.0f / COLS);
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) { float d = v[i][j] - mu; ss += d * d; }
    const float rs = rsqrtf(warp_sum(ss) * (1.0f / COLS) + eps);
    if (lane == 0) {
      if (mean) mean[row] = mu;
      if (rstd) rstd[row] = rs;
    }
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      float g8[8], b8[8];
      if (gamma) unpack8(g_s[i * 32 + lane], g8);
      if (beta) unpack8(b_s[i * 32 + lane], b8);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float o = (v[i][j] - mu) * rs;
        v[i][j] = gamma ? o * g8[j] + (beta ? b8[j] : 0.f) : o;
      }
      st8(y + base + (i * 32 + lane) * 8, v[i]);
    }
  }
}
// dx (and optionally dx2) (+)= LN backward; per-block partial sums of dgamma/dbeta -> partial[2][grid][cols]
template <int VPT>
__global__ void layernorm_bwd_vec_kernel(const bf16 *dy, const bf16 *x, const bf16 *gamma,
                                         const float *mean, const float *rstd, bf16 *__restrict__ dx,
                                         bf16 *__restrict__ dx2, float *__restrict__ partial, int rows, int cols, int acc1, int acc2) {
  pdl_entry(dx, dx2);
  // the two row sums are reduced together through a double-buffered slot: one barrier per row
  __shared__ float2 red2[2][32];
  int parity = 0;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  float gm[VPT][8], dg[VPT][8], db[VPT][8];
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    int c0 = (i * blockDim.x + threadIdx.x) * 8;
    if (gamma) ld8(gamma + c0, gm[i]);
#pragma unroll
    for (int j = 0; j < 8; ++j) { dg[i][j] = 0.f; db[i][j] = 0.f; if (!gamma) gm[i][j] = 1.f; }
  }
  // the next row's pieces of dy and x travel while this row is reduced and written (see the forward kernel)
  uint4 ng[VPT], nx[VPT];
  if ((int)blockIdx.x < rows) {
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      long long off = (long long)blockIdx.x * cols + (i * blockDim.x + threadIdx.x) * 8;
      ng[i] = *reinterpret_cast<const uint4 *>(dy + off);
      nx[i] = *reinterpret_cast<const uint4 *>(x + off);
    }
  }
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const float mu = mean[row], rs = rstd[row];
    float g[VPT][8], xh[VPT][8];
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      unpack8(ng[i], g[i]);
      unpack8(nx[i], xh[i]);
    }
    const int next = row + gridDim.x;
    if (next < rows) {
#pragma unroll
      for (int i = 0; i < VPT; ++i) {
        long long off = (long long)next * cols + (i * blockDim.x + threadIdx.x) * 8;
        ng[i] = *reinterpret_cast<const uint4 *>(dy + off);
        nx[i] = *reinterpret_cast<const uint4 *>(x + off);
      }
    }
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        xh[i][j] = (xh[i][j] - mu) * rs;
        dg[i][j] += g[i][j] * xh[i][j];
        db[i][j] += g[i][j];
        g[i][j] *= gm[i][j];
        s1 += g[i][j];
        s2 += g[i][j] * xh[i][j];
      }
    }
    s1 = warp_sum(s1);
    s2 = warp_sum(s2);
    if (lane == 0) red2[parity][wid] = make_float2(s1, s2);
    __syncthreads();
    float t1 = 0.f, t2 = 0.f;
    for (int k = 0; k < nw; ++k) { float2 q = red2[parity][k]; t1 += q.x; t2 += q.y; }
    parity ^= 1;
    const float m1 = t1 / cols, m2 = t2 / cols;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      long long off = (long long)row * cols + (i * blockDim.x + threadIdx.x) * 8;
      float o[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = rs * (g[i][j] - m1 - xh[i][j] * m2);
      if (dx2) {
        float t[8];
        if (acc2) {
          ld8(dx2 + off, t);
#pragma unroll
          for (int j = 0; j < 8; ++j) t[j] += o[j];
          st8(dx2 + off, t);
        } else st8(dx2 + off, o);
      }
      if (acc1) {
        float t[8];
        ld8(dx + off, t);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] += t[j];
      }
      st8(dx + off, o);
    }
  }
  if (partial) {
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      int c0 = (i * blockDim.x + threadIdx.x) * 8;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        partial[(long long)blockIdx.x * cols + c0 + j] = dg[i][j];
        partial[((long long)gridDim.x + blockIdx.x) * cols + c0 + j] = db[i][j];
      }
    }
  }
}

// LayerNorm backward, one warp per row: cols = 256 * VPT, VPT <= 4 (the column sums of a lane's 8 * VPT columns stay in registers
// over all its rows).  No block-wide barrier per row, the next row's pieces in flight while this one is reduced, and one partial
// row of dgamma / dbeta per block of 8 warps instead of one per row group: at 2048 x 512 the block-per-row form spent as many
// bytes on 1184 partial rows as on the data (8.7 us and 4.5 us to fold them).
template <int VPT>
__global__ void __launch_bounds__(256, VPT <= 2 ? 2 : 1)
layernorm_bwd_warp_kernel(const bf16 *dy, const bf16 *x, const bf16 *gamma, const float *mean,
                          const float *rstd, bf16 *__restrict__ dx, bf16 *__restrict__ dx2, float *__restrict__ partial, int rows,
                          int acc1, int acc2) {
  pdl_entry(dx, dx2);
  constexpr int COLS = 256 * VPT;
  __shared__ float red[8][COLS];
  __shared__ float g_s[COLS];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < COLS; i += 256) g_s[i] = gamma ? bf2f(gamma[i]) : 1.f;
  __syncthreads();
  float dg[VPT][8], db[VPT][8];
#pragma unroll
  for (int i = 0; i < VPT; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) { dg[i][j] = 0.f; db[i][j] = 0.f; }
  uint4 ng[VPT], nx[VPT];
  const int first = blockIdx.x * 8 + wid, step = gridDim.x * 8;
  float nmu = 0.f, nrs = 0.f;
  auto fetch = [&](int row) {
    const uint4 *pg = reinterpret_cast<const uint4 *>(dy + (long long)row * COLS), *px = reinterpret_cast<const uint4 *>(x + (long long)row * COLS);
#pragma unroll
    for (int i = 0; i < VPT; ++i) { ng[i] = pg[i * 32 + lane]; nx[i] = px[i * 32 + lane]; }
    nmu = mean[row];
    nrs = rstd[row];
  };
  if (first < rows) fetch(first);
  for (int row = first; row < rows; row += step) {
    float g[VPT][8], xh[VPT][8];
    const float mu = nmu, rs = nrs;
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) { unpack8(ng[i], g[i]); unpack8(nx[i], xh[i]); }
    if (row + step < rows) fetch(row + step);
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const float4 ga = *reinterpret_cast<const float4 *>(g_s + (i * 32 + lane) * 8), gb = *reinterpret_cast<const float4 *>(g_s + (i * 32 + lane) * 8 + 4);
      const float gm[8] = {ga.x, ga.y, ga.z, ga.w, gb.x, gb.y, gb.z, gb.w};
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        xh[i][j] = (xh[i][j] - mu) * rs;
        dg[i][j] += g[i][j] * xh[i][j];
        db[i][j] += g[i][j];
        g[i][j] *= gm[j];
        s1 += g[i][j];
        s2 += g[i][j] * xh[i][j];
      }
    }
    s1 = warp_sum(s1);
    s2 = warp_sum(s2);
    const float m1 = s1 / COLS, m2 = s2 / COLS;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const long long off = (long long)row * COLS + (i * 32 + lane) * 8;
      float o[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = rs * (g[i][j] - m1 - xh[i][j] * m2);
      if (dx2) {
        float t[8];
        if (acc2) {
          ld8(dx2 + off, t);
#pragma unroll
          for (int j = 0; j < 8; ++j) t[j] += o[j];
          st8(dx2 + off, t);
        } else st8(dx2 + off, o);
      }
      if (acc1) {
        float t[8];
        ld8(dx + off, t);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] += t[j];
      }
      st8(dx + off, o);
    }
  }
  if (!partial) return;
#pragma unroll
  for (int which = 0; which < 2; ++which) {
    if (which) __syncthreads();
#pragma unroll
    for (int i = 0; i < VPT; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) red[wid][(i * 32 + lane) * 8 + j] = which ? db[i][j] : dg[i][j];
    __syncthreads();
    for (int c = threadIdx.x; c < COLS; c += 256) {
      float s = 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) s += red[k][c];
      partial[((long long)which * gridDim.x + blockIdx.x) * COLS + c] = s;
    }
  }
}

// ---------------------------------------------------------------- bias / activation backward
// block (32, 8): thread (tx, ty) owns columns [blockIdx.x*256 + tx*8, +8) of rows ty, ty+8*gridDim.y, ...
// dz = dy * act'(saved); partial[blockIdx.y][col] = column sums over this block's rows.
// With drop_p > 0 the incoming gradient first goes back through the dropout that the forward GEMM epilogue
// applied after the activation (mask regenerated from (seed, flat index)).
static __global__ void bias_act_bwd_vec_kernel(const bf16 *dy, const bf16 *saved, bf16 *__restrict__ dz,
                                        float *__restrict__ partial, int rows, int cols, int act, float drop_p,
                                        unsigned long long drop_salt, const unsigned long long *drop_seed_ptr) {
  pdl_entry();
  const unsigned long long dseed = drop_seed_ptr ? drop_salt * 0x9E3779B97F4A7C15ull + *drop_seed_ptr : drop_salt;
  const uint32_t dthr = ffk_drop_threshold(drop_p);
  const float dscale = drop_p > 0.f ? 1.f / (1.f - drop_p) : 1.f;
  __shared__ float red[8][32][9];
  const int c0 = blockIdx.x * 256 + threadIdx.x * 8;
  float acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.f;
  if (c0 < cols) {
    for (int r = blockIdx.y * 8 + threadIdx.y; r < rows; r += gridDim.y * 8) {
      long long off = (long long)r * cols + c0;
      float g[8];
      ld8(dy + off, g);
      if (drop_p > 0.f) {
        const uint32_t k0 = ffk_keep4(dseed, (unsigned long long)(off >> 2), dthr), k1 = ffk_keep4(dseed, (unsigned long long)(off >> 2) + 1, dthr);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          g[j] = ((k0 >> j) & 1u) ? g[j] * dscale : 0.f;
          g[4 + j] = ((k1 >> j) & 1u) ? g[4 + j] * dscale : 0.f;
        }
      }
      if (act != ACT_NONE) {
        float sv[8];
        ld8(saved + off, sv);
#pragma unroll
        for (int j = 0; j < 8; ++j) g[j] *= act_bwd(sv[j], act);
      }
      if (dz) st8(dz + off, g);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += g[j];
    }
  }
  if (!partial) return;
#pragma unroll
  for (int j = 0; j < 8; ++j) red[threadIdx.y][threadIdx.x][j] = acc[j];
  __syncthreads();
  if (threadIdx.y == 0 && c0 < cols) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float s = 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) s += red[k][threadIdx.x][j];
      partial[(long long)blockIdx.y * cols + c0 + j] = s;
    }
  }
}

// out[c] (+)= sum over p < nparts of partial[p][c], for two stacked partial arrays at once (the second at
// partial + nparts * cols, out2 may be null).  Block (32 columns x 32 part lanes): a lane strides over the parts with
// independent loads, the lanes' sums meet in shared memory in a fixed order (deterministic).  The one-thread-per-column
// form took 60 us for 1184 parts of 768 columns: three blocks, each thread a chain of 1184 dependent additions.
template <typename T>
__global__ void fold_partials_kernel(const float *partial, int nparts, int cols, T *out, T *out2, int accumulate) {
  pdl_entry();
  __shared__ float s1[32][33], s2[32][33];
  const int tx = threadIdx.x, ty = threadIdx.y, c = blockIdx.x * 32 + tx;
  float a = 0.f, b = 0.f;
  if (c < cols) {
    const float *p1 = partial + c, *p2 = partial + (long long)nparts * cols + c;
#pragma unroll 4
    for (int p = ty; p < nparts; p += 32) {
      a += p1[(long long)p * cols];
      if (out2) b += p2[(long long)p * cols];
    }
  }
  s1[ty][tx] = a;
  s2[ty][tx] = b;
  __syncthreads();
  if (ty == 0 && c < cols) {
    float ta = 0.f, tb = 0.f;
#pragma unroll
    for (int k = 0; k < 32; ++k) { ta += s1[k][tx]; tb += s2[k][tx]; }
    if (out) out[c] = (T)(accumulate ? (float)out[c] + ta : ta);
    if (out2) out2[c] = (T)(accumulate ? (float)out2[c] + tb : tb);
  }
}

}  // namespace vec
