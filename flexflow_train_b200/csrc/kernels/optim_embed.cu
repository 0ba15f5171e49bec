// optim_embed.cu -- optimizer updates over flat parameter arenas and the
// embedding gather / scatter-add kernels.
//
// Optimizer math follows lib/kernels/src/cuda/optimizer_kernels.cu:23-44 (SGD
// with weight decay, momentum, Nesterov) and :111-133 (Adam with the
// bias-corrected step size alpha_t supplied by the host, cf.
// lib/pcg/src/pcg/optimizer_attrs.cc:7-25).  One launch updates a whole arena:
// fp32 master weights and optimizer state, gradients in bf16 or fp32, and an
// optional bf16 shadow copy written in the same pass for the next forward.
// Embedding kernels correspond to lib/kernels/src/cuda/embedding_kernels.cu:48-310.
#include "common.cuh"

namespace {

template <typename G> __device__ __forceinline__ float ldg(const G *p, long long i);
template <> __device__ __forceinline__ float ldg<float>(const float *p, long long i) { return p[i]; }
template <> __device__ __forceinline__ float ldg<bf16>(const bf16 *p, long long i) { return bf2f(p[i]); }

template <typename G>
__global__ void adam_kernel(float *__restrict__ w, float *__restrict__ m, float *__restrict__ v,
                            const G *g, bf16 *__restrict__ shadow, long long n, float alpha_t,
                            float beta1, float beta2, float eps, float wd, float gscale,
                            const float *alpha_ptr) {
  pdl_entry(w, m, v);
  // alpha_ptr (optional): bias-corrected step size kept in device memory so that a captured CUDA graph
  // sees the value of the current step.
  if (alpha_ptr) alpha_t = *alpha_ptr;
  long long stride = (long long)gridDim.x * blockDim.x * 4;
  for (long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 4; i < n; i += stride) {
    if (i + 4 <= n) {
      float4 w4 = *reinterpret_cast<float4 *>(w + i), m4 = *reinterpret_cast<float4 *>(m + i),
             v4 = *reinterpret_cast<float4 *>(v + i);
      float gg[4] = {ldg(g, i) * gscale, ldg(g, i + 1) * gscale, ldg(g, i + 2) * gscale, ldg(g, i + 3) * gscale};
      float ww[4] = {w4.x, w4.y, w4.z, w4.w}, mm[4] = {m4.x, m4.y, m4.z, m4.w}, vv[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float gt = gg[j] + wd * ww[j];
        mm[j] = beta1 * mm[j] + (1.f - beta1) * gt;
        vv[j] = beta2 * vv[j] + (1.f - beta2) * gt * gt;
        ww[j] -= alpha_t * mm[j] / (sqrtf(vv[j]) + eps);
      }
      *reinterpret_cast<float4 *>(w + i) = make_float4(ww[0], ww[1], ww[2], ww[3]);
      *reinterpret_cast<float4 *>(m + i) = make_float4(mm[0], mm[1], mm[2], mm[3]);
      *reinterpret_cast<float4 *>(v + i) = make_float4(vv[0], vv[1], vv[2], vv[3]);
      if (shadow) {
        uint2 s = make_uint2(pack_bf162(ww[0], ww[1]), pack_bf162(ww[2], ww[3]));
        *reinterpret_cast<uint2 *>(shadow + i) = s;
      }
    } else {
      for (long long k = i; k < n; ++k) {
        float gt = ldg(g, k) * gscale + wd * w[k];
        float mk = beta1 * m[k] + (1.f - beta1) * gt;
        float vk = beta2 * v[k] + (1.f - beta2) * gt * gt;
        float wk = w[k] - alpha_t * mk / (sqrtf(vk) + eps);
        w[k] = wk; m[k] = mk; v[k] = vk;
        if (shadow) shadow[k] = f2bf(wk);
      }
    }
  }
}

// four gradients from an address of a whole piece
__device__ __forceinline__ void ldg4(const float *p, float (&v)[4]) {
  const float4 u = __ldcs(reinterpret_cast<const float4 *>(p));
  v[0] = u.x; v[1] = u.y; v[2] = u.z; v[3] = u.w;
}
__device__ __forceinline__ void ldg4(const bf16 *p, float (&v)[4]) {
  const uint2 u = __ldcs(reinterpret_cast<const uint2 *>(p));
  const float2 a = unpack_bf162(u.x), b = unpack_bf162(u.y);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void to4(const float4 &q, float (&v)[4]) { v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w; }

// SGD is bound by HBM (20 bytes per parameter with momentum, bf16 gradients and a shadow).  A thread takes two groups of four
// parameters per trip and asks for all their state before it computes; what the step does not read again is streamed past L2.
// Element by element it ran at 4.8 TB/s (33.6 million parameters 139 us, now 115); the same form gave Adam, whose state already
// came in 16-byte pieces, nothing (163 us both).
__device__ __forceinline__ float sgd_step(float wk, float gk, float *mom, float lr, float momentum, int nesterov, float wd, float gscale) {
  float gt = gk * gscale + wd * wk;
  if (momentum > 0.f) {
    const float vk = *mom * momentum + gt;
    *mom = vk;
    gt = nesterov ? gt + momentum * vk : vk;
  }
  return wk - lr * gt;
}
template <typename G>
__global__ void __launch_bounds__(256) sgd_kernel(float *__restrict__ w, float *__restrict__ mom, const G *g,
                                                  bf16 *__restrict__ shadow, long long n, float lr, float momentum, int nesterov, float wd,
                                                  float gscale) {
  pdl_entry(w, mom);
  // groups of four where the arenas' addresses allow it (a slice may start anywhere)
  const bool vec = (((uintptr_t)w | (uintptr_t)(momentum > 0.f ? mom : w)) & 15) == 0 && ((uintptr_t)g & (4 * sizeof(G) - 1)) == 0 &&
                   ((uintptr_t)shadow & 7) == 0;
  const long long half = (long long)gridDim.x * blockDim.x * 4, n4 = vec ? n & ~3ll : 0;
  for (long long i0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 4; i0 < n4; i0 += 2 * half) {
    float ww[2][4], mm[2][4] = {}, gg[2][4];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const long long i = i0 + u * half;
      if (i < n4) {
        to4(__ldcs(reinterpret_cast<const float4 *>(w + i)), ww[u]);
        if (momentum > 0.f) to4(__ldcs(reinterpret_cast<const float4 *>(mom + i)), mm[u]);
        ldg4(g + i, gg[u]);
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const long long i = i0 + u * half;
      if (i < n4) {
#pragma unroll
        for (int j = 0; j < 4; ++j) ww[u][j] = sgd_step(ww[u][j], gg[u][j], &mm[u][j], lr, momentum, nesterov, wd, gscale);
        __stcs(reinterpret_cast<float4 *>(w + i), make_float4(ww[u][0], ww[u][1], ww[u][2], ww[u][3]));
        if (momentum > 0.f) __stcs(reinterpret_cast<float4 *>(mom + i), make_float4(mm[u][0], mm[u][1], mm[u][2], mm[u][3]));
        if (shadow) *reinterpret_cast<uint2 *>(shadow + i) = make_uint2(pack_bf162(ww[u][0], ww[u][1]), pack_bf162(ww[u][2], ww[u][3]));
      }
    }
  }
  for (long long k = n4 + (long long)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    float mk = momentum > 0.f ? mom[k] : 0.f;
    const float wk = sgd_step(w[k], ldg(g, k), &mk, lr, momentum, nesterov, wd, gscale);
    w[k] = wk;
    if (momentum > 0.f) mom[k] = mk;
    if (shadow) shadow[k] = f2bf(wk);
  }
}

// out[t, :] = sum_{j<bag} W[idx[t, j], :] (optionally averaged).  One warp per
// (token, 32-column chunk group); rows are read with 16-byte loads when possible.
template <typename W, typename I, typename O>
__global__ void embedding_fwd_kernel(const I *idx, const W *table, O *__restrict__ out,
                                     long long tokens, int bag, int dim, long long entries, int avg) {
  pdl_entry();
  long long total = tokens * dim;
  long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    long long t = i / dim;
    int c = (int)(i - t * dim);
    float acc = 0.f;
    for (int j = 0; j < bag; ++j) {
      long long e = (long long)idx[t * bag + j];
      if (e >= 0 && e < entries) acc += (float)table[e * dim + c];
    }
    if (avg) acc /= bag;
    out[i] = (O)acc;
  }
}
__device__ __forceinline__ void atomic_add_any(float *p, float v) { atomicAdd(p, v); }
__device__ __forceinline__ void atomic_add_any(bf16 *p, float v) { atomicAdd(p, f2bf(v)); }

template <typename W, typename I, typename O>
__global__ void embedding_bwd_kernel(const I *idx, const O *dout, W *__restrict__ dtable,
                                     long long tokens, int bag, int dim, long long entries, int avg) {
  pdl_entry();
  long long total = tokens * dim;
  long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    long long t = i / dim;
    int c = (int)(i - t * dim);
    float g = (float)dout[i];
    if (avg) g /= bag;
    for (int j = 0; j < bag; ++j) {
      long long e = (long long)idx[t * bag + j];
      if (e >= 0 && e < entries) atomic_add_any(dtable + e * dim + c, g);
    }
  }
}

// 16-byte forms: rows of a multiple of 8 elements, a thread per 16 bytes of the table (4 fp32 elements, 8 bf16), the index split in 32
// bits.  Bound by HBM (tokens x dim read and written); with one element and one 64-bit division per thread the lookup of
// 32768 x 2048 took 384 us and the scatter, whose 16-bit atomics went out one by one, 586 us.  The reductions are those of the scalar
// form (one rounding to the table's type per addition), issued a piece at a time.  A warp's pieces are neighbours: with two pieces
// of fp32 per thread each reduction covered every other 16 bytes, and a row that many tokens share took twice as long as element by element.
template <int N> __device__ __forceinline__ void load_piece(const float *p, float (&v)[N]) {
#pragma unroll
  for (int k = 0; k < N; k += 4) {
    const float4 a = *reinterpret_cast<const float4 *>(p + k);
    v[k] = a.x; v[k + 1] = a.y; v[k + 2] = a.z; v[k + 3] = a.w;
  }
}
__device__ __forceinline__ void load_piece(const bf16 *p, float (&v)[8]) {
  const uint4 u = *reinterpret_cast<const uint4 *>(p);
  const float2 a = unpack_bf162(u.x), b = unpack_bf162(u.y), c = unpack_bf162(u.z), d = unpack_bf162(u.w);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y; v[6] = d.x; v[7] = d.y;
}
__device__ __forceinline__ void load_piece(const bf16 *p, float (&v)[4]) {
  const uint2 u = *reinterpret_cast<const uint2 *>(p);
  const float2 a = unpack_bf162(u.x), b = unpack_bf162(u.y);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void store_piece(float *p, const float (&v)[4]) { *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ void store_piece(bf16 *p, const float (&v)[4]) {
  *reinterpret_cast<uint2 *>(p) = make_uint2(pack_bf162(v[0], v[1]), pack_bf162(v[2], v[3]));
}
__device__ __forceinline__ void store_piece(bf16 *p, const float (&v)[8]) {
  *reinterpret_cast<uint4 *>(p) = make_uint4(pack_bf162(v[0], v[1]), pack_bf162(v[2], v[3]), pack_bf162(v[4], v[5]), pack_bf162(v[6], v[7]));
}
__device__ __forceinline__ void red_piece(float *p, const float (&v)[4]) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]) : "memory");
}
__device__ __forceinline__ void red_piece(bf16 *p, const float (&v)[8]) {
  asm volatile("red.global.add.noftz.v4.bf16x2 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(pack_bf162(v[0], v[1])), "r"(pack_bf162(v[2], v[3])),
               "r"(pack_bf162(v[4], v[5])), "r"(pack_bf162(v[6], v[7]))
               : "memory");
}
template <typename W, typename I, typename O>
__global__ void embedding_fwd_vec_kernel(const I *idx, const W *table, O *__restrict__ out, unsigned pieces, int bag,
                                         unsigned per_row, long long entries, int avg) {
  pdl_entry();
  constexpr int N = 16 / sizeof(W);
  const unsigned stride = gridDim.x * blockDim.x;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < pieces; i += stride) {
    const unsigned t = i / per_row;
    const long long c = (long long)(i - t * per_row) * N;
    float acc[N] = {};
#pragma unroll 4
    for (int j = 0; j < bag; ++j) {
      const long long e = (long long)idx[(long long)t * bag + j];
      if (e >= 0 && e < entries) {
        float v[N];
        load_piece(table + e * per_row * N + c, v);
#pragma unroll
        for (int k = 0; k < N; ++k) acc[k] += v[k];
      }
    }
    if (avg) {
#pragma unroll
      for (int k = 0; k < N; ++k) acc[k] /= bag;
    }
    store_piece(out + (long long)i * N, acc);
  }
}
// dtable[idx] += scale * dout (avg: divided by the bag first), also the sparse SGD step with scale = -lr
template <typename W, typename I, typename O>
__global__ void embedding_scatter_vec_kernel(const I *idx, const O *dout, W *__restrict__ table, unsigned pieces,
                                             int bag, unsigned per_row, long long entries, int avg, float scale) {
  pdl_entry();
  constexpr int N = 16 / sizeof(W);
  const unsigned stride = gridDim.x * blockDim.x;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < pieces; i += stride) {
    const unsigned t = i / per_row;
    const long long c = (long long)(i - t * per_row) * N;
    float g[N];
    load_piece(dout + (long long)i * N, g);
#pragma unroll
    for (int k = 0; k < N; ++k) {
      if (avg) g[k] /= bag;
      g[k] *= scale;
    }
#pragma unroll 4
    for (int j = 0; j < bag; ++j) {
      const long long e = (long long)idx[(long long)t * bag + j];
      if (e >= 0 && e < entries) red_piece(table + e * per_row * N + c, g);
    }
  }
}
// pieces of the 16-byte forms, 0 where rows or addresses do not allow them
template <typename W> static unsigned emb_pieces(long long tokens, int dim, const void *a, const void *b) {
  const long long n = tokens * (dim / (int)(16 / sizeof(W)));
  return dim % 8 == 0 && (((uintptr_t)a | (uintptr_t)b) & 15) == 0 && n < (1ll << 31) - 148ll * 16 * 256 ? (unsigned)n : 0u;
}

// Sparse SGD for embedding tables: W[idx] -= lr * dout, applied straight from
// the output gradient (no dense table gradient is materialised).
template <typename I, typename O>
__global__ void embedding_sgd_kernel(const I *idx, const O *dout, float *__restrict__ table,
                                     long long tokens, int bag, int dim, long long entries, float lr) {
  pdl_entry();
  long long total = tokens * dim;
  long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    long long t = i / dim;
    int c = (int)(i - t * dim);
    float g = (float)dout[i] * lr;
    for (int j = 0; j < bag; ++j) {
      long long e = (long long)idx[t * bag + j];
      if (e >= 0 && e < entries) atomicAdd(table + e * dim + c, -g);
    }
  }
}

}  // namespace

// grad_dt: 0 = fp32, 1 = bf16.  shadow may be null.
FFK_API int ffk_adam_update(float *w, float *m, float *v, const void *g, void *shadow, long long n, float alpha_t,
                            float beta1, float beta2, float eps, float wd, float gscale, const float *alpha_ptr,
                            int grad_dt, cudaStream_t st) {
  if (n <= 0) return 0;
  FfkTraffic traffic(n * 28);
  int grid = ffk_blocks(n / 4 + 1, 256, 148 * 8);
  if (grad_dt == 1)
    ffk_launch(adam_kernel<bf16>, grid, 256, 0, st, w, m, v, (const bf16 *)g, (bf16 *)shadow, n, alpha_t, beta1, beta2, eps, wd, gscale, alpha_ptr);
  else
    ffk_launch(adam_kernel<float>, grid, 256, 0, st, w, m, v, (const float *)g, (bf16 *)shadow, n, alpha_t, beta1, beta2, eps, wd, gscale, alpha_ptr);
  return (int)cudaGetLastError();
}
FFK_API int ffk_sgd_update(float *w, float *mom, const void *g, void *shadow, long long n, float lr, float momentum,
                           int nesterov, float wd, float gscale, int grad_dt, cudaStream_t st) {
  if (n <= 0) return 0;
  FfkTraffic traffic(n * 20);
  int grid = ffk_blocks(n / 4 + 1, 256, 148 * 8);
  if (grad_dt == 1)
    ffk_launch(sgd_kernel<bf16>, grid, 256, 0, st, w, mom, (const bf16 *)g, (bf16 *)shadow, n, lr, momentum, nesterov, wd, gscale);
  else
    ffk_launch(sgd_kernel<float>, grid, 256, 0, st, w, mom, (const float *)g, (bf16 *)shadow, n, lr, momentum, nesterov, wd, gscale);
  return (int)cudaGetLastError();
}

template <typename W, typename I, typename O>
static int emb_launch(int which, const void *idx, const void *table_or_dtable, const void *out_or_dout, long long tokens,
                      int bag, int dim, long long entries, int avg, cudaStream_t st) {
  FfkTraffic traffic(tokens * dim * 4);
  if (const unsigned pieces = emb_pieces<W>(tokens, dim, table_or_dtable, out_or_dout)) {
    const unsigned per_row = (unsigned)(dim / (int)(16 / sizeof(W)));
    const int vgrid = ffk_blocks(pieces, 256);
    if (which == 0)
      ffk_launch(embedding_fwd_vec_kernel<W, I, O>, vgrid, 256, 0, st, (const I *)idx, (const W *)table_or_dtable, (O *)out_or_dout, pieces, bag,
                 per_row, entries, avg);
    else
      ffk_launch(embedding_scatter_vec_kernel<W, I, O>, vgrid, 256, 0, st, (const I *)idx, (const O *)out_or_dout, (W *)table_or_dtable, pieces,
                 bag, per_row, entries, avg, 1.f);
    return (int)cudaGetLastError();
  }
  int grid = ffk_blocks(tokens * dim, 256);
  if (which == 0)
    ffk_launch(embedding_fwd_kernel<W, I, O>, grid, 256, 0, st, (const I *)idx, (const W *)table_or_dtable, (O *)out_or_dout,
                                                         tokens, bag, dim, entries, avg);
  else
    ffk_launch(embedding_bwd_kernel<W, I, O>, grid, 256, 0, st, (const I *)idx, (const O *)out_or_dout, (W *)table_or_dtable,
                                                         tokens, bag, dim, entries, avg);
  return (int)cudaGetLastError();
}
static int emb_dispatch(int which, const void *idx, const void *table, const void *out, long long tokens, int bag,
                        int dim, long long entries, int avg, int table_dt, int idx_dt, int out_dt, cudaStream_t st) {
  if (tokens <= 0) return 0;
#define EMB_CASE(TD, ID, OD, W, I, O) \
  if (table_dt == TD && idx_dt == ID && out_dt == OD) return emb_launch<W, I, O>(which, idx, table, out, tokens, bag, dim, entries, avg, st);
  EMB_CASE(0, 3, 1, float, long long, bf16)
  EMB_CASE(0, 2, 1, float, int, bf16)
  EMB_CASE(0, 3, 0, float, long long, float)
  EMB_CASE(0, 2, 0, float, int, float)
  EMB_CASE(1, 3, 1, bf16, long long, bf16)
  EMB_CASE(1, 2, 1, bf16, int, bf16)
#undef EMB_CASE
  return -2;
}

// table_dt/out_dt: 0 = fp32, 1 = bf16; idx_dt: 2 = int32, 3 = int64; aggr: 0 = sum, 1 = avg
FFK_API int ffk_embedding_fwd(const void *idx, const void *table, void *out, long long tokens, int bag, int dim,
                              long long entries, int aggr, int table_dt, int idx_dt, int out_dt, cudaStream_t st) {
  return emb_dispatch(0, idx, table, out, tokens, bag, dim, entries, aggr, table_dt, idx_dt, out_dt, st);
}
// dtable += scatter(dout); the caller zeroes dtable at the start of a step.
FFK_API int ffk_embedding_bwd(const void *idx, const void *dout, void *dtable, long long tokens, int bag, int dim,
                              long long entries, int aggr, int table_dt, int idx_dt, int out_dt, cudaStream_t st) {
  return emb_dispatch(1, idx, dtable, dout, tokens, bag, dim, entries, aggr, table_dt, idx_dt, out_dt, st);
}
// fp32 table, plain SGD applied sparsely: table[idx] -= lr * dout
FFK_API int ffk_embedding_sgd(const void *idx, const void *dout, float *table, long long tokens, int bag, int dim,
                              long long entries, float lr, int idx_dt, int out_dt, cudaStream_t st) {
  if (tokens <= 0) return 0;
  if (const unsigned pieces = emb_pieces<float>(tokens, dim, table, dout)) {
    const unsigned per_row = (unsigned)(dim / 4);
    const int vgrid = ffk_blocks(pieces, 256);
#define EMB_SGD(ID, OD, I, O)                                                                                                                \
  if (idx_dt == ID && out_dt == OD) {                                                                                                        \
    ffk_launch(embedding_scatter_vec_kernel<float, I, O>, vgrid, 256, 0, st, (const I *)idx, (const O *)dout, table, pieces, bag, per_row,    \
               entries, 0, -lr);                                                                                                             \
    return (int)cudaGetLastError();                                                                                                          \
  }
    EMB_SGD(3, 1, long long, bf16)
    EMB_SGD(2, 1, int, bf16)
    EMB_SGD(3, 0, long long, float)
    EMB_SGD(2, 0, int, float)
#undef EMB_SGD
  }
  int grid = ffk_blocks(tokens * dim, 256);
  if (idx_dt == 3 && out_dt == 1) ffk_launch(embedding_sgd_kernel<long long, bf16>, grid, 256, 0, st, (const long long *)idx, (const bf16 *)dout, table, tokens, bag, dim, entries, lr);
  else if (idx_dt == 2 && out_dt == 1) ffk_launch(embedding_sgd_kernel<int, bf16>, grid, 256, 0, st, (const int *)idx, (const bf16 *)dout, table, tokens, bag, dim, entries, lr);
  else if (idx_dt == 3 && out_dt == 0) ffk_launch(embedding_sgd_kernel<long long, float>, grid, 256, 0, st, (const long long *)idx, (const float *)dout, table, tokens, bag, dim, entries, lr);
  else if (idx_dt == 2 && out_dt == 0) ffk_launch(embedding_sgd_kernel<int, float>, grid, 256, 0, st, (const int *)idx, (const float *)dout, table, tokens, bag, dim, entries, lr);
  else return -2;
  return (int)cudaGetLastError();
}
