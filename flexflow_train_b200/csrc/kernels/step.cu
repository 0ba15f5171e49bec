// step.cu -- what a training step does around its operators: the batch and the step's scalars brought into the plan's
// buffers, and the mean loss handed to the host.
#include "common.cuh"

// One launch per step.  A step used to start with a copy or cast per input, one for the labels and two fills for the
// scalars: launches of 1.3-2 us that each cost a gap on the device and several microseconds of host time (11 of them for a
// model with 9 inputs).
enum FfkStageKind : int { STAGE_BYTES = 0, STAGE_F32_BF16 = 1, STAGE_I64_I32 = 2, STAGE_I32_I64 = 3 };
struct FfkStageSeg {
  const void *src;
  void *dst;
  long long n;      // elements (STAGE_BYTES: bytes)
  int kind;
  int first_block;  // filled in by ffk_stage_batch
};
constexpr int STAGE_MAX = 16;
struct FfkStageArgs {
  FfkStageSeg seg[STAGE_MAX];
  int nseg;
  float alpha;
  float *alpha_ptr;                // null: no scalars
  unsigned long long seed;
  unsigned long long *seed_ptr;
};

namespace {

constexpr int STAGE_THREADS = 256;
constexpr int STAGE_UNITS = STAGE_THREADS * 4;  // 16-byte units of a segment's source that one block moves: 4 loads in flight per thread

__global__ void __launch_bounds__(STAGE_THREADS) stage_batch_kernel(const __grid_constant__ FfkStageArgs a) {
  pdl_entry();
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (a.alpha_ptr) *a.alpha_ptr = a.alpha;
    if (a.seed_ptr) *a.seed_ptr = a.seed;
  }
  int k = 0;
  while (k + 1 < a.nseg && (int)blockIdx.x >= a.seg[k + 1].first_block) ++k;
  if (k >= a.nseg) return;
  const FfkStageSeg s = a.seg[k];
  const long long blk = blockIdx.x - s.first_block;
  const bool aligned = ((((uintptr_t)s.src) | ((uintptr_t)s.dst)) & 15) == 0;
  if (s.kind == STAGE_BYTES) {
    const long long nv = aligned ? s.n / 16 : 0, u0 = blk * STAGE_UNITS + threadIdx.x;
    uint4 v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (u0 + j * STAGE_THREADS < nv) v[j] = ((const uint4 *)s.src)[u0 + j * STAGE_THREADS];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (u0 + j * STAGE_THREADS < nv) ((uint4 *)s.dst)[u0 + j * STAGE_THREADS] = v[j];
    // what no 16-byte unit covers: the tail, or everything when an address is not aligned
    const long long b0 = blk * STAGE_UNITS * 16, b1 = b0 + STAGE_UNITS * 16 < s.n ? b0 + STAGE_UNITS * 16 : s.n;
    for (long long i = (nv * 16 > b0 ? nv * 16 : b0) + threadIdx.x; i < b1; i += STAGE_THREADS)
      ((unsigned char *)s.dst)[i] = ((const unsigned char *)s.src)[i];
  } else if (s.kind == STAGE_F32_BF16) {
    const long long nv = aligned ? s.n / 4 : 0, u0 = blk * STAGE_UNITS + threadIdx.x;
    float4 v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (u0 + j * STAGE_THREADS < nv) v[j] = ((const float4 *)s.src)[u0 + j * STAGE_THREADS];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (u0 + j * STAGE_THREADS < nv)
        ((uint2 *)s.dst)[u0 + j * STAGE_THREADS] = make_uint2(pack_bf162(v[j].x, v[j].y), pack_bf162(v[j].z, v[j].w));
    const long long e0 = blk * STAGE_UNITS * 4, e1 = e0 + STAGE_UNITS * 4 < s.n ? e0 + STAGE_UNITS * 4 : s.n;
    for (long long i = (nv * 4 > e0 ? nv * 4 : e0) + threadIdx.x; i < e1; i += STAGE_THREADS) ((bf16 *)s.dst)[i] = f2bf(((const float *)s.src)[i]);
  } else {
    const long long e0 = blk * STAGE_UNITS * 4, e1 = e0 + STAGE_UNITS * 4 < s.n ? e0 + STAGE_UNITS * 4 : s.n;
    if (s.kind == STAGE_I64_I32)
      for (long long i = e0 + threadIdx.x; i < e1; i += STAGE_THREADS) ((int *)s.dst)[i] = (int)((const long long *)s.src)[i];
    else
      for (long long i = e0 + threadIdx.x; i < e1; i += STAGE_THREADS) ((long long *)s.dst)[i] = ((const int *)s.src)[i];
  }
}

// Mean of the per-row losses, written straight into page-locked host memory: one launch in the place of a reduction and a
// device-to-host copy (5.8 us on the device at the end of every step that reports its loss, and one more launch).
__global__ void __launch_bounds__(1024) loss_mean_kernel(const float *rows, long long n, float *out) {
  pdl_entry();
  __shared__ float red[32];
  float s = 0.f;
  const bool aligned = (((uintptr_t)rows) & 15) == 0;
  const long long nv = aligned ? n / 4 : 0;
#pragma unroll 4
  for (long long i = threadIdx.x; i < nv; i += 1024) {
    const float4 v = ((const float4 *)rows)[i];
    s += (v.x + v.y) + (v.z + v.w);
  }
  for (long long i = nv * 4 + threadIdx.x; i < n; i += 1024) s += rows[i];
  s = block_sum(s, red);
  if (threadIdx.x == 0) *out = s / (float)n;
}

}  // namespace

FFK_API int ffk_stage_batch(const FfkStageArgs *in, cudaStream_t st) {
  FfkStageArgs a = *in;
  if (a.nseg < 0 || a.nseg > STAGE_MAX) return -2;
  int blocks = 0;
  for (int k = 0; k < a.nseg; ++k) {
    a.seg[k].first_block = blocks;
    const long long per = a.seg[k].kind == STAGE_BYTES ? STAGE_UNITS * 16 : STAGE_UNITS * 4;
    const long long b = (a.seg[k].n + per - 1) / per;
    if (b > (1 << 24)) return -2;
    blocks += (int)b;
  }
  if (blocks == 0) blocks = 1;
  ffk_launch(stage_batch_kernel, blocks, STAGE_THREADS, 0, st, a);
  return (int)cudaGetLastError();
}
FFK_API int ffk_loss_mean(const float *rows, long long n, float *out_host, cudaStream_t st) {
  if (n <= 0) return -2;
  ffk_launch(loss_mean_kernel, 1, 1024, 0, st, rows, n, out_host);
  return (int)cudaGetLastError();
}
