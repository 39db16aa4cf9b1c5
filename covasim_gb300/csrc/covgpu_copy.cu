// covgpu_copy: one launch over many arrays (a state's rewind, checkpoint or
// snapshot), and the outcome sums of a finished run.
#include <cuda_runtime.h>
#include <stdint.h>
#include "covgpu.h"
#include "covgpu_device.cuh"
#include "covgpu_launch.cuh"

using namespace covgpu;

namespace {

// A rewind copies or clears about 25 arrays, most of them a few bytes to a few
// megabytes: as launches of their own they cost the host 8-10 us each. Here they
// are one launch: the spans travel as the kernel's parameters, each is cut into
// chunks of COPY_CHUNK bytes, and blocks take chunks with a grid stride, 16 bytes
// a thread with COPY_VEC of them in flight (memory-bound: a chunk is 8 KB read
// and 8 KB written).
constexpr int COPY_SPANS = 40;       // spans per launch (their records fit the parameter space)
constexpr int COPY_THREADS = 256, COPY_VEC = 2;
constexpr int64_t COPY_CHUNK = COPY_THREADS * COPY_VEC * 16;
struct CopyArgs {
  covgpu_span s[COPY_SPANS];
  int64_t first[COPY_SPANS + 1];  // each span's first chunk
  int n;
};

__global__ void __launch_bounds__(COPY_THREADS) k_copy_spans(const __grid_constant__ CopyArgs a) {
  for (int64_t c = blockIdx.x; c < a.first[a.n]; c += gridDim.x) {
    int k = 0;
    while (c >= a.first[k + 1]) ++k;
    const covgpu_span& s = a.s[k];
    const int64_t lo = (c - a.first[k]) * COPY_CHUNK, len = min(COPY_CHUNK, s.bytes - lo);
    unsigned char* dst = static_cast<unsigned char*>(s.dst) + lo;
    const unsigned char* src = s.src ? static_cast<const unsigned char*>(s.src) + lo : nullptr;
    const bool vec = ((reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(src)) & 15u) == 0;
    const int64_t words = vec ? len >> 4 : 0;  // whole 16-byte words; the rest byte by byte
    const uint32_t f = (uint32_t)(s.fill & 0xFF) * 0x01010101u;
    uint4 x[COPY_VEC];
#pragma unroll
    for (int u = 0; u < COPY_VEC; ++u) {
      const int64_t w = threadIdx.x + (int64_t)u * COPY_THREADS;
      x[u] = src && w < words ? reinterpret_cast<const uint4*>(src)[w] : make_uint4(f, f, f, f);
    }
#pragma unroll
    for (int u = 0; u < COPY_VEC; ++u) {
      const int64_t w = threadIdx.x + (int64_t)u * COPY_THREADS;
      if (w < words) reinterpret_cast<uint4*>(dst)[w] = x[u];
    }
    for (int64_t b = 16 * words + threadIdx.x; b < len; b += COPY_THREADS)
      dst[b] = src ? src[b] : (unsigned char)s.fill;
  }
}

// sim.py:920-932: per block, the number of outcomes (recoveries and deaths), the sum
// of their dates and the sum of those agents' infectious dates (float64, each thread
// over its agents in order, then a tree: the same for every run). A barrier after each
// step of the tree, the last one included: its sums are stored by other threads of the
// warp than the one that formed them.
constexpr int SUM_THREADS = 256;
__global__ void __launch_bounds__(SUM_THREADS) k_outcome_sums(const float* __restrict__ rec,
                                                              const float* __restrict__ dead,
                                                              const float* __restrict__ inf, int64_t n,
                                                              double* __restrict__ out) {
  double cnt = 0.0, s_out = 0.0, s_inf = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * SUM_THREADS + threadIdx.x; i < n; i += (int64_t)gridDim.x * SUM_THREADS) {
    const float r = rec[i], d = dead[i], f = inf[i];
    if (!isnan(r)) { cnt += 1.0; s_out += (double)r; s_inf += (double)f; }
    if (!isnan(d)) { cnt += 1.0; s_out += (double)d; s_inf += (double)f; }
  }
  __shared__ double s[3][SUM_THREADS];
  s[0][threadIdx.x] = cnt;
  s[1][threadIdx.x] = s_out;
  s[2][threadIdx.x] = s_inf;
  __syncthreads();
  for (int o = SUM_THREADS / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o)
      for (int k = 0; k < 3; ++k) s[k][threadIdx.x] += s[k][threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x < 3) out[3 * (int64_t)blockIdx.x + threadIdx.x] = s[threadIdx.x][0];
}

}  // namespace

extern "C" {

int covgpu_copy_spans(const covgpu_span* spans, int32_t n, void* stream) {
  if (n < 0 || (n > 0 && !spans)) return COVGPU_BADARG;
  for (int32_t k = 0; k < n; ++k)
    if (spans[k].bytes < 0 || (spans[k].bytes > 0 && !spans[k].dst)) return COVGPU_BADARG;
  for (int32_t k = 0; k < n;) {
    CopyArgs a;
    a.n = 0;
    a.first[0] = 0;
    for (; k < n && a.n < COPY_SPANS; ++k) {
      if (spans[k].bytes == 0) continue;
      a.s[a.n] = spans[k];
      a.first[a.n + 1] = a.first[a.n] + (spans[k].bytes + COPY_CHUNK - 1) / COPY_CHUNK;
      ++a.n;
    }
    if (a.n == 0) continue;
    const int64_t chunks = a.first[a.n], wave = 152 * 8;
    k_copy_spans<<<(unsigned)(chunks < wave ? chunks : wave), COPY_THREADS, 0, S(stream)>>>(a);
  }
  return launch_status();
}

int covgpu_outcome_sums(const float* date_recovered, const float* date_dead, const float* date_infectious, int64_t n,
                        double* out, void* stream) {
  if (n < 1 || !date_recovered || !date_dead || !date_infectious || !out) return COVGPU_BADARG;
  k_outcome_sums<<<COVGPU_OUTCOME_BLOCKS, SUM_THREADS, 0, S(stream)>>>(date_recovered, date_dead, date_infectious, n,
                                                                       out);
  return launch_status();
}

}  // extern "C"
