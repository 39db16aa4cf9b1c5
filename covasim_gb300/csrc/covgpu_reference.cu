// covgpu_reference: the reference's three numba functions (covasim/utils.py:38-128)
// as standalone GPU drop-ins -- compute_viral_load, compute_trans_sus and
// compute_infections (ordered output, bit-exact), with the allocation-free
// variant of compute_infections.
#include <cuda.h>
#include <cuda_runtime.h>
#include <atomic>
#include <stdint.h>
#include <stddef.h>
#include <math.h>
#include "covgpu.h"
#include "covgpu_device.cuh"
#include "covgpu_ff.cuh"
#include "covgpu_launch.cuh"

using namespace covgpu;

namespace {

constexpr int INF_TILE = 2048;         // edges per block of the ordered compute_infections
constexpr int INF_THREADS = 256;
constexpr int INF_PER_THREAD = INF_TILE / INF_THREADS;

// ============================================================ standalone kernels

__global__ void k_viral_load(int t, const float* __restrict__ ts, const float* __restrict__ tr,
                             const float* __restrict__ td, int64_t n, float frac_time, float load_ratio,
                             float high_cap, float* __restrict__ out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = viral_load_one(t, ts[i], tr[i], td[i], frac_time, load_ratio, high_cap);
}

// utils.py:82-90: rel_trans*inf*f_quar*f_asymp*f_iso*beta_layer*viral_load and
// rel_sus*sus*f_quar*(1-immunity), float32 left to right (a factor of 1.0 is exact).
__global__ void k_trans_sus(const float* __restrict__ rt, const float* __restrict__ rs,
                            const uint8_t* __restrict__ inf, const uint8_t* __restrict__ sus, float beta_layer,
                            const float* __restrict__ vl, const uint8_t* __restrict__ symp,
                            const uint8_t* __restrict__ iso, const uint8_t* __restrict__ quar, float asymp_factor,
                            float iso_factor, float quar_factor, const float* __restrict__ imm, int64_t n,
                            float* __restrict__ ort, float* __restrict__ ors) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const bool q = quar[i];
    float a = __fmul_rn(rt[i], inf[i] ? 1.0f : 0.0f);
    a = __fmul_rn(a, q ? quar_factor : 1.0f);
    a = __fmul_rn(a, symp[i] ? 1.0f : asymp_factor);
    a = __fmul_rn(a, iso[i] ? iso_factor : 1.0f);
    a = __fmul_rn(a, beta_layer);
    a = __fmul_rn(a, vl[i]);
    float b = __fmul_rn(rs[i], sus[i] ? 1.0f : 0.0f);
    b = __fmul_rn(b, q ? quar_factor : 1.0f);
    b = __fmul_rn(b, __fsub_rn(1.0f, imm[i]));
    ort[i] = a;
    ors[i] = b;
  }
}

// utils.py:113-124 for one (direction, edge): in inf_inds (source trans != 0),
// drawn (beta != 0) and u < p in float64.
struct InfArgs {
  float beta; const int32_t* p1; const int32_t* p2; const float* lb; int64_t E;
  const float* rt; const float* rs; int64_t n_agents; const double* uni; uint32_t k0, k1; int day, variant, layer;
  int32_t* status;
};
__device__ __forceinline__ bool inf_hit(const InfArgs& a, int dir, int64_t e, int32_t& src, int32_t& tgt) {
  src = dir ? a.p2[e] : a.p1[e];
  tgt = dir ? a.p1[e] : a.p2[e];
  if ((uint32_t)src >= (uint64_t)a.n_agents || (uint32_t)tgt >= (uint64_t)a.n_agents) {  // bad index: skip
    if (a.status) atomicOr(a.status, COVGPU_BADARG);
    return false;
  }
  const float st = a.rt[src];
  if (st == 0.0f) return false;
  const float p = __fmul_rn(__fmul_rn(__fmul_rn(a.beta, a.lb[e]), st), a.rs[tgt]);
  if (p == 0.0f) return false;
  double u;
  if (a.uni) {
    u = a.uni[(int64_t)dir * a.E + e];
  } else {
    const uint4 w = philox(make_uint4((uint32_t)e, (uint32_t)(e >> 32), (uint32_t)a.day,
                                      TAG_EDGE | ((uint32_t)a.variant << 8) | (uint32_t)a.layer), a.k0, a.k1);
    return dir ? bern52(w.z, w.w, p) : bern52(w.x, w.y, p);
  }
  return u < (double)p;
}

__global__ void __launch_bounds__(INF_THREADS) k_infections_count(InfArgs a, int64_t ntiles, int32_t* counts) {
  const int dir = blockIdx.y;
  const int64_t tile = blockIdx.x;
  const int64_t e0 = tile * INF_TILE + (int64_t)threadIdx.x * INF_PER_THREAD;
  int c = 0;
  for (int j = 0; j < INF_PER_THREAD; ++j) {
    const int64_t e = e0 + j;
    int32_t s, g;
    if (e < a.E && inf_hit(a, dir, e, s, g)) ++c;
  }
  __shared__ int s_sum;
  if (threadIdx.x == 0) s_sum = 0;
  __syncthreads();
  c = __reduce_add_sync(0xffffffffu, (unsigned)c);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(&s_sum, c);
  __syncthreads();
  if (threadIdx.x == 0) counts[(int64_t)dir * ntiles + tile] = s_sum;
}

// single-block exclusive scan of m counts into int64 offsets; total into *total
__global__ void __launch_bounds__(1024) k_scan(const int32_t* counts, int64_t m, int64_t* offs, int64_t* total,
                                               int64_t capacity, int32_t* status) {
  __shared__ int64_t s_part[1024];
  const int64_t per = (m + blockDim.x - 1) / blockDim.x;
  const int64_t b = threadIdx.x * per, e = min(b + per, m);
  int64_t sum = 0;
  for (int64_t i = b; i < e; ++i) sum += counts[i];
  s_part[threadIdx.x] = sum;
  __syncthreads();
  for (int off = 1; off < (int)blockDim.x; off <<= 1) {  // Hillis-Steele inclusive scan
    const int64_t v = threadIdx.x >= (unsigned)off ? s_part[threadIdx.x - off] : 0;
    __syncthreads();
    s_part[threadIdx.x] += v;
    __syncthreads();
  }
  int64_t run = s_part[threadIdx.x] - sum;
  for (int64_t i = b; i < e; ++i) { offs[i] = run; run += counts[i]; }
  if (threadIdx.x == blockDim.x - 1) {
    *total = s_part[threadIdx.x];
    if (s_part[threadIdx.x] > capacity && status) atomicOr(status, COVGPU_OVERFLOW);
  }
}

// ordered write: block-level exclusive scan of per-thread hit counts keeps edge order
__global__ void __launch_bounds__(INF_THREADS) k_infections_write(InfArgs a, int64_t ntiles, const int64_t* offs,
                                                                  int32_t* out_src, int32_t* out_tgt, int64_t cap) {
  const int dir = blockIdx.y;
  const int64_t tile = blockIdx.x;
  const int64_t e0 = tile * INF_TILE + (int64_t)threadIdx.x * INF_PER_THREAD;
  uint32_t hits = 0;
  int32_t hs[INF_PER_THREAD], ht[INF_PER_THREAD];
#pragma unroll
  for (int j = 0; j < INF_PER_THREAD; ++j) {
    const int64_t e = e0 + j;
    int32_t s = 0, g = 0;
    if (e < a.E && inf_hit(a, dir, e, s, g)) hits |= 1u << j;
    hs[j] = s;
    ht[j] = g;
  }
  const int c = __popc(hits);
  // block exclusive scan of c (warp shuffle scan + warp totals in shared memory)
  __shared__ int s_warp[INF_THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int w = lane < INF_THREADS / 32 ? s_warp[lane] : 0;
    int wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += v;
    }
    if (lane < INF_THREADS / 32) s_warp[lane] = wi - w;
  }
  __syncthreads();
  int64_t pos = offs[(int64_t)dir * ntiles + tile] + s_warp[warp] + (incl - c);
#pragma unroll
  for (int j = 0; j < INF_PER_THREAD; ++j) {
    if (hits & (1u << j)) {
      if (pos < cap) { out_src[pos] = hs[j]; out_tgt[pos] = ht[j]; }
      ++pos;
    }
  }
}

// ============================================================ infections: find, then emit
//
// compute_infections in one evaluation of each edge instead of two. k_inf_find
// streams the edge lists once, each block a contiguous range: a round's eight
// rel_trans lookups are issued together, then the rel_sus lookups of the
// directions whose source transmits, and the directions with both nonzero are
// queued per warp in shared memory with the two values, so that the weight, the
// Philox block and the comparison run 32 candidates at a time on full warps. A bit
// per (direction, edge) that transmits goes to a mask, which keeps the reference's
// order for any order of evaluation; k_inf_emit turns the bits into the ordered
// lists and touches only the edges that hit.
// What bounds it: 32-byte sectors from L2 (one a random rel_trans lookup, one a
// rel_sus lookup, the weights of the candidate edges), about 600 MB of them for
// 10M edges of 1M agents, 15% infectious. Measured there: 57 us and 5-9 us for the
// emit, against 114 + 9 + 119 us for the two-pass form (200,000 edges of 20,000
// agents: 6.5 us). Two blocks of 512 threads per SM: one takes 68 us, three (40
// registers) 72 us, four (32, spilling) 93 us: past 32 warps the lookups of more
// ranges only contend. A source bitmap, built first and held in shared memory,
// took 62 us with the values gathered again for the candidates.
constexpr int FIND_THREADS = 512;
constexpr int FIND_PER_SM = 2;
constexpr int FIND_WARPS = FIND_THREADS / 32;
constexpr int FIND_ROUND = 128;        // edges a warp reads per round (one int4 of each list per lane)
constexpr int FIND_Q = 96;             // queue entries per warp: fewer than 32 left over + 64 pushed per edge slot
constexpr int EMIT_THREADS = 256;
constexpr int64_t FIND_MAX_BLOCKS = 2048;  // count slots in scratch
constexpr int64_t FIND_MAX_EDGES = 1ll << 36;  // a block's range stays below the queue's 2^31 edges

struct FindQueue {
  float st[FIND_Q], rs[FIND_Q];
  uint32_t m[FIND_Q];  // (edge within the block's range) << 1 | direction
};

// the block's edges: [b * per, min(E, (b + 1) * per)), per a multiple of FIND_ROUND
struct FindArgs {
  InfArgs a;
  int64_t per;
  uint32_t* mask;        // hit bits: direction 0 then direction 1, mask_words each
  int64_t mask_words;
  int32_t* counts;       // [2][gridDim.x] hits per direction and block
  int64_t* total;        // their sum is added to it
};

// one queued direction (source's trans st, target's sus rs, both nonzero): p as
// inf_hit forms it, the draw, and the hit's bit
__device__ __forceinline__ void find_try(const FindArgs& f, int64_t e_lo, float st, float rs, uint32_t m, int& n0,
                                         int& n1) {
  const InfArgs& a = f.a;
  const int64_t e = e_lo + (m >> 1);
  const int dir = (int)(m & 1u);
  const float p = __fmul_rn(__fmul_rn(__fmul_rn(a.beta, __ldg(a.lb + e)), st), rs);
  if (p == 0.0f) return;
  bool hit;
  if (a.uni) {
    hit = a.uni[(int64_t)dir * a.E + e] < (double)p;
  } else {
    const uint4 w = philox(make_uint4((uint32_t)e, (uint32_t)(e >> 32), (uint32_t)a.day,
                                      TAG_EDGE | ((uint32_t)a.variant << 8) | (uint32_t)a.layer), a.k0, a.k1);
    hit = bern52(dir ? w.z : w.x, dir ? w.w : w.y, p);
  }
  if (!hit) return;
  atomicOr(f.mask + (int64_t)dir * f.mask_words + (e >> 5), 1u << (e & 31));
  if (dir) ++n1; else ++n0;
}

__global__ void __launch_bounds__(FIND_THREADS, FIND_PER_SM) k_inf_find(FindArgs f) {
  __shared__ FindQueue s_q[FIND_WARPS];
  __shared__ int s_n[2];
  const InfArgs& a = f.a;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  FindQueue& q = s_q[warp];
  if (threadIdx.x < 2) s_n[threadIdx.x] = 0;
  const int64_t e_lo = (int64_t)blockIdx.x * f.per, e_hi = min(a.E, e_lo + f.per);
  const bool vec = ((reinterpret_cast<uintptr_t>(a.p1) | reinterpret_cast<uintptr_t>(a.p2)) & 15u) == 0;
  auto fetch = [&](int64_t eb, int4& xa, int4& xb) {  // edges eb .. eb + 3; 0 past the end
    if (vec && eb + 4 <= e_hi) {
      xa = ld_stream_v4(a.p1 + eb);
      xb = ld_stream_v4(a.p2 + eb);
    } else {
      xa.x = eb < e_hi ? a.p1[eb] : 0;          xb.x = eb < e_hi ? a.p2[eb] : 0;
      xa.y = eb + 1 < e_hi ? a.p1[eb + 1] : 0;  xb.y = eb + 1 < e_hi ? a.p2[eb + 1] : 0;
      xa.z = eb + 2 < e_hi ? a.p1[eb + 2] : 0;  xb.z = eb + 2 < e_hi ? a.p2[eb + 2] : 0;
      xa.w = eb + 3 < e_hi ? a.p1[eb + 3] : 0;  xb.w = eb + 3 < e_hi ? a.p2[eb + 3] : 0;
    }
  };
  const int64_t stride = (int64_t)FIND_WARPS * FIND_ROUND;
  int64_t rb = e_lo + (int64_t)warp * FIND_ROUND;
  int4 na = make_int4(0, 0, 0, 0), nb = na;
  if (rb < e_hi) fetch(rb + 4 * lane, na, nb);
  // the range's mask words start clear (a block's words are its own: per is whole words)
  const int64_t w_lo = e_lo >> 5, w_hi = (e_hi + 31) >> 5;
  for (int64_t w = w_lo + threadIdx.x; w < w_hi; w += FIND_THREADS) f.mask[w] = f.mask[f.mask_words + w] = 0u;
  __syncthreads();
  int qn = 0, n0 = 0, n1 = 0;
  bool bad = false;
  for (; rb < e_hi; rb += stride) {
    const int32_t pa[4] = {na.x, na.y, na.z, na.w}, pb[4] = {nb.x, nb.y, nb.z, nb.w};
    if (rb + stride < e_hi) fetch(rb + stride + 4 * lane, na, nb);
    float ta[4], tb[4], va[4], vb[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const bool in = rb + 4 * lane + j < e_hi;
      const bool ok = (uint64_t)(uint32_t)pa[j] < (uint64_t)a.n_agents && (uint64_t)(uint32_t)pb[j] < (uint64_t)a.n_agents;
      bad |= in && !ok;
      ta[j] = in && ok ? __ldg(a.rt + pa[j]) : 0.0f;
      tb[j] = in && ok ? __ldg(a.rt + pb[j]) : 0.0f;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {  // a NaN counts as nonzero, as in the reference's comparison
      va[j] = ta[j] != 0.0f ? __ldg(a.rs + pb[j]) : 0.0f;
      vb[j] = tb[j] != 0.0f ? __ldg(a.rs + pa[j]) : 0.0f;
    }
    const uint32_t m0 = (uint32_t)(rb - e_lo + 4 * lane) << 1;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const bool ca = va[j] != 0.0f, cb = vb[j] != 0.0f;
      const unsigned ba = __ballot_sync(0xffffffffu, ca), bb = __ballot_sync(0xffffffffu, cb);
      if (!(ba | bb)) continue;
      if (ca) {
        const int k = qn + __popc(ba & below);
        q.st[k] = ta[j]; q.rs[k] = va[j]; q.m[k] = m0 + 2 * j;
      }
      qn += __popc(ba);
      if (cb) {
        const int k = qn + __popc(bb & below);
        q.st[k] = tb[j]; q.rs[k] = vb[j]; q.m[k] = m0 + 2 * j + 1;
      }
      qn += __popc(bb);
      __syncwarp();
      while (qn >= 32) {  // full warps from the top of the queue (the order does not matter)
        qn -= 32;
        find_try(f, e_lo, q.st[qn + lane], q.rs[qn + lane], q.m[qn + lane], n0, n1);
      }
      __syncwarp();
    }
  }
  if (lane < qn) find_try(f, e_lo, q.st[lane], q.rs[lane], q.m[lane], n0, n1);
  n0 = __reduce_add_sync(0xffffffffu, (unsigned)n0);
  n1 = __reduce_add_sync(0xffffffffu, (unsigned)n1);
  if (lane == 0 && n0) atomicAdd(&s_n[0], n0);
  if (lane == 0 && n1) atomicAdd(&s_n[1], n1);
  if (bad && a.status) atomicOr(a.status, COVGPU_BADARG);
  __syncthreads();
  if (threadIdx.x < 2) f.counts[threadIdx.x * gridDim.x + blockIdx.x] = s_n[threadIdx.x];
  if (threadIdx.x == 0 && s_n[0] + s_n[1])
    atomicAdd(reinterpret_cast<unsigned long long*>(f.total), (unsigned long long)(s_n[0] + s_n[1]));
}

// One block per (range of k_inf_find, direction): its first output position is the
// sum of the counts before it (all of direction 0 for direction 1), then its mask
// words, a contiguous run per thread, are scanned and written in order.
__global__ void __launch_bounds__(EMIT_THREADS) k_inf_emit(FindArgs f, int nblocks, int32_t* out_src, int32_t* out_tgt,
                                                           int64_t cap, int32_t* status) {
  pdl_wait();
  const int dir = blockIdx.x >= (unsigned)nblocks ? 1 : 0, b = (int)blockIdx.x - dir * nblocks;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __shared__ long long s_red[EMIT_THREADS / 32];
  __shared__ int s_warp[EMIT_THREADS / 32];
  if (blockIdx.x == 0 && threadIdx.x == 0 && status && f.total && *f.total > cap) atomicOr(status, COVGPU_OVERFLOW);
  if (f.counts[blockIdx.x] == 0) return;  // block-uniform
  long long before = 0;
  for (int k = threadIdx.x; k < (int)blockIdx.x; k += EMIT_THREADS) before += f.counts[k];
  before = warp_sum_ll(before);
  if (lane == 0) s_red[warp] = before;
  const int64_t w_lo = (int64_t)b * (f.per >> 5), w_hi = min((f.a.E + 31) >> 5, w_lo + (f.per >> 5));
  const int64_t per_thread = (w_hi - w_lo + EMIT_THREADS - 1) / EMIT_THREADS;
  const int64_t w0 = min(w_hi, w_lo + (int64_t)threadIdx.x * per_thread), w1 = min(w_hi, w0 + per_thread);
  const uint32_t* mask = f.mask + (int64_t)dir * f.mask_words;
  int c = 0;
  for (int64_t w = w0; w < w1; ++w) c += __popc(mask[w]);
  int incl = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  long long pos = incl - c;
  for (int k = 0; k < EMIT_THREADS / 32; ++k) {
    pos += s_red[k];
    if (k < warp) pos += s_warp[k];
  }
  for (int64_t w = w0; w < w1; ++w)
    for (uint32_t x = mask[w]; x; x &= x - 1) {
      if (pos >= cap) return;
      const int64_t e = 32 * w + (__ffs(x) - 1);
      const int32_t i1 = f.a.p1[e], i2 = f.a.p2[e];
      out_src[pos] = dir ? i2 : i1;
      out_tgt[pos] = dir ? i1 : i2;
      ++pos;
    }
}

// the scratch of find and emit: the counts, then the hit masks
int64_t find_mask_words(int64_t n_edges) { return (n_edges + 31) >> 5; }
int64_t find_bytes(int64_t n_edges) {
  return 2 * FIND_MAX_BLOCKS * (int64_t)sizeof(int32_t) + 8 * find_mask_words(n_edges);
}

// one wave of blocks over ranges of whole rounds (a range is at least one)
FindArgs find_args(const InfArgs& a, void* scratch, int64_t* total, int& blocks) {
  FindArgs f;
  f.a = a;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1) {
    cudaGetLastError();
    sms = 152;
  }
  int64_t wave = (int64_t)sms * FIND_PER_SM;
  if (wave > FIND_MAX_BLOCKS) wave = FIND_MAX_BLOCKS;
  f.per = (a.E + wave - 1) / wave;
  f.per = (f.per + FIND_ROUND - 1) / FIND_ROUND * FIND_ROUND;
  blocks = (int)((a.E + f.per - 1) / f.per);
  f.counts = reinterpret_cast<int32_t*>(scratch);
  f.mask = reinterpret_cast<uint32_t*>(f.counts + 2 * FIND_MAX_BLOCKS);
  f.mask_words = find_mask_words(a.E);
  f.total = total;
  return f;
}

// The two-pass form (each edge evaluated by the count and again by the write), for
// scratch too small for the hit masks (covgpu_infections_noalloc's fixed array).
int two_pass_launch(const InfArgs& a, void* scratch, int32_t* out_src, int32_t* out_tgt, int64_t capacity,
                    int64_t* out_count, cudaStream_t s) {
  const int64_t ntiles = (a.E + INF_TILE - 1) / INF_TILE;
  if (ntiles > 0x7FFFFFFF) return COVGPU_BADARG;
  const int64_t m = 2 * ntiles;
  int64_t* offs = reinterpret_cast<int64_t*>(scratch);
  int32_t* counts = reinterpret_cast<int32_t*>(offs + m);
  dim3 grid((unsigned)ntiles, 2);
  k_infections_count<<<grid, INF_THREADS, 0, s>>>(a, ntiles, counts);
  k_scan<<<1, 1024, 0, s>>>(counts, m, offs, out_count, capacity, a.status);
  k_infections_write<<<grid, INF_THREADS, 0, s>>>(a, ntiles, offs, out_src, out_tgt, capacity);
  return launch_status();
}
int64_t two_pass_bytes(int64_t n_edges) {
  const int64_t ntiles = (n_edges + INF_TILE - 1) / INF_TILE;
  const int64_t m = 2 * (ntiles > 0 ? ntiles : 1);
  return m * (int64_t)sizeof(int64_t) + m * (int64_t)sizeof(int32_t) + 256;
}

}  // namespace

extern "C" {

int covgpu_viral_load(int32_t t, const float* date_inf, const float* date_rec, const float* date_dead, int64_t n,
                      float frac_time, float load_ratio, float high_cap, float* out_load, void* stream) {
  if (n < 0 || (n > 0 && (!date_inf || !date_rec || !date_dead || !out_load))) return COVGPU_BADARG;
  if (n == 0) return COVGPU_OK;
  k_viral_load<<<grid_for(n, 256), 256, 0, S(stream)>>>(t, date_inf, date_rec, date_dead, n, frac_time, load_ratio,
                                                         high_cap, out_load);
  return launch_status();
}

int covgpu_trans_sus(const float* rel_trans, const float* rel_sus, const uint8_t* inf, const uint8_t* sus,
                     float beta_layer, const float* viral_load, const uint8_t* symp, const uint8_t* iso,
                     const uint8_t* quar, float asymp_factor, float iso_factor, float quar_factor,
                     const float* immunity_factors, int64_t n, float* out_rel_trans, float* out_rel_sus,
                     void* stream) {
  if (n < 0) return COVGPU_BADARG;
  if (n == 0) return COVGPU_OK;
  if (!rel_trans || !rel_sus || !inf || !sus || !viral_load || !symp || !iso || !quar || !immunity_factors ||
      !out_rel_trans || !out_rel_sus)
    return COVGPU_BADARG;
  k_trans_sus<<<grid_for(n, 256), 256, 0, S(stream)>>>(rel_trans, rel_sus, inf, sus, beta_layer, viral_load, symp, iso,
                                                        quar, asymp_factor, iso_factor, quar_factor, immunity_factors,
                                                        n, out_rel_trans, out_rel_sus);
  return launch_status();
}

int64_t covgpu_infections_scratch_bytes(int64_t n_edges) {
  if (n_edges < 0) return -1;
  const int64_t two = two_pass_bytes(n_edges), one = find_bytes(n_edges);
  return one > two ? one : two;
}

int covgpu_infections(float beta, const int32_t* p1, const int32_t* p2, const float* layer_betas, int64_t n_edges,
                      const float* rel_trans, const float* rel_sus, int64_t n_agents, const double* uniforms,
                      uint64_t seed, int32_t day,
                      int32_t variant, int32_t layer, int32_t* out_src, int32_t* out_tgt, int64_t capacity,
                      int64_t* out_count, int32_t* status, void* scratch, int64_t scratch_bytes, void* stream) {
  if (n_edges < 0 || capacity < 0 || n_agents < 0 || !out_count) return COVGPU_BADARG;
  if (variant < 0 || variant >= COVGPU_MAX_VARIANTS || layer < 0 || layer >= COVGPU_MAX_LAYERS) return COVGPU_BADARG;
  if (scratch_bytes < two_pass_bytes(n_edges) || !scratch) return COVGPU_BADARG;
  cudaStream_t s = S(stream);
  if (n_edges == 0) {
    return cudaMemsetAsync(out_count, 0, sizeof(int64_t), s) == cudaSuccess ? COVGPU_OK : COVGPU_CUDA_ERROR;
  }
  if (!p1 || !p2 || !layer_betas || !rel_trans || !rel_sus || (capacity > 0 && (!out_src || !out_tgt)))
    return COVGPU_BADARG;
  InfArgs a;
  a.beta = beta; a.p1 = p1; a.p2 = p2; a.lb = layer_betas; a.E = n_edges; a.rt = rel_trans; a.rs = rel_sus;
  a.n_agents = n_agents; a.status = status; a.uni = uniforms; a.k0 = (uint32_t)seed; a.k1 = (uint32_t)(seed >> 32); a.day = day; a.variant = variant;
  a.layer = layer;
  // scratch sized for the two-pass form, or a range of edges past the queue's 31-bit offsets
  if (scratch_bytes < find_bytes(n_edges) || n_edges > FIND_MAX_EDGES)
    return two_pass_launch(a, scratch, out_src, out_tgt, capacity, out_count, s);
  if (cudaMemsetAsync(out_count, 0, sizeof(int64_t), s) != cudaSuccess) return COVGPU_CUDA_ERROR;
  int blocks = 0;
  const FindArgs f = find_args(a, scratch, out_count, blocks);
  k_inf_find<<<blocks, FIND_THREADS, 0, s>>>(f);
  launch_pdl(k_inf_emit, 2u * (unsigned)blocks, EMIT_THREADS, 0, s, f, blocks, out_src, out_tgt, capacity, status);
  return launch_status();
}

int covgpu_infections_find(float beta, const int32_t* p1, const int32_t* p2, const float* layer_betas, int64_t n_edges,
                           const float* rel_trans, const float* rel_sus, int64_t n_agents, const double* uniforms,
                           uint64_t seed, int32_t day, int32_t variant, int32_t layer, int64_t* out_count,
                           void* scratch, int64_t scratch_bytes, void* stream) {
  if (n_edges < 1 || n_edges > FIND_MAX_EDGES || n_agents < 0 || !out_count || !scratch || !p1 || !p2 ||
      !layer_betas || !rel_trans || !rel_sus || variant < 0 || variant >= COVGPU_MAX_VARIANTS || layer < 0 ||
      layer >= COVGPU_MAX_LAYERS || scratch_bytes < find_bytes(n_edges))
    return COVGPU_BADARG;
  InfArgs a;
  a.beta = beta; a.p1 = p1; a.p2 = p2; a.lb = layer_betas; a.E = n_edges; a.rt = rel_trans; a.rs = rel_sus;
  a.n_agents = n_agents; a.status = reinterpret_cast<int32_t*>(out_count + 1); a.uni = uniforms;
  a.k0 = (uint32_t)seed; a.k1 = (uint32_t)(seed >> 32); a.day = day; a.variant = variant; a.layer = layer;
  int blocks = 0;
  const FindArgs f = find_args(a, scratch, out_count, blocks);
  if (cudaMemsetAsync(out_count, 0, 2 * sizeof(int64_t), S(stream)) != cudaSuccess) return COVGPU_CUDA_ERROR;
  k_inf_find<<<blocks, FIND_THREADS, 0, S(stream)>>>(f);
  return launch_status();
}

int covgpu_infections_emit(const int32_t* p1, const int32_t* p2, int64_t n_edges, const void* scratch, int64_t count,
                           int32_t* out_src, int32_t* out_tgt, void* stream) {
  if (n_edges < 1 || n_edges > FIND_MAX_EDGES || count < 0 || !p1 || !p2 || !scratch || (count > 0 && (!out_src || !out_tgt))) return COVGPU_BADARG;
  if (count == 0) return COVGPU_OK;
  InfArgs a = {};
  a.p1 = p1; a.p2 = p2; a.E = n_edges;
  int blocks = 0;
  const FindArgs f = find_args(a, const_cast<void*>(scratch), nullptr, blocks);
  k_inf_emit<<<2u * (unsigned)blocks, EMIT_THREADS, 0, S(stream)>>>(f, blocks, out_src, out_tgt, count, nullptr);
  return launch_status();
}

// ---- compute_infections without allocation: scratch in a file-scope device array
//
// For callers that may not allocate device memory at all (see the declaration in
// covgpu.h). The tile counts and offsets that covgpu_infections keeps in caller
// scratch live here instead; every call rewrites all of the part it reads, so
// nothing needs clearing between calls, and calls whose kernels overlap on the
// GPU race on it.
constexpr int64_t NOALLOC_MAX_EDGES = COVGPU_NOALLOC_MAX_EDGES;
constexpr int64_t NOALLOC_TILES = (NOALLOC_MAX_EDGES + INF_TILE - 1) / INF_TILE;
constexpr int64_t NOALLOC_SCRATCH = 2 * NOALLOC_TILES * (int64_t)(sizeof(int64_t) + sizeof(int32_t));
static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_SCRATCH];
constexpr int NOALLOC_MAX_DEVICES = 64;
// The device address of g_noalloc_scratch per device, with the context it was
// looked up in: a device reset or a new primary context (the module loaded
// again, possibly elsewhere) makes the next call look it up again. Atomic, so
// that host threads calling at the same time do not race on the cache.
struct NoallocSlot {
  std::atomic<void*> ptr{nullptr};
  std::atomic<void*> ctx{nullptr};
};
static NoallocSlot g_noalloc[NOALLOC_MAX_DEVICES];

// The current CUDA context, through the driver's cuCtxGetCurrent resolved by
// the runtime (no link against the driver library); null when unavailable.
typedef CUresult (*CtxGetCurrentFn)(CUcontext*);
static CUcontext current_context() {
  static std::atomic<CtxGetCurrentFn> fn{nullptr};
  CtxGetCurrentFn f = fn.load(std::memory_order_acquire);
  if (!f) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &p, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !p)
      return nullptr;
    f = reinterpret_cast<CtxGetCurrentFn>(p);
    fn.store(f, std::memory_order_release);
  }
  CUcontext c = nullptr;
  return f(&c) == CUDA_SUCCESS ? c : nullptr;
}

// The array's host-side name is not a device address: look the address up once
// per device (and context), with that device current.
static int noalloc_scratch(void** out) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return COVGPU_CUDA_ERROR;
  if (dev < 0 || dev >= NOALLOC_MAX_DEVICES) return COVGPU_BADARG;
  NoallocSlot& slot = g_noalloc[dev];
  void* ctx = reinterpret_cast<void*>(current_context());
  void* p = slot.ptr.load(std::memory_order_acquire);
  if (!p || !ctx || slot.ctx.load(std::memory_order_acquire) != ctx) {
    p = nullptr;
    if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) return COVGPU_CUDA_ERROR;
    slot.ctx.store(reinterpret_cast<void*>(current_context()), std::memory_order_release);
    slot.ptr.store(p, std::memory_order_release);
  }
  *out = p;
  return COVGPU_OK;
}

int covgpu_infections_noalloc(float beta, const int32_t* p1, const int32_t* p2, const float* layer_betas,
                              int64_t n_edges, const float* rel_trans, const float* rel_sus, int64_t n_agents,
                              const double* uniforms, uint64_t seed, int32_t day, int32_t variant, int32_t layer,
                              int32_t* out_src, int32_t* out_tgt, int64_t capacity, int64_t* out_count,
                              int32_t* status, void* stream) {
  if (n_edges < 0 || n_edges > NOALLOC_MAX_EDGES) return COVGPU_BADARG;
  if (capacity < 0 || n_agents < 0 || !out_count) return COVGPU_BADARG;
  if (variant < 0 || variant >= COVGPU_MAX_VARIANTS || layer < 0 || layer >= COVGPU_MAX_LAYERS) return COVGPU_BADARG;
  cudaStream_t s = S(stream);
  if (n_edges == 0) {
    return cudaMemsetAsync(out_count, 0, sizeof(int64_t), s) == cudaSuccess ? COVGPU_OK : COVGPU_CUDA_ERROR;
  }
  if (!p1 || !p2 || !layer_betas || !rel_trans || !rel_sus || (capacity > 0 && (!out_src || !out_tgt)))
    return COVGPU_BADARG;
  void* scratch = nullptr;
  const int rc = noalloc_scratch(&scratch);
  if (rc != COVGPU_OK) return rc;
  InfArgs a;
  a.beta = beta; a.p1 = p1; a.p2 = p2; a.lb = layer_betas; a.E = n_edges; a.rt = rel_trans; a.rs = rel_sus;
  a.n_agents = n_agents; a.status = status; a.uni = uniforms; a.k0 = (uint32_t)seed; a.k1 = (uint32_t)(seed >> 32);
  a.day = day; a.variant = variant; a.layer = layer;
  return two_pass_launch(a, scratch, out_src, out_tgt, capacity, out_count, s);
}

}  // extern "C"
