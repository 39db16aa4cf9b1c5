// covgpu_testing: test_prob, contact_tracing and update_states_post on the device
// (covasim/interventions.py:858-1145, covasim/people.py:189-196,315-366,589-640),
// and the agent index of stored layers that tracing walks.
#include <cuda_runtime.h>
#include <stdint.h>
#include <stddef.h>
#include <math.h>
#include "covgpu.h"
#include "covgpu_device.cuh"
#include "covgpu_ff.cuh"
#include "covgpu_scan.cuh"
#include "covgpu_launch.cuh"

using namespace covgpu;

namespace {

// ============================================================ testing and tracing
//
// Day t with a test_prob / contact_tracing sim, after the agent pass and any
// importations (sim.py:596-600): k_test_pass draws who tests and marks the
// contacts of the agents to trace, and k_post_pass notifies the contacts and runs
// update_states_post. A tracing capacity, or a stored layer without an index, takes
// the marking out of the test pass: k_trace_cap, k_trace_scan and k_trace_marks
// then work from its bitmap of the traced.

__device__ __forceinline__ bool day_active(int t, int start, int end) { return t >= start && t <= end; }

// interventions.py:682-710: is agent i a quarantined tester on day t?
__device__ __forceinline__ bool quar_tester(const covgpu_state& st, const covgpu_testing& T, int64_t i, int t,
                                            uint32_t f) {
  const int qp = T.quar_policy;
  if (!qp) return false;
  bool q = false;
  if (qp & (COVGPU_QP_START | COVGPU_QP_OFFSETS)) {
    const float dq = date_row(st, COVGPU_DATE_QUARANTINED)[i];
    if ((qp & COVGPU_QP_START) && dq == (float)(t - 1)) q = true;
    if ((qp & COVGPU_QP_OFFSETS) && defined(dq)) {
      const float back = (float)(t - 1) - dq;  // exact: both are small integers when it matters
      if (back >= 0.0f && back < 32.0f && back == floorf(back) && ((T.quar_offsets >> (int)back) & 1u)) q = true;
    }
  }
  if ((qp & COVGPU_QP_END) && date_row(st, COVGPU_DATE_END_QUARANTINE)[i] == (float)(t + 1)) q = true;
  if ((qp & COVGPU_QP_DAILY) && (f & B_QUAR)) q = true;
  return q;
}

// whole days since symptom onset, as test_prob forms them: the float32 difference
// t - date_symptomatic truncated to int32 (cvd.default_int)
__device__ __forceinline__ int symp_days(const covgpu_state& st, int64_t i, int t) {
  return (int)__fsub_rn((float)t, date_row(st, COVGPU_DATE_SYMPTOMATIC)[i]);
}

// ceil(p * 2^53) (the host's prob_threshold): the Bernoulli threshold of a float64 p
__device__ __forceinline__ uint64_t prob_thr(double p) {
  if (!(p > 0.0)) return 0ull;
  if (p >= 1.0) return (1ull << 53) + 1ull;
  return __double2ull_ru(__dmul_rn(p, 9007199254740992.0));
}

// test_prob's symptomatic probability under a swab delay (interventions.py:930-938):
// pdf(days) * adjusted symp_prob * (symptomatic agents / those with the same days),
// in float64 with the reference's operations and order
__device__ __forceinline__ uint64_t swab_threshold(const covgpu_state& st, const covgpu_testing& T, int64_t i, int t) {
  const int d = symp_days(st, i, t);
  if (d < 0 || d >= T.swab_len) return 0ull;
  const double inv = __ddiv_rn((double)T.swab_bins[d], (double)T.swab_bins[T.swab_len]);
  const double cnt = __ddiv_rn(1.0, inv);
  const double x = __dmul_rn((double)d, T.symp_prob);
  const double adj = 1.0 > x ? __ddiv_rn(T.symp_prob, __dsub_rn(1.0, x)) : 1.0;
  return prob_thr(__dmul_rn(__dmul_rn(T.swab_pdf[d], adj), cnt));
}

// contact_tracing.identify_contacts, the find_contacts half (utils.py:131-147), for
// one layer of one traced agent: the other endpoint of each of its edges is marked in
// the layer's bitmap by a group of MARK_LANES lanes (sub: the lane within it), as p1
// and p2 through a stored layer's index, and the partners of its two lists (the draws
// the edge pass makes for that agent as a source) in a redrawn layer.
constexpr int MARK_LANES = 8;
__device__ __noinline__ void mark_layer(const covgpu_state& st, const covgpu_sim_params& sp, uint32_t a, int l, int sub,
                                        int t) {
  const int seg = l < sp.n_layers ? sp.seg_of_layer[l] : -1;
  if (seg < 0 || sp.testing.thr_trace[l] == 0) return;
  const covgpu_layer& L = st.segments[seg];
  const int32_t off = (int32_t)sp.agent_off;
  uint32_t* contact = st.contact_bits + (int64_t)l * ((st.n + 31) >> 5);
  if (L.dynamic) {
    const uint32_t n_local = (uint32_t)sp.n_agents, thr = bounded_thr(n_local);
    int k[2];
    dyn_counts(L.dyn_cdf, L.dyn_k, a, (uint32_t)t, (uint32_t)l, sp.key0, sp.key1, k[0], k[1]);
    const int nb0 = (k[0] + 3) >> 2, nb = nb0 + ((k[1] + 3) >> 2);  // four-entry blocks of both lists
    for (int b = sub; b < nb; b += MARK_LANES) {
      const int d = b >= nb0 ? 1 : 0, j0 = 4 * (d ? b - nb0 : b);
      const uint4 pw = dyn_partner_block(a, d, j0, (uint32_t)t, (uint32_t)l, sp.key0, sp.key1);
      for (int j = j0; j < j0 + 4 && j < k[d]; ++j) {
        const int32_t g = off + (int32_t)dyn_partner(word_of(pw, j & 3), n_local, thr, a, d, j, (uint32_t)t,
                                                     (uint32_t)l, sp.key0, sp.key1);
        atomicOr(contact + (g >> 5), 1u << (g & 31));
      }
    }
  } else if (L.rp1) {
    const uint32_t b1 = L.rp1[a], e1 = L.rp1[a + 1], b2 = L.rp2[a], e2 = L.rp2[a + 1];
    for (uint32_t k = b1 + sub; k < e1; k += MARK_LANES) {
      const int32_t g = L.p2[k];
      atomicOr(contact + (g >> 5), 1u << (g & 31));
    }
    for (uint32_t k = b2 + sub; k < e2; k += MARK_LANES) {
      const int32_t g = L.rev1 ? L.rev1[k] : L.p1[L.perm2[k]];
      atomicOr(contact + (g >> 5), 1u << (g & 31));
    }
  }
}

// The traced agents of one thread block's agent-block range, in shared memory: once
// the range is done (mark_block), the (layer, agent) pairs are shared by the block's
// groups of lanes, a warp's groups on the same layer where there are enough agents,
// so that the chains of dependent loads (row, edge, endpoint, or the lists' draws)
// run side by side instead of one after another in the warp that found the agent
// (10M agents with testing: 91.2 -> 89.7 ms a run). A median day of 300,000 agents: the
// test pass with the marks 14.3 us, against 7.8 us without them, 21.1 us for a thread
// of its own per traced agent and 12.4 us for the redrawn layer's lists, three
// launches.
constexpr int MARK_CAP = 512;
struct MarkList {
  uint32_t agent[MARK_CAP];
  unsigned n;
};
// the traced agents of one warp's 32 (bit r: agent i0 + r); those past the list's end
// are marked here, by the whole warp
__device__ __forceinline__ void mark_push(const covgpu_state& st, const covgpu_sim_params& sp, int64_t i0,
                                          uint32_t traced, int t, MarkList& list) {
  const int lane = threadIdx.x & 31;
  unsigned pos = 0;
  if (lane == 0) pos = atomicAdd(&list.n, (unsigned)__popc(traced));
  pos = __shfl_sync(0xffffffffu, pos, 0) + __popc(traced & ((1u << lane) - 1u));
  const bool mine = (traced >> lane) & 1u;
  if (mine && pos < MARK_CAP) list.agent[pos] = (uint32_t)(i0 + lane);
  for (unsigned over = __ballot_sync(0xffffffffu, mine && pos >= MARK_CAP); over; over &= over - 1) {
    const uint32_t a = (uint32_t)(i0 + (__ffs(over) - 1) - sp.agent_off);
    for (int l = lane / MARK_LANES; l < sp.n_layers; l += 32 / MARK_LANES)
      mark_layer(st, sp, a, l, lane & (MARK_LANES - 1), t);
    __syncwarp();
  }
}
__device__ __forceinline__ void mark_block(const covgpu_state& st, int t, const MarkList& list) {
  __syncthreads();
  const unsigned n = min(list.n, (unsigned)MARK_CAP);
  for (unsigned j = threadIdx.x / MARK_LANES; j < n * (unsigned)st.n_contact_layers; j += AGENT_THREADS / MARK_LANES) {
    const uint32_t i = list.agent[j % n];
    int lo = 0, hi = st.n_sims - 1;  // the agent's sim
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (st.sims[mid].agent_off <= (int64_t)i) lo = mid; else hi = mid - 1;
    }
    const covgpu_sim_params& sp = st.sims[lo];
    mark_layer(st, sp, (uint32_t)((int64_t)i - sp.agent_off), (int)(j / n), threadIdx.x & (MARK_LANES - 1), t);
  }
}

// test_prob.apply (interventions.py:921-981) + People.test (people.py:589-617),
// then the agents contact_tracing.select_cases picks (interventions.py:1066-1072).
// One agent block of the test pass (thread k on agent begin + k, its flags f and
// diagnosis date dd already loaded); the tested are counted into the thread's
// accumulator. MARK: the traced go to the block's list, else to their bitmap.
template <bool MARK>
__device__ __forceinline__ void test_block(const covgpu_state& st, int t, const covgpu_agent_block& blk, uint32_t f,
                                           float dd, unsigned& tested_acc, MarkList& list) {
  const covgpu_sim_params& sp = st.sims[blk.sim];
  const covgpu_testing& T = sp.testing;
  const bool test_on = day_active(t, T.test_start, T.test_end);
  const bool trace_on = day_active(t, T.trace_start, T.trace_end);
  if (!test_on && !trace_on) return;  // uniform over the agent block (one sim per agent block)
  const int64_t i = blk.begin + threadIdx.x;
  const bool valid = i < blk.end;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t tested = 0, trace = 0;
  if (valid) {
    if (test_on) {
      uint64_t thr = 0;
      if (!(f & B_DIAG)) {  // the diagnosed do not test
        const bool symp = f & B_SYMP;
        const int64_t loc = i - sp.agent_off;
        // quarantined testers with everyone's probabilities need not be told apart
        const bool quar_differs = T.swab_pdf || T.thr_symp_quar != T.thr_symp || T.thr_asymp_quar != T.thr_asymp;
        // an influenza-like illness without COVID symptoms: the symptomatic probability,
        // never the quarantine ones (interventions.py:966-969)
        if (!symp && T.ili_mark && T.ili_mark[loc] == t)
          thr = T.thr_symp;
        else if (quar_differs && quar_tester(st, T, i, t, f))
          thr = symp ? T.thr_symp_quar : T.thr_asymp_quar;
        else
          thr = !symp ? T.thr_asymp : (T.swab_pdf ? swab_threshold(st, T, i, t) : T.thr_symp);
        if (T.sub_thr) {  // subtargets (interventions.py:970-972)
          const uint64_t sv = T.sub_thr[loc];
          if (sv != COVGPU_NO_SUBTARGET) thr = sv;
        }
      }
      if (thr) {
        const uint32_t local = (uint32_t)(i - sp.agent_off);
        const uint4 w = philox(make_uint4(local, 0u, (uint32_t)t, TAG_TEST), sp.key0, sp.key1);
        if (bern52_thr(w.x, w.y, thr)) {
          tested = 1;
          st.flags[i] = f | B_TESTED;
          date_row(st, COVGPU_DATE_TESTED)[i] = (float)t;
          if ((f & B_INF) && bern52_thr(w.z, w.w, T.thr_sensitivity) && isnan(dd)) {
            const uint4 w1 = philox(make_uint4(local, 1u, (uint32_t)t, TAG_TEST), sp.key0, sp.key1);
            if (bern52_thr(w1.x, w1.y, T.thr_not_lost)) {
              dd = (float)(t + T.test_delay);
              date_row(st, COVGPU_DATE_DIAGNOSED)[i] = dd;
              date_row(st, COVGPU_DATE_POS_TEST)[i] = (float)t;
            }
          }
        }
      }
    }
    if (trace_on) {
      if (T.presumptive)
        trace = (date_row(st, COVGPU_DATE_TESTED)[i] == (float)t && (f & B_EXP)) ? 1u : 0u;
      else
        trace = (dd == (float)t) ? 1u : 0u;
    }
  }
  tested_acc += tested;
  const uint32_t tm = __ballot_sync(0xffffffffu, trace);
  if (MARK) {
    if (tm) mark_push(st, sp, blk.begin + warp * 32, tm, t, list);
    return;
  }
  if (trace_on && lane == 0 && blk.begin + warp * 32 < blk.end) st.trace_bits[(blk.begin + warp * 32) >> 5] = tm;
  if (tm && T.cap_list) {  // the day's cases, for the capacity's selection (k_trace_cap)
    uint32_t base = 0u;
    if (lane == 0) base = atomicAdd(T.cap_count, (uint32_t)__popc(tm));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (trace) T.cap_list[base + __popc(tm & ((1u << lane) - 1u))] = (int32_t)(i - sp.agent_off);
  }
  if (lane == 0 && tm) atomicAdd(st.trace_count + blk.sim, (unsigned)__popc(tm));
}

__device__ __forceinline__ void test_flush(const covgpu_state& st, int t, int sim, unsigned& tested_acc) {
  const unsigned n_tested = __reduce_add_sync(0xffffffffu, tested_acc);
  if ((threadIdx.x & 31) == 0 && n_tested)
    atomicAdd(reinterpret_cast<unsigned long long*>(&st.sims[sim].res_int[(int64_t)t * COVGPU_N_RES_INT + R_TESTS]),
              (unsigned long long)n_tested);
  tested_acc = 0;
}

// The per-sim preparation of day t's test pass, one block per sim: the count of the
// day's traced cases is cleared (on every day: cases with a delayed diagnosis are traced
// after test_prob's last day), test_prob's swab-delay histogram is cleared (k_swab_hist fills it), and the
// day's influenza-like illnesses (interventions.py:941-947), drawn on the host
// (they do not depend on the state), are marked with t.
__global__ void k_test_prep(covgpu_state st, int t) {
  if (held(st, t)) return;
  const int s = blockIdx.x;
  if (s >= st.n_sims) return;
  const covgpu_testing& T = st.sims[s].testing;
  if (T.cap_list && threadIdx.x == 0) *T.cap_count = 0u;
  if (!day_active(t, T.test_start, T.test_end)) return;
  if (T.swab_pdf)
    for (int k = threadIdx.x; k <= T.swab_len; k += blockDim.x) T.swab_bins[k] = 0;
  if (!T.ili_mark) return;
  const int d = t - T.test_start;
  if (d < 0 || d >= T.ili_days) return;
  const int n = st.sims[s].n_agents;
  for (int64_t k = T.ili_off[d] + threadIdx.x; k < T.ili_off[d + 1]; k += blockDim.x) {
    const int32_t a = T.ili_inds[k];
    if (a >= 0 && a < n) T.ili_mark[a] = t;
  }
}

// The passes over agents run as (at most) one wave of blocks, each walking a
// contiguous range of agent blocks [b, b_end); counts are flushed once per sim.
__device__ __forceinline__ bool agent_range(const covgpu_state& st, int64_t& b, int64_t& b_end) {
  const int64_t nb = st.n_agent_blocks;
  const int64_t per = (nb + gridDim.x - 1) / gridDim.x;
  b = (int64_t)blockIdx.x * per;
  b_end = min(nb, b + per);
  return b < b_end;
}

// test_prob's swab-delay histogram of day t (interventions.py:931-932): the
// symptomatic agents by whole days since onset, and their total in the last bin
__global__ void __launch_bounds__(AGENT_THREADS) k_swab_hist(covgpu_state st, int t) {
  if (held(st, t)) return;
  int64_t b, b_end;
  if (!agent_range(st, b, b_end)) return;
  for (; b < b_end; ++b) {
    const covgpu_agent_block blk = st.agent_blocks[b];
    const covgpu_testing& T = st.sims[blk.sim].testing;
    if (!T.swab_pdf || !day_active(t, T.test_start, T.test_end)) continue;  // uniform over the agent block
    const int64_t i = blk.begin + threadIdx.x;
    if (i >= blk.end || !(st.flags[i] & B_SYMP)) continue;
    const int d = symp_days(st, i, t);
    if (d >= 0 && d < T.swab_len) atomicAdd(T.swab_bins + d, 1);
    atomicAdd(T.swab_bins + T.swab_len, 1);
  }
}

// contact_tracing's capacity (interventions.py:1074-1078), one block per sim: when
// the day's cases exceed int(capacity / scale), a radix select over their unique
// 64-bit keys finds the capacity-th smallest, and the trace bits of the cases above
// it are cleared (a uniform random subset of exactly that size)
__device__ __forceinline__ uint64_t cap_key(const covgpu_sim_params& sp, int32_t local, int t) {
  const uint4 w = philox(make_uint4((uint32_t)local, 2u, (uint32_t)t, TAG_TEST), sp.key0, sp.key1);
  return ((uint64_t)w.x << 32) | (uint32_t)local;
}
__global__ void k_trace_cap(covgpu_state st, int t) {
  if (held(st, t)) return;
  const int s = blockIdx.x;
  if (s >= st.n_sims) return;
  const covgpu_sim_params& sp = st.sims[s];
  const covgpu_testing& T = sp.testing;
  if (!T.cap_list || !day_active(t, T.trace_start, T.trace_end)) return;
  const double scale = sp.rescale_vec ? sp.rescale_vec[t] : T.cap_scale;
  const double capd = T.capacity / scale;
  const uint32_t c = *T.cap_count;
  const int64_t cap = capd < 0.0 ? 0 : (int64_t)capd;
  if ((int64_t)c <= cap) return;
  __shared__ unsigned int hist[256];
  __shared__ unsigned long long s_prefix;
  __shared__ unsigned int s_rank;
  unsigned long long prefix = 0ull, mask = 0ull;
  unsigned int rank = (unsigned int)cap;  // the rank (1-based) of the largest key kept
  if (rank > 0) {
    for (int shift = 56; shift >= 0; shift -= 8) {
      for (int b = threadIdx.x; b < 256; b += blockDim.x) hist[b] = 0u;
      __syncthreads();
      for (uint32_t j = threadIdx.x; j < c; j += blockDim.x) {
        const uint64_t key = cap_key(sp, T.cap_list[j], t);
        if ((key & mask) == prefix) atomicAdd(&hist[(key >> shift) & 255u], 1u);
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        unsigned int cum = 0u;
        int d = 0;
        while (d < 255 && cum + hist[d] < rank) cum += hist[d++];
        s_prefix = prefix | ((unsigned long long)d << shift);
        s_rank = rank - cum;
      }
      __syncthreads();
      prefix = s_prefix;
      rank = s_rank;
      mask |= 0xFFull << shift;
      __syncthreads();
    }
  }
  for (uint32_t j = threadIdx.x; j < c; j += blockDim.x) {
    const int32_t local = T.cap_list[j];
    if (cap == 0 || cap_key(sp, local, t) > prefix) {
      const int64_t i = sp.agent_off + local;
      atomicAnd(st.trace_bits + (i >> 5), ~(1u << (i & 31)));
    }
  }
  if (threadIdx.x == 0) st.trace_count[s] = (uint32_t)cap;
}

// The test and post passes wait on memory (8 and 16 bytes an agent, little
// arithmetic), so they run at full occupancy: eight blocks of 32 registers per SM.
// On the 10M-agent testing run (the 80 days after the last variant's arrival):
// 99.3 ms, against 103.5 ms with six blocks (two agent blocks loaded at a time),
// 111.7 ms with four (four at a time) and 115.0 ms with three. A day of it, test
// 111 -> 73 us (marks included), post 172 -> 95 us: the bytes take 12 and 24 us.
constexpr int PASS_BLOCKS = 8;

template <bool MARK>
__global__ void __launch_bounds__(AGENT_THREADS, PASS_BLOCKS) k_test_pass(covgpu_state st, int t) {
  pdl_wait();
  pdl_trigger();  // one wave, all resident: the next kernel's set-up overlaps this pass
  if (held(st, t)) return;
  int64_t b, b_end;
  if (!agent_range(st, b, b_end)) return;
  __shared__ MarkList s_list;
  if (threadIdx.x == 0) s_list.n = 0;
  __syncthreads();
  int sim = st.agent_blocks[b].sim;
  unsigned tested_acc = 0;
  for (; b < b_end; ++b) {
    const covgpu_agent_block blk = st.agent_blocks[b];
    const int64_t i = blk.begin + threadIdx.x;
    uint32_t f = 0u;
    float dd = 0.0f;
    if (i < blk.end) {
      f = st.flags[i];
      dd = date_row(st, COVGPU_DATE_DIAGNOSED)[i];
    }
    if (blk.sim != sim) {
      test_flush(st, t, sim, tested_acc);
      sim = blk.sim;
    }
    test_block<MARK>(st, t, blk, f, dd, tested_acc, s_list);
  }
  test_flush(st, t, sim, tested_acc);
  if (MARK) mark_block(st, t, s_list);
}

// The marking on its own, from the test pass's bitmap of the traced (after the
// capacity's selection): one warp per agent block's word
__global__ void __launch_bounds__(AGENT_THREADS) k_trace_marks(covgpu_state st, int t) {
  if (held(st, t)) return;
  int64_t b, b_end;
  if (!agent_range(st, b, b_end)) return;
  __shared__ MarkList s_list;
  if (threadIdx.x == 0) s_list.n = 0;
  __syncthreads();
  const int warp = threadIdx.x >> 5;
  for (; b < b_end; ++b) {
    const covgpu_agent_block blk = st.agent_blocks[b];
    const covgpu_sim_params& sp = st.sims[blk.sim];
    const int64_t i0 = blk.begin + warp * 32;
    if (i0 >= blk.end || !day_active(t, sp.testing.trace_start, sp.testing.trace_end) ||
        st.trace_count[blk.sim] == 0)
      continue;
    const uint32_t tm = st.trace_bits[i0 >> 5];
    if (tm) mark_push(st, sp, i0, tm, t, s_list);
  }
  mark_block(st, t, s_list);
}

__device__ __forceinline__ uint32_t bit_of(const uint32_t* bits, int32_t a) {
  return (bits[a >> 5] >> (a & 31)) & 1u;
}

// contact_tracing.identify_contacts, the find_contacts half (utils.py:131-147):
// every edge of a stored layer without an index with a traced endpoint marks the
// other endpoint in its layer's bitmap (the others: mark_layer)
template <int ROUNDS>
__global__ void __launch_bounds__(EDGE_THREADS) k_trace_scan(covgpu_state st, int t) {
  if (held(st, t)) return;
  constexpr int64_t TILE = (int64_t)ROUNDS * EDGE_ROUND;
  __shared__ int s_seg;
  if (threadIdx.x == 0) {
    int lo = 0, hi = st.n_segments - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (st.segments[mid].tile_begin <= (int64_t)blockIdx.x) lo = mid; else hi = mid - 1;
    }
    s_seg = lo;
  }
  __syncthreads();
  const covgpu_layer* L = st.segments + s_seg;
  const covgpu_sim_params& sp = st.sims[L->sim];
  const covgpu_testing& T = sp.testing;
  if (!day_active(t, T.trace_start, T.trace_end) || T.thr_trace[L->layer] == 0 || st.trace_count[L->sim] == 0) return;
  if (L->rp1) return;  // indexed: mark_layer visits the traced agents' edges
  const int64_t words = (st.n + 31) >> 5;
  uint32_t* contact = st.contact_bits + (int64_t)L->layer * words;
  const int64_t e0 = ((int64_t)blockIdx.x - L->tile_begin) * TILE;
  const int64_t e1 = min(e0 + TILE, L->n_edges);
  const int32_t off = (int32_t)sp.agent_off;
  for (int r = 0; r < ROUNDS; ++r) {
    const int64_t eb = e0 + ((int64_t)r * EDGE_THREADS + threadIdx.x) * EDGE_VEC;
    if (eb >= e1) break;
    int32_t a[EDGE_VEC], b[EDGE_VEC];
#pragma unroll
    for (int j = 0; j < EDGE_VEC; ++j) {
      a[j] = eb + j < e1 ? __ldg(L->p1 + eb + j) : off;
      b[j] = eb + j < e1 ? __ldg(L->p2 + eb + j) : off;
    }
#pragma unroll
    for (int j = 0; j < EDGE_VEC; ++j) {
      if (eb + j >= e1) break;
      if (bit_of(st.trace_bits, a[j])) atomicOr(contact + (b[j] >> 5), 1u << (b[j] & 31));
      if (bit_of(st.trace_bits, b[j])) atomicOr(contact + (a[j] >> 5), 1u << (a[j] & 31));
    }
  }
}

// contact_tracing.notify_contacts (interventions.py:1120-1145) with the
// binomial_filter of identify_contacts, then update_states_post
// (people.py:189-196: check_diagnosed, check_quar, check_enter_iso)
// One agent block of the post pass, its fields already loaded (PostIn); the day's
// diagnoses, quarantines and isolations are counted into the thread's accumulators
struct PostIn {
  uint32_t f;
  float dpt, dd;   // date_pos_test, date_diagnosed
  int32_t pq;      // today's pending-quarantine slot
  uint32_t word;   // lane l: the warp's contact word of layer l, on tracing days
};
__device__ __forceinline__ void post_block(const covgpu_state& st, int t, const covgpu_agent_block& blk,
                                           const PostIn& in, unsigned& acc_diag, unsigned& acc_quar,
                                           unsigned& acc_iso) {
  const covgpu_sim_params& sp = st.sims[blk.sim];
  const covgpu_testing& T = sp.testing;
  const int64_t i = blk.begin + threadIdx.x;
  const bool valid = i < blk.end;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t words = (st.n + 31) >> 5;
  const int64_t w = (blk.begin + warp * 32) >> 5;
  const float tf = (float)t;
  const int R = st.pending_slots;
  unsigned c_diag = 0, c_quar = 0, c_iso = 0;
  const float nanf_ = __int_as_float(0x7fc00000);
  uint32_t f = in.f;
  const float a_dpt = in.dpt, a_dd = in.dd;
  int32_t a_pq = in.pq;
  const uint32_t f_in = f;

  // ---- notify the contacts found on this tracing day, layer by layer
  for (unsigned layers = __ballot_sync(0xffffffffu, in.word != 0u); layers; layers &= layers - 1) {
    const int l = __ffs(layers) - 1;
    const uint32_t word = __shfl_sync(0xffffffffu, in.word, l);
    if (lane == 0) st.contact_bits[(int64_t)l * words + w] = 0u;  // clear for the next tracing day
    if (!valid || !((word >> lane) & 1u)) continue;
    const uint32_t local = (uint32_t)(i - sp.agent_off);
    const uint4 u = philox(make_uint4(local, (uint32_t)l, (uint32_t)t, TAG_TRACE), sp.key0, sp.key1);
    if (!bern52_thr(u.x, u.y, T.thr_trace[l]) || (f & B_DEAD)) continue;
    f |= B_KCONT;
    float* dkc = date_row(st, COVGPU_DATE_KNOWN_CONTACT) + i;
    const float cand = __double2float_rn(__dadd_rn((double)t, T.trace_time[l]));
    if (isnan(*dkc) || cand < *dkc) *dkc = cand;  // np.fmin
    const int start = t + T.trace_start_off[l];
    const int32_t end = start + T.trace_period[l];
    if (start == t) {  // today's slot: check_quar below reads it from a_pq
      if (a_pq < 0 || end > a_pq) a_pq = end;
      continue;
    }
    int32_t* pq = st.pending_quar + (int64_t)(start % R) * st.n + i;
    if (*pq < 0 || end > *pq) *pq = end;  // check_quar keeps the latest end of a day's requests
  }

  if (valid) {
    // ---- check_diagnosed, people.py:315-332
    const float dd = a_dd;
    if (!(f & B_DIAG)) {
      if (defined(a_dpt) && tf >= a_dpt) { date_row(st, COVGPU_DATE_POS_TEST)[i] = nanf_; c_diag = 1; }
      if (defined(dd) && tf >= dd) f |= B_DIAG;
    }
    // ---- check_quar, people.py:335-358
    const int32_t end = a_pq;
    // only the quarantined, or those asked to be, have an end of quarantine to look at
    float* p_deq = date_row(st, COVGPU_DATE_END_QUARANTINE) + i;
    const float a_deq = ((f & B_QUAR) || end >= 0) ? *p_deq : nanf_;
    float deq = a_deq;
    if (end >= 0) {
      if (in.pq >= 0) st.pending_quar[(int64_t)(t % R) * st.n + i] = -1;
      if (f & B_QUAR) {
        if ((float)end > deq) deq = (float)end;  // max(current, end_day), first argument kept on ties/NaN
      } else if (!(f & (B_DEAD | B_REC | B_DIAG | B_ISO))) {
        f |= B_QUAR;
        date_row(st, COVGPU_DATE_QUARANTINED)[i] = tf;
        deq = (float)end;
        c_quar = 1;
      }
    }
    if ((f & B_QUAR) && dd == tf) deq = tf;
    if (__float_as_uint(deq) != __float_as_uint(a_deq)) *p_deq = deq;
    if ((f & B_QUAR) && defined(deq) && tf >= deq) f &= ~B_QUAR;
    // ---- check_enter_iso, people.py:361-366
    if (dd == tf) {
      f |= B_ISO;
      date_row(st, COVGPU_DATE_END_ISOLATION)[i] = date_row(st, COVGPU_DATE_RECOVERED)[i];
      c_iso = 1;
    }
    if (f != f_in) st.flags[i] = f;
    // a source's record carries its flags to the edge pass: keep its quarantine / isolation current
    if (((f ^ f_in) & (B_QUAR | B_ISO)) && ((st.roles[i >> 5] >> (i & 31)) & 1u)) st.src_rec[4 * i + 3] = __uint_as_float(f);
    // and a target's record carries its quarantine in the sign bit
    if (((f ^ f_in) & B_QUAR) && ((st.roles[words + (i >> 5)] >> (i & 31)) & 1u))
      for (int v = 0; v < sp.n_variants; ++v) {
        uint32_t* r = reinterpret_cast<uint32_t*>(st.tgt_rec + (int64_t)v * st.n + i);
        *r = (f & B_QUAR) ? (*r | 0x80000000u) : (*r & 0x7FFFFFFFu);
      }
  }
  acc_diag += c_diag;
  acc_quar += c_quar;
  acc_iso += c_iso;
  // the day's trace count is read only by the tracing passes, which have finished
  if (threadIdx.x == 0 && blk.begin == sp.agent_off) st.trace_count[blk.sim] = 0u;
}

__device__ __forceinline__ void post_flush(const covgpu_state& st, int t, int sim, unsigned& acc_diag,
                                           unsigned& acc_quar, unsigned& acc_iso) {
  const covgpu_sim_params& sp = st.sims[sim];
  const unsigned cd = __reduce_add_sync(0xffffffffu, acc_diag), cq = __reduce_add_sync(0xffffffffu, acc_quar),
                 ci = __reduce_add_sync(0xffffffffu, acc_iso);
  int64_t* res = sp.res_int + (int64_t)t * COVGPU_N_RES_INT;
  if ((threadIdx.x & 31) == 0 && t < sp.npts) {
    if (cd) atomicAdd(reinterpret_cast<unsigned long long*>(res + R_DIAGNOSES), (unsigned long long)cd);
    if (cq) atomicAdd(reinterpret_cast<unsigned long long*>(res + R_QUARANTINED), (unsigned long long)cq);
    if (ci) atomicAdd(reinterpret_cast<unsigned long long*>(res + R_ISOLATED), (unsigned long long)ci);
  }
  acc_diag = acc_quar = acc_iso = 0;
}

__global__ void __launch_bounds__(AGENT_THREADS, PASS_BLOCKS) k_post_pass(covgpu_state st, int t) {
  pdl_wait();
  pdl_trigger();  // one wave, all resident: the next kernel's set-up overlaps this pass
  if (held(st, t)) return;
  int64_t b, b_end;
  if (!agent_range(st, b, b_end)) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t words = (st.n + 31) >> 5;
  int sim = st.agent_blocks[b].sim;
  unsigned acc_diag = 0, acc_quar = 0, acc_iso = 0;
  const int32_t* pending = st.pending_quar + (int64_t)(t % st.pending_slots) * st.n;
  for (; b < b_end; ++b) {
    const covgpu_agent_block blk = st.agent_blocks[b];
    const covgpu_sim_params& sp = st.sims[blk.sim];
    const int64_t i = blk.begin + threadIdx.x, i0 = blk.begin + warp * 32;
    const float nanf_ = __int_as_float(0x7fc00000);
    PostIn in{0u, nanf_, nanf_, -1, 0u};
    if (i < blk.end) {
      in.f = st.flags[i];
      in.dpt = date_row(st, COVGPU_DATE_POS_TEST)[i];
      in.dd = date_row(st, COVGPU_DATE_DIAGNOSED)[i];
      in.pq = pending[i];
    }
    if (lane < sp.n_layers && i0 < blk.end && day_active(t, sp.testing.trace_start, sp.testing.trace_end))
      in.word = st.contact_bits[(int64_t)lane * words + (i0 >> 5)];
    if (blk.sim != sim) {
      post_flush(st, t, sim, acc_diag, acc_quar, acc_iso);
      sim = blk.sim;
    }
    post_block(st, t, blk, in, acc_diag, acc_quar, acc_iso);
  }
  post_flush(st, t, sim, acc_diag, acc_quar, acc_iso);
}

// ------------------------------------------------------------ contact-tracing index
__global__ void k_row_ptr(const int32_t* p, int64_t n_edges, int64_t off, int64_t n_local, uint32_t* rp) {
  const int64_t a = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (a > n_local) return;
  const int64_t key = off + a;  // first edge with p >= key
  int64_t lo = 0, hi = n_edges;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if ((int64_t)p[mid] < key) lo = mid + 1; else hi = mid;
  }
  rp[a] = (uint32_t)lo;
}
__global__ void k_rev_count(const int32_t* p2, int64_t n_edges, int64_t off, int64_t n_local, int64_t* counts) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n_edges) return;
  const int64_t a = (int64_t)p2[e] - off;
  if (a >= 0 && a < n_local) atomicAdd(reinterpret_cast<unsigned long long*>(counts + a), 1ull);
}
__global__ void k_rev_offsets(const int64_t* offsets, int64_t n, uint32_t* rp2) {
  const int64_t a = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (a <= n) rp2[a] = (uint32_t)offsets[a];
}
__global__ void k_rev_place(const int32_t* p2, int64_t n_edges, int64_t off, int64_t n_local, int64_t* cursor,
                            uint32_t* perm2, const int32_t* p1, int32_t* rev1) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n_edges) return;
  const int64_t a = (int64_t)p2[e] - off;
  if (a < 0 || a >= n_local) return;
  const unsigned long long pos = atomicAdd(reinterpret_cast<unsigned long long*>(cursor + a), 1ull);
  perm2[pos] = (uint32_t)e;
  if (rev1) rev1[pos] = p1[e];
}

}  // namespace

namespace covgpu {

int launch_test_trace(const covgpu_state* st, int t, cudaStream_t s) {
  if (!st->has_testing) return COVGPU_OK;
  // bit 4: no sim has anything to prepare (no swab delay, capacity or influenza-like illness)
  if (!(st->has_testing & 16)) k_test_prep<<<(unsigned)st->n_sims, 256, 0, s>>>(*st, t);
  if (st->has_testing & 2) {  // some sim has a swab delay
    static const int64_t hist_wave = wave_blocks(k_swab_hist, AGENT_THREADS);
    k_swab_hist<<<wave_grid(st, hist_wave), AGENT_THREADS, 0, s>>>(*st, t);
  }
  const bool scan = st->n_tiles > 0 && !(st->has_testing & 8);  // some stored layer is traced without an index
  const bool capacity = st->has_testing & 4;
  if (!scan && !capacity) {
    static const int64_t mark_wave = wave_blocks(k_test_pass<true>, AGENT_THREADS);
    launch_pdl(k_test_pass<true>, wave_grid(st, mark_wave), AGENT_THREADS, 0, s, *st, t);
  } else {
    static const int64_t test_wave = wave_blocks(k_test_pass<false>, AGENT_THREADS);
    launch_pdl(k_test_pass<false>, wave_grid(st, test_wave), AGENT_THREADS, 0, s, *st, t);
    if (capacity) k_trace_cap<<<(unsigned)st->n_sims, 256, 0, s>>>(*st, t);
    if (scan) {
      const dim3 grid((unsigned)st->n_tiles);
      switch (st->edge_tile) {
        case 1024: k_trace_scan<1><<<grid, EDGE_THREADS, 0, s>>>(*st, t); break;
        case 2048: k_trace_scan<2><<<grid, EDGE_THREADS, 0, s>>>(*st, t); break;
        case 8192: k_trace_scan<8><<<grid, EDGE_THREADS, 0, s>>>(*st, t); break;
        default: k_trace_scan<4><<<grid, EDGE_THREADS, 0, s>>>(*st, t); break;
      }
    }
    static const int64_t marks_wave = wave_blocks(k_trace_marks, AGENT_THREADS);
    k_trace_marks<<<wave_grid(st, marks_wave), AGENT_THREADS, 0, s>>>(*st, t);
  }
  static const int64_t post_wave = wave_blocks(k_post_pass, AGENT_THREADS);
  launch_pdl(k_post_pass, wave_grid(st, post_wave), AGENT_THREADS, 0, s, *st, t);
  return launch_status();
}

}  // namespace covgpu

extern "C" {

int covgpu_test_trace(const covgpu_state* st, int32_t t, void* stream) {
  int rc = check_state(st);
  if (rc) return rc;
  if (t < 0 || t >= 0xFFFF) return COVGPU_BADARG;
  return launch_test_trace(st, t, S(stream));
}

int64_t covgpu_trace_index_scratch(int64_t n_local) {
  return 2 * (n_local + 1) + (int64_t)scan_blocks_for(n_local, SCAN_TILE) + 1;
}

int covgpu_agent_index(const int32_t* p1, const int32_t* p2, int64_t n_edges, int64_t agent_off, int64_t n_local,
                       uint32_t* rp1, uint32_t* rp2, uint32_t* perm2, int32_t* rev1, int64_t* scratch, void* stream) {
  if (n_edges < 1 || n_edges > 0xFFFFFFFFLL || n_local < 1 || agent_off < 0 || !p1 || !p2 || !rp1 || !rp2 ||
      !perm2 || !scratch)
    return COVGPU_BADARG;
  cudaStream_t s = S(stream);
  int64_t* counts = scratch;
  int64_t* offsets = scratch + (n_local + 1);
  int64_t* tiles = scratch + 2 * (n_local + 1);
  k_row_ptr<<<grid_for(n_local + 1, 256, 1 << 30), 256, 0, s>>>(p1, n_edges, agent_off, n_local, rp1);
  if (cudaMemsetAsync(counts, 0, sizeof(int64_t) * (size_t)n_local, s) != cudaSuccess) return COVGPU_CUDA_ERROR;
  k_rev_count<<<grid_for(n_edges, 256, 1 << 30), 256, 0, s>>>(p2, n_edges, agent_off, n_local, counts);
  int rc = scan_i64(counts, offsets, n_local, tiles, s);
  if (rc) return rc;
  k_rev_offsets<<<grid_for(n_local + 1, 256, 1 << 30), 256, 0, s>>>(offsets, n_local, rp2);
  k_rev_place<<<grid_for(n_edges, 256, 1 << 30), 256, 0, s>>>(p2, n_edges, agent_off, n_local, offsets, perm2, p1, rev1);
  return launch_status();
}

int covgpu_trace_index(const int32_t* p1, const int32_t* p2, int64_t n_edges, int64_t agent_off, int64_t n_local,
                       uint32_t* rp1, uint32_t* rp2, uint32_t* perm2, int64_t* scratch, void* stream) {
  return covgpu_agent_index(p1, p2, n_edges, agent_off, n_local, rp1, rp2, perm2, nullptr, scratch, stream);
}

}  // extern "C"
