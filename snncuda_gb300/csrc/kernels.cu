// Tick kernels of the GB300 engine (sm_103a).
//
// One tick t processes wheel slot t mod W, whose buffer holds the events due
// at t in the exact order the reference scheduler would pop them
// (SpikeScheduler.cpp:25-47: bucket FIFO order).  Per tick, on the main
// stream:
//
//  1. k_bcount     count due events per bucket of consecutive targets, per
//                   chunk of the due list (and copy far-future injections
//                   that become reachable into the wheel)
//  2. k_bscatter   bucket starts; place every event in its bucket
//  3. k_events     a block per bucket: its events grouped by target in due
//                   order in shared memory, then per synapse the event's
//                   pre-spike STDP, pre-spike count and spike-code pattern
//                   (SynapseDendriteProcessor.cpp:104-133, :318-365), per
//                   target the neuron's physics over its events in due order
//                   (:175-229), redoing the STDP of events that follow a fire
//                   of the target, and its temporal pattern (:294-316); fires
//                   into a due-position bitmap
//  4. k_fire_list  fires in due order (= reference fire order), raster
//  5. k_fire_count events per (fire block, delay class); the last block scans
//                  destinations and finishes the tick
//  6. k_expand     copy each fire's pre-expanded (synapse, offset) events into
//                  their delivery slots, order-preserving
//
// and two more, on a second stream (graph fork/join) beside 4-6, or for
// networks of 2^28+ synapses on the main stream after 3 (Engine::side_serial):
//
//  7. k_post       post-spike STDP over the in-rows of targets that fired
//                  (:138-173)
//  8. k_temporal   the neuron temporal pattern of touched targets that keep
//                  several reference patterns (networks that have any)
//
// Main-stream kernels that directly follow another are launched as
// programmatic dependents (tick_enter), so each is scheduled while the one
// before it drains.
//
// Every wait is a kernel boundary (a programmatic dependent's grid
// dependency wait included), a "last block" hand-off (an atomic counter, no
// spinning), the time-bounded mbarrier wait of a staging copy, or, in k_small, the
// hardware barrier of its cluster, whose blocks all reach it or have exited (which
// counts), so no kernel here can hang.
// Float arithmetic uses explicitly rounded intrinsics so nothing is
// contracted into an FMA: each operation rounds exactly as the reference's
// separately evaluated float expressions.

#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "engine.h"

namespace snngb {
namespace {

constexpr int kThreads = 256;
constexpr int kFireCountThreads = 1024;  // k_fire_count's last block scans up to 32 delay classes at once

// Minimum resident blocks per SM requested for k_events (register budget).
#ifndef SNNGB_EVENT_THREADS
#define SNNGB_EVENT_THREADS 128
#endif
#ifndef SNNGB_EVENTS_MIN_BLOCKS
#define SNNGB_EVENTS_MIN_BLOCKS 5
#endif

__device__ __forceinline__ float rec_gain(uint32_t r) { return r == 1 ? 0.55f : (r == 3 ? 0.65f : 1.0f); }
__device__ __forceinline__ float rec_sign(uint32_t r) { return r >= 2 ? -1.0f : 1.0f; }

__device__ __forceinline__ void raise_status(const Engine& e, uint32_t bit) { atomicOr(&e.ts->status, bit); }

// First statement of every main-stream tick kernel.  A kernel launched as a
// programmatic dependent of the previous kernel on its stream is scheduled
// while that kernel still runs and waits here until it has completed and its
// writes are visible (for any other launch the wait returns at once); then it
// lets its own dependent be scheduled.  The wait is the hardware's grid
// dependency, not a spin on memory.
__device__ __forceinline__ void tick_enter() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// ---------------------------------------------------------------------------
// bulk copies into shared memory (TMA, cp.async.bulk) with an mbarrier
// ---------------------------------------------------------------------------

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(unsigned long long* bar, uint32_t arrivals) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(arrivals) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// One thread: expect `bytes` on the barrier and copy them from global memory
// (16-byte aligned, a multiple of 16 bytes) into shared memory.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, unsigned long long* bar) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long v;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(v));
    return v;
}

// Waits for phase `parity` of the barrier to complete, for at most
// `limit_ns` nanoseconds (and at most 2^24 polls); returns false if it did
// not.  A limit of 0 gives up without polling.
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, uint32_t parity, unsigned long long limit_ns) {
    if (limit_ns == 0) return false;
    const uint32_t a = smem_addr(bar);
    const unsigned long long t0 = global_ns();
    for (uint32_t it = 0; it < (1u << 24); ++it) {
        uint32_t done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
        if ((it & 255u) == 255u && global_ns() - t0 > limit_ns) break;
    }
    return false;
}

// Limit of the wait that drains a bulk copy still in flight before its
// shared-memory buffer is reused or the block exits (1 s: a copy of at most
// 64 KB completes in microseconds).
constexpr unsigned long long kDrainWaitNs = 1000000000ull;

// ---------------------------------------------------------------------------
// block-level helpers
// ---------------------------------------------------------------------------

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t n = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= d) v += n;
    }
    return v;
}

// Exclusive block scan of one value per thread (blockDim.x == kThreads).
// Returns the exclusive prefix; *total receives the block sum.
template <int kBlock>
__device__ uint32_t block_excl_scan_t(uint32_t v, uint32_t* total) {
    constexpr int kWarps = kBlock / 32;
    static_assert(kWarps >= 1 && kWarps <= 32, "block size");
    __shared__ uint32_t warp_sums[kWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t incl = warp_incl_scan(v);
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        uint32_t s = lane < kWarps ? warp_sums[lane] : 0;
        s = warp_incl_scan(s);
        if (lane < kWarps) warp_sums[lane] = s;
    }
    __syncthreads();
    const uint32_t base = warp > 0 ? warp_sums[warp - 1] : 0;
    if (total) *total = warp_sums[kWarps - 1];
    __syncthreads();
    return base + incl - v;
}

__device__ uint32_t block_excl_scan(uint32_t v, uint32_t* total) { return block_excl_scan_t<kThreads>(v, total); }

// "Last block" hand-off: returns true in exactly one block, after every
// block's prior global writes are visible.
__device__ bool last_block(uint32_t* counter) {
    __shared__ bool is_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        const uint32_t v = atomicAdd(counter, 1u);
        is_last = (v == gridDim.x - 1);
        if (is_last) *counter = 0;
    }
    __syncthreads();
    if (is_last) __threadfence();
    return is_last;
}

// ---------------------------------------------------------------------------
// per-event physics
// ---------------------------------------------------------------------------

// Approximate u64 -> f32 (relative error < 2^-22) from 32-bit bit operations.
// Conversions with 64-bit operands run on the FP64 pipe, which GB300 keeps
// small; this estimate only feeds the threshold screen below.
__device__ __forceinline__ float u64_to_f32_approx(unsigned long long x) {
    if (x < (1ull << 23)) return __int_as_float(0x4B000000u | static_cast<uint32_t>(x)) - 8388608.0f;
    const int sh = 41 - __clzll(static_cast<long long>(x));  // x >> sh < 2^23
    const uint32_t m = static_cast<uint32_t>(x >> sh);
    const float f = __int_as_float(0x4B000000u | m) - 8388608.0f;
    return f * __int_as_float((127 + sh) << 23);
}

// The reference's exact expression, in double.  Kept out of line: inlined,
// its 64-bit conversions get hoisted above the branch into every call and
// occupy GB300's small FP64 pipe.
__device__ __noinline__ bool cos_ge_exact(unsigned long long dot, unsigned long long rn, unsigned long long cn,
                                          float sim) {
    const double q = __ddiv_rn(__ull2double_rn(dot),
                               __dmul_rn(__dsqrt_rn(__ull2double_rn(rn)), __dsqrt_rn(__ull2double_rn(cn))));
    return __double2float_rn(q) >= sim;
}

// float(dot / (sqrt(rn) * sqrt(cn))) >= sim for sim > 0
// (TemporalPattern.cpp:35-60, :20-22).  dot, rn, cn are the exact integer
// sums the reference accumulates in double.  A single-precision estimate
// (relative error < 1e-6) decides every case farther than 2e-5 from the
// threshold; the rest take the reference's exact double expression.
__device__ __forceinline__ bool cos_ge(unsigned long long dot, unsigned long long rn, unsigned long long cn,
                                       float sim) {
    if (rn == 0 || cn == 0) return false;  // similarity 0.0f < sim
    const float est = __fmul_rn(__fmul_rn(u64_to_f32_approx(dot), rsqrtf(u64_to_f32_approx(rn))),
                                rsqrtf(u64_to_f32_approx(cn)));
    if (est >= sim * 1.00002f) return true;
    if (est <= sim * 0.99998f) return false;
    return cos_ge_exact(dot, rn, cn, sim);
}

// cos_ge for sums that fit 32 bits: rn and cn share one reciprocal square root
// (their product stays below 2^64; the estimate's relative error stays below
// 1e-6).
__device__ __forceinline__ bool cos_ge_u32(uint32_t dot, uint32_t rn, uint32_t cn, float sim) {
    if (rn == 0 || cn == 0) return false;  // similarity 0.0f < sim
    const float est = __fmul_rn(__uint2float_rn(dot), rsqrtf(__fmul_rn(__uint2float_rn(rn), __uint2float_rn(cn))));
    if (est >= sim * 1.00002f) return true;
    if (est <= sim * 0.99998f) return false;
    return cos_ge_exact(dot, rn, cn, sim);
}

// (a + b) mod m for a < m and b <= m, without an integer division.
__device__ __forceinline__ uint32_t wrap_add(uint32_t a, uint32_t b, uint32_t m) {
    const uint32_t x = a + b;
    return x >= m ? x - m : x;
}

struct NState {
    float cur[4];
    uint32_t upd[4];
    uint32_t flags;  // tau codes (2 bits each); in temporal_tick: last_match << 8
    float membrane;
    uint32_t spikes, last_fired1, last_active, match_count, ws, len;
    unsigned long long cn;
    uint32_t nruns, ref_head, ref_count, ring_head, ring_used;
    unsigned long long last_run;  // cand[nruns-1], kept in a register while nruns > 0
    RefMeta one;                  // the learned pattern when max_reference_patterns == 1
    // kOne: the newest pattern's runs are copied into the ring once, at the
    // end of the target's tick (until then nothing reads them)
    bool snap_pending;
    uint32_t snap_nruns;
    unsigned long long snap_last;
};

__device__ __forceinline__ float decay_factor(const Tables& tb, uint32_t code, uint32_t elapsed) {
    const uint32_t i = elapsed < tb.decay_len ? elapsed : tb.decay_len - 1;
    return tb.decay[code * tb.decay_len + i];
}

// SynapseDendriteProcessor.cpp:294-316 (+ :14-41), on the exact run-length
// representation: offsets inside a window never decrease, so the window is
// kept as runs (value, count); learned patterns are run lists in a per-neuron
// ring, each with running integer sums of its cosine against the window.
//
// Applied once per target and tick for all k of its events: every event of
// tick t appends the same offset t - window_start (only the first can restart
// the window), and nothing in the neuron's temporal state feeds the membrane,
// so the reference's per-event sequence of appends is reproduced here in one
// pass.  Once no learned pattern is still being compared element by element
// and a cached result already matches, every remaining append matches too
// (the sums are frozen), which makes the common case O(1) per tick.
//
// Targets that keep one reference pattern, a thread each: the pattern lives in
// s.one.
__device__ void temporal_tick(NState& s, const NeuronParam& p, uint32_t t, const Engine& e, int enabled, uint32_t k) {
    if (k == 0) return;
    if (!enabled) {
        s.flags &= ~(1u << 8);
        return;
    }
    unsigned long long* cand = e.cand + p.cand_base;
    unsigned long long* ring = e.ring + p.ring_base;
    RefMeta& m = s.one;
    if (s.len == 0 || t - s.ws > p.window) {
        s.ws = t;
        s.len = 0;
        s.nruns = 0;
        s.cn = 0;
        m.dot = 0;
        m.rn = 0;
        m.cn = 0;
        m.cur_run = 0;
        m.cur_pos = 0;
        m.match = 2;
    }
    const uint32_t o = t - s.ws;
    const uint32_t oo = o * o;  // o < 2^16, so o * o fits 32 bits
    auto matches = [&]() {
        if (0.0f >= p.similarity) return true;
        if (m.match == 2) m.match = cos_ge(m.dot, m.rn, m.cn, p.similarity) ? 1 : 0;
        return m.match == 1;
    };
    for (uint32_t j = 0; j < k; ++j) {
        if (s.len >= 1 && s.ref_count > 0 && s.nruns > 0 && run_value(s.last_run) == o && s.len >= m.len && matches()) {
            const uint32_t n = k - j;
            s.last_run += static_cast<unsigned long long>(n) << 16;
            s.len += n;
            s.cn += static_cast<unsigned long long>(oo) * n;
            s.match_count += n;
            s.flags |= (1u << 8);
            return;
        }
        // one append (spike_offsets.push_back, :309)
        if (s.nruns > 0 && run_value(s.last_run) == o) {
            s.last_run += (1ull << 16);
        } else {
            if (s.nruns > p.window) {  // cannot happen: at most window+1 distinct offsets
                raise_status(e, kStatusRunOverflow);
                return;
            }
            if (s.nruns > 0) cand[s.nruns - 1] = s.last_run;
            s.last_run = static_cast<unsigned long long>(o) | (1ull << 16);
            s.nruns += 1;
        }
        s.len += 1;
        s.cn += oo;
        if (s.ref_count > 0 && s.len <= m.len) {
            const unsigned long long run = ring[wrap_add(m.start, m.cur_run, p.ring_cap)];
            const uint32_t v = run_value(run);
            if (++m.cur_pos == run_count(run)) {
                m.cur_run += 1;
                m.cur_pos = 0;
            }
            m.dot += v * o;  // 16-bit values: 32-bit products
            m.rn += v * v;
            m.cn += oo;
            m.match = 2;
        }
        if (s.ref_count > 0 && s.len >= 2 && matches()) {
            s.flags |= (1u << 8);
            s.match_count += 1;
            continue;
        }
        s.flags &= ~(1u << 8);
        if (s.len < 2) continue;
        // learn_pattern (:31-41): the window takes the one pattern's place
        if (s.ref_count > 0) {
            s.ring_used -= m.nruns;
            s.ref_count = 0;
        }
        if (s.ring_used + s.nruns > p.ring_cap) {
            raise_status(e, kStatusRingOverflow);
            return;
        }
        s.snap_pending = true;
        s.snap_nruns = s.nruns;
        s.snap_last = s.last_run;
        const uint32_t start = s.ring_head;
        s.ring_head = wrap_add(start, s.nruns, p.ring_cap);
        s.ring_used += s.nruns;
        m.dot = s.cn;
        m.rn = s.cn;
        m.cn = s.cn;
        m.start = start;
        m.nruns = s.nruns;
        m.len = s.len;
        m.cur_run = 0;
        m.cur_pos = 0;
        m.match = 2;
        s.ref_count = 1;
    }
}

// The decay step of SynapseDendriteProcessor.cpp:175-229: every compartment
// is brought forward to tick t.  All events of a target in one tick share t,
// so after the first event every compartment is already at t and the step
// does nothing; it is therefore applied once per target and tick, before the
// first event (a fire's reset also leaves every compartment at t).
__device__ __forceinline__ void decay_to(NState& s, uint32_t t, const Engine& e) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (t <= s.upd[k] || s.cur[k] == 0.0f) {
            s.upd[k] = t;
        } else {
            const uint32_t code = (s.flags >> (2 * k)) & 3u;
            s.cur[k] = __fmul_rn(s.cur[k], decay_factor(e.tab, code, t - s.upd[k]));
            s.upd[k] = t;
        }
    }
}

// The rest of SynapseDendriteProcessor.cpp:175-229 for one event at tick t,
// every compartment already at t (decay_to).  Returns whether the neuron
// fired.
__device__ __forceinline__ bool process_input(NState& s, float threshold, uint32_t comp, uint32_t rec, float w,
                                              uint32_t t) {
    const float applied = __fmul_rn(__fmul_rn(w, rec_gain(rec)), rec_sign(rec));
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (static_cast<uint32_t>(k) == comp) {
            s.cur[k] = __fadd_rn(s.cur[k], applied);  // its update tick is already t
            s.flags = (s.flags & ~(3u << (2 * k))) | (rec << (2 * k));
        }
    }
    s.last_active = t;  // the temporal-pattern update of this event is done by temporal_tick
    s.membrane = __fadd_rn(__fadd_rn(__fadd_rn(s.cur[0], s.cur[1]), s.cur[2]), s.cur[3]);
    if (s.membrane >= threshold) {
        s.membrane = 0.0f;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            s.cur[k] = 0.0f;
            s.upd[k] = t;
        }
        // reset taus: soma AMPA, basal AMPA, apical NMDA, inhibitory GABA_A
        s.flags = (s.flags & ~0xFFu) | (0u << 0) | (0u << 2) | (1u << 4) | (2u << 6);
        s.last_fired1 = t + 1;
        s.spikes += 1;
        return true;
    }
    return false;
}

// StdpRule::weight_delta + apply (STDP.cpp:20-40) and the update bookkeeping
// of SynapseDendriteProcessor.cpp:108-122 / :158-172.  `ltp` is the LTP delta
// table.
__device__ __forceinline__ void stdp_apply(SynA& a, uint32_t pre, uint32_t post, const Engine& e, int stdp, const float* ltp) {
    const float before = a.weight;
    float delta = 0.0f;
    if (stdp && !((a.meta >> kMetaRuleOffBit) & 1u) && post != pre) {
        const float* table = post > pre ? ltp : e.tab.ltd;
        const uint32_t dt = post > pre ? post - pre : pre - post;
        delta = table[dt < e.tab.stdp_len ? dt : e.tab.stdp_len - 1];
    }
    float v = __fadd_rn(a.weight, delta);
    v = v < e.min_weight ? e.min_weight : (a.clamp_hi < v ? a.clamp_hi : v);
    a.weight = v;
    a.last_delta = __fsub_rn(v, before);
    if (a.last_delta != 0.0f) a.updates += 1;
}

// apply_post_spike_plasticity for every target fire at tick t not yet
// applied to this synapse (fires = target fires so far this tick).
__device__ __forceinline__ bool post_catch_up(SynA& a, uint32_t t, uint32_t fires, const Engine& e, int stdp,
                                              const float* ltp) {
    const uint32_t applied = a.last_post1 == t + 1 ? a.post_cnt : 0u;
    if (fires <= applied) return false;
    const bool plastic = (a.meta >> kMetaPlasticBit) & 1u;
    for (uint32_t k = applied; k < fires; ++k) {
        a.last_post1 = t + 1;
        if (plastic && a.last_pre1 != 0) stdp_apply(a, a.last_pre1 - 1, t, e, stdp, ltp);
    }
    a.post_cnt = fires;
    return true;
}

// The parameters of a target that its events and its walk need.
struct TargetParam {
    float threshold;
    uint32_t window;
    float similarity;
    uint32_t max_refs;
};

__device__ __forceinline__ void ring_set(unsigned long long& lo, unsigned long long& hi, uint32_t j,
                                         uint32_t v) {
    if (j < 4) {
        const int sh = 16 * j;
        lo = (lo & ~(0xFFFFull << sh)) | (static_cast<unsigned long long>(v) << sh);
    } else {
        const int sh = 16 * (j - 4);
        hi = (hi & ~(0xFFFFull << sh)) | (static_cast<unsigned long long>(v) << sh);
    }
}

// A learned code pattern of `stride` 16-bit offsets, loaded with the widest
// aligned access the stride allows.
__device__ __forceinline__ void load_pattern(const uint16_t* pat, uint32_t stride, unsigned long long& lo,
                                             unsigned long long& hi) {
    if (stride == 4) {
        lo = *reinterpret_cast<const unsigned long long*>(pat);
        hi = 0;
    } else if (stride == 8) {
        const uint4 v = *reinterpret_cast<const uint4*>(pat);
        lo = (static_cast<unsigned long long>(v.y) << 32) | v.x;
        hi = (static_cast<unsigned long long>(v.w) << 32) | v.z;
    } else if (stride == 2) {
        lo = *reinterpret_cast<const uint32_t*>(pat);
        hi = 0;
    } else {
        lo = hi = 0;
        for (uint32_t j = 0; j < stride; ++j) ring_set(lo, hi, j, pat[j]);
    }
}

__device__ __forceinline__ void store_pattern(uint16_t* pat, uint32_t stride, unsigned long long lo,
                                              unsigned long long hi) {
    if (stride == 4) {
        *reinterpret_cast<unsigned long long*>(pat) = lo;
    } else if (stride == 8) {
        *reinterpret_cast<uint4*>(pat) = make_uint4(static_cast<uint32_t>(lo), static_cast<uint32_t>(lo >> 32),
                                                    static_cast<uint32_t>(hi), static_cast<uint32_t>(hi >> 32));
    } else if (stride == 2) {
        *reinterpret_cast<uint32_t*>(pat) = static_cast<uint32_t>(lo);
    } else {
        for (uint32_t j = 0; j < stride; ++j) pat[j] = static_cast<uint16_t>(ring_get(lo, hi, j));
    }
}

// SynapseDendriteProcessor.cpp:318-365 on a fixed ring of `expected` offsets
// held in two 64-bit words.  `inline_pattern`: the target keeps one reference
// pattern and codes have at most 4 offsets, so the single learned code
// pattern is stored in ring_hi instead of the pattern pool.
// Four 16-bit offsets in two words.
struct Lanes {
    uint32_t a, b;
};

// Sum of the products of four 16-bit lanes.  kWide: offsets up to 65,535 (a
// 64-bit sum); otherwise below 2^15, where four products fit 32 bits.
template <bool kWide>
__device__ __forceinline__ auto lanes_dot(Lanes x, Lanes y) {
    using Sum = std::conditional_t<kWide, unsigned long long, uint32_t>;
    return static_cast<Sum>((x.a & 0xFFFFu) * (y.a & 0xFFFFu)) + static_cast<Sum>((x.a >> 16) * (y.a >> 16)) +
           static_cast<Sum>((x.b & 0xFFFFu) * (y.b & 0xFFFFu)) + static_cast<Sum>((x.b >> 16) * (y.b >> 16));
}

// SynapseDendriteProcessor.cpp:318-365 for inline_code_pattern (one reference
// pattern, at most 4 offsets): the window is the four 16-bit lanes of ring_lo,
// the learned pattern those of ring_hi; lanes at or above `expected` are
// always zero, so the sums run over all four lanes.
__device__ __forceinline__ void code_update_inline(SynB& b, uint32_t window, float sim, uint32_t t) {
    uint32_t flags = b.flags & 0xF0u;  // last_code_match = false
    uint32_t len = b.code_len;
    const uint32_t expected = flags >> 4;
    if (len == 0 || t - b.code_ws > window) {
        b.code_ws = t;
        len = 0;
    }
    const uint32_t o = t - b.code_ws;  // at most `window`
    Lanes x{static_cast<uint32_t>(b.ring_lo), static_cast<uint32_t>(b.ring_lo >> 32)};
    uint32_t at = len;  // the new offset's lane
    if (len < expected) {
        ++len;
    } else {
        x.a = __byte_perm(x.a, x.b, 0x5432);
        x.b >>= 16;
        at = expected - 1;
    }
    const uint32_t put = (at & 1u) ? 0x5410u : 0x3254u;  // o into the upper or the lower half
    x.a = at < 2 ? __byte_perm(x.a, o, put) : x.a;
    x.b = at < 2 ? x.b : __byte_perm(x.b, o, put);
    b.ring_lo = (static_cast<unsigned long long>(x.b) << 32) | x.a;
    b.code_len = static_cast<uint8_t>(len);
    if (len >= expected) {
        bool match = 0.0f >= sim;
        if (!match && b.learned_count > 0) {
            const Lanes y{static_cast<uint32_t>(b.ring_hi), static_cast<uint32_t>(b.ring_hi >> 32)};
            if (window < (1u << 15)) {
                match = cos_ge_u32(lanes_dot<false>(y, x), lanes_dot<false>(y, y), lanes_dot<false>(x, x), sim);
            } else {
                match = cos_ge(lanes_dot<true>(y, x), lanes_dot<true>(y, y), lanes_dot<true>(x, x), sim);
            }
        }
        if (match) {
            b.code_matches += 1;
            flags |= 1u;
        } else {
            b.ring_hi = b.ring_lo;
            b.learned_count = 1;
        }
    }
    b.flags = static_cast<uint8_t>(flags);
}

// code_update for the pattern pool (`lc`: the synapse's learned patterns, up
// to p.max_refs of `stride` offsets each).
__device__ void code_update_pool(SynB& b, const TargetParam& p, uint32_t t, uint16_t* lc, uint32_t stride) {
    b.flags &= 0xF0u;  // last_code_match = false
    if (b.code_len == 0 || t - b.code_ws > p.window) {
        b.code_ws = t;
        b.code_len = 0;
    }
    const uint32_t o = t - b.code_ws;
    const uint32_t expected = b.flags >> 4;
    if (b.code_len < expected) {
        ring_set(b.ring_lo, b.ring_hi, b.code_len, o);
        b.code_len += 1;
    } else {
        b.ring_lo = (b.ring_lo >> 16) | (b.ring_hi << 48);
        b.ring_hi >>= 16;
        ring_set(b.ring_lo, b.ring_hi, expected - 1, o);
    }
    if (b.code_len < expected) return;
    bool match = 0.0f >= p.similarity;
    unsigned long long cn = 0;
    for (uint32_t j = 0; j < expected; ++j) {
        const uint32_t v = ring_get(b.ring_lo, b.ring_hi, j);
        cn += v * v;  // 16-bit offsets: 32-bit products, 64-bit sums
    }
    for (uint32_t i = 0; i < b.learned_count && !match; ++i) {
        unsigned long long plo, phi;
        load_pattern(lc + static_cast<size_t>(i) * stride, stride, plo, phi);
        unsigned long long dot = 0, rn = 0;
        for (uint32_t j = 0; j < expected; ++j) {
            const uint32_t pv = ring_get(plo, phi, j);
            dot += pv * ring_get(b.ring_lo, b.ring_hi, j);
            rn += pv * pv;
        }
        match = cos_ge(dot, rn, cn, p.similarity);
    }
    if (match) {
        b.code_matches += 1;
        b.flags |= 1u;
        return;
    }
    if (b.learned_count >= p.max_refs) {
        for (uint32_t i = 1; i < b.learned_count; ++i)
            for (uint32_t j = 0; j < stride; ++j)
                lc[static_cast<size_t>(i - 1) * stride + j] = lc[static_cast<size_t>(i) * stride + j];
        b.learned_count -= 1;
    }
    store_pattern(lc + static_cast<size_t>(b.learned_count) * stride, stride, b.ring_lo, b.ring_hi);
    b.learned_count += 1;
}

template <bool kInline>
__device__ __forceinline__ void code_update(SynB& b, const TargetParam& p, uint32_t t, uint16_t* lc, uint32_t stride,
                                            int enabled, bool inline_pattern) {
    if (!enabled) {
        b.flags &= 0xF0u;  // last_code_match = false
    } else if (kInline || inline_pattern) {
        code_update_inline(b, p.window, p.similarity, t);
    } else {
        code_update_pool(b, p, t, lc, stride);
    }
}

// ---------------------------------------------------------------------------
// kernels
// ---------------------------------------------------------------------------

// ---------------------------------------------------------------------------
// grouping: the tick's due list regrouped by target (ascending), each
// target's events in due order, in three or four kernels:
//   k_bcount    a block per contiguous chunk of the due list: events per
//               bucket of 2^bucket_shift consecutive targets, counted in
//               shared memory; the block's row of counts goes to bcnt and is
//               added into the bucket totals (one atomic per nonzero bucket)
//   k_bscatter  a block per chunk: the bucket starts (every block scans the
//               totals itself), one reservation per (chunk, bucket), then
//               every event goes to its bucket's range of grp_tmp (order
//               inside a bucket arbitrary)
//   k_group     a block per bucket: the bucket's events by target in due order,
//               and the segment starts (the grouping entry points only: the
//               tick's k_events sorts its buckets itself); of buckets too
//               large for its shared memory, k_group_rest sorts the segments
// Per event that is two or more reads of the due list (k_bscatter places a
// long list in passes over disjoint bucket ranges, so the lines it fills stay
// in L2 until complete), one scattered write, and a coalesced read and write
// per bucket: no per-target global atomics.
// ---------------------------------------------------------------------------

// Threads of a k_events block, and the events it holds in shared memory.
constexpr int kEventThreads = SNNGB_EVENT_THREADS;
constexpr uint32_t kBlockPerThread = 10;
constexpr uint32_t kBlockEvents = kBlockPerThread * kEventThreads;
constexpr uint32_t kPartShift = 15;  // Engine::parts: bucket | part << kPartShift
static_assert(kMaxTickBuckets <= 1u << kPartShift && kMaxBucketShift + kPartShift <= 32, "Engine::parts");

// Block-wide exclusive scan of a[0 .. n) in shared memory, in place; returns
// the total.  Every thread takes a run of consecutive entries.
template <int kBlock>
__device__ uint32_t block_scan_shared(uint32_t* a, uint32_t n) {
    const uint32_t per = (n + kBlock - 1) / kBlock;
    const uint32_t b = threadIdx.x * per;
    const uint32_t en = b + per < n ? b + per : n;
    uint32_t sum = 0;
    for (uint32_t i = b; i < en; ++i) sum += a[i];
    uint32_t total;
    uint32_t run = block_excl_scan_t<kBlock>(sum, &total);
    for (uint32_t i = b; i < en; ++i) {
        const uint32_t v = a[i];
        a[i] = run;
        run += v;
    }
    __syncthreads();
    return total;
}

// The far-future injections whose delivery tick t + W - 1 becomes
// addressable at tick t: far_ev[b, en), for wheel slot `slot`.
__device__ __forceinline__ bool far_range(const Engine& e, uint32_t t, uint32_t& b, uint32_t& en, uint32_t& slot) {
    const uint32_t ft = e.ts->far_ticks;
    if (ft == 0) return false;
    const long long rel = static_cast<long long>(t) + e.W - 1 - e.ts->far_first_tick;
    if (rel < 0 || rel >= ft) return false;
    b = e.far_idx[rel];
    en = e.far_idx[rel + 1];
    slot = (t + e.W - 1) & e.wmask;
    return en > b;
}

// Copies them behind the slot's current events, spread over the whole grid
// (k_bcount; the slot is not the one being grouped, and its count changes
// only in k_bscatter, after every block has copied its share).
__device__ void copy_far_injections(const Engine& e, uint32_t t) {
    uint32_t b, en, slot;
    if (!far_range(e, t, b, en, slot)) return;
    const uint32_t base = e.slot_count[slot];
    if (static_cast<unsigned long long>(base) + (en - b) > e.slot_cap) return;  // k_bscatter raises it
    unsigned long long* dst = e.wheel + static_cast<size_t>(slot) * e.slot_cap + base;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < en - b; i += gridDim.x * blockDim.x)
        dst[i] = e.far_ev[b + i];
}

// Their slot's new count (one thread of k_bscatter).
__device__ void count_far_injections(const Engine& e, uint32_t t) {
    uint32_t b, en, slot;
    if (!far_range(e, t, b, en, slot)) return;
    const uint32_t base = e.slot_count[slot];
    if (static_cast<unsigned long long>(base) + (en - b) > e.slot_cap) {
        raise_status(e, kStatusSlotOverflow);
        return;
    }
    e.slot_count[slot] = base + (en - b);
}

// This block's chunk [beg, end) of a due list of n events.
__device__ __forceinline__ void chunk_of(uint32_t n, uint32_t& beg, uint32_t& end) {
    const uint32_t chunk = (n + gridDim.x - 1) / gridDim.x;
    const unsigned long long b = static_cast<unsigned long long>(blockIdx.x) * chunk;
    beg = b < n ? static_cast<uint32_t>(b) : n;
    end = n - beg < chunk ? n : beg + chunk;
}

// Threads of the counting and placing blocks, and the due-list entries each
// thread has in flight per round (independent loads: the kernels stream the
// due list and would otherwise wait a DRAM latency per entry).
constexpr int kBucketThreads = 1024;

// The counting and placing blocks stream their chunk of the due list through
// shared memory: tiles of kStreamTile entries (32 KB) by bulk copy (TMA),
// kStreamBufs copies in flight per block, each waited for at most
// Engine::stage_wait_ns.
constexpr uint32_t kStreamTile = 4096;
constexpr uint32_t kStreamBufs = 2;

struct DueStream {
    unsigned long long* buf;  // kStreamBufs x kStreamTile entries (shared memory)
    unsigned long long* bar;  // kStreamBufs mbarriers (shared memory)
    uint32_t parity;          // bit b: phase buffer b's barrier completes next
    bool staging;             // false after a copy outlived its wait: no more copies
};

// Shared memory of k_bcount / k_bscatter: the bucket counters, then the
// stream's two tiles (16-byte aligned).
__host__ __device__ inline size_t stream_buf_offset(uint32_t nbuckets) {
    return (static_cast<size_t>(nbuckets) * sizeof(uint32_t) + 15) & ~static_cast<size_t>(15);
}

// Calls f(i, src[i]) once for every i in [beg, end), spread over the block's
// threads (every thread of the block must call it: it has block barriers;
// the order of the calls is unspecified).  The 16-byte aligned even-length
// body comes in by bulk copies; an unaligned first entry and an odd last
// entry are read directly.  If a copy outlives
// its wait, the block raises kStatusStageTimeout, drains the copies in
// flight (bounded), and reads the rest from global memory, now and in later
// calls.  Returns false only if a drain also failed (the block must exit).
template <typename F>
__device__ bool stream_due(const Engine& e, const unsigned long long* src, uint32_t beg, uint32_t end, DueStream& s,
                           F&& f) {
    uint32_t a0 = beg;
    if (a0 < end && (reinterpret_cast<uintptr_t>(src + a0) & 15u) != 0) ++a0;
    const uint32_t a1 = a0 + ((end - a0) & ~1u);
    if (threadIdx.x == 0 && beg < a0) f(beg, src[beg]);
    if (threadIdx.x == blockDim.x - 1 && a1 < end) f(a1, src[a1]);
    // Read directly (four loads in flight per thread): a chunk shorter than
    // two tiles, where waiting for a whole tile costs more than it hides, an
    // array that is not even 8-byte aligned, and after a failed copy.
    if (!s.staging || a1 - a0 < 2 * kStreamTile || (reinterpret_cast<uintptr_t>(src + a0) & 15u) != 0) {
        for (uint32_t i0 = a0 + threadIdx.x; i0 < a1; i0 += 4 * blockDim.x) {
            unsigned long long v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t i = i0 + u * blockDim.x;
                v[u] = i < a1 ? __ldcs(src + i) : 0ull;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (i0 + u * blockDim.x < a1) f(i0 + u * blockDim.x, v[u]);
        }
        return true;
    }
    const uint32_t ntiles = (a1 - a0 + kStreamTile - 1) / kStreamTile;
    auto tile_len = [&](uint32_t k) {
        const uint32_t st = a0 + k * kStreamTile;
        return a1 - st < kStreamTile ? a1 - st : kStreamTile;
    };
    auto issue = [&](uint32_t k) {
        const uint32_t b = k % kStreamBufs;
        bulk_load(s.buf + b * kStreamTile, src + a0 + k * kStreamTile,
                  tile_len(k) * static_cast<uint32_t>(sizeof(unsigned long long)), &s.bar[b]);
    };
    if (threadIdx.x == 0)
        for (uint32_t k = 0; k < kStreamBufs && k < ntiles; ++k) issue(k);
    for (uint32_t k = 0; k < ntiles; ++k) {
        const uint32_t b = k % kStreamBufs;
        const uint32_t st = a0 + k * kStreamTile;
        const uint32_t cnt = tile_len(k);
        // one thread polls the barrier; the block barrier then orders its
        // observation of the completed copy before every thread's reads
        bool ready = true;
        if (threadIdx.x == 0) ready = mbar_wait(&s.bar[b], (s.parity >> b) & 1u, e.stage_wait_ns);
        if (!__syncthreads_and(ready)) {
            // tiles k .. k + kStreamBufs - 1 (those that exist) are still in
            // flight: drain them before the block goes on without shared memory
            bool drained = true;
            if (threadIdx.x == 0) raise_status(e, kStatusStageTimeout);
            for (uint32_t j = 0; j < kStreamBufs && k + j < ntiles; ++j) {
                const uint32_t bj = (k + j) % kStreamBufs;
                if (threadIdx.x == 0) drained = mbar_wait(&s.bar[bj], (s.parity >> bj) & 1u, kDrainWaitNs) && drained;
                s.parity ^= 1u << bj;
            }
            if (!__syncthreads_and(drained)) return false;
            s.staging = false;
            for (uint32_t i = st + threadIdx.x; i < a1; i += blockDim.x) f(i, __ldcs(src + i));
            return true;
        }
        const unsigned long long* tile = s.buf + b * kStreamTile;
        for (uint32_t i = threadIdx.x; i < cnt; i += blockDim.x) f(st + i, tile[i]);
        s.parity ^= 1u << b;
        __syncthreads();  // the buffer is read: it may take tile k + kStreamBufs
        if (threadIdx.x == 0 && k + kStreamBufs < ntiles) issue(k + kStreamBufs);
    }
    return true;
}

__global__ void __launch_bounds__(kBucketThreads) k_bcount(Engine e) {
    tick_enter();
    extern __shared__ __align__(16) uint32_t s_hist[];  // [nbuckets], then the stream's tiles
    __shared__ unsigned long long s_bar[kStreamBufs];
    const uint32_t t = e.ts->tick;
    copy_far_injections(e, t);
    const uint32_t B = e.nbuckets;
    for (uint32_t b = threadIdx.x; b < B; b += blockDim.x) s_hist[b] = 0;
    if (threadIdx.x == 0)
        for (uint32_t j = 0; j < kStreamBufs; ++j) mbar_init(&s_bar[j], 1);
    __syncthreads();
    const uint32_t slot = t & e.wmask;
    const uint32_t n = e.slot_count[slot];
    const unsigned long long* ev = e.wheel + static_cast<size_t>(slot) * e.slot_cap;
    uint32_t beg, end;
    chunk_of(n, beg, end);
    DueStream ds{reinterpret_cast<unsigned long long*>(reinterpret_cast<unsigned char*>(s_hist) + stream_buf_offset(B)),
                 s_bar, 0u, true};
    uint32_t ext = 0;
    const bool ok = stream_due(e, ev, beg, end, ds, [&](uint32_t, unsigned long long v) {
        const uint32_t lo = static_cast<uint32_t>(v);
        const uint32_t tgt = lo & ~kExternalBit;
        if (tgt >= e.N) {  // only reachable through snncuda_group_events with bad input
            raise_status(e, kStatusBadEvent);
            return;
        }
        atomicAdd(&s_hist[tgt >> e.bucket_shift], 1u);
        ext += lo >> 31;
    });
    // (if a drain failed the counts are partial and the tick is already
    // flagged; the row is still written, and the kernels after it keep every
    // access in bounds whatever the counts)
    (void)ok;
    ext = __reduce_add_sync(0xffffffffu, ext);
    if ((threadIdx.x & 31) == 0 && ext) atomicAdd(&e.ts->external, static_cast<unsigned long long>(ext));
    __syncthreads();
    uint32_t* row = e.bcnt + static_cast<size_t>(blockIdx.x) * B;
    for (uint32_t b = threadIdx.x; b < B; b += blockDim.x) {
        const uint32_t c = s_hist[b];
        row[b] = c;
        if (c) atomicAdd(&e.btot[b], c);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        e.ts->n_due = n;
        e.ts->post_tick = t;        // the previous tick's k_post has finished
        e.ts->n_fired_targets = 0;
        e.ts->n_parts = 0;
    }
}

// Lists the parts of the buckets that are too large for a block of k_events
// (`large`: events in those of this thread's buckets [b0, b1)); one block.
__device__ __noinline__ void list_parts(const Engine& e, uint32_t b0, uint32_t b1, uint32_t large) {
    uint32_t total;
    block_excl_scan_t<kBucketThreads>(large, &total);
    const uint32_t part_events = min(max(total / kPartBlocks, kPartEventsMin), kPartEvents);
    if (threadIdx.x == 0) e.ts->part_events = part_events;
    if (large == 0) return;
    for (uint32_t b = b0; b < b1; ++b) {
        const uint32_t c = __ldcg(e.btot + b);
        if (c <= kBlockEvents) continue;
        const uint32_t parts = 1u << part_shift(c, part_events, e.bucket_shift);
        const uint32_t at = atomicAdd(&e.ts->n_parts, parts);
        for (uint32_t k = 0; k < parts; ++k) e.parts[at + k] = b | (k << kPartShift);
    }
}

__global__ void __launch_bounds__(kBucketThreads) k_bscatter(Engine e) {
    tick_enter();
    extern __shared__ __align__(16) uint32_t s_pos[];  // [nbuckets] next position of this chunk in each bucket
    __shared__ unsigned long long s_bar[kStreamBufs];
    const uint32_t B = e.nbuckets;
    {
        // bucket starts: every block scans the bucket totals itself (a run of
        // consecutive buckets per thread); block 0 publishes them
        const uint32_t per = (B + blockDim.x - 1) / blockDim.x;
        const uint32_t b0 = threadIdx.x * per < B ? threadIdx.x * per : B;
        const uint32_t b1 = b0 + per < B ? b0 + per : B;
        uint32_t sum = 0, large = 0;
        for (uint32_t b = b0; b < b1; ++b) {
            const uint32_t c = __ldcg(e.btot + b);
            s_pos[b] = c;
            sum += c;
            if (c > kBlockEvents) large += c;
        }
        uint32_t total;
        uint32_t run = block_excl_scan_t<kBucketThreads>(sum, &total);
        for (uint32_t b = b0; b < b1; ++b) {
            const uint32_t c = s_pos[b];
            s_pos[b] = run;
            if (blockIdx.x == 0) e.bstart[b] = run;
            run += c;
        }
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            e.bstart[B] = total;
            e.seg_start[e.N] = total;
            count_far_injections(e, e.ts->tick);
        }
        const bool list = blockIdx.x == gridDim.x - 1 && e.parts != nullptr;
        if (__syncthreads_or(list && large > 0)) list_parts(e, b0, b1, large);
    }
    // this chunk's place in each bucket: behind the chunks that reserved
    // before it (the cursors start at zero every tick; k_events clears them)
    const uint32_t* row = e.bcnt + static_cast<size_t>(blockIdx.x) * B;
    for (uint32_t b = threadIdx.x; b < B; b += blockDim.x) {
        const uint32_t c = row[b];
        if (c) s_pos[b] += atomicAdd(&e.bcur[b], c);
    }
    if (threadIdx.x == 0)
        for (uint32_t j = 0; j < kStreamBufs; ++j) mbar_init(&s_bar[j], 1);
    __syncthreads();
    DueStream ds{reinterpret_cast<unsigned long long*>(reinterpret_cast<unsigned char*>(s_pos) + stream_buf_offset(B)),
                 s_bar, 0u, true};
    const uint32_t slot = e.ts->tick & e.wmask;
    const uint32_t n = e.ts->n_due;
    const unsigned long long* ev = e.wheel + static_cast<size_t>(slot) * e.slot_cap;
    const uint32_t lmask = (1u << e.bucket_shift) - 1u;
    uint32_t beg, end;
    chunk_of(n, beg, end);
    // passes over disjoint bucket ranges (Engine::scatter_pass_events): the
    // due list is streamed again per pass
    const uint32_t per = e.scatter_pass_events;
    const uint32_t passes = per != 0 && n > per ? (n + per - 1) / per : 1u;
    for (uint32_t pass = 0; pass < passes; ++pass) {
        const uint32_t blo = static_cast<uint32_t>(static_cast<unsigned long long>(B) * pass / passes);
        const uint32_t bhi = static_cast<uint32_t>(static_cast<unsigned long long>(B) * (pass + 1) / passes);
        const bool ok = stream_due(e, ev, beg, end, ds, [&](uint32_t i, unsigned long long v) {
            const uint32_t lo = static_cast<uint32_t>(v);
            const uint32_t tgt = lo & ~kExternalBit;
            if (tgt >= e.N) return;
            const uint32_t b = tgt >> e.bucket_shift;
            if (b < blo || b >= bhi) return;
            const uint32_t pos = atomicAdd(&s_pos[b], 1u);
            if (pos >= e.slot_cap) return;  // only after a failed stream (counts partial)
            reinterpret_cast<uint4*>(e.grp_tmp)[pos] =
                make_uint4(i | (lo & kExternalBit), static_cast<uint32_t>(v >> 32), tgt & lmask, 0u);
        });
        if (!ok) return;
    }
}

// Sort key of a grouped entry: its due index (unique within one due list).
__device__ __forceinline__ uint32_t grp_key(unsigned long long v) { return static_cast<uint32_t>(v) & ~kExternalBit; }

// Ascending bitonic sort of one entry per lane by key (lanes without an
// entry carry key 0xFFFFFFFF and sort last).
__device__ __forceinline__ void warp_bitonic(unsigned long long& v, uint32_t& key) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int size = 2; size <= 32; size <<= 1) {
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            const uint32_t ok = __shfl_xor_sync(0xffffffffu, key, stride);
            const unsigned long long ov = __shfl_xor_sync(0xffffffffu, v, stride);
            const bool up = ((lane & size) == 0);
            const bool lower = (lane & stride) == 0;
            const bool take_min = (lower == up);
            if (take_min ? (ok < key) : (ok > key)) {
                key = ok;
                v = ov;
            }
        }
    }
}

// One warp sorts entries [0, len) of `a` by key into `b` (a is scratch and
// is overwritten).  Runs of 32 are sorted in registers, then runs are merged
// pairwise, doubling their width: an entry's place in the merged run is its
// index in its own run plus the number of keys below it in the other run
// (a binary search; keys are unique).  O(len log^2 len) work per warp, so a
// segment of 2^20 entries takes milliseconds, not the len^2 of a rank count.
__device__ void warp_merge_sort(unsigned long long* a, unsigned long long* b, uint32_t len) {
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t c = 0; c < len; c += 32) {
        const uint32_t n = len - c < 32 ? len - c : 32;
        unsigned long long v = lane < n ? a[c + lane] : ~0ull;
        uint32_t key = lane < n ? grp_key(v) : 0xFFFFFFFFu;
        warp_bitonic(v, key);
        if (lane < n) a[c + lane] = v;
    }
    __syncwarp();
    unsigned long long* src = a;
    unsigned long long* dst = b;
    for (uint32_t w = 32; w < len; w <<= 1) {
        for (uint32_t base = 0; base < len; base += 2 * w) {
            const uint32_t la = len - base < w ? len - base : w;
            const uint32_t lb = len - base - la < w ? len - base - la : w;
            const unsigned long long* L = src + base;
            const unsigned long long* R = L + la;
            for (uint32_t j = lane; j < la + lb; j += 32) {
                const bool left = j < la;
                const unsigned long long v = left ? L[j] : R[j - la];
                const uint32_t key = grp_key(v);
                const unsigned long long* other = left ? R : L;
                uint32_t lo = 0, hi = left ? lb : la;  // keys of `other` below key
                while (lo < hi) {
                    const uint32_t mid = (lo + hi) >> 1;
                    if (grp_key(other[mid]) < key) {
                        lo = mid + 1;
                    } else {
                        hi = mid;
                    }
                }
                dst[base + (left ? j : j - la) + lo] = v;
            }
        }
        __syncwarp();
        unsigned long long* t = src;
        src = dst;
        dst = t;
    }
    if (src != b) {
        for (uint32_t j = lane; j < len; j += 32) b[j] = src[j];
        __syncwarp();
    }
}



// The lanes of a whole warp with the same 8-bit digit as this one (`in`: the
// lane has one); eight ballots, where a match instruction over mostly
// different digits kept the SM's match unit busy five times as long.
__device__ __forceinline__ uint32_t same_digit(uint32_t digit, bool in) {
    const uint32_t active = __ballot_sync(0xffffffffu, in);
    uint32_t same = active;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const bool one = (digit >> b) & 1u;
        const uint32_t ones = __ballot_sync(0xffffffffu, one);
        same &= one ? ones : ~ones;
    }
    return same;
}

// Whole block: a[0 .. len) by key (below 2^bits), with b[0 .. len) as scratch;
// the result is in a.  Stable radix sort by 8-bit digits: every warp counts
// and then places a contiguous share of the entries, 32 at a time in order, in
// its own row of counters (s_cnt: kBlock / 32 rows of 256, and 256 totals), so
// an entry's place is the digit's start, the earlier warps' entries, this
// warp's earlier ones, and its rank among the 32.  Work linear in len.
template <int kBlock>
__device__ void block_radix_sort(unsigned long long* a, unsigned long long* b, uint32_t len, uint32_t bits,
                                 uint32_t* s_cnt) {
    constexpr uint32_t kWarps = kBlock / 32, kInFlight = 4;  // loads per lane before the first is used
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t* mine = s_cnt + 256 * warp;
    uint32_t* s_tot = s_cnt + 256 * kWarps;
    constexpr uint32_t kStep = 32 * kInFlight;  // a warp's shares are whole steps: none of them mostly empty
    const uint32_t share = (len + kWarps * kStep - 1) / (kWarps * kStep) * kStep;
    const uint32_t i0 = min(len, warp * share), i1 = min(len, i0 + share);
    unsigned long long *src = a, *dst = b;
    for (uint32_t shift = 0; shift < bits; shift += 8) {
        for (uint32_t i = threadIdx.x; i < 256 * kWarps; i += kBlock) s_cnt[i] = 0;
        __syncthreads();
        for (uint32_t c = i0; c < i1; c += kStep) {
            unsigned long long v[kInFlight];
#pragma unroll
            for (uint32_t u = 0; u < kInFlight; ++u) {
                const uint32_t i = c + 32 * u + lane;
                v[u] = i < i1 ? src[i] : 0ull;
            }
#pragma unroll
            for (uint32_t u = 0; u < kInFlight; ++u) {
                const bool in = c + 32 * u + lane < i1;
                const uint32_t digit = (grp_key(v[u]) >> shift) & 255u;
                const uint32_t same = same_digit(digit, in);
                if (in && lane == __ffs(same) - 1) mine[digit] += __popc(same);
                __syncwarp();
            }
        }
        __syncthreads();
        for (uint32_t d = threadIdx.x; d < 256; d += kBlock) {
            uint32_t run = 0;
            for (uint32_t w = 0; w < kWarps; ++w) {
                const uint32_t c = s_cnt[256 * w + d];
                s_cnt[256 * w + d] = run;
                run += c;
            }
            s_tot[d] = run;
        }
        __syncthreads();
        block_scan_shared<kBlock>(s_tot, 256);
        for (uint32_t c = i0; c < i1; c += kStep) {
            unsigned long long v[kInFlight];
#pragma unroll
            for (uint32_t u = 0; u < kInFlight; ++u) {
                const uint32_t i = c + 32 * u + lane;
                v[u] = i < i1 ? src[i] : 0ull;
            }
#pragma unroll
            for (uint32_t u = 0; u < kInFlight; ++u) {
                const bool in = c + 32 * u + lane < i1;
                const uint32_t digit = (grp_key(v[u]) >> shift) & 255u;
                const uint32_t same = same_digit(digit, in);
                const uint32_t at = in ? mine[digit] : 0u;
                __syncwarp();
                if (in) dst[s_tot[digit] + at + __popc(same & ((1u << lane) - 1u))] = v[u];
                if (in && lane == __ffs(same) - 1) mine[digit] = at + __popc(same);
                __syncwarp();
            }
        }
        __syncthreads();
        unsigned long long* t = src;
        src = dst;
        dst = t;
    }
    if (src != a) {
        for (uint32_t i = threadIdx.x; i < len; i += kBlock) a[i] = src[i];
        __syncthreads();
    }
}

// Bits of the due indices 0 .. n-1.
__device__ __forceinline__ uint32_t due_bits(uint32_t n) { return n > 1 ? 32 - __clz(n - 1) : 1; }

// Adds one to counter[j] for each lane's j (of a whole warp; j == none: no
// count) and returns the count before the lane's own.  The lanes that agree
// with lane 0 share one atomic: a bucket that is large because of one busy
// target then costs a warp's entries about one atomic, not 32 on one counter.
__device__ __forceinline__ uint32_t warp_count(uint32_t* counter, uint32_t j, uint32_t none) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t j0 = __shfl_sync(0xffffffffu, j, 0);
    const uint32_t same = __ballot_sync(0xffffffffu, j == j0);
    uint32_t first = 0;
    if (j != none && (lane == 0 || j != j0)) first = atomicAdd(&counter[j], lane == 0 ? __popc(same) : 1u);
    const uint32_t shared = __shfl_sync(0xffffffffu, first, 0);
    return j == j0 ? shared + __popc(same & ((1u << lane) - 1u)) : first;
}

// One warp puts a target's group of `len` events in due order (up to 32
// bitonic-sorted in registers, longer groups merge-sorted with tmp[0 .. len)
// as scratch).
__device__ __forceinline__ void sort_group(unsigned long long* g, unsigned long long* tmp, uint32_t len) {
    const uint32_t lane = threadIdx.x & 31;
    if (len <= 1) return;
    if (len <= 32) {
        unsigned long long v = lane < len ? g[lane] : ~0ull;
        uint32_t key = lane < len ? grp_key(v) : 0xFFFFFFFFu;
        warp_bitonic(v, key);
        if (lane < len) g[lane] = v;
    } else {
        warp_merge_sort(g, tmp, len);  // sorted into tmp
        for (uint32_t k = lane; k < len; k += 32) g[k] = tmp[k];
        __syncwarp();
    }
}

// The most events of one target that a block ranks in shared memory (every
// pair of them is compared).
constexpr uint32_t kRankEvents = 512;

constexpr uint32_t kNoTarget = 0xFFFFFFFFu;

// Whole block: f(entry) for the entries in[0 .. m), by whole warps (a thread
// without an entry gets one with target `none`), four loads per thread in
// flight.
template <typename F>
__device__ __forceinline__ void for_entries(const uint4* in, uint32_t m, uint32_t none, F&& f) {
    constexpr uint32_t kInFlight = 4;
    for (uint32_t c = 0; c < m; c += blockDim.x * kInFlight) {
        uint4 q[kInFlight];
#pragma unroll
        for (uint32_t u = 0; u < kInFlight; ++u) {
            const uint32_t i = c + u * blockDim.x + threadIdx.x;
            q[u] = i < m ? in[i] : make_uint4(0u, 0u, none, 0u);
        }
#pragma unroll
        for (uint32_t u = 0; u < kInFlight; ++u) f(q[u]);
    }
}

// Events k_group holds in shared memory (each thread its share in registers
// first).
constexpr uint32_t kSortSmemEvents = 4096;
constexpr uint32_t kSortPerThread = kSortSmemEvents / kThreads;
constexpr size_t kSortSmemBytes = kSortSmemEvents * (sizeof(unsigned long long) + sizeof(uint16_t));

// Grouping entry points: one block per bucket.  A bucket that fits is counted
// by target, placed in shared memory by target, and every event goes to its
// rank in due order among its target's events (as k_events does); a larger
// one, or one with a long segment, is counted and placed in grp from global
// memory, and k_group_rest sorts its segments.  Streams the events once in (16
// bytes each) and once out (8); the due order used to be a pass of its own
// over grp, a warp per target: 55 + 358 -> 120 us for 13 M events over 1e6
// targets.
__global__ void __launch_bounds__(kThreads) k_group(const __grid_constant__ Engine e) {
    tick_enter();
    extern __shared__ __align__(16) unsigned long long s_sort[];  // kSortSmemEvents words, their targets, counters
    uint16_t* s_tgt = reinterpret_cast<uint16_t*>(s_sort + kSortSmemEvents);
    uint32_t* s_cnt = reinterpret_cast<uint32_t*>(s_tgt + kSortSmemEvents);  // [2^bucket_shift + 1]
    const uint32_t width = 1u << e.bucket_shift;
    for (uint32_t b = blockIdx.x; b < e.nbuckets; b += gridDim.x) {
        const uint32_t lo = e.bstart[b], hi = e.bstart[b + 1], m = hi - lo;
        const uint32_t n0 = b << e.bucket_shift;
        const uint32_t nw = e.N - n0 < width ? e.N - n0 : width;
        const uint4* in = reinterpret_cast<const uint4*>(e.grp_tmp) + lo;
        unsigned long long* out = e.grp + lo;
        bool small = m <= kSortSmemEvents;
        unsigned long long v[kSortPerThread];
        uint32_t at[kSortPerThread];  // target, and its place among the target's events << 16
        if (small) {
#pragma unroll
            for (uint32_t k = 0; k < kSortPerThread; ++k) {
                const uint32_t i = threadIdx.x + k * kThreads;
                const uint4 q = i < m ? in[i] : make_uint4(0u, 0u, 0xFFFFu, 0u);
                v[k] = (static_cast<unsigned long long>(q.y) << 32) | q.x;
                at[k] = q.z < nw ? q.z : 0xFFFFu;
            }
        }
        for (uint32_t j = threadIdx.x; j < nw; j += blockDim.x) s_cnt[j] = 0;
        __syncthreads();
        if (small) {
#pragma unroll
            for (uint32_t k = 0; k < kSortPerThread; ++k)
                if (at[k] != 0xFFFFu) at[k] |= atomicAdd(&s_cnt[at[k]], 1u) << 16;
        } else {
            for_entries(in, m, nw, [&](const uint4& q) { warp_count(s_cnt, q.z < nw ? q.z : nw, nw); });
        }
        __syncthreads();
        uint32_t longest = 0;
        for (uint32_t j = threadIdx.x; j < nw; j += blockDim.x) longest = max(longest, s_cnt[j]);
        small = !__syncthreads_or(longest > kRankEvents) && small;
        const uint32_t total = block_scan_shared<kThreads>(s_cnt, nw);  // segment starts relative to lo
        for (uint32_t j = threadIdx.x; j < nw; j += blockDim.x) e.seg_start[n0 + j] = lo + s_cnt[j];
        if (threadIdx.x == 0) s_cnt[nw] = total;
        __syncthreads();
        if (small) {
#pragma unroll
            for (uint32_t k = 0; k < kSortPerThread; ++k) {
                const uint32_t j = at[k] & 0xFFFFu;
                if (j == 0xFFFFu) continue;
                const uint32_t p = s_cnt[j] + (at[k] >> 16);
                s_sort[p] = v[k];
                s_tgt[p] = static_cast<uint16_t>(j);
            }
            __syncthreads();
            for (uint32_t i = threadIdx.x; i < total; i += blockDim.x) {
                const unsigned long long x = s_sort[i];
                const uint32_t j = s_tgt[i], key = grp_key(x), q1 = s_cnt[j + 1];
                uint32_t p = s_cnt[j];
                for (uint32_t q = p; q < q1; ++q) p += grp_key(s_sort[q]) < key;
                out[p] = x;
            }
        } else {
            // placed with cursors that start at the segment starts (s_cnt[j]
            // ends at the segment's end, target j + 1's start)
            for_entries(in, m, nw, [&](const uint4& q) {
                const uint32_t p = warp_count(s_cnt, q.z < nw ? q.z : nw, nw);
                if (q.z < nw) out[p] = (static_cast<unsigned long long>(q.y) << 32) | q.x;
            });
            // the segments are sorted by k_group_rest, over the whole GPU: the
            // totals and counts are used up, their memory takes its lists
            // (group_counters)
            if (threadIdx.x == 0) e.btot[atomicAdd(&e.ts->n_touched, 1u)] = b;
            __syncthreads();
            for (uint32_t j = threadIdx.x; j < nw; j += blockDim.x) {
                const uint32_t beg = j > 0 ? s_cnt[j - 1] : 0u;
                if (s_cnt[j] - beg > kWarpSortEvents) e.bcnt[atomicAdd(&e.ts->n_fired_targets, 1u)] = n0 + j;
            }
        }
        __syncthreads();
    }
}

constexpr int kLongThreads = 1024;
// The longest listed segment that a warp sorts when there is one for every warp:
// a block takes about 10 us for it whatever its length (20,000 segments of 650
// events 1.5 ms by warps, 2.0 by blocks; of 1,000 events 2.4 and 2.7).
constexpr uint32_t kWarpSortMany = 1024;
constexpr size_t kLongSmemBytes = 256 * (kLongThreads / 32 + 1) * sizeof(uint32_t);

// Grouping entry points: due order of the segments k_group left: a warp for
// each target of the buckets it listed, and a block for each target it listed
// (more than kWarpSortEvents events; of many, a warp for the shorter ones).  One warp merged such a long segment: 200
// ms for the 450,000 events of one target among 9 M, now 1.6 (and 0.7 in
// k_group before it, from 1.5 with every entry's own atomic on the one counter).
// The entries of a listed bucket are all placed: their memory is the scratch.
__global__ void __launch_bounds__(kLongThreads) k_group_rest(const __grid_constant__ Engine e) {
    tick_enter();
    extern __shared__ uint32_t s_radix[];
    const uint32_t buckets = e.ts->n_touched, targets = e.ts->n_fired_targets;
    auto segment = [&](uint32_t n, unsigned long long*& g, unsigned long long*& tmp) {
        const uint32_t beg = e.seg_start[n], lo = e.bstart[n >> e.bucket_shift];
        g = e.grp + beg;
        tmp = reinterpret_cast<unsigned long long*>(e.grp_tmp + lo) + (beg - lo);
        return e.seg_start[n + 1] - beg;
    };
    unsigned long long *g, *tmp;
    const unsigned long long items = static_cast<unsigned long long>(buckets) << e.bucket_shift;
    const uint32_t warps = gridDim.x * (kLongThreads / 32);
    const bool many = targets >= warps;
    // (item i's target: neighbouring warps take different blocks' SMs; the
    // listed targets come behind the buckets')
    for (unsigned long long i = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; i < items + (many ? targets : 0u); i += warps) {
        const bool listed = i >= items;
        const uint32_t n = listed ? e.bcnt[i - items]
                                  : (e.btot[i >> e.bucket_shift] << e.bucket_shift) +
                                        static_cast<uint32_t>(i & ((1u << e.bucket_shift) - 1u));
        if (n >= e.N) continue;
        const uint32_t len = segment(n, g, tmp);
        if (listed ? len <= kWarpSortMany : len <= kWarpSortEvents) sort_group(g, tmp, len);
    }
    const uint32_t bits = due_bits(e.ts->n_due);
    for (uint32_t k = blockIdx.x; k < targets; k += gridDim.x) {
        const uint32_t len = segment(e.bcnt[k], g, tmp);
        if (many && len <= kWarpSortMany) continue;
        __syncthreads();
        block_radix_sort<kLongThreads>(g, tmp, len, bits, s_radix);
    }
}

// Grouping entry points: the scratch as the counting kernels expect it.
__global__ void k_group_init(const __grid_constant__ Engine e, uint32_t count) {
    for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b < e.nbuckets; b += gridDim.x * blockDim.x) {
        e.btot[b] = 0;
        e.bcur[b] = 0;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *e.ts = TickState{};
        *e.slot_count = count;
    }
}

// Pre-spike part of one synaptic event on its synapse record, in the
// reference's order (SynapseDendriteProcessor.cpp:104-133): pre-spike STDP
// against the last post spike, last_pre, the pre-spike count, and the
// spike-code pattern (:318-365).  None of it depends on the target's neuron
// state; only the STDP part depends on whether the target fired earlier in the
// tick, which the walk handles by redoing it (walk_after_fire).
template <bool kInline>
__device__ __forceinline__ void pre_event(SynAB& r, const TargetParam& p, uint32_t t, uint16_t* lc,
                                          const Engine& e, int stdp, int temporal, bool inl) {
    SynA& a = r.a;
    const uint32_t delay = a.meta & kMetaDelayMask;
    const uint32_t pre_tick = t >= delay ? t - delay : t;
    if (((a.meta >> kMetaPlasticBit) & 1u) && a.last_post1 != 0)
        stdp_apply(a, pre_tick, a.last_post1 - 1, e, stdp, e.tab.ltp);
    a.last_pre1 = pre_tick + 1;
    r.b.pre_count += 1;
    code_update<kInline>(r.b, p, t, lc, e.code_stride, temporal, inl);
}

__device__ __forceinline__ SynPre pre_fields(const SynA& a) {
    SynPre f;
    f.weight = a.weight;
    f.last_pre1 = a.last_pre1;
    f.updates = a.updates;
    f.last_delta = a.last_delta;
    return f;
}

// The record as it was before an event: the fields pre_event changes from
// the event's SynPre, the others (static fields, last_post1, post_cnt) from
// the record, which nothing but the post-spike catch-up changes.
__device__ __forceinline__ SynA before_event(SynA a, const SynPre& f) {
    a.weight = f.weight;
    a.last_pre1 = f.last_pre1;
    a.updates = f.updates;
    a.last_delta = f.last_delta;
    return a;
}

__device__ __forceinline__ uint32_t ev_bits(const SynA& a) {
    return ((a.meta >> kMetaCompShift) & 3u) | (((a.meta >> kMetaRecShift) & 3u) << 2);
}

// Starts bringing a line from DRAM into L2.
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// A synapse record moved with 32-byte accesses, one per half (half the
// requests of 16-byte ones; each half is one DRAM sector).
__device__ __forceinline__ void load_words(const void* p, uint32_t* v) {
    asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "l"(p)
                 : "memory");
}

__device__ __forceinline__ SynA load_half(const SynA* p) {
    uint32_t v[8];
    load_words(p, v);
    SynA a;
    a.weight = __uint_as_float(v[0]);
    a.last_pre1 = v[1];
    a.last_post1 = v[2];
    a.meta = v[3];
    a.clamp_hi = __uint_as_float(v[4]);
    a.updates = v[5];
    a.last_delta = __uint_as_float(v[6]);
    a.post_cnt = v[7];
    return a;
}

__device__ __forceinline__ void store_half(SynA* p, const SynA& a) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(__float_as_uint(a.weight)),
                 "r"(a.last_pre1), "r"(a.last_post1), "r"(a.meta), "r"(__float_as_uint(a.clamp_hi)), "r"(a.updates),
                 "r"(__float_as_uint(a.last_delta)), "r"(a.post_cnt)
                 : "memory");
}

__device__ __forceinline__ SynAB load_record(const SynAB* p) {
    SynAB r;
    uint32_t v[8];
    r.a = load_half(&p->a);
    load_words(&p->b, v);
    r.b.pre_count = v[0];
    r.b.code_ws = v[1];
    r.b.code_matches = v[2];
    r.b.code_len = static_cast<uint8_t>(v[3]);
    r.b.flags = static_cast<uint8_t>(v[3] >> 8);
    r.b.learned_count = static_cast<uint16_t>(v[3] >> 16);
    r.b.ring_lo = (static_cast<unsigned long long>(v[5]) << 32) | v[4];
    r.b.ring_hi = (static_cast<unsigned long long>(v[7]) << 32) | v[6];
    return r;
}

__device__ __forceinline__ void store_record(SynAB* p, const SynAB& r) {
    store_half(&p->a, r.a);
    const uint32_t bits = r.b.code_len | (static_cast<uint32_t>(r.b.flags) << 8) |
                          (static_cast<uint32_t>(r.b.learned_count) << 16);
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(&p->b), "r"(r.b.pre_count), "r"(r.b.code_ws),
                 "r"(r.b.code_matches), "r"(bits), "r"(static_cast<uint32_t>(r.b.ring_lo)),
                 "r"(static_cast<uint32_t>(r.b.ring_lo >> 32)), "r"(static_cast<uint32_t>(r.b.ring_hi)),
                 "r"(static_cast<uint32_t>(r.b.ring_hi >> 32))
                 : "memory");
}

// The parameters of a block's targets: in shared memory, or (k_small, and buckets
// wider than kSharedParams targets: networks beyond 2^23 neurons) in the first 16
// bytes of each NeuronParam.
constexpr uint32_t kSharedParams = 256;

__device__ __forceinline__ TargetParam load_param(const NeuronParam* p) {
    const uint4 q = *reinterpret_cast<const uint4*>(p);
    return TargetParam{__uint_as_float(q.x), q.y, __uint_as_float(q.z), q.w};
}

// The blocks of k_small share out the neurons by runs of kSmallChunk: every block
// has one of eight neighbouring runs, at a place that the number of their group
// turns by a little less than three.  Neighbours, which are often busy together
// (an output layer), so go to different blocks, and so do groups of them at any
// regular distance (a layer of every column: the busiest block has 1.04 times
// its share on average, 1.2 at worst, over widths of 5 to 32 and 3 to 32 layers).
// One by one, the records' reads would take twice the lines (38 us a tick of
// 5,000 events with runs of 8 or 32, 45 with 1).
constexpr uint32_t kSmallChunk = 8;
static_assert(kSmallBlocks == 8, "a group is eight runs");

__device__ __forceinline__ uint32_t small_turn(uint32_t group) { return group * 93 >> 5; }
__device__ __forceinline__ uint32_t small_block(uint32_t n) {
    return (n / kSmallChunk + small_turn(n / (kSmallChunk * kSmallBlocks))) % kSmallBlocks;
}
// A neuron's place among its block's, and the neuron at place j of block c.
__device__ __forceinline__ uint32_t small_place(uint32_t n) {
    return n / (kSmallChunk * kSmallBlocks) * kSmallChunk + n % kSmallChunk;
}
__device__ __forceinline__ uint32_t small_neuron(uint32_t c, uint32_t j) {
    const uint32_t group = j / kSmallChunk, run = group * kSmallBlocks + (c - small_turn(group)) % kSmallBlocks;
    return run * kSmallChunk + j % kSmallChunk;
}

// Target j of a block: neuron first + j, or (kSmall) k_small's.
template <bool kSmall>
__device__ __forceinline__ uint32_t neuron_of(uint32_t first, uint32_t j) {
    return kSmall ? small_neuron(first, j) : first + j;
}

template <bool kSmall>
struct BucketParams {
    const TargetParam* shared;
    const NeuronParam* global;
    uint32_t first;  // (neuron_of)
    bool in_shared;
    __device__ __forceinline__ TargetParam operator[](uint32_t j) const {
        return in_shared ? shared[j] : load_param(global + neuron_of<kSmall>(first, j));
    }
};

constexpr uint32_t kSharedSynapse = 0x8000u;  // beside an event's target: its synapse has other events in the tick
static_assert(kBlockEvents * sizeof(BucketEntry) >= 256 * (kEventThreads / 32 + 1) * sizeof(uint32_t), "s_radix");
static_assert((1u << kMaxBucketShift) <= kSharedSynapse, "targets of a bucket");

// A bucket's events grouped by target in due order, as the event and walk
// phases of k_events see them.  Indices count from the bucket's first event.
//
// In shared memory.
struct SharedEvents {
    unsigned long long* word;  // payload << 32 | due index << 1 | external
    float* w;                  // weight the event delivers
    uint8_t* bits;             // EvIn::bits
    __device__ __forceinline__ EvIn at(uint32_t i) const {
        const unsigned long long v = word[i];
        EvIn x;
        x.weight = w[i];
        x.bits = bits[i];
        x.tm = static_cast<uint32_t>(v >> 32);
        x.due = static_cast<uint32_t>(v) >> 1;
        return x;
    }
    __device__ __forceinline__ uint32_t bits_of(uint32_t i) const { return bits[i]; }
    __device__ __forceinline__ float weight_of(uint32_t i) const { return w[i]; }
    __device__ __forceinline__ bool external(uint32_t i) const { return static_cast<uint32_t>(word[i]) & 1u; }
    __device__ __forceinline__ uint32_t payload(uint32_t i) const { return static_cast<uint32_t>(word[i] >> 32); }
    __device__ __forceinline__ void put(uint32_t i, float weight, uint32_t b) const {
        w[i] = weight;
        bits[i] = static_cast<uint8_t>(b);
    }
};

// In global memory (a bucket with more events than a block holds, or a long
// group): the grouped words of Engine::grp and one EvIn each.
struct GlobalEvents {
    const unsigned long long* word;  // payload << 32 | due index | external bit
    EvIn* in;
    __device__ __forceinline__ EvIn at(uint32_t i) const { return in[i]; }
    __device__ __forceinline__ uint32_t bits_of(uint32_t i) const { return in[i].bits; }
    __device__ __forceinline__ float weight_of(uint32_t i) const { return in[i].weight; }
    __device__ __forceinline__ bool external(uint32_t i) const {
        return static_cast<uint32_t>(word[i]) & kExternalBit;
    }
    __device__ __forceinline__ uint32_t payload(uint32_t i) const { return static_cast<uint32_t>(word[i] >> 32); }
    __device__ __forceinline__ void put(uint32_t i, float weight, uint32_t b) const {
        EvIn x;
        x.weight = weight;
        x.bits = b;
        const unsigned long long v = word[i];
        x.tm = static_cast<uint32_t>(v >> 32);
        x.due = static_cast<uint32_t>(v) & ~kExternalBit;
        in[i] = x;
    }
};

// Event i's synapse record: the fields before the event (Engine::ev_a0), its
// pre-spike work and its input for the walk.  `last` is the end of the
// target's events if the synapse may have further ones there (they follow in
// due order), else i + 1.
template <bool kInline, typename Events>
__device__ __forceinline__ void synapse_events(const Engine& e, const Events& ev, uint32_t lo, uint32_t i,
                                               uint32_t last, const TargetParam& p, uint32_t n, uint32_t t, int stdp,
                                               int temporal) {
    const uint32_t tm = ev.payload(i);
    const bool inl = kInline || inline_code_pattern(p.max_refs, e.code_stride);
    uint16_t* lc = nullptr;
    if (!inl) {
        const NeuronParam& q = e.nparam[n];
        lc = e.lcode + q.lcode_base + static_cast<size_t>(tm - q.in_begin) * p.max_refs * e.code_stride;
    }
    SynAB r = load_record(e.syn + tm);
    // one body for the first and the further events, so that a warp's lanes
    // go through it together whatever the distance to their next event
    for (uint32_t q = i, repeat = 0;;) {
        e.ev_a0[lo + q] = pre_fields(r.a);
        pre_event<kInline>(r, p, t, lc, e, stdp, temporal, inl);
        ev.put(q, r.a.weight, ev_bits(r.a) | repeat);
        do {
            ++q;
        } while (q < last && (ev.payload(q) != tm || ev.external(q)));
        if (q >= last) break;
        repeat = kEvRepeat;
    }
    store_record(e.syn + tm, r);
}

// Applies to a synapse record the post-spike STDP owed for the target's fires
// so far and the event's pre-spike STDP (the record is the synapse's state
// before the event) and returns the weight the event delivers.  Both STDP
// steps have post >= pre, so they read only the LTP table.
__device__ __forceinline__ float redo_pre_stdp(const Engine& e, SynA& a, uint32_t t, uint32_t fires, int stdp,
                                               const float* ltp) {
    post_catch_up(a, t, fires, e, stdp, ltp);
    const uint32_t delay = a.meta & kMetaDelayMask;
    const uint32_t pre_tick = t >= delay ? t - delay : t;
    if (((a.meta >> kMetaPlasticBit) & 1u) && a.last_post1 != 0)
        stdp_apply(a, pre_tick, a.last_post1 - 1, e, stdp, ltp);
    a.last_pre1 = pre_tick + 1;
    return a.weight;
}

__device__ __forceinline__ SynA shfl_syn(const SynA& a, uint32_t src) {
    SynA r;
    r.weight = __shfl_sync(0xffffffffu, a.weight, src);
    r.last_pre1 = __shfl_sync(0xffffffffu, a.last_pre1, src);
    r.last_post1 = __shfl_sync(0xffffffffu, a.last_post1, src);
    r.meta = __shfl_sync(0xffffffffu, a.meta, src);
    r.clamp_hi = __shfl_sync(0xffffffffu, a.clamp_hi, src);
    r.updates = __shfl_sync(0xffffffffu, a.updates, src);
    r.last_delta = __shfl_sync(0xffffffffu, a.last_delta, src);
    r.post_cnt = __shfl_sync(0xffffffffu, a.post_cnt, src);
    return r;
}

// The physics fields of a neuron's state.
__device__ __forceinline__ void load_physics(NState& s, const NeuronRec* rec) {
    const float4 c = reinterpret_cast<const float4*>(rec->cur)[0];
    const uint4 u = reinterpret_cast<const uint4*>(rec->upd)[0];
    const uint4 m = *reinterpret_cast<const uint4*>(&rec->membrane);
    s.cur[0] = c.x;
    s.cur[1] = c.y;
    s.cur[2] = c.z;
    s.cur[3] = c.w;
    s.upd[0] = u.x;
    s.upd[1] = u.y;
    s.upd[2] = u.z;
    s.upd[3] = u.w;
    s.membrane = __uint_as_float(m.x);
    s.spikes = m.y;
    s.last_fired1 = m.z;
    s.last_active = m.w;
    s.flags = rec->flags;
}

__device__ __forceinline__ void store_physics(const NState& s, NeuronRec* rec) {
    reinterpret_cast<float4*>(rec->cur)[0] = make_float4(s.cur[0], s.cur[1], s.cur[2], s.cur[3]);
    reinterpret_cast<uint4*>(rec->upd)[0] = make_uint4(s.upd[0], s.upd[1], s.upd[2], s.upd[3]);
    *reinterpret_cast<uint4*>(&rec->membrane) =
        make_uint4(__float_as_uint(s.membrane), s.spikes, s.last_fired1, s.last_active);
    rec->flags = s.flags;
}

// A fire of neuron n at due position `due`: its bit in the fire bitmap, the
// neuron, and one more fire in the bitmap tile (kThreads words) for
// k_fire_list.
__device__ __forceinline__ void record_fire(const Engine& e, uint32_t n, uint32_t due) {
    atomicOr(&e.fire_bits[due >> 5], 1u << (due & 31));
    e.fire_at[due] = n;
    atomicAdd(&e.fire_tile[(due >> 5) / kThreads], 1u);
}

// Where a walk's fires go: the engine's bitmap and list of fired targets.
struct EngineFires {
    const Engine& e;
    __device__ __forceinline__ void fire(uint32_t n, uint32_t due) const { record_fire(e, n, due); }
    // A target that fired `fires` times this tick (k_post).
    __device__ __forceinline__ void target(uint32_t n, uint32_t fires) const {
        const uint32_t j = atomicAdd(&e.ts->n_fired_targets, 1u);
        e.fired_tgt[j] = n;
        e.fired_cnt[j] = fires;
    }
};

// A target whose walk goes on after its first fire.
struct Refire {
    uint32_t j;     // target within the bucket
    uint32_t next;  // its event after the fire
};

// The rest of a fired target's walk, one warp.  Every synaptic event after a
// fire redoes its STDP with the target's fire count so far, starting from the
// synapse's state before the event: its snapshot, or, when the same synapse
// already had an event after the first fire, the record that event left.  The
// warp redoes up to 32 events at once (an event whose predecessor is in the
// same chunk waits a round and takes its record by shuffle); then the neuron
// physics run over them in order (in lane 0: state `s`).  If the target fires
// again inside the chunk, the events after that fire are redone with the new
// count; only the records of events before it are stored (the last event of
// each synapse stores).  The result is the sequential order's.  `beg`: the
// target's first event in the bucket, `lo`: the bucket's first event in the
// tick (Engine::ev_a0 counts from there).  Returns the target's fires.
template <typename Events, typename Fires>
__device__ __forceinline__ uint32_t walk_after_fire(const Engine& e, NState& s, float threshold, uint32_t n,
                                                    uint32_t beg, uint32_t len, uint32_t after, uint32_t t, int stdp,
                                                    const Events& ev, uint32_t lo, float* s_wt, const Fires& out) {
    const uint32_t lane = threadIdx.x & 31;
    const float* ltp = e.tab.ltp;
    uint32_t pos = after, fires = 1;
    while (pos < len) {
        const uint32_t m = len - pos < 32 ? len - pos : 32;
        const uint32_t j = pos + lane;
        EvIn x{};
        if (lane < m) x = ev.at(beg + j);
        const bool syn = lane < m && !(x.bits & kEvExternal);
        // the synapse's latest earlier event after the first fire
        uint32_t pred = 0xFFFFFFFFu;
        if (syn && (x.bits & kEvRepeat)) {
            for (uint32_t q = j; q-- > after;) {
                const EvIn y = ev.at(beg + q);
                if (!(y.bits & kEvExternal) && y.tm == x.tm) {
                    pred = q;
                    break;
                }
            }
        }
        const bool wait = pred != 0xFFFFFFFFu && pred >= pos;  // predecessor in this chunk
        SynA a{};
        float wt = x.weight;
        bool done = !syn;
        if (syn && !wait) {
            a = pred != 0xFFFFFFFFu ? e.syn[x.tm].a : before_event(e.syn[x.tm].a, e.ev_a0[lo + beg + j]);
            wt = redo_pre_stdp(e, a, t, fires, stdp, ltp);
            done = true;
        }
        while (!__all_sync(0xffffffffu, done)) {
            const uint32_t src = wait ? pred - pos : lane;
            const SynA pa = shfl_syn(a, src);
            const bool pdone = __shfl_sync(0xffffffffu, done, src);
            if (!done && pdone) {
                a = pa;
                wt = redo_pre_stdp(e, a, t, fires, stdp, ltp);
                done = true;
            }
        }
        if (lane < m) s_wt[lane] = wt;
        __syncwarp();
        uint32_t next = pos + m;
        if (lane == 0) {
            for (uint32_t c = 0; c < m; ++c) {
                const uint32_t bits = ev.bits_of(beg + pos + c);
                if (process_input(s, threshold, bits & 3u, (bits >> 2) & 3u, s_wt[c], t)) {
                    out.fire(n, ev.at(beg + pos + c).due);
                    fires += 1;
                    if (c + 1 < m) {
                        next = pos + c + 1;
                        break;
                    }
                }
            }
        }
        next = __shfl_sync(0xffffffffu, next, 0);
        // store the records of the events before `next`, the last one of
        // each synapse
        const bool store = syn && j < next;
        const unsigned long long key = store ? x.tm : (1ull << 32) | lane;
        const unsigned same = __match_any_sync(0xffffffffu, key);
        if (store && lane == 31u - __clz(same)) e.syn[x.tm].a = a;
        pos = next;
        fires = __shfl_sync(0xffffffffu, fires, 0);
        __syncwarp();
    }
    return fires;
}

__device__ __forceinline__ void temporal_target(const Engine& e, uint32_t n, uint32_t k, uint32_t t, int temporal);

// The walks of a bucket's targets (the reference's sequential per-event loop,
// NetworkPropagator.cpp:80-131, restricted to each target).  A thread per
// target processes its events in due order up to and including its first fire
// (every event before it uses the weight its synapse's work computed).  The
// few targets with events after their first fire are then shared out to the
// block's warps (one warp did its own 32 targets' one after the other: up to
// 20 us with three or four of them, where the walk itself takes 4; sharing them
// took the kernel from 36 to 32 us at 250,000 events, 197 to 187 at 2.5 M).
// The targets: the block's nw, or of them the nw in `list` (if not null).
template <int kT, bool kSmall, typename Events, typename Fires>
__device__ __forceinline__ void walk_bucket(const Engine& e, const Events& ev, uint32_t lo, uint32_t n0, uint32_t nw,
                                            const uint16_t* list, const uint32_t* s_seg,
                                            const BucketParams<kSmall>& par, uint32_t t, int stdp, float* s_wt,
                                            Refire* s_refire, uint32_t* s_refires, const Fires& out) {
    for (uint32_t j0 = 0; j0 < nw; j0 += kT) {
        if (threadIdx.x == 0) *s_refires = 0;
        __syncthreads();
        const uint32_t at = j0 + threadIdx.x, j = at < nw && list ? list[at] : at;
        const uint32_t n = neuron_of<kSmall>(n0, j);
        const uint32_t beg = at < nw ? s_seg[j] : 0u, len = at < nw ? s_seg[j + 1] - beg : 0u;
        if (len > 0) {
            NeuronRec* rec = e.nrec + n;
            const float threshold = par[j].threshold;
            NState s;
            load_physics(s, rec);
            decay_to(s, t, e);
            for (uint32_t i = 0; i < len; ++i) {
                const uint32_t bits = ev.bits_of(beg + i);
                if (process_input(s, threshold, bits & 3u, (bits >> 2) & 3u, ev.weight_of(beg + i), t)) {
                    out.fire(n, ev.at(beg + i).due);
                    if (i + 1 < len) {
                        s_refire[atomicAdd(s_refires, 1u)] = Refire{j, i + 1};
                    } else {
                        out.target(n, 1);
                    }
                    break;
                }
            }
            store_physics(s, rec);
        }
        __syncthreads();
        const uint32_t refires = *s_refires, warp = threadIdx.x >> 5;
        for (uint32_t k = warp; k < refires; k += kT / 32) {
            const Refire f = s_refire[k];
            const uint32_t n = neuron_of<kSmall>(n0, f.j), first = s_seg[f.j];
            NState s;
            load_physics(s, e.nrec + n);
            const uint32_t fires = walk_after_fire(e, s, par[f.j].threshold, n, first, s_seg[f.j + 1] - first, f.next, t,
                                                   stdp, ev, lo, s_wt + 32 * warp, out);
            if ((threadIdx.x & 31) == 0) {
                store_physics(s, e.nrec + n);
                out.target(n, fires);
            }
        }
        __syncthreads();
    }
}

// A part with more events than the block's shared memory, or a bucket or part
// with a long group: grouped in Engine::grp (a counting sort by target, then a
// warp per target, or the block for a long group, puts its events in due
// order), its event inputs in Engine::evin.  `in`: the whole bucket's `all`
// entries, of which those of the targets j0 .. j0 + nw - 1 are meant (`lo`: the
// first one's position in the tick).  s_radix: the block's shared memory,
// otherwise unused on this path.
template <bool kInline>
__device__ __noinline__ void bucket_in_global(const Engine& e, const uint4* in, uint32_t all, uint32_t j0,
                                              uint32_t lo, uint32_t n0, uint32_t nw, uint32_t* s_seg,
                                              const BucketParams<false>& par, uint32_t t, int stdp, int temporal,
                                              float* s_wt, Refire* s_refire, uint32_t* s_refires,
                                              uint32_t* s_radix) {
    unsigned long long* grp = e.grp + lo;
    // s_seg[j + 1] holds target j's count, then its cursor, then its end
    for (uint32_t j = threadIdx.x; j <= nw; j += blockDim.x) s_seg[j] = 0;
    __syncthreads();
    for_entries(in, all, kNoTarget, [&](const uint4& q) { warp_count(s_seg + 1, min(q.z - j0, nw), nw); });
    __syncthreads();
    block_scan_shared<kEventThreads>(s_seg + 1, nw);
    for_entries(in, all, kNoTarget, [&](const uint4& q) {
        const uint32_t j = min(q.z - j0, nw), p = warp_count(s_seg + 1, j, nw);
        if (j < nw) grp[p] = (static_cast<unsigned long long>(q.y) << 32) | q.x;
    });
    __syncthreads();
    // the events' inputs are written after the sorts: until then their memory
    // is the merges' scratch (the entries may still be read for other parts)
    unsigned long long* tmp = reinterpret_cast<unsigned long long*>(e.evin + lo);
    for (uint32_t j = threadIdx.x >> 5; j < nw; j += blockDim.x / 32) {
        const uint32_t beg = s_seg[j], len = s_seg[j + 1] - beg;
        if (len <= kWarpSortEvents) sort_group(grp + beg, tmp + beg, len);
    }
    for (uint32_t j = 0; j < nw; ++j) {
        const uint32_t beg = s_seg[j], len = s_seg[j + 1] - beg;
        if (len > kWarpSortEvents)
            block_radix_sort<kEventThreads>(grp + beg, tmp + beg, len, due_bits(e.ts->n_due), s_radix);
    }
    __syncthreads();
    const GlobalEvents ev{grp, e.evin + lo};
    const uint32_t total = s_seg[nw];
    for (uint32_t i = threadIdx.x; i < total; i += blockDim.x) {
        if (ev.external(i)) {
            ev.put(i, __uint_as_float(ev.payload(i)), kEvExternal);
            continue;
        }
        uint32_t j = 0, above = nw;  // s_seg[j] <= i < s_seg[above]
        while (above - j > 1) {
            const uint32_t mid = (j + above) >> 1;
            if (s_seg[mid] <= i) {
                j = mid;
            } else {
                above = mid;
            }
        }
        const uint32_t tm = ev.payload(i);
        bool first = true;
        for (uint32_t q = s_seg[j]; q < i && first; ++q) first = ev.external(q) || ev.payload(q) != tm;
        if (first) synapse_events<kInline>(e, ev, lo, i, s_seg[j + 1], par[j], n0 + j, t, stdp, temporal);
    }
    for (uint32_t j = threadIdx.x; j < nw; j += blockDim.x) {
        const uint32_t k = s_seg[j + 1] - s_seg[j];
        if (k > 0 && par[j].max_refs == 1) temporal_target(e, n0 + j, k, t, temporal);
    }
    __syncthreads();
    walk_bucket<kEventThreads>(e, ev, lo, n0, nw, nullptr, s_seg, par, t, stdp, s_wt, s_refire, s_refires,
                               EngineFires{e});
}

// Shared memory of a bucket's events besides SharedEvents.
struct BucketSpace {
    unsigned long long* word;  // the events' words grouped by target
    uint16_t* tgt;             // their targets
    uint16_t* list;            // first events of the synapses with several
    uint32_t* seg;             // seg[j + 1], seg[j + 2]: first and end of target j's events
    float* wt;                 // 32 per warp: weights of the events redone after a fire
    Refire* refire;            // a block's threads: targets that go on after their first fire
    uint32_t *repeats, *next, *refires;  // counters (the first two zero)
    uint16_t* multi;                     // kAlone: targets with several reference patterns,
    uint32_t* multis;                    // and their number (zero)
    const uint16_t* touched;             // targets with events (null: all are looked at)
};

template <int kGroup>
__device__ __forceinline__ void temporal_group(const Engine& e, uint32_t n, uint32_t k, uint32_t t, int enabled);

// Steps 2 (from the grouped words on) to 4 of k_events for one bucket.  kAlone:
// the block is not k_events': the temporal patterns of targets with several
// reference patterns are done here too.  The targets: the nw in b.touched, or all
// nw.
template <bool kInline, int kT, bool kAlone, typename Fires>
__device__ __forceinline__ void bucket_events(const Engine& e, const BucketSpace& b, const SharedEvents& ev,
                                              uint32_t total, uint32_t lo, uint32_t n0, uint32_t nw,
                                              const BucketParams<kAlone>& par, uint32_t t, int stdp, int temporal,
                                              const Fires& out) {
    auto target = [&](uint32_t i) { return kAlone && b.touched ? b.touched[i] : i; };
    if (kAlone && e.multi_refs)
        for (uint32_t i = threadIdx.x; i < nw; i += kT) {
            const uint32_t j = target(i);
            if (b.seg[j + 2] > b.seg[j + 1] && par[j].max_refs != 1) b.multi[atomicAdd(b.multis, 1u)] = static_cast<uint16_t>(j);
        }
    // each event's rank in due order among its target's events
    // (by position: the lanes of a warp read the same or the next
    // group's words); of the synapses with several events, the
    // first event goes on a list
    for (uint32_t i = threadIdx.x; i < total; i += kT) {
        const unsigned long long v = b.word[i];
        const uint32_t j = b.tgt[i] & ~kSharedSynapse, s0 = b.seg[j + 1], s1 = b.seg[j + 2];
        const uint32_t due = static_cast<uint32_t>(v), pay = static_cast<uint32_t>(v >> 32);
        uint32_t p = s0, same = 0, before = 0;  // synaptic events with this payload, those due earlier
        for (uint32_t q = s0; q < s1; ++q) {
            const unsigned long long x = b.word[q];
            const uint32_t d = static_cast<uint32_t>(x);
            const bool hit = static_cast<uint32_t>(x >> 32) == pay && !(d & 1u);
            p += d < due;
            same += hit;
            before += hit && d < due;
        }
        ev.word[p] = v;
        if (same > 1 && !(due & 1u)) {
            b.tgt[p] = static_cast<uint16_t>(j | kSharedSynapse);
            if (before == 0) b.list[atomicAdd(b.repeats, 1u)] = static_cast<uint16_t>(p);
        }
    }
    __syncthreads();
    if (!kAlone && e.multi_refs)
        for (uint32_t j = threadIdx.x; j < nw; j += kT) e.seg_start[n0 + j] = lo + b.seg[j + 1];
    // The warps share out the rest but the walk: the temporal
    // patterns (they need only the targets' event counts) 32
    // targets at a time from the first warps, the synapses with
    // several events, then all other events.
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t i = threadIdx.x; i < nw; i += kT) {
        const uint32_t j = target(i), k = b.seg[j + 2] - b.seg[j + 1];
        if (k > 0 && par[j].max_refs == 1) temporal_target(e, neuron_of<kAlone>(n0, j), k, t, temporal);
    }
    __syncwarp();
    constexpr uint32_t kGroup = 8;  // lanes per target with several reference patterns
    const uint32_t multis = kAlone ? *b.multis : 0u, patterns = (multis + 32 / kGroup - 1) / (32 / kGroup);
    const uint32_t repeats = *b.repeats, lists = (repeats + 31) / 32, tasks = patterns + lists + (total + 31) / 32;
    for (;;) {
        uint32_t task = lane == 0 ? atomicAdd(b.next, 1u) : 0u;
        task = __shfl_sync(0xffffffffu, task, 0);
        if (task >= tasks) break;
        if constexpr (kAlone) {
            if (task < patterns) {
                const uint32_t k = (task * 32 + lane) / kGroup;
                if (k < multis) {
                    const uint32_t j = b.multi[k];
                    temporal_group<kGroup>(e, neuron_of<kAlone>(n0, j), b.seg[j + 2] - b.seg[j + 1], t, temporal);
                }
                __syncwarp();
                continue;
            }
            task -= patterns;
        }
        uint32_t i = (task - lists) * 32 + lane, last = 0;
        bool run;
        if (task < lists) {
            const uint32_t k = task * 32 + lane;
            run = k < repeats;
            if (run) {
                i = b.list[k];
                last = b.seg[(b.tgt[i] & ~kSharedSynapse) + 2];
            }
        } else {
            run = i < total;
            if (run && ev.external(i)) {
                ev.put(i, __uint_as_float(ev.payload(i)), kEvExternal);
                run = false;
            }
            run = run && !(b.tgt[i] & kSharedSynapse);
            last = i + 1;
        }
        if (run) {
            const uint32_t j = b.tgt[i] & ~kSharedSynapse;
            synapse_events<kInline>(e, ev, lo, i, last, par[j], neuron_of<kAlone>(n0, j), t, stdp, temporal);
        }
        __syncwarp();
    }
    __syncthreads();
    walk_bucket<kT>(e, ev, lo, n0, nw, kAlone ? b.touched : nullptr, b.seg + 1, par, t, stdp, b.wt, b.refire, b.refires,
                    out);
}

// The entries of the targets j0 .. j0 + nw - 1 among a bucket's `all`, as far as
// they fit, into s_in (targets from j0); whole block.  Returns their number and
// that of the entries before j0.
__device__ __noinline__ uint2 pick_part(const uint4* in, uint32_t all, uint32_t j0, uint32_t nw, uint4* s_in) {
    __shared__ uint32_t s_mine, s_before;
    __syncthreads();
    if (threadIdx.x == 0) s_mine = s_before = 0;
    __syncthreads();
    uint32_t before = 0;
    for_entries(in, all, kNoTarget, [&](const uint4& q) {
        const uint32_t j = q.z - j0, mine = __ballot_sync(0xffffffffu, j < nw);
        before += q.z < j0;
        if (mine == 0) return;
        uint32_t p = 0;
        if ((threadIdx.x & 31) == 0) p = atomicAdd(&s_mine, __popc(mine));
        p = __shfl_sync(0xffffffffu, p, 0) + __popc(mine & ((1u << (threadIdx.x & 31)) - 1u));
        if (j < nw && p < kBlockEvents) s_in[p] = make_uint4(q.x, q.y, j, 0u);
    });
    before = __reduce_add_sync(0xffffffffu, before);
    if ((threadIdx.x & 31) == 0 && before) atomicAdd(&s_before, before);
    __syncthreads();
    return make_uint2(s_mine, s_before);
}

// Everything a tick does at its targets, a block per bucket of consecutive
// targets (a bucket's events are one contiguous run of grp_tmp), or per part of
// a bucket that is too large for a block (part_shift), whose entries the block
// picks out of the bucket's:
//
//   1. the bucket's entries come in with one bulk copy (bounded mbarrier
//      wait) while the targets' parameters are loaded; every thread holds its
//      share in registers;
//   2. a counting sort by target into shared memory, then each event's place
//      in due order is its rank among its target's events; the same
//      comparison finds the synapses with several events;
//   3. a thread per event, the warps taking 32 at a time as they get free: its
//      synapse record (one 64-byte read and write, random), pre-spike STDP,
//      spike code, the weight it delivers; a synapse with several events has
//      one thread do them all (together with its like, so that the others'
//      warps need not wait); beside them the neurons' temporal patterns, a
//      thread per target;
//   4. a thread per target: the neuron's physics over its events in due
//      order, exact because everything an event reads or writes belongs to its
//      target; post-spike STDP of a fire is applied lazily to synapses with
//      later events in the tick and in bulk by k_post for the rest.
//
// The records' DRAM traffic (a 128-byte line in and one out per event: 39 ps
// an event at the measured copy bandwidth) is the floor; the kernel is bound by
// the length of its instruction streams before that (about 1,080 warp
// instructions per 32 events, 35 % of the issue slots, 20 warps per SM at 96
// registers; more blocks with fewer registers, and records loaded one round
// ahead, measured the same or slower).  As four kernels (bucket sort, synapse
// events by a warp per target, walk, temporal pattern) the events' words and
// inputs went through global memory between them, 20 of 32 lanes idled, and
// each waited for the slowest block of the one before.  Sum of the four ->
// this one, per tick: 309 -> 187 us (2.5 M events, 200,000 neurons), 82 -> 32
// us (250,000 events, 20,000 neurons).
//
// kInline: every synapse's learned code pattern is in its record
// (inline_code_pattern holds for every target).
template <bool kInline>
__global__ void __launch_bounds__(kEventThreads, SNNGB_EVENTS_MIN_BLOCKS) k_events(const __grid_constant__ Engine e) {
    tick_enter();
    extern __shared__ __align__(128) unsigned char s_raw[];  // EventsLayout
    __shared__ __align__(8) unsigned long long s_bar;
    __shared__ float s_wt[kEventThreads / 32][32];  // per warp: weights of the events redone after a fire
    __shared__ uint32_t s_repeats;                  // synapses with several events
    __shared__ uint32_t s_next;                     // next task of the events phase
    __shared__ Refire s_refire[kEventThreads];      // targets that go on after their first fire
    __shared__ uint32_t s_refires;
    __shared__ uint32_t s_longest;                  // events of the busiest target
    const uint32_t width = 1u << e.bucket_shift;
    // the staged entries (16 bytes per event); once they are in registers, the
    // words grouped by target (8) and the words in due order (8); once those
    // are there, w and bits in place of the grouped words
    uint4* s_in = reinterpret_cast<uint4*>(s_raw);
    unsigned long long* s_word = reinterpret_cast<unsigned long long*>(s_raw);
    const SharedEvents ev{s_word + kBlockEvents, reinterpret_cast<float*>(s_raw), s_raw + 4 * kBlockEvents};
    uint16_t* s_tgt = reinterpret_cast<uint16_t*>(s_raw + sizeof(BucketEntry) * kBlockEvents);
    uint16_t* s_list = s_tgt + kBlockEvents;  // first events of the synapses with several
    TargetParam* s_par = reinterpret_cast<TargetParam*>(s_list + kBlockEvents);
    const bool keep_params = width <= kSharedParams;
    uint32_t* s_seg = reinterpret_cast<uint32_t*>(s_par + (keep_params ? width : 0u));  // [width + 2]
    const BucketSpace space{s_word, s_tgt, s_list, s_seg, &s_wt[0][0], s_refire, &s_repeats, &s_next, &s_refires,
                            nullptr, nullptr, nullptr};
    const uint32_t t = e.ts->tick;
    const int stdp = e.ts->stdp_enabled;
    const int temporal = e.ts->temporal_enabled;
    if (threadIdx.x == 0) mbar_init(&s_bar, 1);
    __syncthreads();
    uint32_t parity = 0;
    bool staging = true;  // false after a copy outlived its wait: no more copies
    // the parts of the large buckets, then the buckets
    const uint32_t parts = e.ts->n_parts, part_events = e.ts->part_events;
    for (uint32_t w = blockIdx.x; w < parts + e.nbuckets; w += gridDim.x) {
        const bool part = w < parts;
        const uint32_t item = part ? e.parts[w] : w - parts, b = item & ((1u << kPartShift) - 1u);
        uint32_t lo = e.bstart[b], m = e.bstart[b + 1] - lo;
        uint32_t n0 = b << e.bucket_shift;
        uint32_t nw = e.N - n0 < width ? e.N - n0 : width;
        const uint4* in = reinterpret_cast<const uint4*>(e.grp_tmp) + lo;
        const uint32_t all = m;
        uint32_t j0 = 0;  // the part's first target
        if (part) {
            const uint32_t range = ((nw - 1) >> part_shift(all, part_events, e.bucket_shift)) + 1;
            j0 = (item >> kPartShift) * range;
            if (j0 >= nw) continue;  // past the last target
            nw = min(nw - j0, range);
            n0 += j0;
            const uint2 got = pick_part(in, all, j0, nw, s_in);
            m = got.x;
            lo += got.y;
        } else {
            if (threadIdx.x == 0) {  // the bucket's total and cursor start at zero next tick
                e.btot[b] = 0;
                e.bcur[b] = 0;
            }
            if (m > kBlockEvents) continue;  // its parts do it
        }
        if (m == 0) {
            if (e.multi_refs)
                for (uint32_t j = threadIdx.x; j < nw; j += kEventThreads) e.seg_start[n0 + j] = lo;
            continue;
        }
        bool small = m <= kBlockEvents;
        const bool staged = !part && staging;
        if (staged && threadIdx.x == 0) bulk_load(s_raw, in, m * static_cast<uint32_t>(sizeof(BucketEntry)), &s_bar);
        const BucketParams<false> par{s_par, e.nparam, n0, keep_params};
        if (keep_params)
            for (uint32_t j = threadIdx.x; j < nw; j += kEventThreads) s_par[j] = load_param(e.nparam + n0 + j);
        for (uint32_t j = threadIdx.x; j < nw; j += kEventThreads) {
            prefetch_l2(e.nrec + n0 + j);
            prefetch_l2(e.ntp + n0 + j);
        }
        for (uint32_t j = threadIdx.x; j <= nw; j += kEventThreads) s_seg[j] = 0;
        bool ready = true;
        if (staged && threadIdx.x == 0) ready = mbar_wait(&s_bar, parity, e.stage_wait_ns);
        ready = __syncthreads_and(ready);
        if (staged) {
            if (!ready) {
                // the copy is still in flight: wait for it once more before
                // its buffer is used or the block exits
                bool drained = true;
                if (threadIdx.x == 0) {
                    raise_status(e, kStatusStageTimeout);
                    drained = mbar_wait(&s_bar, parity, kDrainWaitNs);
                }
                if (!__syncthreads_and(drained)) return;
                staging = false;
            }
            parity ^= 1u;
        }
        if (!part && !(staged && ready)) {  // no copy: the entries come in directly
            for (uint32_t i = threadIdx.x; i < m; i += kEventThreads) s_in[i] = in[i];
            __syncthreads();
        }
        if (small) {
            // counting sort by target: an entry's place among its target's is
            // the count before it
            uint2 v[kBlockPerThread];
            uint32_t at[kBlockPerThread];  // target | place << 16
#pragma unroll
            for (uint32_t k = 0; k < kBlockPerThread; ++k) {
                const uint32_t i = threadIdx.x + k * kEventThreads;
                at[k] = 0xFFFFu;
                if (i >= m) continue;
                const uint4 q = s_in[i];
                if (!(q.x & kExternalBit)) prefetch_l2(e.syn + q.y);
                v[k] = make_uint2(q.x, q.y);
                if (q.z < nw) at[k] = q.z | (atomicAdd(&s_seg[q.z + 1], 1u) << 16);
            }
            __syncthreads();
            // exclusive scan of the counts by one warp (a bucket has 32 to 64
            // targets unless the network is huge): s_seg[j + 1], s_seg[j + 2]
            // become the first and the end of target j's events
            if (threadIdx.x < 32) {
                uint32_t busy = 0, longest = 0, run = 0;
                for (uint32_t j0 = 0; j0 < nw; j0 += 32) {
                    const uint32_t j = j0 + threadIdx.x, c = j < nw ? s_seg[j + 1] : 0u;
                    const uint32_t incl = warp_incl_scan(c);
                    if (j < nw) s_seg[j + 1] = run + incl - c;
                    run += __shfl_sync(0xffffffffu, incl, 31);
                    busy += c != 0;
                    longest = max(longest, c);
                }
                busy = __reduce_add_sync(0xffffffffu, busy);
                longest = __reduce_max_sync(0xffffffffu, longest);
                if (threadIdx.x == 0) {
                    if (busy) atomicAdd(&e.ts->n_touched, busy);
                    s_seg[nw + 1] = run;
                    s_repeats = 0;
                    s_next = 0;
                    s_longest = longest;
                }
            }
            __syncthreads();
            small = s_longest <= kRankEvents;
            if (small) {
                const uint32_t total = s_seg[nw + 1];
#pragma unroll
                for (uint32_t k = 0; k < kBlockPerThread; ++k) {
                    const uint32_t j = at[k] & 0xFFFFu;
                    if (j == 0xFFFFu) continue;
                    const uint32_t p = s_seg[j + 1] + (at[k] >> 16);
                    s_word[p] = (static_cast<unsigned long long>(v[k].y) << 32) | __funnelshift_l(v[k].x, v[k].x, 1);
                    s_tgt[p] = static_cast<uint16_t>(j);
                }
                __syncthreads();
                bucket_events<kInline, kEventThreads, false>(e, space, ev, total, lo, n0, nw, par, t, stdp, temporal,
                                                             EngineFires{e});
            }
        }
        if (!small) {
            bucket_in_global<kInline>(e, in, all, j0, lo, n0, nw, s_seg, par, t, stdp, temporal, &s_wt[0][0], s_refire,
                                      &s_refires, reinterpret_cast<uint32_t*>(s_raw));
            __syncthreads();
            if (m > kBlockEvents) {
                uint32_t busy = 0;
                for (uint32_t j = threadIdx.x; j < nw; j += kEventThreads) busy += s_seg[j + 1] != s_seg[j];
                busy = __reduce_add_sync(0xffffffffu, busy);
                if ((threadIdx.x & 31) == 0 && busy) atomicAdd(&e.ts->n_touched, busy);
            }
            if (e.multi_refs)
                for (uint32_t j = threadIdx.x; j < nw; j += kEventThreads) e.seg_start[n0 + j] = lo + s_seg[j];
        }
        __syncthreads();
    }
}

// The temporal pattern of a touched target that keeps one reference pattern
// (SynapseDendriteProcessor.cpp:294-316), once per tick for all its k events.
// It reads and writes only the neuron's temporal fields.
__device__ __noinline__ void temporal_target(const Engine& e, uint32_t n, uint32_t k, uint32_t t, int temporal) {
    const NeuronParam p = e.nparam[n];
    NeuronRec* rec = e.nrec + n;
    const NeuronTp q = e.ntp[n];
    NState s;
    s.match_count = rec->match_count;
    s.ws = rec->ws;
    s.len = rec->len;
    s.flags = q.last_match << 8;
    s.cn = q.cn;
    s.nruns = q.nruns;
    s.ref_head = q.ref_head;
    s.ref_count = q.ref_count;
    s.ring_head = q.ring_head;
    s.ring_used = q.ring_used;
    s.last_run = s.nruns > 0 ? e.cand[p.cand_base + s.nruns - 1] : 0ull;
    s.one = RefMeta{};
    if (s.ref_count > 0) s.one = e.refmeta[p.meta_base];
    s.snap_pending = false;
    temporal_tick(s, p, t, e, temporal, k);
    if (s.nruns > 0) e.cand[p.cand_base + s.nruns - 1] = s.last_run;
    if (s.ref_count > 0) e.refmeta[p.meta_base] = s.one;
    if (s.snap_pending) {
        // runs 0 .. snap_nruns-2 are final in cand; the last one was saved
        unsigned long long* ring = e.ring + p.ring_base;
        const unsigned long long* cand = e.cand + p.cand_base;
        for (uint32_t j = 0; j + 1 < s.snap_nruns; ++j) ring[wrap_add(s.one.start, j, p.ring_cap)] = cand[j];
        ring[wrap_add(s.one.start, s.snap_nruns - 1, p.ring_cap)] = s.snap_last;
    }
    rec->match_count = s.match_count;
    rec->ws = s.ws;
    rec->len = s.len;
    NeuronTp wq;
    wq.cn = s.cn;
    wq.nruns = s.nruns;
    wq.ref_head = s.ref_head;
    wq.ref_count = s.ref_count;
    wq.ring_head = s.ring_head;
    wq.ring_used = s.ring_used;
    wq.last_match = (s.flags >> 8) & 1u;
    e.ntp[n] = wq;
}

// The temporal pattern of the touched targets that keep several reference
// patterns: kGroup lanes per target, a pattern per lane and round, so that
// the patterns' sums and comparisons (up to 65,535 of them, each a 48-byte
// entry) are in flight together.  A thread per target walked them one after
// the other: 12 us of a 34-us tick with 2 patterns per neuron on a
// 1,000-neuron network, and 30 us more with 43.  Runs after k_events, beside
// the fire ordering, so it takes the tick from post_tick.
template <int kGroup>
__device__ __forceinline__ void temporal_group(const Engine& e, uint32_t n, uint32_t k, uint32_t t, int enabled) {
    const uint32_t sub = threadIdx.x & (kGroup - 1);
    const uint32_t mask = kGroup == 32 ? 0xffffffffu : ((1u << (kGroup & 31)) - 1u) << (threadIdx.x & 31 & ~(kGroup - 1));
    const NeuronParam p = e.nparam[n];
    NeuronRec* rec = e.nrec + n;
    NeuronTp q = e.ntp[n];
    if (!enabled) {
        __syncwarp(mask);
        if (sub == 0) e.ntp[n].last_match = 0;
        return;
    }
    uint32_t match_count = rec->match_count, ws = rec->ws, len = rec->len;
    unsigned long long* cand = e.cand + p.cand_base;
    RefMeta* meta = e.refmeta + p.meta_base;
    unsigned long long* ring = e.ring + p.ring_base;
    unsigned long long last_run = q.nruns > 0 ? cand[q.nruns - 1] : 0ull;
    __syncwarp(mask);  // the group has read its state
    auto ref = [&](uint32_t r) -> RefMeta& { return meta[wrap_add(q.ref_head, r, p.max_refs)]; };
    if (len == 0 || t - ws > p.window) {
        ws = t;
        len = 0;
        q.nruns = 0;
        q.cn = 0;
        for (uint32_t r = sub; r < q.ref_count; r += kGroup) {
            RefMeta& m = ref(r);
            m.dot = 0;
            m.rn = 0;
            m.cn = 0;
            m.cur_run = 0;
            m.cur_pos = 0;
            m.match = 2;
        }
    }
    const uint32_t o = t - ws;
    const uint32_t oo = o * o;
    const bool always = 0.0f >= p.similarity;
    for (uint32_t j = 0; j < k; ++j) {
        // one append, and every pattern's comparison with the longer
        // window; `frozen`: no pattern takes part in a further one
        const bool grow = q.nruns > 0 && run_value(last_run) == o;
        if (grow) {
            last_run += (1ull << 16);
        } else {
            if (q.nruns > p.window) {  // cannot happen: at most window+1 distinct offsets
                if (sub == 0) raise_status(e, kStatusRunOverflow);
                break;
            }
            if (sub == 0 && q.nruns > 0) cand[q.nruns - 1] = last_run;
            last_run = static_cast<unsigned long long>(o) | (1ull << 16);
            q.nruns += 1;
        }
        len += 1;
        q.cn += oo;
        bool match = always && q.ref_count > 0 && len >= 2;
        bool frozen = true;
        for (uint32_t r0 = 0; r0 < q.ref_count; r0 += kGroup) {
            bool hit = false, done = true;
            if (r0 + sub < q.ref_count) {
                RefMeta& m = ref(r0 + sub);
                const uint32_t mlen = m.len;
                uint32_t state = m.match;
                done = len >= mlen;
                const bool advance = len <= mlen;
                if (advance || (state == 2 && !match && len >= 2)) {
                    RefMeta x = m;
                    if (advance) {
                        const unsigned long long run = ring[wrap_add(x.start, x.cur_run, p.ring_cap)];
                        const uint32_t v = run_value(run);
                        if (++x.cur_pos == run_count(run)) {
                            x.cur_run += 1;
                            x.cur_pos = 0;
                        }
                        x.dot += v * o;  // 16-bit values: 32-bit products
                        x.rn += v * v;
                        x.cn += oo;
                        x.match = 2;
                    }
                    if (!match && len >= 2) x.match = cos_ge(x.dot, x.rn, x.cn, p.similarity) ? 1 : 0;
                    state = x.match;
                    m = x;
                }
                hit = state == 1;
            }
            match = __any_sync(mask, hit && len >= 2) || match;
            frozen = __all_sync(mask, done) && frozen;
        }
        if (match) {
            q.last_match = 1;
            match_count += 1;
            if (frozen) {
                // the remaining appends change no pattern's sums: they match too
                const uint32_t rest = k - j - 1;
                last_run += static_cast<unsigned long long>(rest) << 16;
                len += rest;
                q.cn += static_cast<unsigned long long>(oo) * rest;
                match_count += rest;
                break;
            }
            continue;
        }
        q.last_match = 0;
        if (len < 2) continue;
        // learn_pattern (:31-41): FIFO with max_reference_patterns entries
        if (q.ref_count >= p.max_refs) {
            q.ring_used -= ref(0).nruns;
            __syncwarp(mask);
            q.ref_head = wrap_add(q.ref_head, 1, p.max_refs);
            q.ref_count -= 1;
        }
        if (q.ring_used + q.nruns > p.ring_cap) {
            if (sub == 0) raise_status(e, kStatusRingOverflow);
            break;
        }
        if (sub == 0) cand[q.nruns - 1] = last_run;
        __syncwarp(mask);
        for (uint32_t i = sub; i < q.nruns; i += kGroup) ring[wrap_add(q.ring_head, i, p.ring_cap)] = cand[i];
        if (sub == 0) {
            RefMeta x;
            x.dot = x.rn = x.cn = q.cn;
            x.start = q.ring_head;
            x.nruns = q.nruns;
            x.len = len;
            x.cur_run = 0;
            x.cur_pos = 0;
            x.match = 2;
            ref(q.ref_count) = x;
        }
        q.ring_head = wrap_add(q.ring_head, q.nruns, p.ring_cap);
        q.ring_used += q.nruns;
        q.ref_count += 1;
        __syncwarp(mask);
    }
    if (sub == 0) {
        if (q.nruns > 0) cand[q.nruns - 1] = last_run;
        rec->match_count = match_count;
        rec->ws = ws;
        rec->len = len;
        e.ntp[n] = q;
    }
    __syncwarp(mask);
}

template <int kGroup>
__global__ void __launch_bounds__(kThreads) k_temporal(Engine e) {
    const uint32_t t = e.ts->post_tick;
    const int enabled = e.ts->temporal_enabled;
    const uint32_t groups = gridDim.x * blockDim.x / kGroup;
    for (uint32_t n = (blockIdx.x * blockDim.x + threadIdx.x) / kGroup; n < e.N; n += groups) {
        const uint32_t k = e.seg_start[n + 1] - e.seg_start[n];
        if (k > 0 && e.nparam[n].max_refs != 1)  // (1: done by k_events)
            temporal_group<kGroup>(e, n, k, t, enabled);
    }
}

__global__ void k_init_syn(SynAB* syn, const SynA* a, unsigned long long S) {
    for (unsigned long long i = blockIdx.x * static_cast<unsigned long long>(blockDim.x) + threadIdx.x; i < S;
         i += static_cast<unsigned long long>(gridDim.x) * blockDim.x) {
        SynAB r;
        r.a = a[i];
        r.b = SynB{};
        r.b.flags = static_cast<uint8_t>(((r.a.meta >> kMetaExpectedShift) & 15u) << 4);
        syn[i] = r;
    }
}

// Post-spike STDP over the incoming rows of every target that fired
// (NetworkPropagator.cpp:95-102), one block per fired target, coalesced over
// the target-major row.  Runs on the side stream beside k_fire_list ..
// k_expand (none of which touches synapse records), so it reads the tick
// from post_tick, not from the tick counter k_fire_count advances.
// Bound by the latency of the records' reads: each thread has four on their
// way before it updates the first, as 32-byte halves (one request a half).
// Alone 12.9 -> 10.2 us at 20,000 targets x 1,000 rows; beside the fire
// ordering it takes a tick of 2e8 synapses from 341 to 334 us.
constexpr uint32_t kPostInFlight = 4;  // records each thread has on their way

__global__ void __launch_bounds__(kThreads) k_post(const __grid_constant__ Engine e) {
    const uint32_t t = e.ts->post_tick;
    const uint32_t nf = e.ts->n_fired_targets;
    const int stdp = e.ts->stdp_enabled;
    for (uint32_t j = blockIdx.x; j < nf; j += gridDim.x) {
        const uint32_t n = e.fired_tgt[j];
        const uint32_t fires = e.fired_cnt[j];
        if (fires >= 0x10000u) {
            if (threadIdx.x == 0) raise_status(e, kStatusPostCountOverflow);
            continue;
        }
        const unsigned long long en = e.in_ptr[n + 1];
        for (unsigned long long tm = e.in_ptr[n] + threadIdx.x; tm < en; tm += kPostInFlight * kThreads) {
            SynA a[kPostInFlight];
#pragma unroll
            for (uint32_t u = 0; u < kPostInFlight; ++u)
                if (tm + u * kThreads < en) a[u] = load_half(&e.syn[tm + u * kThreads].a);
#pragma unroll
            for (uint32_t u = 0; u < kPostInFlight; ++u)
                if (tm + u * kThreads < en && post_catch_up(a[u], t, fires, e, stdp, e.tab.ltp))
                    store_half(&e.syn[tm + u * kThreads].a, a[u]);
        }
    }
}

// Fires in due order, one thread per bitmap word (a tile is kThreads words).
// k_events counted every tile's fires, so a block finds the first rank of
// its tile by adding the counts of the tiles before it.  A fire's rank r is
// its position in the reference's fire order (due order,
// NetworkPropagator.cpp:80-93); the fire list and the raster are written here
// and the bitmap is cleared.
__global__ void k_fire_list(Engine e) {
    tick_enter();
    const uint32_t t = e.ts->tick;
    const uint32_t words = (e.ts->n_due + 31) / 32;
    const uint32_t tiles = (words + kThreads - 1) / kThreads;
    const unsigned long long raster0 = e.ts->raster_count;
    uint32_t part = 0, base = 0;
    for (uint32_t i = threadIdx.x; i < blockIdx.x && i < tiles; i += blockDim.x) part += __ldcg(e.fire_tile + i);
    block_excl_scan(part, &base);
    for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const uint32_t w = tile * kThreads + threadIdx.x;
        uint32_t bits = w < words ? e.fire_bits[w] : 0u;
        uint32_t r = base + block_excl_scan(__popc(bits), nullptr);
        if (bits) e.fire_bits[w] = 0;
        while (bits) {
            const uint32_t bit = __ffs(bits) - 1;
            bits &= bits - 1;
            const uint32_t n = e.fire_at[w * 32 + bit];
            if (r < e.fire_cap) e.fire_list[r] = n;
            if (e.raster_cap > 0) {
                const unsigned long long pos = raster0 + r;
                if (pos < e.raster_cap) {
                    e.raster[2 * pos] = t;
                    e.raster[2 * pos + 1] = n;
                }
            }
            r += 1;
        }
        // the base of this block's next tile
        part = 0;
        for (uint32_t i = tile + threadIdx.x; i < tile + gridDim.x && i < tiles; i += blockDim.x)
            part += __ldcg(e.fire_tile + i);
        uint32_t step;
        block_excl_scan(part, &step);
        base += step;
    }
}

// Events per (expansion block of kExpandFires fires, delay class), one warp
// per fire and one lane per class.  The last block turns the counts into wheel positions
// (exclusive scan over blocks per class, appended behind each delivery slot's
// current contents) and finishes the tick.
__global__ void __launch_bounds__(kFireCountThreads, 1) k_fire_count(Engine e) {
    tick_enter();
    const uint32_t t = e.ts->tick;
    // the tick's fire count: the sum of k_events' per-tile counts
    const uint32_t tiles = ((e.ts->n_due + 31) / 32 + kThreads - 1) / kThreads;
    __shared__ uint32_t s_nf;
    if (threadIdx.x == 0) s_nf = 0;
    __syncthreads();
    uint32_t part = 0;
    for (uint32_t i = threadIdx.x; i < tiles; i += blockDim.x) part += __ldcg(e.fire_tile + i);
    part = __reduce_add_sync(0xffffffffu, part);
    if ((threadIdx.x & 31) == 0 && part) atomicAdd(&s_nf, part);
    __syncthreads();
    const uint32_t nfires = s_nf;
    const uint32_t nf = nfires < e.fire_cap ? nfires : e.fire_cap;
    const uint32_t D = e.D;
    // one warp per fire, one lane per delay class
    const uint32_t lane0 = threadIdx.x & 31;
    const uint32_t nwarps = gridDim.x * (blockDim.x / 32);
    for (uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < nf; r += nwarps) {
        const uint32_t* row = e.pre_off + static_cast<size_t>(e.fire_list[r]) * (D + 1);
        uint32_t* xs = e.xsum + static_cast<size_t>(r / kExpandFires) * D;
        for (uint32_t d = lane0; d < D; d += 32) {
            const uint32_t c = row[d + 1] - row[d];
            if (c) atomicAdd(xs + d, c);
        }
    }
    if (!last_block(&e.ts->done_fire_list)) return;
    for (uint32_t i = threadIdx.x; i < tiles; i += blockDim.x) e.fire_tile[i] = 0;  // zero for the next tick
    if (nfires > e.fire_cap && threadIdx.x == 0) raise_status(e, kStatusFireOverflow);
    const uint32_t blocks = (nf + kExpandFires - 1) / kExpandFires;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // one warp per class; lane i scans a contiguous run of expansion blocks
    // (its loads are independent, so they are all in flight at once), then
    // the lanes' totals are scanned across the warp
    const uint32_t per = (blocks + 31) / 32;
    const uint32_t b0 = lane * per < blocks ? lane * per : blocks;
    const uint32_t b1 = b0 + per < blocks ? b0 + per : blocks;
    for (uint32_t d = warp; d < D; d += blockDim.x / 32) {
        const uint32_t slot = (t + e.cls_delta[d]) & e.wmask;
        const uint32_t start = e.slot_count[slot];
        uint32_t sum = 0;
        for (uint32_t b = b0; b < b1; ++b) sum += __ldcg(e.xsum + static_cast<size_t>(b) * D + d);
        const uint32_t incl = warp_incl_scan(sum);
        const uint32_t carry = __shfl_sync(0xffffffffu, incl, 31);
        unsigned long long pos = static_cast<unsigned long long>(slot) * e.slot_cap + start + (incl - sum);
        for (uint32_t b = b0; b < b1; ++b) {
            e.xdst[static_cast<size_t>(b) * D + d] = pos;
            pos += __ldcg(e.xsum + static_cast<size_t>(b) * D + d);
        }
        if (lane == 0) {
            if (static_cast<unsigned long long>(start) + carry > e.slot_cap) {
                raise_status(e, kStatusSlotOverflow);
                e.xdst_ok[d] = 0;
            } else {
                e.xdst_ok[d] = 1;
                e.slot_count[slot] = start + carry;
            }
        }
    }
    // the class counts back to zero for the next tick, once every warp has
    // read its classes
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < blocks * D; i += blockDim.x) e.xsum[i] = 0;
    if (threadIdx.x == 0) {
        TickState* ts = e.ts;
        ts->n_fires = nfires;
        const uint32_t due = ts->n_due;
        const unsigned long long raster0 = ts->raster_count;
        ts->delivered += due;
        ts->fired += nfires;
        ts->touched_total += ts->n_touched;
        if (due > ts->max_slot_events) ts->max_slot_events = due;
        if (e.raster_cap > 0) {
            if (raster0 + nfires > e.raster_cap) raise_status(e, kStatusRasterOverflow);
            ts->raster_count = raster0 + nfires;
        }
        ts->expand_fires = nf;
        e.slot_count[t & e.wmask] = 0;
        ts->n_touched = 0;
        ts->tick = t + 1;
    }
}

// Spike-code offset expansion (NetworkPropagator.cpp:104-130): one block per
// fire, one warp per delay class.  A fire's events of one class are
// contiguous in its pre-expanded list and go to one contiguous range of their
// delivery slot: the range k_fire_count reserved for the fire's expansion
// block, behind the block's earlier fires.  So the wheel ends up in exactly
// the reference's scheduling order.
__global__ void __launch_bounds__(kThreads) k_expand(Engine e) {
    tick_enter();
    __shared__ uint32_t s_rows[kExpandFires][kMaxClasses + 1];
    __shared__ unsigned long long s_dst[kMaxClasses];
    __shared__ uint8_t s_ok[kMaxClasses];  // the class's slot had room
    __shared__ unsigned long long s_base;
    const uint32_t nf = e.ts->expand_fires;
    const uint32_t D = e.D;
    for (uint32_t r = blockIdx.x; r < nf; r += gridDim.x) {
        const uint32_t first = r - r % kExpandFires;
        const uint32_t m = r - first + 1;  // fires first .. r of the expansion block
        // everything the copies depend on, fetched together: the class rows of
        // the block's fires, the block's destinations, the fire's event list
        for (uint32_t i = threadIdx.x; i < m * (D + 1); i += blockDim.x) {
            const uint32_t q = i / (D + 1), d = i - q * (D + 1);
            s_rows[q][d] = e.pre_off[static_cast<size_t>(e.fire_list[first + q]) * (D + 1) + d];
        }
        for (uint32_t d = threadIdx.x; d < D; d += blockDim.x) {
            s_ok[d] = e.xdst_ok[d] ? 1 : 0;
            s_dst[d] = s_ok[d] ? __ldcg(e.xdst + static_cast<size_t>(r / kExpandFires) * D + d) : 0ull;
        }
        if (threadIdx.x == 0) s_base = e.pre_base[e.fire_list[r]];
        __syncthreads();
        const uint32_t* row = s_rows[m - 1];
        // this fire's place in each class: the block's destination behind
        // the class's events of the block's earlier fires
        for (uint32_t d = threadIdx.x; d < D; d += blockDim.x) {
            uint32_t before = 0;
            for (uint32_t q = 0; q + 1 < m; ++q) before += s_rows[q][d + 1] - s_rows[q][d];
            // then event k of class d goes to s_dst[d] + k (64-bit wrap-around
            // arithmetic: exact once k >= row[d] is added back)
            s_dst[d] = s_dst[d] + static_cast<unsigned long long>(before) - static_cast<unsigned long long>(row[d]);
        }
        __syncthreads();
        // every event by its own thread (consecutive threads, consecutive
        // events: coalesced within a class); its class by binary search of
        // the fire's class offsets
        const unsigned long long* src = e.pre_ev + s_base;
        const uint32_t k0 = row[0], k1 = row[D];
        auto class_of = [&](uint32_t k) {
            uint32_t lo = 0, hi = D;  // row[lo] <= k < row[hi]
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) >> 1;
                if (row[mid] <= k) {
                    lo = mid;
                } else {
                    hi = mid;
                }
            }
            return lo;
        };
        for (uint32_t k = k0 + threadIdx.x; k < k1; k += 4 * blockDim.x) {
            unsigned long long v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t kk = k + u * blockDim.x;
                v[u] = kk < k1 ? src[kk] : 0ull;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t kk = k + u * blockDim.x;
                if (kk >= k1) continue;
                const uint32_t d = class_of(kk);
                if (s_ok[d]) e.wheel[s_dst[d] + kk] = v[u];
            }
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// small networks: whole ticks in one cluster of blocks
// ---------------------------------------------------------------------------

constexpr int kSmallThreads = 512;
constexpr uint32_t kSmallPlaces = 4096;  // wheel positions a block keeps (fires x classes) between finding and using them
constexpr uint32_t kSmallGroups = 64;    // shares of a tick's fires whose events are summed side by side

constexpr size_t kSmallA = (kSmallEvents + 2) * sizeof(unsigned long long);  // staged due list, words in due order; then fires
constexpr size_t kSmallB = kSmallEvents * sizeof(unsigned long long);        // words by target; then w and bits
constexpr size_t kSmallOffTgt = kSmallA + kSmallB;
constexpr size_t kSmallOffList = kSmallOffTgt + kSmallEvents * sizeof(uint16_t);
constexpr size_t kSmallOffSeg = kSmallOffList + kSmallEvents * sizeof(uint16_t);
constexpr size_t kSmallOffSlot = kSmallOffSeg + (kSmallTargets + 2) * sizeof(uint32_t);
constexpr size_t kSmallSmem = kSmallOffSlot + kSmallSlots * sizeof(uint32_t);
// The list of the targets with events takes the end of the words' memory, where
// a block has no more than this many events (8 KB more shared memory, which L1
// then lacks, took a tick of 7,000 events from 41 to 44 us).
constexpr size_t kSmallOffTouched = kSmallOffTgt - kSmallTargets * sizeof(uint16_t);
constexpr uint32_t kSmallListed = (kSmallOffTouched - kSmallA) / sizeof(unsigned long long);
static_assert(kSmallEvents * (sizeof(float) + 1) <= kSmallOffTouched - kSmallA, "w and bits before the list");
static_assert((kSmallEvents + kSmallPlaces) * sizeof(uint32_t) <= kSmallA, "fires and places");
static_assert(kSmallTargets <= kSmallEvents / 2, "fired targets in the lists' place, targets in their second half");
static_assert(kSmallTargets < kSharedSynapse, "targets of a block");

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// Orders this thread's generic accesses with bulk copies (the async proxy).
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async;" ::: "memory"); }

// A block's fires of the tick (for every block of the cluster) and its fired
// targets.
struct SmallFires {
    uint2* fires;        // (due position, neuron) in global memory
    uint32_t* targets;   // target within the block << 16 | fires
    uint32_t *n_fires, *n_targets;
    __device__ __forceinline__ void fire(uint32_t n, uint32_t due) const { fires[atomicAdd(n_fires, 1u)] = make_uint2(due, n); }
    __device__ __forceinline__ void target(uint32_t n, uint32_t f) const {
        targets[atomicAdd(n_targets, 1u)] = small_place(n) << 16 | f;
    }
};

// Ticks ts->tick .. end-1 of a small network, kSmallBlocks blocks in one
// cluster, each with an eighth of the targets (small_block).  Per tick a block reads
// the whole due list into shared memory and groups the events of its own
// targets (no pass over the other blocks' data), does what k_events does with
// them, and the post-spike STDP of its fired targets; the blocks exchange
// their fires through global memory and a cluster barrier; every block then
// orders all of them (a bitmap of due positions), finds their events' places
// in the wheel, and copies its share; a second barrier ends the tick.  Every
// block keeps the wheel's slot counts and changes them alike.
//
// Bound by the latency of these steps (a global read is about 0.4 us, and the
// barriers' acquires empty L1).  As the tick's seven kernels a tick of a
// 1,000-neuron network with 935 events took 28.8 us, four or five of them per
// kernel boundary; here 18.8: 3.0 due list and grouping, 8.1 synapses, patterns
// and walk, 1.4 post-spike STDP, 4.5 fires and their events, 1.5 barriers.  A
// burst of 27,648 relayed events over 7 ticks: 42 -> 35 us a tick.  Eight blocks (a portable cluster) of 512
// threads; a tick with more than `limit` events due (kSmallEvents, or an
// eighth of a wheel slot: the scratch is shared out), a target with more than
// kRankEvents of them, or ticks that lost too much (kSmallDebt) end the run of
// this kernel (ts->small_stop: the first tick left to the other kernels): there
// the whole GPU is quicker.  The first block to set small_stop decides for all (a
// later and larger value would be seen by some blocks only).
template <bool kInline>
__global__ void __cluster_dims__(kSmallBlocks, 1, 1) __launch_bounds__(kSmallThreads, 1)
    k_small(const __grid_constant__ Engine e, uint32_t end, uint32_t limit) {
    extern __shared__ __align__(128) unsigned char s_raw[];
    __shared__ __align__(8) unsigned long long s_bar;
    __shared__ float s_wt[kSmallThreads / 32][32];
    __shared__ Refire s_refire[kSmallThreads];
    __shared__ uint32_t s_refires, s_repeats, s_next, s_fires, s_fired, s_multis, s_touches, s_rows, s_widest;
    __shared__ uint32_t s_part[kSmallThreads], s_sum[kMaxClasses], s_start[kMaxClasses], s_slot_of[kMaxClasses];
    __shared__ uint32_t s_done[kMaxClasses];
    __shared__ uint32_t s_bits[kSmallEvents / 32], s_before[kSmallEvents / 32], s_count[kSmallBlocks];
    unsigned long long* s_due = reinterpret_cast<unsigned long long*>(s_raw);
    unsigned long long* s_word = reinterpret_cast<unsigned long long*>(s_raw + kSmallA);
    uint16_t* s_tgt = reinterpret_cast<uint16_t*>(s_raw + kSmallOffTgt);
    uint16_t* s_list = reinterpret_cast<uint16_t*>(s_raw + kSmallOffList);
    uint32_t* s_end = reinterpret_cast<uint32_t*>(s_raw + kSmallOffSeg);  // s_end[j], s_end[j + 1]: first and end of target j
    uint32_t* s_seg = s_end + 1;
    uint32_t* s_slot = reinterpret_cast<uint32_t*>(s_raw + kSmallOffSlot);  // events in each wheel slot
    uint16_t* s_touched = reinterpret_cast<uint16_t*>(s_raw + kSmallOffTouched);  // targets with events
    uint32_t* s_fire = reinterpret_cast<uint32_t*>(s_raw);                  // firing neurons in due order
    uint32_t* s_place = s_fire + kSmallEvents;
    const uint32_t c = blockIdx.x;
    uint32_t t = e.ts->tick;
    // (every block looks before any of them can write to the tick state)
    const bool nothing = e.ts->small_stop != 0 || t >= end;
    __syncwarp();
    cluster_arrive();
    cluster_wait();
    if (nothing) return;
    const int stdp = e.ts->stdp_enabled;
    const int temporal = e.ts->temporal_enabled;
    unsigned long long raster = e.ts->raster_count;
    const uint32_t D = e.D;
    // its targets: whole runs, then what there is of the last one
    const uint32_t whole = e.N / (kSmallChunk * kSmallBlocks) * kSmallChunk, last = small_neuron(c, whole);
    const uint32_t nw = whole + (e.N > last ? min(e.N - last, kSmallChunk) : 0u);
    const BucketParams<true> par{nullptr, e.nparam, c, false};
    const SharedEvents ev{s_due, reinterpret_cast<float*>(s_word), reinterpret_cast<uint8_t*>(s_word) + 4 * kSmallEvents};
    uint2* all_fires = reinterpret_cast<uint2*>(e.evin);  // [block][limit]
    const SmallFires out{all_fires + c * limit, reinterpret_cast<uint32_t*>(s_list), &s_fires, &s_fired};
    // lanes per share of the fires: a lane per class
    uint32_t span = 1;
    while (span < D) span <<= 1;
    const uint32_t groups = min(kSmallGroups, kSmallThreads / span);
    const uint32_t cls = threadIdx.x & (span - 1), group = threadIdx.x / span;
    const uint32_t chunk = D > 0 ? kSmallBlocks * (kSmallPlaces / D) : kSmallEvents;  // fires placed at a time
    for (uint32_t i = threadIdx.x; i < e.W; i += kSmallThreads) s_slot[i] = e.slot_count[i];
    if (threadIdx.x == 0) mbar_init(&s_bar, 1);
    unsigned long long delivered = 0, external = 0, fired = 0, most = 0;
    uint32_t parity = 0;
    bool staging = true;
    uint32_t debt = threadIdx.x == 0 ? e.ts->small_debt[c] : 0u;  // (thread 0 keeps it)
    const uint32_t gain = kSmallGain - e.N / 4 + kSmallClassGain * D;
    __syncthreads();
    for (;;) {
        const uint32_t slot = t & e.wmask, n = s_slot[slot];
        if (n > limit) break;
        // far-future injections that become reachable (as k_bcount)
        uint32_t fb, fe, fslot;
        if (far_range(e, t, fb, fe, fslot)) {
            const uint32_t base = s_slot[fslot];
            const bool fits = static_cast<unsigned long long>(base) + (fe - fb) <= e.slot_cap;
            unsigned long long* dst = e.wheel + static_cast<size_t>(fslot) * e.slot_cap + base;
            if (fits)
                for (uint32_t i = c * kSmallThreads + threadIdx.x; i < fe - fb; i += kSmallBlocks * kSmallThreads)
                    dst[i] = e.far_ev[fb + i];
            __syncthreads();
            if (threadIdx.x == 0) {
                if (fits) {
                    s_slot[fslot] = base + (fe - fb);
                } else if (c == 0) {
                    raise_status(e, kStatusSlotOverflow);
                }
            }
        }
        if (threadIdx.x == 0) s_fires = s_fired = s_repeats = s_next = s_multis = s_touches = s_rows = s_widest = 0;
        if (n > 0) {
            const unsigned long long* due = e.wheel + static_cast<size_t>(slot) * e.slot_cap;
            bool ready = true;
            if (staging && threadIdx.x == 0) {
                proxy_fence();
                bulk_load(s_due, due, ((n + 1) & ~1u) * 8u, &s_bar);
            }
            for (uint32_t j = threadIdx.x; j <= nw; j += kSmallThreads) s_end[j] = 0;
            if (staging && threadIdx.x == 0) ready = mbar_wait(&s_bar, parity, e.stage_wait_ns);
            ready = __syncthreads_and(ready);
            if (staging) {
                if (!ready) {
                    bool drained = true;
                    if (threadIdx.x == 0) {
                        raise_status(e, kStatusStageTimeout);
                        drained = mbar_wait(&s_bar, parity, kDrainWaitNs);
                    }
                    if (!__syncthreads_and(drained)) {
                        // (the cluster's barriers do not wait for threads that have exited)
                        if (threadIdx.x == 0) {
                            e.bcnt[c] = 0;
                            __threadfence();
                        }
                        return;
                    }
                    staging = false;
                }
                parity ^= 1u;
            }
            if (!staging) {
                for (uint32_t i = threadIdx.x; i < n; i += kSmallThreads) s_due[i] = due[i];
                __syncthreads();
            }
            // this block's events, grouped by target: counts, starts, words
            uint32_t ext = 0;
            for (uint32_t i = threadIdx.x; i < n; i += kSmallThreads) {
                const uint32_t lo = static_cast<uint32_t>(s_due[i]);
                const uint32_t tgt = lo & ~kExternalBit;
                ext += lo >> 31;
                if (small_block(tgt) == c) atomicAdd(&s_seg[small_place(tgt)], 1u);
            }
            if (c == 0) external += __reduce_add_sync(0xffffffffu, ext);  // (per warp; lane 0 reports)
            __syncthreads();
            uint32_t busy = 0, longest = 0;
            if (nw <= kSmallThreads) {
                longest = threadIdx.x < nw ? s_seg[threadIdx.x] : 0u;
                busy = longest != 0;
            } else {
                // a thread has several targets: those with events are listed
                // (of 4,096 mostly a few hundred)
                const uint32_t lane = threadIdx.x & 31;
                for (uint32_t j0 = threadIdx.x - lane; j0 < nw; j0 += kSmallThreads) {
                    const uint32_t j = j0 + lane, k = j < nw ? s_seg[j] : 0u;
                    const uint32_t some = __ballot_sync(0xffffffffu, k > 0);
                    longest = max(longest, k);
                    busy += k > 0;
                    uint32_t p = 0;
                    if (lane == 0 && some) p = atomicAdd(&s_touches, __popc(some));
                    p = __shfl_sync(0xffffffffu, p, 0) + __popc(some & ((1u << lane) - 1u));
                    if (k > 0) s_touched[p] = static_cast<uint16_t>(j);
                }
            }
            busy = __reduce_add_sync(0xffffffffu, busy);
            if ((threadIdx.x & 31) == 0 && busy) atomicAdd(&e.ts->touched_total, static_cast<unsigned long long>(busy));
            if (longest > kRankEvents) atomicCAS(&e.ts->small_stop, 0u, t + 1);
            __syncthreads();
            const uint32_t total = block_scan_shared<kSmallThreads>(s_seg, nw);
            const bool listed = nw > kSmallThreads && total <= kSmallListed;
            for (uint32_t i = threadIdx.x; i < n; i += kSmallThreads) {
                const unsigned long long v = s_due[i];
                const uint32_t lo = static_cast<uint32_t>(v), tgt = lo & ~kExternalBit, j = small_place(tgt);
                if (small_block(tgt) != c) continue;
                const uint32_t p = atomicAdd(&s_seg[j], 1u);  // ends at the target's end
                s_word[p] = (v & 0xFFFFFFFF00000000ull) | (i << 1) | (lo >> 31);
                s_tgt[p] = static_cast<uint16_t>(j);
            }
            __syncthreads();
            if (total > 0) {
                const BucketSpace space{s_word,      s_tgt,     s_list,     s_end - 1,  &s_wt[0][0],
                                        s_refire,    &s_repeats, &s_next,   &s_refires, s_list + kSmallEvents / 2,
                                        &s_multis, listed ? s_touched : nullptr};
                bucket_events<kInline, kSmallThreads, true>(e, space, ev, total, c * limit, c, listed ? s_touches : nw, par,
                                                            t, stdp, temporal, out);
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) e.bcnt[c] = s_fires;
        __syncthreads();
        cluster_arrive();
        // meanwhile the post-spike STDP of this block's fired targets (k_post)
        // (a warp per target when there are as many as warps, else the block)
        const bool by_warp = s_fired >= kSmallThreads / 32;
        uint32_t rows = 0;
        for (uint32_t k = by_warp ? threadIdx.x >> 5 : 0u; k < s_fired; k += by_warp ? kSmallThreads / 32 : 1u) {
            const uint32_t f = out.targets[k], tgt = small_neuron(c, f >> 16);
            const unsigned long long first = e.in_ptr[tgt], last = e.in_ptr[tgt + 1];
            const uint32_t me = by_warp ? threadIdx.x & 31 : threadIdx.x;
            if (me == 0) rows += static_cast<uint32_t>(min(last - first, 1ull << 17));
            for (unsigned long long tm = first + me; tm < last; tm += by_warp ? 32 : kSmallThreads) {
                SynA a = e.syn[tm].a;
                if (post_catch_up(a, t, f & 0xFFFFu, e, stdp, e.tab.ltp)) e.syn[tm].a = a;
            }
        }
        if (rows > kSmallThreads / 4) atomicAdd(&s_rows, rows);  // (a few are no loss)
        __syncwarp();
        cluster_wait();
        if (threadIdx.x < kSmallBlocks) s_count[threadIdx.x] = __ldcg(e.bcnt + threadIdx.x);
        __syncthreads();
        uint32_t nf = 0;
        for (uint32_t k = 0; k < kSmallBlocks; ++k) nf += s_count[k];
        if (nf > 0) {
            // all fires in due order: fire i of the blocks' lists, the first
            // one of each thread kept for the second look
            auto load_fire = [&](uint32_t i) {
                uint32_t k = 0;
                while (i >= s_count[k]) i -= s_count[k++];
                return __ldcg(all_fires + k * limit + i);
            };
            const uint32_t words = (n + 31) / 32;
            const uint2 mine = threadIdx.x < nf ? load_fire(threadIdx.x) : make_uint2(0u, 0u);
            for (uint32_t w = threadIdx.x; w < words; w += kSmallThreads) s_bits[w] = 0;
            __syncthreads();
            for (uint32_t i = threadIdx.x; i < nf; i += kSmallThreads) {
                const uint2 x = i < kSmallThreads ? mine : load_fire(i);
                atomicOr(&s_bits[x.x >> 5], 1u << (x.x & 31));
            }
            __syncthreads();
            static_assert(kSmallEvents / 32 <= kSmallThreads, "a thread per bitmap word");
            const uint32_t before =
                block_excl_scan_t<kSmallThreads>(threadIdx.x < words ? __popc(s_bits[threadIdx.x]) : 0u, nullptr);
            if (threadIdx.x < words) s_before[threadIdx.x] = before;
            __syncthreads();
            for (uint32_t i = threadIdx.x; i < nf; i += kSmallThreads) {
                const uint2 x = i < kSmallThreads ? mine : load_fire(i);
                s_fire[s_before[x.x >> 5] + __popc(s_bits[x.x >> 5] & ((1u << (x.x & 31)) - 1u))] = x.y;
            }
            __syncthreads();
            if (c == 0 && e.raster_cap > 0)
                for (uint32_t r = threadIdx.x; r < nf; r += kSmallThreads) {
                    const unsigned long long pos = raster + r;
                    if (pos < e.raster_cap) {
                        e.raster[2 * pos] = t;
                        e.raster[2 * pos + 1] = s_fire[r];
                    }
                }
            // events per class of a share of the fires [f0, f0 + m)
            auto share = [&](uint32_t m, uint32_t& q0, uint32_t& q1) {
                const uint32_t each = (m + groups - 1) / groups;
                q0 = min(m, group * each);
                q1 = group < groups ? min(m, q0 + each) : q0;
            };
            auto events_of = [&](uint32_t r) {
                const uint32_t* row = e.pre_off + static_cast<size_t>(s_fire[r]) * (D + 1);
                return row[cls + 1] - row[cls];
            };
            auto sum_shares = [&](uint32_t f0, uint32_t m) {
                uint32_t q0, q1, sum = 0;
                share(m, q0, q1);
                if (cls < D)
                    for (uint32_t q = q0; q < q1; ++q) sum += events_of(f0 + q);
                s_part[threadIdx.x] = sum;
                __syncthreads();
            };
            // the classes' totals decide whether their slots have room
            sum_shares(0, nf);
            if (threadIdx.x < D) {
                uint32_t sum = 0;
                for (uint32_t g = 0; g < groups; ++g) sum += s_part[g * span + threadIdx.x];
                const uint32_t sl = (t + e.cls_delta[threadIdx.x]) & e.wmask;
                s_slot_of[threadIdx.x] = sl;
                s_start[threadIdx.x] = s_slot[sl];
                s_done[threadIdx.x] = 0;
                const bool fits = static_cast<unsigned long long>(s_slot[sl]) + sum <= e.slot_cap;
                if (!fits && c == 0) raise_status(e, kStatusSlotOverflow);
                s_sum[threadIdx.x] = fits ? sum : 0xFFFFFFFFu;
            }
            __syncthreads();
            for (uint32_t f0 = 0; f0 < nf; f0 += chunk) {
                const uint32_t m = min(chunk, nf - f0);
                if (nf > chunk) sum_shares(f0, m);
                uint32_t q0, q1;
                share(m, q0, q1);
                uint32_t pos = 0, sum = 0;
                if (cls < D && group < groups) {
                    pos = s_done[cls];
                    for (uint32_t g = 0; g < groups; ++g) {
                        const uint32_t x = s_part[g * span + cls];
                        pos += g < group ? x : 0u;
                        sum += x;
                    }
                    for (uint32_t q = q0; q < q1; ++q) {
                        if (q % kSmallBlocks == c) s_place[q / kSmallBlocks * D + cls] = pos;
                        pos += events_of(f0 + q);
                    }
                }
                __syncthreads();
                if (threadIdx.x < D) s_done[threadIdx.x] += sum;  // (group 0: sum over all groups)
                // this block's fires' events, a warp per fire (k_expand)
                for (uint32_t i = threadIdx.x >> 5; i * kSmallBlocks + c < m; i += kSmallThreads / 32) {
                    const uint32_t src = s_fire[f0 + i * kSmallBlocks + c];
                    const uint32_t* row = e.pre_off + static_cast<size_t>(src) * (D + 1);
                    const unsigned long long* from = e.pre_ev + e.pre_base[src];
                    const uint32_t lane = threadIdx.x & 31;
                    // the fire's class offsets: in the lanes when they fit
                    const uint32_t own = D < 32 && lane <= D ? row[lane] : 0u;
                    const uint32_t k0 = D < 32 ? __shfl_sync(0xffffffffu, own, 0) : row[0];
                    const uint32_t k1 = D < 32 ? __shfl_sync(0xffffffffu, own, D & 31) : row[D];
                    if (lane == 0 && k1 - k0 > 256) atomicMax(&s_widest, min(k1 - k0, 1u << 24));
                    for (uint32_t kb = k0; kb < k1; kb += 32) {
                        const uint32_t k = kb + lane;
                        const unsigned long long v = k < k1 ? from[k] : 0ull;
                        uint32_t d = 0, first = 0;  // row[d] = first <= k < row[d + 1]
                        if (D < 32) {
#pragma unroll
                            for (uint32_t step = 16; step > 0; step >>= 1) {
                                const uint32_t x = __shfl_sync(0xffffffffu, own, (d + step) & 31);
                                if (d + step < D && x <= k) d += step;
                            }
                            first = __shfl_sync(0xffffffffu, own, d);
                        } else {
                            uint32_t above = D;
                            while (above - d > 1) {
                                const uint32_t mid = (d + above) >> 1;
                                if (row[mid] <= k) {
                                    d = mid;
                                } else {
                                    above = mid;
                                }
                            }
                            first = row[d];
                        }
                        if (k < k1 && s_sum[d] != 0xFFFFFFFFu)
                            e.wheel[static_cast<size_t>(s_slot_of[d]) * e.slot_cap + s_start[d] + s_place[i * D + d] +
                                    (k - first)] = v;
                    }
                }
                __syncthreads();
            }
            if (threadIdx.x < D && s_sum[threadIdx.x] != 0xFFFFFFFFu)
                s_slot[s_slot_of[threadIdx.x]] += s_sum[threadIdx.x];
            if (e.raster_cap > 0) {
                if (c == 0 && threadIdx.x == 0 && raster + nf > e.raster_cap) raise_status(e, kStatusRasterOverflow);
                raster += nf;
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) s_slot[slot] = 0;
        delivered += n;
        fired += nf;
        most = n > most ? n : most;
        proxy_fence();  // (the next due list, written here, comes in by a bulk copy)
        __syncwarp();
        cluster_arrive();
        if (threadIdx.x == 0) {
            debt += kSmallRow * s_rows + kSmallCopy * s_widest + nf * span / 10 * kSmallClass10 +
                    (nw > kSmallThreads && n > kSmallEven ? (n - kSmallEven) * kSmallEvent : 0u);
            debt = debt > gain ? debt - gain : 0u;
            // (the other blocks may not see this before their next tick's
            // barrier: the run ends after that tick)
            if (debt > kSmallDebt) atomicCAS(&e.ts->small_stop, 0u, t + 2);
        }
        __syncwarp();
        cluster_wait();
        ++t;
        if (t >= end) break;
        const uint32_t stop = __ldcg(&e.ts->small_stop);
        if (stop != 0 && stop <= t) break;
        __syncthreads();
    }
    __syncthreads();
    if (threadIdx.x == 0) e.ts->small_debt[c] = debt;
    if (c != 0) return;
    for (uint32_t i = threadIdx.x; i < e.W; i += kSmallThreads) e.slot_count[i] = s_slot[i];
    if ((threadIdx.x & 31) == 0 && external) atomicAdd(&e.ts->external, external);
    if (threadIdx.x == 0) {
        TickState* ts = e.ts;
        if (t < end) atomicCAS(&ts->small_stop, 0u, t == 0 ? 1u : t);
        ts->tick = t;
        ts->delivered += delivered;
        ts->fired += fired;
        if (most > ts->max_slot_events) ts->max_slot_events = most;
        ts->raster_count = raster;
    }
}

__global__ void k_inject(Engine e, const unsigned long long* ev, const uint32_t* slot_of_group,
                         const uint32_t* group_off, uint32_t groups) {
    for (uint32_t gi = blockIdx.x; gi < groups; gi += gridDim.x) {
        const uint32_t slot = slot_of_group[gi];
        const uint32_t b = group_off[gi], en = group_off[gi + 1];
        const uint32_t base = e.slot_count[slot];
        if (static_cast<unsigned long long>(base) + (en - b) > e.slot_cap) {
            if (threadIdx.x == 0) raise_status(e, kStatusSlotOverflow);
            continue;
        }
        unsigned long long* dst = e.wheel + static_cast<size_t>(slot) * e.slot_cap + base;
        for (uint32_t i = threadIdx.x; i < en - b; i += blockDim.x) dst[i] = ev[b + i];
        __syncthreads();
        if (threadIdx.x == 0) e.slot_count[slot] = base + (en - b);
        __syncthreads();
    }
}

__global__ void k_rule_off(SynAB* syn, unsigned long long b, unsigned long long en) {
    for (unsigned long long i = b + blockIdx.x * static_cast<unsigned long long>(blockDim.x) + threadIdx.x; i < en;
         i += static_cast<unsigned long long>(gridDim.x) * blockDim.x)
        syn[i].a.meta |= 1u << kMetaRuleOffBit;
}

__global__ void k_range_counts(Engine e, uint32_t nb, uint32_t ne, unsigned long long tb, unsigned long long te,
                               unsigned long long* out) {
    const unsigned long long stride = static_cast<unsigned long long>(gridDim.x) * blockDim.x;
    const unsigned long long first = blockIdx.x * static_cast<unsigned long long>(blockDim.x) + threadIdx.x;
    unsigned long long spikes = 0, pre = 0, wheel = 0, matches = 0, code_matches = 0;
    for (unsigned long long n = nb + first; n < ne; n += stride) {
        spikes += e.nrec[n].spike_count;
        matches += e.nrec[n].match_count;
    }
    for (unsigned long long i = tb + first; i < te; i += stride) {
        pre += e.syn[i].b.pre_count;
        code_matches += e.syn[i].b.code_matches;
    }
    // the wheel: every block has all slots' counts at once (one after the other
    // they were W waits); wheels of more slots than a block has threads are shared
    // out by slots
    auto count_events = [&](uint32_t slot, uint32_t cnt, unsigned long long from, unsigned long long step) {
        const unsigned long long* ev = e.wheel + static_cast<size_t>(slot) * e.slot_cap;
        for (unsigned long long i = from; i < cnt; i += step) {
            const uint32_t tgt = static_cast<uint32_t>(ev[i]) & ~kExternalBit;
            wheel += tgt >= nb && tgt < ne;
        }
    };
    __shared__ uint32_t s_count[kThreads];
    if (e.W <= kThreads) {
        if (threadIdx.x < e.W) s_count[threadIdx.x] = e.slot_count[threadIdx.x];
        __syncthreads();
        // (a slot's first events go to another block each time: few events would
        // otherwise be the first blocks' work, slot after slot)
        const uint32_t turn = gridDim.x / e.W;
        for (uint32_t slot = 0; slot < e.W; ++slot) {
            const uint32_t at = blockIdx.x + slot * turn, b = at < gridDim.x ? at : at - gridDim.x;
            count_events(slot, s_count[slot], b * blockDim.x + threadIdx.x, stride);
        }
    } else {
        const uint32_t parts = gridDim.x > e.W ? gridDim.x / e.W : 1u;
        for (uint32_t task = blockIdx.x; task < e.W * parts; task += gridDim.x)
            count_events(task % e.W, e.slot_count[task % e.W], task / e.W * blockDim.x + threadIdx.x, parts * blockDim.x);
    }
    // one atomic a block and sum (a thread each, they took longer than the reads)
    __shared__ unsigned long long s_sum[5];
    __syncthreads();
    if (threadIdx.x < 5) s_sum[threadIdx.x] = 0;
    __syncthreads();
    unsigned long long sums[5] = {spikes, pre, wheel, matches, code_matches};
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        for (int d = 16; d > 0; d >>= 1) sums[k] += __shfl_down_sync(0xffffffffu, sums[k], d);
        if ((threadIdx.x & 31) == 0 && sums[k]) atomicAdd(&s_sum[k], sums[k]);
    }
    __syncthreads();
    if (threadIdx.x < 5 && s_sum[threadIdx.x]) atomicAdd(out + threadIdx.x, s_sum[threadIdx.x]);
}

// Readers: a thread per neuron or synapse; the outputs are coalesced, the
// synapse records come in Connectome order (one random 64-byte read each).
__global__ void k_unpack_neurons(Engine e, uint32_t n0, uint32_t count, NeuronArrays o) {
    constexpr float kTau[4] = {5.0f, 100.0f, 10.0f, 150.0f};  // receptor decay taus
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        const NeuronRec r = e.nrec[n0 + i];
        const NeuronTp q = e.ntp[n0 + i];
        if (o.current) {
            reinterpret_cast<float4*>(o.current)[i] = make_float4(r.cur[0], r.cur[1], r.cur[2], r.cur[3]);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t code = (r.flags >> (2 * k)) & 3u;
                o.tau[4ull * i + k] = code == 0 ? kTau[0] : (code == 1 ? kTau[1] : (code == 2 ? kTau[2] : kTau[3]));
                o.update[4ull * i + k] = r.upd[k];
            }
        } else {
            o.membrane[i] = r.membrane;
            o.spikes[i] = r.spike_count;
            o.fired[i] = static_cast<int64_t>(r.last_fired1) - 1;  // 0: none, reads -1
            o.active[i] = r.last_active;
            o.window[i] = r.ws;
            o.offsets[i] = r.len;
            o.learned[i] = q.ref_count;
            o.matches[i] = r.match_count;
            o.match[i] = static_cast<uint8_t>(q.last_match);
        }
    }
}

__global__ void k_unpack_synapses(Engine e, const uint32_t* order, unsigned long long count, SynapseArrays o) {
    for (unsigned long long i = blockIdx.x * static_cast<unsigned long long>(blockDim.x) + threadIdx.x; i < count;
         i += static_cast<unsigned long long>(gridDim.x) * blockDim.x) {
        const SynAB r = load_record(e.syn + order[i]);
        o.weight[i] = r.a.weight;
        o.pre[i] = static_cast<int64_t>(r.a.last_pre1) - 1;  // 0: none, reads -1
        o.post[i] = static_cast<int64_t>(r.a.last_post1) - 1;
        o.pre_count[i] = r.b.pre_count;
        o.updates[i] = r.a.updates;
        o.delta[i] = r.a.last_delta;
        o.window[i] = r.b.code_ws;
        o.offsets[i] = r.b.code_len;
        o.learned[i] = r.b.learned_count;
        o.matches[i] = r.b.code_matches;
        o.match[i] = r.b.flags & 1u;
    }
}

// 64-bit mix of one word into a running hash (multiply / xor-shift rounds).
__device__ __forceinline__ unsigned long long mix64(unsigned long long h, unsigned long long w) {
    h ^= w + 0x9e3779b97f4a7c15ull + (h << 6) + (h >> 2);
    h *= 0xbf58476d1ce4e5b9ull;
    h ^= h >> 31;
    return h;
}

template <int kWords>
__device__ __forceinline__ unsigned long long record_hash(unsigned long long index, const uint32_t* w) {
    unsigned long long h = mix64(0x6a09e667f3bcc908ull, index);
#pragma unroll
    for (int i = 0; i < kWords; ++i) h = mix64(h, w[i]);
    return h;
}

constexpr int checksum_blocks(bool inline_codes) { return inline_codes ? 8 : 4; }  // per SM

// Order-independent checksums of neurons [nb, ne) (NeuronRec + NeuronTp)
// and of their incoming synapses: the sum over records of a hash of (index
// within the range, the record's meaning).  A synapse contributes its SynA
// words (the rule-off bit masked), its code-pattern counters, its code
// offsets and its learned code patterns, wherever the layout keeps them
// (inline in the record or in the pattern pool, which depends on the widest
// code of the whole simulation), so a batch member and its solo run give
// equal sums exactly when their states are equal (up to hash collisions).
//
// Bound by the hash's instructions (about 19 words a record, a 64-bit multiply
// each).  kInline (every learned code pattern in its record): a thread per
// synapse over the whole range with eight blocks per SM, 5.4 -> 3.3 ms for 2e8
// synapses (12.8 GB, 3.9 TB/s); a warp per target had four, ran a partial
// round at the end of every target and chose the patterns' place per record.
template <bool kInline>
__global__ void __launch_bounds__(kThreads, checksum_blocks(kInline)) k_checksum(const __grid_constant__ Engine e, uint32_t nb, uint32_t ne, unsigned long long tb, unsigned long long* out) {
    const unsigned long long stride = static_cast<unsigned long long>(gridDim.x) * blockDim.x;
    const unsigned long long first = blockIdx.x * static_cast<unsigned long long>(blockDim.x) + threadIdx.x;
    unsigned long long hn = 0, hs = 0;
    for (unsigned long long n = nb + first; n < ne; n += stride) {
        uint32_t w[24];
        const uint4* r = reinterpret_cast<const uint4*>(e.nrec + n);
        const uint4* q = reinterpret_cast<const uint4*>(e.ntp + n);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint4 v = r[i];
            w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const uint4 v = q[i];
            w[16 + 4 * i] = v.x; w[17 + 4 * i] = v.y; w[18 + 4 * i] = v.z; w[19 + 4 * i] = v.w;
        }
        hn += record_hash<24>(n - nb, w);
    }
    // a record's words but its learned code patterns
    auto synapse_hash = [&](unsigned long long index, const SynAB& rec) {
        const SynA& a = rec.a;
        const SynB& sb = rec.b;
        unsigned long long h = mix64(0x6a09e667f3bcc908ull, index);
        h = mix64(h, __float_as_uint(a.weight));
        h = mix64(h, a.last_pre1);
        h = mix64(h, a.last_post1);
        h = mix64(h, a.meta & ~(1u << kMetaRuleOffBit));
        h = mix64(h, __float_as_uint(a.clamp_hi));
        h = mix64(h, a.updates);
        h = mix64(h, __float_as_uint(a.last_delta));
        h = mix64(h, a.post_cnt);
        h = mix64(h, sb.pre_count);
        h = mix64(h, sb.code_ws);
        h = mix64(h, sb.code_matches);
        return mix64(h, sb.code_len | (static_cast<uint32_t>(sb.flags) << 8) |
                            (static_cast<uint32_t>(sb.learned_count) << 16));
    };
    if constexpr (kInline) {
        const unsigned long long te = e.in_ptr[ne];
        for (unsigned long long i = tb + first; i < te; i += stride) {
            const SynAB rec = load_record(e.syn + i);
            unsigned long long h = synapse_hash(i - tb, rec);
            const uint32_t expected = (rec.a.meta >> kMetaExpectedShift) & 15u;
            const uint32_t learned = rec.b.learned_count ? expected : 0u;  // one pattern at most
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j)
                if (j < rec.b.code_len) h = mix64(h, static_cast<uint32_t>(rec.b.ring_lo >> (16 * j)) & 0xFFFFu);
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j)
                if (j < learned) h = mix64(h, static_cast<uint32_t>(rec.b.ring_hi >> (16 * j)) & 0xFFFFu);
            hs += h;
        }
    } else {
        // a warp per target
        const uint32_t lane = threadIdx.x & 31;
        const unsigned long long warps = stride / 32;
        for (unsigned long long n = nb + first / 32; n < ne; n += warps) {
            const NeuronParam p = e.nparam[n];
            const bool inl = inline_code_pattern(p.max_refs, e.code_stride);
            for (unsigned long long i = e.in_ptr[n] + lane; i < e.in_ptr[n + 1]; i += 32) {
                const SynAB rec = load_record(e.syn + i);
                const SynB& sb = rec.b;
                unsigned long long h = synapse_hash(i - tb, rec);
                for (uint32_t j = 0; j < sb.code_len; ++j) h = mix64(h, ring_get(sb.ring_lo, sb.ring_hi, j));
                const uint32_t expected = (rec.a.meta >> kMetaExpectedShift) & 15u;
                const uint16_t* lc =
                    e.lcode + p.lcode_base + static_cast<size_t>(i - p.in_begin) * p.max_refs * e.code_stride;
                for (uint32_t k = 0; k < sb.learned_count; ++k)
                    for (uint32_t j = 0; j < expected; ++j)
                        h = mix64(h, inl ? ring_get(sb.ring_hi, 0ull, j) : lc[static_cast<size_t>(k) * e.code_stride + j]);
                hs += h;
            }
        }
    }
    for (int d = 16; d > 0; d >>= 1) {
        hn += __shfl_down_sync(0xffffffffu, hn, d);
        hs += __shfl_down_sync(0xffffffffu, hs, d);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(out, hn);
        atomicAdd(out + 1, hs);
    }
}

}  // namespace

void launch_checksum(const Engine& e, uint32_t n_begin, uint32_t n_end, unsigned long long tm_begin,
                     unsigned long long* out, cudaStream_t stream) {
    const uint32_t grid = e.grid_wide / 2 * checksum_blocks(e.inline_codes);
    if (e.inline_codes) {
        k_checksum<true><<<grid, kThreads, 0, stream>>>(e, n_begin, n_end, tm_begin, out);
    } else {
        k_checksum<false><<<grid, kThreads, 0, stream>>>(e, n_begin, n_end, tm_begin, out);
    }
}

void launch_unpack_neurons(const Engine& e, uint32_t n0, uint32_t count, const NeuronArrays& out, cudaStream_t stream) {
    k_unpack_neurons<<<e.grid_wide * 4, kThreads, 0, stream>>>(e, n0, count, out);
}

void launch_unpack_synapses(const Engine& e, const uint32_t* order, uint64_t count, const SynapseArrays& out,
                            cudaStream_t stream) {
    k_unpack_synapses<<<e.grid_wide * 4, kThreads, 0, stream>>>(e, order, count, out);
}

void launch_rule_off(const Engine& e, unsigned long long tm_begin, unsigned long long tm_end, cudaStream_t stream) {
    if (tm_end > tm_begin) k_rule_off<<<1024, kThreads, 0, stream>>>(e.syn, tm_begin, tm_end);
}

void launch_range_counts(const Engine& e, uint32_t n_begin, uint32_t n_end, unsigned long long tm_begin,
                         unsigned long long tm_end, unsigned long long* out, cudaStream_t stream) {
    k_range_counts<<<e.grid_wide, kThreads, 0, stream>>>(e, n_begin, n_end, tm_begin, tm_end, out);
}

// Launch of a main-stream tick kernel.  `dependent` makes it a programmatic
// dependent of the kernel before it on the stream (see tick_enter): its
// blocks are scheduled while that kernel drains instead of after it.
static void launch_main(void (*kernel)(Engine), uint32_t grid, uint32_t block, size_t smem, cudaStream_t stream,
                        bool dependent, const Engine& e) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = dependent ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, e);
}

// Dynamic shared memory of the grouping kernels and of k_events.
static size_t bucket_smem(const Engine& e) {
    return stream_buf_offset(e.nbuckets) + kStreamBufs * kStreamTile * sizeof(unsigned long long);
}
static size_t group_smem(uint32_t bucket_shift) {
    return kSortSmemBytes + ((static_cast<size_t>(1) << bucket_shift) + 1) * sizeof(uint32_t);
}
static size_t events_smem(uint32_t bucket_shift) {
    const size_t width = static_cast<size_t>(1) << bucket_shift;
    return kBlockEvents * (sizeof(BucketEntry) + 2 + 2) + (width <= kSharedParams ? width * sizeof(TargetParam) : 0) +
           (width + 2) * sizeof(uint32_t);
}

// k_temporal's lanes per target: a whole warp while every target has one
// resident at once, on larger networks as many as patterns, up to 8 (50,000
// targets of 2 patterns: 41 us with 8 lanes, 23 with 2).
static void launch_temporal(const Engine& e, cudaStream_t stream) {
    if (e.N <= e.grid_wide * 32u) {
        k_temporal<32><<<(e.N + kThreads / 32 - 1) / (kThreads / 32), kThreads, 0, stream>>>(e);
    } else if (e.multi_refs <= 2) {
        k_temporal<2><<<e.grid_process, kThreads, 0, stream>>>(e);
    } else if (e.multi_refs <= 4) {
        k_temporal<4><<<e.grid_process, kThreads, 0, stream>>>(e);
    } else {
        k_temporal<8><<<e.grid_process, kThreads, 0, stream>>>(e);
    }
}

void launch_tick(const Engine& e, const TickStreams& s, cudaEvent_t* marks) {
    const uint32_t wide = e.grid_wide;
    cudaStream_t stream = s.main;
    // Kernels that follow another kernel directly on the main stream are
    // programmatic dependents; the per-kernel profile (event marks between
    // the kernels) launches them plainly so each kernel is timed alone.
    const bool dep = marks == nullptr;
    int k = 0;
    auto mark = [&](bool after) {
        if (marks) cudaEventRecordWithFlags(marks[2 * k + (after ? 1 : 0)], stream, cudaEventRecordExternal);
        if (after) ++k;
    };
    auto side_mark = [&](int index, bool after) {
        if (marks)
            cudaEventRecordWithFlags(marks[2 * index + (after ? 1 : 0)],
                                     e.side_serial ? stream : s.side,
                                     cudaEventRecordExternal);
    };
    // k_bcount follows a wait on the side stream: a full dependency
    mark(false); launch_main(k_bcount, e.grid_bucket, kBucketThreads, bucket_smem(e), stream, false, e); mark(true);
    mark(false); launch_main(k_bscatter, e.grid_bucket, kBucketThreads, bucket_smem(e), stream, dep, e); mark(true);
    mark(false);
    launch_main(e.inline_codes ? k_events<true> : k_events<false>,
                std::min(e.grid_events, std::max(e.nbuckets, wide)), kEventThreads,
                events_smem(e.bucket_shift), stream, dep, e);
    mark(true);
    if (e.side_serial) {
        // everything in tick order on the main stream; k_post and the fire
        // ordering take full dependencies (as programmatic dependents they
        // made the tick 7 % slower on recog_1m: their blocks, launched early,
        // held SM resources the kernel before them needed)
        side_mark(6, false);
        launch_main(k_post, wide * 2, kThreads, 0, stream, false, e);
        side_mark(6, true);
        side_mark(7, false);
        if (e.multi_refs) launch_temporal(e, stream);
        side_mark(7, true);
        mark(false); launch_main(k_fire_list, e.grid_fire, kThreads, 0, stream, false, e); mark(true);
        mark(false); launch_main(k_fire_count, e.grid_wide / 4 + 1, kFireCountThreads, 0, stream, false, e); mark(true);
        mark(false); launch_main(k_expand, e.grid_wide * 4, kThreads, 0, stream, dep, e); mark(true);
        return;
    }
    // post-spike STDP of the fired targets and the temporal patterns of the
    // targets with several reference patterns run beside the fire ordering
    // and the expansion (which touch neither)
    cudaEventRecord(s.ev[0], stream);
    cudaStreamWaitEvent(s.side, s.ev[0], 0);
    side_mark(6, false);
    k_post<<<wide, kThreads, 0, s.side>>>(e);
    side_mark(6, true);
    side_mark(7, false);
    if (e.multi_refs) launch_temporal(e, s.side);
    side_mark(7, true);
    cudaEventRecord(s.ev[1], s.side);
    mark(false); launch_main(k_fire_list, e.grid_fire, kThreads, 0, stream, dep, e); mark(true);
    mark(false); launch_main(k_fire_count, e.grid_wide / 4 + 1, kFireCountThreads, 0, stream, dep, e); mark(true);
    mark(false); launch_main(k_expand, e.grid_wide * 4, kThreads, 0, stream, dep, e); mark(true);
    cudaStreamWaitEvent(stream, s.ev[1], 0);  // the next tick's k_events reads the records k_post updates
}

const char* kernel_name(int index) {
    static const char* names[kKernelCount] = {"k_bcount",     "k_bscatter", "k_events", "k_fire_list",
                                              "k_fire_count", "k_expand",   "k_post",   "k_temporal"};
    return index >= 0 && index < kKernelCount ? names[index] : "";
}

void launch_group(const Engine& e, uint32_t count, cudaStream_t stream) {
    // (programmatic dependents: each kernel waits in tick_enter)
    const uint32_t init = e.nbuckets / kThreads + 1;
    k_group_init<<<init < 64 ? init : 64, kThreads, 0, stream>>>(e, count);
    launch_main(k_bcount, e.grid_bucket, kBucketThreads, bucket_smem(e), stream, false, e);
    launch_main(k_bscatter, e.grid_bucket, kBucketThreads, bucket_smem(e), stream, true, e);
    launch_main(k_group, e.nbuckets, kThreads, group_smem(e.bucket_shift), stream, true, e);
    // (a bucket or a segment it cannot rank needs more events than that)
    if (count > kRankEvents) launch_main(k_group_rest, e.grid_wide / 2, kLongThreads, kLongSmemBytes, stream, true, e);
}

void configure_kernels() {
    const int bucket_bytes =
        static_cast<int>(stream_buf_offset(kMaxTickBuckets) + kStreamBufs * kStreamTile * sizeof(unsigned long long));
    cudaFuncSetAttribute(k_bcount, cudaFuncAttributeMaxDynamicSharedMemorySize, bucket_bytes);
    cudaFuncSetAttribute(k_bscatter, cudaFuncAttributeMaxDynamicSharedMemorySize, bucket_bytes);
    const int events_bytes = static_cast<int>(std::max(events_smem(kMaxBucketShift), events_smem(8)));
    cudaFuncSetAttribute(k_events<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, events_bytes);
    cudaFuncSetAttribute(k_events<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, events_bytes);
    cudaFuncSetAttribute(k_small<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmallSmem));
    cudaFuncSetAttribute(k_small<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmallSmem));
}

void configure_group() {
    const int bucket_bytes =
        static_cast<int>(stream_buf_offset(kMaxTickBuckets) + kStreamBufs * kStreamTile * sizeof(unsigned long long));
    cudaFuncSetAttribute(k_bcount, cudaFuncAttributeMaxDynamicSharedMemorySize, bucket_bytes);
    cudaFuncSetAttribute(k_bscatter, cudaFuncAttributeMaxDynamicSharedMemorySize, bucket_bytes);
    cudaFuncSetAttribute(k_group, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         static_cast<int>(group_smem(kMaxBucketShift)));
}

void launch_small(const Engine& e, uint32_t end, uint32_t limit, cudaStream_t stream) {
    if (e.inline_codes) {
        k_small<true><<<kSmallBlocks, kSmallThreads, kSmallSmem, stream>>>(e, end, limit);
    } else {
        k_small<false><<<kSmallBlocks, kSmallThreads, kSmallSmem, stream>>>(e, end, limit);
    }
}

void launch_init_syn(const Engine& e, const SynA* a, cudaStream_t stream) {
    if (e.S == 0) return;
    k_init_syn<<<1024, kThreads, 0, stream>>>(e.syn, a, e.S);
}

void launch_inject(const Engine& e, const unsigned long long* ev, const uint32_t* slot_of_group,
                   const uint32_t* group_off, uint32_t groups, cudaStream_t stream) {
    if (groups == 0) return;
    k_inject<<<groups < 1024 ? groups : 1024, kThreads, 0, stream>>>(e, ev, slot_of_group, group_off, groups);
}

}  // namespace snngb
