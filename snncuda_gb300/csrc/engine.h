// Device data layout and kernel interface of the GB300 tick engine.
//
// One simulation = one network resident in HBM:
//   * neurons: NeuronRec (64 B, dynamic state), NeuronTp (32 B, temporal
//     bookkeeping), NeuronParam (64 B, read-only) -- one per neuron;
//   * synapses in target-major order (incoming lists of each target
//     contiguous, Connectome order inside a list), one 64 B record each:
//     SynA (weight, STDP state, static fields) + SynB (code-pattern state,
//     counters), so the per-event work touches one DRAM line per event;
//   * pre-expanded outgoing events: for every source, its (synapse, code
//     offset) events grouped by delivery delay class, each class in
//     Connectome x offset order -- spike-code expansion is then a copy;
//   * a timing wheel of W slots, each a buffer of 64-bit events in exact
//     scheduling order (the reference bucket FIFO order).
#pragma once

#include <cstddef>
#include <cstdint>

namespace snngb {

// Event word: low 32 bits = target neuron, bit 31 set for an external input;
// high 32 bits = target-major synapse index, or the float weight bits of an
// external input.
constexpr uint32_t kExternalBit = 0x80000000u;

// Status bits raised by kernels (host maps them to SNNCUDA_ERR_*).
constexpr uint32_t kStatusSlotOverflow = 1u << 0;
constexpr uint32_t kStatusRingOverflow = 1u << 1;
constexpr uint32_t kStatusRasterOverflow = 1u << 2;
constexpr uint32_t kStatusPostCountOverflow = 1u << 3;
constexpr uint32_t kStatusRunOverflow = 1u << 4;
constexpr uint32_t kStatusFireOverflow = 1u << 5;
constexpr uint32_t kStatusBadEvent = 1u << 6;       // event target out of range (grouping input)
constexpr uint32_t kStatusStageTimeout = 1u << 7;   // a bounded wait for a bulk copy ran out

// SynA.meta bit fields.
constexpr uint32_t kMetaDelayMask = 0xFFFFu;
constexpr int kMetaCompShift = 16;      // 2 bits
constexpr int kMetaRecShift = 18;       // 2 bits
constexpr int kMetaPlasticBit = 20;     // 1 bit
constexpr int kMetaExpectedShift = 21;  // 4 bits: max(2, #code offsets), <= 8
constexpr int kMetaRuleOffBit = 25;     // the synapse's network runs with the STDP rule disabled

constexpr int kMaxExpected = 8;

struct alignas(32) SynA {
    float weight;
    uint32_t last_pre1;   // last_pre_spike_tick + 1, 0 = none
    uint32_t last_post1;  // last_post_spike_tick + 1, 0 = none
    uint32_t meta;
    float clamp_hi;       // min(StdpConfig::max_weight, synapse max_weight)
    uint32_t updates;     // plasticity_update_count
    float last_delta;     // last_weight_delta
    uint32_t post_cnt;    // target fires already applied at tick last_post1-1
};

struct alignas(32) SynB {
    uint32_t pre_count;
    uint32_t code_ws;       // code_window_start_tick
    uint32_t code_matches;  // code_match_count
    uint8_t code_len;       // code_offsets.size() (<= expected)
    uint8_t flags;          // bit 0: last_code_match; bits 4-7: expected = max(2, #code offsets)
    uint16_t learned_count; // learned_code_patterns.size()
    // code_offsets in order, 16 bits each: offsets 0-3 in ring_lo, 4-7 in
    // ring_hi.  When the target keeps a single reference pattern and no code
    // has more than 4 offsets (inline_code_pattern), ring_hi instead holds the
    // synapse's one learned code pattern.
    unsigned long long ring_lo;
    unsigned long long ring_hi;
};

struct alignas(64) SynAB {
    SynA a;
    SynB b;
};

// Per-event input of the neuron walk, in due order inside
// every target's group: the weight after the event's pre-spike STDP (computed
// as if the target had not fired earlier in the tick), compartment, receptor
// and flags, the synapse and the due position.
struct alignas(16) EvIn {
    float weight;
    uint32_t bits;  // comp | rec << 2 | external << 4 | repeat << 5
    uint32_t tm;    // target-major synapse index (synaptic events)
    uint32_t due;   // position in the tick's due list
};
// The fields of a synapse record that an event's pre-spike work changes, as
// they were before the event (k_events writes one per synaptic event; the
// per-target walk redoes an event that follows a fire of its target from
// them and the record's other fields, which that work does not change).
struct alignas(16) SynPre {
    float weight;
    uint32_t last_pre1;
    uint32_t updates;
    float last_delta;
};
constexpr uint32_t kEvExternal = 1u << 4;
constexpr uint32_t kEvRepeat = 1u << 5;  // not the first event of its synapse in this tick

__host__ __device__ inline bool inline_code_pattern(uint32_t max_refs, uint32_t code_stride) {
    return max_refs == 1 && code_stride <= 4;
}

__host__ __device__ inline uint32_t ring_get(unsigned long long lo, unsigned long long hi, uint32_t j) {
    return static_cast<uint32_t>((j < 4 ? lo >> (16 * j) : hi >> (16 * (j - 4))) & 0xFFFFu);
}

struct alignas(64) NeuronRec {
    float cur[4];          // soma, basal, apical, inhibitory current
    uint32_t upd[4];       // compartment last_update_tick
    float membrane;
    uint32_t spike_count;
    uint32_t last_fired1;  // last_fired_tick + 1, 0 = none
    uint32_t last_active;
    uint32_t flags;        // 4 x 2-bit tau code
    // temporal pattern fields
    uint32_t match_count;
    uint32_t ws;           // temporal window_start_tick
    uint32_t len;          // spike_offsets.size()
};

struct alignas(32) NeuronTp {
    unsigned long long cn;  // sum of squares of the current window's offsets
    uint32_t nruns;         // runs in the current window's run list
    uint32_t ref_head;      // FIFO index of the oldest learned pattern
    uint32_t ref_count;
    uint32_t ring_head;     // next free run slot of the learned-pattern run ring
    uint32_t ring_used;
    uint32_t last_match;    // temporal_pattern.last_match
};

struct alignas(64) NeuronParam {
    float threshold;
    uint32_t window;        // pattern_window_ticks
    float similarity;
    uint32_t max_refs;      // max_reference_patterns
    uint32_t ring_cap;      // runs in the learned-pattern ring
    uint32_t pad;
    unsigned long long in_begin;    // first target-major synapse index
    unsigned long long cand_base;   // run list of the current window (window+1 runs)
    unsigned long long meta_base;   // max_refs RefMeta entries
    unsigned long long ring_base;   // ring_cap runs
    unsigned long long lcode_base;  // learned code patterns of the incoming synapses
};

// A learned temporal pattern: runs in the neuron's ring plus the running
// prefix sums of its cosine against the current window.
struct alignas(16) RefMeta {
    unsigned long long dot, rn, cn;  // exact integer sums over min(len, window length)
    uint32_t start;                  // first run (ring position)
    uint32_t nruns;
    uint32_t len;                    // pattern length
    uint32_t cur_run;                // cursor into the pattern (run, position)
    uint32_t cur_pos;
    uint32_t match;                  // 0 no, 1 yes, 2 unknown (recompute from sums)
};

// A run of equal offsets: value in the low 16 bits, count in the high 48.
__host__ __device__ inline uint32_t run_value(unsigned long long r) { return static_cast<uint32_t>(r & 0xFFFFu); }
__host__ __device__ inline unsigned long long run_count(unsigned long long r) { return r >> 16; }

// Per-tick scratch and counters that live on the device.
struct TickState {
    unsigned long long delivered;
    unsigned long long external;
    unsigned long long fired;
    unsigned long long max_slot_events;
    unsigned long long raster_count;
    unsigned long long touched_total;  // sum of n_touched over ticks
    uint32_t status;
    uint32_t tick;            // tick being processed
    uint32_t n_due;           // events due this tick
    uint32_t n_touched;       // targets with at least one due event
    uint32_t n_fires;         // fires this tick
    uint32_t n_fired_targets; // distinct targets that fired this tick (reset by k_bcount)
    uint32_t post_tick;       // tick of the pending post-spike STDP (set by k_bcount; read by k_post)
    uint32_t expand_fires;    // fires whose events k_expand copies
    uint32_t far_first_tick;  // delivery tick of far_idx[0] for the current run
    uint32_t far_ticks;       // entries of far_idx minus one (0 = none)
    int32_t stdp_enabled;     // StdpRule::enabled (runtime toggle)
    int32_t temporal_enabled; // SynapseDendriteConfig::temporal_learning_enabled
    uint32_t done_fire_list;  // "last block" counter
    uint32_t small_stop;      // not 0: k_small ended before its last tick (launch_small)
    uint32_t n_parts;         // entries of Engine::parts this tick (reset by k_bcount),
    uint32_t part_events;     // and events of a part (part_shift)
    uint32_t small_debt[8];   // per block of k_small: ns that its ticks have lost (kSmallDebt)
};

struct Tables {
    const float* decay;     // [4][decay_len]: expf(-e / tau_k), e = 0..decay_len-1
    uint32_t decay_len;
    const float* ltp;       // [stdp_len]: A+ expf(-dt / tau+)
    const float* ltd;       // [stdp_len]: -A- expf(-dt / tau-)
    uint32_t stdp_len;
};

// Everything a tick needs, passed by value to the kernels.
// One due event placed in its bucket by k_bscatter: the due-list word with
// its due index in the low bits (payload << 32 | due index | external bit)
// and its target within the bucket.  16 bytes, so the scattered placement is
// one store per event.
struct alignas(16) BucketEntry {
    unsigned long long ev;
    uint32_t ltgt;
    uint32_t unused;
};

struct Engine {
    uint32_t N;
    uint32_t W;             // wheel slots (power of two)
    uint32_t wmask;
    uint32_t D;             // delay classes
    unsigned long long S;
    unsigned long long slot_cap;
    uint32_t code_stride;   // max expected over the network
    unsigned long long raster_cap;
    uint32_t fire_cap;
    uint32_t fire_tiles_cap;
    float min_weight;
    unsigned long long stage_wait_ns;  // limit of a block's wait for a staging copy

    // network
    const unsigned long long* in_ptr;      // [N+1] target-major row pointers
    const NeuronParam* nparam;             // [N]
    NeuronRec* nrec;                       // [N]
    NeuronTp* ntp;                         // [N]
    unsigned long long* cand;              // run lists of current windows
    RefMeta* refmeta;
    unsigned long long* ring;              // learned-pattern runs
    SynAB* syn;                            // [S] target-major
    uint16_t* lcode;                       // learned code patterns
    const unsigned long long* pre_base;    // [N] first pre-expanded event of a source
    const uint32_t* pre_off;               // [N*(D+1)] class offsets within a source
    const unsigned long long* pre_ev;      // pre-expanded events
    const uint32_t* cls_delta;             // [D] delivery delay of each class (>= 1)

    // wheel
    unsigned long long* wheel;             // [W * slot_cap]
    uint32_t* slot_count;                  // [W]

    // per-tick scratch: grouping by target.  Targets are bucketed by
    // bucket_shift (2^bucket_shift consecutive targets per bucket: tick_bucket_shift,
    // at most kMaxTickBuckets buckets; bucket_shift_for, at most kMaxBuckets, in
    // grouping calls); grid_bucket blocks each count and place one contiguous chunk
    // of the due list.
    uint32_t bucket_shift;
    uint32_t nbuckets;
    uint32_t grid_bucket;
    // Due-list events per placing pass of k_bscatter (0: one pass): a due
    // list longer than this is placed in passes over disjoint bucket ranges,
    // so the lines of grp_tmp being filled stay in L2 until
    // complete instead of going to DRAM half-written.
    uint32_t scatter_pass_events;
    // 1: k_post and k_temporal run on the main stream in tick order instead
    // of on the side stream beside the fire ordering (on very large networks
    // the two slow each other by more than the overlap gives).
    uint32_t side_serial;
    uint32_t inline_codes;                 // 1: inline_code_pattern holds for every target
    uint32_t multi_refs;                   // most reference patterns of a target if several (k_temporal runs), else 0
    uint32_t* bcnt;                        // [grid_bucket][nbuckets] events of each (chunk, bucket)
    uint32_t* btot;                        // [nbuckets] events per bucket (zero between ticks)
    uint32_t* bstart;                      // [nbuckets + 1] first grouped position of each bucket
    uint32_t* bcur;                        // [nbuckets] placement cursor of each bucket
    uint32_t* parts;                       // [parts_cap] parts of the buckets that k_events shares out to
                                           // several blocks: bucket | part << 15 (null: grouping calls)
    uint32_t* seg_start;                   // [N + 1] first grouped position of each target
    unsigned long long* grp;               // [slot_cap] due events grouped by target, due order inside
                                           // a target: (payload << 32) | (due index | ext << 31)
    BucketEntry* grp_tmp;                  // [slot_cap] the due events in bucket order (unsorted inside)
    EvIn* evin;                            // [slot_cap] event inputs of buckets grouped in grp, due order
    SynPre* ev_a0;                         // [slot_cap] each synaptic event's changing fields before it
    uint32_t* fire_bits;                   // [slot_cap/32] bitmap of due positions that fired
    uint32_t* fire_at;                     // [slot_cap] firing neuron at a due position
    uint32_t* fire_tile;                   // fires per bitmap tile of kThreads words (zero between ticks)
    uint32_t* fire_list;                   // [fire_cap] firing neurons in reference order
    uint32_t* fired_tgt;                   // [N] targets that fired this tick
    uint32_t* fired_cnt;                   // [N] their fire counts
    uint32_t* xsum;                        // [fire_cap/8][D] events per (expansion block, class)
    unsigned long long* xdst;              // [fire_cap/8][D] wheel position of each
    uint32_t* xdst_ok;                     // [D] class destination fits its slot
    uint32_t* raster;                      // [raster_cap * 2] (tick, neuron)

    // far-future injections for the current run (see TickState)
    const unsigned long long* far_ev;
    const uint32_t* far_idx;

    TickState* ts;
    Tables tab;

    // launch shapes (results do not depend on them; snncuda_sim_autotune
    // picks grid_events, grid_bucket and grid_process)
    uint32_t grid_wide;
    uint32_t grid_process;  // k_temporal blocks
    uint32_t grid_fire;
    uint32_t grid_events;   // k_events blocks at most (one per bucket)
};

constexpr uint32_t kMaxBuckets = 16384;   // target buckets of the grouping (shared-memory counters)
constexpr uint32_t kScatterPassEvents = 1u << 22;  // default Engine::scatter_pass_events (64 MB of grp_tmp)
constexpr uint32_t kMaxBucketShift = 14;  // at most 2^14 targets per bucket: N <= 2^28

// Targets per bucket (log2) for N targets: the smallest 2^s >= 256 with at
// most kMaxBuckets buckets.  Returns 0 when N needs more than 2^28 targets.
__host__ __device__ constexpr uint32_t bucket_shift_for(uint32_t N) {
    uint32_t s = 8;
    while (((static_cast<unsigned long long>(N) + (1ull << s) - 1) >> s) > kMaxBuckets) ++s;
    return s <= kMaxBucketShift ? s : 0;
}
// The tick's buckets may be more and narrower than bucket_shift_for's:
// k_events takes a block per bucket, and 64 targets' events (about 12 per
// target and tick on the dense workloads, 800 of the 1,280 a block's shared
// memory holds) were the best fit there: 128 targets with twice the threads
// took 273 us where 64 took 219 (recog_1m distributions at 200,000 neurons).
// 32 targets where 64 would leave fewer than three blocks per SM.  Wider, up to
// 256 targets, where they have fewer than kBucketSynapses synapses, so that a
// bucket's events would not keep a block busy, and at least kWideBuckets buckets
// per SM are left (1e6 neurons of 50 synapses, 100,000 events: 266 us a tick with
// 64 targets, 124 with 256; 2e6 of 5, 200,000 events: 736 and 492; at 5 buckets
// per SM ticks of 1e6 and more events took 2 to 6 % longer), or when there would be
// more than kMaxTickBuckets (their counters fill the placing blocks' shared
// memory).
constexpr uint32_t kMaxTickBuckets = 32768;
constexpr uint32_t kWideBuckets = 20, kBucketSynapses = 16384;
inline uint32_t tick_bucket_shift(uint32_t N, uint64_t synapses, uint32_t sms) {
    if (bucket_shift_for(N) == 0) return 0;
    uint32_t s = (N >> 6) < 3 * sms ? 5 : 6;
    while (s < 8 && (N >> (s + 1)) >= kWideBuckets * sms && (synapses << s) / N < kBucketSynapses) ++s;
    while (((static_cast<unsigned long long>(N) + (1ull << s) - 1) >> s) > kMaxTickBuckets) ++s;
    return s;
}
inline uint32_t tick_buckets(uint32_t N, uint64_t synapses, uint32_t sms) {
    const uint32_t s = tick_bucket_shift(N, synapses, sms);
    const uint64_t n = (static_cast<uint64_t>(N) + (1u << s) - 1) >> s;
    return n > 0 ? static_cast<uint32_t>(n) : 1u;
}
// Counting and placing blocks per SM, at most (the rows of Engine::bcnt).
constexpr uint32_t kBucketBlocksPerSm = 4;

// Grouping entry points: blocks of the counting and placing kernels, at most
// (fixed, so that the static scratch has a fixed size), and the longest segment
// that a warp of k_group_rest sorts.
constexpr uint32_t kGroupGrid = 256;
constexpr uint32_t kWarpSortEvents = 512;

constexpr uint32_t group_buckets(uint32_t neuron_count) {
    const uint32_t shift = bucket_shift_for(neuron_count);
    const uint64_t n = (static_cast<uint64_t>(neuron_count) + (1u << shift) - 1) >> shift;
    return n > 0 ? static_cast<uint32_t>(n) : 1u;
}

// Entries of a grouping call's Engine::bcnt: the counting blocks' rows of
// counters, in whose memory k_group then lists the targets that have more than
// kWarpSortEvents events each.  `count` events hold at most count /
// (kWarpSortEvents + 1) of them: more than the rows hold where a bucket is
// wider than kGroupGrid targets (above 2^22 neurons) and most targets are busy.
constexpr size_t group_counters(uint32_t count, uint32_t neuron_count) {
    const size_t rows = static_cast<size_t>(kGroupGrid) * group_buckets(neuron_count);
    const size_t listed = count / (kWarpSortEvents + 1);
    return rows > listed ? rows : listed;
}

// Byte offsets (256-byte aligned) of a grouping call's arrays in its scratch.
struct GroupLayout {
    size_t bcnt, btot, bstart, bcur, grp_tmp, slot_count, ts, bytes;
};
constexpr GroupLayout group_layout(uint32_t count, uint32_t neuron_count) {
    const size_t buckets = group_buckets(neuron_count);
    GroupLayout l{};
    l.btot = l.bcnt + (group_counters(count, neuron_count) * 4 + 255) / 256 * 256;
    l.bstart = l.btot + (buckets * 4 + 255) / 256 * 256;
    l.bcur = l.bstart + ((buckets + 1) * 4 + 255) / 256 * 256;
    l.grp_tmp = l.bcur + (buckets * 4 + 255) / 256 * 256;
    l.slot_count = l.grp_tmp + ((count > 0 ? count : 1u) * sizeof(BucketEntry) + 255) / 256 * 256;
    l.ts = l.slot_count + 256;
    l.bytes = l.ts + (sizeof(TickState) + 255) / 256 * 256;
    return l;
}

// A bucket with more events than a block's shared memory holds is taken in
// 2^part_shift parts of equal target ranges (fewer where it has fewer targets),
// a block for each.  One block took such a bucket from global memory, target
// after target: a layer of 100 output neurons behind 200,000 others (100 events
// each in a tick, two buckets) kept one or two SMs busy for 1.8 ms, now 0.096;
// with every bucket too large (50,000 neurons, 25 events per target) 340 us a
// tick, now 250.  A part has part_events of the events if they are spread
// evenly: as few as make kPartBlocks parts (the blocks the GPU holds at once) of
// all such buckets, but not fewer than a block's threads, nor more than leave
// room for uneven targets in a block's 1,280 (a part that does not fit goes
// through global memory).
constexpr uint32_t kPartEvents = 800, kPartEventsMin = 160, kPartBlocks = 760;
__host__ __device__ inline uint32_t part_shift(uint32_t events, uint32_t part_events, uint32_t bucket_shift) {
    uint32_t p = 0;
    while (p < bucket_shift && (events >> p) > part_events) ++p;
    return p;
}
// Parts of a tick, at most: a bucket has fewer than 2 events / part_events.
constexpr size_t parts_cap(unsigned long long slot_cap) { return slot_cap / (kPartEvents / 2) + 2 * kPartBlocks; }

constexpr int kExpandFires = 8;          // fires per expansion block (one warp each)
constexpr uint32_t kMaxClasses = 256;    // distinct delivery delays

// Host-side launchers (kernels.cu).
// `marks` (optional) holds 2 * kKernelCount events recorded around every
// kernel (before, after) for profiling graphs.
constexpr int kKernelCount = 8;
// The streams of a tick: k_post and k_temporal run on `side`, forked from
// `main` with ev[0] and joined back with ev[1].
struct TickStreams {
    cudaStream_t main;
    cudaStream_t side;
    cudaEvent_t ev[2];
};
void launch_tick(const Engine& e, const TickStreams& s, cudaEvent_t* marks = nullptr);
const char* kernel_name(int index);
// Ticks ts->tick .. end-1 of a small network (small_network) in one kernel; it
// stops before a tick it does not take (ts->small_stop, until which the
// launches behind it return at once): one with more than `limit` events due
// (small_limit), or any after its ticks have lost more than kSmallDebt.
constexpr uint32_t kSmallBlocks = 8;
constexpr uint32_t kSmallTargets = 4096;  // per block
constexpr uint32_t kSmallEvents = 8192;
constexpr uint32_t kSmallSlots = 1024;
// What eight SMs take longer for than the launched kernels, which have them all,
// in ns: a row of post-spike STDP of one block (512 at a time, about 1 us), an
// event of the fire with the most (one warp copies them: 32 in 0.5 us), a fire
// and delay class (190 fires x 250 classes: 54 us, launched 46), an event above
// kSmallEven where the blocks have more targets than threads (8,000 neurons: 4,000
// events 31 us, launched 33, 6,000 39 and 37, 7,000 43 and 38; 16,000: 4,000 both
// 32, 7,000 44 and 35).  A
// quiet tick gains kSmallGain (1,000 neurons: 500 events 18 us, launched 28;
// 1,452 neurons, fires of 650 events: 43 and 49) less N / 4 and, as the launched
// kernels count the fires by class, kSmallClassGain per class more.  Once a
// block's ticks have lost kSmallDebt more than they gained, the launched kernels
// take over: rare heavy ticks do not do that, a layer of 100 output neurons with
// 30,000 inputs each that fires all the time (4,700 us a tick here, 126 launched)
// does in a few.
constexpr uint32_t kSmallRow = 2, kSmallCopy = 16, kSmallClass10 = 5, kSmallEvent = 6, kSmallEven = 4096;
constexpr uint32_t kSmallGain = 12000, kSmallClassGain = 32;
constexpr uint32_t kSmallDebt = 1u << 20;
static_assert(sizeof(TickState::small_debt) == kSmallBlocks * sizeof(uint32_t), "a block's debt");
static_assert(kSmallGain >= kSmallBlocks * kSmallTargets / 4, "a gain for every size");
inline uint32_t small_limit(const Engine& e) {
    const unsigned long long share = e.slot_cap / kSmallBlocks;  // a block's part of the per-event scratch
    return static_cast<uint32_t>(share < kSmallEvents ? share : kSmallEvents);
}
inline bool small_network(const Engine& e) {
    return e.N > 0 && e.N <= kSmallBlocks * kSmallTargets && e.W <= kSmallSlots && small_limit(e) >= 512;
}
void launch_small(const Engine& e, uint32_t end, uint32_t limit, cudaStream_t stream);
void launch_inject(const Engine& e, const unsigned long long* ev, const uint32_t* slot_of_group,
                   const uint32_t* group_off, uint32_t groups, cudaStream_t stream);
// Groups the W == 1 "wheel" of e (a caller's buffer of `count` events) by
// target: the tick's counting and placing kernels, then k_group.
void launch_group(const Engine& e, uint32_t count, cudaStream_t stream);
// The kernel attributes launch_group needs (as configure_kernels).
void configure_group();
// Batched form: one handle simulates several networks side by side.
// Sets kMetaRuleOffBit on target-major synapses [tm_begin, tm_end).
void launch_rule_off(const Engine& e, unsigned long long tm_begin, unsigned long long tm_end, cudaStream_t stream);
// out[0] += spike counts of neurons [n_begin, n_end); out[1] += pre-spike
// counts of target-major synapses [tm_begin, tm_end); out[2] += wheel events
// (all slots) whose target is in [n_begin, n_end); out[3] += the neurons'
// temporal match counts; out[4] += the synapses' code match counts.  out (5
// entries) must start at zero.
void launch_range_counts(const Engine& e, uint32_t n_begin, uint32_t n_end, unsigned long long tm_begin,
                         unsigned long long tm_end, unsigned long long* out, cudaStream_t stream);
// out[0] += checksum of neurons [n_begin, n_end), out[1] += checksum of
// their incoming synapses, whose target-major range starts at tm_begin
// (k_checksum); out must start at zero.
void launch_checksum(const Engine& e, uint32_t n_begin, uint32_t n_end, unsigned long long tm_begin,
                     unsigned long long* out, cudaStream_t stream);
// The readers' fields, one device array each (null: not wanted), in the types
// of snncuda_neuron_state / snncuda_synapse_state.
struct NeuronArrays {
    float* membrane;
    uint64_t* spikes;
    int64_t* fired;
    uint64_t* active;
    float* current;    // 4 per neuron
    uint64_t* update;  // 4 per neuron
    float* tau;        // 4 per neuron
    uint64_t* window;
    uint64_t* offsets;
    uint64_t* learned;
    uint64_t* matches;
    uint8_t* match;
};
struct SynapseArrays {
    float* weight;
    int64_t* pre;
    int64_t* post;
    uint64_t* pre_count;
    uint64_t* updates;
    float* delta;
    uint64_t* window;
    uint64_t* offsets;
    uint64_t* learned;
    uint64_t* matches;
    uint8_t* match;
};
// Neurons [n0, n0 + count) into the arrays.
void launch_unpack_neurons(const Engine& e, uint32_t n0, uint32_t count, const NeuronArrays& out, cudaStream_t stream);
// The synapses in target-major slots order[0 .. count) into the arrays.
void launch_unpack_synapses(const Engine& e, const uint32_t* order, uint64_t count, const SynapseArrays& out,
                            cudaStream_t stream);
// One-time kernel attributes (dynamic shared memory); call with
// the device current before the first tick.
void configure_kernels();
// Builds the synapse records from SynA images (`a`, S entries): code-pattern
// state zeroed, each synapse's `expected` stored.
void launch_init_syn(const Engine& e, const SynA* a, cudaStream_t stream);

}  // namespace snngb
