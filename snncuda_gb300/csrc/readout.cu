// Inference readouts of the GB300 backend: the reference inference
// session's one-hop feed-forward readout and its recurrent hidden/readout
// iteration (CudaInferenceSession::run_feedforward_batch and
// run_recurrent_feedforward_batch, CudaBackend.cu:1725-2100), over the
// Connectome's initial weights.
//
// The reference pushes every contribution with a float atomicAdd, so its
// sums come out in an unspecified order.  Here every sum is pulled by one
// thread in a fixed order -- a readout's (or hidden neuron's) incoming
// synapses in Connectome order, and the time steps in order -- so results
// are deterministic and equal to the same sums computed sequentially.
//
//   k_feedforward   a warp per (sample, readout): the sum over the readout's
//                   incoming synapses whose source is one of the sample's
//                   (merged) inputs of input weight x synapse weight
//   k_rows_*        the recurrent iteration's two edge lists (hidden ->
//                   readout and readout -> hidden), filtered out of the
//                   incoming lists once per call
//   k_recurrent     one block per sample running every time step: top-k of
//                   the hidden events, hidden -> readout propagation (delay
//                   d lands d steps later), readout gates (threshold or
//                   top-k), gated feedback readout -> hidden scaled by the
//                   feedback decay; the readout events summed over the steps

#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <string>
#include <type_traits>
#include <utility>
#include <vector>

#include "pack.h"
#include "snncuda_gb300.h"

namespace {

constexpr int kThreads = 256;
constexpr float kLowest = -3.402823466e+38F;

struct InEdges {
    const unsigned long long* ptr;  // [N+1]
    const uint32_t* src;
    const uint32_t* delay;           // max(1, delay_ticks)
    const float* w;                  // initial weight
};

// ---- one hop ---------------------------------------------------------------

constexpr uint32_t kNoNeuron = 0xFFFFFFFFu;
// Inputs of a sample a block's hash table takes (four slots per input, 8
// bytes each: 128 KB at this limit); larger samples search their sorted
// inputs in global memory.
constexpr uint32_t kHashInputs = 4096;

__host__ __device__ inline uint32_t hash_slots(uint32_t inputs) {
    uint32_t h = 64;
    while (h < 4 * inputs) h <<= 1;
    return h;
}
__device__ __forceinline__ uint32_t hash_of(uint32_t n, uint32_t mask) { return (n * 2654435761u >> 7) & mask; }

struct ForwardArgs {
    InEdges g;
    const unsigned long long* in_ptr;  // [samples + 1]
    const uint32_t* in_n;              // merged inputs (sorted by neuron when !hashed)
    const float* in_w;
    uint32_t R;
    uint32_t hashed;
    uint32_t samples;
    const uint32_t* readouts;
    const float* thresholds;
    float* scores;
    unsigned long long* spikes;
};

// Weight of neuron n among a sample's merged inputs (sorted by neuron), or 0.
__device__ __forceinline__ float input_weight(const uint32_t* nb, const float* wb, uint32_t m, uint32_t n) {
    uint32_t lo = 0, hi = m;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (nb[mid] < n) {
            lo = mid + 1;
        } else {
            hi = mid;
        }
    }
    return lo < m && nb[lo] == n ? wb[lo] : 0.0F;
}

// Bound by the latency of the synapse and table reads.  A block takes one
// sample and a share of the readouts, a warp per readout: a thread per readout
// walked its 500 synapses one after the other, each with a dependent binary
// search, and left the SM to 100 threads.  The lanes look up 32 synapses'
// sources at once in a hash table of the sample's inputs in shared memory (a
// quarter full: a source that is no input, the common case, ends at its first
// slot); the few contributions are then added in synapse order, as one thread
// would.  A call with 64 samples x 100 inputs and 100 readouts of 500 synapses
// went from 1.55 to 0.67 ms, together with the call's one copy each way; what
// is left is the conversion of the samples in Python.
//
// kThread: a thread per readout all the same (forward_by_thread).
template <bool kThread>
__global__ void __launch_bounds__(kThreads) k_feedforward(ForwardArgs a) {
    extern __shared__ uint32_t s_key[];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint32_t s = blockIdx.y; s < a.samples; s += gridDim.y) {
        const unsigned long long b = a.in_ptr[s];
        const uint32_t m = static_cast<uint32_t>(a.in_ptr[s + 1] - b);
        const uint32_t slots = hash_slots(m), mask = slots - 1;
        float* s_val = reinterpret_cast<float*>(s_key + slots);
        if (a.hashed) {
            __syncthreads();  // the previous sample's table is no longer read
            for (uint32_t i = threadIdx.x; i < slots; i += kThreads) s_key[i] = kNoNeuron;
            __syncthreads();
            for (uint32_t i = threadIdx.x; i < m; i += kThreads) {
                const uint32_t n = a.in_n[b + i];
                uint32_t at = hash_of(n, mask);
                while (atomicCAS(&s_key[at], kNoNeuron, n) != kNoNeuron) at = (at + 1) & mask;
                s_val[at] = a.in_w[b + i];
            }
            __syncthreads();
        }
        auto weight_of = [&](uint32_t src) {
            if (!a.hashed) return input_weight(a.in_n + b, a.in_w + b, m, src);
            uint32_t at = hash_of(src, mask), key;
            while ((key = s_key[at]) != kNoNeuron && key != src) at = (at + 1) & mask;
            return key == src ? s_val[at] : 0.0F;
        };
        auto put = [&](uint32_t r, float score) {
            a.scores[static_cast<size_t>(s) * a.R + r] = score;
            a.spikes[static_cast<size_t>(s) * a.R + r] = score >= a.thresholds[r] ? 1ull : 0ull;
        };
        if constexpr (kThread) {
            for (uint32_t r = blockIdx.x * kThreads + threadIdx.x; r < a.R; r += gridDim.x * kThreads) {
                const uint32_t n = a.readouts[r];
                const unsigned long long e1 = a.g.ptr[n + 1];
                float score = 0.0F;
                for (unsigned long long e = a.g.ptr[n]; e < e1; ++e) {
                    const float x = weight_of(a.g.src[e]);
                    if (x != 0.0F) score = __fadd_rn(score, __fmul_rn(x, a.g.w[e]));
                }
                put(r, score);
            }
        } else {
            for (uint32_t r = blockIdx.x * (kThreads / 32) + warp; r < a.R; r += gridDim.x * (kThreads / 32)) {
                const uint32_t n = a.readouts[r];
                const unsigned long long e0 = a.g.ptr[n], e1 = a.g.ptr[n + 1];
                float score = 0.0F;
                for (unsigned long long c = e0; c < e1; c += 32) {
                    const bool in = c + lane < e1;
                    const float x = in ? weight_of(a.g.src[c + lane]) : 0.0F;
                    const float v = x != 0.0F ? __fmul_rn(x, a.g.w[c + lane]) : 0.0F;
                    for (uint32_t hit = __ballot_sync(0xffffffffu, x != 0.0F); hit; hit &= hit - 1)
                        score = __fadd_rn(score, __shfl_sync(0xffffffffu, v, __ffs(hit) - 1));
                }
                if (lane == 0) put(r, score);
            }
        }
    }
}

// ---- recurrent iteration -----------------------------------------------------

// An edge of the recurrent iteration: its weight, its delay and the index of
// the event it reads (a hidden index, or a readout index).
struct alignas(16) RecEdge {
    float w;
    uint32_t delay;
    uint32_t from;
    uint32_t unused;
};

struct RecurrentArgs {
    InEdges g;
    uint32_t N, H, R, T, L, samples;
    const unsigned long long* in_ptr;  // [samples + 1] merged inputs
    const uint32_t* in_n;
    const float* in_w;
    const uint32_t* readouts;       // [R]
    const uint32_t* hidden;         // [H] dense neuron of each hidden index
    int* to_hidden;                 // [N] hidden index of a neuron, -1
    int* to_readout;                // [N] readout index of a neuron, -1
    const float* thresholds;        // [R]
    unsigned long long* row;        // [R + H + 1] first edge of each row: the readouts' rows, then the hidden ones'
    uint32_t* busy;                 // [H] hidden indices whose row is not empty, ascending
    uint32_t* busy_count;
    RecEdge* edge;
    // The events of steps t .. t + max_delay: step t's are in slot t mod L,
    // zero again once the step is done.
    float* hid;                     // [samples][L][H] hidden events
    float* out;                     // [samples][L][R] readout events
    float* gate;                    // [samples][R]
    float decay;
    uint32_t topk_readouts, topk_hidden;
    int use_scores;
    float* scores;                  // [samples][R]
    unsigned long long* spikes;     // [samples][R]
};

__global__ void k_index(RecurrentArgs a) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < a.H || i < a.R; i += gridDim.x * blockDim.x) {
        if (i < a.H) a.to_hidden[a.hidden[i]] = static_cast<int>(i);
        if (i < a.R) a.to_readout[a.readouts[i]] = static_cast<int>(i);
    }
}

// Row i's neuron, and whether its incoming synapse e belongs to the row: a
// readout's row takes the synapses from hidden neurons, a hidden neuron's row
// those from readouts.
__device__ __forceinline__ uint32_t row_neuron(const RecurrentArgs& a, uint32_t i) {
    return i < a.R ? a.readouts[i] : a.hidden[i - a.R];
}
__device__ __forceinline__ int row_from(const RecurrentArgs& a, uint32_t i, uint32_t src) {
    return i < a.R ? a.to_hidden[src] : a.to_readout[src];
}

// Edges of every row (row[i] = its count), a warp per row.
__global__ void __launch_bounds__(kThreads) k_rows_count(RecurrentArgs a) {
    const uint32_t lane = threadIdx.x & 31, rows = a.R + a.H;
    for (uint32_t i = (blockIdx.x * kThreads + threadIdx.x) >> 5; i < rows; i += gridDim.x * (kThreads / 32)) {
        const uint32_t n = row_neuron(a, i);
        uint32_t count = 0;
        for (unsigned long long e = a.g.ptr[n] + lane; e < a.g.ptr[n + 1]; e += 32)
            count += row_from(a, i, a.g.src[e]) >= 0;
        count = __reduce_add_sync(0xffffffffu, count);
        if (lane == 0) a.row[i] = count;
    }
}

constexpr int kScanThreads = 1024;

// Exclusive scan of the counts, and the list of hidden rows with edges; one
// block (each thread a run of consecutive rows).
__global__ void __launch_bounds__(kScanThreads) k_rows_scan(RecurrentArgs a) {
    __shared__ unsigned long long s_sum[kScanThreads];
    __shared__ uint32_t s_busy[kScanThreads];
    const uint32_t rows = a.R + a.H, per = (rows + kScanThreads - 1) / kScanThreads;
    const uint32_t b = min(rows, threadIdx.x * per), en = min(rows, b + per);
    unsigned long long sum = 0;
    uint32_t busy = 0;
    for (uint32_t i = b; i < en; ++i) {
        sum += a.row[i];
        busy += i >= a.R && a.row[i] > 0;
    }
    s_sum[threadIdx.x] = sum;
    s_busy[threadIdx.x] = busy;
    for (int d = 1; d < kScanThreads; d <<= 1) {
        __syncthreads();
        const unsigned long long x = threadIdx.x >= d ? s_sum[threadIdx.x - d] : 0ull;
        const uint32_t y = threadIdx.x >= d ? s_busy[threadIdx.x - d] : 0u;
        __syncthreads();
        s_sum[threadIdx.x] += x;
        s_busy[threadIdx.x] += y;
    }
    unsigned long long at = s_sum[threadIdx.x] - sum;
    uint32_t k = s_busy[threadIdx.x] - busy;
    for (uint32_t i = b; i < en; ++i) {
        const unsigned long long c = a.row[i];
        a.row[i] = at;
        at += c;
        if (i >= a.R && c > 0) a.busy[k++] = i - a.R;
    }
    if (threadIdx.x == kScanThreads - 1) {
        a.row[rows] = s_sum[threadIdx.x];
        *a.busy_count = s_busy[threadIdx.x];
    }
}

// The rows' edges, in synapse order; a warp per row.
__global__ void __launch_bounds__(kThreads) k_rows_fill(RecurrentArgs a) {
    const uint32_t lane = threadIdx.x & 31, rows = a.R + a.H;
    for (uint32_t i = (blockIdx.x * kThreads + threadIdx.x) >> 5; i < rows; i += gridDim.x * (kThreads / 32)) {
        unsigned long long at = a.row[i];
        if (at == a.row[i + 1]) continue;
        const uint32_t n = row_neuron(a, i);
        for (unsigned long long c = a.g.ptr[n]; c < a.g.ptr[n + 1]; c += 32) {
            const unsigned long long e = c + lane;
            const int from = e < a.g.ptr[n + 1] ? row_from(a, i, a.g.src[e]) : -1;
            const uint32_t mine = __ballot_sync(0xffffffffu, from >= 0);
            if (from >= 0)
                a.edge[at + __popc(mine & ((1u << lane) - 1u))] =
                    RecEdge{a.g.w[e], a.g.delay[e], static_cast<uint32_t>(from), 0u};
            at += __popc(mine);
        }
    }
}

constexpr int kRecThreads = 512;
constexpr int kRecWarps = kRecThreads / 32;

// Order of the values top-k picks by: larger is larger, -0 equals 0; 0 for a
// value that is never picked (not above the lowest finite one, or NaN).
__device__ __forceinline__ uint32_t order_key(float v) {
    if (!(v > kLowest)) return 0;
    const uint32_t u = v == 0.0F ? 0u : __float_as_uint(v);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ uint32_t block_sum(uint32_t v, uint32_t* s_part) {
    v = __reduce_add_sync(0xffffffffu, v);
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = v;
    __syncthreads();
    uint32_t t = 0;
    for (int i = 0; i < kRecWarps; ++i) t += s_part[i];
    __syncthreads();
    return t;
}

struct TopK {
    uint32_t key;    // entries with a larger order_key are picked,
    uint32_t equal;  // and the first `equal` entries with this one
    bool all;        // `equal` covers every entry with this key
};

// The k largest of v[0 .. n) (the first of equal values), whole block: the
// key of the k-th one by four 8-bit digits from the top, each a histogram in
// shared memory of the entries that share the digits found so far.
__device__ TopK top_k(const float* v, uint32_t n, uint32_t k, uint32_t* s_hist) {
    __shared__ uint32_t s_digit, s_left, s_in;
    uint32_t prefix = 0, left = k;
    for (int shift = 24; shift >= 0; shift -= 8) {
        for (uint32_t i = threadIdx.x; i < 256; i += kRecThreads) s_hist[i] = 0;
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < n; i += kRecThreads) {
            const uint32_t key = order_key(v[i]);
            if (key != 0 && (shift == 24 || key >> (shift + 8) == prefix)) atomicAdd(&s_hist[(key >> shift) & 255u], 1u);
        }
        __syncthreads();
        if (threadIdx.x < 32) {
            // lane l holds digits 255 - 8 l .. 248 - 8 l: the first digit
            // (from the top) at which the running count reaches `left`
            uint32_t sum = 0;
            for (int j = 0; j < 8; ++j) sum += s_hist[255 - 8 * threadIdx.x - j];
            uint32_t incl = sum;
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
                if (threadIdx.x >= d) incl += y;
            }
            const uint32_t reach = __ballot_sync(0xffffffffu, incl >= left);
            if (reach == 0) {
                if (threadIdx.x == 0) s_digit = 256;  // fewer than k entries can be picked
            } else if (threadIdx.x == __ffs(reach) - 1) {
                uint32_t before = incl - sum;
                int j = 0;
                while (before + s_hist[255 - 8 * threadIdx.x - j] < left) before += s_hist[255 - 8 * threadIdx.x - j++];
                s_digit = 255 - 8 * threadIdx.x - j;
                s_left = left - before;
                s_in = s_hist[s_digit];
            }
        }
        __syncthreads();
        const uint32_t digit = s_digit;
        if (digit == 256) {
            __syncthreads();
            return TopK{0u, 0u, true};  // every entry with a key is picked
        }
        prefix = (prefix << 8) | digit;
        left = s_left;
    }
    const bool all = s_in == left;
    __syncthreads();
    return TopK{prefix, left, all};
}

// f(i, picked) for every entry i of v[0 .. n), whole block.
template <typename F>
__device__ void for_picked(const float* v, uint32_t n, const TopK& p, uint32_t* s_part, F&& f) {
    uint32_t before = 0;  // entries with the boundary key ahead of this round's
    for (uint32_t i0 = 0; i0 < n; i0 += kRecThreads) {
        const uint32_t i = i0 + threadIdx.x;
        const uint32_t key = i < n ? order_key(v[i]) : 0u;
        bool pick = key > p.key;
        const bool tie = key != 0 && key == p.key;
        if (p.all) {
            pick = pick || tie;
        } else {
            // the boundary entries are picked in index order
            const uint32_t ties = __ballot_sync(0xffffffffu, tie);
            if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = __popc(ties);
            __syncthreads();
            uint32_t rank = before + __popc(ties & ((1u << (threadIdx.x & 31)) - 1u));
            for (uint32_t w = 0; w < kRecWarps; ++w) {
                if (w < threadIdx.x >> 5) rank += s_part[w];
                before += s_part[w];
            }
            __syncthreads();
            pick = pick || (tie && rank < p.equal);
        }
        if (i < n) f(i, pick);
    }
}

// Index of the largest of v[0 .. n) (the first of equal ones), n if none can
// be picked; whole block.
__device__ uint32_t top_one(const float* v, uint32_t n, unsigned long long* s_best) {
    unsigned long long best = 0;
    for (uint32_t i = threadIdx.x; i < n; i += kRecThreads) {
        const uint32_t key = order_key(v[i]);
        const unsigned long long x = (static_cast<unsigned long long>(key) << 32) | (0xFFFFFFFFu - i);
        if (key != 0 && x > best) best = x;
    }
    for (int d = 16; d > 0; d >>= 1) {
        const unsigned long long y = __shfl_xor_sync(0xffffffffu, best, d);
        best = y > best ? y : best;
    }
    if ((threadIdx.x & 31) == 0) s_best[threadIdx.x >> 5] = best;
    __syncthreads();
    for (int w = 0; w < kRecWarps; ++w) best = s_best[w] > best ? s_best[w] : best;
    __syncthreads();
    return best ? 0xFFFFFFFFu - static_cast<uint32_t>(best) : n;
}

// One block per sample, every time step inside (a step depends on the one
// before it: the length is steps x the latency of a step's phases, so each
// phase touches only what can be nonzero).  The first version let one thread
// pick the top k (k passes over the hidden events) and walked every incoming
// synapse of every hidden neuron at every step: a call with 32 samples on a
// 2,000-neuron network (101 steps, top 40 of 1,984 hidden neurons, 16
// readouts) went from 327 to 0.72 ms.  Contributions to one
// event are added in the same order: time steps in order, synapses in order
// within a step.
__global__ void __launch_bounds__(kRecThreads) k_recurrent(RecurrentArgs a) {
    __shared__ uint32_t s_hist[256], s_part[kRecWarps];
    __shared__ unsigned long long s_best[kRecWarps];
    const uint32_t s = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float* hid = a.hid + static_cast<size_t>(s) * a.L * a.H;
    float* out = a.out + static_cast<size_t>(s) * a.L * a.R;
    float* gate = a.gate + static_cast<size_t>(s) * a.R;
    float* scores = a.scores + static_cast<size_t>(s) * a.R;
    const uint32_t busy = *a.busy_count;
    const bool select = a.topk_hidden > 0 && a.topk_hidden < a.H;
    // hidden events of step 0: the merged inputs that are hidden neurons
    for (unsigned long long i = a.in_ptr[s] + threadIdx.x; i < a.in_ptr[s + 1]; i += kRecThreads) {
        const int h = a.to_hidden[a.in_n[i]];
        if (h >= 0) hid[h] = a.in_w[i];
    }
    for (uint32_t r = threadIdx.x; r < a.R; r += kRecThreads) scores[r] = 0.0F;
    __syncthreads();
    uint32_t slot = 0;  // t mod L
    for (uint32_t t = 0; t < a.T; ++t, slot = slot + 1 == a.L ? 0 : slot + 1) {
        float* ht = hid + static_cast<size_t>(slot) * a.H;
        float* ot = out + static_cast<size_t>(slot) * a.R;
        uint32_t pos = 0, zero = 0;
        for (uint32_t h = threadIdx.x; h < a.H; h += kRecThreads) {
            const float x = ht[h];
            pos += x > 0.0F;
            zero += x == 0.0F;
        }
        zero = block_sum(zero, s_part);
        const bool any = zero < a.H;  // some hidden event is not zero
        if (any && select) {
            pos = block_sum(pos, s_part);
            if (pos <= a.topk_hidden && pos + zero >= a.topk_hidden) {
                // every positive event is among the k largest, and zeros fill the rest
                for (uint32_t h = threadIdx.x; h < a.H; h += kRecThreads)
                    if (!(ht[h] > 0.0F)) ht[h] = 0.0F;
            } else {
                const TopK p = top_k(ht, a.H, a.topk_hidden, s_hist);
                for_picked(ht, a.H, p, s_part, [&](uint32_t h, bool pick) {
                    if (!pick) ht[h] = 0.0F;
                });
            }
            __syncthreads();
        }
        // hidden events of step t reach the readouts d steps later: a warp
        // per readout, 32 edges' events at once, the nonzero ones added in
        // edge order
        if (any) {
            for (uint32_t r = warp; r < a.R; r += kRecWarps) {
                const unsigned long long e1 = a.row[r + 1];
                for (unsigned long long c = a.row[r]; c < e1; c += 32) {
                    RecEdge e{};
                    float x = 0.0F;
                    if (c + lane < e1) {
                        e = a.edge[c + lane];
                        if (e.delay < a.T - t) x = ht[e.from];
                    }
                    const float v = __fmul_rn(x, e.w);
                    const uint32_t at = slot + e.delay >= a.L ? slot + e.delay - a.L : slot + e.delay;
                    for (uint32_t hit = __ballot_sync(0xffffffffu, x != 0.0F); hit; hit &= hit - 1) {
                        if (lane == __ffs(hit) - 1) {
                            float* o = out + static_cast<size_t>(at) * a.R + r;
                            *o = __fadd_rn(*o, v);
                        }
                        __syncwarp();
                    }
                }
            }
            __syncthreads();
        }
        // readout gates of step t
        if (a.topk_readouts == 0) {
            for (uint32_t r = threadIdx.x; r < a.R; r += kRecThreads)
                gate[r] = ot[r] >= a.thresholds[r] ? (a.use_scores ? ot[r] : 1.0F) : 0.0F;
        } else if (a.topk_readouts == 1) {
            const uint32_t best = top_one(ot, a.R, s_best);
            for (uint32_t r = threadIdx.x; r < a.R; r += kRecThreads)
                gate[r] = r == best ? (a.use_scores ? ot[r] : 1.0F) : 0.0F;
        } else {
            const TopK p = top_k(ot, a.R, a.topk_readouts, s_hist);
            for_picked(ot, a.R, p, s_part, [&](uint32_t r, bool pick) {
                gate[r] = pick ? (a.use_scores ? ot[r] : 1.0F) : 0.0F;
            });
        }
        bool open = false;
        for (uint32_t r = threadIdx.x; r < a.R; r += kRecThreads) {
            open = open || gate[r] != 0.0F;  // the thread's own entries
            scores[r] = __fadd_rn(scores[r], ot[r]);
            ot[r] = 0.0F;
        }
        open = __syncthreads_or(open);
        if (any)
            for (uint32_t h = threadIdx.x; h < a.H; h += kRecThreads) ht[h] = 0.0F;
        // gated readouts feed back to the hidden neurons d steps later: a
        // thread per hidden neuron with an edge from a readout
        if (open) {
            for (uint32_t k = threadIdx.x; k < busy; k += kRecThreads) {
                const uint32_t h = a.busy[k];
                for (unsigned long long c = a.row[a.R + h]; c < a.row[a.R + h + 1]; ++c) {
                    const RecEdge e = a.edge[c];
                    const float gr = gate[e.from];
                    if (gr == 0.0F || e.delay >= a.T - t) continue;
                    const uint32_t at = slot + e.delay >= a.L ? slot + e.delay - a.L : slot + e.delay;
                    float* y = hid + static_cast<size_t>(at) * a.H + h;
                    *y = __fadd_rn(*y, __fmul_rn(__fmul_rn(a.decay, gr), e.w));
                }
            }
        }
        __syncthreads();
    }
    for (uint32_t r = threadIdx.x; r < a.R; r += kRecThreads)
        a.spikes[static_cast<size_t>(s) * a.R + r] = scores[r] >= a.thresholds[r] ? 1ull : 0ull;
}

struct Fail {
    int code;
    std::string msg;
};

void check(cudaError_t err, const char* what) {
    if (err == cudaSuccess) return;
    const int code = err == cudaErrorMemoryAllocation ? SNNCUDA_ERR_OUT_OF_MEMORY : SNNCUDA_ERR_DEVICE;
    cudaGetLastError();
    throw Fail{code, std::string(what) + ": " + cudaGetErrorString(err)};
}

// A sample's inputs merged per neuron (weights of one neuron summed in input
// order), in the order of their first appearance, or sorted by neuron.
struct MergedInputs {
    std::vector<unsigned long long> ptr;
    std::vector<uint32_t> n;
    std::vector<float> w;
    uint32_t most{0};  // inputs of the largest sample
};

MergedInputs merge_inputs(uint32_t samples, const uint64_t* ptr, const uint32_t* neurons, const float* weights,
                          uint32_t N, uint64_t* delivered) {
    MergedInputs m;
    m.ptr.assign(static_cast<size_t>(samples) + 1, 0);
    std::vector<uint32_t> seen(N, 0), place(N, 0);  // sample + 1 that last used the neuron, and where
    for (uint32_t s = 0; s < samples; ++s) {
        const size_t first = m.n.size();
        for (uint64_t i = ptr[s]; i < ptr[s + 1]; ++i) {
            const uint32_t n = neurons[i];
            if (n >= N) throw Fail{SNNCUDA_ERR_INVALID_ARGUMENT, "input neuron out of range"};
            if (seen[n] == s + 1) {
                m.w[place[n]] = m.w[place[n]] + weights[i];
            } else {
                seen[n] = s + 1;
                place[n] = static_cast<uint32_t>(m.n.size());
                m.n.push_back(n);
                m.w.push_back(0.0F + weights[i]);
            }
        }
        const size_t count = m.n.size() - first;
        m.most = std::max(m.most, static_cast<uint32_t>(count));
        m.ptr[s + 1] = m.n.size();
        if (delivered) delivered[s] = count;
    }
    return m;
}

void sort_inputs(MergedInputs& m) {
    std::vector<std::pair<uint32_t, float>> v;
    for (size_t s = 0; s + 1 < m.ptr.size(); ++s) {
        v.clear();
        for (unsigned long long i = m.ptr[s]; i < m.ptr[s + 1]; ++i) v.emplace_back(m.n[i], m.w[i]);
        std::sort(v.begin(), v.end(), [](const auto& x, const auto& y) { return x.first < y.first; });
        for (size_t i = 0; i < v.size(); ++i) {
            m.n[m.ptr[s] + i] = v[i].first;
            m.w[m.ptr[s] + i] = v[i].second;
        }
    }
}

}  // namespace

struct snncuda_readout {
    uint32_t N{0};
    std::vector<float> threshold;
    uint32_t max_delay{1};
    unsigned long long* ptr{nullptr};
    uint32_t* src{nullptr};
    uint32_t* delay{nullptr};
    float* w{nullptr};
    std::vector<uint64_t> degree;  // [N] incoming plus outgoing synapses
    std::vector<unsigned long long> in_ptr;  // [N+1] ptr's contents
    // A call's device buffers are carved out of one that the handle keeps
    // (grown when a call needs more, freed with the handle, or after the call if
    // it is larger than the handle may keep: 256 MB, 64 MB pinned), and its inputs
    // and results pass through one pinned host buffer: a call is one copy to
    // the device, its kernels and one copy back.  One call at a time has them.
    std::mutex in_use;
    unsigned char* work{nullptr};
    size_t work_bytes{0};
    unsigned char* host{nullptr};
    size_t host_bytes{0};
    ~snncuda_readout() {
        cudaFree(ptr);
        cudaFree(src);
        cudaFree(delay);
        cudaFree(w);
        cudaFree(work);
        if (host) cudaFreeHost(host);
    }
    InEdges edges() const { return InEdges{ptr, src, delay, w}; }
    void trim() {
        if (work_bytes > (256u << 20)) {
            cudaFree(work);
            work = nullptr;
            work_bytes = 0;
        }
        if (host_bytes > (64u << 20)) {
            cudaFreeHost(host);
            host = nullptr;
            host_bytes = 0;
        }
    }
    void need(size_t device_bytes, size_t pinned_bytes) {
        if (device_bytes > work_bytes) {
            cudaFree(work);
            work = nullptr;
            work_bytes = 0;
            check(cudaMalloc(reinterpret_cast<void**>(&work), device_bytes), "device allocation");
            work_bytes = device_bytes;
        }
        if (pinned_bytes > host_bytes) {
            if (host) cudaFreeHost(host);
            host = nullptr;
            host_bytes = 0;
            check(cudaMallocHost(reinterpret_cast<void**>(&host), pinned_bytes), "pinned staging");
            host_bytes = pinned_bytes;
        }
    }
};

namespace {

int fail_code(const Fail& f) {
    snngb::set_last_error_message(f.msg);
    return f.code;
}

// A call on a handle: no other at the same time, large buffers given back.
struct Call {
    snncuda_readout* r;
    std::lock_guard<std::mutex> lock{r->in_use};
    ~Call() { r->trim(); }
};

// Places of a call's arrays in the handle's buffers, each 256-byte aligned:
// the inputs (copied from the pinned buffer, where they have the same
// offsets), then the results, then what only the kernels use.
struct Layout {
    size_t at{0};
    size_t take(size_t bytes) {
        const size_t here = at;
        at = (at + std::max<size_t>(bytes, 1) + 255) & ~static_cast<size_t>(255);
        return here;
    }
    template <typename T>
    size_t array(size_t count) {
        return take(count * sizeof(T));
    }
};

template <typename T>
void stage(snncuda_readout* r, size_t at, const std::vector<T>& v) {
    if (!v.empty()) std::memcpy(r->host + at, v.data(), v.size() * sizeof(T));
}
template <typename T>
T* placed(snncuda_readout* r, size_t at) {
    return reinterpret_cast<T*>(r->work + at);
}

// Results up to this size come back through the pinned buffer: one copy, and
// nothing to map in arrays that the caller has just allocated (100 x 100 results
// 87 us a call, copied directly 143; 300 x 300 both 235).  Larger ones would only
// be moved twice (4,096 x 4,096: 22.6 ms, directly 11.4).
constexpr size_t kStagedResults = 1u << 20;

// The results [res, end) of the work buffer to the caller's arrays.
void fetch_results(snncuda_readout* r, size_t res, size_t spikes_at, size_t end, size_t count, float* scores,
                   uint64_t* spikes) {
    if (end - res > kStagedResults) {
        check(cudaMemcpyAsync(scores, r->work + res, count * sizeof(float), cudaMemcpyDeviceToHost), "copy");
        check(cudaMemcpyAsync(spikes, r->work + spikes_at, count * sizeof(uint64_t), cudaMemcpyDeviceToHost), "copy");
        check(cudaStreamSynchronize(nullptr), "readout synchronize");
        return;
    }
    check(cudaMemcpyAsync(r->host + res, r->work + res, end - res, cudaMemcpyDeviceToHost), "copy");
    check(cudaStreamSynchronize(nullptr), "readout synchronize");
    std::memcpy(scores, r->host + res, count * sizeof(float));
    std::memcpy(spikes, r->host + spikes_at, count * sizeof(uint64_t));
}

// Whether a call's `results` (samples x readouts) take a thread each rather than
// a warp: with enough of them to fill the GPU, and readouts of few synapses, whose
// rows leave most of a warp's lanes idle.  1e6 results of 10 synapses 30 us by
// threads, 239 by warps, 8.4e6 of 300 4.1 and 4.2 ms; 6,400 of 40 22 and 6 us.
bool forward_by_thread(size_t results, uint64_t synapses) { return results >= (1u << 18) && synapses <= 256; }

// Pinned bytes of a call whose inputs are [0, res) and results [res, end).
size_t pinned_bytes(size_t res, size_t end) { return end - res > kStagedResults ? res : end; }

// Readout neurons and their thresholds; rejects repeats.
void readout_list(const snncuda_readout* r, uint32_t count, const uint32_t* neurons, std::vector<uint32_t>& list,
                  std::vector<float>& thr) {
    std::vector<char> seen(r->N, 0);
    for (uint32_t i = 0; i < count; ++i) {
        if (neurons[i] >= r->N) throw Fail{SNNCUDA_ERR_INVALID_ARGUMENT, "neuron out of range"};
        if (seen[neurons[i]]) throw Fail{SNNCUDA_ERR_INVALID_ARGUMENT, "a neuron is listed twice"};
        seen[neurons[i]] = 1;
        list.push_back(neurons[i]);
        thr.push_back(r->threshold[neurons[i]]);
    }
}

}  // namespace

extern "C" {

int snncuda_readout_create(const snncuda_network* net, snncuda_readout** out) {
    if (net == nullptr || out == nullptr) return SNNCUDA_ERR_INVALID_ARGUMENT;
    snncuda_readout* r = new (std::nothrow) snncuda_readout();
    if (r == nullptr) return SNNCUDA_ERR_OUT_OF_MEMORY;
    int code = SNNCUDA_OK;
    try {
        const uint32_t N = net->neuron_count;
        const uint64_t S = net->synapse_count;
        if (N > 0 && net->threshold == nullptr) throw Fail{SNNCUDA_ERR_INVALID_ARGUMENT, "thresholds are required"};
        if (S > 0 && (!net->source || !net->target || !net->weight || !net->delay_ticks))
            throw Fail{SNNCUDA_ERR_INVALID_ARGUMENT, "synapse arrays are required"};
        r->N = N;
        r->degree.assign(N, 0);
        r->threshold.assign(net->threshold, net->threshold + N);
        // incoming synapses of each neuron in Connectome order (stable
        // counting sort by target)
        std::vector<unsigned long long> ptr(static_cast<size_t>(N) + 1, 0);
        uint64_t run = 0;  // first synapse of the current run of one source
        for (uint64_t k = 0; k < S; ++k) {
            if (net->source[k] >= N || net->target[k] >= N)
                throw Fail{SNNCUDA_ERR_INVALID_ARGUMENT, "synapse endpoint out of range"};
            ++ptr[net->target[k] + 1];
            // synapses usually come source by source: one update a run
            if (k > 0 && net->source[k] != net->source[run]) {
                r->degree[net->source[run]] += k - run;
                run = k;
            }
        }
        if (S > 0) r->degree[net->source[run]] += S - run;
        for (uint32_t n = 0; n < N; ++n) {
            r->degree[n] += ptr[n + 1];  // still the count of n's incoming synapses
            ptr[n + 1] += ptr[n];
        }
        std::vector<unsigned long long> fill(ptr.begin(), ptr.end() - 1);
        std::vector<uint32_t> src(S), dly(S);
        std::vector<float> w(S);
        for (uint64_t k = 0; k < S; ++k) {
            const unsigned long long at = fill[net->target[k]]++;
            src[at] = net->source[k];
            dly[at] = std::max(1u, net->delay_ticks[k]);
            w[at] = net->weight[k];
            r->max_delay = std::max(r->max_delay, dly[at]);
        }
        auto upload = [](auto*& d, const auto& v) {
            using T = std::remove_reference_t<decltype(v[0])>;
            check(cudaMalloc(reinterpret_cast<void**>(&d), std::max<size_t>(v.size(), 1) * sizeof(T)), "device allocation");
            if (!v.empty()) check(cudaMemcpy(d, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice), "copy");
        };
        upload(r->ptr, ptr);
        upload(r->src, src);
        upload(r->delay, dly);
        upload(r->w, w);
        r->in_ptr = std::move(ptr);
    } catch (const Fail& f) {
        code = fail_code(f);
    } catch (const std::bad_alloc&) {
        snngb::set_last_error_message("host allocation failed");
        code = SNNCUDA_ERR_OUT_OF_MEMORY;
    }
    if (code != SNNCUDA_OK) {
        delete r;
        return code;
    }
    *out = r;
    return SNNCUDA_OK;
}

int snncuda_readout_destroy(snncuda_readout* r) {
    delete r;
    return SNNCUDA_OK;
}

int snncuda_readout_feedforward(snncuda_readout* r, uint32_t samples, const uint64_t* input_ptr,
                                const uint32_t* input_neurons, const float* input_weights, uint32_t readout_count,
                                const uint32_t* readout_neurons, float* scores, uint64_t* spikes,
                                uint64_t* delivered) {
    if (r == nullptr || (samples > 0 && input_ptr == nullptr)) return SNNCUDA_ERR_INVALID_ARGUMENT;
    int code = SNNCUDA_OK;
    const Call call{r};
    try {
        if (delivered) std::fill(delivered, delivered + samples, 0);
        if (samples == 0 || readout_count == 0) return SNNCUDA_OK;
        std::vector<uint32_t> list;
        std::vector<float> thr;
        readout_list(r, readout_count, readout_neurons, list, thr);
        MergedInputs m = merge_inputs(samples, input_ptr, input_neurons, input_weights, r->N, delivered);
        ForwardArgs a{};
        a.hashed = m.most <= kHashInputs;
        if (!a.hashed) sort_inputs(m);
        const size_t count = static_cast<size_t>(samples) * readout_count;
        Layout l;
        const size_t o_ptr = l.array<unsigned long long>(m.ptr.size()), o_n = l.array<uint32_t>(m.n.size()),
                     o_w = l.array<float>(m.w.size()), o_list = l.array<uint32_t>(list.size()),
                     o_thr = l.array<float>(thr.size());
        const size_t res = l.at, o_scores = l.array<float>(count), o_spikes = l.array<unsigned long long>(count);
        r->need(l.at, pinned_bytes(res, l.at));
        stage(r, o_ptr, m.ptr);
        stage(r, o_n, m.n);
        stage(r, o_w, m.w);
        stage(r, o_list, list);
        stage(r, o_thr, thr);
        check(cudaMemcpyAsync(r->work, r->host, res, cudaMemcpyHostToDevice), "copy");
        a.g = r->edges();
        a.in_ptr = placed<unsigned long long>(r, o_ptr);
        a.in_n = placed<uint32_t>(r, o_n);
        a.in_w = placed<float>(r, o_w);
        a.R = readout_count;
        a.samples = samples;
        a.readouts = placed<uint32_t>(r, o_list);
        a.thresholds = placed<float>(r, o_thr);
        a.scores = placed<float>(r, o_scores);
        a.spikes = placed<unsigned long long>(r, o_spikes);
        const size_t smem = a.hashed ? hash_slots(m.most) * 8ull : 0;
        uint64_t synapses = 0;
        for (uint32_t n : list) synapses += r->in_ptr[n + 1] - r->in_ptr[n];
        const bool by_thread = forward_by_thread(count, synapses / readout_count);
        auto* kernel = by_thread ? k_feedforward<true> : k_feedforward<false>;
        check(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   static_cast<int>(hash_slots(kHashInputs) * 8)),
              "feedforward attribute");
        const uint32_t each = by_thread ? kThreads : kThreads / 32;  // readouts of a block at a time
        const uint32_t share = std::min(65535u, (readout_count + each - 1) / each);
        kernel<<<dim3(share, std::min(65535u, samples)), kThreads, smem>>>(a);
        check(cudaGetLastError(), "feedforward launch");
        fetch_results(r, res, o_spikes, l.at, count, scores, spikes);
    } catch (const Fail& f) {
        code = fail_code(f);
    } catch (const std::bad_alloc&) {
        snngb::set_last_error_message("host allocation failed");
        code = SNNCUDA_ERR_OUT_OF_MEMORY;
    }
    return code;
}

void snncuda_recurrent_options_default(snncuda_recurrent_options* o) {
    if (o == nullptr) return;
    std::memset(o, 0, sizeof(*o));
    o->iterations = 1;
    o->feedback_decay = 0.5F;
    o->top_k_feedback_readouts = 1;
    o->top_k_hidden = 0;
    o->use_scores_not_spikes = 1;
}

int snncuda_readout_recurrent(snncuda_readout* r, uint32_t samples, const uint64_t* input_ptr,
                              const uint32_t* input_neurons, const float* input_weights, uint32_t readout_count,
                              const uint32_t* readout_neurons, uint32_t hidden_count, const uint32_t* hidden_neurons,
                              const snncuda_recurrent_options* options, float* scores, uint64_t* spikes,
                              uint64_t* delivered, uint64_t* time_steps) {
    if (r == nullptr || options == nullptr || (samples > 0 && input_ptr == nullptr))
        return SNNCUDA_ERR_INVALID_ARGUMENT;
    int code = SNNCUDA_OK;
    const Call call{r};
    try {
        if (delivered) std::fill(delivered, delivered + samples, 0);
        const uint64_t T = static_cast<uint64_t>(r->max_delay) * (1 + 2ull * options->iterations) + 1;
        if (time_steps) *time_steps = T;
        if (samples == 0 || readout_count == 0) return SNNCUDA_OK;
        std::vector<uint32_t> rl, hl;
        std::vector<float> thr, hthr;
        readout_list(r, readout_count, readout_neurons, rl, thr);
        if (hidden_count > 0) {
            readout_list(r, hidden_count, hidden_neurons, hl, hthr);
        } else {  // every neuron that is not a readout, in index order
            std::vector<char> is_readout(r->N, 0);
            for (uint32_t n : rl) is_readout[n] = 1;
            for (uint32_t n = 0; n < r->N; ++n)
                if (!is_readout[n]) hl.push_back(n);
        }
        const uint32_t H = static_cast<uint32_t>(hl.size());
        if (H == 0) return SNNCUDA_OK;
        if (T > (1u << 20)) throw Fail{SNNCUDA_ERR_UNSUPPORTED, "more than 2^20 time steps"};
        const MergedInputs m = merge_inputs(samples, input_ptr, input_neurons, input_weights, r->N, delivered);
        const size_t count = static_cast<size_t>(samples) * readout_count;
        const size_t L = static_cast<size_t>(r->max_delay) + 1, rows = static_cast<size_t>(H) + readout_count;
        size_t edges = 0;  // at most: every edge ends at a readout or starts at one
        for (uint32_t n : rl) edges += r->degree[n];
        Layout l;
        const size_t o_ptr = l.array<unsigned long long>(m.ptr.size()), o_n = l.array<uint32_t>(m.n.size()),
                     o_w = l.array<float>(m.w.size()), o_rl = l.array<uint32_t>(rl.size()),
                     o_hl = l.array<uint32_t>(hl.size()), o_thr = l.array<float>(thr.size());
        const size_t res = l.at, o_scores = l.array<float>(count), o_spikes = l.array<unsigned long long>(count);
        const size_t end = l.at;
        const size_t o_map = l.array<int>(2 * static_cast<size_t>(r->N)), o_row = l.array<unsigned long long>(rows + 1),
                     o_busy = l.array<uint32_t>(static_cast<size_t>(H) + 1), o_edge = l.array<RecEdge>(edges);
        const size_t zeroed = l.at, o_hid = l.array<float>(samples * L * H),
                     o_out = l.array<float>(samples * L * readout_count), o_gate = l.array<float>(count);
        r->need(l.at, pinned_bytes(res, end));
        stage(r, o_ptr, m.ptr);
        stage(r, o_n, m.n);
        stage(r, o_w, m.w);
        stage(r, o_rl, rl);
        stage(r, o_hl, hl);
        stage(r, o_thr, thr);
        RecurrentArgs a{};
        a.g = r->edges();
        a.N = r->N;
        a.H = H;
        a.R = readout_count;
        a.T = static_cast<uint32_t>(T);
        a.L = static_cast<uint32_t>(L);
        a.samples = samples;
        a.in_ptr = placed<unsigned long long>(r, o_ptr);
        a.in_n = placed<uint32_t>(r, o_n);
        a.in_w = placed<float>(r, o_w);
        a.readouts = placed<uint32_t>(r, o_rl);
        a.hidden = placed<uint32_t>(r, o_hl);
        a.to_hidden = placed<int>(r, o_map);
        a.to_readout = a.to_hidden + r->N;
        a.thresholds = placed<float>(r, o_thr);
        a.row = placed<unsigned long long>(r, o_row);
        a.busy = placed<uint32_t>(r, o_busy);
        a.busy_count = a.busy + H;
        a.edge = placed<RecEdge>(r, o_edge);
        a.hid = placed<float>(r, o_hid);
        a.out = placed<float>(r, o_out);
        a.gate = placed<float>(r, o_gate);
        a.decay = options->feedback_decay;
        a.topk_readouts = options->top_k_feedback_readouts;
        a.topk_hidden = options->top_k_hidden;
        a.use_scores = options->use_scores_not_spikes ? 1 : 0;
        a.scores = placed<float>(r, o_scores);
        a.spikes = placed<unsigned long long>(r, o_spikes);
        check(cudaMemcpyAsync(r->work, r->host, res, cudaMemcpyHostToDevice), "copy");
        check(cudaMemsetAsync(a.to_hidden, 0xFF, 2 * sizeof(int) * r->N), "memset");
        check(cudaMemsetAsync(r->work + zeroed, 0, l.at - zeroed), "memset");
        const uint32_t wide = static_cast<uint32_t>(std::min<size_t>(4096, (rows + kThreads / 32 - 1) / (kThreads / 32)));
        k_index<<<static_cast<uint32_t>(std::min<size_t>(1024, (rows + kThreads - 1) / kThreads)), kThreads>>>(a);
        k_rows_count<<<wide, kThreads>>>(a);
        k_rows_scan<<<1, kScanThreads>>>(a);
        k_rows_fill<<<wide, kThreads>>>(a);
        k_recurrent<<<samples, kRecThreads>>>(a);
        check(cudaGetLastError(), "recurrent launch");
        fetch_results(r, res, o_spikes, end, count, scores, spikes);
    } catch (const Fail& f) {
        code = fail_code(f);
    } catch (const std::bad_alloc&) {
        snngb::set_last_error_message("host allocation failed");
        code = SNNCUDA_ERR_OUT_OF_MEMORY;
    }
    return code;
}

}  // extern "C"
