// Sampling on the device: greedy argmax, and temperature sampling with optional top-k / top-p.
//
// Semantics of the reference sampler (src/sampler/sampler.h:3-27, src/sampler/sampler.cpp:55-129):
//   greedy: the largest logit, the lowest index among equals;
//   otherwise p_i = exp((logit_i - max) / temperature) * (float)(1 / sum), sum in double;
//   top-k keeps the k most likely tokens (probability descending, index ascending among equals),
//   top-p then keeps the shortest prefix of that order whose mass reaches top_p * (kept mass);
//   the draw returns the first kept token, in that order (index order when no filter is on),
//   whose cumulative probability exceeds u * (kept mass).
// The uniform number u of every row comes from the caller (the per-request xorshift64* stream is
// kept on the host so that a request's stream does not depend on the batch it is in).
//
// The sorted order is never materialised. A position in it (the k-th token, the place where the
// cumulative mass crosses a threshold) is found by a radix descent over the bits of the
// probabilities: histograms of counts and of exact masses per 10-bit digit, three
// passes, then index order inside the last group of equal probabilities. One cluster of CTAs per row.
#include <climits>
#include <type_traits>

#include <cooperative_groups.h>

#include "common.cuh"

namespace gi {

namespace cg = cooperative_groups;

constexpr int kSampleThreads = 1024;

// Greedy argmax in two steps: kArgmaxParts blocks per row each find the best of a slice of the
// vocabulary (lowest index among equals), then one block per row picks among the slice winners.
// One block per row would read 0.5 MB through a single SM.
constexpr int kArgmaxParts = 32;

__device__ __forceinline__ void argmax_block_reduce(float& best, int& best_i, float* s_val, int* s_idx) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
        if (ov > best || (ov == best && oi < best_i)) { best = ov; best_i = oi; }
    }
    if (lane == 0) { s_val[warp] = best; s_idx[warp] = best_i; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (blockDim.x >> 5); ++w) {
            if (s_val[w] > best || (s_val[w] == best && s_idx[w] < best_i)) { best = s_val[w]; best_i = s_idx[w]; }
        }
    }
}

// grid (kArgmaxParts, rows): the best of one slice -> part_val / part_idx [rows, kArgmaxParts]
__global__ void __launch_bounds__(256)
argmax_partial_kernel(const float* __restrict__ logits, int V, float* __restrict__ part_val, int* __restrict__ part_idx) {
    pdl_prologue();
    __shared__ float s_val[8];
    __shared__ int s_idx[8];
    const float* row = logits + static_cast<size_t>(blockIdx.y) * V;
    const int per = (V + kArgmaxParts - 1) / kArgmaxParts;
    const int begin = blockIdx.x * per, end = min(V, begin + per);
    float best = -INFINITY;
    int best_i = 0x7fffffff;
    for (int i = begin + threadIdx.x; i < end; i += 256) {
        const float v = row[i];
        if (v > best || best_i == 0x7fffffff) { best = v; best_i = i; }   // increasing i: ties keep the lower index
    }
    argmax_block_reduce(best, best_i, s_val, s_idx);
    if (threadIdx.x == 0) {
        part_val[blockIdx.y * kArgmaxParts + blockIdx.x] = best;
        part_idx[blockIdx.y * kArgmaxParts + blockIdx.x] = best_i;
    }
}

// one warp per row
__global__ void __launch_bounds__(32)
argmax_final_kernel(const float* __restrict__ part_val, const int* __restrict__ part_idx, int* __restrict__ out) {
    pdl_prologue();
    float best = part_val[blockIdx.x * kArgmaxParts + threadIdx.x];
    int best_i = part_idx[blockIdx.x * kArgmaxParts + threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
        if (ov > best || (ov == best && oi < best_i)) { best = ov; best_i = oi; }
    }
    if (threadIdx.x == 0) out[blockIdx.x] = best_i == 0x7fffffff ? 0 : best_i;
}

// ---- temperature sampling: one cluster of kSampleParts CTAs per row ----
//
// A row is bound by latency, not by its bytes (0.5 MB at a vocabulary of 128,256, read once from memory and a few times from
// L1): one block of 1024 threads per row took 1,560 us for six rows, most of it in double-precision atomics on
// histograms in shared memory (loops of compare-and-swap, all on the few digits that the exponents have) and in loops of one
// thread over 1024 ranges. Here eight CTAs share a row, every warp owns a contiguous piece of it, and a histogram's masses
// are integers: the values of one bin have one exponent, so their sum is a sum of 24-bit mantissas, added exactly in two
// 32-bit words by the hardware's integer atomics: 90 us for the same rows.
constexpr int kSampleParts = 8, kBins = 1024, kDigit = 10;
constexpr int kMassBits = 12;                  // a mantissa goes into two words of 12 bits: slices of up to 2^20 values cannot overflow them
constexpr int kNarrowVocab = kSampleParts << 20;      // above: whole mantissas in 64-bit words (whose atomics are slower)

// A warp's piece stays in registers, up to 16 values a lane, where it fits (vocabularies of up to 131,072): read once instead of
// in every pass, each a wait for L2 (six rows of 128,256, drawn with every kind of filter: 92 -> 62 us).
constexpr int kHeldMost = 16, kHeldFew = 4;       // (vocabularies of up to 32,768: places without a value cost time, too: forty rows of 1,000 31.2 -> 24.7 us)

template <bool kWide> struct SampleShared {
    using Low = typename std::conditional<kWide, unsigned long long, unsigned>::type;
    static constexpr int kSets = kWide ? 2 : 3;      // histograms of this CTA's piece: two sets take turns, the third keeps the
    unsigned count[kSets][kBins];                    // first pass, which is the same for every descent of a row
    Low low[kSets][kBins];
    unsigned high[kSets][kBins];
    double cta_max, cta_sum, cta_mass;         // each written once and read by the cluster behind its own barrier
    int cta_equal;
    double warp_mass[32];
    double red[32];
    int counts[32];
    double scan_mass[32];
    int scan_count[32];
    int first, last;                           // positions of the bin chosen
    double chosen_mass;
    int chosen_count;
};

// What a descent has found: the value's bits, what is strictly above it, and how many values equal it.
struct Found {
    unsigned bits;
    double mass_above;
    int count_above, equal;
};

__device__ __forceinline__ unsigned long long sample_mantissa(unsigned bits) {
    return (bits & 0x7fffffu) | ((bits >> 23) ? 0x800000u : 0u);
}
__device__ __forceinline__ double sample_scale(unsigned bits) {                    // the weight of the mantissa's last bit
    const int e = static_cast<int>((bits >> 23) & 255u);
    return ldexp(1.0, (e > 0 ? e : 1) - 150);
}

__device__ __forceinline__ double warp_sum_double(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// Sum over the block in the order of the warps; each thread has it.
__device__ __forceinline__ double block_sum_double(double v, double* scratch) {
    v = warp_sum_double(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = v;
    __syncthreads();
    double total = 0.0;
    for (int w = 0; w < kSampleThreads / 32; ++w) total += scratch[w];
    return total;
}

// Walks the row's values from the largest downwards, ten bits of them per pass (values are at most 1: 30 bits): in each pass
// the bin is chosen in which the running total (of ones if by_count, else of probabilities) first reaches (inclusive) or
// exceeds the target. Where rounding never lets it, the lowest bin that weighs anything is chosen.
// `each` calls its argument with every place and value of the calling warp's piece. `turn` counts the passes that take turns with the
// histograms, `descents` the row's descents.
template <bool kWide, typename Each>
__device__ __forceinline__ Found sample_descend(const Each& each, bool by_count, double target, bool inclusive,
                                SampleShared<kWide>& s, int& turn, int& descents, cg::cluster_group& cluster) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Found f{0u, 0.0, 0, 0};
    unsigned mask = 0u;
    for (int shift = 20; shift >= 0; shift -= kDigit) {
        const bool first_pass = !kWide && shift == 20;
        const int set = first_pass ? SampleShared<kWide>::kSets - 1 : turn++ & 1;
        const bool fill = !(first_pass && descents > 0);
        if (fill) {
            s.count[set][threadIdx.x] = 0u;
            s.low[set][threadIdx.x] = 0u;
            s.high[set][threadIdx.x] = 0u;
        }
        if (threadIdx.x == 0) { s.first = kBins; s.last = -1; }
        __syncthreads();
        if (fill) {
            each([&](int, float value) {
                const unsigned bits = __float_as_uint(value);
                if ((bits & mask) == f.bits) {
                    const unsigned digit = (bits >> shift) & (kBins - 1);
                    const unsigned m = static_cast<unsigned>(sample_mantissa(bits));
                    atomicAdd(&s.count[set][digit], 1u);
                    if constexpr (kWide) {
                        atomicAdd(&s.low[set][digit], static_cast<unsigned long long>(m));
                    } else {
                        atomicAdd(&s.low[set][digit], m & ((1u << kMassBits) - 1));
                        atomicAdd(&s.high[set][digit], m >> kMassBits);
                    }
                }
            });
            cluster.sync();
        }
        // thread t has the t-th bin from the top: its totals over the cluster, then a scan over the block
        const int bin = kBins - 1 - threadIdx.x;
        unsigned long long low = 0, high = 0;
        int count = 0;
#pragma unroll
        for (int p = 0; p < kSampleParts; ++p) {
            count += static_cast<int>(*cluster.map_shared_rank(&s.count[set][bin], p));
            low += *cluster.map_shared_rank(&s.low[set][bin], p);
            high += *cluster.map_shared_rank(&s.high[set][bin], p);
        }
        const double mass = static_cast<double>(low + (high << kMassBits)) * sample_scale(f.bits | (static_cast<unsigned>(bin) << shift));
        double run = mass;
        int runs = count;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double m = __shfl_up_sync(0xffffffffu, run, o);
            const int c = __shfl_up_sync(0xffffffffu, runs, o);
            if (lane >= o) { run += m; runs += c; }
        }
        if (lane == 31) { s.scan_mass[warp] = run; s.scan_count[warp] = runs; }
        __syncthreads();
        double ahead = f.mass_above;
        int aheads = f.count_above;
        for (int w = 0; w < warp; ++w) { ahead += s.scan_mass[w]; aheads += s.scan_count[w]; }
        run += ahead;
        runs += aheads;
        const bool weighs = by_count ? count > 0 : mass > 0.0;
        const double total = by_count ? static_cast<double>(runs) : run;
        if (weighs && (inclusive ? total >= target : total > target)) atomicMin(&s.first, static_cast<int>(threadIdx.x));
        if (weighs) atomicMax(&s.last, static_cast<int>(threadIdx.x));
        __syncthreads();
        const int chosen = s.first < kBins ? s.first : max(s.last, 0);
        if (static_cast<int>(threadIdx.x) == chosen) {
            s.chosen_mass = run - mass;
            s.chosen_count = runs - count;
            s.counts[0] = count;
        }
        __syncthreads();
        f.mass_above = s.chosen_mass;
        f.count_above = s.chosen_count;
        f.equal = s.counts[0];
        f.bits |= static_cast<unsigned>(kBins - 1 - chosen) << shift;
        mask |= static_cast<unsigned>(kBins - 1) << shift;
    }
    ++descents;
    return f;
}

// The smallest c of 1 .. n with above + c * w >= target (inclusive) or > target; n where there is none, as for a target that is
// no number (which must not become the integer that a search starts from: the conversion gives the smallest there is).
__device__ __forceinline__ int sample_count_to(double above, double w, int n, double target, bool inclusive) {
    if (!(w > 0.0) || !(target == target)) return n;
    const double guess = (target - above) / w;
    int c = guess >= n ? n : guess > 1.0 ? static_cast<int>(guess) : 1;
    auto reached = [&](int k) { const double cum = above + k * w; return inclusive ? cum >= target : cum > target; };
    while (c > 1 && reached(c - 1)) --c;
    while (c < n && !reached(c)) ++c;
    return c;
}

// probs: scratch [rows, V] floats.
// kHeld > 0: every warp's piece fits kHeld values a lane, and probs is not used.
template <bool kWide, int kHeld>
__global__ void __cluster_dims__(kSampleParts, 1, 1) __launch_bounds__(kSampleThreads)
sample_kernel(const float* __restrict__ logits, float* __restrict__ probs_all, int V,
              const float* __restrict__ temperature, const int* __restrict__ top_k,
              const float* __restrict__ top_p, const float* __restrict__ uniform, int* __restrict__ out) {
    pdl_prologue();
    __shared__ SampleShared<kWide> s;
    cg::cluster_group cluster = cg::this_cluster();
    const int r = blockIdx.x / kSampleParts, part = blockIdx.x % kSampleParts;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float* row = logits + static_cast<size_t>(r) * V;
    float* probs = probs_all + static_cast<size_t>(r) * V;
    const float temp = temperature[r];
    if (!(temp > 0.f)) return;          // a greedy row (for the whole cluster): out[r] keeps what the caller put there (its argmax)

    // this CTA's piece of the row, and this warp's piece of that
    const int slice = (V + kSampleParts - 1) / kSampleParts, piece = (slice + 31) / 32;
    const int slice_begin = min(V, part * slice), slice_end = min(V, slice_begin + slice);
    const int begin = min(slice_end, slice_begin + warp * piece), end = min(slice_end, begin + piece);

    constexpr bool kInRegs = kHeld > 0;
    float held[kInRegs ? kHeld : 1];
    // every place of this lane and its value, in order
    auto each = [&](auto f) {
        if constexpr (kInRegs) {
#pragma unroll
            for (int u = 0; u < kHeld; ++u)
                if (begin + lane + 32 * u < end) f(begin + lane + 32 * u, held[u]);
        } else {
            for (int i = begin + lane; i < end; i += 32) f(i, probs[i]);
        }
    };
    // every value of this lane replaced: in registers, else in probs (from the logits the first time)
    auto replace = [&](const float* from, auto f) {
        if constexpr (kInRegs) {
#pragma unroll
            for (int u = 0; u < kHeld; ++u)
                if (begin + lane + 32 * u < end) held[u] = f(held[u]);
        } else {
            for (int i = begin + lane; i < end; i += 32) probs[i] = f(from[i]);
        }
    };

    // max
    float mx = -INFINITY;
    if constexpr (kInRegs) {
#pragma unroll
        for (int u = 0; u < kHeld; ++u) held[u] = begin + lane + 32 * u < end ? row[begin + lane + 32 * u] : -INFINITY;
#pragma unroll
        for (int u = 0; u < kHeld; ++u) mx = fmaxf(mx, held[u]);
    } else {
        for (int i = begin + lane; i < end; i += 32) mx = fmaxf(mx, row[i]);
    }
    mx = warp_max(mx);
    if (lane == 0) s.red[warp] = static_cast<double>(mx);
    __syncthreads();
    if (threadIdx.x == 0) {
        double m = s.red[0];
        for (int w = 1; w < 32; ++w) m = fmax(m, s.red[w]);
        s.cta_max = m;
    }
    cluster.sync();
    mx = -INFINITY;
    for (int p = 0; p < kSampleParts; ++p) mx = fmaxf(mx, static_cast<float>(*cluster.map_shared_rank(&s.cta_max, p)));

    // p_i = exp((l_i - max)/T), sum in double, then scaled by (float)(1/sum)
    double mine = 0.0;
    replace(row, [&](float x) {
        const float e = expf((x - mx) / temp);
        mine += static_cast<double>(e);
        return e;
    });
    mine = block_sum_double(mine, s.red);
    if (threadIdx.x == 0) s.cta_sum = mine;
    cluster.sync();
    double sum = 0.0;
    for (int p = 0; p < kSampleParts; ++p) sum += *cluster.map_shared_rank(&s.cta_sum, p);
    const float inv_sum = static_cast<float>(1.0 / sum);
    mine = 0.0;
    replace(probs, [&](float x) {
        const float p = x * inv_sum;
        mine += static_cast<double>(p);
        return p;
    });
    mine = warp_sum_double(mine);
    if (lane == 0) s.warp_mass[warp] = mine;
    __syncthreads();
    mine = 0.0;
    for (int w = 0; w < 32; ++w) mine += s.warp_mass[w];
    if (threadIdx.x == 0) s.cta_mass = mine;
    cluster.sync();
    double before = 0.0, all_mass = 0.0;              // `before`: the mass of the pieces ahead of this CTA's
    for (int p = 0; p < kSampleParts; ++p) {
        if (p == part) before = all_mass;
        all_mass += *cluster.map_shared_rank(&s.cta_mass, p);
    }

    const int k = top_k[r];
    const float tp = top_p[r];
    const bool use_k = k > 0 && k < V;
    const bool use_p = tp < 1.0f;
    const double u = static_cast<double>(uniform[r]);

    if (!(sum == sum)) {                              // a row without probabilities (NaN, or infinities of one sign only)
        if (part == 0 && threadIdx.x == 0) out[r] = use_p ? 0 : use_k ? k - 1 : V - 1;
    } else if (!use_k && !use_p) {
        // index order: the CTA, the warp, then the value at which the running mass exceeds the target
        const double target = u * all_mass;
        if (!(target < all_mass)) {
            if (part == 0 && threadIdx.x == 0) out[r] = V - 1;          // rounding guard: u was (almost) 1, or no number
        } else if (target < 0.0) {
            if (part == 0 && threadIdx.x == 0) out[r] = 0;              // (no piece begins below 0)
        } else if (target >= before && target < before + mine) {
            double run = before, next = before;       // run: the mass ahead of the owner, a warp that has some
            int owner = -1;
            for (int w = 0; w < 32 && !(target < next); ++w) {
                if (s.warp_mass[w] > 0.0) { owner = w; run = next; }
                next += s.warp_mass[w];
            }
            if (owner == warp) {
                int pick = -1, fallback = max(begin, end - 1);
                auto look = [&](int base, float value) {          // the 32 values from base on
                    const int i = base + lane;
                    double cum = i < end ? static_cast<double>(value) : 0.0;
                    const unsigned some = __ballot_sync(0xffffffffu, cum > 0.0);
                    if (some) fallback = base + 31 - __clz(some);
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const double m = __shfl_up_sync(0xffffffffu, cum, o);
                        if (lane >= o) cum += m;
                    }
                    cum += run;
                    const unsigned over = __ballot_sync(0xffffffffu, i < end && target < cum);
                    if (over) pick = base + __ffs(over) - 1;
                    run = __shfl_sync(0xffffffffu, cum, 31);
                };
                if constexpr (kInRegs) {
#pragma unroll
                    for (int u = 0; u < kHeld; ++u)
                        if (begin + 32 * u < end && pick < 0) look(begin + 32 * u, held[u]);
                } else {
                    for (int base = begin; base < end && pick < 0; base += 32) look(base, base + lane < end ? probs[base + lane] : 0.f);
                }
                if (lane == 0) out[r] = pick >= 0 ? pick : fallback;
            }
        }
    } else {
        // ---- the kept set is a prefix of the order (probability descending, index ascending) ----
        // Its end is described by (boundary bits, number of boundary-valued elements kept).
        // Start: everything kept.
        double kept_mass = all_mass;
        unsigned bound_bits = 0u;        // smallest kept probability's bits
        int bound_take = 0;              // how many elements equal to it are kept (index order)
        bool bounded = false;
        int turn = 0, descents = 0;

        if (use_k) {
            const Found f = sample_descend<kWide>(each, true, static_cast<double>(k), true, s, turn, descents, cluster);
            bound_bits = f.bits;
            bound_take = k - f.count_above;
            bounded = true;
            kept_mass = f.mass_above + static_cast<double>(bound_take) * static_cast<double>(__uint_as_float(bound_bits));
        }
        if (use_p) {
            // shortest prefix with cum >= top_p * kept_mass, inside the current kept set. The descent runs over all elements;
            // as the kept set is a prefix of the same order, the crossing lies inside it unless rounding pushes it out.
            const double threshold = static_cast<double>(tp) * kept_mass;
            const Found f = sample_descend<kWide>(each, false, threshold, true, s, turn, descents, cluster);
            const double w = static_cast<double>(__uint_as_float(f.bits));
            const int take = w > 0.0 ? sample_count_to(f.mass_above, w, f.equal, threshold, true) : 1;
            if (!bounded || f.bits > bound_bits || (f.bits == bound_bits && take <= bound_take)) {
                bound_bits = f.bits;
                bound_take = take;
                bounded = true;
                kept_mass = f.mass_above + static_cast<double>(take) * w;
            }
        }

        // ---- draw: first token in the order with u * kept_mass < cum ----
        const double target = u * kept_mass;
        const Found f = sample_descend<kWide>(each, false, target, false, s, turn, descents, cluster);
        unsigned pick_bits = f.bits;
        int rank = sample_count_to(f.mass_above, static_cast<double>(__uint_as_float(pick_bits)), f.equal, target, false) - 1;
        // clamp to the kept set (rounding guard: the last kept token)
        if (bounded && (pick_bits < bound_bits || (pick_bits == bound_bits && rank >= bound_take))) {
            pick_bits = bound_bits;
            rank = bound_take - 1;
        }
        // the rank-th (0-based) index with those bits: the CTA, the warp, then the place
        int c = 0;
        each([&](int, float value) { c += __float_as_uint(value) == pick_bits; });
        c = __reduce_add_sync(0xffffffffu, c);
        __syncthreads();
        if (lane == 0) s.counts[warp] = c;
        __syncthreads();
        int own = 0, ahead = 0;
        for (int w = 0; w < 32; ++w) {
            if (w == warp) ahead = own;
            own += s.counts[w];
        }
        if (threadIdx.x == 0) s.cta_equal = own;
        cluster.sync();
        for (int p = 0; p < part; ++p) ahead += *cluster.map_shared_rank(&s.cta_equal, p);
        if (rank >= ahead && rank < ahead + c) {
            bool done = false;
            auto look = [&](int base, float value) {              // the 32 values from base on
                const int i = base + lane;
                const unsigned same = __ballot_sync(0xffffffffu, i < end && __float_as_uint(value) == pick_bits);
                if (rank < ahead + __popc(same)) {
                    if ((same >> lane & 1u) && ahead + __popc(same & ((1u << lane) - 1)) == rank) out[r] = i;
                    done = true;
                }
                ahead += __popc(same);
            };
            if constexpr (kInRegs) {
#pragma unroll
                for (int u = 0; u < kHeld; ++u)
                    if (begin + 32 * u < end && !done) look(begin + 32 * u, held[u]);
            } else {
                for (int base = begin; base < end && !done; base += 32) look(base, base + lane < end ? probs[base + lane] : 0.f);
            }
        }
    }
    cluster.sync();                                   // no CTA leaves while another may read its shared memory
}

int launch_sample(const float* logits, float* probs, int rows, int V, const float* temperature, const int* top_k, const float* top_p,
                  const float* uniform, int* out, cudaStream_t st) {
    GI_REQUIRE(rows <= INT_MAX / kSampleParts, "sample: %d rows exceed the grid limit", rows);
    const dim3 grid(rows * kSampleParts), block(kSampleThreads);
    if (V <= kSampleParts * kSampleThreads * kHeldFew) launch_kernel((sample_kernel<false, kHeldFew>), grid, block, 0, st, logits, probs, V, temperature, top_k, top_p, uniform, out);
    else if (V <= kSampleParts * kSampleThreads * kHeldMost) launch_kernel((sample_kernel<false, kHeldMost>), grid, block, 0, st, logits, probs, V, temperature, top_k, top_p, uniform, out);
    else if (V <= kNarrowVocab) launch_kernel((sample_kernel<false, 0>), grid, block, 0, st, logits, probs, V, temperature, top_k, top_p, uniform, out);
    else launch_kernel((sample_kernel<true, 0>), grid, block, 0, st, logits, probs, V, temperature, top_k, top_p, uniform, out);
    return check_launch("sample");
}

}  // namespace gi

using namespace gi;

// part_val / part_idx: caller's scratch of rows * 32 floats / ints.
static int gi_argmax_impl(const float* logits, int rows, int V, int* out, float* part_val, int* part_idx, void* stream) {
    if (rows == 0) return 0;
    GI_REQUIRE(rows > 0 && V > 0, "argmax: sizes must be positive (rows=%d, V=%d)", rows, V);
    GI_REQUIRE(rows <= 65535, "argmax: %d rows exceed the grid limit", rows);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    launch_kernel((argmax_partial_kernel), dim3(kArgmaxParts, rows), dim3(256), 0, st, logits, V, part_val, part_idx);
    if (check_launch("argmax")) return 1;
    launch_kernel((argmax_final_kernel), dim3(rows), dim3(32), 0, st, static_cast<const float*>(part_val),
                  static_cast<const int*>(part_idx), out);
    return check_launch("argmax");
}

// probs_scratch: [rows, V] floats owned by the caller. Rows with temperature[r] <= 0 are skipped:
// out[r] is left as it is (the caller writes the row's argmax there first).
static int gi_sample_impl(const float* logits, float* probs_scratch, int rows, int V, const float* temperature,
                         const int* top_k, const float* top_p, const float* uniform, int* out, void* stream) {
    if (rows == 0) return 0;
    GI_REQUIRE(rows > 0 && V > 0, "sample: sizes must be positive (rows=%d, V=%d)", rows, V);
    return launch_sample(logits, probs_scratch, rows, V, temperature, top_k, top_p, uniform, out, static_cast<cudaStream_t>(stream));
}

// ------------------------------------------------------------------------------------------------
// The allocation-free variant of gi_sample (declared and explained in no_alloc.h).
#include "no_alloc.h"

#include <mutex>

namespace gi {

// The work area of gi_sample_no_alloc. In host code this name is only a handle for the runtime's
// symbol table, not a device address: the address is looked up once per device below.
static __device__ __align__(256) float g_sample_work_area[GI_SAMPLE_NO_ALLOC_MAX_FLOATS];

constexpr int kMaxDevices = 64;
static float* g_work_area_address[kMaxDevices] = {};
static std::mutex g_work_area_mutex;

// Device address of the work area on the current device; looked up on the first call per device.
static int work_area_for_current_device(float** out) {
    int device = -1;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) {
        set_error("sample_no_alloc: cudaGetDevice failed: %s", cudaGetErrorString(e));
        return 1;
    }
    if (device < 0 || device >= kMaxDevices) {
        set_error("sample_no_alloc: device index %d is outside the supported range 0..%d", device, kMaxDevices - 1);
        return 2;
    }
    std::lock_guard<std::mutex> lock(g_work_area_mutex);
    if (g_work_area_address[device] == nullptr) {
        float* ptr = nullptr;
        e = cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_sample_work_area);
        if (e != cudaSuccess || ptr == nullptr) {
            set_error("sample_no_alloc: cudaGetSymbolAddress failed on device %d: %s", device, cudaGetErrorString(e));
            return 1;
        }
        g_work_area_address[device] = ptr;
    }
    *out = g_work_area_address[device];
    return 0;
}

}  // namespace gi

extern "C" int gi_sample_no_alloc(const float* logits, int rows, int vocab, const float* temperature,
                                  const int* top_k, const float* top_p, const float* uniform, int* out,
                                  void* stream) {
    if (rows == 0) return 0;
    GI_REQUIRE(rows > 0 && vocab > 0, "sample_no_alloc: sizes must be positive (rows=%d, vocab=%d)", rows, vocab);
    const long long need = static_cast<long long>(rows) * vocab;
    GI_REQUIRE(need <= GI_SAMPLE_NO_ALLOC_MAX_FLOATS,
               "sample_no_alloc: %d rows x %d vocabulary = %lld floats exceed the built-in work area of %d floats; "
               "sample fewer rows per call or use gi_sample with a scratch buffer of your own",
               rows, vocab, need, GI_SAMPLE_NO_ALLOC_MAX_FLOATS);
    float* work = nullptr;
    const int rc = work_area_for_current_device(&work);
    if (rc != 0) return rc;
    return launch_sample(logits, work, rows, vocab, temperature, top_k, top_p, uniform, out, static_cast<cudaStream_t>(stream));
}

// The exported names: each runs its implementation above and, while a launch program is recorded, leaves a copy of
// its arguments in the program (common.cuh).
extern "C" int gi_argmax(const float* logits, int rows, int V, int* out, float* part_val, int* part_idx, void* stream) {
    return gi::dispatch(gi_argmax_impl, logits, rows, V, out, part_val, part_idx, stream);
}

extern "C" int gi_sample(const float* logits, float* probs_scratch, int rows, int V, const float* temperature, const int* top_k, const float* top_p, const float* uniform, int* out, void* stream) {
    return gi::dispatch(gi_sample_impl, logits, probs_scratch, rows, V, temperature, top_k, top_p, uniform, out, stream);
}
