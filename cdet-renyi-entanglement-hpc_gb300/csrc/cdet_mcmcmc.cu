// Device-resident MCMCMC chains: run_mcmcmc_step (mcmcmc_sampler.h:524-577) on
// the all-subset integrand values of each chain's envelope, so a batch of chains advances one step per launch pair
// (integrand, step) with no host round trip. The seed kernel is the uniform
// one (mcmcmc_seed.h:41-61) or the factorized histogram (:71-229), whose
// conditional generation probabilities (mcmcmc_sampler.h:252-335) weight the
// fluxes.
//
// Each chain keeps the reference's std::mt19937_64 stream (the published
// MT19937-64 generator with libstdc++'s seeding) and draws from it exactly as
// libstdc++'s distributions do: std::generate_canonical<double, 53> takes one
// 64-bit output, converts it to double (round to nearest) and divides by 2^64;
// std::uniform_int_distribution<int> downscales with a 128-bit product
// (nearly-divisionless rejection). With the FP64 integrand the device chains
// therefore follow the reference's chains step for step. The generator state
// is stored interleaved ([word][chain]) so that the threads of a warp touch
// consecutive addresses.
#include "cdet_device.cuh"
#include "cdet_kernels.cuh"

#include <algorithm>

namespace cdet {

namespace {

constexpr int kMtN = 312;
constexpr int kMtM = 156;

// One word of the state transition, from words i, i + 1 and i + 156.
__device__ __forceinline__ uint64_t mt_twist(uint64_t word, uint64_t next, uint64_t far) {
    const uint64_t x = (word & 0xFFFFFFFF80000000ull) | (next & 0x7FFFFFFFull);
    return far ^ (x >> 1) ^ ((x & 1ull) ? 0xB5026F5AA96619E9ull : 0ull);
}
__device__ __forceinline__ uint64_t mt_temper(uint64_t y) {
    y ^= (y >> 29) & 0x5555555555555555ull;
    y ^= (y << 17) & 0x71D67FFFEDA60000ull;
    y ^= (y << 37) & 0xFFF7EEE000000000ull;
    return y ^ (y >> 43);
}

// std::generate_canonical<double, 53> of one word as libstdc++ computes it.
// The division by 2^64 is exact, and so is the product with 2^-64.
__device__ __forceinline__ double mt_canonical(uint64_t word) {
    const double r = dmul(__ull2double_rn(word), 0x1p-64);
    return r >= 1.0 ? __longlong_as_double(0x3FEFFFFFFFFFFFFFll) : r;
}

// std::uniform_int_distribution<int>(0, n - 1)
template <class Generator>
__device__ __forceinline__ int mt_uniform_int(Generator& g, int n) {
    const uint64_t range = static_cast<uint64_t>(n);
    uint64_t x = g.next();
    uint64_t low = x * range;
    uint64_t high = __umul64hi(x, range);
    if (low < range) {
        const uint64_t threshold = (0ull - range) % range;
        while (low < threshold) {
            x = g.next();
            low = x * range;
            high = __umul64hi(x, range);
        }
    }
    return static_cast<int>(high);
}

// A chain's generator on one thread.
struct Mt64 {
    uint64_t* words;  // word i of this chain at words[i * stride]
    int64_t stride;
    int32_t* index;

    __device__ __forceinline__ uint64_t& at(int i) const { return words[static_cast<int64_t>(i) * stride]; }

    __device__ uint64_t next() const {
        if (*index >= kMtN) {
            for (int i = 0; i < kMtN; ++i)
                at(i) = mt_twist(at(i), at(i + 1 < kMtN ? i + 1 : 0),
                                 at(i + kMtM < kMtN ? i + kMtM : i + kMtM - kMtN));
            *index = 0;
        }
        return mt_temper(at((*index)++));
    }
    __device__ double canonical() const { return mt_canonical(next()); }
};

// A chain's generator on one warp, every lane calling together: lane k holds
// word base + k of the state, tempered, so that a draw is a shuffle, and the
// state transition runs on all lanes (32 words at a time; a word's new value
// needs only its neighbour's old one, which the next 32 have not replaced
// yet). The same words in the same order as Mt64's.
struct WarpMt64 {
    uint64_t* words;
    int64_t stride;
    int lane;
    int32_t index;
    int32_t base;
    uint64_t buffer;

    __device__ WarpMt64(uint64_t* w, int64_t s, int32_t i, int l)
        : words(w), stride(s), lane(l), index(i), base(-kWarp), buffer(0) {}
    __device__ __forceinline__ uint64_t& at(int i) const { return words[static_cast<int64_t>(i) * stride]; }

    __device__ void transition() {
        for (int part = 0; part < 2; ++part) {  // words 0..155, then 156..311 from the new 0..155
            for (int i0 = part * kMtM; i0 < (part + 1) * kMtM; i0 += kWarp) {
                const int i = i0 + lane;
                const bool in = i < (part + 1) * kMtM;
                uint64_t v = 0;
                if (in) v = mt_twist(at(i), at(i + 1 < kMtN ? i + 1 : 0), at(part == 0 ? i + kMtM : i - kMtM));
                __syncwarp();
                if (in) at(i) = v;
                __syncwarp();
            }
        }
    }
    // The buffer holds words index .. index + count - 1 (count <= 32, index + count <= 312).
    __device__ __forceinline__ void fill(int count) {
        if (index >= base && index + count <= base + kWarp) return;
        base = index;
        buffer = base + lane < kMtN ? mt_temper(at(base + lane)) : 0;
    }
    __device__ uint64_t next() {
        if (index >= kMtN) {
            transition();
            index = 0;
            base = -kWarp;
        }
        fill(1);
        return __shfl_sync(0xffffffffu, buffer, index++ - base);
    }
    __device__ double canonical() { return mt_canonical(next()); }
    // Four canonical draws in order, the k-th on every lane l with l & 3 == k.
    __device__ double canonical4() {
        uint64_t word = 0;
        if (index + 4 <= kMtN) {
            fill(4);
            word = __shfl_sync(0xffffffffu, buffer, index - base + (lane & 3));
            index += 4;
        } else {
            for (int k = 0; k < 4; ++k) {
                const uint64_t w = next();
                if ((lane & 3) == k) word = w;
            }
        }
        return mt_canonical(word);
    }
};

// unit_coordinate_to_index (mcmcmc_seed.h:30-39)
__device__ __forceinline__ int unit_index(double value, int extent) {
    const int index = static_cast<int>(floor(dmul(value, static_cast<double>(extent))));
    if (index < 0) return 0;
    if (index >= extent) return extent - 1;
    return index;
}

// sample_from_row (mcmcmc_seed.h:205-218): std::lower_bound (the binary search
// for the first entry not below the draw) in one CDF row; past the end, the
// last column
template <class Generator>
__device__ int sample_row(const double* __restrict__ cdf, int columns, int row, Generator& g) {
    const double threshold = g.canonical();
    const double* b = cdf + static_cast<int64_t>(row) * columns;
    int first = 0, len = columns;
    while (len > 0) {
        const int half = len >> 1;
        if (b[first + half] < threshold) {
            first += half + 1;
            len -= half + 1;
        } else {
            len = half;
        }
    }
    return first == columns ? columns - 1 : first;
}

// density_child_given_parent (mcmcmc_seed.h:130-150)
__device__ double hist_density(const McmcmcStepArgs& a, const double* child, const double* parent) {
    const int sites = a.n1 * a.n2;
    const double tau_d = dmul(a.tau_prob[unit_index(parent[0], a.tau_bins) * a.tau_bins +
                                         unit_index(child[0], a.tau_bins)],
                              static_cast<double>(a.tau_bins));
    const int ps = unit_index(parent[1], a.n1) * a.n2 + unit_index(parent[2], a.n2);
    const int cs = unit_index(child[1], a.n1) * a.n2 + unit_index(child[2], a.n2);
    const double space_d = dmul(a.space_prob[static_cast<int64_t>(ps) * sites + cs], static_cast<double>(sites));
    const double rep_d = dmul(a.replica_prob[unit_index(parent[3], 2) * 2 + unit_index(child[3], 2)], 2.0);
    return dmul(dmul(tau_d, space_d), rep_d);
}

// sample_child_from_parent (mcmcmc_seed.h:106-128): three row draws, then the
// four in-cell offsets in vertex order
template <class Generator>
__device__ void hist_child(const McmcmcStepArgs& a, Generator& g, const double* parent, double (&child)[4]) {
    const int child_tau = sample_row(a.tau_cdf, a.tau_bins, unit_index(parent[0], a.tau_bins), g);
    const int parent_site = unit_index(parent[1], a.n1) * a.n2 + unit_index(parent[2], a.n2);
    const int child_site = sample_row(a.space_cdf, a.n1 * a.n2, parent_site, g);
    const int child_x = child_site / a.n2;
    const int child_y = child_site - child_x * a.n2;
    const int child_rep = sample_row(a.replica_cdf, 2, unit_index(parent[3], 2), g);
    child[0] = ddiv(dadd(static_cast<double>(child_tau), g.canonical()), static_cast<double>(a.tau_bins));
    child[1] = ddiv(dadd(static_cast<double>(child_x), g.canonical()), static_cast<double>(a.n1));
    child[2] = ddiv(dadd(static_cast<double>(child_y), g.canonical()), static_cast<double>(a.n2));
    child[3] = ddiv(dadd(static_cast<double>(child_rep), g.canonical()), 2.0);
}

// compute_conditional_generation_probabilities_typed_into<double>
// (mcmcmc_sampler.h:252-335), one warp per chain. The reference tabulates the
// remaining child densities cd[gm][c] by peeling the lowest bit of gm; here
// each one is formed on the spot from the row sum with the same subtractions
// in the same order (the highest bit of gm first), each result clamped as the
// table's is, so only the 2^n probabilities are stored. The subsets of one
// popcount level depend only on the level below, so the lanes share each
// level; every subset's sum runs on one lane in the reference's order, so the
// values are the reference's bit for bit. sd: this warp's n x n densities in
// shared memory. false (on every lane): a density is negative or not finite.
__device__ bool conditional_probabilities_warp(const McmcmcStepArgs& a, const double* v, int n, double* prob,
                                               double* sd, double* cd0, int lane) {
    bool bad = false;
    for (int idx = lane; idx < n * n; idx += 32) {
        const int c = idx / n, p = idx - (idx / n) * n;
        double d = 0.0;
        if (c != p) {
            d = hist_density(a, v + 4 * c, v + 4 * p);
            bad |= d < 0.0 || !isfinite(d);
        }
        sd[idx] = d;
    }
    if (__any_sync(0xffffffffu, bad)) return false;
    __syncwarp();
    if (lane < n) {
        double sum = 0.0;
        for (int p = 0; p < n; ++p) sum = dadd(sum, sd[lane * n + p]);
        cd0[lane] = sum;
    }
    const uint64_t full = (uint64_t{1} << n) - 1;
    if (lane == 0) {
        prob[0] = 1.0;
        prob[full] = 0.0;
    }
    __syncwarp();
    for (int level = 1; level < n; ++level) {
        const int pc = n - level;
        const double denom = dmul(static_cast<double>(level), static_cast<double>(pc));
        const uint32_t per = kBinomial.c[n][level];
        for (uint32_t r = lane; r < per; r += 32) {
            const uint64_t gm = colex_subset(r, level, n);  // the level's subsets dealt out evenly
            double sum = 0.0;
            for (int c = 0; c < n; ++c) {
                const uint64_t cb = uint64_t{1} << c;
                if (!(gm & cb)) continue;
                double d = cd0[c];
                for (uint64_t rest = gm; rest;) {
                    const int b = 63 - __clzll(static_cast<long long>(rest));
                    rest ^= uint64_t{1} << b;
                    d = dsub(d, sd[c * n + b]);
                    if (d < 0.0 && d > -1.0e-12) d = 0.0;
                }
                sum = dadd(sum, dmul(prob[gm ^ cb], d));
            }
            prob[gm] = ddiv(sum, denom);
        }
        __syncwarp();  // the next level reads this one
    }
    return true;
}

// std::mt19937_64(seed) and sample_uniform_vertex_set (mcmcmc_sampler.h:187-198)
__global__ void mcmcmc_init(int64_t chains, int envelope, const uint64_t* __restrict__ seeds, uint64_t* mt,
                            int32_t* mt_index, double* vertices) {
    const int64_t c = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (c >= chains) return;
    Mt64 g{mt + c, chains, mt_index + c};
    uint64_t x = seeds[c];
    g.at(0) = x;
    for (int i = 1; i < kMtN; ++i) {
        x = 6364136223846793005ull * (x ^ (x >> 62)) + static_cast<uint64_t>(i);
        g.at(i) = x;
    }
    *g.index = kMtN;
    double* v = vertices + c * envelope * 4;
    for (int k = 0; k < envelope * 4; ++k) v[k] = g.canonical();
}

// The serial part of run_mcmcmc_step (:540-577) for chain c, after the seed
// kernel's conditional probabilities (cprob; null for the uniform kernel).
template <bool Hist>
__device__ void finish_step(const McmcmcStepArgs& a, int64_t c, int64_t row, const double* cprob) {
    const int env = a.envelope;
    const uint64_t subsets = uint64_t{1} << env;
    const double* values = a.values + c * static_cast<int64_t>(subsets);
    const double* lam = a.lambdas + c * (env + 1);
    Mt64 g{a.mt + c, a.chains, a.mt_index + c};
    const double* v = a.vertices + c * env * 4;
    const uint64_t full = subsets - 1;
    // flux = lambda * value * conditional probability of the complement
    // (1 for the uniform kernel)
    auto flux_of = [&](uint64_t mask, int o) {
        return dmul(dmul(lam[o], values[mask]), Hist ? cprob[full ^ mask] : 1.0);
    };
    // fluxes and selection weights in the mask plan's order (:411-430, :540-560)
    double norm = 0.0;
    for (uint64_t mask = 1; mask < subsets; ++mask) {
        const int o = __popcll(mask);
        if (o < a.order_min || o > a.order_max) continue;
        norm = dadd(norm, dmul(fabs(flux_of(mask, o)), a.inv_binom[o]));
    }
    // sample_weighted_candidate_mask (:225-250)
    if (!(norm > 0.0) || !isfinite(norm)) {
        a.error[c] = 2;  // "MCMCMC local normalization is zero or non-finite"
        return;
    }
    const double threshold = dadd(dmul(g.canonical(), dsub(norm, 0.0)), 0.0);
    double cumulative = 0.0;
    uint64_t chosen = 0, last_positive = 0;
    bool found = false;
    for (uint64_t mask = 1; mask < subsets && !found; ++mask) {
        const int o = __popcll(mask);
        if (o < a.order_min || o > a.order_max) continue;
        const double w = dmul(fabs(flux_of(mask, o)), a.inv_binom[o]);
        if (!(w > 0.0)) continue;
        if (isfinite(w)) last_positive = mask;
        cumulative = dadd(cumulative, w);
        if (cumulative > threshold) {
            chosen = mask;
            found = true;
        }
    }
    if (!found) chosen = last_positive;
    // order signal: time = flux / local_normalization, weighted by 1/binomial (:566-571)
    if (a.signal_out) {
        double* sig = a.signal_out + (row * a.chains + c) * (env + 1);
        for (int o = 0; o <= env; ++o) sig[o] = 0.0;
        for (uint64_t mask = 1; mask < subsets; ++mask) {
            const int o = __popcll(mask);
            if (o < a.order_min || o > a.order_max) continue;
            const double time = ddiv(flux_of(mask, o), norm);
            sig[o] = dadd(sig[o], dmul(time, a.inv_binom[o]));
        }
    }
    // create_next_vertices_from_seed_into (:380-400): the retained vertices in
    // order, then children of uniformly chosen parents among the vertices so
    // far (the uniform kernel, mcmcmc_seed.h:51-55, ignores the parent)
    double* nv = a.next_vertices + c * env * 4;
    int size = 0;
    for (int i = 0; i < env; ++i)
        if (chosen & (uint64_t{1} << i)) {
            for (int k = 0; k < 4; ++k) nv[4 * size + k] = v[4 * i + k];
            ++size;
        }
    while (size < env) {
        const int parent = mt_uniform_int(g, size);
        if constexpr (Hist) {
            double child[4];
            hist_child(a, g, nv + 4 * parent, child);
            for (int k = 0; k < 4; ++k) nv[4 * size + k] = child[k];
        } else {
            (void)parent;
            for (int k = 0; k < 4; ++k) nv[4 * size + k] = g.canonical();
        }
        ++size;
    }
    const int order = __popcll(chosen);
    if (a.chosen_out) a.chosen_out[row * a.chains + c] = chosen;
    if (a.retained_out) a.retained_out[c] = chosen;
    if (a.norm_out) a.norm_out[row * a.chains + c] = norm;
    if (a.warmup) ++a.counts[c * (env + 1) + order];
}

// The step, one thread per chain (after mcmcmc_hist_probs for the histogram
// seed kernel).
template <bool Hist>
__global__ void __launch_bounds__(128) mcmcmc_step(const __grid_constant__ McmcmcStepArgs a) {
    const int64_t c = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (c >= a.chains) return;
    const int64_t row = a.ring_row ? *a.ring_row : 0;
    if (a.chosen_out) a.chosen_out[row * a.chains + c] = 0;  // 0: no step (a failed chain)
    if (a.retained_out) a.retained_out[c] = 0;
    if (a.error[c]) return;  // a chain that failed stays where it stopped
    if (a.integrand_status[c] & kStatusNonFinite) {
        a.error[c] = 1;  // "Error (all-subset integrand): Value is not finite"
        return;
    }
    finish_step<Hist>(a, c, row, Hist ? a.cprob + c * (int64_t{1} << a.envelope) : nullptr);
}

// The step with one warp per chain (fewer than step_warp_max_chains chains), one
// to eight chains per block. Everything elementwise runs on the chain's lanes:
// the fluxes and selection weights, the signal terms, the search for the drawn
// mask, the generator. What the reference adds up in mask order stays a serial
// sum, but shares its FP64 instructions: the local normalisations of the
// block's chains run on neighbouring lanes of one warp, and so do their
// per-order signal sums. The weighted draw needs no second sum: its running
// weight is the normalisation's (masks of weight zero change neither), so the
// prefixes are kept and the first one above the threshold is found in
// parallel. Same values as finish_step.
//
// Bound: the 2^envelope dependent FP64 additions of the normalisation.
// Measured at envelope 9 against lane 0 doing all serial work with its own
// divisions and global generator state: 128 chains 215 -> 50 us, 2,048 chains 588 -> 74 us (one
// thread per chain before).
constexpr int kStepWarpMaxEnvelope = 12;
constexpr int kStepMaxChainsPerBlock = 8;

// Doubles of shared memory per chain: fluxes and weight prefixes (each padded
// by one, so that neighbouring chains' entries fall into other banks), for the
// histogram seed kernel the conditional probabilities, densities and row sums.
__host__ __device__ inline size_t step_doubles(int env, bool hist) {
    const size_t subsets = size_t{1} << env;
    return 2 * (subsets + 1) + (hist ? subsets + static_cast<size_t>(env) * (env + 1) : 0);
}

// From how many chains on a thread per chain is the faster step. A warp per
// chain loses its lead where the envelope leaves its lanes nothing to do (2, 3)
// and where the shared memory of few chains fills an SM, so that many chains are
// many rounds (from envelope 11; earlier with the histogram seed, whose
// probabilities the other form makes on full SMs). Whole steps, thread form over
// warp form (2x2, degree 8; uniform seed, then histogram): envelope 2, 2,048 chains
// 1.00 and 0.98, 8,192 0.94 and 0.90; envelope 3, 4,096 1.05 and 1.04, 8,192 1.02 and
// 0.96; 4 to 10, 8,192 1.11 to 1.26 and 1.08 to 1.17, 16,383 1.05 to 1.14 and 0.99 to
// 1.07; 11 (six and four chains per SM), 3,000 1.31 and 1.05, 4,096 1.21 and 0.96,
// 12,000 1.02 and 0.81; 12 (three and two), 3,000 1.01 and 0.95, 8,192 1.00 and 0.88.
int64_t step_warp_max_chains(int env, bool hist) {
    if (env > kStepWarpMaxEnvelope) return 0;
    constexpr int64_t kLeast = 2048, kMost = 16384;
    if (env <= 3) return env <= 2 ? kLeast : 4 * kLeast;
    const int64_t per_sm = (227 * 1024) / static_cast<int64_t>(step_doubles(env, hist) * sizeof(double));
    return per_sm >= 8 ? kMost : std::max<int64_t>(kLeast, per_sm * (hist ? 768 : 2048));
}

template <bool Hist>
__global__ void __launch_bounds__(kStepMaxChainsPerBlock * kWarp) mcmcmc_step_warp(const __grid_constant__ McmcmcStepArgs a) {
    extern __shared__ double step_smem[];
    __shared__ double s_norm[kStepMaxChainsPerBlock];
    __shared__ int s_state[kStepMaxChainsPerBlock];  // 1: the chain makes a step; 2: its normalisation is good
    const int lane = threadIdx.x & (kWarp - 1), warp = threadIdx.x / kWarp, per_block = blockDim.x / kWarp;
    const int64_t c = static_cast<int64_t>(blockIdx.x) * per_block + warp;
    const int env = a.envelope;
    const uint32_t subsets = 1u << env, full = subsets - 1;
    const size_t per_chain = step_doubles(env, Hist);
    double* flux = step_smem + static_cast<size_t>(warp) * per_chain;
    double* prefix = flux + subsets + 1;
    double* prob = prefix + subsets + 1;
    const int64_t row = a.ring_row ? *a.ring_row : 0;
    bool active = c < a.chains;
    if (active) {
        if (lane == 0 && a.chosen_out) a.chosen_out[row * a.chains + c] = 0;  // 0: no step (a failed chain)
        if (lane == 0 && a.retained_out) a.retained_out[c] = 0;
        if (a.error[c]) {  // the same value on every lane
            active = false;
        } else if (a.integrand_status[c] & kStatusNonFinite) {
            __syncwarp();
            if (lane == 0) a.error[c] = 1;  // "Error (all-subset integrand): Value is not finite"
            active = false;
        }
    }
    if constexpr (Hist) {
        if (active) {
            if (!conditional_probabilities_warp(a, a.vertices + c * env * 4, env, prob, prob + subsets,
                                                prob + subsets + env * env, lane)) {
                if (lane == 0) a.error[c] = 3;  // "MCMCMC seed density is negative or non-finite"
                active = false;
            }
            __syncwarp();
        }
    }
    if (active) {
        // fluxes and selection weights (:411-430, :540-560); masks outside the orders weigh nothing
        const double* values = a.values + c * static_cast<int64_t>(subsets);
        const double* lam = a.lambdas + c * (env + 1);
        for (uint32_t mask = lane; mask < subsets; mask += kWarp) {
            const int o = __popc(mask);
            double f = 0.0, weight = 0.0;
            if (mask != 0 && o >= a.order_min && o <= a.order_max) {
                f = dmul(dmul(lam[o], values[mask]), Hist ? prob[full ^ mask] : 1.0);
                weight = dmul(fabs(f), a.inv_binom[o]);
            }
            flux[mask] = f;
            prefix[mask] = weight;
        }
    }
    if (lane == 0) s_state[warp] = active ? 1 : 0;
    __syncthreads();
    // the local normalisations: lane k adds up chain k's weights in mask order
    if (warp == 0 && lane < per_block && s_state[lane]) {
        double* w = step_smem + static_cast<size_t>(lane) * per_chain + subsets + 1;
        double norm = 0.0;
        for (uint32_t m0 = 0; m0 < subsets; m0 += 8) {  // (mask 0 weighs nothing; subsets >= 8 or the tail below)
            double x[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) x[k] = m0 + k < subsets ? w[m0 + k] : 0.0;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                norm = dadd(norm, x[k]);
                x[k] = norm;
            }
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (m0 + k < subsets) w[m0 + k] = x[k];
        }
        s_norm[lane] = norm;
        if (norm > 0.0 && isfinite(norm)) s_state[lane] = 2;
        else a.error[static_cast<int64_t>(blockIdx.x) * per_block + lane] = 2;  // "MCMCMC local normalization is zero or non-finite"
    }
    __syncthreads();
    if (s_state[warp] == 2) {
        const double norm = s_norm[warp];
        WarpMt64 g(a.mt + c, a.chains, a.mt_index[c], lane);
        // sample_weighted_candidate_mask (:225-250): the first mask whose running weight exceeds the
        // threshold; failing that, the last one of positive finite weight
        const double threshold = dadd(dmul(g.canonical(), dsub(norm, 0.0)), 0.0);
        uint32_t chosen = 0, last_positive = 0;
        bool found = false;
        for (uint32_t m0 = 0; m0 < subsets && !found; m0 += kWarp) {
            const uint32_t mask = m0 + lane;
            const uint32_t hit = __ballot_sync(0xffffffffu, mask > 0 && mask < subsets && prefix[mask] > threshold);
            if (hit) {
                chosen = m0 + __ffs(hit) - 1;
                found = true;
            }
        }
        if (!found) {
            for (uint32_t m0 = 0; m0 < subsets; m0 += kWarp) {
                const uint32_t mask = m0 + lane;
                const int o = __popc(mask);
                bool positive = false;
                if (mask > 0 && mask < subsets && o >= a.order_min && o <= a.order_max) {
                    const double weight = dmul(fabs(flux[mask]), a.inv_binom[o]);
                    positive = weight > 0.0 && isfinite(weight);
                }
                const uint32_t hit = __ballot_sync(0xffffffffu, positive);
                if (hit) last_positive = m0 + 31 - __clz(static_cast<int>(hit));
            }
            chosen = last_positive;
        }
        // the signal's terms: time = flux / local_normalization, weighted by 1/binomial (:566-571)
        if (a.signal_out)
            for (uint32_t mask = lane; mask < subsets; mask += kWarp)
                flux[mask] = dmul(ddiv(flux[mask], norm), a.inv_binom[__popc(mask)]);
        // create_next_vertices_from_seed_into (:380-400): the retained vertices in
        // order, then children of uniformly chosen parents among the vertices so
        // far (the uniform kernel, mcmcmc_seed.h:51-55, ignores the parent)
        const double* v = a.vertices + c * env * 4;
        double* nv = a.next_vertices + c * env * 4;
        int size = __popc(chosen);
        for (int e = lane; e < 4 * size; e += kWarp) nv[e] = v[4 * nth_set_bit(chosen, e >> 2) + (e & 3)];
        for (; size < env; ++size) {
            const int parent = mt_uniform_int(g, size);
            if constexpr (Hist) {
                __syncwarp();  // the parent's coordinates, written by other lanes
                double child[4];
                hist_child(a, g, nv + 4 * parent, child);
                if (lane < 4) nv[4 * size + lane] = lane == 0 ? child[0] : (lane == 1 ? child[1] : (lane == 2 ? child[2] : child[3]));
            } else {
                (void)parent;
                const double x = g.canonical4();
                if (lane < 4) nv[4 * size + lane] = x;
            }
        }
        if (lane == 0) {
            a.mt_index[c] = g.index;
            if (a.chosen_out) a.chosen_out[row * a.chains + c] = chosen;
            if (a.retained_out) a.retained_out[c] = chosen;
            if (a.norm_out) a.norm_out[row * a.chains + c] = norm;
            if (a.warmup) ++a.counts[c * (env + 1) + __popc(chosen)];
        }
    }
    if (!a.signal_out) return;  // every thread
    __syncthreads();
    // each order's terms in mask order, (chain, order) pairs dealt to the block's threads
    for (int item = threadIdx.x; item < per_block * (env + 1); item += blockDim.x) {
        const int k = item / (env + 1), order = item - k * (env + 1);
        if (s_state[k] != 2) continue;
        const double* terms = step_smem + static_cast<size_t>(k) * per_chain;
        double sig = 0.0;
        if (order >= 1 && order >= a.order_min && order <= a.order_max) {
            const uint32_t masks = kBinomial.c[env][order];
            uint32_t m = (1u << order) - 1u;
            for (uint32_t r = 0; r < masks; ++r, m = next_same_popcount(m)) sig = dadd(sig, terms[m]);
        }
        a.signal_out[(row * a.chains + static_cast<int64_t>(blockIdx.x) * per_block + k) * (env + 1) + order] = sig;
    }
}

// The histogram seed kernel's conditional generation probabilities, one warp
// per chain, into a.cprob; a negative or non-finite seed density stops the
// chain (error 3), which the step kernel then skips.
constexpr int kHistWarps = 4;
__global__ void __launch_bounds__(kHistWarps * 32) mcmcmc_hist_probs(const __grid_constant__ McmcmcStepArgs a) {
    __shared__ double sd_all[kHistWarps][kMcmcmcMaxEnvelope * kMcmcmcMaxEnvelope];
    __shared__ double cd0_all[kHistWarps][kMcmcmcMaxEnvelope];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t c = static_cast<int64_t>(blockIdx.x) * kHistWarps + warp;
    if (c >= a.chains) return;  // whole warps
    // both read the same value on every lane; the step kernel reports a non-finite integrand
    if (a.error[c] || (a.integrand_status[c] & kStatusNonFinite)) return;
    const int env = a.envelope;
    double* cprob = a.cprob + c * (int64_t{1} << env);
    const double* v = a.vertices + c * env * 4;
    if (!conditional_probabilities_warp(a, v, env, cprob, sd_all[warp], cd0_all[warp], lane) && lane == 0)
        a.error[c] = 3;  // "MCMCMC seed density is negative or non-finite"
}

__global__ void mcmcmc_advance_row(int64_t* row, int64_t rows) {
    if (threadIdx.x == 0 && blockIdx.x == 0) *row = (*row + 1) % rows;
}

}  // namespace

cudaError_t launch_mcmcmc_advance_row(int64_t* row, int64_t rows, cudaStream_t stream) {
    mcmcmc_advance_row<<<1, 32, 0, stream>>>(row, rows);
    return cudaGetLastError();
}

cudaError_t launch_mcmcmc_init(int64_t chains, int envelope, const uint64_t* seeds, uint64_t* mt, int32_t* mt_index,
                               double* vertices, cudaStream_t stream) {
    if (chains <= 0) return cudaSuccess;
    mcmcmc_init<<<static_cast<unsigned>((chains + 127) / 128), 128, 0, stream>>>(chains, envelope, seeds, mt,
                                                                                mt_index, vertices);
    return cudaGetLastError();
}

cudaError_t launch_mcmcmc_step(const McmcmcStepArgs& args, cudaStream_t stream, int* kernels) {
    *kernels = 0;
    if (args.chains <= 0) return cudaSuccess;
    const bool hist = args.tau_bins > 0;
    if (args.chains < step_warp_max_chains(args.envelope, hist)) {
        // as many chains per block as leave every SM a block, while shared memory holds them
        const size_t per_chain = step_doubles(args.envelope, hist) * sizeof(double);
        int per_block = 1;
        while (per_block * 2 <= kStepMaxChainsPerBlock && args.chains >= 2 * 152 * static_cast<int64_t>(per_block) &&
               per_chain * per_block * 2 <= 96 * 1024)
            per_block *= 2;
        const size_t smem = per_chain * per_block;
        auto kernel = hist ? mcmcmc_step_warp<true> : mcmcmc_step_warp<false>;
        cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        if (err != cudaSuccess) return err;
        kernel<<<static_cast<unsigned>((args.chains + per_block - 1) / per_block), per_block * kWarp, smem, stream>>>(args);
        *kernels = 1;
        return cudaGetLastError();
    }
    const unsigned grid = static_cast<unsigned>((args.chains + 127) / 128);
    *kernels = hist ? 2 : 1;
    if (hist) {
        mcmcmc_hist_probs<<<static_cast<unsigned>((args.chains + kHistWarps - 1) / kHistWarps), kHistWarps * 32, 0,
                            stream>>>(args);
        const cudaError_t err = cudaGetLastError();
        if (err != cudaSuccess) return err;
        mcmcmc_step<true><<<grid, 128, 0, stream>>>(args);
    } else {
        mcmcmc_step<false><<<grid, 128, 0, stream>>>(args);
    }
    return cudaGetLastError();
}

}  // namespace cdet
