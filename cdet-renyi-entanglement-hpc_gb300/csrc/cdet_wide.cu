// The double-double integrand behind the split assembly (orders <= 10), in
// 113-bit integer arithmetic (cdet_widefloat.cuh).
//
// On the FP64 assembly the double-double mode is the reference's DoubleDouble
// arithmetic bit for bit (cdet_dd.cu). On the split assembly's Green matrices
// only the accuracy counts, and there the FP64 pipe is the wrong unit: a
// double-double pair update of the recursion is 16 operations of 64 to 74
// clocks. Here every step runs on the 32-bit integer pipes, to 113 bits.
//
// One block of four warps (of one warp up to order 7) runs a configuration,
// both sets in turn: the compact Schur recursion of the minors (the FP64 form's
// layout, 16-byte elements: 39 KB at order 10, five blocks per SM), a level's
// items dealt to all of its threads, then a[mask] = up * down and the connected
// recursion in the same shared memory. In the recursion a and dp are kept unpacked (mantissa
// and exponent arrays), and a mask's sum is a 192-bit integer (WideSum) on a scale
// that bounds every term of its popcount level, or, where the mask's terms may lie
// far below that (a vertex far from all others), its own largest term: integer
// addition is associative, so the submasks of a mask are split over up to 32 lanes
// and the parts added in any order without changing the value. Blocks take
// configurations from the order-sorted slots (decreasing order) through an atomic
// queue head.
//
// Bound: the integer pipes and, next to them, shared-memory bandwidth (two
// 16-byte reads of scattered masks per pair update). Measured at 6x6 / degree
// 96 / order 10, 8,192 configurations, against double-double minors by warps
// and one lane per configuration for the recursion: 35.2 -> 4.1 ms after the
// assembly (5.32 ms the call; with the level's scale for every mask, which leaves a
// graded matrix fewer bits than double-double steps, 5.27; with a scale of its own
// for every mask 5.53). Against a binary128 evaluation both have the same errors (256
// configurations per order 2..10 on three lattices: medians 4e-16 to 2e-15,
// maxima below 2e-12): the Green entries set them.
#include "cdet_dd.cuh"
#include "cdet_widefloat.cuh"

#include <algorithm>

namespace cdet {

namespace {

// Orders up to 7 keep four warps waiting on one another and run a warp per
// configuration, 20 of them per SM (a lone configuration takes as long): order
// 7, 4,096 configurations, one spin, 911 us with four warps each, 510 with one;
// order 2: 478 and 269. Order 1 needs neither, only a thread. Four-warp blocks
// leave the small configurations of a mixed batch to a second launch of one-warp
// blocks when more than wide_tail per block are there; fewer they take along while
// the others still run the large ones. Truncated-geometric orders, one launch and
// two: up to 8, one spin, 4,096 (2.2 per block) 478 and 470 us, 6,500 650 and 531;
// up to 9, 4,096 (3.4) 501 and 526, 6,500 688 and 590; up to 10, 4,096 (5.4) 547
// and 742, two spins, 2,800 (6.1) 750 and 970.
constexpr int kWideWarpMaxOrder = 7;
__host__ __device__ inline int64_t wide_tail(int max_order) { return max_order <= 8 ? 3 : max_order == 9 ? 5 : 8; }
constexpr int32_t kNoExponent = -(1 << 24);

__device__ __forceinline__ Wide from_double(double x) {
    return wide_from_bits(static_cast<uint64_t>(__double_as_longlong(x)));
}
__device__ __forceinline__ Wide from_dd(DD x) { return wide_add(from_double(x.hi), from_double(x.lo)); }

__device__ __forceinline__ Wide inverse(const Wide& a) {
    return wide_inverse(a, [](uint64_t bits) {
        return static_cast<uint64_t>(__double_as_longlong(__drcp_rn(__longlong_as_double(static_cast<long long>(bits)))));
    });
}

// The leading 106 bits as a DoubleDouble.
__device__ DD to_dd(const uint32_t (&m)[4], int32_t e, uint32_t sign) {
    if (e < kWideFlush) return DD{0.0, 0.0};
    const uint64_t top = (static_cast<uint64_t>(m[3]) << 32) | m[2], low = (static_cast<uint64_t>(m[1]) << 32) | m[0];
    const uint64_t hi = top >> 10;                                            // bits 126..74
    const uint64_t lo = ((top & 0x3FFu) << 43) | (low >> 21);                 // bits 73..21
    double h = ldexp(static_cast<double>(hi), e - 53), l = ldexp(static_cast<double>(lo), e - 106);
    if (sign) {
        h = -h;
        l = -l;
    }
    DD r;
    r.hi = quick_two_sum(h, l, r.lo);
    return r;
}

// item / d for item * d < 2^32 with magic = 0xFFFFFFFF / d + 1
__device__ __forceinline__ int div_magic(int item, uint32_t magic) {
    return static_cast<int>(__umulhi(static_cast<uint32_t>(item), magic));
}

// mat2pm_from_buffer (fast_principle_minors.h:120-246) of one n x n matrix A
// (in shared memory) by the whole block; shifted[mask] ends as the principal
// minor of mask. Returns true when the LU fallback ran.
template <int Threads>
__device__ bool wide_minors(const DD* A, int n, const Problem& p, WidePacked* shifted, int arena, DD* lu_lane) {
    const int tid = threadIdx.x;
    const int msize = n * n;
    const uint32_t subsets = 1u << n;
    double max_abs = 0.0;  // every thread scans all of A: n^2 <= 100 broadcast reads
    for (int k = 0; k < msize; ++k) max_abs = fmax(max_abs, fabs(A[k].hi));
    const DD thresh{p.dd_fpm_shift.hi, p.dd_fpm_shift.lo}, tol{p.dd_tol.hi, p.dd_tol.lo}, zero{0.0, 0.0};
    const DD shift = !dd_lt(thresh, zero) ? thresh : dd_div(DD{max_abs, 0.0}, DD{static_cast<double>(msize), 0.0});
    if (max_abs == 0.0 && dd_zero(shift)) {
        for (uint32_t m = tid; m < subsets; m += Threads) shifted[m] = WidePacked{0u, 0u, 0u, 0u};
        __syncthreads();
        return false;
    }
    const Wide ps = from_dd(shift);
    const bool eps_on = dd_gt(tol, zero) && max_abs > 0.0;
    const WidePacked eps = wide_pack(from_dd(eps_on ? dd_mul(tol, DD{max_abs, 0.0}) : zero));

    WidePacked* old_list = shifted + compact_list_offset(n, 0, arena);
    for (int k = tid; k < msize; k += Threads) old_list[k] = wide_pack(from_double(A[k].hi));
    if (tid == 0) {
        shifted[0] = wide_pack(from_double(1.0));
        shifted[1] = wide_pack(wide_add(ps, from_double(A[0].hi)));
    }
    __syncthreads();
    uint32_t minor_index = 2;
    bool fell_back = false;
    for (int level = 0; level < n - 1; ++level) {
        const int old_size = n - level, old_msize = old_size * old_size;
        const int new_size = old_size - 1, new_msize = new_size * new_size;
        const int sets = 1 << level;
        // pivots' inverses, then the first-column factors, in place
        bool bad_pivot = false;
        for (int set = tid; set < sets; set += Threads) {
            const Wide pivot = wide_add(ps, wide_unpack(old_list[set * old_msize]));
            const WidePacked pa = wide_pack(pivot);
            if ((pa.x | pa.y | pa.z | pa.w) == 0u || (eps_on && wide_abs_le(pa, eps))) bad_pivot = true;
            old_list[set * old_msize] = wide_pack(inverse(pivot));
        }
        if (__syncthreads_or(bad_pivot)) {
            fell_back = true;
            break;
        }
        const uint32_t by_size = 0xFFFFFFFFu / static_cast<uint32_t>(new_size) + 1u;
        for (int item = tid; item < sets * new_size; item += Threads) {
            const int set = new_size == 1 ? item : div_magic(item, by_size);
            WidePacked* entry = old_list + set * old_msize + (item - set * new_size + 1) * old_size;
            *entry = wide_pack(wide_mul(wide_unpack(*entry), wide_unpack(old_list[set * old_msize])));
        }
        __syncthreads();
        if (level == n - 2) {  // the 1 x 1 children, straight to their shifted minors
            for (int set = tid; set < sets; set += Threads) {
                const WidePacked* m = old_list + set * 4;
                const Wide base = wide_unpack(m[3]);
                const Wide l = wide_unpack(m[1]), r = wide_unpack(m[2]);
                // the last list ends at the arena's end, above the minors this level writes
                shifted[minor_index + set] = wide_pack(wide_add(ps, base));
                shifted[minor_index + sets + set] = wide_pack(wide_add(ps, wide_sub_prod(l, r, base)));
            }
            __syncthreads();
            minor_index += 2 * sets;
            break;
        }
        WidePacked* new_list = shifted + compact_list_offset(n, level + 1, arena);
        const int items = sets * new_msize;
        const uint32_t by_msize = 0xFFFFFFFFu / static_cast<uint32_t>(new_msize) + 1u;
        for (int item = tid; item < items; item += Threads) {
            const int set = div_magic(item, by_msize);
            const int e = item - set * new_msize;
            const int row = div_magic(e, by_size);
            const int col = e - row * new_size;
            const WidePacked* src = old_list + set * old_msize;
            const WidePacked base = src[(row + 1) * old_size + col + 1];
            new_list[item] = base;
            new_list[items + item] = wide_pack(
                wide_sub_prod(wide_unpack(src[1 + col]), wide_unpack(src[(row + 1) * old_size]), wide_unpack(base)));
        }
        __syncthreads();
        for (int m = tid; m < 2 * sets; m += Threads)
            shifted[minor_index + m] = wide_pack(wide_add(ps, wide_unpack(new_list[m * new_msize])));
        minor_index += 2 * sets;
        old_list = new_list;
        __syncthreads();
    }
    if (fell_back) {
        // determinant_principal_minors_from_buffer<DoubleDouble> (fast_principle_minors.h:107-115), on the (at
        // most two) warps that have LU scratch
        constexpr int kLu = Threads < 64 ? Threads : 64;
        if (tid < kLu)
            for (uint32_t m = 1 + tid; m < subsets; m += kLu) shifted[m] = wide_pack(from_dd(minor_by_lu_dd(A, n, m, lu_lane)));
        __syncthreads();
        return true;
    }
    for (uint32_t step = 1; step < subsets; step <<= 1) {  // the prefix product over levels
        for (uint32_t set = step + 1 + tid; set < 2 * step; set += Threads)
            shifted[set] = wide_pack(wide_mul(wide_unpack(shifted[set]), wide_unpack(shifted[set - step])));
        __syncthreads();
    }
    for (uint32_t step = subsets; step > 1; step >>= 1) {  // the shift removal, bit by bit from the top
        const uint32_t half = step >> 1;
        const int hb = __ffs(half) - 1;
        for (uint32_t q = tid; q < subsets / 2; q += Threads) {
            const uint32_t ss = ((q >> hb) << (hb + 1)) + half + (q & (half - 1u));
            shifted[ss] = wide_pack(wide_sub_prod(ps, wide_unpack(shifted[ss - half]), wide_unpack(shifted[ss])));
        }
        __syncthreads();
    }
    return false;
}

// The recursion's arrays inside the arena: mantissas of a (the even masks at
// mask >> 1, then the odd ones), their exponent words (e << 1 | sign), and
// those of dp of the odd masks at mask >> 1.
struct RecursionArrays {
    uint4 *a, *dp;
    int32_t *ae, *de;
};
__device__ __forceinline__ RecursionArrays recursion_arrays(void* arena, int n) {
    char* base = static_cast<char*>(arena);
    const size_t count = size_t{1} << n;
    RecursionArrays r;
    r.a = reinterpret_cast<uint4*>(base);
    r.ae = reinterpret_cast<int32_t*>(base + 16 * count);
    r.dp = reinterpret_cast<uint4*>(base + 20 * count);
    r.de = reinterpret_cast<int32_t*>(base + 28 * count);
    return r;
}

// Largest exponents per popcount: of a's even masks, a's odd masks, dp.
struct LevelBounds {
    int32_t even[kDDMaxOrder + 1], odd[kDDMaxOrder + 1], dp[kDDMaxOrder + 1];
};

// compute_dp_ztransform (integrand_replica_randomly_sampled.h:226-290) by the
// whole block, order n >= 2, a in place; returns dp of the full mask on every
// thread.
template <int Threads>
__device__ Wide wide_recursion(const RecursionArrays& r, int n, double threshold, LevelBounds& bounds) {
    const int tid = threadIdx.x;
    const int nbits = n - 1;
    const uint32_t half = 1u << nbits;
    const int thr_log = threshold > 0.0 ? ilogb(threshold) : 0;
    if (tid == 0) {
        r.dp[0] = r.a[half];
        r.de[0] = r.ae[half];
        bounds.dp[1] = r.ae[half] >> 1;
    }
    __syncthreads();
    for (int k = 2; k <= n; ++k) {
        const int kk = k - 1;
        const int masks = static_cast<int>(kBinomial.c[nbits][kk]);
        const int subs = 1 << kk;
        // every |a[mask]| and |dp[sub] a[mask ^ sub]| of the level is below 2^(level_bound + 1)
        int32_t level_bound = bounds.odd[k];
        for (int j = 1; j < k; ++j) level_bound = max(level_bound, bounds.dp[j] + bounds.even[k - j]);
        for (int base = 0; base < masks;) {
            const int remaining = masks - base;
            int L = 1, take = Threads;
            if (remaining < Threads) {
                while (L * 2 * remaining <= Threads && L * 2 <= subs && L < kWarp) L *= 2;
                take = remaining;
                if (4 * L * remaining < 3 * Threads && L * 2 <= subs && L < kWarp) {  // < 75 % of the threads busy
                    L *= 2;
                    take = Threads / L;
                }
            }
            const int q = __ffs(L) - 1;
            const int idx = base + (tid >> q);
            const int j = tid & (L - 1);
            const bool active = (tid >> q) < take && idx < masks;
            uint32_t rest = 0, low = 0, fixed = 0;
            if (active) {
                rest = colex_subset(static_cast<uint32_t>(idx), kk, nbits);
                // the lane fixes the q highest bits of rest and walks the submasks of the others
                uint32_t top = 0;
                low = rest;
                for (int t = 0; t < q; ++t) {
                    const uint32_t hb = 1u << (31 - __clz(static_cast<int>(low)));
                    top |= hb;
                    low ^= hb;
                }
                uint32_t tb = top;
                for (int t = 0; t < q; ++t) {
                    const uint32_t lb = tb & (~tb + 1u);
                    if ((j >> t) & 1) fixed |= lb;
                    tb ^= lb;
                }
            }
            // the sum's scale: the level's where a[mask] alone shows that the terms come near it, else the
            // largest exponent among the mask's own terms
            int32_t bound = level_bound;
            const int32_t own = active ? (r.ae[half + rest] >> 1) - 1 : level_bound;
            const bool far = own < level_bound - kSumSlack;
            if (__any_sync(0xffffffffu, far)) {
                if (far) {
                    bound = own;
                    for (uint32_t sl = low;; sl = (sl - 1u) & low) {
                        const uint32_t sm = fixed | sl;
                        if (sm != rest) bound = max(bound, (r.de[sm] >> 1) + (r.ae[rest ^ sm] >> 1));
                        if (sl == 0) break;
                    }
                }
                for (int off = 1; off < L; off <<= 1) bound = max(bound, __shfl_xor_sync(0xffffffffu, bound, off));
            }
            WideSum sum;
            if (active) {
                if (j == 0) {  // a[mask]: m 2^(e - 127) = m 2^((e - 1) - 126)
                    const uint4 m = r.a[half + rest];
                    const uint32_t am[4] = {m.x, m.y, m.z, m.w};
                    sum.add(am, bound - own, r.ae[half + rest] & 1);
                }
                for (uint32_t sl = low;; sl = (sl - 1u) & low) {
                    const uint32_t sm = fixed | sl;
                    if (sm != rest) {  // (dp of rest itself is what is being formed)
                        const uint4 x = r.dp[sm], y = r.a[rest ^ sm];
                        const int32_t ex = r.de[sm], ey = r.ae[rest ^ sm];
                        const uint32_t xm[4] = {x.x, x.y, x.z, x.w}, ym[4] = {y.x, y.y, y.z, y.w};
                        uint32_t pm[4];
                        mul_top(xm, ym, pm);
                        sum.add(pm, bound - ((ex >> 1) + (ey >> 1)), ((ex ^ ey) & 1) == 0);  // sum -= dp a
                    }
                    if (sl == 0) break;
                }
            }
            for (int off = 1; off < L; off <<= 1) {
                WideSum other;
#pragma unroll
                for (int i = 0; i < kSumWords; ++i) other.acc[i] = __shfl_xor_sync(0xffffffffu, sum.acc[i], off);
#pragma unroll
                for (int i = 0; i < kMagWords; ++i) other.mag[i] = __shfl_xor_sync(0xffffffffu, sum.mag[i], off);
                sum.merge(other);
            }
            if (active && j == 0) {
                const Wide v = sum.value(bound, threshold, thr_log);
                r.dp[rest] = make_uint4(v.m[0], v.m[1], v.m[2], v.m[3]);
                r.de[rest] = (v.e << 1) | static_cast<int32_t>(v.sign);
                atomicMax(&bounds.dp[k], v.e);
            }
            base += take;
        }
        __syncthreads();
    }
    const uint4 m = r.dp[half - 1u];
    const int32_t es = r.de[half - 1u];
    Wide top;
    top.m[0] = m.x;
    top.m[1] = m.y;
    top.m[2] = m.z;
    top.m[3] = m.w;
    top.e = es >> 1;
    top.sign = es & 1;
    return top;
}

template <int Threads, int MaxOrder>
__global__ void __launch_bounds__(Threads, 640 / Threads) integrand_wide(const __grid_constant__ Problem p,
                                                                           const __grid_constant__ Scratch w, int arena,
                                                                           bool singles, bool split) {
    extern __shared__ __align__(16) unsigned char wide_smem[];
    __shared__ DD A[kDDMaxOrder * kDDMaxOrder];
    __shared__ LevelBounds bounds;
    __shared__ uint32_t next_slot;
    WidePacked* minors = reinterpret_cast<WidePacked*>(wide_smem);
    WidePacked* up_minors = minors + arena;  // the spin-up minors while the spin-down ones are formed
    const int tid = threadIdx.x;
    const int nmax = p.max_order;
    // a lane's LU-fallback matrix: two lanes' FP64 regions of the scratch, at most two of the block's warps
    constexpr int kLu = Threads < 64 ? Threads : 64;
    DD* lu_lane =
        reinterpret_cast<DD*>(w.lu_scratch + (static_cast<size_t>(blockIdx.x) * kLu + tid % kLu) * 2 * nmax * nmax);
    uint32_t* head = w.order_count + kQueueHeadIndex;
    // every block leaves the small configurations to the second launch, or none does: the sort left the end of the
    // order-8 slots in its bucket
    const bool leave = split && static_cast<uint32_t>(p.batch) - __ldg(w.order_count + nmax - kWideWarpMaxOrder - 1) >
                                    static_cast<uint32_t>(wide_tail(nmax)) * gridDim.x;
    if (singles) {  // order 1, a product of two diagonal entries: a thread per configuration
        for (int64_t c = static_cast<int64_t>(blockIdx.x) * Threads + tid; c < p.batch;
             c += static_cast<int64_t>(gridDim.x) * Threads) {
            if (__ldg(p.orders + c) != 1) continue;
            const DD result = dd_sub(dd_order1_value(p, w, c, 0), dd_mul(DD{2.0, 0.0}, dd_order1_value(p, w, c, 1)));
            p.values[c] = dadd(result.hi, result.lo);
        }
    }
    for (bool last = false; !last;) {
        if (tid == 0) next_slot = atomicAdd(head, 1u);
        __syncthreads();
        const uint32_t slot = next_slot;
        if (slot >= static_cast<uint32_t>(p.batch)) break;
        const int64_t c = __ldg(w.config_at + slot);
        const int n = __ldg(p.orders + c);
        __syncthreads();  // next_slot is read before the next pop
        if (n <= 1 || n > nmax) break;  // the slots' end: order 1 (above), then invalid orders (flagged by the assembly)
        last = leave && n <= kWideWarpMaxOrder;
        int32_t status = 0;
        DD value[2];
        for (int set = 0; set < 2; ++set) {
            const double* green = w.green + (c * 2 + set) * 2 * static_cast<int64_t>(nmax) * nmax;
            const bool one_spin = p.same_spin[set] != 0;
            const uint32_t count = 1u << n, half = count / 2;
            bool fell_back = false, finite = true;
            for (int spin = 0; spin < (one_spin ? 1 : 2); ++spin) {
                bool bad = false;
                for (int k = tid; k < n * n; k += Threads) {
                    const double x = green[spin * static_cast<int64_t>(nmax) * nmax + k];
                    bad |= !isfinite(x);
                    A[k] = DD{x, 0.0};
                }
                if (spin == 1)
                    for (uint32_t m = tid; m < count; m += Threads) up_minors[m] = minors[m];
                if (__syncthreads_or(bad)) {
                    finite = false;
                    break;
                }
                fell_back |= wide_minors<Threads>(A, n, p, minors, arena, lu_lane);
            }
            if (!finite) {  // no number to compute: the double-double arithmetic would end in NaN
                value[set] = DD{__longlong_as_double(0x7FF8000000000000ll), 0.0};
                status |= kStatusNonFinite;
                __syncthreads();
                continue;
            }
            // a[mask] = up[mask] * down[mask] (:254-257), unpacked into the recursion's arrays
            const RecursionArrays r = recursion_arrays(minors, n);
            constexpr int kPer = (1 << MaxOrder) / Threads;
            Wide a[kPer];
#pragma unroll
            for (int i = 0; i < kPer; ++i) {
                const uint32_t m = tid + i * Threads;
                if (m < count) {
                    const Wide down = wide_unpack(minors[m]);
                    a[i] = wide_mul(one_spin ? down : wide_unpack(up_minors[m]), down);
                }
            }
            if (tid <= kDDMaxOrder) bounds.even[tid] = bounds.odd[tid] = bounds.dp[tid] = kNoExponent;
            __syncthreads();
#pragma unroll
            for (int i = 0; i < kPer; ++i) {
                const uint32_t m = tid + i * Threads;
                if (m > 0 && m < count) {
                    const uint32_t at = ((m & 1u) ? half : 0u) + (m >> 1);
                    r.a[at] = make_uint4(a[i].m[0], a[i].m[1], a[i].m[2], a[i].m[3]);
                    r.ae[at] = (a[i].e << 1) | static_cast<int32_t>(a[i].sign);
                    atomicMax(((m & 1u) ? bounds.odd : bounds.even) + __popc(m), a[i].e);
                }
            }
            __syncthreads();
            const Wide top = wide_recursion<Threads>(r, n, p.dd_threshold.hi, bounds);
            value[set] = dd_mul(DD{p.pref_dd[set][n].hi, p.pref_dd[set][n].lo}, to_dd(top.m, top.e, top.sign));
            if (!dd_finite(value[set])) status |= kStatusNonFinite;
            if (fell_back) status |= kStatusFpmFallback;
            __syncthreads();  // the next set reuses the workspace
        }
        if (tid == 0) {
            // twisted - DoubleDouble(2) * ordinary (cdet_integrand_evaluator.h:233-263), then to double
            const DD result = dd_sub(value[0], dd_mul(DD{2.0, 0.0}, value[1]));
            p.values[c] = dadd(result.hi, result.lo);
            if (status) atomicOr(p.status + c, status);
        }
    }
}

}  // namespace

namespace {
struct WideGrid {
    int arena, threads;
    size_t smem;
    int64_t blocks;
};

WideGrid wide_grid(const Problem& p, const Scratch& w, int sm_count, int max_order, int threads) {
    const bool two_spins = !(p.same_spin[0] && p.same_spin[1]);
    WideGrid g;
    g.threads = threads;
    g.arena = compact_minors_layout(max_order, false).arena;
    g.smem = (static_cast<size_t>(g.arena) + (two_spins ? size_t{1} << max_order : 0)) * sizeof(WidePacked);
    const int sms = sm_count > 0 ? sm_count : 152;
    // as many blocks as the shared memory holds (five of four warps at order 10)
    const int per_sm = static_cast<int>(
        std::max<size_t>(1, std::min<size_t>(threads == kWarp ? 20 : 12, (227 * 1024) / (g.smem + 4096))));
    g.blocks = std::min<int64_t>(static_cast<int64_t>(sms) * per_sm, p.batch);
    // the LU-fallback regions of the scratch: two lanes' for each lane of a block's first (at most two) warps
    const int64_t lu_warps = threads == kWarp ? 2 : 4;
    g.blocks = std::min<int64_t>(g.blocks, std::max<int64_t>(1, static_cast<int64_t>(w.ws_warps) / lu_warps));
    return g;
}

template <int Threads, int MaxOrder>
cudaError_t launch_wide(const Problem& p, const Scratch& w, const WideGrid& g, bool singles, bool split,
                        cudaStream_t stream) {
    const auto kernel = integrand_wide<Threads, MaxOrder>;
    const cudaError_t err =
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(g.smem));
    if (err != cudaSuccess) return err;
    kernel<<<static_cast<unsigned>(g.blocks), Threads, g.smem, stream>>>(p, w, g.arena, singles, split);
    return cudaGetLastError();
}

// A batch so large that a warp per small configuration may pay a second launch (the kernel knows how many are
// small; a sort in one launch leaves no bucket ends).
bool wide_splits(const Problem& p, int64_t blocks) {
    return p.max_order > kWideWarpMaxOrder && p.batch > wide_tail(p.max_order) * blocks && order_sort_launches(p.batch) > 1;
}
}  // namespace

int wide_launches(const Problem& p, const Scratch& w, int sm_count) {
    return wide_splits(p, wide_grid(p, w, sm_count, p.max_order, 4 * kWarp).blocks) ? 2 : 1;
}

cudaError_t launch_integrand_wide(const Problem& p, const Scratch& w, int sm_count, cudaStream_t stream) {
    if (p.batch <= 0) return cudaSuccess;
    const int small = std::min(p.max_order, kWideWarpMaxOrder);
    const WideGrid warps = wide_grid(p, w, sm_count, small, kWarp);
    if (p.max_order <= kWideWarpMaxOrder)
        return launch_wide<kWarp, kWideWarpMaxOrder>(p, w, warps, true, false, stream);
    const WideGrid g = wide_grid(p, w, sm_count, p.max_order, 4 * kWarp);
    const bool split = wide_splits(p, g.blocks);
    const cudaError_t err = launch_wide<4 * kWarp, kDDMaxOrder>(p, w, g, true, split, stream);
    if (err != cudaSuccess || !split) return err;
    return launch_wide<kWarp, kWideWarpMaxOrder>(p, w, warps, false, false, stream);
}

}  // namespace cdet
