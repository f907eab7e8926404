// The reference's double-double integrand mode on the GPU:
// INTEGRAND_REAL=double_double with VECTOR_REAL=double
// (cdet_integrand_evaluator.h:431-465, precision_config.h:15-26).
//
// The Green matrices are the FP64 form's (the same Clenshaw sums, shifts and
// scale in double, integrand_replica_randomly_sampled.h:434-484). Each entry
// is widened to DoubleDouble(x, 0), and from there every operation is the
// reference's DoubleDouble arithmetic (utility/types.h:30-182) in the
// reference's order: the shifted Schur-complement recursion with its
// whole-matrix LU fallback (fast_principle_minors.h:39-246), the connected
// recursion with the round-off filter (integrand_replica_randomly_sampled.h:
// 226-290), the double-double prefactor and twisted - 2 ordinary. The order-1
// branch widens the unshifted diagonal value and adds the DoubleDouble shifts
// alpha / U (:173-213). With the reference's DoubleDouble being error-free
// transforms of doubles, the values are the reference's bit for bit.
//
// One persistent kernel after the assembly: warps take configurations from
// the order-sorted slots (decreasing order) through an atomic queue head; a
// warp runs one configuration's minors and recursion in its shared-memory
// workspace (the compact minors layout in DoubleDouble elements, A and one
// arena per spin: 40.5 KB per warp at order 10 with one spin per set, five
// warps per SM), the masks of a popcount level dealt to its lanes, each mask's
// submask sum on one lane in the reference's order.
#include "cdet_dd.cuh"

#include <algorithm>

namespace cdet {

namespace {

__device__ __forceinline__ DD shfl_dd(DD v, int src_lane_xor) {
    return DD{__shfl_xor_sync(0xffffffffu, v.hi, src_lane_xor), __shfl_xor_sync(0xffffffffu, v.lo, src_lane_xor)};
}

// mat2pm_from_buffer<DoubleDouble> (fast_principle_minors.h:120-246) for one
// matrix on one warp: shifted[mask] (mask >= 1) ends as the principal minor of
// the rows and columns in mask. Returns true when the LU fallback ran.
__device__ bool mat2pm_dd_warp(const DD* A, int n, DD tol, DD thresh, const WsLayout& lay, DD* ws, DD* shifted,
                               DD* lu_lane, int lane) {
    const int msize = n * n;
    const uint32_t subsets = 1u << n;
    const DD zero{0.0, 0.0};
    DD max_abs = zero;  // the first maximal entry, as the sequential scan keeps it
    for (int k = lane; k < msize; k += kWarp) {
        const DD e = dd_abs(A[k]);
        if (dd_gt(e, max_abs)) max_abs = e;
    }
    for (int off = 16; off > 0; off >>= 1) {
        const DD o = shfl_dd(max_abs, off);
        if (dd_gt(o, max_abs)) max_abs = o;
    }
    const bool explicit_shift = !dd_lt(thresh, zero);
    const DD p = explicit_shift ? thresh : dd_div(max_abs, DD{static_cast<double>(msize), 0.0});
    if (dd_eq(max_abs, zero) && dd_eq(p, zero)) {
        for (uint32_t m = lane; m < subsets; m += kWarp) shifted[m] = zero;
        __syncwarp();
        return false;
    }
    const DD fallback_eps = (dd_gt(tol, zero) && dd_gt(max_abs, zero)) ? dd_mul(tol, max_abs) : zero;
    const bool eps_on = dd_gt(fallback_eps, zero);
    // The compact arena (compact_minors_layout): the level lists share
    // shifted's arena with the minors, each node's pivot inverse replaces its
    // pivot entry and its factors column 0, each shifted minor is written once
    // as p + its pivot entry (the initialise-then-add form's value).
    DD* old_list = shifted + compact_list_offset(n, 0, lay.arena);
    DD* new_list = nullptr;
    for (int k = lane; k < msize; k += kWarp) old_list[k] = A[k];
    if (lane == 0) shifted[0] = DD{1.0, 0.0};
    __syncwarp();
    if (lane == 0) shifted[1] = dd_add(p, old_list[0]);
    __syncwarp();
    uint32_t minor_index = 2;
    bool fell_back = false;
    for (int level = 0; level < n - 1; ++level) {
        const int old_size = n - level;
        const int old_msize = old_size * old_size;
        const int new_size = old_size - 1;
        const int new_msize = new_size * new_size;
        const int sets = 1 << level;
        bool bad_pivot = false;
        for (int set = lane; set < sets; set += kWarp) {
            const DD pivot = dd_add(old_list[set * old_msize], p);
            const DD pa = dd_abs(pivot);
            if (dd_eq(pa, zero) || (eps_on && !dd_gt(pa, fallback_eps))) bad_pivot = true;
            old_list[set * old_msize] = dd_div(DD{1.0, 0.0}, pivot);
        }
        if (__any_sync(0xffffffffu, bad_pivot)) {
            fell_back = true;
            break;
        }
        __syncwarp();
        for (int item = lane; item < sets * new_size; item += kWarp) {
            const int set = item / new_size;
            const int row = item - set * new_size;
            DD* entry = old_list + set * old_msize + (row + 1) * old_size;
            *entry = dd_mul(*entry, old_list[set * old_msize]);
        }
        __syncwarp();
        if (level == n - 2) {
            // the last level's 1 x 1 children, straight to their shifted minors
            for (int set = lane; set < sets; set += kWarp) {
                const DD* m = old_list + set * 4;
                const DD base = m[3];
                shifted[minor_index + set] = dd_add(p, base);
                shifted[minor_index + sets + set] = dd_add(p, dd_sub_prod(m[1], m[2], base));
            }
            __syncwarp();
            minor_index += 2 * sets;
            break;
        }
        new_list = shifted + compact_list_offset(n, level + 1, lay.arena);
        const int items = sets * new_msize;
#pragma unroll 4
        for (int item = lane; item < items; item += kWarp) {  // independent items: chains in flight
            const int set = item / new_msize;
            const int e = item - set * new_msize;
            const int row = e / new_size;
            const int col = e - row * new_size;
            const int src = set * old_msize;
            const DD base = old_list[src + (row + 1) * old_size + col + 1];
            new_list[item] = base;
            new_list[items + item] =
                dd_sub_prod(old_list[src + 1 + col], old_list[src + (row + 1) * old_size], base);
        }
        __syncwarp();
        for (int m = lane; m < 2 * sets; m += kWarp)
            shifted[minor_index + m] = dd_add(p, new_list[m * new_msize]);
        minor_index += 2 * sets;
        old_list = new_list;
        __syncwarp();
    }
    if (fell_back) {
        // determinant_principal_minors_from_buffer<DoubleDouble> (fast_principle_minors.h:107-115)
        for (uint32_t m = 1 + lane; m < subsets; m += kWarp) shifted[m] = minor_by_lu_dd(A, n, m, lu_lane);
        __syncwarp();
        return true;
    }
    for (uint32_t step = 1; step < subsets; step <<= 1) {  // the prefix product over levels
#pragma unroll 4
        for (uint32_t set = step + 1 + lane; set < 2 * step; set += kWarp)
            shifted[set] = dd_mul(shifted[set], shifted[set - step]);
        __syncwarp();
    }
    for (uint32_t step = subsets; step > 1; step >>= 1) {  // the shift removal, bit by bit from the top
        const uint32_t half = step >> 1;
        const int hb = __ffs(half) - 1;  // half = 2^hb
#pragma unroll 4
        for (uint32_t q = lane; q < subsets / 2; q += kWarp) {
            const uint32_t ss = ((q >> hb) << (hb + 1)) + half + (q & (half - 1u));
            shifted[ss] = dd_sub_prod(p, shifted[ss - half], shifted[ss]);
        }
        __syncwarp();
    }
    return false;
}

// compute_dp_ztransform<DoubleDouble> (integrand_replica_randomly_sampled.h:
// 226-290) on one warp for order n >= 2: a[mask] for every mask, dp of the
// masks holding vertex 0 into dp_s[mask >> 1]; each mask's submask sum on one
// lane, its terms in the reference's descending order.
__device__ DD cdet_dd_warp(const DD* a, DD* dp_s, int n, DD threshold, int lane) {
    const DD zero{0.0, 0.0};
    const bool filter = dd_gt(threshold, zero);
    if (lane == 0) dp_s[0] = a[1];
    __syncwarp();
    const int nbits = n - 1;
    for (int k = 2; k <= n; ++k) {
        const int kk = k - 1;
        const uint32_t masks = kBinomial.c[nbits][kk];
        for (uint32_t idx = lane; idx < masks; idx += kWarp) {
            const uint32_t rest = colex_subset(idx, kk, nbits);
            DD acc = a[(rest << 1) | 1u];
            DD rhs = dd_abs(acc);
            for (uint32_t sm = (rest - 1u) & rest;; sm = (sm - 1u) & rest) {
                const DD term = dd_mul(dp_s[sm], a[(rest ^ sm) << 1]);
                acc = dd_sub(acc, term);
                rhs = dd_add(rhs, dd_abs(term));
                if (sm == 0) break;
            }
            if (filter && dd_lt(dd_abs(acc), dd_mul(threshold, rhs))) acc = zero;
            dp_s[rest] = acc;
        }
        __syncwarp();  // the next level reads this one
    }
    return dp_s[(1u << nbits) - 1u];
}

// One set of configuration c (order n): its prefactored DoubleDouble value.
__device__ DD dd_set_value(const Problem& p, const Scratch& w, int64_t c, int set, int n, const WsLayout& lay,
                           DD* ws, DD* lu_lane, int lane, int32_t& status) {
    const int nmax = p.max_order;
    if (n == 1) return dd_order1_value(p, w, c, set);
    const double* green = w.green + (c * 2 + set) * 2 * static_cast<int64_t>(nmax) * nmax;
    DD* A = ws + lay.a;
    const DD tol{p.dd_tol.hi, p.dd_tol.lo}, thresh{p.dd_fpm_shift.hi, p.dd_fpm_shift.lo};
    bool fb = false;
    for (int k = lane; k < n * n; k += kWarp) A[k] = DD{green[k], 0.0};
    __syncwarp();
    DD* su = ws + lay.shifted_up;
    fb |= mat2pm_dd_warp(A, n, tol, thresh, lay, ws, su, lu_lane, lane);
    const bool one_spin = p.same_spin[set] != 0;
    if (!one_spin) {
        for (int k = lane; k < n * n; k += kWarp) A[k] = DD{green[static_cast<int64_t>(nmax) * nmax + k], 0.0};
        __syncwarp();
        fb |= mat2pm_dd_warp(A, n, tol, thresh, lay, ws, ws + lay.shifted_down, lu_lane, lane);
    }
    const DD* sd = one_spin ? su : ws + lay.shifted_down;
    // a[mask] = up[mask - 1] * down[mask - 1] (:254-257), in place of the up minors
    for (uint32_t m = lane; m < (1u << n); m += kWarp) su[m] = m == 0 ? DD{0.0, 0.0} : dd_mul(su[m], sd[m]);
    __syncwarp();
    const DD top = cdet_dd_warp(su, ws + lay.old_list, n, DD{p.dd_threshold.hi, p.dd_threshold.lo}, lane);
    const DD value = dd_mul(DD{p.pref_dd[set][n].hi, p.pref_dd[set][n].lo}, top);
    if (!dd_finite(value)) status |= kStatusNonFinite;
    if (fb) status |= kStatusFpmFallback;
    __syncwarp();  // the next set reuses the workspace
    return value;
}

__global__ void __launch_bounds__(kDDMaxWarps * 32) integrand_dd(const __grid_constant__ Problem p,
                                                   const __grid_constant__ Scratch w) {
    extern __shared__ double dd_smem[];
    const int lane = threadIdx.x & (kWarp - 1);
    const int warp_in_block = threadIdx.x / kWarp;
    const int warps_per_block = blockDim.x / kWarp;
    const int64_t global_warp = static_cast<int64_t>(blockIdx.x) * warps_per_block + warp_in_block;
    const int nmax = p.max_order;
    const WsLayout lay = compact_minors_layout(nmax, !(p.same_spin[0] && p.same_spin[1]), true);
    DD* ws = reinterpret_cast<DD*>(dd_smem) + static_cast<size_t>(warp_in_block) * lay.total;
    // a lane's LU-fallback matrix: two lanes' FP64 regions of the scratch
    DD* lu_lane = reinterpret_cast<DD*>(w.lu_scratch + (static_cast<size_t>(global_warp) * kWarp + lane) * 2 *
                                                           nmax * nmax);
    uint32_t* head = w.order_count + kQueueHeadIndex;
    const uint32_t batch = static_cast<uint32_t>(p.batch);
    for (;;) {
        uint32_t slot = 0;
        if (lane == 0) slot = atomicAdd(head, 1u);
        slot = __shfl_sync(0xffffffffu, slot, 0);
        if (slot >= batch) break;
        const int64_t c = __ldg(w.config_at + slot);
        const int n = __ldg(p.orders + c);
        if (n < 1 || n > nmax) continue;  // flagged by the assembly
        int32_t status = 0;
        const DD twisted = dd_set_value(p, w, c, 0, n, lay, ws, lu_lane, lane, status);
        const DD ordinary = dd_set_value(p, w, c, 1, n, lay, ws, lu_lane, lane, status);
        if (lane == 0) {
            // twisted - DoubleDouble(2) * ordinary (cdet_integrand_evaluator.h:233-263), then to double
            const DD result = dd_sub(twisted, dd_mul(DD{2.0, 0.0}, ordinary));
            p.values[c] = dadd(result.hi, result.lo);
            if (status) atomicOr(p.status + c, status);
        }
    }
}

// ---- lane form: minors by warps into lane-interleaved a, CDet by lanes ----
// For large batches: principal_minors_dd gives each (configuration, set) a
// warp, as the FP64 form does, and writes a = up * down into [group][set]
// [mask][lane] (the slot's lane of its order-sorted group of 32); cdet_dd_lane
// then gives each slot a lane, so the 32 lanes of a warp run the recursions of
// 32 configurations of (nearly) one order in step, every load a coalesced
// 512-byte row. The same operations as the warp form: the same values.
__device__ __forceinline__ DD* lane_a(const Scratch& w, int64_t slot, int set, int nmax) {
    const int64_t subsets = int64_t{1} << nmax;
    return reinterpret_cast<DD*>(w.dd_lanes) + ((slot >> 5) * 2 + set) * subsets * kWarp + (slot & 31);
}
__device__ __forceinline__ DD* lane_dp(const Scratch& w, int64_t slot, int set, int nmax, int64_t groups) {
    const int64_t subsets = int64_t{1} << nmax;
    return reinterpret_cast<DD*>(w.dd_lanes) + groups * 2 * subsets * kWarp +
           ((slot >> 5) * 2 + set) * (subsets / 2) * kWarp + (slot & 31);
}

__global__ void __launch_bounds__(kDDMaxWarps * 32) principal_minors_dd(const __grid_constant__ Problem p,
                                                          const __grid_constant__ Scratch w) {
    extern __shared__ double dd_smem[];
    const int lane = threadIdx.x & (kWarp - 1);
    const int warp_in_block = threadIdx.x / kWarp;
    const int warps_per_block = blockDim.x / kWarp;
    const int64_t global_warp = static_cast<int64_t>(blockIdx.x) * warps_per_block + warp_in_block;
    const int64_t total_warps = static_cast<int64_t>(gridDim.x) * warps_per_block;
    const int nmax = p.max_order;
    const WsLayout lay = compact_minors_layout(nmax, !(p.same_spin[0] && p.same_spin[1]), true);
    DD* ws = reinterpret_cast<DD*>(dd_smem) + static_cast<size_t>(warp_in_block) * lay.total;
    DD* lu_lane = reinterpret_cast<DD*>(w.lu_scratch + (static_cast<size_t>(global_warp) * kWarp + lane) * 2 *
                                                           nmax * nmax);
    const DD tol{p.dd_tol.hi, p.dd_tol.lo}, thresh{p.dd_fpm_shift.hi, p.dd_fpm_shift.lo};
    for (int64_t item = global_warp; item < p.batch * 2; item += total_warps) {
        const int64_t c = item >> 1;
        const int set = static_cast<int>(item & 1);
        const int n = __ldg(p.orders + c);
        if (n < 2 || n > nmax) continue;  // order 1 needs no minors
        const double* green = w.green + (c * 2 + set) * 2 * static_cast<int64_t>(nmax) * nmax;
        DD* A = ws + lay.a;
        bool fb = false;
        for (int k = lane; k < n * n; k += kWarp) A[k] = DD{green[k], 0.0};
        __syncwarp();
        DD* su = ws + lay.shifted_up;
        fb |= mat2pm_dd_warp(A, n, tol, thresh, lay, ws, su, lu_lane, lane);
        const bool one_spin = p.same_spin[set] != 0;
        if (!one_spin) {
            for (int k = lane; k < n * n; k += kWarp) A[k] = DD{green[static_cast<int64_t>(nmax) * nmax + k], 0.0};
            __syncwarp();
            fb |= mat2pm_dd_warp(A, n, tol, thresh, lay, ws, ws + lay.shifted_down, lu_lane, lane);
        }
        const DD* sd = one_spin ? su : ws + lay.shifted_down;
        DD* a = lane_a(w, __ldg(w.slot_of + c), set, nmax);
        for (uint32_t m = lane; m < (1u << n); m += kWarp)
            a[static_cast<int64_t>(m) * kWarp] = m == 0 ? DD{0.0, 0.0} : dd_mul(su[m], sd[m]);
        if (fb && lane == 0) atomicOr(p.status + c, kStatusFpmFallback);
        __syncwarp();
    }
}

// compute_dp_ztransform<DoubleDouble> for the slot's configuration on one
// lane, masks holding vertex 0 in popcount order, each one's submasks in the
// reference's descending order; then the prefactors and the combine.
__global__ void __launch_bounds__(32) cdet_dd_lane(const __grid_constant__ Problem p,
                                                   const __grid_constant__ Scratch w) {
    const int64_t slot = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (slot >= p.batch) return;
    const int64_t c = __ldg(w.config_at + slot);
    const int n = __ldg(p.orders + c);
    const int nmax = p.max_order;
    if (n < 1 || n > nmax) return;
    const int64_t groups = (p.batch + kWarp - 1) / kWarp;
    const DD zero{0.0, 0.0};
    const DD threshold{p.dd_threshold.hi, p.dd_threshold.lo};
    const bool filter = dd_gt(threshold, zero);
    int32_t status = 0;
    DD value[2];
    for (int set = 0; set < 2; ++set) {
        if (n == 1) {
            value[set] = dd_order1_value(p, w, c, set);
            continue;
        }
        const DD* a = lane_a(w, slot, set, nmax);
        DD* dp = lane_dp(w, slot, set, nmax, groups);
        dp[0] = a[1 * kWarp];
        const uint32_t rest_limit = 1u << (n - 1);
        for (int bits = 2; bits <= n; ++bits) {
            for (uint32_t rest = (1u << (bits - 1)) - 1u; rest < rest_limit; rest = next_same_popcount(rest)) {
                DD acc = a[static_cast<int64_t>((rest << 1) | 1u) * kWarp];
                DD rhs = dd_abs(acc);
                for (uint32_t sm = (rest - 1u) & rest;; sm = (sm - 1u) & rest) {
                    const DD term = dd_mul(dp[static_cast<int64_t>(sm) * kWarp],
                                           a[static_cast<int64_t>((rest ^ sm) << 1) * kWarp]);
                    acc = dd_sub(acc, term);
                    rhs = dd_add(rhs, dd_abs(term));
                    if (sm == 0) break;
                }
                if (filter && dd_lt(dd_abs(acc), dd_mul(threshold, rhs))) acc = zero;
                dp[static_cast<int64_t>(rest) * kWarp] = acc;
                if (bits == n) break;  // one mask at the top level
            }
        }
        const DD top = dp[static_cast<int64_t>(rest_limit - 1u) * kWarp];
        value[set] = dd_mul(DD{p.pref_dd[set][n].hi, p.pref_dd[set][n].lo}, top);
        if (!dd_finite(value[set])) status |= kStatusNonFinite;
    }
    const DD result = dd_sub(value[0], dd_mul(DD{2.0, 0.0}, value[1]));
    p.values[c] = dadd(result.hi, result.lo);
    if (status) atomicOr(p.status + c, status);
}

}  // namespace

// Smallest batch that runs the lane form (a warp of configurations per SM).
static int64_t dd_lane_min_batch(int sm_count) { return static_cast<int64_t>(sm_count > 0 ? sm_count : 152) * kWarp; }

DDShape dd_launch_shape(const Problem& p, bool lanes, size_t ws_warps, int sm_count) {
    const bool two_spins = !(p.same_spin[0] && p.same_spin[1]);
    const size_t ws_bytes = compact_minors_layout(p.max_order, two_spins, true).total * sizeof(DD);
    const size_t budget = 227 * 1024;
    const int64_t warps = std::max<int64_t>(1, static_cast<int64_t>(ws_warps) / 2);  // warps the LU regions are enough for
    DDShape d;
    d.wpb = static_cast<int>(std::max<int64_t>(
        1, std::min<int64_t>({kDDMaxWarps, static_cast<int64_t>(budget / ws_bytes), warps})));
    const int sms = sm_count > 0 ? sm_count : 152;
    const int per_sm = std::max(1, static_cast<int>(budget / (ws_bytes * d.wpb + 1024)));
    const int64_t items = p.batch * (lanes ? 2 : 1);
    d.blocks = std::min<int64_t>({static_cast<int64_t>(sms) * per_sm, (items + d.wpb - 1) / d.wpb, warps / d.wpb});
    d.smem = ws_bytes * d.wpb;
    return d;
}

cudaError_t launch_integrand_dd(const Problem& p, const Scratch& w, int sm_count, cudaStream_t stream) {
    if (p.batch <= 0) return cudaSuccess;
    // on the split assembly the reference's DoubleDouble steps are not the contract: 113-bit integer arithmetic
    if (p.fused_cdet) return launch_integrand_wide(p, w, sm_count, stream);
    const bool lanes = w.dd_lanes && (p.integrand_form == kIntegrandStaged ||
                                      (p.integrand_form == kIntegrandAuto && p.batch >= dd_lane_min_batch(sm_count)));
    const DDShape d = dd_launch_shape(p, lanes, w.ws_warps, sm_count);
    const auto kernel = lanes ? principal_minors_dd : integrand_dd;
    cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(d.smem));
    if (err != cudaSuccess) return err;
    kernel<<<static_cast<unsigned>(d.blocks), d.wpb * kWarp, d.smem, stream>>>(p, w);
    err = cudaGetLastError();
    if (err != cudaSuccess || !lanes) return err;
    // one warp per block, so that a small batch still spreads over every SM
    cdet_dd_lane<<<static_cast<unsigned>((p.batch + kWarp - 1) / kWarp), kWarp, 0, stream>>>(p, w);
    return cudaGetLastError();
}

}  // namespace cdet
