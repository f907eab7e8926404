// FP64 Green-matrix assembly for sm_103a: decode, lookup descriptor and the
// reference's Clenshaw recurrences (g_funcs.h:395-463, 609-763), bit for bit.
//
// A lookup is one 2-D Chebyshev sum: nu independent row sums over v, then one
// sum of the row values over u. One block of four warps takes up to 16 lookups
// (more where the rows are few) of one configuration, or of several whose lookups
// are fewer. Its row sums (lookups x rows) are dealt to lanes in runs of 32, so a
// single configuration already fills a block with independent chains and no lane
// idles on an invalid entry of a mixed-order batch; the row values go to shared
// memory, and one lane per lookup runs the outer sum over them.
//
// Row sums: each lane walks one row of nv coefficients downwards. The 32 rows
// of a warp are copied eight columns at a time with cp.async (two buffers per
// warp, the next chunk in flight while one is consumed), so the global reads
// are 64-byte pieces of rows; read straight from global memory each
// lane's 8-byte loads were 32 separate L1 wavefronts per step, about what the
// FP64 work of the step takes.
//
// Arithmetic: a step b_k = c_k + 2x b_{k+1} - b_{k+2} is a product and two
// additions, each rounded. The FP64 pipe would bound the kernel (two lane
// operations per clock and SM), so the product and every other step's first
// addition are formed on the integer pipes (cdet_softmul.cuh): 1.5 FP64
// operations per step. A chunk in which some lane's operands may not be the
// common case is repeated from its first step on the FP64 pipe. Chunks of
// eight columns and 96 registers let five blocks share an SM (a step is a long
// dependent chain: with chunks of 16 and four blocks the same arithmetic took
// 51.6 ms instead of 44.0).
//
// Measured against one thread per lookup (product on the FP64 pipe, 8-byte
// loads), whole calls: 8x8 / degree 128 / order 10, 4,096 configurations
// 106.5 -> 44.0 ms (three FP64 operations per coefficient at the pipe's 527
// G/s: 76 ms; one and a half: 38 ms); 6x6 / degree 96, 4,096 mixed orders 1..10
// 26.6 -> 4.1 ms (no lanes on entries past a configuration's order); 4x4 / 45 x
// 37 coefficients, two spins, order 7 x 391 1.47 -> 0.55 ms; one order-6
// configuration 2.08 -> 0.14 ms (all rows at once); 128 chains of envelope 9, a
// step with reused pairs 3.35 -> 0.54 ms (copies and evaluations in one launch).
#include "cdet_device.cuh"
#include "cdet_kernels.cuh"
#include "cdet_softmul.cuh"

#include <algorithm>
#include <type_traits>

namespace cdet {

namespace {

// sampled_coordinate_to_index (g_funcs.h:315-342) on value*extent; flags
// values the reference would reject (non-finite, outside the int range).
__device__ __forceinline__ int coordinate_index(double scaled, int extent, bool& bad) {
    if (!(scaled > -2147483648.0 && scaled < 2147483648.0)) {
        bad = true;
        return 0;
    }
    int index = static_cast<int>(floor(scaled));
    if (index < 0) index = 0;
    if (index >= extent) index = extent - 1;
    return index;
}

struct Vertex {
    double tau, tau_unit;
    int x, y, replica;
};

// Vertex decode of integrand_temp_typed (integrand_replica_randomly_sampled.h:422-432).
__device__ __forceinline__ Vertex decode_vertex(const double* __restrict__ v, const Scalars& s,
                                                int replica_count, bool& bad) {
    Vertex out;
    const double tu = __ldg(v + 0);
    if (!isfinite(tu)) bad = true;
    out.tau_unit = tu;
    out.tau = dmul(s.beta, tu);
    out.x = coordinate_index(dmul(static_cast<double>(s.n1), __ldg(v + 1)), s.n1, bad);
    out.y = coordinate_index(dmul(static_cast<double>(s.n2), __ldg(v + 2)), s.n2, bad);
    out.replica = replica_count <= 1
                      ? 0
                      : coordinate_index(dmul(static_cast<double>(replica_count), __ldg(v + 3)),
                                         replica_count, bad);
    return out;
}

__device__ __forceinline__ double clamp_unit(double value) {
    if (value < -1.0) return -1.0;
    if (value > 1.0) return 1.0;
    return value;
}

constexpr int kThreads = 128;
constexpr int kWarps = kThreads / kWarp;
constexpr int kMaxLookups = 128;  // lookups of one block, a thread each for the decode and the outer sum
constexpr int kMaxConfigs = kWarp;  // configurations of one block
constexpr int kRowBlock = 128;   // row values kept per lookup; more rows are taken block by block
constexpr int kChunk = 8;        // columns of a staged chunk
constexpr int kStride = 10;      // doubles between the rows of a staged chunk: 16-byte aligned, 16-byte reads free of bank conflicts

// One lookup of the block.
struct Lookup {
    const double* coeffs;  // its block of nu x nv coefficients
    double u, v;
    int8_t config;  // which of the block's configurations, and its order
    int8_t n;
    int8_t set, i, j;
    int8_t spin;    // the spin evaluated
    int8_t active;  // 0: nothing to evaluate (value already written, or a rejected vertex)
};

struct Shared {
    double stage[kWarps][2][kWarp * kStride];
    const double* row[kWarps][2][kWarp];  // the rows of the run being staged
};

// fill_pair_range (integrand_replica_randomly_sampled.h:467-473) for one
// evaluated entry: both spins when they share the evaluation.
__device__ __forceinline__ void store_entry(const Problem& p, const Scratch& w, int64_t c, int n, int set, int i, int j,
                                            int spin, bool both, double value) {
    const int nmax = p.max_order;
    const int64_t per_set = static_cast<int64_t>(nmax) * nmax;
    const int64_t mslot = (c * 2 + set) * 2;
    for (int sp = both ? 0 : spin; sp <= (both ? 1 : spin); ++sp) {
        double g = value;
        if (i == j) {
            g = dadd(g, sp == 0 ? p.s.diag_up_shift : p.s.diag_down_shift);
            // the double-double order-1 branch adds its own shifts to the unshifted value
            w.diag[(mslot + sp) * nmax + i] = p.raw_diag ? value : g;
        }
        w.green[(mslot + sp) * per_set + i * n + j] = dmul(g, p.s.scale);
    }
}

// What a lane needs of its lookup's x: the recurrence's 2x as a double and
// unpacked for the integer product.
struct Argument {
    double x, two_x;
    SoftFactor soft;
};
__device__ __forceinline__ Argument argument(double x) {
    Argument a;
    a.x = x;
    a.two_x = dmul(2.0, x);
    a.soft = soft_factor(static_cast<uint32_t>(__double2hiint(a.two_x)), static_cast<uint32_t>(__double2loint(a.two_x)));
    return a;
}
__device__ __forceinline__ bool soft_argument(const Argument& a) {
    return soft_factor_in_range(static_cast<uint32_t>(__double2hiint(a.two_x)));
}

// The recurrence's start c + 2x 0 - 0. With a finite x it is c itself unless c
// is a zero (whose sign 2x decides).
template <bool kSoft>
__device__ __forceinline__ double first_step(double c, const Argument& a) {
    if (kSoft && ((__double2hiint(c) << 1) | __double2loint(c)) != 0) return c;
    return dsub(dadd(c, dmul(a.two_x, 0.0)), 0.0);
}
// The product 2x b (kSoft: on the integer pipes, `bad` set where that may not be the FP64 pipe's).
template <bool kSoft>
__device__ __forceinline__ double times_two_x(const Argument& a, double b, bool& bad) {
    return kSoft ? soft_mul(a.soft, b, bad) : dmul(a.two_x, b);
}
// The row's end c_0 + x b_1 - b_2; the integer product is half of 2x b (its
// exponent one less: never subnormal where soft_mul reports nothing).
template <bool kSoft>
__device__ __forceinline__ double last_step(double c, const Argument& a, double b1, double b2, bool& bad) {
    double t;
    if (kSoft) {
        const double twice = soft_mul(a.soft, b1, bad);
        t = __hiloint2double(__double2hiint(twice) - 0x100000, __double2loint(twice));
    } else {
        t = dmul(b1, a.x);
    }
    return dsub(dadd(c, t), b2);
}

// The columns of a chunk whose first addition runs on the integer pipes too
// (soft_add): every other one, where the FP64 pipe and the integer pipes finish
// about together. 8x8 / degree 128 / order 10, 4,096 configurations: none of
// eight 55.5 ms, two 49.2, three 46.1, four 44.0, five 45.2, six 48.4.
constexpr uint32_t kSoftSums = 0x55;

// The Clenshaw steps of one full staged chunk (its columns in decreasing
// order). kFirst: its top column starts the recurrence; kLast: its lowest
// column ends it.
template <bool kSoft, bool kFirst, bool kLast>
__device__ __forceinline__ void chunk_steps(const double* st, const Argument& arg, double& b1, double& b2, bool& bad) {
#pragma unroll
    for (int q = kChunk / 2 - 1; q >= 0; --q) {
        const double2 pair = *reinterpret_cast<const double2*>(st + 2 * q);
#pragma unroll
        for (int h = 1; h >= 0; --h) {
            const double c = h ? pair.y : pair.x;
            if (kFirst && q == kChunk / 2 - 1 && h == 1) {
                b1 = first_step<kSoft>(c, arg);
                b2 = 0.0;
            } else if (kLast && q == 0 && h == 0) {
                b1 = last_step<kSoft>(c, arg, b1, b2, bad);
            } else {
                const double t = times_two_x<kSoft>(arg, b1, bad);
                const bool soft_sum = kSoft && ((kSoftSums >> (2 * q + h)) & 1) != 0;
                const double bk = dsub(soft_sum ? soft_add(c, t, bad) : dadd(c, t), b2);
                b2 = b1;
                b1 = bk;
            }
        }
    }
}

// The same for a chunk of `count` < kChunk columns (the top of a row).
template <bool kSoft>
__device__ __forceinline__ void partial_chunk_steps(const double* st, int count, bool last, const Argument& arg,
                                                    double& b1, double& b2, bool& bad) {
    b1 = first_step<kSoft>(st[count - 1], arg);
    b2 = 0.0;
    const int end = last ? 1 : 0;
    for (int k = count - 2; k >= end; --k) {
        const double bk = dsub(dadd(st[k], times_two_x<kSoft>(arg, b1, bad)), b2);
        b2 = b1;
        b1 = bk;
    }
    if (last) b1 = last_step<kSoft>(st[0], arg, b1, b2, bad);
}

template <bool kSoft>
__device__ __forceinline__ void row_chunk(const double* st, int count, bool first, bool last, const Argument& arg,
                                          double& b1, double& b2, bool& bad) {
    if (count < kChunk) partial_chunk_steps<kSoft>(st, count, last, arg, b1, b2, bad);
    else if (first && last) chunk_steps<kSoft, true, true>(st, arg, b1, b2, bad);
    else if (first) chunk_steps<kSoft, true, false>(st, arg, b1, b2, bad);
    else if (last) chunk_steps<kSoft, false, true>(st, arg, b1, b2, bad);
    else chunk_steps<kSoft, false, false>(st, arg, b1, b2, bad);
}

template <bool kVec16>
__device__ __forceinline__ void stage_chunk(double* st, const double* const* row, int column, int count, int lane) {
    const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(st));
    // lanes of one row: 16 bytes each where the rows are aligned to it, else 8
    constexpr int kLanes = kVec16 ? kChunk / 2 : kChunk;
    const int part = (lane & (kLanes - 1)) * (kVec16 ? 2 : 1);
    if (part < count) {
#pragma unroll
        for (int r0 = 0; r0 < kWarp; r0 += kWarp / kLanes) {
            const int r = r0 + lane / kLanes;
            const double* src = row[r] + column + part;
            if constexpr (kVec16)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst + (r * kStride + part) * 8), "l"(src));
            else
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + (r * kStride + part) * 8), "l"(src));
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// One block: lookups [first, first + count) of configuration blockIdx.x, first =
// blockIdx.y * lookups_per_block, or (per_block > 1, gridDim.y == 1) all lookups
// of per_block configurations. The lookups of a configuration of order n, set by
// set and spin by spin: its n^2 entries, or, with Green-pair reuse, the entries
// of pairs not both retained (rows i < k at columns k..n-1, then rows i >= k at
// every column), where the blocks with blockIdx.y == 0 also copy the retained
// ones.
template <bool kVec16>
__global__ void __launch_bounds__(kThreads, 5) green_assembly_fp64(const __grid_constant__ Problem p,
                                                                  const __grid_constant__ Scratch w,
                                                                  int lookups_per_block, int per_block, int row_block) {
    extern __shared__ __align__(16) unsigned char assembly_smem[];
    __shared__ int s_start[kMaxConfigs + 1];  // per_block > 1: first lookup of each configuration, and the total
    Shared& sm = *reinterpret_cast<Shared*>(assembly_smem);
    Lookup* lookups = reinterpret_cast<Lookup*>(assembly_smem + sizeof(Shared));
    double* values = reinterpret_cast<double*>(lookups + lookups_per_block);  // [lookup][row_block | 1]
    const int value_stride = row_block | 1;
    const Scalars& s = p.s;
    const int nmax = p.max_order;
    const int tid = threadIdx.x, lane = tid & (kWarp - 1), warp = tid / kWarp;
    const int64_t c0 = static_cast<int64_t>(blockIdx.x) * per_block;
    const int configs = static_cast<int>(min(static_cast<int64_t>(per_block), p.batch - c0));
    const int spins0 = p.same_spin[0] ? 1 : 2, spins1 = p.same_spin[1] ? 1 : 2;
    auto order_of = [&](int64_t c) { return p.all_subsets ? nmax : __ldg(p.orders + c); };
    auto kept_of = [&](int64_t c) { return p.reuse_mask ? __popcll(__ldg(p.reuse_mask + c)) : 0; };
    auto evaluated = [&](int n, int kept) { return n < 1 || n > nmax ? 0 : n * n - kept * kept; };  // of a set and spin

    if (blockIdx.y == 0 && tid < configs) {
        const int n = order_of(c0 + tid);
        if (n < 1 || n > nmax) atomicOr(p.status + c0 + tid, kStatusBadInput);
    }
    if (p.reuse_mask && blockIdx.y == 0) {
        const int per_config = 2 * nmax * nmax;
        for (int t = tid; t < configs * per_config; t += kThreads) {
            const int64_t c = c0 + t / per_config;
            const int e = t % per_config, n = order_of(c), kept = kept_of(c);
            const int set = e >= nmax * nmax ? 1 : 0;
            const int r = e - set * nmax * nmax, i = r / nmax, j = r - i * nmax;
            if (n < 1 || n > nmax || i >= kept || j >= kept) continue;
            const double* vbase = p.vertices + c * static_cast<int64_t>(nmax) * 4;
            bool bad = false;  // the decode's checks, so the status bits are a fresh evaluation's
            decode_vertex(vbase + 4 * i, s, set == 0 ? 2 : 1, bad);
            decode_vertex(vbase + 4 * j, s, set == 0 ? 2 : 1, bad);
            if (bad) atomicOr(p.status + c, kStatusBadInput);
            else copy_reused_pair(p, w.green, w.diag, c, set, i, j, n);
        }
    }

    const int first = blockIdx.y * lookups_per_block;
    int total, config = 0, e = first + tid;
    if (per_block == 1) {
        total = evaluated(order_of(c0), kept_of(c0)) * (spins0 + spins1);
    } else {
        if (warp == 0) {
            const int mine = lane < configs ? evaluated(order_of(c0 + lane), kept_of(c0 + lane)) * (spins0 + spins1) : 0;
            int end = mine;
            for (int off = 1; off < kWarp; off <<= 1) {
                const int below = __shfl_up_sync(0xffffffffu, end, off);
                if (lane >= off) end += below;
            }
            s_start[lane] = end - mine;
            if (lane == kWarp - 1) s_start[kMaxConfigs] = end;
        }
        __syncthreads();
        total = s_start[kMaxConfigs];
        for (int half = kMaxConfigs / 2; half > 0; half /= 2)  // the last configuration that starts at or before e
            if (s_start[config + half] <= e) config += half;
        e -= s_start[config];
    }
    if (first >= total) return;
    const int count = min(lookups_per_block, total - first);
    if (tid < count) {
        const int64_t c = c0 + config;
        const int n = order_of(c), kept = kept_of(c), per = evaluated(n, kept);
        const double* vbase = p.vertices + c * static_cast<int64_t>(nmax) * 4;
        const int set = e >= per * spins0 ? 1 : 0;
        e -= set * per * spins0;
        const int spin = e >= per ? 1 : 0;
        e -= spin * per;
        int i, j;
        if (e < kept * (n - kept)) {
            i = e / (n - kept);
            j = kept + (e - i * (n - kept));
        } else {
            const int q = e - kept * (n - kept);
            i = kept + q / n;
            j = q - (q / n) * n;
        }
        Lookup l;
        l.config = static_cast<int8_t>(config);
        l.n = static_cast<int8_t>(n);
        l.set = static_cast<int8_t>(set);
        l.spin = static_cast<int8_t>(spin);
        l.i = static_cast<int8_t>(i);
        l.j = static_cast<int8_t>(j);
        l.u = l.v = 1.0;  // a lookup with nothing to evaluate walks its rows harmlessly
        l.active = 0;
        bool bad = false;
        const int replica_count = set == 0 ? 2 : 1;
        const Vertex vi = decode_vertex(vbase + 4 * i, s, replica_count, bad);
        const Vertex vj = decode_vertex(vbase + 4 * j, s, replica_count, bad);
        // prepare_green_lookup_descriptor (g_funcs.h:609-653).
        const bool upper = (i != j) && (vi.tau_unit > vj.tau_unit);
        const uint64_t sitepair =
            ((((static_cast<uint64_t>(vi.replica) * 2u + static_cast<uint64_t>(vj.replica)) * s.n1 + vi.x) * s.n2 +
              vi.y) * s.n1 + vj.x) * s.n2 + vj.y;
        const TableDev& t = spin == 0 ? p.up[set] : p.down[set];
        l.coeffs = (upper ? t.upper : t.lower) + sitepair * static_cast<uint64_t>(s.nu) * static_cast<uint64_t>(s.nv);
        const double t_outer = upper ? vi.tau : vj.tau;  // the later time of the pair
        const double t_inner = upper ? vj.tau : vi.tau;
        if (bad) {
            atomicOr(p.status + c, kStatusBadInput);
        } else if (t_outer < s.branch_eps) {
            store_entry(p, w, c, n, set, i, j, spin, p.same_spin[set] != 0,
                        __ldg((upper ? t.upper_corners : t.lower_corners) + sitepair));
        } else {
            l.u = clamp_unit(dsub(ddiv(dmul(2.0, t_outer), s.beta), 1.0));
            l.v = clamp_unit(dsub(ddiv(dmul(2.0, t_inner), t_outer), 1.0));
            l.active = 1;
        }
        lookups[tid] = l;
    }
    __syncthreads();

    const int nu = s.nu, nv = s.nv;
    const int chunks = (nv + kChunk - 1) / kChunk;
    const int top_count = nv - (chunks - 1) * kChunk;  // columns of a row's first (highest) chunk
    // the outer sum of lookup tid, fed row values in decreasing order (the
    // recurrence of a row, over u)
    Argument outer_arg;
    double outer_b1 = 0.0, outer_b2 = 0.0;
    if (tid < count) outer_arg = argument(lookups[tid].u);

    for (int hi = nu; hi > 0; hi -= row_block) {
        const int rows = min(row_block, hi);
        const int base_row = hi - rows;
        const int tasks = count * rows;  // task = lookup * rows + (row - base_row)
        const int runs = (tasks + kWarp - 1) / kWarp;
        if (nv < 3) {
            for (int task = tid; task < tasks; task += kThreads) {
                const int l = task / rows, r = task - l * rows;
                values[l * value_stride + r] = clenshaw_row(
                    lookups[l].coeffs + static_cast<int64_t>(base_row + r) * nv, nv - 1, lookups[l].v);
            }
        } else {
            // this warp's runs warp, warp + 4, ...: a flat sequence of (run, chunk) with one chunk staged ahead
            const int my_runs = runs > warp ? (runs - warp + kWarps - 1) / kWarps : 0;
            auto point_rows = [&](int m) {  // the m-th run's rows; lanes past the end repeat the last task
                const int task = min((warp + m * kWarps) * kWarp + lane, tasks - 1);
                const int l = task / rows, r = task - l * rows;
                sm.row[warp][m & 1][lane] = lookups[l].coeffs + static_cast<int64_t>(base_row + r) * nv;
                __syncwarp();
            };
            auto stage = [&](int m, int j, int slot) {  // chunk j of run m: columns from the top
                const int column = (chunks - 1 - j) * kChunk;
                stage_chunk<kVec16>(sm.stage[warp][slot], sm.row[warp][m & 1], column, j == 0 ? top_count : kChunk,
                                    lane);
            };
            if (my_runs > 0) {
                point_rows(0);
                stage(0, 0, 0);
            }
            int slot = 0;
            for (int m = 0; m < my_runs; ++m) {
                const int task = (warp + m * kWarps) * kWarp + lane;
                const int task_c = min(task, tasks - 1);
                const int l = task_c / rows, r = task_c - l * rows;
                const Argument arg = argument(lookups[l].v);
                // integer products while every lane's factor allows them and no chunk of this run failed
                bool soft = __all_sync(0xffffffffu, soft_argument(arg));
                double b1 = 0.0, b2 = 0.0;
                for (int j = 0; j < chunks; ++j) {
                    // stage the next chunk, then wait for this one
                    if (j + 1 < chunks) {
                        stage(m, j + 1, slot ^ 1);
                    } else if (m + 1 < my_runs) {
                        point_rows(m + 1);
                        stage(m + 1, 0, slot ^ 1);
                    } else {
                        asm volatile("cp.async.commit_group;" ::: "memory");
                    }
                    asm volatile("cp.async.wait_group 1;" ::: "memory");
                    __syncwarp();
                    const double* st = sm.stage[warp][slot] + lane * kStride;
                    const int columns = j == 0 ? top_count : kChunk;
                    const double b1_in = b1, b2_in = b2;
                    bool redo = !soft;
                    if (soft) {
                        bool bad = false;
                        row_chunk<true>(st, columns, j == 0, j == chunks - 1, arg, b1, b2, bad);
                        redo = __any_sync(0xffffffffu, bad);
                    }
                    if (redo) {
                        soft = false;
                        bool unused = false;
                        b1 = b1_in;
                        b2 = b2_in;
                        row_chunk<false>(st, columns, j == 0, j == chunks - 1, arg, b1, b2, unused);
                    }
                    __syncwarp();  // the buffer is free for the chunk after next
                    slot ^= 1;
                }
                if (task < tasks) values[l * value_stride + r] = b1;
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
        }
        __syncthreads();
        if (tid < count) {
            const double* row_value = values + tid * value_stride;
            const bool first = hi == nu, last = base_row == 0;
            if (nu < 3) {  // degree 0 or 1: the sum's own short forms
                outer_b1 = nu == 1 ? row_value[0] : dadd(row_value[0], dmul(row_value[1], outer_arg.x));
            } else {
                const double b1_in = outer_b1, b2_in = outer_b2;
                auto sum = [&](auto use_soft) {
                    constexpr bool kSoft = decltype(use_soft)::value;
                    bool bad = false;
                    int r = rows - 1;
                    if (first) {
                        outer_b1 = first_step<kSoft>(row_value[r--], outer_arg);
                        outer_b2 = 0.0;
                    }
                    for (; r >= (last ? 1 : 0); --r) {
                        const double bk = dsub(dadd(row_value[r], times_two_x<kSoft>(outer_arg, outer_b1, bad)), outer_b2);
                        outer_b2 = outer_b1;
                        outer_b1 = bk;
                    }
                    if (last) outer_b1 = last_step<kSoft>(row_value[0], outer_arg, outer_b1, outer_b2, bad);
                    return bad;
                };
                if (!soft_argument(outer_arg) || sum(std::true_type())) {
                    outer_b1 = b1_in;
                    outer_b2 = b2_in;
                    sum(std::false_type());
                }
            }
        }
        __syncthreads();
    }
    if (tid < count && lookups[tid].active) {
        const Lookup& l = lookups[tid];
        store_entry(p, w, c0 + l.config, l.n, l.set, l.i, l.j, l.spin, p.same_spin[l.set] != 0, outer_b1);
    }
}

}  // namespace

cudaError_t launch_fp64_assembly(const Problem& p, const Scratch& w, int sm_count, cudaStream_t stream) {
    if (p.batch <= 0) return cudaSuccess;
    const int spins = (p.same_spin[0] ? 1 : 2) + (p.same_spin[1] ? 1 : 2);
    const int64_t per_config = static_cast<int64_t>(spins) * p.max_order * p.max_order;
    // lookups per block: 16 (or 512 row sums, four runs of each warp, where the rows are fewer than 32) once the
    // batch gives every SM its five blocks several times over, fewer for small batches, down to one lookup per
    // block, so that they spread over all SMs
    const int64_t blocks_wanted = 16 * static_cast<int64_t>(sm_count > 0 ? sm_count : 152);
    const int64_t most = std::max<int64_t>(16, std::min<int64_t>(kMaxLookups, 512 / p.s.nu));
    const int lookups =
        static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(most, p.batch * per_config / blocks_wanted)));
    // as many configurations as have at most that many (a block costs about 5 us whatever it has to do; Green
    // matrices alone, one thread per lookup / a block per configuration of 16 lookups / this rule: order 1 x
    // 65,536 at degree 12 444 / 707 / 180 us, at degree 32 2,500 / 1,234 / 609; order 8 x 4,096 at degree 4 226 /
    // 295 / 174; from order 3 on at degree 32 the rule changes nothing)
    const int per_block = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(kMaxConfigs, lookups / per_config)));
    const int row_block = std::min(p.s.nu, kRowBlock);
    const size_t smem = sizeof(Shared) + lookups * (sizeof(Lookup) + static_cast<size_t>(row_block | 1) * sizeof(double));
    // 16-byte copies need 16-byte aligned rows
    bool vec16 = p.s.nv % 2 == 0;
    for (int set = 0; set < 2; ++set)
        for (const TableDev* t : {&p.up[set], &p.down[set]})
            for (const double* c : {t->upper, t->lower})
                if (reinterpret_cast<uintptr_t>(c) % 16 != 0) vec16 = false;
    auto kernel = vec16 ? green_assembly_fp64<true> : green_assembly_fp64<false>;
    const cudaError_t err =
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (err != cudaSuccess) return err;
    const dim3 grid(static_cast<unsigned>((p.batch + per_block - 1) / per_block),
                    static_cast<unsigned>((per_config + lookups - 1) / lookups));
    kernel<<<grid, kThreads, smem, stream>>>(p, w, lookups, per_block, row_block);
    return cudaGetLastError();
}

}  // namespace cdet
