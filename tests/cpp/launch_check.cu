// Host check of the launch shapes that index the LU-fallback scratch
// (minors_launch_shape, queue_launch_shape, dd_launch_shape): for every order,
// batches from one to 200,000, one and two spins, and scratches of 8 (the
// fewest) to a few thousand warps' regions, no launch has more warps (workspaces)
// than the scratch has regions. Links the library; calls no CUDA function.
// Prints each violation and exits non-zero if there is one.
#include "cdet_kernels.cuh"

#include <cstdio>

using namespace cdet;

static long failures = 0;

static void check(const char* what, bool ok, const Problem& p, size_t ws_warps, long long used) {
    if (ok) return;
    if (++failures <= 20)
        std::printf("%s: order %d batch %lld spins %d scratch %zu: %lld\n", what, p.max_order,
                    static_cast<long long>(p.batch), p.same_spin[0] ? 1 : 2, ws_warps, used);
}

int main() {
    const int64_t batches[] = {1, 2, 3, 151, 152, 305, 608, 911, 912, 1000, 3000, 11349, 11355, 57798, 200000};
    const size_t scratch[] = {8, 9, 10, 11, 12, 13, 15, 16, 17, 23, 24, 100, 608, 1824, 4864};
    long shapes = 0;
    for (int order = 1; order <= kMaxOrder; ++order)
        for (int spins = 1; spins <= 2; ++spins)
            for (int64_t batch : batches)
                for (size_t ws : scratch)
                    for (int sms : {1, 76, 152}) {
                        Problem p{};
                        p.max_order = order;
                        p.batch = batch;
                        p.same_spin[0] = p.same_spin[1] = spins == 1;
                        const MinorsShape m = minors_launch_shape(p, ws, sms);
                        ++shapes;
                        check("minors", m.blocks >= 1 && m.per_block >= 1 &&
                              m.blocks * m.per_block <= static_cast<int64_t>(ws), p, ws, m.blocks * m.per_block);
                        check("minors block", m.per_block * m.warps * 32 <= (m.use_smem ? 1024 : m.chunked ? 512 : 256) &&
                              m.smem <= 227 * 1024, p, ws, m.per_block * m.warps);
                        if (order > 10) continue;
                        for (int pair = 0; pair < 2; ++pair)
                            for (int per_sm : {0, 1, 5, 24}) {
                                p.queue.pair = pair;
                                p.queue.warps_per_sm = per_sm;
                                Scratch w{};
                                w.ws_warps = ws;
                                int wpb = 0, blocks = 0;
                                size_t smem = 0;
                                queue_launch_shape(p, w, sms, &wpb, &blocks, &smem);
                                ++shapes;
                                check("queue", blocks >= 1 && wpb >= 1 + pair && wpb % (1 + pair) == 0 &&
                                      static_cast<int64_t>(blocks) * wpb <= static_cast<int64_t>(ws), p, ws,
                                      static_cast<long long>(blocks) * wpb);
                            }
                        for (int lanes = 0; lanes < 2; ++lanes) {
                            const DDShape d = dd_launch_shape(p, lanes != 0, ws, sms);
                            ++shapes;
                            check("double-double", d.blocks >= 1 && d.wpb >= 1 && d.wpb <= kDDMaxWarps &&
                                  2 * d.blocks * d.wpb <= static_cast<int64_t>(ws), p, ws, 2 * d.blocks * d.wpb);
                        }
                    }
    std::printf("%ld launch shapes checked, %ld violations\n", shapes, failures);
    return failures == 0 ? 0 : 1;
}
