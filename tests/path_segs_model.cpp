// Launches of the whole-path kernel and of the wavefront on the host, from the functions that
// the kernel itself calls (path_segs.h): every block reads the counters when it starts, block 0
// marks the lanes, warps take their first paths by their place and the rest from the cursor.
// One line a case on standard output: whether all blocks agreed, and whether every path was taken once.
#include "path_segs.h"

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <random>
#include <set>
#include <vector>

using namespace lux;

namespace {

constexpr int kWarpsPerBlock = 4;

struct Model {
    std::vector<WaveCounters> ctr;
    int blocks;
    std::mt19937 rng;
    bool agree = true, cover = true;
    explicit Model(int lanes, int nblocks, unsigned seed) : ctr(size_t(lanes)), blocks(nblocks), rng(seed) {}

    void start_wave(int lane, int paths) {
        std::memset(&ctr[size_t(lane)], 0, sizeof(WaveCounters));
        ctr[size_t(lane)].count[0] = paths;
    }

    static bool same(const PathSegs& a, const PathSegs& b) {
        return std::equal(a.first, a.first + kMaxSegs + 1, b.first) && a.lane == b.lane;
    }

    // One launch; the paths it takes die one by one over the bounces that follow. Blocks start
    // in random order, so some find what others have already marked. `want`: the paths it should take.
    void launch(const Segs& G, int limit, int want) {
        std::vector<int> order(static_cast<size_t>(blocks));
        for (int b = 0; b < blocks; ++b) order[size_t(b)] = b;
        std::shuffle(order.begin(), order.end(), rng);
        std::vector<PathSegs> table(static_cast<size_t>(blocks));
        for (int b : order) {
            table[size_t(b)] = path_segments(ctr.data(), G);
            const int total = table[size_t(b)].first[kMaxSegs];
            if (b == 0 && total > 0 && total <= limit)
                for (int k = 0; k < G.n; ++k) mark_segment(ctr.data(), G, k);
        }
        for (int b = 1; b < blocks; ++b)
            agree = agree && same(table[0], table[size_t(b)]);
        const PathSegs& T = table[0];
        const int total = T.first[kMaxSegs];
        cover = cover && total == want;
        if (total == 0 || total > limit) return;
        // work assignment of paths.cu
        const int warps = blocks * kWarpsPerBlock;
        const int cap = std::min(32, (total + warps - 1) / warps);
        std::vector<int> seen(static_cast<size_t>(total), 0);
        auto take = [&](int base, int n) {
            for (int r = base; r < std::min(base + n, total); ++r) ++seen[size_t(r)];
            return base + n >= total;
        };
        std::vector<int> busy;
        for (int w = 0; w < warps; ++w)
            if (!take(w * cap, cap) && cap == 32) busy.push_back(w);
        int& cursor = ctr[size_t(T.lane)].fetch_p;
        while (!busy.empty()) {  // a warp with free lanes fetches for them
            const size_t i = rng() % busy.size();
            const int need = 1 + int(rng() % 32);
            const int base = cursor + warps * 32;
            cursor += need;
            if (take(base, need)) {
                busy[i] = busy.back();
                busy.pop_back();
            }
        }
        for (int s : seen) cover = cover && s == 1;
        // survivors entering each later bounce, as the kernel counts them
        for (int k = 0; k < G.n; ++k) {
            int left = T.first[k + 1] - T.first[k];
            for (int b = G.bounce[k] + 1; b < kMaxDepth && left > 0; ++b) {
                left -= left / 16;
                ctr[size_t(G.lane[k])].count[b] += left;
            }
        }
    }
};

Segs segs_of(std::initializer_list<std::pair<int, int>> s) {
    Segs G{};
    for (auto& p : s) {
        G.lane[G.n] = p.first;
        G.bounce[G.n] = p.second;
        ++G.n;
    }
    return G;
}

// The job engine's steps: wave A (lane 0) is finished at bounce 3 and stays in flight, wave B
// (lane 1) starts beside it, and the launch at {A at 9, B at 3} has to take all of B and none of A.
// Then a third wave, with both others still among the segments.
Model interleaved(int blocks, int a, int b, unsigned seed) {
    Model M(3, blocks, seed);
    const int limit = 2 * blocks * kWarpsPerBlock * 32;
    auto start_at_3 = [&](int lane, int paths) {
        M.start_wave(lane, paths);
        M.ctr[size_t(lane)].count[3] = paths;
    };
    start_at_3(0, a);
    M.launch(segs_of({{0, 3}}), limit, a);
    start_at_3(1, b);
    M.launch(segs_of({{0, 9}, {1, 3}}), limit, b);
    start_at_3(2, a);
    M.launch(segs_of({{0, 11}, {1, 9}, {2, 3}}), limit, a);
    for (const WaveCounters& c : M.ctr) M.cover = M.cover && c.finished != 0;
    return M;
}

}  // namespace

int main() {
    // paths against the grid's lanes: far fewer, a few more, and up to the limit of two a lane
    const int blocks = 12, lanes = blocks * kWarpsPerBlock * 32;
    for (int a : {300, lanes - 1, lanes + 40, 2 * lanes})
        for (int b : {300, lanes - 1, lanes + 40, 2 * lanes - 7})
            for (unsigned seed = 0; seed < 8; ++seed) {
                const Model M = interleaved(blocks, a, b, seed);
                std::printf("%d %d %u %s %s\n", a, b, seed, M.agree ? "agree" : "DISAGREE", M.cover ? "cover" : "LOST");
            }
    return 0;
}
