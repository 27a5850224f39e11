// The row masks and counts of the small closure's cluster (csrc/cluster_rows.cuh,
// the code that the kernel runs) under random schedules: some CTAs of some warps
// each, every shared-memory access of the protocol a step of its own, any warp that
// is not waiting at a barrier may take the next step.  After each cluster barrier
// every warp counts rows and new bits for the decision to go on: all of them must
// find the same numbers, those of the rows published up to then.
//
// cluster_rows_main SCHEDULES [shared]: with "shared", a mistake is planted: rows
// are published into every CTA's masks of the current matrices too, as if these
// could be written from outside.  Prints the number of decisions and of those that
// were wrong.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#include "cluster_rows.cuh"

using cfpq::ClusterRows;

namespace {

constexpr uint32_t kCtas = 3, kWarps = 2, kNm = 2, kT = 2, kIters = 8;

struct Cta {
    std::vector<uint64_t> masks = std::vector<uint64_t>(4 * kNm * kT);
    std::vector<uint32_t> cnt = std::vector<uint32_t>(3 * ClusterRows::kMats);
    ClusterRows rows() { return {masks.data(), masks.data() + 3 * kNm * kT, cnt.data(), kNm, kT}; }
    uint32_t at_sync = 0, syncs = 0;
};

struct Decision {
    uint32_t rows[kNm], delta[kNm], fresh[kNm];
    bool operator!=(const Decision &o) const { return memcmp(this, &o, sizeof(*this)) != 0; }
};

// What a warp does next.
struct Warp {
    uint32_t it = 0, phase = 0, at = 0;
    uint32_t wait_sync = 0, wait_cluster = 0;
    Decision d;
};

struct Sim {
    std::mt19937 rng;
    bool shared;
    Cta cta[kCtas];
    Warp warp[kCtas][kWarps];
    uint32_t at_cluster = 0, barriers = 0;
    // what CTA c publishes at the end of iteration it for matrix m: rows of word w
    struct News { uint32_t w, lo, hi, bits; } news[kIters][kCtas][kNm];
    Decision truth[kIters];
    unsigned long long decisions = 0, wrong = 0;

    Sim(unsigned seed, bool s) : rng(seed), shared(s) {
        uint64_t cur[kNm][kT] = {};
        for (uint32_t it = 0; it < kIters; ++it) {
            uint64_t dl[kNm][kT] = {};
            memset(&truth[it], 0, sizeof(Decision));
            for (uint32_t c = 0; c < kCtas; ++c)
                for (uint32_t m = 0; m < kNm; ++m) {
                    const uint32_t any = rng() & 1u ? 0xffffffffu : 0u;
                    News &n = news[it][c][m];
                    n.w = c % kT;
                    n.lo = (uint32_t)(rng() & rng()) & any;
                    n.hi = (uint32_t)(rng() & rng()) & any;
                    n.bits = n.lo || n.hi ? 1 + (uint32_t)(rng() % 100) : 0;
                    dl[m][n.w] |= n.lo | ((uint64_t)n.hi << 32);
                    truth[it].fresh[m] += n.bits;
                }
            for (uint32_t m = 0; m < kNm; ++m)
                for (uint32_t w = 0; w < kT; ++w) {
                    cur[m][w] |= dl[m][w];
                    truth[it].rows[m] += __builtin_popcountll(cur[m][w]);
                    truth[it].delta[m] += __builtin_popcountll(dl[m][w]);
                }
        }
    }

    void publish(uint32_t c, uint32_t it, uint32_t m, uint32_t to) {
        const News &n = news[it][c][m];
        if (!n.bits) return;
        ClusterRows own = cta[c].rows();
        auto there = [&](uint32_t *p) -> uint32_t * {  // the same word of CTA `to`
            const size_t off = reinterpret_cast<char *>(p) - reinterpret_cast<char *>(cta[c].masks.data());
            if (off < cta[c].masks.size() * 8)
                return reinterpret_cast<uint32_t *>(reinterpret_cast<char *>(cta[to].masks.data()) + off);
            return cta[to].cnt.data() + (p - cta[c].cnt.data());
        };
        own.publish(ClusterRows::write_buffer(it), m, n.w, n.lo, n.hi, n.bits,
                    [&](uint32_t *p, uint32_t v) { *there(p) |= v; }, [&](uint32_t *p, uint32_t v) { *there(p) += v; });
        if (shared) cta[to].rows().current[m * kT + n.w] |= n.lo | ((uint64_t)n.hi << 32);
    }

    // One step of warp w of CTA c; false: it waits or is done.
    bool step(uint32_t c, uint32_t w) {
        Warp &x = warp[c][w];
        ClusterRows r = cta[c].rows();
        if (x.it == kIters) return false;
        switch (x.phase) {
        case 0:  // the thread x.at of this warp opens the iteration
            r.open(x.it, w + kWarps * x.at, 2 * kWarps);
            if (++x.at < 2) return true;
            break;
        case 1:  // block barrier: the CTA's new rows are complete
        case 3:  // (and the publishing warps are done)
            if (!x.at) {
                x.at = 1;
                x.wait_sync = cta[c].syncs;
                if (++cta[c].at_sync == kWarps) {
                    cta[c].at_sync = 0;
                    ++cta[c].syncs;
                }
                return true;
            }
            if (cta[c].syncs == x.wait_sync) return false;
            break;
        case 2:  // matrices w, w + kWarps, ..: one copy at a time
            if (w + x.at / kCtas * kWarps < kNm) {
                publish(c, x.it, w + x.at / kCtas * kWarps, x.at % kCtas);
                ++x.at;
                return true;
            }
            break;
        case 4:  // cluster barrier
            if (!x.at) {
                x.at = 1;
                x.wait_cluster = barriers;
                if (++at_cluster == kCtas * kWarps) {
                    at_cluster = 0;
                    ++barriers;
                }
                return true;
            }
            if (barriers == x.wait_cluster) return false;
            memset(&x.d, 0, sizeof(x.d));
            break;
        case 5: {  // the decision's reads, a word at a time
            const uint32_t buf = ClusterRows::write_buffer(x.it), m = x.at / (kT + 1), k = x.at % (kT + 1);
            if (m < kNm) {
                if (k == kT) {
                    x.d.fresh[m] = r.count[buf * ClusterRows::kMats + m];
                } else {
                    x.d.rows[m] += __builtin_popcountll(r.rows(buf, m, k));
                    x.d.delta[m] += __builtin_popcountll(r.delta_rows(buf, m)[k]);
                }
                ++x.at;
                return true;
            }
            ++decisions;
            wrong += x.d != truth[x.it];
            ++x.it;
            x.phase = x.at = 0;
            return true;
        }
        }
        ++x.phase;
        x.at = 0;
        return true;
    }

    bool run() {
        // one warp after the other in random turns; a bias makes some warps slow
        uint32_t slow = rng() % (kCtas * kWarps + 1);
        for (uint32_t idle = 0; idle < 100000;) {
            uint32_t i = rng() % (kCtas * kWarps);
            if (i == slow && rng() % 64) i = rng() % (kCtas * kWarps);
            idle = step(i / kWarps, i % kWarps) ? 0 : idle + 1;
            bool done = true;
            for (auto &c : warp)
                for (auto &w : c) done = done && w.it == kIters;
            if (done) return true;
        }
        return false;  // every warp waits
    }
};

}  // namespace

int main(int argc, char **argv) {
    const int n = argc > 1 ? atoi(argv[1]) : 1000;
    const bool shared = argc > 2 && !strcmp(argv[2], "shared");
    unsigned long long decisions = 0, wrong = 0;
    for (int s = 0; s < n; ++s) {
        Sim sim((unsigned)s, shared);
        if (!sim.run()) {
            printf("schedule %d: stuck\n", s);
            return 1;
        }
        decisions += sim.decisions;
        wrong += sim.wrong;
    }
    printf("%llu %llu\n", decisions, wrong);
    return 0;
}
