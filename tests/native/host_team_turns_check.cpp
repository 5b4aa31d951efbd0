// Long copies on a shared copy team (csrc/host_io.h), run by tests/test_host_team_turns.py: a short job
// that another thread posts while a long copy, touch or pack runs does not wait for all of it; and the
// pieces of several feeds, running at once, each run exactly once and in claimed order.
#include <cstdio>
#include <cstring>

#include "../../fherma-polynomial-cuda_b200/csrc/host_io.h"

using namespace negacyclic;

static int failures = 0;
#define EXPECT(cond)                                                          \
    do {                                                                      \
        if (!(cond)) {                                                        \
            std::fprintf(stderr, "%s:%d: %s\n", __FILE__, __LINE__, #cond);   \
            ++failures;                                                       \
        }                                                                     \
    } while (0)

static unsigned char load(const std::vector<unsigned char>& v, size_t at) {
    return *static_cast<const volatile unsigned char*>(&v[at]);
}

// Starts `work`, which zeroes `big` from its start on, on a thread; once it has begun, a short job of this
// thread is through before the work is.
template <class Work>
static void beside(HostTeam& team, std::vector<unsigned char>& big, const Work& work) {
    std::memset(big.data(), 0xff, big.size());
    std::thread caller(work);
    while (load(big, 0)) std::this_thread::yield();
    std::atomic<unsigned> ran{0};
    team.wait(team.post([&](unsigned, unsigned) { ran.fetch_add(1); }));
    EXPECT(load(big, big.size() - 1) == 0xff);
    EXPECT(ran.load() == team.workers());
    caller.join();
    for (size_t at = 0; at < big.size(); at += 4093) EXPECT(big[at] == 0);
    EXPECT(big.back() == 0);
}

static void pack(HostTeam& team, std::vector<unsigned char>& big) {
    constexpr size_t kPiece = 256 << 10;
    const uint32_t total = uint32_t(big.size() / kPiece);
    std::atomic<uint32_t> done{0};
    PieceFeed feed(team, total, 8, [&](uint32_t piece) {
        std::memset(&big[piece * kPiece], 0, kPiece);
        done.fetch_add(1, std::memory_order_release);
    });
    spin_until(done, total, team.spin_time(), [&] { feed.feed(); });
    team.wait(feed.last());
}

int main() {
    std::vector<unsigned char> big(size_t(1) << 30), zeros(big.size(), 0);
    {
        HostTeam team(2);
        beside(team, big, [&] { team.touch(big.data(), big.size()); });
        beside(team, big, [&] { team.copy(big.data(), zeros.data(), big.size()); });
        beside(team, big, [&] { pack(team, big); });
    }
    for (unsigned workers : {1u, 3u, 7u}) {
        HostTeam team(workers, std::chrono::microseconds(200));
        std::vector<std::thread> callers;
        for (uint32_t c = 0; c < 3; ++c)
            callers.emplace_back([&, c] {
                for (uint32_t total : {0u, 1u, 7u, 8u, 9u, 1000u + c}) {
                    std::vector<std::atomic<uint32_t>> runs(total);
                    std::atomic<uint32_t> done{0};
                    PieceFeed feed(team, total, 8, [&](uint32_t piece) {
                        runs[piece].fetch_add(1);
                        done.fetch_add(1, std::memory_order_release);
                    });
                    for (uint32_t part = 0; part <= total; part += 1 + total / 5)  // as chunks complete
                        spin_until(done, part, team.spin_time(), [&] { feed.feed(); });
                    spin_until(done, total, team.spin_time(), [&] { feed.feed(); });
                    team.wait(feed.last());
                    for (auto& r : runs) EXPECT(r.load() == 1);
                }
            });
        for (auto& t : callers) t.join();
    }
    std::printf("%d failures\n", failures);
    return failures != 0;
}
