// The process's shared copy team (csrc/host_io.h): holders of one size and spin time get the same
// team, another size gets its own, the team ends with its last holder, and jobs that two threads
// post at once each run on every worker.
#include "../../fherma-polynomial-cuda_b200/csrc/host_io.h"

#include <cstdio>
#include <cstdlib>

using namespace negacyclic;

#define CHECK(x)                                                    \
    do {                                                            \
        if (!(x)) {                                                 \
            std::printf("line %d: %s\n", __LINE__, #x);             \
            return 1;                                               \
        }                                                           \
    } while (0)

int main() {
    const std::chrono::microseconds spin(200);
    std::weak_ptr<HostTeam> ended;
    {
        auto a = shared_host_team(3, spin), b = shared_host_team(3, spin), c = shared_host_team(2, spin);
        CHECK(a == b && a != c && a->workers() == 3 && c->workers() == 2);
        CHECK(shared_host_team(3, std::chrono::microseconds(300)) != a);
        ended = a;
        a.reset();
        CHECK(!ended.expired() && shared_host_team(3, spin) == b);

        constexpr int kThreads = 4, kCalls = 200;
        std::atomic<int> bad{0};
        std::vector<std::thread> callers;
        for (int t = 0; t < kThreads; ++t)
            callers.emplace_back([&] {
                auto team = shared_host_team(3, spin);
                for (int i = 0; i < kCalls; ++i) {
                    std::atomic<int> first{0}, second{0};
                    team->post([&](unsigned, unsigned) { first.fetch_add(1); });
                    team->wait(team->post([&](unsigned, unsigned) { second.fetch_add(1); }));
                    if (first.load() != 3 || second.load() != 3) bad.fetch_add(1);
                }
            });
        for (auto& t : callers) t.join();
        CHECK(bad.load() == 0);
    }
    CHECK(ended.expired());
    CHECK(shared_host_team(3, spin)->workers() == 3);
    std::printf("ok\n");
    return 0;
}
