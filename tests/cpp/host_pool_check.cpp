// A pool whose threads cannot all be started runs every task once all the same, and a pool can grow, stop
// and start again.
#include <sys/resource.h>

#include <atomic>
#include <cstdio>
#include <vector>

#include "csp_pool.h"

static bool runs(csp::HostPool& pool, size_t tasks) {
    std::vector<std::atomic<int>> done(tasks);
    pool.run(tasks, [&](size_t k) { ++done[k]; });
    for (auto& d : done)
        if (d != 1) return false;
    return true;
}

int main() {
    csp::HostPool pool;
    bool ok = runs(pool, 100);
    pool.start(2);
    ok = ok && runs(pool, 1000);
    pool.start(4);
    ok = ok && runs(pool, 1000);
    pool.stop();
    ok = ok && runs(pool, 10);
    // room for a few thread stacks only
    rlimit lim{};
    getrlimit(RLIMIT_AS, &lim);
    lim.rlim_cur = 192u << 20;
    if (setrlimit(RLIMIT_AS, &lim) != 0) return 2;
    pool.start(64);
    ok = ok && runs(pool, 1000);
    std::puts(ok ? "OK" : "FAIL");
    return ok ? 0 : 1;
}
