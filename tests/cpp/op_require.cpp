// Threads that ask for the same operators' tables (mw_internal.hpp, op_require): each (operator, depth) is built once, the
// root before any other depth.  Prints the number of tables built, and whether an order was violated.
#include <atomic>
#include <chrono>
#include <cstdio>
#include <thread>

#include "mw_internal.hpp"

namespace mwb {
void* dalloc(Ctx*, size_t bytes) { return ::operator new(bytes); }
void dfree(Ctx*, void* p) { ::operator delete(p); }
void upload_bytes(Ctx*, void*, const void*, size_t) {}
Op::~Op() {}
}  // namespace mwb

int main() {
    using namespace mwb;
    Ctx ctx;
    Mra m;
    m.ctx = &ctx;
    Op ops[3];
    Op* all[4] = {&ops[0], &ops[1], &ops[2], &ops[1]};  // one listed twice
    for (Op& o : ops) o.mra = &m;
    std::atomic<int> built{0}, bad{0};
    auto build = [&](const std::vector<Op*>& need, int depth) {
        for (Op* o : need) {
            if (depth > 0 && o->B0 != 1.0) ++bad;
            std::this_thread::sleep_for(std::chrono::milliseconds(2));
            if (depth == 0) o->B0 += 1.0;
            if (!o->depths.emplace(depth, std::make_unique<OpDepth>(&ctx)).second) ++bad;
            ++built;
        }
    };
    std::vector<std::thread> th;
    for (int t = 0; t < 8; ++t)
        th.emplace_back([&, t] {
            for (int depth = 0; depth < 4; ++depth) op_require(m, all + t % 2, 3, (depth + t) % 4, build);
        });
    for (std::thread& t : th) t.join();
    std::printf("%d %d\n", built.load(), bad.load());
    return 0;
}
