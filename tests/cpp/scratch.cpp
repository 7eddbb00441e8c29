// Ownership of device memory (mw_internal.hpp) with a counting allocator in place of the device pool: prints the
// arrays still held after each scope that ends with an exception or without one.
#include <cstdio>
#include <set>

#include "mw_internal.hpp"

static std::set<void*> live;
static int left = -1;  // allocations until one fails (-1: never)

namespace mwb {
void* dalloc(Ctx*, size_t bytes) {
    if (left == 0) throw Error(-2, "out of memory");
    if (left > 0) --left;
    void* p = ::operator new(bytes);
    live.insert(p);
    return p;
}
void dfree(Ctx*, void* p) {
    if (p && live.erase(p)) ::operator delete(p);
}
void upload_bytes(Ctx*, void* dst, const void* src, size_t bytes) { std::memcpy(dst, src, bytes); }
}  // namespace mwb

using namespace mwb;

template <typename F>
static void scope(const char* name, int fail_at, F&& f) {
    left = fail_at;
    bool thrown = false;
    try {
        f();
    } catch (const Error&) {
        thrown = true;
    }
    left = -1;
    std::printf("%s %d %zu\n", name, (int)thrown, live.size());
}

int main() {
    Ctx ctx;
    for (int at : {-1, 0, 2, 3})
        scope("scratch", at, [&] {
            Scratch s(&ctx);
            s.get<int>(5);
            s.get<double>(0);
            const double* d = s.up(std::vector<double>{1.0, 2.0});
            if (d[1] != 2.0) throw std::runtime_error("upload");
            if (at == 3) s.get<char>(1);
        });
    for (int at : {-1, 1})
        scope("tables", at, [&] {
            auto od = std::make_unique<OpDepth>(&ctx);
            od->d_mats = (double*)dalloc(&ctx, 8);
            od->d_terms = (TermRec*)dalloc(&ctx, 8);
        });
    scope("duplicate", -1, [&] {  // a table that finds its place taken goes away whole
        std::map<int, std::unique_ptr<OpDepth>> depths;
        for (int q = 0; q < 2; ++q) {
            auto od = std::make_unique<OpDepth>(&ctx);
            od->d_matsX = (unsigned char*)dalloc(&ctx, 8);
            depths.emplace(1, std::move(od));
        }
        if (live.size() != 1) throw std::runtime_error("duplicate kept");
    });
    scope("kept", -1, [&] {
        Scratch s(&ctx);
        s.get<int>(1);
        s.keep();
    });
    return 0;
}
