// A world's operator tables (mw_internal.hpp, world_operator_tables) when one of their allocations fails: prints, per
// failing allocation, whether the call failed, whether the world then counts as having tables, and after a second call
// whether all of them are there.
#include <cstdio>

#include "mw_internal.hpp"

static int left = -1;  // allocations until one fails (-1: never)

namespace mwb {
void* dalloc(Ctx*, size_t bytes) {
    if (left == 0) {
        left = -1;
        throw Error(-2, "out of memory");
    }
    if (left > 0) --left;
    return ::operator new(bytes);
}
void dfree(Ctx*, void* p) { ::operator delete(p); }
void upload_bytes(Ctx*, void* dst, const void* src, size_t bytes) { std::memcpy(dst, src, bytes); }
}  // namespace mwb

int main() {
    using namespace mwb;
    Ctx ctx;
    for (int at = 0; at < 4; ++at) {
        Mra m;
        m.ctx = &ctx;
        m.basis.init(0, 5);
        m.k = m.basis.k;
        m.F = two_scale_filter(m.basis);
        left = at;
        bool failed = false;
        try {
            world_operator_tables(m);
        } catch (const Error&) {
            failed = true;
        }
        left = -1;
        const bool has = m.builder != nullptr;
        world_operator_tables(m);
        std::printf("%d %d %d\n", (int)failed, (int)has, (int)(m.builder && m.d_cc && m.d_px && m.d_pw && m.d_pw[0] > 0.0));
        for (double* p : {m.d_cc, m.d_px, m.d_pw}) dfree(&ctx, p);
    }
    return 0;
}
