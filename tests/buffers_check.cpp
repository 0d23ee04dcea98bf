// Drives replace_buffers (sprout_b200/csrc/buffers.hpp) with an allocator that fails at each of its
// calls in turn and prints "ok <name>" per passed check.
#include <cstdio>
#include <cstdlib>
#include <set>

#include "buffers.hpp"

using spb::render::buffer;
using spb::render::replace_buffers;

static int failures = 0;
#define CHECK(name, cond)                                      \
    do {                                                       \
        if (cond) {                                            \
            std::printf("ok %s\n", name);                      \
        } else {                                               \
            std::printf("FAILED %s (line %d)\n", name, __LINE__); \
            ++failures;                                        \
        }                                                      \
    } while (0)

struct Heap {
    std::set<void*> live;
    int             calls = 0;
    int             fail  = -1;  // the call that fails
    int             bad   = 0;   // releases of what is not allocated

    int replace(std::vector<spb::render::Buffer> const& set) {
        return replace_buffers(
            set,
            [&](void** p, size_t bytes) {
                if (calls++ == fail) {
                    *p = &calls;  // an allocator may leave anything behind
                    return 2;
                }
                *p = std::malloc(bytes);
                live.insert(*p);
                return 0;
            },
            [&](void* p) {
                if (p) {
                    bad += live.erase(p) == 0;
                    std::free(p);
                }
            });
    }
};

int main() {
    bool all_null = true, none_left = true, told = true, again = true;
    for (int fail = 0; fail < 3; ++fail) {
        Heap     h;
        float*   a = nullptr;
        int*     b = nullptr;
        double*  c = nullptr;
        char*    unused = nullptr;
        auto const set = [&](size_t n) {
            return std::vector<spb::render::Buffer>{buffer(a, n), buffer(unused, 0), buffer(b, 2 * n), buffer(c, n)};
        };
        again     = again && h.replace(set(8)) == 0 && h.live.size() == 3 && a && b && c && !unused;
        h.calls   = 0;
        h.fail    = fail;
        told      = told && h.replace(set(1000)) == 2;
        all_null  = all_null && !a && !b && !c;
        none_left = none_left && h.live.empty();
        h.fail    = -1;
        again     = again && h.replace(set(8)) == 0 && h.live.size() == 3 && a && b && c && h.bad == 0;
        h.replace(set(0));
        none_left = none_left && h.live.empty() && !a;
    }
    CHECK("failure_is_told", told);
    CHECK("failure_leaves_no_pointer", all_null);
    CHECK("failure_releases_everything", none_left);
    CHECK("a_later_request_succeeds", again);
    return failures ? EXIT_FAILURE : EXIT_SUCCESS;
}
