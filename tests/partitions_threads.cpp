// b200s_sort_partitions (csrc/partitions.cu) over a fake of the plan functions:
// several host threads on one stream, with growing partition counts and a
// thread that releases the cached plans.  Prints the calls, the calls that
// overlapped on one plan, and the uses of a plan after its end.
#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <string>
#include <thread>
#include <vector>

#include "b200sort.h"
#include <cuda_runtime.h>

struct b200s_plan {  // never freed, so that a use after its end can be counted
    std::atomic<int> users{0};
    std::atomic<bool> alive{true};
    int64_t capacity = 0;
};
static std::atomic<int> g_calls{0}, g_overlaps{0}, g_dead{0}, g_small{0};

namespace b200s {
b200s_status set_error(b200s_status s, const std::string&) { return s; }
b200s_status cuda_error(cudaError_t, const char*) { return B200S_ERR_CUDA; }
int effective_stable(int, uint32_t flags) { return int(flags & B200S_STABLE); }
}  // namespace b200s

extern "C" {
cudaError_t cudaGetDevice(int* dev) {
    *dev = 0;
    return cudaSuccess;
}
b200s_status b200s_plan_create(b200s_plan** out, b200s_dtype, uint32_t, int64_t max_arrays, int32_t) {
    *out = new b200s_plan;
    (*out)->capacity = max_arrays;
    return B200S_OK;
}
b200s_status b200s_plan_destroy(b200s_plan* p) {
    if (p->users.load() != 0 || !p->alive.exchange(false)) ++g_dead;
    return B200S_OK;
}
b200s_status b200s_sort_ragged(b200s_plan* p, const void*, void*, const int32_t*, int64_t arrays, void*) {
    ++g_calls;
    if (!p) {
        ++g_dead;
        return B200S_ERR_INVALID_ARGUMENT;
    }
    if (p->users.fetch_add(1) != 0) ++g_overlaps;
    if (p->capacity < arrays) ++g_small;
    std::this_thread::sleep_for(std::chrono::microseconds(20));
    if (!p->alive.load()) ++g_dead;
    --p->users;
    return B200S_OK;
}
}

int main() {
    std::vector<std::thread> threads;
    for (int t = 0; t < 4; ++t)
        threads.emplace_back([t] {
            for (int i = 0; i < 200; ++i) {
                int32_t off = 0;
                const int parts = i < 100 ? 10 + i : 1000 * (1 + (i + t) % 9);
                if (b200s_sort_partitions(B200S_I32, 0, &off, &off, &off, nullptr, parts, nullptr) != B200S_OK) std::abort();
            }
        });
    threads.emplace_back([] {
        for (int i = 0; i < 20; ++i) {
            std::this_thread::sleep_for(std::chrono::microseconds(300));
            b200s_release_partition_plans();
        }
    });
    for (auto& t : threads) t.join();
    std::printf("%d %d %d %d\n", g_calls.load(), g_overlaps.load(), g_dead.load(), g_small.load());
    return 0;
}
