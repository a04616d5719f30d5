// b200s_sort_partitions: the leaf of the reference's large-array sort.
//
// The reference's partitioned sort (HybridSortPartitionedV3, cusort.hpp:2493-
// 2653) splits one large array into up to 1024 key-range partitions (CSR
// counters), then sorts every small partition in one launch of
// SortPartitionsAdaptive_outofplace (cusort.hpp:2309-2352, launched at
// cusort.hpp:2616-2628) and each larger one with a merge sort.  This entry
// point has that kernel's contract -- values, CSR counters, per-partition
// single-value flags, partition count, out of place -- and runs the ragged
// launch (b200s_sort_ragged) over the partitions, so a partitioned sort that
// calls it inherits the persistent bucketed kernels, including partitions up
// to b200s_ragged_max_length that the reference sends to its merge path.
//
// The ragged launch needs a plan (bucket counters, id lists, a captured
// graph).  Plans are cached per (device, element type, stable, stream) and
// grown to the largest partition count seen; b200s_release_partition_plans
// frees them.  Calls on one stream are ordered by the stream; calls on
// different streams use different plans.  A plan serves one call at a time: a
// call holds its entry until its whole sequence is enqueued, so that the
// launches of two host threads on one stream do not mix on one control block,
// and no other call grows or frees the plan meanwhile.
#include <cuda_runtime.h>

#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <tuple>

#include "b200sort.h"

namespace b200s {
b200s_status set_error(b200s_status s, const std::string& msg);
b200s_status cuda_error(cudaError_t e, const char* what);
int effective_stable(int dtype, uint32_t flags);
}  // namespace b200s

using namespace b200s;

namespace {

struct CachedPlan {
    std::mutex mutex;  // held from the lookup of the plan to the end of the call
    b200s_plan* plan = nullptr;
    int64_t capacity = 0;
    void reset() {
        if (plan) b200s_plan_destroy(plan);
        plan = nullptr;
        capacity = 0;
    }
    ~CachedPlan() { reset(); }  // released while a call was waiting for it: the last such call frees it
};
using PlanKey = std::tuple<int, int, int, void*>;  // device, dtype, stable, stream
using PlanCache = std::map<PlanKey, std::shared_ptr<CachedPlan>>;
std::mutex g_plan_mutex;  // the map only
PlanCache& plan_cache() {
    static PlanCache* cache = new PlanCache;  // never destroyed: the device may be gone at exit
    return *cache;
}

}  // namespace

extern "C" {

b200s_status b200s_sort_partitions(b200s_dtype dtype, uint32_t flags, const void* d_in, void* d_out,
                                   const int32_t* d_counters, const int32_t* d_uniform, int32_t nb_parts,
                                   void* stream) {
    (void)d_uniform;  // a single-valued partition sorts to itself: sorting it is the copy
    if (dtype < 0 || dtype > 3) return set_error(B200S_ERR_INVALID_ARGUMENT, "unknown dtype");
    if (flags & ~(B200S_STABLE | B200S_SORTED_CHECK))
        return set_error(B200S_ERR_INVALID_ARGUMENT, "unknown flag bits");
    if (nb_parts < 0) return set_error(B200S_ERR_INVALID_ARGUMENT, "negative partition count");
    if (nb_parts == 0) return B200S_OK;
    if (!d_in || !d_out || !d_counters) return set_error(B200S_ERR_INVALID_ARGUMENT, "null buffer");
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_error(e, "cudaGetDevice");
    const int stable = effective_stable(dtype, flags);
    std::shared_ptr<CachedPlan> c;
    {
        std::lock_guard<std::mutex> lock(g_plan_mutex);
        std::shared_ptr<CachedPlan>& entry = plan_cache()[PlanKey(dev, int(dtype), stable, stream)];
        if (!entry) entry = std::make_shared<CachedPlan>();
        c = entry;
    }
    std::lock_guard<std::mutex> lock(c->mutex);
    if (c->capacity < nb_parts) {
        c->reset();
        int64_t cap = 1024;  // the reference's partition count limit (MaxNbParts)
        while (cap < nb_parts) cap *= 2;
        const b200s_status st = b200s_plan_create(&c->plan, dtype, stable ? B200S_STABLE : 0u, cap, dev);
        if (st != B200S_OK) return st;
        c->capacity = cap;
    }
    return b200s_sort_ragged(c->plan, d_in, d_out, d_counters, nb_parts, stream);
}

b200s_status b200s_release_partition_plans(void) {
    PlanCache old;
    {
        std::lock_guard<std::mutex> lock(g_plan_mutex);
        old.swap(plan_cache());
    }
    for (auto& kv : old) {
        std::lock_guard<std::mutex> lock(kv.second->mutex);
        kv.second->reset();
    }
    return B200S_OK;
}

}  // extern "C"
