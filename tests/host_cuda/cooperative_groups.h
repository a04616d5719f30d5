// Thread-block clusters of the simulated threads (tests/win_network.cpp).
#pragma once
namespace cooperative_groups {
void cluster_sync();
void* cluster_map(void* p, int rank);
struct cluster_group {
    void sync() const { cluster_sync(); }
    unsigned block_rank() const { return 0; }  // the test passes the rank itself
    template <class T>
    T* map_shared_rank(T* p, int rank) const {
        return static_cast<T*>(cluster_map(p, rank));
    }
};
inline cluster_group this_cluster() { return {}; }
}  // namespace cooperative_groups
