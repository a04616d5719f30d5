// The kernels' own windowed network (csrc/win.cuh, csrc/cta_xpose.cuh) on the
// host: one simulated thread per GPU thread, switched only at barriers, so that
// between two barriers the warps run one after another in a chosen order (each
// as far as it gets, lowest or highest first, or at random).  A barrier that is
// left out although another warp's elements are read, or that some warps skip,
// shows as a wrong order or as threads that never end.  Shared memory starts as
// garbage, buffers end in a guard, and the build checks the alignment of every
// access.  Prints one line per tile: "name logw ctas failures".
#include <ucontext.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <memory>
#include <random>
#include <vector>

#include "cuda_runtime.h"

#include "cta_xpose.cuh"

dim3 threadIdx, blockIdx, gridDim, blockDim;

// ---- simulated threads ----------------------------------------------------------
namespace sim {
constexpr size_t kStack = 64 << 10;
struct Barrier {
    int members = 0, waiting = 0;
    int all = 1, result = 1;
    unsigned generation = 0;
};
struct Thread {
    ucontext_t ctx;
    std::unique_ptr<char[]> stack{new char[kStack]};
    Barrier *warp, *cta, *at = nullptr;
    unsigned generation = 0;
    int rank = 0;
    bool done = false;
};
std::vector<std::unique_ptr<Thread>> threads;
std::vector<Barrier> barriers;
Barrier cluster;
ucontext_t scheduler;
size_t current;
std::function<void(int)> body;
std::vector<std::vector<unsigned char>> shared;  // per CTA

bool runnable(const Thread& t) { return !t.done && (!t.at || t.at->generation != t.generation); }
int wait(Barrier* b, int v) {
    Thread& t = *threads[current];
    b->all &= v != 0;
    if (++b->waiting == b->members) {
        b->result = b->all;
        b->all = 1;
        b->waiting = 0;
        ++b->generation;
        return b->result;
    }
    t.at = b;
    t.generation = b->generation;
    swapcontext(&t.ctx, &scheduler);
    t.at = nullptr;
    return b->result;
}
void entry(int i) {
    body(i);
    threads[size_t(i)]->done = true;
    swapcontext(&threads[size_t(i)]->ctx, &scheduler);
}
// ctas CTAs of `count` threads run f(cta, thread); false: they do not all end.
bool run(int ctas, int count, size_t smem, int order, unsigned seed, const std::function<void(int, int)>& f) {
    const size_t total = size_t(ctas) * size_t(count);
    std::mt19937 rng(seed);
    shared.assign(size_t(ctas), std::vector<unsigned char>(smem + 64, 0x85));
    barriers.assign(size_t(ctas) * size_t(1 + count / 32), Barrier{});
    cluster = Barrier{};
    cluster.members = int(total);
    body = [&](int i) { f(i / count, i % count); };
    while (threads.size() < total) threads.push_back(std::make_unique<Thread>());
    for (size_t i = 0; i < total; ++i) {
        Thread& t = *threads[i];
        const size_t base = (i / size_t(count)) * size_t(1 + count / 32);
        t.rank = int(i) / count;
        t.cta = &barriers[base];
        t.warp = &barriers[base + 1 + (i % size_t(count)) / 32];
        t.cta->members = count;
        t.warp->members = 32;
        t.done = false;
        t.at = nullptr;
        getcontext(&t.ctx);
        t.ctx.uc_stack.ss_sp = t.stack.get();
        t.ctx.uc_stack.ss_size = kStack;
        t.ctx.uc_link = nullptr;
        makecontext(&t.ctx, reinterpret_cast<void (*)()>(&entry), 1, int(i));
    }
    for (size_t left = total; left > 0;) {
        // a whole warp at a time, the first runnable one in the order
        const size_t warps = total / 32, start = order == 2 ? rng() % warps : 0;
        bool ran = false;
        for (size_t k = 0; k < warps && !ran; ++k) {
            const size_t w = order == 1 ? warps - 1 - k : (start + k) % warps;
            for (size_t l = 0; l < 32; ++l) {
                Thread& t = *threads[w * 32 + l];
                if (!runnable(t)) continue;
                ran = true;
                current = w * 32 + l;
                swapcontext(&scheduler, &t.ctx);
                if (t.done) --left;
            }
        }
        if (!ran) return false;
    }
    return true;
}
}  // namespace sim

void __syncwarp() { sim::wait(sim::threads[sim::current]->warp, 1); }
void __syncthreads() { sim::wait(sim::threads[sim::current]->cta, 1); }
int __syncthreads_and(int v) { return sim::wait(sim::threads[sim::current]->cta, v); }
void cooperative_groups::cluster_sync() { sim::wait(&sim::cluster, 1); }
void* cooperative_groups::cluster_map(void* p, int rank) {
    unsigned char* mine = sim::shared[size_t(sim::threads[sim::current]->rank)].data();
    return sim::shared[size_t(rank)].data() + (static_cast<unsigned char*>(p) - mine);
}

using namespace b200s;

// ---- element types: the kernels', with the exchanges in plain C++ --------------------
template <class R, class After>
void exchange(R& lo, R& hi, After after) {
    if (after(lo, hi)) std::swap(lo, hi);
}
struct HostU64 : ElemU64 {
    template <int Q>
    static void cexq(Reg& lo, Reg& hi) { exchange(lo, hi, after); }
};
struct HostRec : ElemRecI32L {};
struct HostStable : ElemRecI32G {
    template <int Q>
    static void cexq(Reg& lo, Reg& hi) { exchange(lo, hi, after); }
};
struct alignas(16) HostReg16 {
    uint64_t key;
    int32_t data, spare;
};
struct HostRec16 {
    using Mem = RecU64;
    using Reg = HostReg16;
    static constexpr bool kStable = false;
    static Reg pad() { return Reg{UINT64_MAX, INT32_MAX, 0}; }
    static Reg from_mem(const Mem& m, int) { return Reg{m.key, m.data, 0}; }
    static Mem to_mem(const Reg& r) { return Mem{r.key, r.data, 0}; }
    static bool after(const Reg& a, const Reg& b) { return b.key < a.key; }
    static void cex(Reg& lo, Reg& hi) { exchange(lo, hi, after); }
    static Reg pick(const Reg& own, const Reg& other, bool upper) {
        return (upper ? own.key < other.key : other.key < own.key) ? other : own;
    }
};

void set(int32_t& m, uint64_t key, int) { m = int32_t(uint32_t(key)); }
void set(uint64_t& m, uint64_t key, int) { m = key; }
void set(RecI32& m, uint64_t key, int i) { m = RecI32{int32_t(uint32_t(key)), i}; }
void set(RecU64& m, uint64_t key, int i) { m = RecU64{key, i, 0}; }
bool less(int32_t a, int32_t b) { return a < b; }
bool less(uint64_t a, uint64_t b) { return a < b; }
bool less(const RecI32& a, const RecI32& b) { return a.key < b.key; }
bool less(const RecU64& a, const RecU64& b) { return a.key < b.key; }

// The reference's order: the reflection network with the keep-own rule on the
// array padded to W, or a stable sort.
template <class E>
std::vector<typename E::Mem> expected(std::vector<typename E::Mem> v) {
    using M = typename E::Mem;
    if (E::kStable || keys_only<E>::value) {
        std::stable_sort(v.begin(), v.end(), [](const M& a, const M& b) { return less(a, b); });
        return v;
    }
    const int n = int(v.size());
    for (int st = 0; (1 << st) < n; ++st)
        for (int j = st; j >= 0; --j)
            for (int i = 0; i < n; ++i) {
                const int p = j == st ? i ^ ((2 << st) - 1) : i ^ (1 << j);
                if (i < p && p < n && less(v[size_t(p)], v[size_t(i)])) std::swap(v[size_t(i)], v[size_t(p)]);
            }
    return v;
}

// sort(in, out, n, order, seed) over lengths, distributions, offsets of the
// buffers and orders of the warps; the number of wrong results.
template <class E, class F>
int failures(int w, int shortest, const F& sort) {
    using M = typename E::Mem;
    int bad = 0;
    std::mt19937 rng(unsigned(w) + sizeof(M));
    int c = 0;
    for (int n : {w, w - 1, w / 2 + 1, w / 2, w - w / 4 + 5, 33, 1}) {
        if (n < shortest || n > w) continue;
        for (int kind = 0; kind < 3; ++kind, ++c) {  // few distinct keys, many, in order
            const size_t shift = sizeof(M) > 4 && sizeof(M) != sizeof(uint64_t) ? size_t(4 * (c % 4)) % sizeof(M)
                                 : std::is_same_v<M, RecI32> ? size_t(4 * (c % 2)) : 0;
            const bool in_place = c % 5 == 4;
            std::vector<M> data(static_cast<size_t>(n));
            for (int i = 0; i < n; ++i) {
                uint64_t key = kind == 0 ? (rng() % 5) * 0x3333333333333333ull : uint64_t(rng()) << 32 | rng();
                if (i % 7 == 3) key = std::is_same_v<M, int32_t> || std::is_same_v<M, RecI32> ? 0x7fffffffull : ~0ull;
                set(data[size_t(i)], key, i);
            }
            if (kind == 2) std::stable_sort(data.begin(), data.end(), [](const M& a, const M& b) { return less(a, b); });
            const size_t bytes = data.size() * sizeof(M);
            // 16-byte aligned stores, the arrays `shift` bytes into them
            std::vector<uint4> a(bytes / 16 + 4), b(bytes / 16 + 4);
            std::memset(a.data(), 0x5a, a.size() * 16);
            std::memset(b.data(), 0x5a, b.size() * 16);
            unsigned char* in = reinterpret_cast<unsigned char*>(a.data()) + 16 + shift;
            unsigned char* out = in_place ? in : reinterpret_cast<unsigned char*>(b.data()) + 16 + shift;
            std::memcpy(in, data.data(), bytes);
            const bool ended = sort(reinterpret_cast<M*>(in), reinterpret_cast<M*>(out), n, c % 3, unsigned(c));
            const std::vector<M> want = expected<E>(data);
            bool ok = ended && std::memcmp(out, want.data(), bytes) == 0;
            for (int g = 1; g <= 16; ++g) ok = ok && out[-g] == 0x5a && out[bytes + size_t(g) - 1] == 0x5a;
            bad += !ok;
        }
    }
    return bad;
}

template <class E, int LK, int LW, bool CHECK>
void packed(const char* name) {
    using S = Shape<LK, 5, LW>;
    using R = typename E::Reg;
    const int bad = failures<E>(S::W, 1, [](typename E::Mem* in, typename E::Mem* out, int n, int order, unsigned seed) {
        return sim::run(1, S::TPA, xc_smem_bytes<E, LK, S::LOGW>(), order, seed, [&](int, int t) {
            xc_sort_array<E, S, CHECK>(in, out, n, t, reinterpret_cast<R*>(sim::shared[0].data()));
        });
    });
    std::printf("%s%s %d 1 %d\n", name, CHECK ? "_check" : "", S::LOGW, bad);
}

// As k_sort_cluster_xc, one array by one cluster.
template <class E, int LK, int LT, int LC>
void cluster(const char* name) {
    using R = typename E::Reg;
    using Tile = Win<E, LK, LK + LT>;
    constexpr int W = 1 << (LK + LT);
    const int bad = failures<E>(W << LC, 1, [](typename E::Mem* in, typename E::Mem* out, int n, int order,
                                               unsigned seed) {
        return sim::run(1 << LC, 1 << LT, xc_smem_bytes<E, LK, LK + LT>(), order, seed, [&](int rank, int t) {
            R* sm = reinterpret_cast<R*>(sim::shared[size_t(rank)].data());
            R v[1 << LK];
            Tile::load(v, in, t, rank * W, n, sm);
            xc_cluster_network<E, LK, LT, LC>(v, t, rank, n - rank * W, sm);
            if constexpr (gathers<E>::value)
                Tile::store_gather(v, in, out, t, rank * W, n, sm, nullptr, [] { cooperative_groups::cluster_sync(); });
            else Tile::store(v, out, t, rank * W, n, sm);
        });
    });
    std::printf("%s %d %d %d\n", name, LK + LT, 1 << LC, bad);
}

// One program per PART (0 .. 7), built side by side.
int main() {
#if PART == 0
    packed<ElemI32, 5, 1, false>("i32");
    packed<ElemI32, 5, 2, true>("i32");
    packed<ElemI32, 4, 2, false>("i32_16");
#endif
#if PART == 1
    packed<HostRec, 4, 0, false>("rec");
    packed<HostRec, 4, 1, true>("rec");
    packed<HostRec, 4, 2, false>("rec");
    packed<HostRec, 4, 3, false>("rec");
#endif
#if PART == 2
    packed<HostRec, 5, 1, false>("rec_32");
    packed<HostRec, 5, 2, true>("rec_32");
#endif
#if PART == 3
    packed<HostStable, 4, 0, false>("stable");
    packed<HostStable, 4, 2, true>("stable");
    packed<HostU64, 4, 0, true>("u64");
    packed<HostU64, 4, 2, false>("u64");
#endif
#if PART == 4
    packed<HostRec16, 4, 0, false>("rec16");
    packed<HostRec16, 4, 1, true>("rec16");
    packed<HostRec16, 4, 2, false>("rec16");
    packed<HostRec16, 4, 3, false>("rec16");
#endif
#if PART == 5
    cluster<ElemI32, 5, 6, 1>("i32");
    cluster<ElemI32, 5, 6, 3>("i32");
#endif
#if PART == 6
    cluster<HostRec, 4, 6, 0>("rec");
    cluster<HostRec, 4, 6, 2>("rec");
    cluster<HostRec, 4, 8, 1>("rec");
#endif
#if PART == 7
    cluster<HostStable, 4, 6, 1>("stable");
    cluster<HostU64, 4, 6, 2>("u64");
    cluster<HostRec16, 4, 6, 3>("rec16");
    cluster<HostRec16, 4, 7, 1>("rec16");
#endif
    return 0;
}
