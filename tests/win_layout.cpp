// Host walk of the windowed network's layout tables (csrc/win_layout.h): the
// network run through the windows and the shared-memory addresses against the
// reference network (keep-own ties), unique addresses, and bank conflicts.
// Prints one line per tile: "lk logw m ok worst/total/base".
#include <algorithm>
#include <cstdio>
#include <random>
#include <utility>
#include <vector>

#include "win_layout.h"

using namespace b200s;

struct El {
    int key, pos;
};

static void exchange(El& a, El& b) {
    if (b.key < a.key) std::swap(a, b);
}

template <int LK, int LOGW, int M>
void run(int distinct) {
    using P = WinPlan<LK, LOGW, M>;
    constexpr auto& T = P::kT;
    const int W = 1 << LOGW, K = 1 << LK, threads = 1 << P::LT;
    auto base = [&](const WinLayout& w, int t, bool mir) {
        int a = 0;
        for (int j = 0; j < P::LT; ++j)
            if ((((t >> j) & 1) ^ int(mir && w.thr[j] < w.st))) a += T.weight[w.thr[j]];
        return a;
    };
    auto address = [&](int i) {
        int a = 0;
        for (int b = 0; b < LOGW; ++b)
            if ((i >> b) & 1) a += T.weight[b];
        return a;
    };
    bool ok = true;
    std::vector<char> used(static_cast<size_t>(T.elems), 0);
    for (int i = 0; i < W; ++i) {
        const int a = address(i);
        ok = ok && a < T.elems && !used[size_t(a)];
        used[size_t(a)] = 1;
    }
    std::mt19937 rng(LOGW * 100 + LK);
    std::vector<El> ref(static_cast<size_t>(W));
    for (int i = 0; i < W; ++i) ref[size_t(i)] = El{int(rng() % unsigned(distinct)), i};
    std::vector<El> sm(static_cast<size_t>(T.elems)), v(static_cast<size_t>(W));
    for (int i = 0; i < W; ++i) sm[size_t(address(i))] = ref[size_t(i)];
    for (int st = 0; st < LOGW; ++st)
        for (int j = st; j >= 0; --j)
            for (int i = 0; i < W; ++i) {
                const int p = j == st ? i ^ ((2 << st) - 1) : i ^ (1 << j);
                if (i < p) exchange(ref[size_t(i)], ref[size_t(p)]);
            }
    auto at = [&](const WinLayout& w, int t, int q) { return size_t(base(w, t, P::mirrored(w, q)) + P::reg_off(w, q)); };
    auto put = [&](const WinLayout& w) {
        for (int t = 0; t < threads; ++t)
            for (int q = 0; q < K; ++q) sm[at(w, t, q)] = v[size_t(t * K + q)];
    };
    auto get = [&](const WinLayout& w) {
        for (int t = 0; t < threads; ++t)
            for (int q = 0; q < K; ++q) v[size_t(t * K + q)] = sm[at(w, t, q)];
    };
    // wavefronts of the worst access of a layout, in sweeps of 2^M lanes
    auto sweeps = [&](const WinLayout& w) {
        int worst = 1;
        for (int q = 0; q < K; ++q)
            for (int g = 0; g < 32 >> M; ++g) {
                std::vector<int> bank(size_t(1) << M, 0);
                for (int l = 0; l < 1 << M; ++l) {
                    const int lane = (g << M) + l, t = lane & ((1 << P::LG) - 1), slot = lane >> P::LG;
                    int a = int(at(w, t, q));
                    for (int b = 0; b < 5 - P::LG; ++b)
                        if ((slot >> b) & 1) a += T.slot[b];
                    worst = std::max(worst, ++bank[size_t(a & ((1 << M) - 1))]);
                }
            }
        return worst;
    };
    int total = 2 * sweeps(T.io) + 2 * sweeps(T.win[0]), accesses = 4;
    get(T.win[0]);
    for (int t = 0; t < threads; ++t)
        for (int st = 0; st < LK; ++st)
            for (int j = st; j >= 0; --j)
                for (int q = 0; q < K; ++q) {
                    const int p = j == st ? q ^ ((2 << st) - 1) : q ^ (1 << j);
                    if (q < p) exchange(v[size_t(t * K + q)], v[size_t(t * K + p)]);
                }
    for (int w = 1; w <= T.windows; ++w) {
        const WinLayout& L = T.win[w];
        put(T.win[w - 1]);
        get(L);
        total += 2 * sweeps(L);
        accesses += 2;
        for (int r = L.layers - 1; r >= 0; --r)
            for (int t = 0; t < threads; ++t)
                for (int q = 0; q < K; ++q)
                    if (!((q >> r) & 1))
                        exchange(v[size_t(t * K + q)], v[size_t(t * K + (r == L.refl ? q ^ (K - 1) : q | (1 << r)))]);
    }
    put(T.win[0]);
    for (int i = 0; i < W; ++i) {
        const El& e = sm[size_t(address(i))];
        ok = ok && e.key == ref[size_t(i)].key && e.pos == ref[size_t(i)].pos;
    }
    // a merge of two sorted halves by a plain (not reflected) top layer
    std::vector<El> half(static_cast<size_t>(W), El{0, 0});
    for (int i = 0; i < W; ++i) half[size_t(i)] = El{i < W / 2 ? i : W - i, i};
    std::vector<El> want = half;
    for (int j = LOGW - 1; j >= 0; --j)
        for (int i = 0; i < W; ++i)
            if (!((i >> j) & 1)) exchange(want[size_t(i)], want[size_t(i | (1 << j))]);
    for (int i = 0; i < W; ++i) sm[size_t(address(i))] = half[size_t(i)];
    for (int m = 0; m < T.merges; ++m) {
        const WinLayout& L = T.merge[m];
        get(L);
        for (int r = L.layers - 1; r >= 0; --r)
            for (int t = 0; t < threads; ++t)
                for (int q = 0; q < K; ++q)
                    if (!((q >> r) & 1)) exchange(v[size_t(t * K + q)], v[size_t(t * K + (q | (1 << r)))]);
        put(L);
    }
    for (int i = 0; i < W; ++i) {
        const El& e = sm[size_t(address(i))];
        ok = ok && e.key == want[size_t(i)].key && e.pos == want[size_t(i)].pos;
    }
    std::printf("%d %d %d %d %d %d\n", LK, LOGW, M, int(ok), total, accesses);
}

template <int LK, int M, int A, int B>
void range(int distinct) {
    run<LK, A, M>(distinct);
    if constexpr (A < B) range<LK, M, A + 1, B>(distinct);
}

int main() {
    for (int distinct : {3, 1 << 30}) {
        range<4, 4, 9, 14>(distinct);   // records, uint64 keys, stable records
        range<4, 3, 10, 14>(distinct);  // 16-byte records
        range<5, 5, 10, 14>(distinct);  // int32 keys
        range<4, 5, 9, 13>(distinct);   // int32 keys, 16 per thread
    }
    return 0;
}
