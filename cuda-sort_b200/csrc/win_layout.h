// Layout algebra of the windowed network (win.cuh): which index bits a
// thread's registers hold in each window, in which order the layers run, and
// where an element lives in shared memory.  Plain constexpr C++ with no CUDA,
// so that a CPU test can walk the same tables.
//
// The reflection network on 2^LOGW elements is a sequence of layers: stage ST
// pairs i with i ^ (2^(ST+1) - 1), then with i ^ 2^j for j = ST-1 .. 0.  A
// tile holds 2^LK elements per thread, so a layer whose index bit is one of
// the LK bits that number a thread's registers is a compare-exchange between
// two registers.  Stages 0 .. LK-1 run with the registers on bits 0 .. LK-1
// (window 0, the natural layout).  The layers of the later stages are cut into
// consecutive runs of LK, ACROSS stage boundaries: the layers of one run use LK
// different bits (a bit comes back only ST+2 >= LK+2 layers later), so each
// run is one window whose registers are numbered by just those bits, and a
// window costs one trip through shared memory.  Against one window group per
// stage, ceil((ST+1)/LK) trips each, this takes 8 trips instead of 10 for
// 1024 elements and 13 instead of 16 for 4096 (32 per thread).  The last run
// may be short; it ends in bits f-1 .. 0, so the last window is always the
// natural layout again.
//
// Register bit LK-1 is the first layer's bit, LK-2 the second's, and so on.
// A window that holds the reflection of stage ST (at register bit refl) reads
// and writes the registers with that bit set at the address whose thread-held
// bits below ST are complemented: the reflection partner of register q is then
// register q ^ (2^LK - 1) of the same thread, and every merge keeps its minimum
// at the lower index.
//
// Shared memory.  Element i lives at the sum of weight[b] over its set bits b.
// The first M lane bits of an access (2^M elements of 16, 8 or 4 bytes fill the
// banks: M = 3, 4, 5) hit distinct banks when their weights have the distinct
// 2-adic valuations 0 .. M-1 (their "classes"; M: a multiple of 2^M).  The
// classes below come from a search over all windows of a tile (and the
// natural and the coalesced layout); tests/test_win_layout.py counts the
// conflicts that are left, and tests/test_win_network.py runs the network of
// win.cuh on these tables.  One bit of each class takes the weights 1, 2, 4,
// ..; the others follow in the order of their class, each the smallest value
// of its class above the sum of all before it, which keeps every address
// unique and the region within a few percent of 2^LOGW.
#pragma once

namespace b200s {

constexpr int kWinMaxBits = 16;     // index bits of one tile
constexpr int kWinMaxWindows = 32;  // windows of one tile, the natural one included

struct WinClasses {
    int cls[kWinMaxBits];   // class of each index bit
};

// Classes of the index bits for 2^LOGW-element tiles of 2^lk elements per
// thread and accesses of 2^m elements per bank sweep.
constexpr WinClasses win_classes(int lk, int logw, int m) {
    // 8-byte elements
    if (m == 4 && lk == 4) {
        switch (logw) {
            case 9: return {{1, 3, 2, 0, 1, 3, 1, 2, 0}};
            case 10: return {{0, 3, 2, 1, 0, 3, 0, 2, 1, 4}};
            case 11: return {{0, 3, 2, 1, 0, 3, 0, 2, 1, 3, 1}};
            case 12: return {{1, 0, 2, 1, 3, 0, 1, 2, 3, 1, 0, 4}};
            case 13: return {{0, 1, 2, 3, 0, 1, 0, 2, 3, 4, 1, 3, 1}};
            case 14: return {{0, 1, 2, 3, 0, 1, 0, 2, 3, 3, 1, 2, 2, 0}};
        }
    }
    if (m == 4 && lk == 5) {
        switch (logw) {
            case 11: return {{0, 3, 1, 3, 2, 3, 3, 2, 1, 0, 1}};
            case 12: return {{0, 2, 1, 0, 3, 1, 1, 0, 2, 3, 3, 4}};
            case 13: return {{2, 3, 0, 1, 2, 0, 3, 2, 1, 0, 0, 4, 2}};
        }
    }
    // 16-byte elements
    if (m == 3 && lk == 4) {
        switch (logw) {
            case 9: return {{0, 1, 2, 0, 1, 1, 0, 0, 2}};
            case 10: return {{0, 1, 2, 2, 0, 1, 0, 0, 2, 3}};
            case 11: return {{1, 0, 2, 1, 0, 3, 0, 2, 1, 3, 2}};
            case 12: return {{0, 0, 2, 0, 1, 1, 0, 2, 1, 0, 0, 0}};
            case 13: return {{1, 1, 2, 0, 1, 1, 2, 0, 2, 3, 0, 0, 0}};
            case 14: return {{1, 1, 2, 1, 0, 1, 0, 2, 0, 0, 1, 0, 1, 1}};
        }
    }
    // 4-byte elements
    if (m == 5 && lk == 4) {
        switch (logw) {
            case 9: return {{3, 1, 4, 2, 3, 1, 4, 2, 0}};
            case 10: return {{0, 1, 2, 4, 0, 1, 2, 3, 4, 1}};
            case 11: return {{4, 3, 1, 2, 4, 3, 2, 1, 0, 0, 4}};
            case 12: return {{3, 1, 2, 0, 3, 1, 0, 2, 4, 0, 3, 1}};
            case 13: return {{3, 1, 2, 0, 3, 1, 0, 2, 4, 4, 5, 2, 0}};
        }
    }
    if (m == 5 && lk == 5) {
        switch (logw) {
            case 10: return {{1, 4, 3, 0, 2, 1, 3, 0, 2, 4}};
            case 11: return {{2, 3, 1, 4, 0, 2, 3, 0, 1, 4, 4}};
            case 12: return {{1, 2, 0, 3, 4, 1, 2, 3, 0, 4, 3, 2}};
            case 13: return {{0, 1, 4, 3, 2, 0, 1, 3, 2, 4, 5, 2, 0}};
            case 14: return {{0, 3, 1, 4, 2, 0, 3, 2, 1, 4, 2, 4, 5, 5}};
        }
    }
    // no searched classes: the bits cycle through them
    WinClasses c{};
    for (int b = 0; b < kWinMaxBits; ++b) c.cls[b] = b % (m < lk ? m : lk);
    return c;
}

struct WinLayout {
    int reg[6];               // index bit of each register bit
    int thr[kWinMaxBits];     // index bit of each thread bit
    int refl;                 // register bit at which the reflection runs, -1: none
    int st;                   // its stage
    int layers;               // layers run here: register bits layers-1 .. 0
};

template <int LK, int LOGW, int M>
struct WinPlan {
    static constexpr int LT = LOGW - LK, LG = 5, LW = LT - LG;
    static_assert(LOGW <= kWinMaxBits && LK >= 2 && LK <= 6 && LT >= 5, "tile shape: whole warps");
    struct Tables {
        WinLayout win[kWinMaxWindows];  // [0]: natural
        WinLayout merge[6];             // windows of the merges on bits LOGW-1 .. 0 (after a cluster layer)
        int merges;
        WinLayout io;                   // coalesced global accesses: lanes on the lowest index bits
        int windows;                    // windows after the natural one
        int weight[kWinMaxBits];        // shared-memory weight of each index bit
        static constexpr int slot[5] = {};  // of the bits that number a warp's arrays: none, a tile is whole warps
        int elems;                      // shared-memory elements of the tile
    };

    // Thread bits of a layout: the index bits left over, the lowest LG of them
    // on the lanes (those of distinct classes first, so that the lanes of one
    // bank sweep differ in them), the higher ones on the warps: a warp keeps
    // its part of the tile while no register bit is one of the top LW bits.
    static constexpr void fill_threads(WinLayout& w, const WinClasses& c) {
        int left[kWinMaxBits] = {}, n = 0;
        for (int b = 0; b < LOGW; ++b) {
            bool used = false;
            for (int r = 0; r < LK; ++r) used = used || w.reg[r] == b;
            if (!used) left[n++] = b;
        }
        bool taken[kWinMaxBits] = {};
        int at = 0;
        for (int k = 0; k < M && k < LG; ++k)
            for (int j = 0; j < LG; ++j)
                if (!taken[j] && c.cls[left[j]] == k) {
                    taken[j] = true;
                    w.thr[at++] = left[j];
                    break;
                }
        for (int j = 0; j < LG; ++j)
            if (!taken[j]) w.thr[at++] = left[j];
        for (int j = LG; j < LT; ++j) w.thr[j] = left[j];
    }

    static constexpr Tables make() {
        Tables t{};
        const WinClasses c = win_classes(LK, LOGW, M);
        // windows
        for (int r = 0; r < LK; ++r) t.win[0].reg[r] = r;
        for (int j = 0; j < LT; ++j) t.win[0].thr[j] = LK + j;
        t.win[0].refl = -1;
        fill_threads(t.win[0], c);
        int n = 0, pos = 0;
        for (int st = LK; st < LOGW; ++st)
            for (int j = st; j >= 0; --j) {
                if (pos == 0) {
                    ++n;
                    for (int r = 0; r < LK; ++r) t.win[n].reg[r] = -1;
                    t.win[n].refl = -1;
                    t.win[n].layers = 0;
                }
                t.win[n].reg[LK - 1 - pos] = j;
                if (j == st) {
                    t.win[n].refl = LK - 1 - pos;
                    t.win[n].st = st;
                }
                ++t.win[n].layers;
                pos = pos + 1 == LK ? 0 : pos + 1;
            }
        bool natural = true;  // whether the last window ends in the natural layout
        for (int r = 0; r < LK; ++r) natural = natural && t.win[n].reg[r] == r;
        if (pos != 0) {
            for (int r = 0; r < LK; ++r) t.win[n].reg[r] = r;  // a short run: bits layers-1 .. 0
        } else if (!natural) {
            ++n;
            for (int r = 0; r < LK; ++r) t.win[n].reg[r] = r;
            t.win[n].refl = -1;
            t.win[n].layers = 0;
        }
        t.windows = n;
        for (int w = 1; w <= n; ++w) fill_threads(t.win[w], c);
        // a merge of the whole tile: bits LOGW-1 .. 0, LK at a time, the last
        // run natural as above
        for (int top = LOGW - 1; top >= 0; top -= LK) {
            WinLayout& m = t.merge[t.merges++];
            m.refl = -1;
            m.layers = top + 1 < LK ? top + 1 : LK;
            for (int r = 0; r < LK; ++r) m.reg[r] = top + 1 < LK ? r : top - LK + 1 + r;
            fill_threads(m, c);
        }
        for (int r = 0; r < LK; ++r) t.io.reg[r] = LG + r;
        t.io.refl = -1;
        for (int j = 0; j < LG; ++j) t.io.thr[j] = j;
        for (int j = LG; j < LT; ++j) t.io.thr[j] = LK + j;
        // weights
        int w[kWinMaxBits] = {};
        const auto& cls = c.cls;
        int sum = 0;
        bool base = true;  // one bit of each class 0 .. M-1 among the index bits
        int first[8] = {};
        for (int k = 0; k < M; ++k) {
            first[k] = -1;
            for (int b = LOGW - 1; b >= 0; --b)
                if (cls[b] == k) first[k] = b;
            base = base && first[k] >= 0;
        }
        if (base)
            for (int k = 0; k < M; ++k) {
                w[first[k]] = 1 << k;
                sum += 1 << k;
            }
        // then the others: multiples of 2^M first, then class 0, 1, ..
        for (int pass = 0; pass <= M; ++pass) {
            const int k = pass == 0 ? M : pass - 1;
            for (int b = 0; b < LOGW; ++b)
                if (w[b] == 0 && cls[b] == k) {
                    const int mod = k == M ? 1 << M : 2 << k, want = k == M ? 0 : 1 << k;
                    int v = sum + 1;
                    while (v % mod != want) ++v;
                    w[b] = v;
                    sum += v;
                }
        }
        for (int b = 0; b < LOGW; ++b) t.weight[b] = w[b];
        t.elems = sum + 1;
        return t;
    }
    static constexpr Tables kT = make();

    // Address part of register q in a layout.
    static constexpr int reg_off(const WinLayout& w, int q) {
        int a = 0;
        for (int r = 0; r < LK; ++r)
            if ((q >> r) & 1) a += kT.weight[w.reg[r]];
        return a;
    }
    // Whether register q of window w is stored with complemented thread bits.
    static constexpr bool mirrored(const WinLayout& w, int q) { return w.refl >= 0 && ((q >> w.refl) & 1); }
    // Whether every warp holds the same part of the tile in both layouts.
    static constexpr bool same_warps(const WinLayout& a, const WinLayout& b) {
        for (int j = LG; j < LT; ++j)
            if (a.thr[j] != b.thr[j] || (a.refl >= 0 && a.thr[j] < a.st) || (b.refl >= 0 && b.thr[j] < b.st))
                return false;
        return true;
    }
};

}  // namespace b200s
