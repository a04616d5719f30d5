// Element types and their comparison rules for the batched bitonic sort.
//
// Memory layouts (what the caller's buffers hold):
//   int32_t   keys only                                   4 B
//   RecI32    {int32 key; int32 data;}  == IntAndData     8 B  (intanddata.hpp:9-11)
//   uint64_t  keys only                                   8 B
//   RecU64    {uint64 key; int32 data; int32 reserved;}  16 B  (AoS; reserved is written as 0)
//
// Register forms (what a thread holds while sorting) add an original-position
// word in the stable mode, so that ties are broken by input order.
//
// Ordering follows the reference: records compare by key only
// (intanddata.hpp:20-31) and, on the default path, a comparator keeps its own
// element on ties: min(a,b) = b<a ? b : a, max(a,b) = a<b ? b : a
// (cusort.hpp:460-472).  Padding uses the maximum key with a maximum payload
// (cusort.hpp:257-271, intanddata.hpp:47-52).
#pragma once
#include <climits>
#include <cstdint>

namespace b200s {

struct RecI32 {
    int32_t key;
    int32_t data;
};
struct __align__(16) RecU64 {
    uint64_t key;
    int32_t data;
    int32_t reserved;
};

// Element J of a 16-byte word, and the inverse, for each memory layout; J is
// a compile-time index so the moves stay in registers.
template <int J>
__device__ __forceinline__ void from_u4(const uint4& u, int32_t& m) {
    m = int32_t(J == 0 ? u.x : J == 1 ? u.y : J == 2 ? u.z : u.w);
}
template <int J>
__device__ __forceinline__ void to_u4(uint4& u, int32_t m) {
    if constexpr (J == 0) u.x = uint32_t(m);
    else if constexpr (J == 1) u.y = uint32_t(m);
    else if constexpr (J == 2) u.z = uint32_t(m);
    else u.w = uint32_t(m);
}
template <int J>
__device__ __forceinline__ void from_u4(const uint4& u, uint64_t& m) {
    m = J == 0 ? (uint64_t(u.y) << 32 | u.x) : (uint64_t(u.w) << 32 | u.z);
}
template <int J>
__device__ __forceinline__ void to_u4(uint4& u, uint64_t m) {
    if constexpr (J == 0) {
        u.x = uint32_t(m);
        u.y = uint32_t(m >> 32);
    } else {
        u.z = uint32_t(m);
        u.w = uint32_t(m >> 32);
    }
}
template <int J>
__device__ __forceinline__ void from_u4(const uint4& u, RecI32& m) {
    m.key = int32_t(J == 0 ? u.x : u.z);
    m.data = int32_t(J == 0 ? u.y : u.w);
}
template <int J>
__device__ __forceinline__ void to_u4(uint4& u, const RecI32& m) {
    if constexpr (J == 0) {
        u.x = uint32_t(m.key);
        u.y = uint32_t(m.data);
    } else {
        u.z = uint32_t(m.key);
        u.w = uint32_t(m.data);
    }
}
template <int J>
__device__ __forceinline__ void from_u4(const uint4& u, RecU64& m) {
    m.key = uint64_t(u.y) << 32 | u.x;
    m.data = int32_t(u.z);
    m.reserved = int32_t(u.w);
}
template <int J>
__device__ __forceinline__ void to_u4(uint4& u, const RecU64& m) {
    u.x = uint32_t(m.key);
    u.y = uint32_t(m.key >> 32);
    u.z = uint32_t(m.data);
    u.w = uint32_t(m.reserved);
}

__device__ __forceinline__ uint32_t shfl_x(uint32_t v, int m) {
    return __shfl_xor_sync(0xffffffffu, v, m);
}
__device__ __forceinline__ int32_t shfl_x(int32_t v, int m) {
    return __shfl_xor_sync(0xffffffffu, v, m);
}
__device__ __forceinline__ uint64_t shfl_x(uint64_t v, int m) {
    return __shfl_xor_sync(0xffffffffu, (unsigned long long)v, m);
}
__device__ __forceinline__ int32_t shfl_d(int32_t v, int d) { return __shfl_down_sync(0xffffffffu, v, d); }
__device__ __forceinline__ uint64_t shfl_d(uint64_t v, int d) {
    return __shfl_down_sync(0xffffffffu, (unsigned long long)v, d);
}

// The value 1, opaque to the compiler (every launch has gridDim.z == 1).  A
// multiplication by it is a register move on the FMA pipe.
//
// Why: a compare-exchange written as a compare and selects runs on the ALU pipe
// alone, which takes a warp instruction every two cycles: 5 instructions, 10
// cycles per pair of records (measured in a register-only loop, 8 warps per
// scheduler), while the FMA pipe idles.  Moving the payloads with predicated
// multiplications leaves 3 ALU and 3 FMA instructions: 7.0 cycles.  For 64-bit
// keys the compiler turns compare + selects into a minimum and a maximum with a
// comparison each, 16 cycles; one comparison with one or both words moved on the
// FMA pipe takes 9.3 or 12.5, and two of the first to one of the second 8.7.
__device__ __forceinline__ int opaque_one() {
    int r;
    asm("mov.u32 %0, %%nctaid.z;" : "=r"(r));
    return r;
}

// PTX of one word's exchange under predicate q (operands by number): on the
// FMA pipe (ONE: the operand that holds opaque_one()) or by selects.
#define B200S_SWAP_FMA(A, B, ONE, T) \
    "mul.lo.u32 " T ", %" A ", %" ONE ";\n\t@q mul.lo.u32 %" A ", %" B ", %" ONE ";\n\t@q mul.lo.u32 %" B ", " T \
    ", %" ONE ";\n\t"
#define B200S_SWAP_SEL(A, B, T) \
    "selp.b32 " T ", %" B ", %" A ", q;\n\tselp.b32 %" B ", %" A ", %" B ", q;\n\tmov.b32 %" A ", " T ";\n\t"

// Ascending compare-exchange of two unsigned 64-bit values (strict): the low
// words on the FMA pipe, the high words there too when FMA_HIGH.
template <bool FMA_HIGH>
__device__ __forceinline__ void cex_u64(uint64_t& lo, uint64_t& hi) {
    uint32_t a0 = uint32_t(lo), a1 = uint32_t(lo >> 32), b0 = uint32_t(hi), b1 = uint32_t(hi >> 32);
    const int one = opaque_one();
    if constexpr (FMA_HIGH)
        asm("{\n\t.reg .pred q;\n\t.reg .u32 u, w;\n\t.reg .u64 x, y;\n\t"
            "mov.b64 x, {%0, %1};\n\tmov.b64 y, {%2, %3};\n\tsetp.lt.u64 q, y, x;\n\t"
            B200S_SWAP_FMA("0", "2", "4", "u") B200S_SWAP_FMA("1", "3", "4", "w") "}"
            : "+r"(a0), "+r"(a1), "+r"(b0), "+r"(b1)
            : "r"(one));
    else
        asm("{\n\t.reg .pred q;\n\t.reg .u32 u, w;\n\t.reg .u64 x, y;\n\t"
            "mov.b64 x, {%0, %1};\n\tmov.b64 y, {%2, %3};\n\tsetp.lt.u64 q, y, x;\n\t"
            B200S_SWAP_FMA("0", "2", "4", "u") B200S_SWAP_SEL("1", "3", "w") "}"
            : "+r"(a0), "+r"(a1), "+r"(b0), "+r"(b1)
            : "r"(one));
    lo = uint64_t(a1) << 32 | a0;
    hi = uint64_t(b1) << 32 | b0;
}

// ---- int32 keys --------------------------------------------------------------
struct ElemI32 {
    static constexpr bool kKeysOnly = true;  // tie order unobservable
    using Mem = int32_t;
    using Reg = int32_t;
    static constexpr bool kStable = false;
    static constexpr bool kCompact = false;
    static __device__ __forceinline__ Reg pad() { return INT32_MAX; }
    static __device__ __forceinline__ Reg from_mem(Mem m, int) { return m; }
    static __device__ __forceinline__ Mem to_mem(Reg r) { return r; }
    static __device__ __forceinline__ Reg shfl(Reg v, int m) { return shfl_x(v, m); }
    static __device__ __forceinline__ Reg shfl_down(Reg v, int d) { return shfl_d(v, d); }
    // b belongs before a (the pair (a, b) is out of order).
    static __device__ __forceinline__ bool after(Reg a, Reg b) { return b < a; }
    // Ascending compare-exchange of (lower, upper).  Equal keys are
    // indistinguishable, so min/max is the keep-own rule.
    static __device__ __forceinline__ void cex(Reg& lo, Reg& hi) {
        const Reg a = lo, b = hi;
        lo = min(a, b);
        hi = max(a, b);
    }
    // One side of a cross-thread compare-exchange: the upper side keeps the
    // larger, the lower side the smaller.
    static __device__ __forceinline__ Reg pick(Reg own, Reg other, bool upper) {
        return upper ? max(own, other) : min(own, other);
    }
};

// int32 keys through the compact network: for the 4- and 8-CTA cluster tiles,
// whose fully unrolled network spills at 128 registers (432-728 bytes); the
// compact form does not, and is 5-8 % faster there (16 M keys, n = 65536:
// 0.43 -> 0.40 ms; 131072: 0.61 -> 0.58 ms).  Same comparators, same output.
struct ElemI32C : ElemI32 {
    static constexpr bool kCompact = true;
};

// ---- uint64 keys -------------------------------------------------------------
struct ElemU64 {
    static constexpr bool kKeysOnly = true;
    using Mem = uint64_t;
    using Reg = uint64_t;
    static constexpr bool kStable = false;
    static constexpr bool kCompact = true;
    static __device__ __forceinline__ Reg pad() { return UINT64_MAX; }
    static __device__ __forceinline__ Reg from_mem(Mem m, int) { return m; }
    static __device__ __forceinline__ Mem to_mem(Reg r) { return r; }
    static __device__ __forceinline__ Reg shfl(Reg v, int m) { return shfl_x(v, m); }
    static __device__ __forceinline__ Reg shfl_down(Reg v, int d) { return shfl_d(v, d); }
    static __device__ __forceinline__ bool after(Reg a, Reg b) { return b < a; }
    // Number Q of a layer: one in three moves both words on the FMA pipe,
    // which balances the two pipes.
    template <int Q>
    static __device__ __forceinline__ void cexq(Reg& lo, Reg& hi) {
        cex_u64<Q % 3 == 0>(lo, hi);
    }
    static __device__ __forceinline__ void cex(Reg& lo, Reg& hi) { cex_u64<false>(lo, hi); }
    static __device__ __forceinline__ Reg pick(Reg own, Reg other, bool upper) {
        const bool take = upper ? (own < other) : (other < own);
        return take ? other : own;
    }
};

// The same with compare and selects, the latency form of the tiles of W = 64 ..
// 2048 (see ElemRecI32L).
struct ElemU64L : ElemU64 {
    template <int Q>
    static __device__ __forceinline__ void cexq(Reg& lo, Reg& hi) {
        cex(lo, hi);
    }
    static __device__ __forceinline__ void cex(Reg& lo, Reg& hi) {
        const Reg a = lo, b = hi;
        const bool sw = b < a;
        lo = sw ? b : a;
        hi = sw ? a : b;
    }
};

// ---- records: int32 key + int32 payload (IntAndData) ------------------------
struct RegRecI32 {
    int32_t key;
    int32_t data;
};
struct ElemRecI32 {
    using Mem = RecI32;
    using Reg = RegRecI32;
    static constexpr bool kStable = false;
    static constexpr bool kCompact = true;
    static __device__ __forceinline__ Reg pad() { return Reg{INT32_MAX, INT32_MAX}; }
    static __device__ __forceinline__ Reg from_mem(Mem m, int) { return Reg{m.key, m.data}; }
    static __device__ __forceinline__ Mem to_mem(Reg r) { return Mem{r.key, r.data}; }
    static __device__ __forceinline__ Reg shfl(Reg v, int m) {
        return Reg{shfl_x(v.key, m), shfl_x(v.data, m)};
    }
    static __device__ __forceinline__ Reg shfl_down(Reg v, int d) { return Reg{shfl_d(v.key, d), shfl_d(v.data, d)}; }
    static __device__ __forceinline__ bool after(const Reg& a, const Reg& b) { return b.key < a.key; }
    // Strict: ties keep their places.
    static __device__ __forceinline__ void cex(Reg& lo, Reg& hi) {
        asm("{\n\t.reg .pred q;\n\t.reg .s32 t;\n\t.reg .u32 u;\n\t"
            "setp.lt.s32 q, %1, %0;\n\tmin.s32 t, %0, %1;\n\tmax.s32 %1, %0, %1;\n\tmov.s32 %0, t;\n\t"
            B200S_SWAP_FMA("2", "3", "4", "u") "}"
            : "+r"(lo.key), "+r"(hi.key), "+r"(lo.data), "+r"(hi.data)
            : "r"(opaque_one()));
    }
    static __device__ __forceinline__ Reg pick(Reg own, Reg other, bool upper) {
        const bool take = upper ? (own.key < other.key) : (other.key < own.key);
        return Reg{take ? other.key : own.key, take ? other.data : own.data};
    }
};

// The same with compare and selects: fewer instructions in all and shorter
// code, for batches that leave the SMs mostly idle, where one warp's latency
// and its instruction fetches count and no pipe is full (W = 256 .. 2048; see
// kLatencyWarps in instantiate.cuh).
struct ElemRecI32L : ElemRecI32 {
    static __device__ __forceinline__ void cex(Reg& lo, Reg& hi) {
        const Reg a = lo, b = hi;
        const bool sw = b.key < a.key;
        lo.key = sw ? b.key : a.key;
        lo.data = sw ? b.data : a.data;
        hi.key = sw ? a.key : b.key;
        hi.data = sw ? a.data : b.data;
    }
};

// Stable mode for IntAndData: (key, original position) is unique, so the
// network output equals a stable sort by key.
struct RegRecI32S {
    int32_t key;
    int32_t data;
    int32_t pos;
};
struct ElemRecI32S {
    using Mem = RecI32;
    using Reg = RegRecI32S;
    static constexpr bool kStable = true;
    static constexpr bool kCompact = true;
    static __device__ __forceinline__ Reg pad() { return Reg{INT32_MAX, INT32_MAX, INT32_MAX}; }
    static __device__ __forceinline__ Reg from_mem(Mem m, int pos) { return Reg{m.key, m.data, pos}; }
    static __device__ __forceinline__ Mem to_mem(Reg r) { return Mem{r.key, r.data}; }
    static __device__ __forceinline__ Reg shfl(Reg v, int m) {
        return Reg{shfl_x(v.key, m), shfl_x(v.data, m), shfl_x(v.pos, m)};
    }
    static __device__ __forceinline__ Reg shfl_down(Reg v, int d) {
        return Reg{shfl_d(v.key, d), shfl_d(v.data, d), shfl_d(v.pos, d)};
    }
    static __device__ __forceinline__ bool lt(const Reg& a, const Reg& b) {
        return a.key < b.key || (a.key == b.key && a.pos < b.pos);
    }
    static __device__ __forceinline__ bool after(const Reg& a, const Reg& b) { return lt(b, a); }
    static __device__ __forceinline__ void cex(Reg& lo, Reg& hi) {
        const Reg a = lo, b = hi;
        const bool sw = lt(b, a);
        lo.key = sw ? b.key : a.key;
        lo.data = sw ? b.data : a.data;
        lo.pos = sw ? b.pos : a.pos;
        hi.key = sw ? a.key : b.key;
        hi.data = sw ? a.data : b.data;
        hi.pos = sw ? a.pos : b.pos;
    }
    static __device__ __forceinline__ Reg pick(Reg own, Reg other, bool upper) {
        const bool take = upper ? lt(own, other) : lt(other, own);
        Reg r;
        r.key = take ? other.key : own.key;
        r.data = take ? other.data : own.data;
        r.pos = take ? other.pos : own.pos;
        return r;
    }
};

// The same order on one 64-bit word per record, the key above the position;
// the payload stays behind and is fetched by position when the sorted record
// is written (kGather).  Two words per compare-exchange instead of three, a
// comparison of one 64-bit value instead of two words with a tie case, and
// 8 bytes per record through shared memory instead of 12; the words are
// distinct, so any sorting network gives the stable order.
struct ElemRecI32G : ElemU64 {
    using Mem = RecI32;
    static constexpr bool kStable = true;
    static constexpr bool kGather = true;
    static __device__ __forceinline__ Reg from_mem(Mem m, int pos) {
        return uint64_t(uint32_t(m.key) ^ 0x80000000u) << 32 | uint32_t(pos);
    }
    static __device__ __forceinline__ int position(Reg r) { return int(uint32_t(r)); }
    static __device__ __forceinline__ Mem to_mem(Reg r, int32_t data) {
        return Mem{int32_t(uint32_t(r >> 32) ^ 0x80000000u), data};
    }
};

// ---- records: uint64 key + int32 payload -------------------------------------
struct alignas(16) RegRecU64 {
    uint64_t key;
    int32_t data;
};
struct ElemRecU64 {
    using Mem = RecU64;
    using Reg = RegRecU64;
    static constexpr bool kStable = false;
    static constexpr bool kCompact = true;
    static __device__ __forceinline__ Reg pad() { return Reg{UINT64_MAX, INT32_MAX}; }
    static __device__ __forceinline__ Reg from_mem(Mem m, int) { return Reg{m.key, m.data}; }
    static __device__ __forceinline__ Mem to_mem(Reg r) { return Mem{r.key, r.data, 0}; }
    static __device__ __forceinline__ Reg shfl(Reg v, int m) {
        return Reg{shfl_x(v.key, m), shfl_x(v.data, m)};
    }
    static __device__ __forceinline__ Reg shfl_down(Reg v, int d) { return Reg{shfl_d(v.key, d), shfl_d(v.data, d)}; }
    static __device__ __forceinline__ bool after(const Reg& a, const Reg& b) { return b.key < a.key; }
    // Word by word (whole-struct selects of this padded register record made
    // the compiler spill), the words shared between the pipes: even numbers of
    // a layer move one word on the FMA pipe, odd ones two.
    template <int Q>
    static __device__ __forceinline__ void cexq(Reg& lo, Reg& hi) {
        uint32_t a0 = uint32_t(lo.key), a1 = uint32_t(lo.key >> 32), b0 = uint32_t(hi.key), b1 = uint32_t(hi.key >> 32);
        const int one = opaque_one();
        if constexpr (Q % 2 == 0)
            asm("{\n\t.reg .pred q;\n\t.reg .u32 u, w, z;\n\t.reg .u64 x, y;\n\t"
                "mov.b64 x, {%0, %1};\n\tmov.b64 y, {%2, %3};\n\tsetp.lt.u64 q, y, x;\n\t"
                B200S_SWAP_FMA("0", "2", "6", "u") B200S_SWAP_SEL("1", "3", "w") B200S_SWAP_SEL("4", "5", "z") "}"
                : "+r"(a0), "+r"(a1), "+r"(b0), "+r"(b1), "+r"(lo.data), "+r"(hi.data)
                : "r"(one));
        else
            asm("{\n\t.reg .pred q;\n\t.reg .u32 u, w, z;\n\t.reg .u64 x, y;\n\t"
                "mov.b64 x, {%0, %1};\n\tmov.b64 y, {%2, %3};\n\tsetp.lt.u64 q, y, x;\n\t"
                B200S_SWAP_FMA("0", "2", "6", "u") B200S_SWAP_SEL("1", "3", "w") B200S_SWAP_FMA("4", "5", "6", "z") "}"
                : "+r"(a0), "+r"(a1), "+r"(b0), "+r"(b1), "+r"(lo.data), "+r"(hi.data)
                : "r"(one));
        lo.key = uint64_t(a1) << 32 | a0;
        hi.key = uint64_t(b1) << 32 | b0;
    }
    // For the loops of the blocked network, where a batch of a few arrays is
    // bound by one warp's latency: the compiler's selects (14 arrays of 345:
    // 9.9 us per call, 12.5 with cexq).
    static __device__ __forceinline__ void cex(Reg& lo, Reg& hi) {
        const Reg a = lo, b = hi;
        const bool sw = b.key < a.key;
        lo.key = sw ? b.key : a.key;
        lo.data = sw ? b.data : a.data;
        hi.key = sw ? a.key : b.key;
        hi.data = sw ? a.data : b.data;
    }
    static __device__ __forceinline__ Reg pick(Reg own, Reg other, bool upper) {
        const bool take = upper ? (own.key < other.key) : (other.key < own.key);
        Reg r;
        r.key = take ? other.key : own.key;
        r.data = take ? other.data : own.data;
        return r;
    }
};

struct alignas(16) RegRecU64S {
    uint64_t key;
    int32_t data;
    int32_t pos;
};
struct ElemRecU64S {
    using Mem = RecU64;
    using Reg = RegRecU64S;
    static constexpr bool kStable = true;
    static constexpr bool kCompact = true;
    static __device__ __forceinline__ Reg pad() { return Reg{UINT64_MAX, INT32_MAX, INT32_MAX}; }
    static __device__ __forceinline__ Reg from_mem(Mem m, int pos) { return Reg{m.key, m.data, pos}; }
    static __device__ __forceinline__ Mem to_mem(Reg r) { return Mem{r.key, r.data, 0}; }
    static __device__ __forceinline__ Reg shfl(Reg v, int m) {
        return Reg{shfl_x(v.key, m), shfl_x(v.data, m), shfl_x(v.pos, m)};
    }
    static __device__ __forceinline__ Reg shfl_down(Reg v, int d) {
        return Reg{shfl_d(v.key, d), shfl_d(v.data, d), shfl_d(v.pos, d)};
    }
    static __device__ __forceinline__ bool lt(const Reg& a, const Reg& b) {
        return a.key < b.key || (a.key == b.key && a.pos < b.pos);
    }
    static __device__ __forceinline__ bool after(const Reg& a, const Reg& b) { return lt(b, a); }
    // b < a as one 96-bit subtraction of (key, position), its borrow the
    // exchange; two of the four words move on the FMA pipe.
    static __device__ __forceinline__ void cex(Reg& lo, Reg& hi) {
        uint32_t a0 = uint32_t(lo.key), a1 = uint32_t(lo.key >> 32), b0 = uint32_t(hi.key), b1 = uint32_t(hi.key >> 32);
        asm("{\n\t.reg .pred q;\n\t.reg .u32 d, u, w, y, z;\n\t"
            "sub.cc.u32 d, %7, %6;\n\tsubc.cc.u32 d, %2, %0;\n\tsubc.cc.u32 d, %3, %1;\n\tsubc.u32 d, 0, 0;\n\t"
            "setp.ne.u32 q, d, 0;\n\t"
            B200S_SWAP_FMA("0", "2", "8", "u") B200S_SWAP_SEL("1", "3", "w") B200S_SWAP_FMA("4", "5", "8", "y")
            B200S_SWAP_SEL("6", "7", "z") "}"
            : "+r"(a0), "+r"(a1), "+r"(b0), "+r"(b1), "+r"(lo.data), "+r"(hi.data), "+r"(lo.pos), "+r"(hi.pos)
            : "r"(opaque_one()));
        lo.key = uint64_t(a1) << 32 | a0;
        hi.key = uint64_t(b1) << 32 | b0;
    }
    static __device__ __forceinline__ Reg pick(Reg own, Reg other, bool upper) {
        const bool take = upper ? lt(own, other) : lt(other, own);
        Reg r;
        r.key = take ? other.key : own.key;
        r.data = take ? other.data : own.data;
        r.pos = take ? other.pos : own.pos;
        return r;
    }
};

// uint64 keys alone are totally ordered values: the stable mode changes nothing.

// Shared-memory (and distributed-shared-memory) element accesses.  The
// 16-byte register records move as one 128-bit access: field by field (an
// 8-byte key, then a 4-byte payload at a 16-byte stride) each access takes
// two wavefronts per half-warp instead of one per quarter-warp.
template <class R>
__device__ __forceinline__ R sh_ld(const R* p) {
    return *p;
}
template <class R>
__device__ __forceinline__ void sh_st(R* p, const R& v) {
    *p = v;
}
// The fourth word is padding: one 128-bit shared-space load in PTX (p is in
// this CTA's shared memory), so that the compiler does not narrow it to an
// 8-byte and a 4-byte load.
__device__ __forceinline__ RegRecU64 sh_ld(const RegRecU64* p) {
    unsigned x, y, z, w;
    const unsigned a = unsigned(__cvta_generic_to_shared(p));
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(x), "=r"(y), "=r"(z), "=r"(w) : "r"(a) : "memory");
    (void)w;
    return RegRecU64{(uint64_t(y) << 32) | x, int32_t(z)};
}
__device__ __forceinline__ void sh_st(RegRecU64* p, const RegRecU64& v) {
    *reinterpret_cast<uint4*>(p) = make_uint4(unsigned(v.key), unsigned(v.key >> 32), unsigned(v.data), 0u);
}
// Reads of a cluster peer's shared memory (a generic pointer from
// map_shared_rank): plain loads, 128 bits for the 16-byte records.
template <class R>
__device__ __forceinline__ R dsm_ld(const R* p) {
    return *p;
}
__device__ __forceinline__ RegRecU64 dsm_ld(const RegRecU64* p) {
    const uint4 u = *reinterpret_cast<const uint4*>(p);
    return RegRecU64{(uint64_t(u.y) << 32) | u.x, int32_t(u.z)};
}
__device__ __forceinline__ RegRecU64S dsm_ld(const RegRecU64S* p) {
    const uint4 u = *reinterpret_cast<const uint4*>(p);
    return RegRecU64S{(uint64_t(u.y) << 32) | u.x, int32_t(u.z), int32_t(u.w)};
}
__device__ __forceinline__ RegRecU64S sh_ld(const RegRecU64S* p) {
    const uint4 u = *reinterpret_cast<const uint4*>(p);
    return RegRecU64S{(uint64_t(u.y) << 32) | u.x, int32_t(u.z), int32_t(u.w)};
}
__device__ __forceinline__ void sh_st(RegRecU64S* p, const RegRecU64S& v) {
    *reinterpret_cast<uint4*>(p) =
        make_uint4(unsigned(v.key), unsigned(v.key >> 32), unsigned(v.data), unsigned(v.pos));
}

}  // namespace b200s
