// Values exchanged between the CTAs of one cooperative launch without fences:
// a 64-bit word carries 32 bits of data and a 32-bit tag (the publication it
// belongs to) and is written and read as one access, so a reader that sees the
// tag has the data. An FP64 value takes two words. A vector access moves two
// words; each is checked by its own tag.
#pragma once

#include <cstdint>

namespace cmcg {

__device__ __forceinline__ uint64_t tagged(uint32_t data, uint32_t tag) {
    return static_cast<uint64_t>(tag) << 32 | data;
}
__device__ __forceinline__ void st_word(uint64_t* p, uint64_t v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void st_word2(uint64_t* p, uint64_t a, uint64_t b) {
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
// Predicated loads (no branch, so a reader's loads stay in flight together);
// where not wanted the words keep their value.
__device__ __forceinline__ void ld_word_if(bool on, const uint64_t* p, uint64_t& v) {
    asm volatile("{\n.reg .pred q;\nsetp.ne.u32 q, %2, 0;\n@q ld.relaxed.gpu.global.u64 %0, [%1];\n}"
                 : "+l"(v) : "l"(p), "r"(static_cast<unsigned>(on)) : "memory");
}
__device__ __forceinline__ void ld_word2_if(bool on, const uint64_t* p, uint64_t& a, uint64_t& b) {
    asm volatile("{\n.reg .pred q;\nsetp.ne.u32 q, %3, 0;\n@q ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];\n}"
                 : "+l"(a), "+l"(b) : "l"(p), "r"(static_cast<unsigned>(on)) : "memory");
}

// words per value: one for 32 bits, two for 64
template <typename VT> constexpr int kWords = static_cast<int>(sizeof(VT) / 4);

__device__ __forceinline__ void put_value(uint64_t* p, float v, uint32_t tag) {
    st_word(p, tagged(__float_as_uint(v), tag));
}
__device__ __forceinline__ void put_value(uint64_t* p, double v, uint32_t tag) {
    const uint64_t u = __double_as_longlong(v);
    st_word2(p, tagged(static_cast<uint32_t>(u), tag), tagged(static_cast<uint32_t>(u >> 32), tag));
}
// The words of one value; the reader loads all it waits for, then checks the
// tags. A word that is not wanted counts as arrived and gives 0.
template <typename VT> struct TaggedValue;
template <> struct TaggedValue<float> {
    uint64_t w;
    __device__ __forceinline__ void load(bool on, const uint64_t* p, uint32_t want) {
        w = tagged(0u, want);
        ld_word_if(on, p, w);
    }
    __device__ __forceinline__ bool arrived(uint32_t want) const { return static_cast<uint32_t>(w >> 32) == want; }
    __device__ __forceinline__ float value() const { return __uint_as_float(static_cast<uint32_t>(w)); }
};
template <> struct TaggedValue<double> {
    uint64_t a, b;
    __device__ __forceinline__ void load(bool on, const uint64_t* p, uint32_t want) {
        a = b = tagged(0u, want);
        ld_word2_if(on, p, a, b);
    }
    __device__ __forceinline__ bool arrived(uint32_t want) const {
        return static_cast<uint32_t>(a >> 32) == want && static_cast<uint32_t>(b >> 32) == want;
    }
    __device__ __forceinline__ double value() const {
        return __longlong_as_double(static_cast<long long>((b << 32) | (a & 0xffffffffu)));
    }
};
// Two neighbouring values (16-byte aligned words); second: whether the second
// one is wanted too.
template <typename VT> struct TaggedPair;
template <> struct TaggedPair<float> {
    uint64_t a, b;
    __device__ __forceinline__ void load(bool on, bool second, const uint64_t* p, uint32_t want) {
        a = b = tagged(0u, want);
        ld_word2_if(on, p, a, b);
        if (!second) b = tagged(0u, want);
    }
    __device__ __forceinline__ bool arrived(uint32_t want) const {
        return static_cast<uint32_t>(a >> 32) == want && static_cast<uint32_t>(b >> 32) == want;
    }
    __device__ __forceinline__ float first() const { return __uint_as_float(static_cast<uint32_t>(a)); }
    __device__ __forceinline__ float second() const { return __uint_as_float(static_cast<uint32_t>(b)); }
};
template <> struct TaggedPair<double> {
    TaggedValue<double> u, v;
    __device__ __forceinline__ void load(bool on, bool second, const uint64_t* p, uint32_t want) {
        u.load(on, p, want);
        v.load(on && second, p + 2, want);
    }
    __device__ __forceinline__ bool arrived(uint32_t want) const { return u.arrived(want) && v.arrived(want); }
    __device__ __forceinline__ double first() const { return u.value(); }
    __device__ __forceinline__ double second() const { return v.value(); }
};
// NV = 1 or 2 values of a partial sum
template <typename VT, int NV> struct TaggedSum {
    TaggedValue<VT> w;
    __device__ __forceinline__ void load(bool on, const uint64_t* p, uint32_t want) { w.load(on, p, want); }
    __device__ __forceinline__ bool arrived(uint32_t want) const { return w.arrived(want); }
    __device__ __forceinline__ VT value(int) const { return w.value(); }
};
template <typename VT> struct TaggedSum<VT, 2> {
    TaggedPair<VT> w;
    __device__ __forceinline__ void load(bool on, const uint64_t* p, uint32_t want) { w.load(on, true, p, want); }
    __device__ __forceinline__ bool arrived(uint32_t want) const { return w.arrived(want); }
    __device__ __forceinline__ VT value(int j) const { return j == 0 ? w.first() : w.second(); }
};
// two neighbouring values (16-byte aligned words)
__device__ __forceinline__ void put_pair(uint64_t* p, float a, float b, uint32_t tag) {
    st_word2(p, tagged(__float_as_uint(a), tag), tagged(__float_as_uint(b), tag));
}
__device__ __forceinline__ void put_pair(uint64_t* p, double a, double b, uint32_t tag) {
    put_value(p, a, tag);
    put_value(p + 2, b, tag);
}

}  // namespace cmcg
