// Sums of products kept unreduced until they end (entry sums: a weight times a table entry of any layout).
//
// A field product mod r is 64 multiply-adds for the product and as many for its reduction; a sum needs the reduction
// once.  An integer entry needs no field product at all: 8 multiply-adds per 32 bits.
#pragma once
#include "family.cuh"

namespace dpb {

// INT: the entries are integers (DPB_*_I32 / DPB_*_I64).
template <class F, bool INT>
struct EntrySum;

template <>
struct EntrySum<FrFam, false> {
    static constexpr bool kPlus31 = false;
    frw::Wide s;
    __device__ __forceinline__ void zero() { s = frw::wide_zero(); }
    __device__ __forceinline__ void mac(const Fr& w, const void* __restrict__ p, int, uint64_t i) {
        frw::wide_mac(s, frw::from_fr(w), frw::from_fr(FrFam::load(p, DPB_FR, i)));
    }
    __device__ __forceinline__ Fr finish() const { return fr_wide_finish(s); }
};
// An entry x enters as x + 2^31, which is an unsigned word for every integer of 32 bits: the result is 2^31 times the
// sum of the weights too large (kPlus31), which the caller takes back.
template <>
struct EntrySum<FrFam, true> {
    static constexpr bool kPlus31 = true;
    FrIntAcc s;
    __device__ __forceinline__ void zero() { s = fr_intacc_zero(); }
    __device__ __forceinline__ void mac(const Fr& w, const void* __restrict__ p, int dtype, uint64_t i) {
        const frw::F8 ww = frw::from_fr(w);
        if (dtype == DPB_FR_I32) {
            frw::intacc_mac_lo(s.a, ww, (uint32_t)((const int32_t*)p)[i] ^ 0x80000000u);
            return;
        }
        const int64_t x = ((const int64_t*)p)[i];
        const uint64_t y = (uint64_t)x + 0x80000000ull;  // hi 2^32 + lo, hi of x's sign and zero for 32-bit integers
        const uint32_t hi = (uint32_t)(y >> 32);
        frw::intacc_mac_lo(s.a, ww, (uint32_t)y);
        if (hi) frw::intacc_mac_hi(s.a, x < 0 ? frw::from_fr(fr_neg(w)) : ww, x < 0 ? (uint32_t)0 - hi : hi);
    }
    __device__ __forceinline__ Fr finish() const { return fr_intacc_finish(s); }
};

template <bool INT>
struct EntrySum<GlFam, INT> {
    static constexpr bool kPlus31 = false;
    glw::A8 s0, s1;
    __device__ __forceinline__ void zero() { s0 = s1 = glw::acc_zero(); }
    __device__ __forceinline__ void mac(const Gl2& w, const void* __restrict__ p, int dtype, uint64_t i) {
        const glw::W2 ww = gl2_words(w), x = gl2_words(GlFam::load(p, dtype, i));
        glw::acc_mac(s0, ww.c0, x.c0);
        glw::acc_mac(s1, ww.c1, x.c0);
        if (!INT && dtype == DPB_GL_EXT) {
            glw::acc_mac(s0, glw::mul7(ww.c1), x.c1);
            glw::acc_mac(s1, ww.c0, x.c1);
        }
    }
    __device__ __forceinline__ Gl2 finish() const {
        return gl2_make(glw::to_u64(glw::canon(glw::acc_reduce(s0))), glw::to_u64(glw::canon(glw::acc_reduce(s1))));
    }
};

// c u + a d, reduced once
template <class F>
struct TwoProducts;
template <>
struct TwoProducts<FrFam> {
    __device__ __forceinline__ static Fr sum(const Fr& c, const Fr& u, const Fr& a, const Fr& d) {
        frw::Wide s = frw::wide_zero();
        frw::wide_mac(s, frw::from_fr(c), frw::from_fr(u));
        frw::wide_mac(s, frw::from_fr(a), frw::from_fr(d));
        return fr_wide_finish(s);
    }
};
template <>
struct TwoProducts<GlFam> {
    __device__ __forceinline__ static Gl2 sum(const Gl2& c, const Gl2& u, const Gl2& a, const Gl2& d) {
        glw::A8 s0 = glw::acc_zero(), s1 = glw::acc_zero();
        auto mac = [&](const glw::W2& x, const glw::W2& y) {
            glw::acc_mac(s0, x.c0, y.c0);
            glw::acc_mac(s0, glw::mul7(x.c1), y.c1);
            glw::acc_mac(s1, x.c0, y.c1);
            glw::acc_mac(s1, x.c1, y.c0);
        };
        mac(gl2_words(c), gl2_words(u));
        mac(gl2_words(a), gl2_words(d));
        return gl2_make(glw::to_u64(glw::canon(glw::acc_reduce(s0))), glw::to_u64(glw::canon(glw::acc_reduce(s1))));
    }
};

}  // namespace dpb
