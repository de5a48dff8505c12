// Partial evaluation (fix_high / fix_low): one pass binds up to five variables,
// out[j] = sum_l w[l] * in[index(j, l)] with the 2^g eq weights of those
// variables.  One thread per output entry runs the whole sum, so nothing is
// exchanged between threads, and because the weights are fixed for the launch
// the products take the cheap forms: both fields accumulate the products
// lazily and reduce once per output, BN254 through precomputed rows of the
// weights.
#pragma once
#include "family.cuh"
#include "gl_words.cuh"
#include "sumcheck_kernels.cuh"

namespace dpb {

template <class F>
struct WSum;

template <>
struct WSum<GlFam> {
    struct Key {
        glw::W c0, c1, c1x7;  // the weight c0 + c1 X, and 7 c1
    };
    struct Acc {
        glw::A8 s0, s1;
    };
    // the block's threads fill keys[0..n) from the weights; the caller synchronises
    __device__ __forceinline__ static void make_keys_block(const Gl2* __restrict__ w, uint32_t n, Key* keys, int) {
        if (threadIdx.x < n) {
            const Gl2 v = w[threadIdx.x];
            Key k;
            k.c0 = glw::make_w((uint32_t)v.c0, (uint32_t)(v.c0 >> 32));
            k.c1 = glw::make_w((uint32_t)v.c1, (uint32_t)(v.c1 >> 32));
            k.c1x7 = glw::mul7(k.c1);
            keys[threadIdx.x] = k;
        }
    }
    __device__ __forceinline__ static Acc zero() {
        Acc a;
        a.s0 = a.s1 = glw::acc_zero();
        return a;
    }
    // acc += key * entry i
    __device__ __forceinline__ static void mac(Acc& a, const Key& k, const void* __restrict__ in, int dtype, uint64_t i) {
        if (dtype == DPB_GL_BASE) {
            const uint64_t x = ((const uint64_t*)in)[i];
            const glw::W xw = glw::make_w((uint32_t)x, (uint32_t)(x >> 32));
            glw::acc_mac(a.s0, xw, k.c0);
            glw::acc_mac(a.s1, xw, k.c1);
        } else if (dtype == DPB_GL_EXT) {
            const uint4 v = ((const uint4*)in)[i];
            const glw::W x0 = glw::make_w(v.x, v.y), x1 = glw::make_w(v.z, v.w);
            glw::acc_mac(a.s0, x0, k.c0);
            glw::acc_mac(a.s0, x1, k.c1x7);
            glw::acc_mac(a.s1, x0, k.c1);
            glw::acc_mac(a.s1, x1, k.c0);
        } else {  // integer tables: the base element the integer stands for
            const uint64_t x = GlFam::load(in, dtype, i).c0;
            const glw::W xw = glw::make_w((uint32_t)x, (uint32_t)(x >> 32));
            glw::acc_mac(a.s0, xw, k.c0);
            glw::acc_mac(a.s1, xw, k.c1);
        }
    }
    // acc += key0 * entry i + key1 * entry i + 1 of a base table, i even: one 16-byte load
    __device__ __forceinline__ static void mac_base_pair(Acc& a, const Key& k0, const Key& k1, const void* __restrict__ in,
                                                         uint64_t i) {
        const uint4 v = ((const uint4*)in)[i >> 1];
        const glw::W x0 = glw::make_w(v.x, v.y), x1 = glw::make_w(v.z, v.w);
        glw::acc_mac(a.s0, x0, k0.c0);
        glw::acc_mac(a.s1, x0, k0.c1);
        glw::acc_mac(a.s0, x1, k1.c0);
        glw::acc_mac(a.s1, x1, k1.c1);
    }
    static constexpr bool kBasePairs = true;
    __device__ __forceinline__ static void mac_int_quad(Acc&, const Key*, const void*, uint64_t) {}
    static constexpr bool kIntRows = false;
    __device__ __forceinline__ static Gl2 finish(const Acc& a, int) {
        return gl2_make(glw::to_u64(glw::canon(glw::acc_reduce(a.s0))), glw::to_u64(glw::canon(glw::acc_reduce(a.s1))));
    }
};

// BN254: the weight's eight rows times the entry's eight words land on the same aligned pairs for every entry, so the
// whole sum stays unreduced (2^5 entries of 8 words: below 2^294) and takes the two reduction words once per output:
// 64 multiply-adds per field entry instead of 80 and an addition mod r.  An integer entry x enters as the unsigned
// word x + 2^31: 8 multiply-adds; the weights of an eq table sum to one, so the sum is 2^31 too large, which finish
// takes back.  A 64-bit integer outside 32 bits adds its upper word times the weight's second row (the weight times
// 2^32), negated for a negative one.  Measured (int32, 2^26 entries, k = 10): 1243 us with every entry widened to a
// field element, 141 us since (HBM 41 us, multiply-adds 62 us).
template <>
struct WSum<FrFam> {
    typedef frw::FixedMul Key;
    typedef frw::RowAcc Acc;
    __device__ __forceinline__ static void make_keys_block(const Fr* __restrict__ w, uint32_t n, Key* keys, int dtype) {
        if (dtype == DPB_FR) {
            for (uint32_t t = threadIdx.x; t < 8 * n; t += blockDim.x) fr_fixed_row(w[t >> 3], (int)(t & 7), keys[t >> 3].c[t & 7]);
        } else {  // the two rows of a plain integer's words
            for (uint32_t t = threadIdx.x; t < 2 * n; t += blockDim.x) fr_fixed_row(w[t >> 1], 8 + (int)(t & 1), keys[t >> 1].c[t & 1]);
        }
    }
    __device__ __forceinline__ static Acc zero() { return frw::rowacc_zero(); }
    __device__ __forceinline__ static void mac_i32(Acc& a, const Key& k, int32_t x) {
        frw::rowacc_mac(a, k.c[0], (uint32_t)x ^ 0x80000000u);
    }
    __device__ __forceinline__ static void mac_i64(Acc& a, const Key& k, int64_t x) {
        // x + 2^31 = hi 2^32 + lo, hi of x's sign and zero for every x of 32 bits
        const uint64_t y = (uint64_t)x + 0x80000000ull;
        const uint32_t hi = (uint32_t)(y >> 32);
        frw::rowacc_mac(a, k.c[0], (uint32_t)y);
        if (hi != 0) {
            frw::F8 row;
#pragma unroll
            for (int w = 0; w < 8; w++) row.w[w] = k.c[1][w];
            if (x < 0) row = frw::from_fr(fr_neg(frw::to_fr(row)));
            frw::rowacc_mac(a, row.w, x < 0 ? (uint32_t)0 - hi : hi);
        }
    }
    __device__ __forceinline__ static void mac(Acc& a, const Key& k, const void* __restrict__ in, int dtype, uint64_t i) {
        if (dtype == DPB_FR_I32) {
            mac_i32(a, k, ((const int32_t*)in)[i]);
        } else if (dtype == DPB_FR_I64) {
            mac_i64(a, k, ((const int64_t*)in)[i]);
        } else {
            const frw::F8 v = frw::from_fr(FrFam::load(in, DPB_FR, i));
#pragma unroll
            for (int w = 0; w < 8; w++) frw::rowacc_mac(a, k.c[w], v.w[w]);
        }
    }
    // entries i .. i + 3 of an int32 table, i a multiple of 4: one 16-byte load
    __device__ __forceinline__ static void mac_int_quad(Acc& a, const Key* k, const void* __restrict__ in, uint64_t i) {
        const int4 v = ((const int4*)in)[i >> 2];
        mac_i32(a, k[0], v.x);
        mac_i32(a, k[1], v.y);
        mac_i32(a, k[2], v.z);
        mac_i32(a, k[3], v.w);
    }
    static constexpr bool kIntRows = true;
    __device__ __forceinline__ static void mac_base_pair(Acc&, const Key&, const Key&, const void*, uint64_t) {}
    static constexpr bool kBasePairs = false;
    __device__ __forceinline__ static Fr finish(Acc& a, int dtype) {
        const Fr v = frw::to_fr(frw::reduce_rows(a.E, a.O));
        return dtype != DPB_FR ? fr_sub(v, fr_two31()) : v;
    }
};

// Bottom g variables (g <= 5): out[j] = sum_{l < 2^g} w[l] * in[j * 2^g + l].
template <class F>
__global__ void __launch_bounds__(kThreads)
    fix_low_sum(const void* __restrict__ in, int dtype_in, const typename F::E* __restrict__ w, uint32_t g,
                uint64_t n_out, typename F::E* __restrict__ out) {
    __shared__ typename WSum<F>::Key keys[32];
    const uint32_t G = 1u << g;
    WSum<F>::make_keys_block(w, G, keys, dtype_in);
    __syncthreads();
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n_out; j += stride) {
        typename WSum<F>::Acc acc = WSum<F>::zero();
        if (WSum<F>::kBasePairs && dtype_in == DPB_GL_BASE) {  // G >= 2 entries of 8 bytes, read two at a time
            for (uint32_t l = 0; l < G; l += 2) WSum<F>::mac_base_pair(acc, keys[l], keys[l + 1], in, (j << g) + l);
        } else if (WSum<F>::kIntRows && dtype_in == DPB_FR_I32 && g >= 2) {  // a thread's entries, 16 bytes at a time
            for (uint32_t l = 0; l < G; l += 4) WSum<F>::mac_int_quad(acc, keys + l, in, (j << g) + l);
        } else {
            for (uint32_t l = 0; l < G; l++) WSum<F>::mac(acc, keys[l], in, dtype_in, (j << g) + l);
        }
        F::store(out, j, WSum<F>::finish(acc, dtype_in));
    }
}

// Top g variables: out[j] = sum_{h < 2^g} w[h] * in[h * n_out + j].
template <class F>
__global__ void __launch_bounds__(kThreads)
    fix_high_sum(const void* __restrict__ in, int dtype_in, const typename F::E* __restrict__ w, uint32_t g,
                 uint64_t n_out, typename F::E* __restrict__ out) {
    __shared__ typename WSum<F>::Key keys[32];
    const uint32_t H = 1u << g;
    WSum<F>::make_keys_block(w, H, keys, dtype_in);
    __syncthreads();
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n_out; j += stride) {
        typename WSum<F>::Acc acc = WSum<F>::zero();
        for (uint32_t h = 0; h < H; h++) WSum<F>::mac(acc, keys[h], in, dtype_in, (uint64_t)h * n_out + j);
        F::store(out, j, WSum<F>::finish(acc, dtype_in));
    }
}

}  // namespace dpb
