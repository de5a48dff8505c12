// Einsum axis fixing: contract the OUTER axes of an integer tensor against
// per-axis eq weights, keep the stacked and contracted axes
// (FixedAxesMapping::mles_from_tensor, zkml/src/layers/einsum/axis.rs:1142-1234).
//
//   out[q] = sum_o W[o] * T[kept_off(q) + outer_off[o]],   W[o] = prod_a w_a[o_a]
//
// The tensor stays in its native form (signed 64-bit quantised values, 8 bytes
// per entry instead of a 32-byte field element).  A term of the sum is
// (integer) * (field element): the products are added up as plain integers
// (16 wide multiply-adds per term for BN254, 4 for Goldilocks, no reduction) and
// reduced once per output; a negative entry adds its magnitude times the
// negated weight.
#pragma once
#include "family.cuh"
#include "gl_words.cuh"
#include "sumcheck_kernels.cuh"

namespace dpb {

constexpr int kMaxEinsumRank = 8;

struct EinsumKept {
    uint32_t n_kept;
    uint64_t dim[kMaxEinsumRank];     // kept axes, outermost first
    uint64_t stride[kMaxEinsumRank];  // their strides in the tensor (entries)
};

template <class F>
struct EinsumAcc;
template <>
struct EinsumAcc<FrFam> {
    FrIntAcc a;
    __device__ __forceinline__ void zero() { a = fr_intacc_zero(); }
    __device__ __forceinline__ void mac(const Fr& w, int64_t x) { fr_intacc_mac(a, w, x); }
    __device__ __forceinline__ Fr finish() const { return fr_intacc_finish(a); }
};
template <>
struct EinsumAcc<GlFam> {
    glw::A8 s0, s1;
    __device__ __forceinline__ void zero() { s0 = s1 = glw::acc_zero(); }
    __device__ __forceinline__ void mac(const Gl2& w, int64_t x) {
        const uint64_t mag = x < 0 ? (uint64_t)0 - (uint64_t)x : (uint64_t)x;
        const uint64_t c0 = x < 0 ? gl_neg(w.c0) : w.c0, c1 = x < 0 ? gl_neg(w.c1) : w.c1;
        const glw::W m = glw::make_w((uint32_t)mag, (uint32_t)(mag >> 32));
        glw::acc_mac(s0, m, glw::make_w((uint32_t)c0, (uint32_t)(c0 >> 32)));
        glw::acc_mac(s1, m, glw::make_w((uint32_t)c1, (uint32_t)(c1 >> 32)));
    }
    __device__ __forceinline__ Gl2 finish() const {
        return gl2_make(glw::to_u64(glw::canon(glw::acc_reduce(s0))), glw::to_u64(glw::canon(glw::acc_reduce(s1))));
    }
};

// W[o] = prod over outer axes of w_a[coordinate of o on axis a]; o is the flat
// row-major index over the outer axes.
template <class F>
__global__ void einsum_outer_weights(const typename F::E* const* __restrict__ w, const uint64_t* __restrict__ dims,
                                     uint32_t n_outer, uint64_t n, typename F::E* __restrict__ out) {
    typedef typename F::E E;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t o = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; o < n; o += stride) {
        uint64_t rem = o;
        E acc = F::one();
        for (int a = (int)n_outer - 1; a >= 0; a--) {
            const uint64_t c = rem % dims[a];
            rem /= dims[a];
            acc = F::mul(acc, w[a][c]);
        }
        F::store(out, o, acc);
    }
}

__device__ __forceinline__ uint64_t einsum_kept_offset(const EinsumKept& k, uint64_t q) {
    uint64_t off = 0;
    for (int a = (int)k.n_kept - 1; a >= 0; a--) {
        off += (q % k.dim[a]) * k.stride[a];
        q /= k.dim[a];
    }
    return off;
}

// The sum over the outer index of one output, cut over threads.  Two layouts, chosen by the innermost tensor axis so
// that neighbouring threads read neighbouring entries:
//  * kept (einsum_contract_lanes): a warp's lanes are 32 outputs, the block's warps and blockIdx.y share the outer index;
//  * outer (einsum_contract_strided): the threads of a group (a warp, or the whole block for long sums) stride over the
//    outer index of one output.
// A dense layer's tensors have few outputs and long sums, so one thread (or warp) per output left most of the GPU idle
// behind serial chains: x[512, 768] by rows 186 us with 768 threads, W[768, 3072] by columns 63 us with 768 warps;
// 11.7 + 2.3 and 26.5 us since (BN254).
// Output entry q = s * C + c lands at out[s * c_pad + c]; the pad is zeroed by the caller.  With gridDim.y > 1 slice y
// of the outer index writes part[y * n_out + q] instead (einsum_add_parts adds them up).
constexpr uint32_t kEinsumLaneWarps = 16;
template <class F>
__global__ void __launch_bounds__(32 * kEinsumLaneWarps)
    einsum_contract_lanes(const int64_t* __restrict__ t, EinsumKept kept, const uint64_t* __restrict__ outer_off,
                          const typename F::E* __restrict__ w, uint64_t n_outer, uint64_t n_out, uint64_t c_size,
                          uint64_t c_pad, typename F::E* __restrict__ out, typename F::E* __restrict__ part) {
    typedef typename F::E E;
    __shared__ E sh[kEinsumLaneWarps][32];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const uint64_t slice = (n_outer + gridDim.y - 1) / gridDim.y;
    const uint64_t begin = blockIdx.y * slice, end = begin + slice < n_outer ? begin + slice : n_outer;
    for (uint64_t q0 = (uint64_t)blockIdx.x * 32; q0 < n_out; q0 += (uint64_t)gridDim.x * 32) {
        const uint64_t q = q0 + lane;
        EinsumAcc<F> acc;
        acc.zero();
        if (q < n_out) {
            const uint64_t base = einsum_kept_offset(kept, q);
            for (uint64_t o = begin + warp; o < end; o += 4 * (uint64_t)warps) {
                int64_t x[4];  // four loads in flight
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const uint64_t ou = o + (uint64_t)u * warps;
                    x[u] = ou < end ? t[base + outer_off[ou]] : 0;
                }
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const uint64_t ou = o + (uint64_t)u * warps;
                    if (ou < end) acc.mac(F::load(w, F::kChalDtype, ou), x[u]);
                }
            }
        }
        E v = acc.finish();
        for (uint32_t half = warps >> 1; half > 0; half >>= 1) {
            if (warp >= half && warp < 2 * half) sh[warp][lane] = v;
            __syncthreads();
            if (warp < half) v = F::add(v, sh[warp + half][lane]);
            __syncthreads();
        }
        if (warp == 0 && q < n_out) {
            if (gridDim.y > 1) F::store(part, blockIdx.y * n_out + q, v);
            else F::store(out, (q / c_size) * c_pad + (q % c_size), v);
        }
    }
}

template <class F>
__global__ void __launch_bounds__(kThreads)
    einsum_add_parts(const typename F::E* __restrict__ part, uint32_t slices, uint64_t n_out, uint64_t c_size, uint64_t c_pad,
                     typename F::E* __restrict__ out) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t q = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n_out; q += stride) {
        typename F::E v = part[q];
        for (uint32_t s = 1; s < slices; s++) v = F::add(v, part[s * n_out + q]);
        F::store(out, (q / c_size) * c_pad + (q % c_size), v);
    }
}

// group: 32 or blockDim.x threads per output
template <class F>
__global__ void __launch_bounds__(kThreads)
    einsum_contract_strided(const int64_t* __restrict__ t, EinsumKept kept, const uint64_t* __restrict__ outer_off,
                            const typename F::E* __restrict__ w, uint64_t n_outer, uint64_t n_out, uint64_t c_size,
                            uint64_t c_pad, uint32_t group, typename F::E* __restrict__ out) {
    typedef typename F::E E;
    const uint32_t in_group = threadIdx.x % group, groups = blockDim.x / group;
    const uint64_t n_groups = (uint64_t)gridDim.x * groups;
    for (uint64_t q = (uint64_t)blockIdx.x * groups + threadIdx.x / group; q < n_out; q += n_groups) {
        const uint64_t base = einsum_kept_offset(kept, q);
        EinsumAcc<F> part;
        part.zero();
        for (uint64_t o = in_group; o < n_outer; o += 4 * (uint64_t)group) {
            int64_t x[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const uint64_t ou = o + (uint64_t)u * group;
                x[u] = ou < n_outer ? t[base + outer_off[ou]] : 0;
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const uint64_t ou = o + (uint64_t)u * group;
                if (ou < n_outer) part.mac(F::load(w, F::kChalDtype, ou), x[u]);
            }
        }
        E acc[1] = {part.finish()};
        if (group == 32) {
            for (int off = 16; off > 0; off >>= 1) acc[0] = F::add(acc[0], F::shfl_down(acc[0], off));
        } else {
            block_sum<F, 1>(acc);  // the whole block works on output q
        }
        if (in_group == 0) F::store(out, (q / c_size) * c_pad + (q % c_size), acc[0]);
    }
}

}  // namespace dpb
