// The Walsh-Hadamard rotation of one row by one warp, shared by the packing (fq_turbo_quant.cu) and the attention (fq_turbo_attn.cu).
// Lane l holds the D/32 consecutive values starting at l*D/32.  Every stage is rounded to the tensor's dtype as the reference's eager
// ops do (kernel/wht.py:26-41).
#pragma once
#include "fq_common.cuh"

namespace fq {

// Packed 16-bit arithmetic for the butterflies.  The reference adds two values of dtype T in
// T: that is the correctly rounded sum, and so is rn_T(fp32 sum) because rounding first to 24
// and then to 11 (or 8) bits is innocuous when 24 >= 2*11 + 2; the packed add is the same
// correctly rounded sum, two values per instruction and no conversions.
template <typename T> struct Pk2;
template <> struct Pk2<__half> {
    using type = __half2;
    __device__ static type make(float a, float b) { return __floats2half2_rn(a, b); }
    __device__ static float2 unpack(type x) { return __half22float2(x); }
};
template <> struct Pk2<__nv_bfloat16> {
    using type = __nv_bfloat162;
    __device__ static type make(float a, float b) { return __floats2bfloat162_rn(a, b); }
    __device__ static float2 unpack(type x) { return __bfloat1622float2(x); }
};
template <typename P2> __device__ __forceinline__ uint32_t p2_bits(P2 x) { return *reinterpret_cast<uint32_t*>(&x); }
template <typename P2> __device__ __forceinline__ P2 p2_from(uint32_t u) { return *reinterpret_cast<P2*>(&u); }

// In-place WHT of the row spread over the warp: v[j] is element lane*EPL + j.
template <typename T, int EPL>
__device__ __forceinline__ void wht_lanes(float (&v)[EPL], int lane, int D) {
    if constexpr (sizeof(T) == 2 && EPL >= 2) {
        using P2 = typename Pk2<T>::type;
        constexpr int NP = EPL / 2;
        P2 x[NP];
#pragma unroll
        for (int i = 0; i < NP; ++i) x[i] = Pk2<T>::make(v[2 * i], v[2 * i + 1]);      // exact: the values are T already
        // stride 1: (a, b) -> (a + b, a - b)
#pragma unroll
        for (int i = 0; i < NP; ++i) {
            const uint32_t u = p2_bits(x[i]);
            const P2 aa = p2_from<P2>(__byte_perm(u, u, 0x1010));                         // (a, a)
            const P2 bm = p2_from<P2>(__byte_perm(u, u, 0x3232) ^ 0x80000000u);           // (b, -b)
            x[i] = __hadd2(aa, bm);
        }
        // strides 2 .. EPL/2: whole registers
#pragma unroll
        for (int h = 1; h < NP; h <<= 1) {
#pragma unroll
            for (int i = 0; i < NP; ++i) {
                if ((i & h) == 0) {
                    const P2 a = x[i], b = x[i + h];
                    x[i] = __hadd2(a, b);
                    x[i + h] = __hsub2(a, b);
                }
            }
        }
        // strides >= EPL: partner lane; the upper lane of a pair computes other - mine
        for (int h = EPL; h < D; h <<= 1) {
            const int lo = h / EPL;
            const uint32_t flip = (lane & lo) ? 0x80008000u : 0u;
#pragma unroll
            for (int i = 0; i < NP; ++i) {
                const uint32_t mine = p2_bits(x[i]);
                const uint32_t other = __shfl_xor_sync(0xffffffffu, mine, lo);
                x[i] = __hadd2(p2_from<P2>(other), p2_from<P2>(mine ^ flip));
            }
        }
        const float cd = (float)sqrt((double)D);
#pragma unroll
        for (int i = 0; i < NP; ++i) {
            const float2 f = Pk2<T>::unpack(x[i]);
            v[2 * i] = Dt<T>::rn(__fdiv_rn(f.x, cd));
            v[2 * i + 1] = Dt<T>::rn(__fdiv_rn(f.y, cd));
        }
    } else {
#pragma unroll
    for (int h = 1; h < EPL; h <<= 1) {
#pragma unroll
        for (int j = 0; j < EPL; ++j) {
            if ((j & h) == 0) {
                const float a = v[j], b = v[j + h];
                v[j] = Dt<T>::rn(__fadd_rn(a, b));
                v[j + h] = Dt<T>::rn(__fsub_rn(a, b));
            }
        }
    }
    for (int h = EPL; h < D; h <<= 1) {
        const int lo = h / EPL;                 // partner lane distance
        const bool upper = (lane & lo) != 0;    // this lane holds the "b" half of the pair
#pragma unroll
        for (int j = 0; j < EPL; ++j) {
            const float other = __shfl_xor_sync(0xffffffffu, v[j], lo);
            v[j] = upper ? Dt<T>::rn(__fsub_rn(other, v[j])) : Dt<T>::rn(__fadd_rn(v[j], other));
        }
    }
    const float cd = (float)sqrt((double)D);    // the divisor the reference uses: fp32(math.sqrt(D))
#pragma unroll
    for (int j = 0; j < EPL; ++j) v[j] = Dt<T>::rn(__fdiv_rn(v[j], cd));
    }
}

template <typename T, int EPL>
__device__ __forceinline__ void load_row(const T* row, int lane, int D, float (&v)[EPL]) {
    if constexpr (EPL == 4 && sizeof(T) == 2) {
        // four 16-bit values of a lane in one 8-byte load when the row allows it
        if ((reinterpret_cast<uintptr_t>(row) & 7) == 0 && D == 128) {
            const uint2 u = *reinterpret_cast<const uint2*>(row + 4 * lane);
            const T* e = reinterpret_cast<const T*>(&u);
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = Dt<T>::to_f32(e[j]);
            return;
        }
    }
#pragma unroll
    for (int j = 0; j < EPL; ++j) {
        const int i = lane * EPL + j;
        v[j] = i < D ? Dt<T>::to_f32(row[i]) : 0.f;
    }
}

}  // namespace fq
