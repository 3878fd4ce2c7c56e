// sweep_labels.cuh -- a node's label from its belief, by four lanes (the
// labels-only half-sweeps of sweep_labels.cu and batch.cu).
#pragma once

#include "sweep_impl.cuh"

namespace ginf_gpu {

// Chunks g, g + 4, ... of B labels from `begin` below `end`.
template <typename T, typename M>
__device__ __forceinline__ void label_part(const unsigned char *r, const SweepParams &p, unsigned zero, int begin,
                                           int end, int g, T &best, int &bl) {
    constexpr int B = MIO<M, T>::B;
    const unsigned char *mb = r + p.d_bytes;
#pragma unroll 2
    for (int c = begin + g * B; c < end; c += 4 * B) {
        T v[B], a[4][B];
        load_t<T, B>(r + c * sizeof(T), v);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            if ((zero >> e) & 1u) {
#pragma unroll
                for (int k = 0; k < B; ++k) a[e][k] = T(0);
            } else {
                MIO<M, T>::load(mb + e * p.m_bytes + c * sizeof(M), a[e]);
            }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int k = 0; k < B; ++k) v[k] = v[k] + a[e][k];
#pragma unroll
        for (int k = 0; k < B; ++k) {
            if (c + k < end && (bl == 0x7fffffff || v[k] < best)) {
                best = v[k];
                bl = c + k;
            }
        }
    }
}

// argmin_combine over lanes 4n .. 4n + 3.
template <typename T>
__device__ __forceinline__ void combine4(T &best, int &bl) {
#pragma unroll
    for (int off = 1; off <= 2; off <<= 1) {
        const T ob = __shfl_xor_sync(0xffffffffu, best, off);
        const int ol = __shfl_xor_sync(0xffffffffu, bl, off);
        if (ol != 0x7fffffff && (bl == 0x7fffffff || ob < best || (!(best < ob) && ol < bl))) {
            best = ob;
            bl = ol;
        }
    }
}

}  // namespace ginf_gpu
