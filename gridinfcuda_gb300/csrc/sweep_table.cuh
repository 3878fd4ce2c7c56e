// sweep_table.cuh -- the checkerboard half-sweep for tables the linear update
// does not cover (4-byte arithmetic): the reference's O(L^2) rule for explicit
// and truncated-quadratic tables (src/bp.cc:55-62) and the standard rule's
// min-convolution.
//
//   reference   out(i) = min_j V(i,j) + from(j), one vector a node, sent in all
//               four directions as it is
//   standard    out(i) = min_j V(i,j) + h(j), h = from - in[dir], one a
//               message, then the mean (or the minimum) subtracted
//
// A min-convolution is a matrix product over (min, +): V (L x L) times the
// tile's L x 16 (reference) or L x 64 (standard) vectors.  A block of 128
// threads holds V in shared memory for all its tiles (16 nodes each) and gives
// every thread TI outputs of TN vectors in registers, so that four steps of j
// read TI floats of V and four of each vector from shared memory for
// 4 TI TN additions and minima.  Additions go two outputs to an instruction
// (add.rn.f32x2, rounded as the scalar one) and minima two steps of j to one
// (three-input minimum).  TI and TN follow L so that the 128 threads have one
// group of outputs each or nearly so (launch_table).  The lane-per-message
// form this replaces read V through the cache once per addition and kept the
// standard rule's vectors in local memory.
//
// Bound: HBM (36 B per updated node and label) for the reference rule and up
// to about 64 labels of the standard rule, then the instruction issue rate.
// Measured, 640x480 FP32, us per half-sweep, before -> now:
//   TABLE_MEASURED
//
// Exactness.  The reference takes (a < b) ? a : b in order of j.  On operands
// that are neither NaN nor a zero of either sign against the other, the
// hardware minimum gives the same value in any order.  A candidate can be -0
// only if its table entry is, and NaN only if an operand is NaN or the two
// are opposite infinities.  So a table with a -0, a -infinity or a NaN, and a
// tile in which a belief is not above -kTableBig or, for the standard rule's
// difference, a message not within +-kTableBig, run the sequential form
// (messages_ref_minconv, message_std_minconv) instead.
#pragma once

#include "sweep_impl.cuh"

namespace ginf_gpu {

constexpr int kTableWarps = 4, kTableSplit = 2, kTableNodes = kTableWarps / kTableSplit * 8;
constexpr int kTableThreads = kTableWarps * 32;
constexpr float kTableBig = 1e38f;
constexpr int kTableMaxGroups = 16;  // output groups per vector: Lp / TI

// Four consecutive elements of shared memory.
template <typename M, typename T>
__device__ __forceinline__ void load4(const unsigned char *p, T *o) {
    if constexpr (sizeof(M) == 2) {
        const uint2 v = *reinterpret_cast<const uint2 *>(p);
        __half2 a, b;
        *reinterpret_cast<uint32_t *>(&a) = v.x;
        *reinterpret_cast<uint32_t *>(&b) = v.y;
        const float2 fa = __half22float2(a), fb = __half22float2(b);
        o[0] = fa.x; o[1] = fa.y; o[2] = fb.x; o[3] = fb.y;
    } else {
        MIO<M, T>::load(p, o);
    }
}
template <typename M, typename T>
__device__ __forceinline__ void store4(unsigned char *p, const T *o) {
    if constexpr (sizeof(M) == 2) {
        const __half2 a = __floats2half2_rn(o[0], o[1]), b = __floats2half2_rn(o[2], o[3]);
        *reinterpret_cast<uint2 *>(p) =
            make_uint2(*reinterpret_cast<const uint32_t *>(&a), *reinterpret_cast<const uint32_t *>(&b));
    } else {
        MIO<M, T>::store(p, o);
    }
}

// acc(i) = min(acc(i), v0(i) + h0, v1(i) + h1) for TI outputs.
template <int TI>
__device__ __forceinline__ void table_step2(float *acc, const float *v0, float h0, const float *v1, float h1) {
#pragma unroll
    for (int i = 0; i < TI; i += 2) {
        const float2 a = add_f32x2(v0[i], v0[i + 1], h0, h0), b = add_f32x2(v1[i], v1[i + 1], h1, h1);
        acc[i] = min3_f32(acc[i], a.x, b.x);
        acc[i + 1] = min3_f32(acc[i + 1], a.y, b.y);
    }
}
template <int TI>
__device__ __forceinline__ void table_step2(int *acc, const int *v0, int h0, const int *v1, int h1) {
#pragma unroll
    for (int i = 0; i < TI; ++i) acc[i] = min(min(acc[i], v0[i] + h0), v1[i] + h1);
}
template <int TI>
__device__ __forceinline__ void table_step1(float *acc, const float *v, float h) {
#pragma unroll
    for (int i = 0; i < TI; ++i) acc[i] = fminf(acc[i], v[i] + h);
}
template <int TI>
__device__ __forceinline__ void table_step1(int *acc, const int *v, int h) {
#pragma unroll
    for (int i = 0; i < TI; ++i) acc[i] = min(acc[i], v[i] + h);
}

// The belief of one node by its four lanes, as belief_part, noting values the
// fast form does not cover.
template <typename T, typename M, bool STD>
__device__ __forceinline__ void table_belief(const SweepParams &p, unsigned char *slot, int L, int dir, T &best,
                                             int &bl, int &odd) {
    const unsigned char *mb = slot + p.d_bytes;
#pragma unroll 2
    for (int c = dir * 4; c < L; c += 16) {
        T v[4], a[4];
        load_t<T, 4>(slot + c * sizeof(T), v);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            load4<M, T>(mb + e * p.m_bytes + c * sizeof(M), a);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                v[k] = v[k] + a[k];
                if constexpr (STD && std::is_same<T, float>::value)
                    if (c + k < L && !(fabsf(a[k]) < kTableBig)) odd = 1;
            }
        }
        store_t<T, 4>(slot + c * sizeof(T), v);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (c + k < L) {
                if constexpr (std::is_same<T, float>::value)
                    if (!(v[k] > -kTableBig)) odd = 1;
                if (bl == 0x7fffffff || v[k] < best) {
                    best = v[k];
                    bl = c + k;
                }
            }
        }
    }
}

// The tile's min-convolutions, fast form.  Vs is V with rows of Lp outputs
// (Vs[j * Lp + i] = V(i, j)).  Vector m is node m (reference: the output goes
// to the node's first message slot) or message (node m / 4, direction m % 4)
// (standard: in place, which is why a round's reads end before its writes).
template <typename T, typename M, bool STD, int TI, int TN>
__device__ __forceinline__ void table_convolve(const SweepParams &p, const T *Vs, unsigned char *smem, int L,
                                               T (*mins)[kTableMaxGroups]) {
    constexpr int NV = STD ? 4 * kTableNodes : kTableNodes;
    const int groups = p.Lp / TI;
    const int per_round = kTableThreads / groups;
    const int ig = (int)threadIdx.x % groups, mine = (int)threadIdx.x / groups;
    for (int m0 = 0; m0 < NV; m0 += per_round * TN) {
        const int mb = m0 + mine * TN;
        const bool on = mine < per_round && mb < NV;
        T acc[TN][TI];
        if (on) {
            const unsigned char *sl[TN], *in[TN];
#pragma unroll
            for (int u = 0; u < TN; ++u) {
                sl[u] = smem + (size_t)(STD ? (mb + u) / 4 : mb + u) * p.slot_bytes;
                in[u] = sl[u] + p.d_bytes + (STD ? (mb + u) % 4 : 0) * p.m_bytes;
            }
#pragma unroll
            for (int u = 0; u < TN; ++u)
#pragma unroll
                for (int i = 0; i < TI; ++i) acc[u][i] = pos_inf<T>();
            const T *vp = Vs + ig * TI;
            // Four steps of j; rows past L are never read.
#pragma unroll 1
            for (int j = 0; j < L; j += 4) {
                T h[TN][4];
#pragma unroll
                for (int u = 0; u < TN; ++u) {
                    load_t<T, 4>(sl[u] + j * sizeof(T), h[u]);
                    if constexpr (STD) {
                        T a[4];
                        load4<M, T>(in[u] + j * sizeof(M), a);
#pragma unroll
                        for (int k = 0; k < 4; ++k) h[u][k] = h[u][k] - a[k];
                    }
                }
#pragma unroll
                for (int k = 0; k < 4; k += 2) {
                    T v0[TI], v1[TI];
                    if (j + k + 1 < L) {
                        load_t<T, TI>(reinterpret_cast<const unsigned char *>(vp + (size_t)(j + k) * p.Lp), v0);
                        load_t<T, TI>(reinterpret_cast<const unsigned char *>(vp + (size_t)(j + k + 1) * p.Lp), v1);
#pragma unroll
                        for (int u = 0; u < TN; ++u) table_step2<TI>(acc[u], v0, h[u][k], v1, h[u][k + 1]);
                    } else if (j + k < L) {
                        load_t<T, TI>(reinterpret_cast<const unsigned char *>(vp + (size_t)(j + k) * p.Lp), v0);
#pragma unroll
                        for (int u = 0; u < TN; ++u) table_step1<TI>(acc[u], v0, h[u][k]);
                    }
                }
            }
        }
        if constexpr (STD && sizeof(M) == 2) {
            // FP16 messages leave rounded once, the minimum already subtracted.
            if (on) {
#pragma unroll
                for (int u = 0; u < TN; ++u) {
                    T m = pos_inf<T>();
#pragma unroll
                    for (int i = 0; i < TI; ++i)
                        if (ig * TI + i < L) m = fminf(m, acc[u][i]);
                    mins[mb + u][ig] = m;
                }
            }
        }
        if constexpr (STD) __syncthreads();
        if (on) {
#pragma unroll
            for (int u = 0; u < TN; ++u) {
                T shift = T(0);
                if constexpr (STD && sizeof(M) == 2) {
                    shift = mins[mb + u][0];
                    for (int g = 1; g < groups; ++g) shift = fminf(shift, mins[mb + u][g]);
                }
                unsigned char *out = smem + (size_t)(STD ? (mb + u) / 4 : mb + u) * p.slot_bytes + p.d_bytes +
                                     (STD ? (mb + u) % 4 : 0) * p.m_bytes + (size_t)ig * TI * sizeof(M);
#pragma unroll
                for (int i = 0; i < TI; i += 4) {
                    T r[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        r[k] = ig * TI + i + k < L ? acc[u][i + k] : T(0);
                        if constexpr (STD && sizeof(M) == 2) r[k] = ig * TI + i + k < L ? r[k] - shift : T(0);
                    }
                    store4<M, T>(out + i * sizeof(M), r);
                }
            }
        }
    }
}

// Subtracts the mean (summed in label order, as the reference does) or the
// minimum from one message of the arithmetic type, in place.
template <typename T>
__device__ __forceinline__ void table_normalise(unsigned char *md, int L, int norm_min) {
    T val;
    if (norm_min) {
        val = *reinterpret_cast<const T *>(md);
        for (int c = 0; c < L; c += 4) {
            T r[4];
            MIO<T, T>::load(md + c * sizeof(T), r);
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (c + k < L) val = rmin(val, r[k]);
        }
    } else {
        val = T(0);
        for (int c = 0; c < L; c += 4) {
            T r[4];
            MIO<T, T>::load(md + c * sizeof(T), r);
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (c + k < L) val += r[k];
        }
        val = div_labels(val, L);
    }
    for (int c = 0; c < L; c += 4) {
        T r[4];
        MIO<T, T>::load(md + c * sizeof(T), r);
#pragma unroll
        for (int k = 0; k < 4; ++k) r[k] = c + k < L ? r[k] - val : T(0);
        MIO<T, T>::store(md + c * sizeof(T), r);
    }
}

// One half-sweep.  Warps come in pairs over eight nodes: the first of a pair
// issues the copies and does what is done once a lane (k, dir) -- beliefs,
// normalisation, stores -- and all four convolve.
template <typename T, typename M, bool STD, int TI, int TN>
__global__ void __launch_bounds__(kTableThreads) sweep_kernel_table(const SweepParams p) {
    constexpr int NW = kTableWarps, SPL = kTableSplit;
    constexpr bool kF32 = std::is_same<T, float>::value;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint64_t full_bar;
    __shared__ T mins[sizeof(M) == 2 && STD ? 4 * kTableNodes : 1][kTableMaxGroups];
    launch_dependents();
    const int L = p.L;
    T *Vs = reinterpret_cast<T *>(smem + (size_t)kTableNodes * p.slot_bytes);
    int odd_table = 0;
    for (int e = threadIdx.x; e < L * p.Lp; e += blockDim.x) {
        const int j = e / p.Lp, i = e - j * p.Lp;
        const T v = i < L ? __ldg(static_cast<const T *>(p.V) + i + (size_t)L * j) : T(0);
        Vs[e] = v;
        if constexpr (kF32)
            if (!(v > -pos_inf<float>()) || __float_as_uint(v) == 0x80000000u) odd_table = 1;
    }
    if (threadIdx.x == 0) {
        mbar_init(&full_bar, NW * 32);
        fence_barrier_init();
    }
    odd_table = __syncthreads_or(odd_table);
    grid_dependency_wait();
    const int dir = (threadIdx.x & 31) >> 3;
    const int node = ((threadIdx.x >> 5) / SPL) * 8 + (threadIdx.x & 7);
    const bool lead = ((threadIdx.x >> 5) % SPL) == 0;
    unsigned char *slot = smem + (size_t)node * p.slot_bytes;
    unsigned char *md = slot + p.d_bytes + dir * p.m_bytes;
    int t = blockIdx.x;
    if (t < p.num_tiles) tile_load<NW, SPL>(p, t, smem, &full_bar);
    uint32_t parity = 0;
    for (; t < p.num_tiles; t += gridDim.x) {
        const bool got = mbar_wait_bounded(&full_bar, parity, p.status);
        parity ^= 1u;
        if (!__syncthreads_and(got)) return;
        int x, y;
        const bool act = tile_node<NW, SPL>(p, t, x, y) && lead;
        if (act && ((zero_mask(p, x, y) >> dir) & 1u)) zero_bytes(md, p.m_bytes);
        __syncwarp();
        T best = pos_inf<T>();
        int label = 0x7fffffff, odd = 0;
        if (act) table_belief<T, M, STD>(p, slot, L, dir, best, label, odd);
        argmin_combine(best, label);
        // The beliefs are complete, and the block agrees on the form.
        const bool slow = __syncthreads_or(odd | odd_table) != 0;
        if (kF32 && slow) {  // int32 minima have one value
            if constexpr (kF32) {
                if (act) {
                    if constexpr (STD) message_std_minconv<T, M, kMaxLabels>(p, slot, L, dir);
                    else messages_ref_minconv<T, M, kMaxLabels>(p, slot, L, dir);
                }
            }
        } else {
            table_convolve<T, M, STD, TI, TN>(p, Vs, smem, L, mins);
            if constexpr (STD && sizeof(M) == sizeof(T)) {
                __syncthreads();
                if (act) table_normalise<T>(md, L, p.norm_min);
            }
        }
        fence_proxy_async_shared();
        __syncthreads();
        if (act) {
            if (dir == 0 && p.write_labels) p.labels[(size_t)y * p.W + x] = label;
            const int qx = x + dir_dx(dir), qy = y + dir_dy(dir);
            unsigned char *dst = p.rec + ((size_t)qy * p.W + qx) * p.rec_bytes + p.d_bytes + opp_dir(dir) * p.m_bytes;
            // The reference rule's one vector lies in the first slot.
            bulk_store(dst, STD ? md : slot + p.d_bytes, p.m_bytes);
            bulk_commit();
            bulk_wait_read_all();
        }
        __syncthreads();
        const int tn = t + gridDim.x;
        if (tn < p.num_tiles) tile_load<NW, SPL>(p, tn, smem, &full_bar);
    }
    bulk_wait_all();
}

template <typename T, typename M, bool STD, int TI, int TN>
cudaError_t launch_table_t(const RecordFormat &f, const SweepParams &p, cudaStream_t s, int num_sms) {
    static LaunchCache cache;
    return launch_tiles(sweep_kernel_table<T, M, STD, TI, TN>, cache, kTableWarps, kTableNodes, p, f.slot_bytes, s,
                        num_sms, (size_t)f.L * f.Lp * sizeof(T));
}

// Outputs per thread: 128 threads cover L / TI groups of 16 / TN (reference)
// or 64 / TN (standard) vectors in one round at the powers of two; between
// them some threads idle or a second round runs.
template <typename T, typename M>
cudaError_t launch_table(const RecordFormat &f, const SweepParams &p, cudaStream_t s, int num_sms) {
    if (p.mode == MODE_REF_MINCONV) {
        if (f.L <= 32) return launch_table_t<T, M, false, 4, 1>(f, p, s, num_sms);
        if (f.L <= 64) return launch_table_t<T, M, false, 4, 2>(f, p, s, num_sms);
        return launch_table_t<T, M, false, 4, 4>(f, p, s, num_sms);
    }
    if (f.L <= 8) return launch_table_t<T, M, true, 4, 1>(f, p, s, num_sms);
    if (f.L <= 24) return launch_table_t<T, M, true, 4, 2>(f, p, s, num_sms);
    if (f.L <= 32) return launch_table_t<T, M, true, 4, 4>(f, p, s, num_sms);
    if (f.L <= 64) return launch_table_t<T, M, true, 8, 4>(f, p, s, num_sms);
    return launch_table_t<T, M, true, 8, 8>(f, p, s, num_sms);
}

}  // namespace ginf_gpu
