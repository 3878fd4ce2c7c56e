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
// tile's L x 16 (reference) or L x 64 (standard) vectors.  A block
// holds V in shared memory for all its tiles (16 nodes each) and gives
// every thread TI outputs of TN vectors in registers, so that four steps of j
// read 4 TI entries of V and four of each vector from shared memory for
// 4 TI TN additions and minima.  Additions and minima go two steps of j to an
// instruction (add.rn.f32x2, rounded as the scalar one; three-input minimum).
// TI and TN follow L so that the block's threads have one group of outputs each
// or nearly so (launch_table).  The lane-per-message form this replaces read V
// through the cache once per addition and kept the standard rule's vectors in
// local memory.
//
// Bound: HBM (36 B per updated node and label) for the reference rule up to
// about 32 labels; above that the latency of a tile's phases with the few
// blocks that the table leaves room for, and for the standard rule the issue
// rate (at L = 64, 12.5 T additions and as many minima a second).  Measured, 640x480
// FP32, us per half-sweep, lane-per-message form -> this one:
//   L           16         32         64          128
//   reference   52 -> 24   146 -> 37  727 -> 85   - -> 256
//   standard    127 -> 39  697 -> 75  3866 -> 200 - -> 720
// (the reference rule at L = 32 33 since launches wait for the last one's blocks
// to go, sweep_impl.cuh).
// Also measured for the standard rule at L = 64: four warps of 8 x 4 outputs
// 237, two of 8 x 8 with the additions paired along i 197 (the reference rule,
// whose vectors need no subtraction, is faster paired along j).
//
// Exactness.  The reference takes (a < b) ? a : b in order of j.  On operands
// that are neither NaN nor a zero of either sign against the other, the
// hardware minimum gives the same value in any order.  A candidate can be -0
// only if its table entry is, and NaN only if an operand is NaN or the two
// are opposite infinities.  So a table with a -0, a -infinity or a NaN, and a
// tile in which a belief is not above -kTableBig or, for the standard rule's
// difference, a message not within +-kTableBig, take the reference's comparison
// in its order instead.  A hand-made table may well hold a -0.  320x240, six
// half-sweeps, us: a lane per output or message with V through the cache and the
// standard rule's vectors in local memory -> eight (four) outputs side by side
// with V from shared memory (ordinary tables):
//   L           16         32                64                   128
//   reference   165 (112)  315 (125)         900 (207)            12520 -> 1655 (500)
//   standard    254 (131)  1366 -> 274 (171) 10830 -> 1170 (385)  111700 -> 9820 (1090)
// Where no second figure stands the first form is still the one (as a kernel
// without V in shared memory it took 175 and 355 us for the reference rule at 16
// and 32 labels, 1450 at 64, 6250 at 128, and 315, 1190, 5900 and 67300 for the
// standard one), since the blocked form beside table_convolve costs ordinary
// tables up to 1 %.  table_convolve itself with these comparisons took 1970 us at
// 128 labels, but ordinary tables then 1245 us for 1155 (640x480, L = 64).
#pragma once

#include "sweep_impl.cuh"

namespace ginf_gpu {

constexpr int kTableNodes = 16;  // nodes per tile
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
// Two consecutive elements.
template <typename M, typename T>
__device__ __forceinline__ void store2(unsigned char *p, T a, T b) {
    if constexpr (sizeof(M) == 2) {
        const __half2 h = __floats2half2_rn(a, b);
        *reinterpret_cast<uint32_t *>(p) = *reinterpret_cast<const uint32_t *>(&h);
    } else if constexpr (std::is_same<T, int>::value) {
        *reinterpret_cast<int2 *>(p) = make_int2(a, b);
    } else {
        *reinterpret_cast<float2 *>(p) = make_float2(a, b);
    }
}

// Steps j and j + 1 of one output: acc = min(acc, v0 + h0, v1 + h1).
__device__ __forceinline__ float table_step(float acc, float v0, float v1, float h0, float h1) {
    const float2 t = add_f32x2(v0, v1, h0, h1);
    return min3_f32(acc, t.x, t.y);
}
__device__ __forceinline__ int table_step(int acc, int v0, int v1, int h0, int h1) {
    return min(min(acc, v0 + h0), v1 + h1);
}
__device__ __forceinline__ void sub4(float *h, const float *a) {
    const float2 x = sub_f32x2(h[0], h[1], a[0], a[1]), y = sub_f32x2(h[2], h[3], a[2], a[3]);
    h[0] = x.x; h[1] = x.y; h[2] = y.x; h[3] = y.y;
}
__device__ __forceinline__ void sub4(int *h, const int *a) {
#pragma unroll
    for (int k = 0; k < 4; ++k) h[k] -= a[k];
}
__device__ __forceinline__ float table_min(float a, float b) { return fminf(a, b); }
__device__ __forceinline__ int table_min(int a, int b) { return min(a, b); }

// The belief of one node by its four lanes, as belief_part (in chunks of four
// labels whatever the store: with FP16 messages' chunks of eight L = 8 took 226 us
// for six half-sweeps at 640x480, so 209), noting values the fast form does not
// cover.
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

// The label of a node by its four lanes from its finished belief, in belief_part's
// chunks.  With a NaN among them the chunks decide the label.
template <typename T, typename M>
__device__ __forceinline__ void table_label(const unsigned char *slot, int L, int dir, T &best, int &bl) {
    constexpr int B = MIO<M, T>::B;
    best = pos_inf<T>();
    bl = 0x7fffffff;
    for (int c = dir * B; c < L; c += 4 * B)
        for (int i = c; i < c + B && i < L; ++i) {
            const T v = reinterpret_cast<const T *>(slot)[i];
            if (bl == 0x7fffffff || v < best) {
                best = v;
                bl = i;
            }
        }
}

// The tile's min-convolutions, fast form.  Vs holds V with the steps of j in
// pairs: V(i, j) at ((j / 2) Lp + i) 2 + j % 2, so that a 16-byte load brings
// two outputs' entries for j and j + 1, each pair an operand of one packed
// addition with the pair h(j), h(j + 1) as it lies in the node's slot.  Vector
// m is node m (reference: the output goes to the node's first message slot) or
// message (node m / 4, direction m % 4) (standard: in place, which is why the
// block's reads end before its writes).  Thread (ig, mb / TN) has the outputs
// 2 (ig + c groups), + 1, c < TI / 2, of the vectors mb .. mb + TN - 1: eight
// neighbouring threads read 128 consecutive bytes of V.
template <typename T, typename M, bool STD, int TI, int TN>
__device__ __forceinline__ void table_convolve(const SweepParams &p, const T *Vs, unsigned char *smem, int L,
                                               T (*mins)[kTableMaxGroups]) {
    constexpr int NV = STD ? 4 * kTableNodes : kTableNodes;
    const int groups = p.Lp / TI;
    const int ig = (int)threadIdx.x % groups, mb = (int)threadIdx.x / groups * TN;
    const bool on = mb < NV;
    T acc[TN][TI];
    if (on) {
        const unsigned char *sl[TN], *in[TN];
#pragma unroll
        for (int u = 0; u < TN; ++u) {
            sl[u] = smem + (size_t)(STD ? (mb + u) / 4 : mb + u) * p.slot_bytes;
            in[u] = sl[u] + p.d_bytes + (STD ? (mb + u) % 4 : 0) * p.m_bytes;
#pragma unroll
            for (int i = 0; i < TI; ++i) acc[u][i] = pos_inf<T>();
        }
        const unsigned char *vp = reinterpret_cast<const unsigned char *>(Vs + ig * 4);
        const int row = 2 * p.Lp * (int)sizeof(T), chunk = 4 * groups * (int)sizeof(T);
        // h(j .. j + 3) of vector u.
        auto load_h = [&](int u, int j, T *h) {
            load_t<T, 4>(sl[u] + j * sizeof(T), h);
            if constexpr (STD) {
                T a[4];
                load4<M, T>(in[u] + j * sizeof(M), a);
                sub4(h, a);
            }
        };
        // Four steps of j at a time; the reference rule's loop has registers to
        // spare for loads ahead (L = 128: 313 us at one step per pass, 280 at four).
        const int L4 = L & ~3;
#pragma unroll(STD ? 1 : 4)
        for (int j = 0; j < L4; j += 4) {
            T h[TN][4];
#pragma unroll
            for (int u = 0; u < TN; ++u) load_h(u, j, h[u]);
#pragma unroll
            for (int k = 0; k < 4; k += 2) {
#pragma unroll
                for (int c = 0; c < TI / 2; ++c) {
                    T v[4];
                    load_t<T, 4>(vp + c * chunk, v);
#pragma unroll
                    for (int u = 0; u < TN; ++u) {
                        acc[u][2 * c] = table_step(acc[u][2 * c], v[0], v[1], h[u][k], h[u][k + 1]);
                        acc[u][2 * c + 1] = table_step(acc[u][2 * c + 1], v[2], v[3], h[u][k], h[u][k + 1]);
                    }
                }
                vp += row;
            }
        }
        if (L4 < L) {  // one to three steps more
#pragma unroll
            for (int u = 0; u < TN; ++u) {
                T h[4];
                load_h(u, L4, h);
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    if (L4 + k < L) {
#pragma unroll
                        for (int c = 0; c < TI / 2; ++c) {
                            const T *v = reinterpret_cast<const T *>(vp + (k / 2) * row + c * chunk) + (k & 1);
                            acc[u][2 * c] = table_min(acc[u][2 * c], v[0] + h[k]);
                            acc[u][2 * c + 1] = table_min(acc[u][2 * c + 1], v[2] + h[k]);
                        }
                    }
                }
            }
        }
        if constexpr (STD && sizeof(M) == 2) {
            // FP16 messages leave rounded once, the minimum already subtracted.
#pragma unroll
            for (int u = 0; u < TN; ++u) {
                T m = pos_inf<T>();
#pragma unroll
                for (int i = 0; i < TI; ++i)
                    if ((ig + i / 2 * groups) * 2 + i % 2 < L) m = fminf(m, acc[u][i]);
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
                                 (STD ? (mb + u) % 4 : 0) * p.m_bytes;
#pragma unroll
            for (int c = 0; c < TI / 2; ++c) {
                const int i0 = (ig + c * groups) * 2;
                store2<M, T>(out + i0 * sizeof(M), i0 < L ? acc[u][2 * c] - shift : T(0),
                             i0 + 1 < L ? acc[u][2 * c + 1] - shift : T(0));
            }
        }
    }
}

// Outputs i0 .. i0 + N - 1 of one vector by the reference's comparison in order
// of j, h(j) the vector; an accumulator starts at infinity, which the first
// candidate replaces whatever it is.
template <int N, typename T, typename Fn>
__device__ __forceinline__ void table_ordered(const T *Vs, int Lp, int L, int i0, Fn h, T *acc) {
#pragma unroll
    for (int i = 0; i < N; ++i) acc[i] = pos_inf<T>();
#pragma unroll 1
    for (int j = 0; j < L; j += 2) {
        const bool two = j + 1 < L;
        const T h0 = h(j), h1 = two ? h(j + 1) : T(0);
#pragma unroll
        for (int q = 0; q < N / 2; ++q) {
            T v[4];  // V(i, j), V(i, j + 1), V(i + 1, j), V(i + 1, j + 1)
            load_t<T, 4>(reinterpret_cast<const unsigned char *>(Vs + j * Lp + 2 * i0 + 4 * q), v);
            acc[2 * q] = rmin(acc[2 * q], v[0] + h0);
            acc[2 * q + 1] = rmin(acc[2 * q + 1], v[2] + h0);
            if (two) {
                acc[2 * q] = rmin(acc[2 * q], v[1] + h1);
                acc[2 * q + 1] = rmin(acc[2 * q + 1], v[3] + h1);
            }
        }
    }
}

// The lane's part of its node's messages in that form: the standard rule's
// message towards dir (4-byte messages in place, not yet normalised), the
// reference rule's outputs 4 dir, 4 dir + 16, ... into the node's first slot.  V
// is read from shared memory, each entry for a warp at once, and eight (four)
// outputs run side by side.
template <typename T, typename M, bool STD>
__device__ __forceinline__ void table_messages_ordered(const SweepParams &p, const T *Vs, unsigned char *slot, int L,
                                                       int dir) {
    if constexpr (STD) {
        unsigned char *md = slot + p.d_bytes + dir * p.m_bytes;
        T h[kMaxLabels], o[sizeof(M) == sizeof(T) ? 1 : kMaxLabels];
        load_h<T, M, kMaxLabels>(slot, md, L, h);
#pragma unroll 1
        for (int i = 0; i < L; i += 8) {
            T r[8];
            table_ordered<8>(Vs, p.Lp, L, i, [&](int j) { return h[j]; }, r);
            if constexpr (sizeof(M) == sizeof(T)) {  // normalised later
                store_t<T, 4>(md + i * sizeof(T), r);
                store_t<T, 4>(md + (i + 4) * sizeof(T), r + 4);
            } else {
#pragma unroll
                for (int k = 0; k < 8; ++k) o[i + k] = r[k];
            }
        }
        if constexpr (sizeof(M) != sizeof(T)) {
            normalise(o, L, p.norm_min);
            store_msg<T, M>(md, o, L);
        }
    } else {
        const T *fr = reinterpret_cast<const T *>(slot);
#pragma unroll 1
        for (int i = dir * 4; i < L; i += 16) {
            T r[4];
            table_ordered<4>(Vs, p.Lp, L, i, [&](int j) { return fr[j]; }, r);
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (i + k >= L) r[k] = T(0);
            unsigned char *out = slot + p.d_bytes + i * sizeof(M);
            store2<M, T>(out, r[0], r[1]);
            store2<M, T>(out + 2 * sizeof(M), r[2], r[3]);
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

// Blocks per SM the registers are allocated for: what shared memory holds at
// the kernel's largest L, or what keeps the accumulators out of local memory.
constexpr int table_blocks(bool std_rule, int spl, int outputs) {
    if (spl == 2) return 2;
    if (!std_rule) return outputs == 4 ? 18 : (outputs == 8 ? 15 : 6);
    return outputs == 8 ? 14 : (outputs == 16 ? 10 : (outputs == 32 ? 8 : 6));
}

// One half-sweep.  SPL warps serve eight nodes: the first of them issues the
// copies and does what is done once a lane (k, dir) -- beliefs, normalisation,
// stores -- and all convolve.
template <typename T, typename M, bool STD, int SPL, int TI, int TN>
__global__ void __launch_bounds__(64 * SPL, table_blocks(STD, SPL, TI * TN)) sweep_kernel_table(const SweepParams p) {
    constexpr int NW = 2 * SPL;
    constexpr bool kF32 = std::is_same<T, float>::value;
    constexpr bool kNormalise = STD && sizeof(M) == sizeof(T);
    // Label counts whose ordered form is the blocked one: where a lane per output
    // was slower beside the table in shared memory than without it (above).
    constexpr bool kBlocked = kF32 && (STD ? TN > 2 : SPL == 2);
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint64_t full_bar;
    __shared__ T mins[sizeof(M) == 2 && STD ? 4 * kTableNodes : 1][kTableMaxGroups];
    const int L = p.L;
    T *Vs = reinterpret_cast<T *>(smem + (size_t)kTableNodes * p.slot_bytes);
    int odd_table = 0;
    // Warp w stages the rows w, w + NW, ..., eight of them in flight.
    for (int j0 = (int)(threadIdx.x >> 5); j0 < L; j0 += 8 * NW)
        for (int i = (int)(threadIdx.x & 31); i < p.Lp; i += 32) {
            T v[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int j = j0 + q * NW;
                v[q] = j < L && i < L ? __ldg(static_cast<const T *>(p.V) + i + (size_t)L * j) : T(0);
            }
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int j = j0 + q * NW;
                if (j < L) Vs[((j >> 1) * p.Lp + i) * 2 + (j & 1)] = v[q];
                if constexpr (kF32)
                    if (!(v[q] > -pos_inf<float>()) || __float_as_uint(v[q]) == 0x80000000u) odd_table = 1;
            }
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
                if constexpr (sizeof(M) == 2) {
                    if (act) table_label<T, M>(slot, L, dir, best, label);
                    argmin_combine(best, label);
                }
                if (act) {
                    if constexpr (kBlocked) table_messages_ordered<T, M, STD>(p, Vs, slot, L, dir);
                    else if constexpr (STD) message_std_minconv<T, M, kMaxLabels>(p, slot, L, dir);
                    else messages_ref_minconv<T, M, kMaxLabels>(p, slot, L, dir);
                }
            }
        } else {
            table_convolve<T, M, STD, TI, TN>(p, Vs, smem, L, mins);
            if constexpr (kNormalise) {
                __syncthreads();
                if (!kBlocked && act) table_normalise<T>(md, L, p.norm_min);
            }
        }
        if constexpr (kNormalise && kBlocked)
            if (act) table_normalise<T>(md, L, p.norm_min);
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

template <typename T, typename M, bool STD, int SPL, int TI, int TN>
cudaError_t launch_table_t(const RecordFormat &f, const SweepParams &p, cudaStream_t s, int num_sms) {
    static LaunchCache cache;
    return launch_tiles(sweep_kernel_table<T, M, STD, SPL, TI, TN>, cache, 2 * SPL, kTableNodes, p, f.slot_bytes, s,
                        num_sms, (size_t)(f.L + 1) / 2 * 2 * f.Lp * sizeof(T));
}

// Threads and outputs per thread: Lp / TI groups times 16 / TN (reference) or
// 64 / TN (standard) vector groups fill the block's 64 (128 above 64 labels)
// threads at the powers of two and leave some idle between them.  The largest
// TI x TN that fills the block reads the least shared memory per addition.
template <typename T, typename M>
cudaError_t launch_table(const RecordFormat &f, const SweepParams &p, cudaStream_t s, int num_sms) {
    if (p.mode == MODE_REF_MINCONV) {
        if (f.L <= 16) return launch_table_t<T, M, false, 1, 4, 1>(f, p, s, num_sms);
        if (f.L <= 32) return launch_table_t<T, M, false, 1, 4, 2>(f, p, s, num_sms);
        if (f.L <= 64) return launch_table_t<T, M, false, 1, 4, 4>(f, p, s, num_sms);
        return launch_table_t<T, M, false, 2, 4, 4>(f, p, s, num_sms);
    }
    if (f.L <= 8) return launch_table_t<T, M, true, 1, 8, 1>(f, p, s, num_sms);
    if (f.L <= 16) return launch_table_t<T, M, true, 1, 8, 2>(f, p, s, num_sms);
    if (f.L <= 32) return launch_table_t<T, M, true, 1, 8, 4>(f, p, s, num_sms);
    if (f.L <= 64) return launch_table_t<T, M, true, 1, 8, 8>(f, p, s, num_sms);
    return launch_table_t<T, M, true, 2, 8, 8>(f, p, s, num_sms);
}

}  // namespace ginf_gpu
