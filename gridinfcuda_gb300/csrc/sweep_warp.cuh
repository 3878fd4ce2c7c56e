// sweep_warp.cuh -- the half-sweep of the truncated-linear / Potts update for
// few labels (4-byte elements, L <= 32): a warp per eight nodes with ordinary
// loads and stores, no block barrier and no copy engine.
//
// With few labels a node's messages are 32 to 128 bytes, and five bulk copies
// per node (one in, four out), an mbarrier phase and two block barriers per
// tile cost more than the bytes.  Here a warp loads its nodes' costs and
// messages straight into registers, passes them through shared memory to the
// lanes that own a message each, and stores the messages through it again, so
// that every global access covers whole sectors.
//
// Bound: HBM above 16 labels (36 B per updated node and label), below it the
// accesses per node, L2-resident grids the latency of a half-sweep.  us per
// half-sweep, block tiles with bulk copies -> this form: 1920x1080 FP32 L = 8
// 145 -> 106, L = 16 131 -> 119 (4.8 TB/s), L = 24 191 -> 168, L = 32 197 ->
// 189 (6.1 TB/s); 384x288 L = 16 9.7 -> 7.4, L = 32 14.9 -> 13.4 (6.5 and 12.0
// since a half-sweep's blocks no longer start beside the last one's).  At L = 40,
// 48 and 64 it is slower on large grids (1920x1080 258 -> 280, 303 -> 331 and
// 351 -> 412) for want of registers, hence kWarpTileLabels.  With the lanes of
// the global accesses laid out as the messages' (a quarter-warp on eight nodes)
// L = 16 took 155 us and L = 32 308.
#pragma once

#include "sweep_impl.cuh"

namespace ginf_gpu {

// Warps per block of a batch's launches, a tile of eight nodes each (the batch
// of twelve grids: two 12.88 ms, four 12.86, eight 12.94).
constexpr int kWarpTileWarps = 4;

// Tile t of one half-sweep by one warp; `slots` holds the warp's eight slots.
template <typename T, int LMAX, int LMIN>
__device__ __forceinline__ void warp_tile(const SweepParams &p, const TableConsts<T> &tc, int t,
                                          unsigned char *slots) {
    constexpr int NCH = LMAX / 4, CPL = (NCH + 3) / 4;  // 16-byte chunks per vector, and per lane
    const int L = LMIN == LMAX ? LMAX : p.L;
    const int lane = threadIdx.x & 31;
    // Two lane layouts: global accesses take node lane / 4, chunks lane % 4, +4,
    // ... (a quarter-warp covers whole sectors of two nodes); messages take node
    // lane % 8, direction lane / 8 (a quarter-warp's 16-byte shared accesses fall
    // into eight bank groups).
    const int n = lane >> 2, q = lane & 3, dir = lane >> 3;
    unsigned char *nslot = slots + (size_t)n * p.slot_bytes;
    unsigned char *slot = slots + (size_t)(lane & 7) * p.slot_bytes;
    const int y = 1 + t / p.tiles_per_row;
    const int x0 = ((y + p.iter) & 1) + 1 + 2 * ((t % p.tiles_per_row) * 8);
    const int x = x0 + 2 * n;
    const bool act = x <= p.W - 2;
    unsigned char *r = p.rec + ((size_t)y * p.W + x) * p.rec_bytes;
    T best = pos_inf<T>();
    int label = 0x7fffffff;
    if (act) {
        const unsigned zero = zero_mask(p, x, y);
        T v[CPL][4], a[CPL][4][4];
#pragma unroll
        for (int j = 0; j < CPL; ++j) {
            const int c = (4 * j + q) * 4;
            if (NCH % 4 == 0 || c < LMAX) MIO<T, T>::load(r + c * sizeof(T), v[j]);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const unsigned char *m = r + p.d_bytes + e * p.m_bytes;
            if (p.read_mode == RD_COARSE) {
                // As tile_load: the coarse sender's message at its receiver.
                const int Rx = ((x + dir_dx(e)) >> 1) - dir_dx(e), Ry = ((y + dir_dy(e)) >> 1) - dir_dy(e);
                m = p.crec + ((ptrdiff_t)Ry * p.cW + Rx) * (ptrdiff_t)p.rec_bytes + p.d_bytes + e * p.m_bytes;
            }
#pragma unroll
            for (int j = 0; j < CPL; ++j) {
                const int c = (4 * j + q) * 4;
                if ((zero >> e) & 1u) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) a[j][e][k] = T(0);
                } else if (NCH % 4 == 0 || c < LMAX) {
                    MIO<T, T>::load(m + c * sizeof(T), a[j][e]);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < CPL; ++j) {
            const int c = (4 * j + q) * 4;
            if (NCH % 4 == 0 || c < LMAX) {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) v[j][k] = v[j][k] + a[j][e][k];
                    MIO<T, T>::store(nslot + p.d_bytes + e * p.m_bytes + c * sizeof(T), a[j][e]);
                }
                MIO<T, T>::store(nslot + c * sizeof(T), v[j]);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if ((LMIN == LMAX || c + k < L) && (label == 0x7fffffff || v[j][k] < best)) {
                        best = v[j][k];
                        label = c + k;
                    }
                }
            }
        }
    }
    if (p.write_labels) {
        // argmin_combine over lanes 4n .. 4n + 3.
#pragma unroll
        for (int off = 1; off <= 2; off <<= 1) {
            const T ob = __shfl_xor_sync(0xffffffffu, best, off);
            const int ol = __shfl_xor_sync(0xffffffffu, label, off);
            if (ol != 0x7fffffff && (label == 0x7fffffff || ob < best || (!(best < ob) && ol < label))) {
                best = ob;
                label = ol;
            }
        }
        if (act && q == 0) p.labels[(size_t)y * p.W + x] = label;
    }
    __syncwarp();
    if (x0 + 2 * (lane & 7) <= p.W - 2) message_linear<T, T, LMAX, LMIN>(p, slot, L, dir, tc.scale, tc.trunc);
    __syncwarp();
    if (act) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            unsigned char *dst = p.rec + ((size_t)(y + dir_dy(e)) * p.W + x + dir_dx(e)) * p.rec_bytes + p.d_bytes +
                                 opp_dir(e) * p.m_bytes;
#pragma unroll
            for (int j = 0; j < CPL; ++j) {
                const int c = (4 * j + q) * 4;
                if (NCH % 4 == 0 || c < LMAX) {
                    T o[4];
                    MIO<T, T>::load(nslot + p.d_bytes + e * p.m_bytes + c * sizeof(T), o);
                    MIO<T, T>::store(dst + c * sizeof(T), o);
                }
            }
        }
    }
    __syncwarp();
}

// One half-sweep, a block's NW warps taking tiles on their own.  MINB: blocks
// per SM the registers are allocated for (0: no bound).
template <typename T, int LMAX, int LMIN, int NW, int MINB>
__global__ void __launch_bounds__(NW * 32, MINB) sweep_kernel_warp(const SweepParams p) {
    extern __shared__ __align__(128) unsigned char smem[];
    const TableConsts<T> tc = table_consts<T, KIND_LINEAR>(p.V, LMIN == LMAX ? LMAX : p.L);
    const int warp = threadIdx.x >> 5;
    unsigned char *slots = smem + (size_t)warp * 8 * p.slot_bytes;
    grid_dependency_wait();
    for (int t = blockIdx.x * NW + warp; t < p.num_tiles; t += gridDim.x * NW)
        warp_tile<T, LMAX, LMIN>(p, tc, t, slots);
}

template <typename T, int LM, int LO, int NW, int MINB = 0>
cudaError_t launch_warp_kernel(const RecordFormat &f, const SweepParams &p, cudaStream_t s, int num_sms) {
    static LaunchCache cache;
    return launch_tiles(sweep_kernel_warp<T, LM, LO, NW, MINB>, cache, NW, 8, p, f.slot_bytes, s, num_sms,
                        (size_t)(NW - 1) * 8 * f.slot_bytes, NW);
}

// Warps per block, us per half-sweep: two at L = 8 (four: 1280x720 55.7 -> 53.2,
// 1920x1080 115 -> 110, small grids equal), four at L = 24, eight at L = 32 (four:
// 384x288 12.5 -> 12.0, 1920x1080 197 -> 192).  At L = 16 four up to
// kWarpTiles4 tiles (800x600, 29900 tiles: 24.8, with two 28.2) and two above
// it, where the records outgrow the L2 cache (1024x768 44.6 -> 43.6, 1600x900
// 90.7 -> 76.5, 1920x1080 124 -> 108), and of four those up to kWarpSmallTiles
// held to 48 registers (40 warps per SM instead of 36: 240x180 3.9 -> 3.6,
// 384x288, 6864 tiles, 6.8 -> 6.5, but 640x480, 19120, 15.8 -> 16.6).
constexpr long kWarpSmallTiles = 12288, kWarpTiles4 = 40960;

template <typename T, int LM, int LO>
cudaError_t launch_warp_tiles(const RecordFormat &f, const SweepParams &p, cudaStream_t s, int num_sms) {
    if constexpr (LM == 16) {
        const int n1 = p.W >= 3 ? (p.W - 3) / 2 + 1 : 0;
        const long tiles = p.H >= 3 ? (long)(p.H - 2) * ((n1 + 7) / 8) : 0;
        if (tiles <= kWarpSmallTiles) return launch_warp_kernel<T, LM, LO, 4, 10>(f, p, s, num_sms);
        if (tiles <= kWarpTiles4) return launch_warp_kernel<T, LM, LO, 4>(f, p, s, num_sms);
        return launch_warp_kernel<T, LM, LO, 2>(f, p, s, num_sms);
    }
    return launch_warp_kernel<T, LM, LO, LM == 8 ? 2 : (LM == 32 ? 8 : 4)>(f, p, s, num_sms);
}

}  // namespace ginf_gpu
