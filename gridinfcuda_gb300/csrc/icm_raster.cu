// icm_raster.cu -- raster-order Gauss-Seidel ICM (src/icm.cc:40-67) as one
// launch: all iterations, exact.
//
// In raster order a node sees its west and north neighbours' labels of this
// iteration and its east and south neighbours' of the one before.  A warp owns
// a strip of four rows for every iteration and runs them in skewed lockstep:
// at step s row r handles the column s - r, eight lanes a node, so a row's
// north label is what the eight lanes beside it found one step earlier (a
// shuffle) and its west label what it found itself.  The rest a step needs --
// the costs, the east and south labels, the first row's north labels -- is
// requested one chunk of kChunk steps ahead.
//
// Strips meet at mailboxes in global memory, one word per column for a strip's
// first and last row: label and iteration tag in one word, written and polled
// with relaxed accesses, so no fence is needed and a word tells by itself
// whether it has arrived.  A strip never runs ahead of its neighbours' words
// by more than the recipe allows, so one word per column is enough: the strip
// below takes a column of iteration t only after the word of iteration t above
// it, and the strip above takes iteration t + 1 there only after the word of
// iteration t below.  All strips must be resident (cooperative launch); every
// poll is bounded.
//
// Bound: the latency of a step -- a shuffle, two table rows from shared memory,
// the additions, the argmin over eight lanes -- times the columns and
// iterations, plus the strips' lags.  One launch per anti-diagonal, as before,
// paid a launch for each: 640x480x32, five iterations, RASTER_MEASURED
//
// The sum's order, the lanes' partition of the labels and their combine are
// icm_node's, so labels agree with the other ICM kernels whatever the costs.
#include <algorithm>

#include "ginf_internal.h"
#include "ptx.cuh"

namespace ginf_gpu {

namespace {

constexpr int kRows = 4;    // rows per strip
constexpr int kChunk = 4;   // steps per request

__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed(uint32_t *p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

template <typename T>
struct Vec {
    static constexpr int E = 16 / sizeof(T);
    alignas(16) T v[E];
    __device__ __forceinline__ void load(const T *p) {
        *reinterpret_cast<uint4 *>(v) = *reinterpret_cast<const uint4 *>(p);
    }
    __device__ __forceinline__ void add(const Vec &o) {
#pragma unroll
        for (int k = 0; k < E; ++k) v[k] += o.v[k];
    }
};

// top / bot: mailboxes [strips][W] of each strip's first / last row, zeroed.
// NQ: 16-byte label chunks per lane.
template <typename T, int NQ>
__global__ void __launch_bounds__(32)
    k_icm_raster(const unsigned char *__restrict__ rec, int W, int H, int L, int Lp, uint32_t rec_bytes,
                 const T *__restrict__ V, int32_t *lab, int iters, uint32_t *top, uint32_t *bot, int *status) {
    extern __shared__ __align__(16) unsigned char raster_smem[];
    constexpr int E = Vec<T>::E;
    T *Vs = reinterpret_cast<T *>(raster_smem);  // Vs[f * Lp + l] = V(l, f)
    const int lane = threadIdx.x, r = lane >> 3, g = lane & 7;
    for (int l = lane; l < Lp; l += 32)
        for (int f0 = 0; f0 < L; f0 += 8) {
            T v[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) v[q] = l < L && f0 + q < L ? V[l + (size_t)L * (f0 + q)] : T(0);
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (f0 + q < L) Vs[(f0 + q) * Lp + l] = v[q];
        }
    __syncwarp();
    const int strip = blockIdx.x;
    const int y = 1 + kRows * strip + r;
    const bool row = y <= H - 2;
    const bool first = strip == 0, last = strip == (int)gridDim.x - 1;
    const size_t yw = (size_t)min(y, H - 2) * W;
    const uint32_t *north = bot + (size_t)(first ? 0 : strip - 1) * W;
    const uint32_t *south = top + (size_t)(last ? 0 : strip + 1) * W;
    uint32_t *my_top = top + (size_t)strip * W, *my_bot = bot + (size_t)strip * W;
    // Where this lane's neighbour words come from: lanes 0-3 of a row hold the
    // south labels of a chunk's steps, lanes 4-7 the east ones; lanes 0-3 of
    // the first row also the north ones.
    const bool south_box = g < kChunk && r == kRows - 1 && !last;
    const bool north_lane = r == 0 && g < kChunk;
    const bool north_box = north_lane && !first;
    const int steps = (W - 2) + (kRows - 1);
    bool bad = false;
    auto checked = [&](int f) {
        if (f < 0 || f >= L) {
            bad = true;
            return 0;
        }
        return f;
    };

    for (int t = 0; t < iters; ++t) {
        __syncwarp();  // the previous iteration's labels, written by other lanes
        const uint32_t tag_s = (uint32_t)t & 0xffffu, tag_n = (uint32_t)(t + 1) & 0xffffu;
        const bool wait_s = south_box && t > 0;
        int cur = row ? checked(__ldcg(lab + yw)) : 0;  // the west border's label
        uint32_t a = 0, b = 0, an = 0, bn = 0;          // neighbour words of this chunk and the next
        Vec<T> d[kChunk][NQ], dn[kChunk][NQ];
        // Column of this lane's word and whether its step exists.
        auto column = [&](int k) { return 1 + k * kChunk + (g & (kChunk - 1)) - r; };
        auto exists = [&](int x) { return row && x >= 1 && x <= W - 2; };
        auto request = [&](int k, uint32_t &wa, uint32_t &wb, Vec<T>(&c)[kChunk][NQ]) {
            const int x = column(k);
            wa = wb = 0;
            if (exists(x)) {
                if (g >= kChunk) wa = (uint32_t)__ldcg(lab + yw + x + 1);
                else if (wait_s) wa = ld_relaxed(south + x);
                else wa = (uint32_t)__ldcg(lab + yw + W + x);
                if (north_lane) wb = north_box ? ld_relaxed(north + x) : (uint32_t)__ldcg(lab + yw - W + x);
            }
#pragma unroll
            for (int j = 0; j < kChunk; ++j) {
                const int xj = 1 + k * kChunk + j - r;
#pragma unroll
                for (int q = 0; q < NQ; ++q) {
                    const int l = (g + 8 * q) * E;
                    if (exists(xj) && l < L)
                        c[j][q].load(reinterpret_cast<const T *>(rec + (yw + xj) * rec_bytes) + l);
                }
            }
        };
        // Polls until this chunk's words carry their tags, then strips them.
        auto arrive = [&](int k, uint32_t &wa, uint32_t &wb) {
            const int x = column(k);
            const bool ws = wait_s && exists(x), wn = north_box && exists(x);
            uint64_t t0 = 0;
            for (uint32_t n = 1; !__all_sync(~0u, (!ws || wa >> 16 == tag_s) && (!wn || wb >> 16 == tag_n)); ++n) {
                if (ws && wa >> 16 != tag_s) wa = ld_relaxed(south + x);
                if (wn && wb >> 16 != tag_n) wb = ld_relaxed(north + x);
                if ((n & 255u) == 0) {
                    const uint64_t now = __shfl_sync(~0u, global_timer_ns(), 0);
                    if (t0 == 0) t0 = now;
                    else if (now - t0 > kWaitLimitNs) {
                        if (lane == 0) atomicOr(status, DEV_ERR_TIMEOUT);
                        return false;
                    }
                }
            }
            if (ws) wa &= 0xffffu;
            if (wn) wb &= 0xffffu;
            if (exists(x)) {
                wa = (uint32_t)checked((int)wa);
                if (north_lane) wb = (uint32_t)checked((int)wb);
            }
            return true;
        };
        request(0, a, b, d);
        if (!arrive(0, a, b)) return;
        for (int k = 0; k * kChunk < steps; ++k) {
            const bool more = (k + 1) * kChunk < steps;
            if (more) request(k + 1, an, bn, dn);
#pragma unroll
            for (int j = 0; j < kChunk; ++j) {
                const int x = 1 + k * kChunk + j - r;
                const int fs = __shfl_sync(~0u, (int)a, (lane & ~7) + j);
                const int fe = __shfl_sync(~0u, (int)a, (lane & ~7) + kChunk + j);
                const int f0 = __shfl_sync(~0u, (int)b, j);
                const int up = __shfl_up_sync(~0u, cur, 8);
                const int fn = r == 0 ? f0 : up;
                const bool act = exists(x);
                T best = T(0);
                int bl = 0x7fffffff;
                if (act) {
#pragma unroll
                    for (int q = 0; q < NQ; ++q) {
                        const int l = (g + 8 * q) * E;
                        if (l < L) {
                            Vec<T> c = d[j][q], vs, ve, vn, vw;
                            vs.load(Vs + fs * Lp + l);
                            ve.load(Vs + fe * Lp + l);
                            vn.load(Vs + fn * Lp + l);
                            vw.load(Vs + cur * Lp + l);
                            c.add(vs);
                            c.add(ve);
                            c.add(vn);
                            c.add(vw);
#pragma unroll
                            for (int e = 0; e < E; ++e) {
                                if (l + e < L && (bl == 0x7fffffff || c.v[e] < best)) {
                                    best = c.v[e];
                                    bl = l + e;
                                }
                            }
                        }
                    }
                }
#pragma unroll
                for (int off = 1; off < 8; off <<= 1) {
                    const T ob = __shfl_xor_sync(~0u, best, off);
                    const int ol = __shfl_xor_sync(~0u, bl, off);
                    if (ol != 0x7fffffff && (bl == 0x7fffffff || ob < best || (!(best < ob) && ol < bl))) {
                        best = ob;
                        bl = ol;
                    }
                }
                if (act) {
                    cur = bl;
                    if (g == 0) {
                        lab[yw + x] = bl;
                        if (r == 0 && !first) st_relaxed(my_top + x, tag_n << 16 | (uint32_t)bl);
                        if (r == kRows - 1 && !last) st_relaxed(my_bot + x, tag_n << 16 | (uint32_t)bl);
                    }
                }
            }
            if (more) {
                if (!arrive(k + 1, an, bn)) return;
                a = an;
                b = bn;
#pragma unroll
                for (int j = 0; j < kChunk; ++j)
#pragma unroll
                    for (int q = 0; q < NQ; ++q) d[j][q] = dn[j][q];
            }
        }
    }
    if (bad) atomicOr(status, DEV_ERR_BOUNDS);
}

template <typename T, int NQ>
cudaError_t launch_raster_t(const RecordFormat &f, const unsigned char *rec, int W, int H, const void *V,
                            int32_t *labels, int iters, uint32_t *boxes, int *status, cudaStream_t s, int num_sms,
                            bool &done) {
    static SmemLimit limit;
    static OccupancyMemo memo;
    auto kern = k_icm_raster<T, NQ>;
    const int strips = icm_raster_strips(H);
    const size_t smem = (size_t)f.L * f.Lp * sizeof(T);
    cudaError_t e = limit.ensure(kern, smem);
    if (e != cudaSuccess) return e;
    int occ = 0;
    e = memo.blocks(kern, 32, smem, occ);
    if (e != cudaSuccess) return e;
    if ((long)occ * num_sms < strips) return cudaSuccess;  // not all strips resident
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)strips);
    lc.blockDim = dim3(32);
    lc.dynamicSmemBytes = smem;
    lc.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    lc.attrs = attr;
    lc.numAttrs = 1;
    done = true;
    return cudaLaunchKernelEx(&lc, kern, rec, W, H, f.L, f.Lp, f.rec_bytes, static_cast<const T *>(V), labels, iters,
                              boxes, boxes + (size_t)strips * W, status);
}

template <typename T>
cudaError_t launch_raster(const RecordFormat &f, const unsigned char *rec, int W, int H, const void *V,
                          int32_t *labels, int iters, uint32_t *boxes, int *status, cudaStream_t s, int num_sms,
                          bool &done) {
    const int per_chunk = 8 * (16 / (int)sizeof(T));  // labels a row's eight lanes take at once
    if (f.L <= per_chunk)
        return launch_raster_t<T, 1>(f, rec, W, H, V, labels, iters, boxes, status, s, num_sms, done);
    if (f.L <= 2 * per_chunk)
        return launch_raster_t<T, 2>(f, rec, W, H, V, labels, iters, boxes, status, s, num_sms, done);
    if (f.L <= 4 * per_chunk)
        return launch_raster_t<T, 4>(f, rec, W, H, V, labels, iters, boxes, status, s, num_sms, done);
    return cudaSuccess;
}

}  // namespace

int icm_raster_strips(int H) { return H >= 3 ? (H - 2 + kRows - 1) / kRows : 0; }

cudaError_t launch_icm_raster(const RecordFormat &f, const unsigned char *rec, int W, int H, const void *V,
                              int32_t *labels, int iters, uint32_t *boxes, int *status, cudaStream_t s, int num_sms,
                              bool &done) {
    done = false;
    if (W < 3 || H < 3 || iters < 1) return cudaSuccess;
    switch (f.ctype) {
        case CT_F32: return launch_raster<float>(f, rec, W, H, V, labels, iters, boxes, status, s, num_sms, done);
        case CT_I32: return launch_raster<int>(f, rec, W, H, V, labels, iters, boxes, status, s, num_sms, done);
        case CT_F64: return launch_raster<double>(f, rec, W, H, V, labels, iters, boxes, status, s, num_sms, done);
    }
    return cudaErrorInvalidValue;
}

}  // namespace ginf_gpu
