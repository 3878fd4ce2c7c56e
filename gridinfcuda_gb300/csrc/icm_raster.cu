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
// Bound: the latency of a step -- a shuffle, a table row from shared memory,
// the additions, the argmin over eight lanes -- times the columns and
// iterations, plus the strips' lags (2.8 us each).  640x480x32 int32: 0.24 us a
// step (one warp on a scheduler, 5.8 cycles an instruction, ncu); five iterations
// 1.19 ms, against 23.0 ms with one launch per anti-diagonal (5590 of them) and
// 1.98 ms with stores per step and the general argmin.
//
// A warp a block and the whole table in its shared memory: grids whose strips do
// not all fit the device at once (128 labels in 4 bytes: 64 KB, three blocks an
// SM, 1826 rows on 152 SMs; 96 labels twice that) and FP64 grids of more than 64
// labels keep one launch per anti-diagonal.
//
// The sum's order is the reference's and ties go to the lowest label.  Chunks
// whose costs hold a NaN or a value near -infinity, and tables that do, take
// icm_node's own partition and combine (raster_node_any), so that labels agree
// with the other ICM kernels whatever the costs.
#include <algorithm>

#include <type_traits>

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
    __device__ __forceinline__ void load(const void *p) {
        *reinterpret_cast<uint4 *>(v) = *reinterpret_cast<const uint4 *>(p);
    }
    __device__ __forceinline__ void add(const Vec &o) {
#pragma unroll
        for (int k = 0; k < E; ++k) v[k] += o.v[k];
    }
};

// Values above every cost, and below which a cost leaves the fast form: a sum
// of five that are not below it is neither NaN nor -infinity.
template <typename T>
__device__ __forceinline__ T top_cost();
template <>
__device__ __forceinline__ float top_cost<float>() { return __int_as_float(0x7f800000); }
template <>
__device__ __forceinline__ double top_cost<double>() { return __longlong_as_double(0x7ff0000000000000ll); }
template <>
__device__ __forceinline__ int top_cost<int>() { return 0x7fffffff; }
__device__ __forceinline__ bool odd_cost(float v) { return !(v > -1e37f); }
__device__ __forceinline__ bool odd_cost(double v) { return !(v > -1e300); }
__device__ __forceinline__ bool odd_cost(int) { return false; }

// (value, label) of the smaller: the lower label of equal values.
template <typename T>
__device__ __forceinline__ void take_less(T &best, int &bl, T ob, int ol) {
    const bool take = ob < best || (ob == best && ol < bl);
    best = take ? ob : best;
    bl = take ? ol : bl;
}

// One node's label by its eight lanes, as icm_node<T, 8> of aux_kernels.cu,
// for any costs: the four table rows at the byte offsets fs, fe, fn, fw of Vs.
template <typename T>
__device__ int raster_node_any(const T *D, const unsigned char *Vs, int fs, int fe, int fn, int fw, int L, int g) {
    constexpr int E = Vec<T>::E;
    T best = T(0);
    int bl = 0x7fffffff;
    for (int l = g * E; l < L; l += 8 * E) {
        Vec<T> c, w;
        c.load(D + l);
        const unsigned char *v = Vs + (size_t)l * sizeof(T);
        w.load(v + fs);
        c.add(w);
        w.load(v + fe);
        c.add(w);
        w.load(v + fn);
        c.add(w);
        w.load(v + fw);
        c.add(w);
#pragma unroll
        for (int e = 0; e < E; ++e) {
            if (l + e < L && (bl == 0x7fffffff || c.v[e] < best)) {
                best = c.v[e];
                bl = l + e;
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
    return bl;
}

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
    bool odd_table = false;
    for (int l = lane; l < Lp; l += 32)
        for (int f0 = 0; f0 < L; f0 += 8) {
            T v[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) v[q] = l < L && f0 + q < L ? V[l + (size_t)L * (f0 + q)] : T(0);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                if (f0 + q < L) Vs[(f0 + q) * Lp + l] = v[q];
                odd_table |= odd_cost(v[q]);
            }
        }
    odd_table = __any_sync(~0u, odd_table);
    __syncwarp();
    const int strip = blockIdx.x;
    const int y = 1 + kRows * strip + r;
    const int cols = y <= H - 2 ? W - 2 : 0;  // of this lane's row
    const bool first = strip == 0, last = strip == (int)gridDim.x - 1;
    const size_t yw = (size_t)min(y, H - 2) * W;
    const int row_bytes = Lp * (int)sizeof(T);  // a table row
    // Where this lane's neighbour words come from: lanes 0-3 of a row hold the
    // south labels of a chunk's steps, lanes 4-7 the east ones; lanes 0-3 of
    // the first row also the north ones.  They are kept as the byte offsets of
    // the labels' table rows.
    const bool south_box = g < kChunk && r == kRows - 1 && !last;
    const bool north_lane = r == 0 && g < kChunk;
    const bool north_box = north_lane && !first;
    const bool out_top = north_lane && !first, out_bot = south_box;  // lanes that publish
    const int steps = (W - 2) + (kRows - 1);
    // This lane's column of chunk 0, less one, and what it reads and writes there.
    const int u0 = (g & (kChunk - 1)) - r;
    const int32_t *east_or_south = lab + yw + 1 + u0 + (g >= kChunk ? 1 : W);
    const int32_t *above = lab + yw + 1 + u0 - W;
    const uint32_t *south = top + (size_t)(last ? 0 : strip + 1) * W + 1 + u0;
    const uint32_t *north = bot + (size_t)(first ? 0 : strip - 1) * W + 1 + u0;
    int32_t *mine = lab + yw + 1 + u0;
    uint32_t *box = (r == 0 ? top : bot) + (size_t)strip * W + 1 + u0;
    const unsigned char *costs = rec + (yw + 1 - r) * rec_bytes + g * 16;
    bool bad = false;
    auto offset = [&](int f) {  // of a label's table row
        if (f < 0 || f >= L) {
            bad = true;
            f = 0;
        }
        return f * row_bytes;
    };

    for (int t = 0; t < iters; ++t) {
        __syncwarp();  // the previous iteration's labels, written by other lanes
        const uint32_t tag_s = (uint32_t)t & 0xffffu, tag_n = (uint32_t)(t + 1) & 0xffffu;
        const bool wait_s = south_box && t > 0;
        int cur = cols ? offset(__ldcg(lab + yw)) : 0;  // the west border's label
        uint32_t a = 0, b = 0, an = 0, bn = 0;          // neighbour words of this chunk and the next
        Vec<T> d[kChunk][NQ], dn[kChunk][NQ];
#pragma unroll
        for (int j = 0; j < kChunk; ++j)
#pragma unroll
            for (int q = 0; q < NQ; ++q)
#pragma unroll
                for (int e = 0; e < E; ++e) d[j][q].v[e] = dn[j][q].v[e] = T(0);
        // Words and costs of the chunk that starts k steps in.
        auto request = [&](int k, uint32_t &wa, uint32_t &wb, Vec<T>(&c)[kChunk][NQ]) {
            if ((unsigned)(u0 + k) < (unsigned)cols) {
                wa = wait_s ? ld_relaxed(south + k) : (uint32_t)__ldcg(east_or_south + k);
                if (north_lane) wb = north_box ? ld_relaxed(north + k) : (uint32_t)__ldcg(above + k);
            }
            const unsigned char *p = costs + (ptrdiff_t)k * rec_bytes;
#pragma unroll
            for (int j = 0; j < kChunk; ++j) {
                if ((unsigned)(k + j - r) < (unsigned)cols) {
#pragma unroll
                    for (int q = 0; q < NQ; ++q)
                        if ((g + 8 * q) * E < L) c[j][q].load(p + q * 128);
                }
                p += rec_bytes;
            }
        };
        // Polls until this chunk's words carry their tags, then makes them
        // offsets; the costs have arrived too and are looked over.
        bool slow = odd_table;
        auto arrive = [&](int k, uint32_t &wa, uint32_t &wb, const Vec<T>(&c)[kChunk][NQ]) {
            const bool in = (unsigned)(u0 + k) < (unsigned)cols;
            const bool ws = wait_s && in, wn = north_box && in;
            uint64_t t0 = 0;
            for (uint32_t n = 1; !__all_sync(~0u, (!ws || wa >> 16 == tag_s) && (!wn || wb >> 16 == tag_n)); ++n) {
                if (ws && wa >> 16 != tag_s) wa = ld_relaxed(south + k);
                if (wn && wb >> 16 != tag_n) wb = ld_relaxed(north + k);
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
            if (in) {
                wa = (uint32_t)offset((int)wa);
                if (north_lane) wb = (uint32_t)offset((int)wb);
            } else {
                wa = wb = 0;
            }
            if constexpr (sizeof(T) == 8 || std::is_same<T, float>::value) {
                bool odd = odd_table;
#pragma unroll
                for (int j = 0; j < kChunk; ++j)
#pragma unroll
                    for (int q = 0; q < NQ; ++q)
#pragma unroll
                        for (int e = 0; e < E; ++e) odd |= odd_cost(c[j][q].v[e]);
                slow = __any_sync(~0u, odd);
            }
            return true;
        };
        request(0, a, b, d);
        if (!arrive(0, a, b, d)) return;
        for (int k = 0; k < steps; k += kChunk) {
            const bool more = k + kChunk < steps;
            if (more) request(k + kChunk, an, bn, dn);
            int found = 0;  // this lane's step's label
#pragma unroll
            for (int j = 0; j < kChunk; ++j) {
                const int fs = __shfl_sync(~0u, (int)a, (lane & ~7) + j);
                const int fe = __shfl_sync(~0u, (int)a, (lane & ~7) + kChunk + j);
                const int f0 = __shfl_sync(~0u, (int)b, j);
                const int up = __shfl_up_sync(~0u, cur, 8);
                const int fn = r == 0 ? f0 : up;
                const bool act = (unsigned)(k + j - r) < (unsigned)cols;
                int bl;
                if (slow) {
                    // Inactive rows read some record of the grid.
                    const size_t node = yw + (act ? 1 + k + j - r : 1);
                    bl = raster_node_any(reinterpret_cast<const T *>(rec + node * rec_bytes), raster_smem, fs, fe, fn,
                                         cur, L, g);
                } else {
                    T best = top_cost<T>();
                    bl = 0x7fffffff;
#pragma unroll
                    for (int q = 0; q < NQ; ++q) {
                        const int l = (g + 8 * q) * E;
                        const unsigned char *v = raster_smem + l * (int)sizeof(T);
                        if (NQ == 1 || l < L) {
                            Vec<T> c = d[j][q], w;
                            w.load(v + fs);
                            c.add(w);
                            w.load(v + fe);
                            c.add(w);
                            w.load(v + fn);
                            c.add(w);
                            w.load(v + cur);
                            c.add(w);
#pragma unroll
                            for (int e = 0; e < E; ++e)
                                if (l + e >= L) c.v[e] = top_cost<T>();
                            // The first minimum of the chunk, in pairs.
                            int m[E];
#pragma unroll
                            for (int e = 0; e < E; ++e) m[e] = l + e;
#pragma unroll
                            for (int w2 = 1; w2 < E; w2 *= 2)
#pragma unroll
                                for (int e = 0; e + w2 < E; e += 2 * w2) {
                                    const bool right = c.v[e + w2] < c.v[e];
                                    c.v[e] = right ? c.v[e + w2] : c.v[e];
                                    m[e] = right ? m[e + w2] : m[e];
                                }
                            if (q == 0) {
                                best = c.v[0];
                                bl = m[0];
                            } else if (c.v[0] < best) {
                                best = c.v[0];
                                bl = m[0];
                            }
                        }
                    }
#pragma unroll
                    for (int off = 1; off < 8; off <<= 1)
                        take_less(best, bl, __shfl_xor_sync(~0u, best, off), __shfl_xor_sync(~0u, bl, off));
                }
                if (act) cur = bl * row_bytes;
                if ((g & (kChunk - 1)) == j) found = bl;
            }
            // The chunk's labels: into the labelling and, for the strips' outer
            // rows, the mailboxes.
            if (g < kChunk && (unsigned)(u0 + k) < (unsigned)cols) {
                mine[k] = found;
                if (out_top || out_bot) st_relaxed(box + k, tag_n << 16 | (uint32_t)found);
            }
            if (more) {
                if (!arrive(k + kChunk, an, bn, dn)) return;
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
    const size_t smem = (size_t)f.L * f.Lp * sizeof(T) + 128;  // lanes beyond L read past the last row
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
