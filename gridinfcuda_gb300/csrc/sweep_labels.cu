// sweep_labels.cu -- the last half-sweep of a solve whose messages nobody
// reads: each node of its colour gets the first argmin of its belief, which is
// all that a stale-belief decode takes from it (src/bp.cc:65-84).
//
// Bound: HBM, costs and four incoming messages per node (20 B per label in
// FP32) instead of the full half-sweep's 36 B.  No shared memory: four lanes
// per node, lane g reading the 16-byte message chunks g, g + 4, ..., two chunks
// in flight each, so eight nodes' loads cover whole 32-byte sectors.
// 1920x1080x64 FP32: 365 us as a full half-sweep, 205 us here; 1280x720x128
// truncated quadratic 347 -> 270 us.
//
// The belief's sum and the argmin's lane partition and combine are the
// half-sweep's (belief_part, and the split kernel's halves at 128 labels), so
// the label is the same whatever the costs hold, NaN included.
#include <algorithm>

#include "sweep_labels.cuh"

namespace ginf_gpu {

namespace {

constexpr int kLabelThreads = 256;

// HALVES: the split kernel's partition -- lanes 4 - 7 of eight take the labels
// from `half` on.
template <typename T, typename M, bool HALVES>
__global__ void __launch_bounds__(kLabelThreads) k_sweep_labels(const SweepParams p, int half) {
    constexpr int LANES = HALVES ? 8 : 4;
    grid_dependency_wait();
    const int g = threadIdx.x & 3;
    const bool upper = HALVES && (threadIdx.x & 4);
    const int n = blockIdx.x * (kLabelThreads / LANES) + threadIdx.x / LANES;  // node of its colour in the row
    for (int y = 1 + blockIdx.y; y <= p.H - 2; y += gridDim.y) {
        const int x = ((y + p.iter) & 1) + 1 + 2 * n;
        const bool act = x <= p.W - 2;
        T best = pos_inf<T>();
        int label = 0x7fffffff;
        if (act)
            label_part<T, M>(p.rec + ((size_t)y * p.W + x) * p.rec_bytes, p, zero_mask(p, x, y), upper ? half : 0,
                             HALVES && !upper ? half : p.L, g, best, label);
        combine4(best, label);
        if constexpr (HALVES) {
            const T ob = __shfl_xor_sync(0xffffffffu, best, 4);
            const int ol = __shfl_xor_sync(0xffffffffu, label, 4);
            if (ol != 0x7fffffff && (label == 0x7fffffff || ob < best || (!(best < ob) && ol < label))) label = ol;
        }
        if (act && threadIdx.x % LANES == 0) p.labels[(size_t)y * p.W + x] = label;
    }
}

template <typename T, typename M, bool HALVES = false>
cudaError_t launch_labels_t(const SweepParams &p, int half, cudaStream_t s) {
    const int n1 = (p.W - 3) / 2 + 1;  // most nodes of a colour in a row
    constexpr int kNodes = kLabelThreads / (HALVES ? 8 : 4);
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)((n1 + kNodes - 1) / kNodes), (unsigned)std::min(p.H - 2, 65535));
    lc.blockDim = dim3(kLabelThreads);
    lc.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = attr;
    lc.numAttrs = 1;
    return cudaLaunchKernelEx(&lc, k_sweep_labels<T, M, HALVES>, p, half);
}

}  // namespace

cudaError_t launch_sweep_labels(const RecordFormat &f, const SweepParams &p, cudaStream_t s) {
    if (p.W < 3 || p.H < 3) return cudaSuccess;
    // The split kernel (launch_variant) with 128 labels parts them in halves.
    const bool split = f.ctype == CT_F32 && f.store == ST_NATIVE && f.L == 128 && p.mode == MODE_STD_QUAD &&
                       p.quad_radius <= kQuadWindow;
    if (split) return launch_labels_t<float, float, true>(p, 64, s);
    if (f.store == ST_F16) return launch_labels_t<float, __half>(p, 0, s);
    switch (f.ctype) {
        case CT_F32: return launch_labels_t<float, float>(p, 0, s);
        case CT_I32: return launch_labels_t<int, int>(p, 0, s);
        case CT_F64: return launch_labels_t<double, double>(p, 0, s);
    }
    return cudaErrorInvalidValue;
}

}  // namespace ginf_gpu
