// conv_tc.cu -- the warm-start network's 3x3 convolutions (the forward pass,
// the data gradient as a forward convolution with flipped weights, and the
// weight gradient) on the fifth-generation tensor cores: tcgen05.mma with the
// accumulator in tensor memory, both operands read from shared memory by
// matrix descriptors, the input rows brought in by TMA tensor copies.
//
// Implicit GEMM.  A tile is M = 128 consecutive pixels of one image row,
// N = COUT output channels, K = 9 taps x CIN input channels, BF16 operands,
// FP32 accumulation.  Activations are NHWC BF16.  A CTA owns a strip of
// tiles going down one column band (up to 128 pixels; a narrower one's last
// accumulator rows are computed from what the buffer held and not read) of an
// image, so each input row is loaded once (plus one halo row above and below
// the strip): a row arrives as one TMA tensor copy of band + 2 pixels x CIN
// channels (the band plus one pixel either side; pixels and rows outside the image read as zero,
// which is the convolution's zero padding) into a 1024-byte aligned buffer,
// swizzled by the copy (128-, 64- or 32-byte swizzle for CIN = 64, 32, 16:
// one pixel's channels per swizzle row), which is the canonical K-major
// layout the tensor cores read: 8-pixel groups SBO = 8 rows apart.  The
// swizzle is a function of the absolute shared-memory address, so the A
// operand of tap (dy, dx) is the buffer of row y + dy read from pixel dx + 1
// on, a descriptor whose start is one swizzle row further per pixel -- the
// nine taps are nine descriptors over three row buffers, nothing is copied
// per tap.
//
// The weights, [dx][8-channel chunk][j * COUT + co][8] in the canonical
// layout without swizzle, stack the three row offsets dy = j - 1 along N, so
// one MMA (N = 3 * COUT) applies an input row r to the accumulators of output
// rows r + 1, r and r - 1 at once; those live in a descending ring of
// tensor-memory slots (adjacent unless the ring wraps, when the run splits in
// two), and the first block into a fresh slot overwrites it.
//
// Roles (10 warps): 8 warps read the accumulators back (warp w owns lanes
// 32 (w % 4) .. + 31, i.e. those pixels of the tile; the warps of one lane
// quarter share out the channels, 16 or more each, or take tiles in turn),
// add the bias, apply ReLU, stage the 32 pixels in shared memory and store
// them, adding the residual in that pass; of the next warp lane 0 issues the
// row copies into a ring of RING buffers; of the last, lane 0 issues, per
// input row, 3 * CIN / 16 steps of one or two MMAs (descriptors formed once
// per row, compile-time step offsets) and commits them to mbarriers (a row
// buffer is free after its own MMAs; an output row's accumulator is full
// after input row r + 1).  Loads of the loss go out in groups of four passes,
// eight spill.  Every wait is bounded (DEV_ERR_TIMEOUT in the status word),
// and the tensor memory is released on every path.
//
// The first layer reads x in FP32: eight warps take the copying warp's place,
// round the rows on their way into the buffers and, in training, store the
// rounding for the weight gradient: 43 us of a 960x540x64 forward pass, where a
// conversion kernel before a layer that reads its output, which moves x's BF16
// through memory twice, took 26 + 33.
//
// Programmatic launches: each kernel sets up (barriers, tensor memory, its
// weights) beside the tail of the one before it and waits before it touches
// anything else.  A kernel lets its successor start only after its own wait,
// so what it reads ahead of that wait -- weights and biases -- must have been
// complete before its predecessor began; the callers see to that.  Without
// them a 960x540x64 forward pass takes about 20 us more.
//
// 960x540x64 forward: 164 us a call, 141 of them in the four kernels.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <atomic>
#include <mutex>

#include "ginf_internal.h"
#include "ptx.cuh"

namespace ginf_gpu {

struct ConvTcParams {
    // [COUT][9][CIN], tap = (dy + 1) * 3 + dx + 1; EPI_MASK: the layer's own
    // weights, [CIN][9][COUT], whose flipped transpose is the data gradient's.
    const __nv_bfloat16 *wt;
    const float *bias;       // COUT, or null
    const float *res;        // FP32 residual [pixel][COUT] added after the activation, or null
    void *out;               // [pixel][COUT], FP32 or BF16
    const float *x;          // IN_F32: the input, [pixel][CIN]
    __nv_bfloat16 *x_bf16;   // IN_F32: its BF16 rounding, or null
    const __nv_bfloat16 *act;  // EPI_MASK: the activations whose ReLU the gradient passes
    const float *target;       // EPI_LOSS: [pixel][COUT]
    float scale;               // EPI_LOSS: 2 / elements
    int wide_squares;          // EPI_LOSS: square in FP64, not four at a time in FP32 ahead of the FP64 sum
    float *bias_part;          // EPI_MASK, EPI_LOSS: [CTA][COUT] sums of the gradient written
    double *loss_part;         // EPI_LOSS: [CTA] sums of squared differences
    int n, h, w;             // images, rows, columns
    int band, bands, chunks, rows_per_chunk, items;  // band: pixels of a full one
    int *status;
};

namespace {

// What the epilogue makes of the convolution.
enum {
    EPI_STORE = 0,  // + bias, ReLU or residual; stored
    EPI_MASK = 1,   // a data gradient through the ReLU below: zero where that activation is not
                    // positive, stored as BF16, its sum per channel being the bias gradient
    EPI_LOSS = 2    // the last layer in training: + bias + residual, the difference to the target,
                    // its square's sum (the loss) and 2 / n times itself as BF16 (the output gradient),
                    // whose sum per channel is the bias gradient
};

constexpr int kTileM = 128;            // pixels per tile (MMA M)
constexpr int kSlab = kTileM + 2;      // pixels per row copy at most: the band and one either side
constexpr int kThreadsTc = 192;        // weight gradient: warps 0-3 epilogue, 4 copies, 5 MMA
constexpr int kCopyWarp = 4, kMmaWarp = 5;

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

// One box of the 4-D row map (channels, x, row, image): a row of the band.
__device__ __forceinline__ void tma_load_row(uint32_t dst, const CUtensorMap *map, int x, int row, int img,
                                             uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
        "[%6];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(0), "r"(x), "r"(row), "r"(img), "r"(smem_addr(bar))
        : "memory");
}

// Shared-memory matrix descriptor: start address, leading byte offset
// (between core matrices adjacent in K; unused when a swizzle row holds the
// instruction's K), stride byte offset (between 8-row groups in M or N),
// version 1, swizzle mode (0 none, 2 128-byte, 4 64-byte, 6 32-byte).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo, uint32_t swizzle = 0) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) |
           (1ull << 46) | ((uint64_t)swizzle << 61);
}

// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both
// K-major, M = 128, N = n.
__host__ __device__ constexpr uint32_t instr_desc_bf16(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kTileM >> 4) << 24);
}

__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}

// Arrives on bar once every tcgen05 operation this thread issued before is done.
__device__ __forceinline__ void umma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar))
                 : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 16 consecutive FP32 columns of this warp's 32 lanes (one lane per thread),
// waited for before returning.
__device__ __forceinline__ void tmem_load16(uint32_t taddr, float *v) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

struct Item {
    int img, x0, y0, rows;
};

// Work item: (image, band of up to 128 pixels, chunk of rows_per_chunk rows), chunks
// of one band adjacent so that neighbouring CTAs share halo rows in L2.
__device__ __forceinline__ Item item_of(const ConvTcParams &p, int it) {
    Item r;
    const int chunk = it % p.chunks, rest = it / p.chunks;
    r.x0 = (rest % p.bands) * p.band;
    r.img = rest / p.bands;
    r.y0 = chunk * p.rows_per_chunk;
    r.rows = min(p.rows_per_chunk, p.h - r.y0);
    return r;
}

// Warps of a convolution: epilogue, row copies, MMA.  With FP32 input eight
// warps round the rows on their way to shared memory, and the epilogue has
// four: with eight there too a 960x540x64 forward pass took 4 % longer.  The
// others have eight: with four or sixteen 16x256x192x64 gradients took 3 % longer.
constexpr int epi_warps(bool in_f32) { return in_f32 ? 4 : 8; }
constexpr int copy_warps(bool in_f32) { return in_f32 ? 8 : 1; }
constexpr int conv_threads(bool in_f32) { return (epi_warps(in_f32) + copy_warps(in_f32) + 1) * 32; }

template <int CIN, int COUT, bool OUT_F32, int RING, bool IN_F32>
struct TcLayout {
    static constexpr int kEpi = epi_warps(IN_F32), kCopy = copy_warps(IN_F32);
    static constexpr int kThreads = conv_threads(IN_F32);  // epilogue, copies, MMA
    static constexpr int kCW = COUT * 4 / kEpi > 16 ? COUT * 4 / kEpi : 16;  // channels per epilogue warp
    static constexpr int kTileWarps = COUT / kCW * 4;    // epilogue warps of a tile
    static constexpr int kTeams = kEpi / kTileWarps;     // tiles are taken in turn by as many teams of warps
    static_assert(kEpi % kTileWarps == 0, "whole teams");
    static constexpr int kChunks = CIN / 8;
    static constexpr int kPixBytes = CIN * 2;                          // one pixel: one swizzle row
    static constexpr uint32_t kSwizzle = CIN == 64 ? 2 : (CIN == 32 ? 4 : 6);
    static constexpr int kRowBytes = (kSlab * kPixBytes + 1023) / 1024 * 1024;  // one row buffer, 1024-byte aligned
    static constexpr int kWBytes = 9 * CIN * COUT * 2;      // [tap][chunk][co][16 B]
    static constexpr int kRows = 0;
    static constexpr int kW = kRows + RING * kRowBytes;
    static constexpr int kBias = kW + kWBytes;
    static constexpr int kOutBytes = kCW * (OUT_F32 ? 4 : 2);  // one pixel's outputs of one warp
    static constexpr int kChunksOut = kOutBytes / 16;
    static constexpr int kStagePitch = kOutBytes + 16;
    static constexpr int kStage = (kBias + COUT * 4 + 15) / 16 * 16;  // epilogue warps x 32 pixel rows
    static constexpr int kBars = kStage + kEpi * 32 * kStagePitch;
    static constexpr int kAcc = COUT == 64 ? 4 : 8;  // accumulator slots in tensor memory
    static constexpr int kNumBars = 2 * RING + 2 * kAcc + 1;  // full, empty, acc_full, acc_empty, done
    static constexpr int kTmemSlot = kBars + kNumBars * 8;
    static constexpr int kAbort = kTmemSlot + 4;
    static constexpr int kBytes = kAbort + 4;
    static constexpr uint32_t kCols = kAcc * COUT;  // 128 or 256 columns: two CTAs fit an SM's 512
    static_assert((kCols & (kCols - 1)) == 0 && kCols >= 32, "tensor-memory allocation is a power of two");
};

// Tensor-memory column of output row (tile) t's accumulator: slots run
// downwards, so the accumulators of rows r + 1, r, r - 1 -- the three an
// input row r feeds -- are adjacent and ascending unless the ring wraps.
template <int COUT, int ACC>
__device__ __forceinline__ uint32_t acc_col(uint32_t t) {
    return (uint32_t)(ACC - 1 - (int)(t % ACC)) * COUT;
}

__device__ __forceinline__ uint2 pack_bf16x4(const float *v) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
    return make_uint2(*reinterpret_cast<const uint32_t *>(&a), *reinterpret_cast<const uint32_t *>(&b));
}

// OUT_F32: FP32 results are staged (and stored, with EPI_STORE).
// IN_F32: the input is FP32; warps round its rows to BF16 on the way into the
// row buffers (no map).
template <int CIN, int COUT, bool RELU, bool OUT_F32, int RING, int EPI, bool IN_F32>
__global__ void __launch_bounds__(conv_threads(IN_F32), 2)
    k_conv_tc(const __grid_constant__ CUtensorMap rows_map, const ConvTcParams p) {
    using Lay = TcLayout<CIN, COUT, OUT_F32, RING, IN_F32>;
    static_assert((CIN == 16 || CIN == 32 || CIN == 64) && COUT % 16 == 0 && COUT <= 256, "tile shape");
    static_assert(EPI == EPI_STORE || (OUT_F32 && !RELU), "the gradients are formed from FP32 rows");
    extern __shared__ __align__(1024) unsigned char sm[];
    uint64_t *bars = reinterpret_cast<uint64_t *>(sm + Lay::kBars);
    uint64_t *full = bars, *empty = bars + RING, *acc_full = bars + 2 * RING, *acc_empty = acc_full + Lay::kAcc,
             *done = acc_empty + Lay::kAcc;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(sm + Lay::kTmemSlot);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(sm + Lay::kAbort);
    float *bias = reinterpret_cast<float *>(sm + Lay::kBias);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned char *stage = sm + Lay::kStage + warp * 32 * Lay::kStagePitch;  // epilogue warps only

    // Weights into [dx][chunk][j * COUT + co][8 channels]: for one column
    // offset dx the three row offsets dy = j - 1 stacked along N, so one MMA
    // applies all three to an input row.  The bias (zero without one).
    for (int e = threadIdx.x; e < 9 * Lay::kChunks * COUT; e += blockDim.x) {
        const int n = e % (3 * COUT), t = e / (3 * COUT), c8 = t % Lay::kChunks, dx = t / Lay::kChunks;
        const int j = n / COUT, co = n % COUT;
        uint4 q;
        if constexpr (EPI == EPI_MASK) {
            uint32_t w2[4];
            const uint16_t *wt =
                reinterpret_cast<const uint16_t *>(p.wt) + ((size_t)c8 * 72 + 8 - j * 3 - dx) * COUT + co;
#pragma unroll
            for (int k = 0; k < 4; ++k)
                w2[k] = (uint32_t)wt[2 * k * 9 * COUT] | ((uint32_t)wt[(2 * k + 1) * 9 * COUT] << 16);
            q = make_uint4(w2[0], w2[1], w2[2], w2[3]);
        } else {
            q = *reinterpret_cast<const uint4 *>(p.wt + ((size_t)co * 9 + j * 3 + dx) * CIN + c8 * 8);
        }
        *reinterpret_cast<uint4 *>(sm + Lay::kW + (size_t)e * 16) = q;
    }
    for (int c = threadIdx.x; c < COUT; c += blockDim.x) bias[c] = p.bias ? p.bias[c] : 0.f;
    if (threadIdx.x == 0) {
        for (int i = 0; i < RING; ++i) {
            mbar_init(&full[i], IN_F32 ? Lay::kCopy * 32 : 1);
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < Lay::kAcc; ++i) {
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_empty[i], Lay::kTileWarps * 32);
        }
        mbar_init(done, 1);
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)),
                     "r"(Lay::kCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_proxy_async_shared();  // the weights, written by threads, are read by the tensor cores
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    if (smem_addr(sm) & 1023u) {  // swizzled row buffers start on 1024-byte boundaries
        if (threadIdx.x == 0 && p.status) atomicOr(p.status, DEV_ERR_BOUNDS);
        *abort_flag = 1;
    }
    __syncthreads();
    grid_dependency_wait();
    launch_dependents();

    if (IN_F32 && warp >= Lay::kEpi && warp < Lay::kEpi + Lay::kCopy) {
        // Rows through registers: quad q of the row is channels 4 (q % kQuads)
        // on of pixel q / kQuads, 8 bytes of the buffer, where the copy's
        // swizzle would put them (address bits 4-6 xor bits 7-9, as many as a
        // swizzle row's chunks take).  All of a thread's loads are in flight
        // at once, ahead of the wait for the buffer.
        constexpr int kCopyThreads = Lay::kCopy * 32, kQuads = CIN / 4;
        constexpr int kEach = (kSlab * kQuads + kCopyThreads - 1) / kCopyThreads;
        constexpr int kAhead = 1;  // rows the L2 prefetch runs ahead
        const int t0 = threadIdx.x - Lay::kEpi * 32, row_quads = (p.band + 2) * kQuads;
        uint32_t ld = 0;
        bool ok = true;
        for (int it = blockIdx.x; it < p.items && ok && !__any_sync(~0u, *abort_flag); it += gridDim.x) {
            const Item t = item_of(p, it);
            for (int r = t.y0 - 1; r <= t.y0 + t.rows; ++r, ++ld) {
                const int ra = r + kAhead;
                if (t0 == 0 && ra >= 0 && ra < p.h && ra <= t.y0 + t.rows) {
                    const int xl = t.x0 > 0 ? t.x0 - 1 : 0, xr = t.x0 + p.band + 1 < p.w ? t.x0 + p.band + 1 : p.w;
                    bulk_prefetch_l2(p.x + (((size_t)t.img * p.h + ra) * p.w + xl) * CIN,
                                     (uint32_t)((xr - xl) * CIN * 4));
                }
                // Quads of the row inside the image: [qlo, qhi).
                const int left = t.x0 == 0 ? kQuads : 0, right = (p.w - t.x0 + 1) * kQuads;
                const int qlo = r >= 0 && r < p.h ? left : row_quads, qhi = right < row_quads ? right : row_quads;
                const ptrdiff_t row = (((ptrdiff_t)t.img * p.h + r) * p.w + t.x0 - 1) * CIN;  // of quad 0
                float4 v[kEach];
#pragma unroll
                for (int i = 0; i < kEach; ++i) {
                    const int q = t0 + i * kCopyThreads;
                    v[i] = q >= qlo && q < qhi ? *reinterpret_cast<const float4 *>(p.x + row + 4 * q)
                                               : make_float4(0.f, 0.f, 0.f, 0.f);
                }
                const int slot = (int)(ld % RING);
                ok = __all_sync(~0u, mbar_wait_bounded(&empty[slot], ((ld / RING) & 1u) ^ 1u, p.status));
                if (!ok) {
                    *abort_flag = 1;
                    break;
                }
                // The rounding kept: the band's own pixels of the strip's own rows, each once.
                const bool keep = p.x_bf16 && r >= t.y0 && r < t.y0 + t.rows;
                const int khi = qhi < (p.band + 1) * kQuads ? qhi : (p.band + 1) * kQuads;
#pragma unroll
                for (int i = 0; i < kEach; ++i) {
                    const int q = t0 + i * kCopyThreads;
                    if (q >= row_quads) break;
                    const uint2 b = pack_bf16x4(&v[i].x);
                    uint32_t at = (uint32_t)q * 8;
                    at ^= ((at >> 7) & (Lay::kChunks - 1)) << 4;
                    *reinterpret_cast<uint2 *>(sm + Lay::kRows + slot * Lay::kRowBytes + at) = b;
                    if (keep && q >= kQuads && q < khi) *reinterpret_cast<uint2 *>(p.x_bf16 + row + 4 * q) = b;
                }
                fence_proxy_async_shared();  // written by threads, read by the tensor cores
                mbar_arrive(&full[slot]);
            }
        }
    } else if (warp == Lay::kEpi) {
        if (lane == 0) {
            uint32_t ld = 0;
            for (int it = blockIdx.x; it < p.items && !*abort_flag; it += gridDim.x) {
                const Item t = item_of(p, it);
                for (int r = t.y0 - 1; r <= t.y0 + t.rows; ++r, ++ld) {
                    const int slot = (int)(ld % RING);
                    if (!mbar_wait_bounded(&empty[slot], ((ld / RING) & 1u) ^ 1u, p.status)) {
                        *abort_flag = 1;
                        break;
                    }
                    mbar_arrive_expect_tx(&full[slot], (uint32_t)(p.band + 2) * Lay::kPixBytes);
                    tma_load_row(smem_addr(sm + Lay::kRows + slot * Lay::kRowBytes), &rows_map, t.x0 - 1, r, t.img,
                                 &full[slot]);
                }
            }
            // Copies still in flight land before the CTA's shared memory goes.
            for (uint32_t q = ld > RING ? ld - RING : 0; q < ld; ++q)
                mbar_wait_bounded(&full[q % RING], (q / RING) & 1u, nullptr);
        }
        __syncwarp();
    } else if (warp == Lay::kEpi + Lay::kCopy) {
        // The whole warp keeps count and one lane issues: with everything in
        // one lane's branch each instruction's descriptors went through
        // vector registers (960x540x64 forward 5 %, 16x256x192x64 gradients 2 %
        // longer).
        const bool leader = elect_one();
        constexpr int ACC = Lay::kAcc;
        const uint32_t rbase = smem_addr(sm + Lay::kRows);
        // Weights: [dx][chunk][3 * COUT rows][16 B], K-adjacent chunks 3 * COUT * 16 bytes apart.
        const uint64_t bdesc = smem_desc(smem_addr(sm + Lay::kW), 3 * COUT * 16, 128);
        uint32_t ld = 0, tile = 0;
        bool ok = true;
        for (int it = blockIdx.x; it < p.items && ok && !__any_sync(~0u, *abort_flag); it += gridDim.x) {
            const Item t = item_of(p, it);
            // Input row r = y0 - 1 + i feeds output rows y = r + 1 - j
            // (dy = j - 1), j in [jlo, jhi] within the strip; output row
            // y0 + m is tile `tile + m`.
            for (int i = 0; i < t.rows + 2 && ok; ++i, ++ld) {
                const int jlo = i - (t.rows - 1) > 0 ? i - (t.rows - 1) : 0, jhi = i < 2 ? i : 2;
                ok = __all_sync(~0u, mbar_wait_bounded(&full[ld % RING], (ld / RING) & 1u, p.status));
                // Block j = 0 starts row y0 + i's accumulator: its slot must be read out.
                if (ok && jlo == 0) {
                    const uint32_t tn = tile + i;
                    ok = __all_sync(~0u, mbar_wait_bounded(&acc_empty[tn % ACC], ((tn / ACC) & 1u) ^ 1u, p.status));
                }
                if (!ok) break;
                tc_fence_after();
                // The blocks j in [jlo, jhi] as at most two runs with
                // adjacent accumulators (the ring wraps at most once),
                // fixed for the row; every step then issues one MMA per
                // run, its descriptors the row's plus constant offsets.
                int k0 = jlo;
                while (k0 < jhi && (tile + i - k0) % ACC != 0) ++k0;
                const int n0 = k0 - jlo + 1, n1 = jhi - k0;  // blocks in run 0, run 1
                const uint32_t d0 = tmem + acc_col<COUT, ACC>(tile + i - jlo);
                const uint32_t d1 = tmem + acc_col<COUT, ACC>(tile + i - k0 - 1);
                const uint32_t i0 = instr_desc_bf16(n0 * COUT), i1 = instr_desc_bf16(n1 > 0 ? n1 * COUT : 16);
                const uint64_t a0 = smem_desc(rbase + (ld % RING) * Lay::kRowBytes, 16, 8 * Lay::kPixBytes,
                                              Lay::kSwizzle);
                const uint64_t b0 = bdesc + (uint64_t)(jlo * COUT), b1 = bdesc + (uint64_t)((k0 + 1) * COUT);
                if (leader) {
#pragma unroll
                    for (int dx = 0; dx < 3; ++dx)
#pragma unroll
                        for (int ks = 0; ks < CIN / 16; ++ks) {
                            // Offsets in 16-byte units of the descriptors' address fields.
                            const uint64_t ao = (uint64_t)((dx * Lay::kPixBytes + ks * 32) >> 4);
                            const uint64_t bo = (uint64_t)((dx * Lay::kChunks + 2 * ks) * 3 * COUT);
                            if (dx == 0 && ks == 0 && jlo == 0) {
                                // Block 0 starts output row y0 + i: overwrite.
                                umma_bf16(d0, a0, b0, instr_desc_bf16(COUT), 0u);
                                if (n0 > 1)
                                    umma_bf16(d0 + COUT, a0, b0 + (uint64_t)COUT, instr_desc_bf16((n0 - 1) * COUT), 1u);
                            } else {
                                umma_bf16(d0, a0 + ao, b0 + bo, i0, 1u);
                            }
                            if (n1 > 0) umma_bf16(d1, a0 + ao, b1 + bo, i1, 1u);
                        }
                    umma_commit(&empty[ld % RING]);  // the row's only MMAs are these
                    if (jhi == 2) umma_commit(&acc_full[(tile + i - 2) % ACC]);  // row y0 + i - 2 is done
                }
                __syncwarp();
            }
            tile += t.rows;
        }
        if (!ok) *abort_flag = 1;
        if (leader) umma_commit(done);
        mbar_wait_bounded(done, 0, nullptr);
        __syncwarp();
    } else {
        // Epilogue: warp w reads lanes 32 (w % 4) .. + 31 of the accumulator,
        // channels c0 .. c0 + CW - 1.
        constexpr int CW = Lay::kCW;
        const int quarter = warp & 3, c0 = warp % Lay::kTileWarps / 4 * CW;
        const uint32_t team = warp / Lay::kTileWarps;
        uint32_t tile = 0;
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
        // EPI_MASK, EPI_LOSS: this lane's four channels (chunk lane % kChunksOut
        // of a pixel, the same in every pass) and its squares.
        float bsum[4] = {0.f, 0.f, 0.f, 0.f};
        double loss = 0.0;
        // The tensor-memory loads are warp-collective: every decision to stop
        // is taken by the whole warp.
        for (int it = blockIdx.x; it < p.items && !__any_sync(~0u, *abort_flag); it += gridDim.x) {
            const Item t = item_of(p, it);
            for (int j = 0; j < t.rows; ++j, ++tile) {
                if (Lay::kTeams > 1 && tile % Lay::kTeams != team) continue;
                const uint32_t acc = tile % Lay::kAcc;
                if (!__all_sync(~0u, mbar_wait_bounded(&acc_full[acc], (tile / Lay::kAcc) & 1u, p.status))) {
                    *abort_flag = 1;
                    break;
                }
                tc_fence_after();
                float v[CW];
#pragma unroll
                for (int c = 0; c < CW; c += 16)
                    tmem_load16(tmem + lane_base + acc_col<COUT, Lay::kAcc>(tile) + c0 + c, v + c);
                tc_fence_before();
                mbar_arrive(&acc_empty[acc]);
#pragma unroll
                for (int c = 0; c < CW; ++c) {
                    v[c] += bias[c0 + c];
                    if (RELU) v[c] = fmaxf(v[c], 0.f);
                }
                // This lane's pixel into the warp's staging rows (a pitch of
                // one 16-byte chunk more than a pixel's outputs keeps eight
                // consecutive lanes on distinct banks) ...
                unsigned char *row = stage + lane * Lay::kStagePitch;
#pragma unroll
                for (int c = 0; c < Lay::kChunksOut; ++c) {
                    uint4 q;
                    if (OUT_F32) {
                        q = make_uint4(__float_as_uint(v[4 * c]), __float_as_uint(v[4 * c + 1]),
                                       __float_as_uint(v[4 * c + 2]), __float_as_uint(v[4 * c + 3]));
                    } else {
                        uint32_t w4[4];
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            w4[k] = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(v[8 * c + 2 * k])) |
                                    ((uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(v[8 * c + 2 * k + 1])) << 16);
                        q = make_uint4(w4[0], w4[1], w4[2], w4[3]);
                    }
                    *reinterpret_cast<uint4 *>(row + c * 16) = q;
                }
                __syncwarp();
                // ... then the warp's 32 pixels, contiguous in the output,
                // written 512 bytes per instruction (the residual read the
                // same way).
                const int x = t.x0 + quarter * 32;
                const int ends = t.x0 + p.band < p.w ? t.x0 + p.band : p.w;  // of the band
                const int valid = ends - x < 32 ? ends - x : 32;
                const size_t pix = ((size_t)t.img * p.h + t.y0 + j) * p.w + x;
                // 16-byte chunk q of the warp's block: pixel q / kChunksOut,
                // chunk q % kChunksOut of its channels, at(q) in the tensor.
                constexpr int kPixChunks = Lay::kChunksOut * (COUT / CW);  // of a whole pixel
                auto at = [&](int q) { return (q / Lay::kChunksOut) * kPixChunks + q % Lay::kChunksOut; };
                const size_t first = pix * COUT + c0;
                uint4 *o = reinterpret_cast<uint4 *>(static_cast<unsigned char *>(p.out) + first * (OUT_F32 ? 4 : 2));
                const uint4 *rs = OUT_F32 && p.res ? reinterpret_cast<const uint4 *>(p.res + first) : nullptr;
                const int nq = valid * Lay::kChunksOut;
                if constexpr (EPI != EPI_STORE) {
                    // Passes in groups whose loads are all in flight at once;
                    // a row's sums first, then the running ones.
                    constexpr int kMost = EPI == EPI_LOSS ? 4 : 8;
                    constexpr int kGroup = Lay::kChunksOut < kMost ? Lay::kChunksOut : kMost;
                    float rsum[4] = {0.f, 0.f, 0.f, 0.f};
                    uint2 *g = reinterpret_cast<uint2 *>(static_cast<__nv_bfloat16 *>(p.out) + first);
                    const uint2 *act = EPI == EPI_MASK ? reinterpret_cast<const uint2 *>(p.act + first) : nullptr;
                    const float4 *res = EPI == EPI_LOSS ? reinterpret_cast<const float4 *>(p.res + first) : nullptr;
                    const float4 *tgt = EPI == EPI_LOSS ? reinterpret_cast<const float4 *>(p.target + first) : nullptr;
#pragma unroll
                    for (int i0 = 0; i0 < Lay::kChunksOut; i0 += kGroup) {
                        uint2 av[kGroup];
                        float4 xv[kGroup], tv[kGroup];
#pragma unroll
                        for (int i = 0; i < kGroup; ++i) {
                            const int q = lane + 32 * (i0 + i);
                            if (q < nq) {
                                if (EPI == EPI_MASK) av[i] = act[at(q)];
                                if (EPI == EPI_LOSS) {
                                    xv[i] = res[at(q)];
                                    tv[i] = tgt[at(q)];
                                }
                            }
                        }
#pragma unroll
                        for (int i = 0; i < kGroup; ++i) {
                            const int q = lane + 32 * (i0 + i);
                            if (q < nq) {
                                const float4 f = *reinterpret_cast<const float4 *>(
                                    stage + (q / Lay::kChunksOut) * Lay::kStagePitch + (q % Lay::kChunksOut) * 16);
                                float o[4] = {f.x, f.y, f.z, f.w};
                                if (EPI == EPI_MASK) {
#pragma unroll
                                    for (int k = 0; k < 4; ++k) {
                                        const uint32_t w2 = k < 2 ? av[i].x : av[i].y;
                                        const uint16_t bits = (uint16_t)(w2 >> (16 * (k & 1)));
                                        if (!(__bfloat162float(__ushort_as_bfloat16(bits)) > 0.f)) o[k] = 0.f;
                                    }
                                } else {
                                    const float4 a = xv[i], b = tv[i];
                                    const float d[4] = {(f.x + a.x) - b.x, (f.y + a.y) - b.y, (f.z + a.z) - b.z,
                                                        (f.w + a.w) - b.w};
                                    if (p.wide_squares) {
#pragma unroll
                                        for (int k = 0; k < 4; ++k) loss += (double)d[k] * (double)d[k];
                                    } else {
                                        loss += (double)(d[0] * d[0] + d[1] * d[1] + d[2] * d[2] + d[3] * d[3]);
                                    }
#pragma unroll
                                    for (int k = 0; k < 4; ++k) o[k] = p.scale * d[k];
                                }
#pragma unroll
                                for (int k = 0; k < 4; ++k) rsum[k] += o[k];
                                g[at(q)] = pack_bf16x4(o);
                            }
                        }
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k) bsum[k] += rsum[k];
                    __syncwarp();
                    continue;
                }
                uint4 r[Lay::kChunksOut];  // all residual loads in flight before the first store
                if (OUT_F32 && rs) {
#pragma unroll
                    for (int i = 0; i < Lay::kChunksOut; ++i)
                        if (lane + 32 * i < nq) r[i] = rs[at(lane + 32 * i)];
                }
#pragma unroll
                for (int i = 0; i < Lay::kChunksOut; ++i) {
                    const int q = lane + 32 * i;
                    if (q >= nq) break;
                    uint4 val = *reinterpret_cast<const uint4 *>(stage + (q / Lay::kChunksOut) * Lay::kStagePitch +
                                                                 (q % Lay::kChunksOut) * 16);
                    if (OUT_F32 && rs)
                        val = make_uint4(__float_as_uint(__uint_as_float(val.x) + __uint_as_float(r[i].x)),
                                         __float_as_uint(__uint_as_float(val.y) + __uint_as_float(r[i].y)),
                                         __float_as_uint(__uint_as_float(val.z) + __uint_as_float(r[i].z)),
                                         __float_as_uint(__uint_as_float(val.w) + __uint_as_float(r[i].w)));
                    o[at(q)] = val;
                }
                __syncwarp();
            }
        }
        if constexpr (EPI != EPI_STORE) {
            // The CTA's sums, in a fixed order: lanes of one channel chunk, then
            // the warps of the same channels.
#pragma unroll
            for (int off = Lay::kChunksOut; off < 32; off <<= 1)
#pragma unroll
                for (int k = 0; k < 4; ++k) bsum[k] += __shfl_xor_sync(~0u, bsum[k], off);
            float *red = reinterpret_cast<float *>(stage);
            if (lane < Lay::kChunksOut)
#pragma unroll
                for (int k = 0; k < 4; ++k) red[4 * lane + k] = bsum[k];
            double *lred = reinterpret_cast<double *>(stage + CW * 4);
            if (EPI == EPI_LOSS) {
                double l = loss;
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) l += __shfl_xor_sync(~0u, l, off);
                if (lane == 0) *lred = l;
            }
            asm volatile("bar.sync 1, %0;" ::"n"(Lay::kEpi * 32) : "memory");  // the epilogue's warps
            constexpr int kWarpStage = 32 * Lay::kStagePitch;
            if (threadIdx.x < COUT) {
                float t = 0.f;
#pragma unroll
                for (int w = 0; w < 4 * Lay::kTeams; ++w)
                    t += reinterpret_cast<const float *>(
                        sm + Lay::kStage +
                        (w / 4 * Lay::kTileWarps + threadIdx.x / CW * 4 + w % 4) * kWarpStage)[threadIdx.x % CW];
                p.bias_part[(size_t)blockIdx.x * COUT + threadIdx.x] = t;
            }
            if (EPI == EPI_LOSS && threadIdx.x == 0) {
                double t = 0.0;
                for (int w = 0; w < Lay::kEpi; ++w)
                    t += *reinterpret_cast<const double *>(sm + Lay::kStage + w * kWarpStage + CW * 4);
                p.loss_part[blockIdx.x] = t;
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(Lay::kCols) : "memory");
    }
}

// Per device, once: the kernel's dynamic shared-memory limit and a
// preference for the largest shared-memory split (without it the driver may
// pick a split that holds one of these CTAs per SM, not two).
struct TcKernelSetup {
    SmemLimit smem;
    Carveout carveout;
    template <typename K>
    cudaError_t ensure(K kern, int bytes) {
        const cudaError_t e = smem.ensure(kern, (size_t)bytes);
        return e != cudaSuccess ? e : carveout.ensure(kern, (int)cudaSharedmemCarveoutMaxShared);
    }
};

PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
        cudaGetLastError();
    });
    return fn;
}

// Rows map over an NHWC BF16 tensor (channels, x, row, image), box of `box_px`
// pixels, swizzled by a pixel's bytes (C = 16, 32 or 64).
bool encode_rows_map(CUtensorMap *map, const void *base, int C, int n, int h, int w, int box_px) {
    PFN_cuTensorMapEncodeTiled_v12000 encode = tensor_map_encoder();
    if (!encode) return false;
    const cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)w, (cuuint64_t)h, (cuuint64_t)n};
    const cuuint64_t strides[3] = {(cuuint64_t)C * 2, (cuuint64_t)w * C * 2, (cuuint64_t)h * w * C * 2};
    const cuuint32_t box[4] = {(cuuint32_t)C, (cuuint32_t)box_px, 1, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    const CUtensorMapSwizzle swz =
        C == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : (C == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void *>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, swz, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// CTA slots of a kernel with `smem` bytes of shared memory: two per SM at most.
cudaError_t cta_slots(int smem, int *slots) {
    int dev = 0, sms = 0, smem_sm = 0, reserved = 0;
    cudaError_t e;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev)) != cudaSuccess)
        return e;
    if ((e = cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev)) != cudaSuccess)
        return e;
    int per_sm = smem_sm / (smem + reserved);
    per_sm = per_sm < 1 ? 1 : (per_sm > 2 ? 2 : per_sm);
    *slots = sms * per_sm;
    return cudaSuccess;
}

// Work items for `slots` CTAs: each band's rows split into chunks (two halo rows
// each), at most one per four rows begun, as many as make the longest CTA
// shortest -- its items times a chunk's rows with their halo.  False when there
// is nothing to do or too much to count.  16 images of 256x192 on 304 slots are
// 288 items of 22 rows; an even split of the rows over the slots, rounded up,
// gives 320 of 21, two chunks' time, and the gradients took 1.4 times as long.
//
// Bands are as even as whole groups of 16 pixels (the weight gradient's K
// step) allow: 192 columns are two bands of 96, not 128 and 64, whose CTAs
// keep unlike SMs busy unlike long (16 images of 192x256 with 64 labels:
// forward 223 us, 248 with those; gradients 550, 602; four of 144x300 227, 249).
struct ItemPlan {
    int band, bands, rows_per_chunk, chunks, items, grid;
};

bool plan_items(int n, int h, int w, int slots, ItemPlan &pl) {
    if (n < 1 || h < 1 || w < 1 || slots < 1) return false;
    pl.bands = (w + kTileM - 1) / kTileM;
    pl.band = ((w + pl.bands - 1) / pl.bands + 15) / 16 * 16;
    const long long strips = (long long)n * pl.bands;
    // The finest split that is done in k waves of CTAs, for the first few k:
    // past them the halo rows cost more than the rounding gains.
    const long long most = (h + 3) / 4, first = (strips + slots - 1) / slots;
    long long best = -1;
    for (long long k = first; k < first + 16; ++k) {
        const long long c = k * slots / strips < most ? k * slots / strips : most;
        const long long rows = (h + c - 1) / c;
        if (best >= 0 && k * (rows + 2) >= best) continue;
        best = k * (rows + 2);
        pl.rows_per_chunk = (int)rows;
        pl.chunks = (int)((h + rows - 1) / rows);
        if (c == most) break;
    }
    const long long items = strips * pl.chunks;
    if (items > 0x7fffffffLL) return false;
    pl.items = (int)items;
    pl.grid = pl.items < slots ? pl.items : slots;
    return true;
}

// parts (may be null): the CTAs launched, each with its partial sums.
template <int CIN, int COUT, bool RELU, bool OUT_F32, int EPI = EPI_STORE, bool IN_F32 = false>
cudaError_t launch_conv_tc(const __nv_bfloat16 *in, ConvTcParams p, cudaStream_t s, int *parts = nullptr) {
    // The deepest ring of row buffers (3 to 8) that leaves room for two CTAs
    // per SM (228 KB of shared memory, 1 KB of it reserved per CTA).
    constexpr int kBudget = 113 * 1024;
    using Most = TcLayout<CIN, COUT, OUT_F32, 8, IN_F32>;
    constexpr int kFit = (kBudget - (Most::kBytes - 8 * Most::kRowBytes)) / Most::kRowBytes;
    constexpr int RING = kFit < 3 ? 3 : (kFit > 8 ? 8 : kFit);
    using Lay = TcLayout<CIN, COUT, OUT_F32, RING, IN_F32>;
    // At least 80 KB, so that no more than two CTAs share an SM's 512
    // tensor-memory columns (a third would wait in its allocation).
    constexpr int kSmem = Lay::kBytes < 80 * 1024 ? 80 * 1024 : Lay::kBytes;
    auto kern = k_conv_tc<CIN, COUT, RELU, OUT_F32, RING, EPI, IN_F32>;
    static TcKernelSetup setup;
    cudaError_t attr_err = setup.ensure(kern, kSmem);
    if (attr_err != cudaSuccess) return attr_err;
    int slots = 0;
    cudaError_t e = cta_slots(kSmem, &slots);
    if (e != cudaSuccess) return e;
    ItemPlan pl;
    if (!plan_items(p.n, p.h, p.w, slots, pl)) return cudaErrorInvalidValue;
    alignas(64) CUtensorMap map{};
    if constexpr (!IN_F32) {
        if (!tensor_map_encoder()) return cudaErrorNotSupported;
        if (!encode_rows_map(&map, in, CIN, p.n, p.h, p.w, pl.band + 2)) return cudaErrorInvalidValue;
    }
    p.band = pl.band;
    p.bands = pl.bands;
    p.rows_per_chunk = pl.rows_per_chunk;
    p.chunks = pl.chunks;
    p.items = pl.items;
    if (parts) *parts = pl.grid;
    if constexpr (IN_F32) {  // the first of a call: nothing before it may be unfinished
        kern<<<pl.grid, Lay::kThreads, kSmem, s>>>(map, p);
        return cudaGetLastError();
    }
    return launch_after(kern, pl.grid, Lay::kThreads, kSmem, s, map, p);
}

// ---------------------------------------------------------------------------
// Weight gradient: dW[co][tap][ci] = sum over pixels p of dout[p][co] *
// in[p shifted by tap][ci], a GEMM with the pixels as K.  Both operands are
// read MN-major (channels contiguous per pixel) from the same swizzled row
// buffers the forward pass uses: A = input rows, M = taps x CIN, where one
// M = 128 tile holds 128 / CIN taps of one row offset dy as MN atoms one
// pixel apart (LBO = a pixel's bytes; the taps past dx = +1 are computed and
// dropped); B = the three output-gradient rows r - 1, r, r + 1 that input row
// r meets (dy = 2, 1, 0), adjacent in the ring of row buffers and so the MN
// atoms of one operand (LBO = a row buffer), N = 3 COUT: one MMA serves the
// three row offsets and reads A once for them.  Where the ring wraps the run
// splits in two.  Each CTA accumulates in tensor memory over all of its rows
// (K steps of 16 pixels) and writes one partial sum; the caller adds the
// partials in a fixed order, so the result is deterministic.
//
// Bound: the shared-memory reads of the operands (4 KB of A and COUT x 96
// bytes of B an MMA).  16x256x192, us a layer (32 -> 64, 32 -> 32, 64 -> 32
// channels): 33, 23, 38, with evenly filled CTAs; before those 46, 35, 56, and
// with one MMA per row offset 59, 57, 90.

struct WgradParams {
    float *partials;  // [CTA][COUT][9][CIN]
    int n, h, w;
    int band, bands, chunks, rows_per_chunk, items;  // band: pixels of a full one
    int *status;
};

template <int CIN, int COUT, int RING>
struct WgLayout {
    static constexpr int kInPix = CIN * 2, kOutPix = COUT * 2;  // bytes per pixel = one swizzle row
    static constexpr uint32_t kSwIn = CIN == 64 ? 2 : (CIN == 32 ? 4 : 6);
    static constexpr uint32_t kSwOut = COUT == 64 ? 2 : (COUT == 32 ? 4 : 6);
    static constexpr int kInRow = (kSlab * kInPix + 1023) / 1024 * 1024;
    static constexpr int kOutRow = (kTileM * kOutPix + 1023) / 1024 * 1024;
    static constexpr int kTaps = 128 / CIN;                // taps per M tile
    static constexpr int kMT = (3 + kTaps - 1) / kTaps;    // M tiles per row offset
    static constexpr int kAcc = 3 * kMT;                   // accumulators of COUT columns
    static constexpr int kIn = 0;
    static constexpr int kOut = kIn + RING * kInRow;
    // Operand reads of the dropped taps run up to 8 pixels past a row
    // buffer's copy; every buffer is padded to 136 pixels or more, and 4 KB
    // of slack follow the last one.
    static constexpr int kBars = kOut + RING * kOutRow + 4096;
    static constexpr int kNumBars = 4 * RING + 1;  // in full / empty, out full / empty, done
    static constexpr int kTmemSlot = kBars + kNumBars * 8;
    static constexpr int kAbort = kTmemSlot + 4;
    static constexpr int kBytes = kAbort + 4;
    static constexpr uint32_t kCols = kAcc * COUT <= 32 ? 32 : (kAcc * COUT <= 64 ? 64 : (kAcc * COUT <= 128 ? 128 : 256));
};

// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both
// MN-major, M = 128, N = n.
__host__ __device__ constexpr uint32_t instr_desc_bf16_mn(int n) {
    return instr_desc_bf16(n) | (1u << 15) | (1u << 16);
}

template <int CIN, int COUT, int RING>
__global__ void __launch_bounds__(kThreadsTc, 2)
    k_conv_wgrad_tc(const __grid_constant__ CUtensorMap in_map, const __grid_constant__ CUtensorMap out_map,
                    const WgradParams p) {
    using Lay = WgLayout<CIN, COUT, RING>;
    static_assert((CIN == 16 || CIN == 32 || CIN == 64) && (COUT == 16 || COUT == 32 || COUT == 64), "shape");
    extern __shared__ __align__(1024) unsigned char sm[];
    uint64_t *bars = reinterpret_cast<uint64_t *>(sm + Lay::kBars);
    uint64_t *in_full = bars, *in_empty = bars + RING, *out_full = bars + 2 * RING, *out_empty = bars + 3 * RING,
             *done = bars + 4 * RING;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(sm + Lay::kTmemSlot);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(sm + Lay::kAbort);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < RING; ++i) {
            mbar_init(&in_full[i], 1);
            mbar_init(&in_empty[i], 1);
            mbar_init(&out_full[i], 1);
            mbar_init(&out_empty[i], 1);
        }
        mbar_init(done, 1);
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)),
                     "r"(Lay::kCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    if (smem_addr(sm) & 1023u) {
        if (threadIdx.x == 0 && p.status) atomicOr(p.status, DEV_ERR_BOUNDS);
        *abort_flag = 1;
    }
    __syncthreads();
    grid_dependency_wait();
    launch_dependents();
    // Items as in the forward pass: a 128-pixel band of one image, a chunk of
    // its rows.  Step i of an item is input row r = y0 - 1 + i.
    ConvTcParams ip{};
    ip.n = p.n;
    ip.h = p.h;
    ip.w = p.w;
    ip.band = p.band;
    ip.bands = p.bands;
    ip.chunks = p.chunks;
    ip.rows_per_chunk = p.rows_per_chunk;

    if (warp == kCopyWarp) {
        if (lane == 0) {
            uint32_t li = 0, lo = 0;  // input rows, output-gradient rows issued
            bool ok = true;
            for (int it = blockIdx.x; it < p.items && ok && !*abort_flag; it += gridDim.x) {
                const Item t = item_of(ip, it);
                for (int i = 0; i < t.rows + 2; ++i) {
                    int slot = (int)(li % RING);
                    ok = mbar_wait_bounded(&in_empty[slot], ((li / RING) & 1u) ^ 1u, p.status);
                    if (!ok) break;
                    mbar_arrive_expect_tx(&in_full[slot], (uint32_t)(p.band + 2) * Lay::kInPix);
                    tma_load_row(smem_addr(sm + Lay::kIn + slot * Lay::kInRow), &in_map, t.x0 - 1, t.y0 - 1 + i, t.img,
                                 &in_full[slot]);
                    ++li;
                    if (i >= t.rows) continue;
                    slot = (int)(lo % RING);
                    ok = mbar_wait_bounded(&out_empty[slot], ((lo / RING) & 1u) ^ 1u, p.status);
                    if (!ok) break;
                    mbar_arrive_expect_tx(&out_full[slot], (uint32_t)p.band * Lay::kOutPix);
                    tma_load_row(smem_addr(sm + Lay::kOut + slot * Lay::kOutRow), &out_map, t.x0, t.y0 + i, t.img,
                                 &out_full[slot]);
                    ++lo;
                }
            }
            if (!ok) *abort_flag = 1;
            for (uint32_t q = li > RING ? li - RING : 0; q < li; ++q)
                mbar_wait_bounded(&in_full[q % RING], (q / RING) & 1u, nullptr);
            for (uint32_t q = lo > RING ? lo - RING : 0; q < lo; ++q)
                mbar_wait_bounded(&out_full[q % RING], (q / RING) & 1u, nullptr);
        }
        __syncwarp();
    } else if (warp == kMmaWarp) {
        const bool leader = elect_one();
        const uint32_t ibase = smem_addr(sm + Lay::kIn), obase = smem_addr(sm + Lay::kOut);
        uint32_t li = 0, lo = 0;  // input row of the step, first output-gradient row of the item
        bool ok = true, first_item = true;
        for (int it = blockIdx.x; it < p.items && ok && !__any_sync(~0u, *abort_flag); it += gridDim.x) {
            const Item t = item_of(ip, it);
            for (int i = 0; i < t.rows + 2 && ok; ++i, ++li) {
                ok = __all_sync(~0u, mbar_wait_bounded(&in_full[li % RING], (li / RING) & 1u, p.status));
                if (ok && i < t.rows)
                    ok = __all_sync(
                        ~0u, mbar_wait_bounded(&out_full[(lo + i) % RING], ((lo + i) / RING) & 1u, p.status));
                if (!ok) break;
                tc_fence_after();
                // Blocks b: output-gradient row y0 + i - 2 + b, dy = 2 - b,
                // accumulator columns b * COUT on.
                const int blo = i < 2 ? 2 - i : 0, bhi = t.rows + 1 - i < 2 ? t.rows + 1 - i : 2;
                const uint64_t a0 = smem_desc(ibase + (li % RING) * Lay::kInRow, Lay::kInPix, 8 * Lay::kInPix,
                                              Lay::kSwIn);
                // Runs of adjacent row buffers; a block's first use starts
                // its accumulator, in a run of its own.
                const bool fresh = first_item && i < 3;
                if (leader) {
                    for (int b = blo; b <= bhi;) {
                        const uint32_t slot = (lo + i - 2 + b) % RING;
                        const bool start = fresh && b == blo;
                        int n = start ? 1 : bhi - b + 1;
                        if ((int)slot + n > RING) n = RING - (int)slot;
                        const uint64_t b0 = smem_desc(obase + slot * Lay::kOutRow, Lay::kOutRow, 8 * Lay::kOutPix,
                                                      Lay::kSwOut);
                        const uint32_t idesc = instr_desc_bf16_mn(n * COUT);
#pragma unroll
                        for (int mt = 0; mt < Lay::kMT; ++mt)
#pragma unroll
                            for (int ks = 0; ks < kTileM / 16; ++ks) {
                                if (ks * 16 >= p.band) break;
                                // Offsets in 16-byte units: tap block mt starts
                                // mt * kTaps pixels in, K step ks 16 pixels on.
                                const uint64_t ao = (uint64_t)((mt * Lay::kTaps + 16 * ks) * Lay::kInPix >> 4);
                                const uint64_t bo = (uint64_t)(16 * ks * Lay::kOutPix >> 4);
                                umma_bf16(tmem + (mt * 3 + b) * COUT, a0 + ao, b0 + bo, idesc, start && ks == 0 ? 0u : 1u);
                            }
                        b += n;
                    }
                    umma_commit(&in_empty[li % RING]);
                    if (blo == 0) umma_commit(&out_empty[(lo + i - 2) % RING]);  // its last use
                }
                __syncwarp();
            }
            first_item = false;
            lo += t.rows;
        }
        if (!ok) *abort_flag = 1;
        if (leader) umma_commit(done);
        __syncwarp();
    } else {
        // Epilogue, once: accumulator (mt, dy), lane m = 32 * warp + lane is
        // tap dx = mt * kTaps + m / CIN, channel m % CIN.
        const bool ok = __all_sync(~0u, mbar_wait_bounded(done, 0, p.status));
        if (ok && !__any_sync(~0u, *abort_flag)) {
            tc_fence_after();
            const int m = warp * 32 + lane, ci = m % CIN;
            float *part = p.partials + (size_t)blockIdx.x * COUT * 9 * CIN;
#pragma unroll 1
            for (int a = 0; a < Lay::kAcc; ++a) {
                const int dy = 2 - a % 3, dx = (a / 3) * Lay::kTaps + m / CIN;
                float v[COUT];
#pragma unroll
                for (int c = 0; c < COUT; c += 16)
                    tmem_load16(tmem + ((uint32_t)(warp * 32) << 16) + a * COUT + c, v + c);
                if (dx < 3) {
#pragma unroll
                    for (int co = 0; co < COUT; ++co) part[((size_t)co * 9 + dy * 3 + dx) * CIN + ci] = v[co];
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(Lay::kCols) : "memory");
    }
}

template <int CIN, int COUT>
cudaError_t launch_wgrad_tc(const __nv_bfloat16 *dout, const __nv_bfloat16 *in, WgradParams p, int max_parts,
                            int *parts, cudaStream_t s) {
    constexpr int kBudget = 113 * 1024;
    constexpr int kFixed = WgLayout<CIN, COUT, 8>::kBytes - 8 * (WgLayout<CIN, COUT, 8>::kInRow + WgLayout<CIN, COUT, 8>::kOutRow);
    constexpr int kFit = (kBudget - kFixed) / (WgLayout<CIN, COUT, 8>::kInRow + WgLayout<CIN, COUT, 8>::kOutRow);
    constexpr int RING = kFit < 3 ? 3 : (kFit > 8 ? 8 : kFit);
    using Lay = WgLayout<CIN, COUT, RING>;
    constexpr int kSmem = Lay::kBytes < 80 * 1024 ? 80 * 1024 : Lay::kBytes;
    auto kern = k_conv_wgrad_tc<CIN, COUT, RING>;
    static TcKernelSetup setup;
    cudaError_t attr_err = setup.ensure(kern, kSmem);
    if (attr_err != cudaSuccess) return attr_err;
    int slots = 0;
    cudaError_t e = cta_slots(kSmem, &slots);
    if (e != cudaSuccess) return e;
    if (slots > max_parts) slots = max_parts;
    ItemPlan pl;
    if (!plan_items(p.n, p.h, p.w, slots, pl)) return cudaErrorInvalidValue;
    alignas(64) CUtensorMap in_map, out_map;
    if (!encode_rows_map(&in_map, in, CIN, p.n, p.h, p.w, pl.band + 2) ||
        !encode_rows_map(&out_map, dout, COUT, p.n, p.h, p.w, pl.band))
        return cudaErrorInvalidValue;
    p.band = pl.band;
    p.bands = pl.bands;
    p.rows_per_chunk = pl.rows_per_chunk;
    p.chunks = pl.chunks;
    p.items = pl.items;
    *parts = pl.grid;
    return launch_after(kern, pl.grid, kThreadsTc, kSmem, s, in_map, out_map, p);
}

}  // namespace

// 3x3 convolution of NHWC BF16 input with weights [COUT][9][CIN] on the
// tcgen05 path: hidden layers (cout 32, ReLU, BF16 out) and the last layer
// (cin 32, FP32 out, + res); cudaErrorInvalidValue for a channel pair it is
// not built for.
cudaError_t conv_fwd_tc(int cin, int cout, bool relu, const __nv_bfloat16 *in, const __nv_bfloat16 *w,
                        const float *bias, int nimg, int h, int wd, void *out, const float *res, int *status,
                        cudaStream_t s) {
    if (((uintptr_t)in | (uintptr_t)w | (uintptr_t)out | (uintptr_t)res) & 15) return cudaErrorMisalignedAddress;
    ConvTcParams p{};
    p.wt = w;
    p.bias = bias;
    p.res = res;
    p.out = out;
    p.n = nimg;
    p.h = h;
    p.w = wd;
    p.status = status;
    if (relu) {
        if (cin != 32 || cout != 32) return cudaErrorInvalidValue;
        return launch_conv_tc<32, 32, true, false>(in, p, s);
    }
    if (cin != 32) return cudaErrorInvalidValue;
    if (cout == 16) return launch_conv_tc<32, 16, false, true>(in, p, s);
    if (cout == 32) return launch_conv_tc<32, 32, false, true>(in, p, s);
    if (cout == 64) return launch_conv_tc<32, 64, false, true>(in, p, s);
    return cudaErrorInvalidValue;
}

// The first layer (cin -> 32, ReLU, BF16 out) from the FP32 x, whose BF16
// rounding goes to x_bf16 unless that is null.
cudaError_t conv_first_tc(int cin, const float *x, __nv_bfloat16 *x_bf16, const __nv_bfloat16 *w, const float *bias,
                          int nimg, int h, int wd, __nv_bfloat16 *out, int *status, cudaStream_t s) {
    if (((uintptr_t)x | (uintptr_t)x_bf16 | (uintptr_t)w | (uintptr_t)out) & 15) return cudaErrorMisalignedAddress;
    ConvTcParams p{};
    p.wt = w;
    p.bias = bias;
    p.x = x;
    p.x_bf16 = x_bf16;
    p.out = out;
    p.n = nimg;
    p.h = h;
    p.w = wd;
    p.status = status;
    if (cin == 16) return launch_conv_tc<16, 32, true, false, EPI_STORE, true>(nullptr, p, s);
    if (cin == 32) return launch_conv_tc<32, 32, true, false, EPI_STORE, true>(nullptr, p, s);
    if (cin == 64) return launch_conv_tc<64, 32, true, false, EPI_STORE, true>(nullptr, p, s);
    return cudaErrorInvalidValue;
}

// The last layer in training (32 -> cout): grad = BF16 of 2 / n (y - target)
// with y = conv + bias + x, per-CTA sums of it per channel in bias_part
// ([parts][cout]) and of the squared differences in loss_part ([parts]).
cudaError_t conv_loss_tc(int cout, const __nv_bfloat16 *in, const __nv_bfloat16 *w, const float *bias, int nimg, int h,
                         int wd, const float *x, const float *target, bool wide_squares, float scale,
                         __nv_bfloat16 *grad, float *bias_part, double *loss_part, int *parts, int *status,
                         cudaStream_t s) {
    if (((uintptr_t)in | (uintptr_t)w | (uintptr_t)x | (uintptr_t)target | (uintptr_t)grad) & 15)
        return cudaErrorMisalignedAddress;
    ConvTcParams p{};
    p.wt = w;
    p.bias = bias;
    p.res = x;
    p.target = target;
    p.scale = scale;
    p.wide_squares = wide_squares;
    p.out = grad;
    p.bias_part = bias_part;
    p.loss_part = loss_part;
    p.n = nimg;
    p.h = h;
    p.w = wd;
    p.status = status;
    if (cout == 16) return launch_conv_tc<32, 16, false, true, EPI_LOSS>(in, p, s, parts);
    if (cout == 32) return launch_conv_tc<32, 32, false, true, EPI_LOSS>(in, p, s, parts);
    if (cout == 64) return launch_conv_tc<32, 64, false, true, EPI_LOSS>(in, p, s, parts);
    return cudaErrorInvalidValue;
}

// Data gradient (cin channels of output gradient -> 32) of the layer with
// weights w ([cin][9][32]), through the ReLU that made act: grad as BF16 and
// its per-CTA sums per channel.
cudaError_t conv_dgrad_tc(int cin, const __nv_bfloat16 *in, const __nv_bfloat16 *w, int nimg, int h, int wd,
                          const __nv_bfloat16 *act, __nv_bfloat16 *grad, float *bias_part, int *parts, int *status,
                          cudaStream_t s) {
    if (((uintptr_t)in | (uintptr_t)w | (uintptr_t)act | (uintptr_t)grad) & 15) return cudaErrorMisalignedAddress;
    ConvTcParams p{};
    p.wt = w;
    p.act = act;
    p.out = grad;
    p.bias_part = bias_part;
    p.n = nimg;
    p.h = h;
    p.w = wd;
    p.status = status;
    if (cin == 16) return launch_conv_tc<16, 32, false, true, EPI_MASK>(in, p, s, parts);
    if (cin == 32) return launch_conv_tc<32, 32, false, true, EPI_MASK>(in, p, s, parts);
    if (cin == 64) return launch_conv_tc<64, 32, false, true, EPI_MASK>(in, p, s, parts);
    return cudaErrorInvalidValue;
}

// Weight gradient of the 3x3 convolution on the tcgen05 path: per-CTA
// partial sums [parts][COUT][9][CIN] into `partials` (room for max_parts),
// their count in *parts; cudaErrorInvalidValue for a channel pair it is not
// built for.
cudaError_t conv_wgrad_tc(int cin, int cout, const __nv_bfloat16 *dout, const __nv_bfloat16 *in, int nimg, int h,
                          int wd, float *partials, int max_parts, int *parts, int *status, cudaStream_t s) {
    if (((uintptr_t)dout | (uintptr_t)in) & 15) return cudaErrorMisalignedAddress;
    WgradParams p{};
    p.partials = partials;
    p.n = nimg;
    p.h = h;
    p.w = wd;
    p.status = status;
#define GINF_WG_TC_CASE(CI, CO) \
    if (cin == CI && cout == CO) return launch_wgrad_tc<CI, CO>(dout, in, p, max_parts, parts, s);
    GINF_WG_TC_CASE(16, 32)
    GINF_WG_TC_CASE(32, 32)
    GINF_WG_TC_CASE(64, 32)
    GINF_WG_TC_CASE(32, 16)
    GINF_WG_TC_CASE(32, 64)
#undef GINF_WG_TC_CASE
    return cudaErrorInvalidValue;
}

}  // namespace ginf_gpu
