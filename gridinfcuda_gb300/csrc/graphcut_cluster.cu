// graphcut_cluster.cu -- the alpha-beta swap of graphcut.cu on one thread-block
// cluster, for grids whose state fits its shared memory: the same results, with
// the ten push and ten relabel sweeps between two global relabels in flight at
// once.
//
// The grid is cut into bands of up to 32 rows, one CTA each, and everything the
// reference keeps per node -- excess, height, the four residues and the sink's,
// the label -- lives in the CTA's shared memory.  A sweep in raster order is a
// wavefront over anti-diagonals, and a later sweep may follow two diagonals
// behind: sweep j may take diagonal k once
//   - sweep j has taken diagonal k - 1 (raster-earlier neighbours are done),
//   - sweep j - 1 has taken diagonal k + 1 (nothing it does touches k later).
// So warp j of every CTA runs sweep j, one lane per row, the warps chained by
// progress counters in shared memory and the bands by mailbox words.
//
// What crosses a band's edge travels as one word per column: the flow pushed
// over the edge, the sender's height after its sweep, and the sweep's number.
// The band below waits for its upper neighbour's word of the same sweep, the
// band above for its lower neighbour's word of the sweep before; a word is read
// before its column's next one can be written (which waits, through the other
// direction's word, for exactly that), so one word per column and direction is
// enough, and no fence is needed between CTAs inside a round.
//
// Concurrent sweeps add to the same excess only by atomics (the additions
// commute; the node is next read after all of them), each residue slot has one
// writer at a time, and heights change only in the order above.
//
// The global relabel and the final reachability are level-synchronous searches
// on bit sets, 32 nodes to a word and a word to a thread, with one cluster
// barrier per level; the few per-pair reductions ride on such barriers.  Every wait inside a round is bounded; one
// that runs out is recorded and the round ends with all CTAs.
//
// Bound: the latency of a wavefront step (shared-memory loads, a handful of
// dependent operations, a progress counter) and the searches' barriers.
// AB_MEASURED
#include <cstdint>

#include "ginf_internal.h"
#include "ptx.cuh"

namespace ginf_gpu {

namespace {

constexpr int kSweeps = 20;  // ten pushes, ten relabels (graphcut.h:8)
constexpr int kThreadsCl = kSweeps * 32;
constexpr int kMaxBands = 16;  // largest cluster
constexpr int kMaxRows = 32;   // rows per band: a lane each
constexpr uint64_t kAlphaBetaLimitNs = 60ull * 1000000000ull;
constexpr int kTagBits = 14, kHeightBits = 18;

struct Head {
    int red[32];
    int slots[2][kMaxBands];  // what the CTAs tell one another (cl_exchange)
    int prog[kSweeps];        // last diagonal each sweep has taken
    int give_up;
};

// Offsets of the arrays in dynamic shared memory; R rows per band, row pitch P.
struct Layout {
    // masks: [6][R][words]; front: [2][R + 2][words].
    uint32_t box_n, box_s, ghost_s, masks, front, ex, ht, res, f, bytes;
    __host__ __device__ Layout(int R, int P, int words) {
        const uint32_t n = (uint32_t)R * P, w = 4u * words;
        box_n = 512;
        box_s = box_n + 8u * P;
        ghost_s = box_s + 8u * P;
        masks = ghost_s + 4u * P;
        front = masks + 6u * R * w;
        ex = front + 2u * (R + 2) * w;
        ht = ex + 4u * n;
        res = ht + 4u * n;
        f = res + 5u * 4u * n;
        bytes = (f + n + 15u) / 16u * 16u;
    }
};
static_assert(sizeof(Head) <= 512, "header");

// Node sets as 32-column words per row: which nodes have residue in direction
// d (0 .. 3), which a search has not reached, which of them reach the sink.
enum { kMaskOpen = 4, kMaskReach = 5 };

// Row pitch: even, so that a diagonal's nodes (stride P - 1 words) lie in
// distinct banks.
__host__ __device__ inline int pitch_of(int W) { return (W + 1) & ~1; }

__device__ __forceinline__ uint64_t make_word(int tag, int height, int flow) {
    return ((uint64_t)(uint32_t)(tag & ((1 << kTagBits) - 1)) << 50) | ((uint64_t)(uint32_t)height << 32) |
           (uint64_t)(uint32_t)flow;
}
__device__ __forceinline__ int word_tag(uint64_t w) { return (int)(w >> 50); }
__device__ __forceinline__ int word_height(uint64_t w) { return (int)((w >> 32) & ((1u << kHeightBits) - 1)); }
__device__ __forceinline__ int word_flow(uint64_t w) { return (int)(uint32_t)w; }

__device__ __forceinline__ uint64_t box_load(uint32_t addr) {
    uint64_t v;
    asm volatile("ld.relaxed.cluster.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void box_store(uint32_t addr, uint64_t v) {
    asm volatile("st.relaxed.cluster.shared::cluster.u64 [%0], %1;" ::"r"(addr), "l"(v) : "memory");
}
__device__ __forceinline__ int dsmem_i32(uint32_t addr) {
    int v;
    asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ int dsmem_u8(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared::cluster.u8 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return (int)v;
}
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t v;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(v));
    return v;
}

struct Band {
    int W, H, L, N, NP2, C;   // grid, N + 2, CTAs
    int rank, y0, rows, P, R; // this band; rows of a full band
    bool up, down;            // bands above and below
    unsigned char *sm;
    Head *hd;
    int *ex, *ht, *res[5];
    uint8_t *f;
    int words;  // per row
    uint32_t *masks;
    Layout lay;
    uint32_t base, base_up, base_down;  // shared-memory addresses: own, neighbours'
    int parity;
};

// Sum (or, for flags, the bitwise or) of the CTAs' block-uniform v; also a
// cluster barrier.
template <bool SUM>
__device__ __forceinline__ int cl_exchange(Band &b, int v) {
    if ((int)threadIdx.x < b.C) {
        const uint32_t a = dsmem_addr(smem_addr(&b.hd->slots[b.parity][b.rank]), threadIdx.x);
        asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
    }
    cluster_sync();
    int t = 0;
    for (int i = 0; i < b.C; ++i) t = SUM ? t + b.hd->slots[b.parity][i] : t | b.hd->slots[b.parity][i];
    b.parity ^= 1;
    return t;
}

__device__ __forceinline__ int block_sum_cl(Band &b, int v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(~0u, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) b.hd->red[threadIdx.x >> 5] = v;
    __syncthreads();
    int t = 0;
    for (int i = 0; i < kThreadsCl / 32; ++i) t += b.hd->red[i];
    __syncthreads();
    return t;
}

// The band's rows by warps, columns by lanes.
#define AB_FOR_NODES(r, x)                                             \
    for (int r = threadIdx.x >> 5; r < b.rows; r += kThreadsCl / 32)   \
        for (int x = threadIdx.x & 31; x < b.W; x += 32)

// The current labelling, or with FLOW the one the pair's cut proposes: nodes
// that reach the sink take alpha, the rest of the partition beta
// (graphcut.cc:253-263, 60-72).  Row -1 is the band above's last row, row
// b.rows the band below's first.
template <bool FLOW>
__device__ __forceinline__ int label_at(const Band &b, int r, int x, int alpha, int beta) {
    int f;
    uint32_t reach = 0;
    const uint32_t reach_off = b.lay.masks + 4u * (uint32_t)(kMaskReach * b.R * b.words + (x >> 5));
    if (r < 0) {
        f = dsmem_u8(b.base_up + b.lay.f + (uint32_t)((b.R - 1) * b.P + x));
        if (FLOW) reach = (uint32_t)dsmem_i32(b.base_up + reach_off + 4u * (uint32_t)((b.R - 1) * b.words));
    } else if (r >= b.rows) {
        f = dsmem_u8(b.base_down + b.lay.f + x);
        if (FLOW) reach = (uint32_t)dsmem_i32(b.base_down + reach_off);
    } else {
        f = b.f[r * b.P + x];
        if (FLOW) reach = b.masks[(kMaskReach * b.R + r) * b.words + (x >> 5)];
    }
    if (FLOW && (f == alpha || f == beta)) f = (reach >> (x & 31)) & 1u ? alpha : beta;
    return f;
}

// getLabelingCost (src/grid.cc:102-125) in int32: this band's share.
template <bool FLOW>
__device__ __forceinline__ int band_energy(const AlphaBetaParams &p, Band &b, int alpha, int beta) {
    int acc = 0;
    AB_FOR_NODES(r, x) {
        const int y = b.y0 + r;
        if (x < 1 || y < 1 || x > b.W - 2 || y > b.H - 2) continue;
        const int fl = label_at<FLOW>(b, r, x, alpha, beta), fn = label_at<FLOW>(b, r - 1, x, alpha, beta),
                  fe = label_at<FLOW>(b, r, x + 1, alpha, beta);
        acc += p.D[(size_t)y * b.W + x + (size_t)b.N * fl];
        acc += p.V[fl + (size_t)b.L * fn];
        acc += p.V[fl + (size_t)b.L * fe];
    }
    return block_sum_cl(b, acc);
}

// Breadth-first search from the nodes with sink residue over residual edges,
// on the node sets: a word's owner thread takes the nodes of its 32 columns
// that have residue towards a frontier node.  One level is a few shared-memory
// words, bit operations and a cluster barrier; the edge rows' frontiers go to
// the neighbours' copies before it.
// LEVELS: the distances go into the heights (1 at the start nodes), as
// graphCutGlobalRelabel's (graphcut.cc:91-140).  Leaves the unreached nodes in
// kMaskOpen and the reached ones in kMaskReach.
template <bool LEVELS>
__device__ __forceinline__ void sink_search_cl(Band &b) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int words = b.words, per_mask = b.R * words;
    uint32_t *front = reinterpret_cast<uint32_t *>(b.sm + b.lay.front);
    const int fsize = (b.R + 2) * words;
    for (int q = warp; q < b.rows * words; q += kThreadsCl / 32) {
        const int r = q / words, c = q - r * words;
        const int x = c * 32 + lane, i = r * b.P + x;
        const bool in = x < b.W;
        uint32_t m[5];
#pragma unroll
        for (int d = 0; d < 5; ++d) m[d] = __ballot_sync(~0u, in && b.res[d][i] != 0);
        const uint32_t all = __ballot_sync(~0u, in);
        if (LEVELS && in && ((m[4] >> lane) & 1u)) b.ht[i] = 1;
        if (lane == 0) {
            // Residues that point off the grid (none in the reference) lead nowhere.
            const int y = b.y0 + r;
            b.masks[q] = y + 1 < b.H ? m[0] : 0u;
            b.masks[per_mask + q] = c == words - 1 ? m[1] & ~(1u << ((b.W - 1) & 31)) : m[1];
            b.masks[2 * per_mask + q] = y > 0 ? m[2] : 0u;
            b.masks[3 * per_mask + q] = c == 0 ? m[3] & ~1u : m[3];
            b.masks[kMaskOpen * per_mask + q] = all & ~m[4];
            b.masks[kMaskReach * per_mask + q] = m[4];
            front[words + q] = m[4];
        }
    }
    __syncthreads();
    const int q = threadIdx.x;
    const bool own = q < b.rows * words;
    const int r = own ? q / words : 0, c = own ? q - r * words : 0;
    uint32_t open = 0, mask[4] = {0u, 0u, 0u, 0u}, reach = 0;
    if (own) {
#pragma unroll
        for (int d = 0; d < 4; ++d) mask[d] = b.masks[d * per_mask + q];
        open = b.masks[kMaskOpen * per_mask + q];
        reach = b.masks[kMaskReach * per_mask + q];
    }
    const bool send_up = own && r == 0 && b.up, send_down = own && r == b.rows - 1 && b.down;
    // The neighbours' copies of this word: row R + 1 of the band above (a full
    // band), row 0 of the band below.
    const uint32_t to_up = b.base_up + b.lay.front + 4u * (uint32_t)((b.R + 1) * words + c);
    const uint32_t to_down = b.base_down + b.lay.front + 4u * (uint32_t)c;
    uint32_t mine = reach;
    int cur = 0;
    for (int level = 1;; ++level) {
        if (send_up) asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(to_up + 4u * cur * fsize), "r"(mine) : "memory");
        if (send_down)
            asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(to_down + 4u * cur * fsize), "r"(mine) : "memory");
        if (!cl_exchange<false>(b, __syncthreads_or(mine != 0))) break;
        mine = 0;
        if (own && open) {
            const uint32_t *fr = front + cur * fsize + (r + 1) * words + c;
            const uint32_t f = fr[0];
            const uint32_t left = c > 0 ? fr[-1] >> 31 : 0u, right = c < words - 1 ? fr[1] << 31 : 0u;
            mine = open & ((mask[0] & fr[words]) | (mask[2] & fr[-words]) | (mask[1] & ((f >> 1) | right)) |
                           (mask[3] & ((f << 1) | left)));
            open &= ~mine;
            reach |= mine;
            if (LEVELS)
                for (uint32_t m = mine; m; m &= m - 1) b.ht[r * b.P + c * 32 + __ffs(m) - 1] = level + 1;
        }
        cur ^= 1;
        if (own) front[cur * fsize + (r + 1) * words + c] = mine;
    }
    if (own) {
        b.masks[kMaskOpen * per_mask + q] = open;
        b.masks[kMaskReach * per_mask + q] = reach;
    }
}

// graphCutGlobalRelabel: the distances; the nodes that reach no sink keep
// max(height, N + 2).
__device__ __forceinline__ void global_relabel(Band &b) {
    sink_search_cl<true>(b);
    cluster_sync();  // the band below's unreached nodes
    const int open_row = kMaskOpen * b.R * b.words;
    AB_FOR_NODES(r, x) {
        const int i = r * b.P + x;
        if ((b.masks[open_row + r * b.words + (x >> 5)] >> (x & 31)) & 1u) b.ht[i] = max(b.ht[i], b.NP2);
    }
    // The band below's first-row heights, for sweep 0 (the later sweeps get
    // them by word): raised here too, since they may not have been yet, and
    // stable until this band's words of sweep 1.
    if (b.down) {
        int *ghost = reinterpret_cast<int *>(b.sm + b.lay.ghost_s);
        for (int x = threadIdx.x; x < b.W; x += kThreadsCl) {
            const int h = dsmem_i32(b.base_down + b.lay.ht + 4u * x);
            const uint32_t o = (uint32_t)dsmem_i32(b.base_down + b.lay.masks + 4u * (uint32_t)(open_row + (x >> 5)));
            ghost[x] = (o >> (x & 31)) & 1u ? max(h, b.NP2) : h;
        }
    }
}

// Sweep j of a round (even: pushes, graphcut.cc:143-177; odd: relabels,
// :180-195) over the band's diagonals by one warp.  first_tag numbers the
// round's sweep 0.
__device__ __forceinline__ void sweep(Band &b, int j, int first_tag, int *status) {
    if (b.rows == 0) return;
    const int lane = threadIdx.x & 31;
    const int klast = b.y0 + b.rows - 1 + b.W - 1;
    const bool row = lane < b.rows;
    const bool top = lane == 0 && b.up, bottom = lane == b.rows - 1 && b.down;
    const int tag_n = (first_tag + j) & ((1 << kTagBits) - 1), tag_s = (first_tag + j - 1) & ((1 << kTagBits) - 1);
    const bool push = (j & 1) == 0;
    volatile int *prog = b.hd->prog;
    const int *ghost = reinterpret_cast<const int *>(b.sm + b.lay.ghost_s);
    int seen = j > 0 ? -1 : 0x7fffffff;
    for (int k = b.y0; k <= klast; ++k) {
        const int x = k - b.y0 - lane;
        const bool in = row && x >= 0 && x < b.W;
        const int i = lane * b.P + x;
        const bool wait_n = in && top, wait_s = in && bottom && j > 0;
        const int need = min(k + 1, klast);
        uint64_t wn = 0, ws = 0;
        bool ok_n = !wait_n, ok_s = !wait_s;
        uint64_t t0 = 0;
        for (uint32_t n = 1;; ++n) {
            if (seen < need) seen = prog[j - 1];
            if (!ok_n) {
                wn = box_load(b.base + b.lay.box_n + 8u * x);
                ok_n = word_tag(wn) == tag_n;
            }
            if (!ok_s) {
                ws = box_load(b.base + b.lay.box_s + 8u * x);
                ok_s = word_tag(ws) == tag_s;
            }
            if (__all_sync(~0u, seen >= need && ok_n && ok_s)) break;
            if ((n & 1023u) == 0) {
                const uint64_t now = __shfl_sync(~0u, global_timer_ns(), 0);
                if (t0 == 0) t0 = now;
                const bool late = now - t0 > kWaitLimitNs;
                if (__any_sync(~0u, late || *(volatile int *)&b.hd->give_up)) {
                    if (late && lane == 0) atomicOr(status, DEV_ERR_TIMEOUT);
                    *(volatile int *)&b.hd->give_up = 1;
                    break;
                }
            }
        }
        __threadfence_block();
        int flow_n = 0, flow_s = 0, h = 0;
        if (in) {
            int e = b.ex[i];
            const int e_was = e;
            h = b.ht[i];
            if (wait_n && word_flow(wn)) {
                e += word_flow(wn);
                b.res[2][i] += word_flow(wn);
            }
            if (wait_s && word_flow(ws)) {
                e += word_flow(ws);
                b.res[0][i] += word_flow(ws);
            }
            if (e && h < b.NP2) {
                const int hs = bottom ? (j > 0 ? word_height(ws) : ghost[x]) : (b.y0 + lane + 1 < b.H ? b.ht[i + b.P] : 0);
                const int hn = top ? word_height(wn) : (b.y0 + lane > 0 ? b.ht[i - b.P] : 0);
                const int he = x + 1 < b.W ? b.ht[i + 1] : 0, hw = x > 0 ? b.ht[i - 1] : 0;
                const int rs = b.res[4][i], r0 = b.res[0][i], r1 = b.res[1][i], r2 = b.res[2][i], r3 = b.res[3][i];
                if (push) {
                    if (rs && h == 1) {
                        const int fl = min(rs, e);
                        e -= fl;
                        b.res[4][i] = rs - fl;
                    }
                    // Directions in order S, E, N, W; a zero flow changes nothing.
                    if (r0 && h == hs + 1) {
                        const int fl = min(r0, e);
                        if (fl) {
                            e -= fl;
                            b.res[0][i] = r0 - fl;
                            if (bottom) {
                                flow_s = fl;
                            } else {
                                atomicAdd(&b.ex[i + b.P], fl);
                                b.res[2][i + b.P] += fl;
                            }
                        }
                    }
                    if (r1 && h == he + 1) {
                        const int fl = min(r1, e);
                        if (fl) {
                            e -= fl;
                            b.res[1][i] = r1 - fl;
                            atomicAdd(&b.ex[i + 1], fl);
                            b.res[3][i + 1] += fl;
                        }
                    }
                    if (r2 && h == hn + 1) {
                        const int fl = min(r2, e);
                        if (fl) {
                            e -= fl;
                            b.res[2][i] = r2 - fl;
                            if (top) {
                                flow_n = fl;
                            } else {
                                atomicAdd(&b.ex[i - b.P], fl);
                                b.res[0][i - b.P] += fl;
                            }
                        }
                    }
                    if (r3 && h == hw + 1) {
                        const int fl = min(r3, e);
                        if (fl) {
                            e -= fl;
                            b.res[3][i] = r3 - fl;
                            atomicAdd(&b.ex[i - 1], fl);
                            b.res[1][i - 1] += fl;
                        }
                    }
                } else {
                    if (rs) {
                        h = 1;
                    } else {
                        int mh = b.NP2;
                        if (r0) mh = min(mh, hs);
                        if (r1) mh = min(mh, he);
                        if (r2) mh = min(mh, hn);
                        if (r3) mh = min(mh, hw);
                        h = mh + 1;
                    }
                    b.ht[i] = h;
                }
            }
            if (e != e_was) b.ex[i] = e;
            if (top) box_store(b.base_up + b.lay.box_s + 8u * x, make_word(tag_n, h, flow_n));
            if (bottom) box_store(b.base_down + b.lay.box_n + 8u * x, make_word(tag_n, h, flow_s));
        }
        __threadfence_block();
        __syncwarp();
        if (lane == 0) prog[j] = k;
    }
}

__global__ void __launch_bounds__(kThreadsCl, 1) k_alpha_beta_cluster(const AlphaBetaParams p, int R) {
    extern __shared__ __align__(16) unsigned char ab_smem[];
    const int P = pitch_of(p.W);
    Band b{p.W, p.H, p.L, p.W * p.H, p.W * p.H + 2, 0, 0, 0, 0, P, R, false, false, ab_smem,
           reinterpret_cast<Head *>(ab_smem), nullptr, nullptr, {}, nullptr, (p.W + 31) / 32, nullptr,
           Layout(R, P, (p.W + 31) / 32), 0, 0, 0, 0};
    b.C = (int)gridDim.x;
    b.rank = (int)cluster_rank();
    b.y0 = b.rank * R;
    b.rows = min(R, p.H - b.y0);
    if (b.rows < 0) b.rows = 0;
    b.up = b.rank > 0 && b.rows > 0;
    b.down = b.rows > 0 && b.y0 + b.rows < p.H;
    b.ex = reinterpret_cast<int *>(ab_smem + b.lay.ex);
    b.ht = reinterpret_cast<int *>(ab_smem + b.lay.ht);
    for (int d = 0; d < 5; ++d) b.res[d] = reinterpret_cast<int *>(ab_smem + b.lay.res) + (size_t)d * R * P;
    b.f = ab_smem + b.lay.f;
    b.masks = reinterpret_cast<uint32_t *>(ab_smem + b.lay.masks);
    b.base = smem_addr(ab_smem);
    b.base_up = dsmem_addr(b.base, b.rank > 0 ? b.rank - 1 : 0);
    b.base_down = dsmem_addr(b.base, b.rank + 1 < b.C ? b.rank + 1 : b.rank);
    const uint64_t t_start = global_timer_ns();

    // The reference's matrices start at zero (matrix.cc:21-27); the labels come
    // as bytes.
    for (uint32_t o = threadIdx.x * 16; o < b.lay.bytes; o += kThreadsCl * 16)
        *reinterpret_cast<uint4 *>(ab_smem + o) = make_uint4(0, 0, 0, 0);
    __syncthreads();
    int bad = 0;
    AB_FOR_NODES(r, x) {
        const int f = p.result[(size_t)(b.y0 + r) * p.W + x];
        bad |= f < 0 || f >= p.L;
        b.f[r * P + x] = (uint8_t)f;
    }
    if (cl_exchange<false>(b, __syncthreads_or(bad))) {
        if (threadIdx.x == 0) atomicOr(p.status, DEV_ERR_BOUNDS);
        return;
    }
    int min_cost = cl_exchange<true>(b, band_energy<false>(p, b, 0, 0));
    int tag = 1;  // number of the next round's sweep 0
    bool success = true, stop = false;
    for (int t = 0; t < p.iters && success && !stop; ++t) {
        success = false;
        for (int alpha = 0; alpha < p.L && !stop; ++alpha) {
            for (int beta = alpha + 1; beta < p.L && !stop; ++beta) {
                // graphCutConstructGraph (graphcut.cc:10-45): partition nodes only.
                const int vab = p.V[alpha + (size_t)p.L * beta];
                AB_FOR_NODES(r, x) {
                    const int i = r * P + x, y = b.y0 + r;
                    const int fl = b.f[i];
                    if (fl != alpha && fl != beta) continue;
                    int ac = 0, bc = 0;
#pragma unroll
                    for (int d = 0; d < 4; ++d) {
                        const int nx = x + (d == 1 ? 1 : (d == 3 ? -1 : 0)), nr = r + (d == 0 ? 1 : (d == 2 ? -1 : 0));
                        int cap = 0;
                        if (nx >= 0 && nx < p.W && b.y0 + nr >= 0 && b.y0 + nr < p.H) {
                            const int fn = label_at<false>(b, nr, nx, alpha, beta);
                            if (fn == alpha || fn == beta) {
                                cap = vab;
                            } else {
                                ac += p.V[alpha + (size_t)p.L * fn];
                                bc += p.V[beta + (size_t)p.L * fn];
                            }
                        }
                        b.res[d][i] = cap;
                    }
                    const size_t n = (size_t)y * p.W + x;
                    b.ex[i] = p.D[n + (size_t)b.N * alpha] + ac;
                    b.res[4][i] = p.D[n + (size_t)b.N * beta] + bc;
                    b.ht[i] = 0;
                }
                __syncthreads();
                for (;;) {
                    // graphCutCountActive (graphcut.cc:75-88), with the time
                    // limit and given-up waits in the same exchange.
                    int act = 0;
                    AB_FOR_NODES(r, x) {
                        const int i = r * P + x;
                        act |= b.ex[i] && b.ht[i] < b.NP2;
                    }
                    int say = __syncthreads_or(act) ? 1 : 0;
                    if (b.hd->give_up || (b.rank == 0 && global_timer_ns() - t_start > kAlphaBetaLimitNs)) say |= 2;
                    say = __syncthreads_or(say & 2) ? say | 2 : say;
                    const int all = cl_exchange<false>(b, say);
                    if (all & 2) {
                        if (threadIdx.x == 0 && b.rank == 0) atomicOr(p.status, DEV_ERR_TIMEOUT);
                        stop = true;
                        break;
                    }
                    if (!all) break;
                    global_relabel(b);
                    if (threadIdx.x < kSweeps) b.hd->prog[threadIdx.x] = -1;
                    __syncthreads();
                    sweep(b, threadIdx.x >> 5, tag, p.status);
                    tag += kSweeps;
                    __syncthreads();
                }
                if (stop) break;
                sink_search_cl<false>(b);
                cluster_sync();  // the neighbours' reached nodes
                const int cost = cl_exchange<true>(b, band_energy<true>(p, b, alpha, beta));
                if (cost < min_cost) {
                    min_cost = cost;
                    success = true;
                    AB_FOR_NODES(r, x) b.f[r * P + x] = (uint8_t)label_at<true>(b, r, x, alpha, beta);
                }
                cluster_sync();  // the next pair reads the neighbours' labels
            }
        }
    }
    AB_FOR_NODES(r, x) p.result[(size_t)(b.y0 + r) * p.W + x] = b.f[r * P + x];
    cluster_sync();  // no CTA's shared memory goes while another may address it
}

}  // namespace

cudaError_t launch_alpha_beta_cluster(const AlphaBetaParams &p, cudaStream_t s, bool &done) {
    done = false;
    // Heights reach N + 3 and travel in kHeightBits bits; labels are bytes.
    if ((long)p.W * p.H + 3 >= (1L << kHeightBits) || p.L > 256) return cudaSuccess;
    int dev = 0, most = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e != cudaSuccess) return e;
    // The fewest bands (a power of two) of at most 32 rows that fit: every
    // further band adds its lag to a sweep.
    int C = 1, R = p.H;
    const int words = (p.W + 31) / 32;
    while (C <= kMaxBands && ((R = (p.H + C - 1) / C) > kMaxRows || R * words > kThreadsCl ||
                              Layout(R, pitch_of(p.W), words).bytes > (uint32_t)most))
        C *= 2;
    if (C > kMaxBands) return cudaSuccess;
    auto kern = k_alpha_beta_cluster;
    static SmemLimit limit;
    const size_t smem = Layout(R, pitch_of(p.W), words).bytes;
    e = limit.ensure(kern, smem);
    if (e != cudaSuccess) return e;
    if (C > 8) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess) return e;
    }
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)C);
    lc.blockDim = dim3(kThreadsCl);
    lc.dynamicSmemBytes = smem;
    lc.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    lc.attrs = attr;
    lc.numAttrs = 1;
    int clusters = 0;
    e = cudaOccupancyMaxActiveClusters(&clusters, kern, &lc);
    if (e != cudaSuccess || clusters < 1) {
        cudaGetLastError();
        return cudaSuccess;
    }
    done = true;
    return cudaLaunchKernelEx(&lc, kern, p, R);
}

}  // namespace ginf_gpu
