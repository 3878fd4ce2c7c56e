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
// What crosses a band's edge travels as one 64-bit word per column: the flow
// pushed over the edge (low half), the sender's height after its sweep and the
// sweep's number.  It is read and written by scalar 64-bit accesses: the two
// elements of a vector access are accesses of their own, in no stated order, so
// a reader could meet a new number beside an old flow.
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
// barrier per level; the few per-pair reductions ride on such barriers.  Every
// wait inside a round is bounded; one that runs out is recorded and the round
// ends with all CTAs.
//
// Bound: the latency of a wavefront step with twenty warps on the SM, five to a
// scheduler (ten cycles an instruction, ncu; 0.33 ms a round of twenty sweeps at
// 384x288: 400 steps a band and the lags of 16 bands), and the searches'
// barriers.  384x288x16, one pass from the BP labels, three inputs: 80, 55 and
// 79 ms (one CTA in global memory 787 ms for the first).  Also measured, for the
// first: searches that walk the unreached nodes instead of bit sets 187 ms before
// a step was shortened, 91 with bit sets; from there four diagonals between two
// waits 137 (the lags grow by more than the waits cost), flows formed branch-free
// and applied by predicated additions 99, no fences in a step 3 % less.
//
// Beyond it (state that sixteen bands do not hold, from about 110,000 nodes on;
// heights or labels that their bits do not) one CTA runs the solve (graphcut.cu).
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
constexpr int kHeightBits = 18;  // of a word's upper half; the sweep's number in the other 14

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

// A mailbox word's accesses: its own CTA reads it, a neighbour writes it.
__device__ __forceinline__ uint64_t box_read(uint32_t addr) {
    uint64_t v;
    asm volatile("ld.relaxed.cluster.shared::cluster.b64 %0, [%1];" : "=l"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void box_write(uint32_t addr, uint64_t v) {
    asm volatile("st.relaxed.cluster.shared::cluster.b64 [%0], %1;" ::"r"(addr), "l"(v) : "memory");
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

// Called now and then by a waiting warp: false when the wait, or another of
// this CTA, has taken too long.
__device__ __noinline__ bool sweep_patience(Band &b, uint32_t n, int *status) {
    volatile int *give_up = &b.hd->give_up;
    // 2^25 polls of at least 60 cycles each are more than a second.
    if (n >= (1u << 25) && !*give_up) {
        if ((threadIdx.x & 31) == 0) atomicOr(status, DEV_ERR_TIMEOUT);
        *give_up = 1;
    }
    return __all_sync(~0u, *give_up == 0);
}

// Flow fl from node i over its residue r at res_i into node q.
__device__ __forceinline__ void push_to(int fl, int r, int *res_i, int *ex_q, int *res_q) {
    *res_i = r - fl;
    atomicAdd(ex_q, fl);
    *res_q += fl;
}

// Sweep j of a round (pushes, graphcut.cc:143-177, or relabels, :180-195) over
// the band's diagonals by one warp.  first_tag numbers the round's sweep 0.
//
// A step's latency is the sweeps' rate, and with twenty warps on the SM an
// instruction of it costs about eight cycles, so what every step does is kept
// short: a lane meets at most one neighbouring band, with one word in and one
// out (every band but the last has R >= 2 rows, and the last, which may have one,
// has none below); progress counters end at a value that needs no comparison
// with the last diagonal.
constexpr int kSweepDone = 0x3fffffff;
template <bool PUSH>
__device__ __forceinline__ void sweep(Band &b, int j, int first_tag, int *status) {
    if (b.rows == 0) return;
    const int lane = threadIdx.x & 31, W = b.W, P = b.P, NP2 = b.NP2;
    const int steps = b.rows - 1 + W;
    const int cols = lane < b.rows ? W : 0;
    const bool top = lane == 0 && b.up, bottom = lane == b.rows - 1 && b.down;
    const bool edge_n = b.y0 + lane == 0, edge_s = b.y0 + lane + 1 >= b.H;  // the grid's
    const bool edge = top || bottom, recv = top || (bottom && j > 0);
    // The neighbour's words of this sweep (above) or the last one (below), the
    // band's own of this sweep; a word's upper half is tag and height.
    const uint32_t tag = (uint32_t)(first_tag + j) << kHeightBits;
    const uint32_t want = top ? tag : (uint32_t)(first_tag + j - 1) << kHeightBits;
    uint32_t box = b.base + (top ? b.lay.box_n : b.lay.box_s) - 8u * lane;
    uint32_t out = (top ? b.base_up + b.lay.box_s : b.base_down + b.lay.box_n) - 8u * lane;
    volatile int *before = &b.hd->prog[j > 0 ? j - 1 : 0], *mine = &b.hd->prog[j];
    const int *ghost = reinterpret_cast<const int *>(b.sm + b.lay.ghost_s) - lane;
    int *ex = b.ex + lane * P - lane, *ht = b.ht + lane * P - lane;
    const int array = b.R * P;  // from one residue array to the next
    int *res = b.res[0] + lane * P - lane;
    int seen = j > 0 ? -1 : kSweepDone;
    // Step k is diagonal y0 + k: column k - lane of each row.
    for (int k = 0; k < steps; ++k) {
        const bool in = (unsigned)(k - lane) < (unsigned)cols;
        uint32_t w_hi = 0, w_lo = 0;
        bool ok = !(in && recv);
        for (uint32_t n = 1;; ++n) {
            if (seen <= k) seen = *before;
            if (!ok) {
                const uint64_t w = box_read(box + 8u * k);
                w_lo = (uint32_t)w;
                w_hi = (uint32_t)(w >> 32);
                ok = (w_hi ^ want) < (1u << kHeightBits);
            }
            if (__all_sync(~0u, ok && seen > k)) break;
            if ((n & 4095u) == 0 && !sweep_patience(b, n, status)) break;
        }
        __threadfence_block();
        int e = 0, h = 0;
        if (in) {
            e = ex[k];
            h = ht[k];
        }
        const int e_was = e;
        if (w_lo) {  // flow over the band's edge
            e += (int)w_lo;
            res[(top ? 2 : 0) * array + k] += (int)w_lo;
        }
        int flow = 0;
        if (e && h < NP2) {
            const int h_word = (int)(w_hi & ((1u << kHeightBits) - 1));
            const int hs = bottom ? (j > 0 ? h_word : ghost[k]) : (edge_s ? 0 : ht[k + P]);
            const int hn = top ? h_word : (edge_n ? 0 : ht[k - P]);
            const int he = k - lane + 1 < W ? ht[k + 1] : 0, hw = k > lane ? ht[k - 1] : 0;
            int *r = res + k, *x = ex + k;
            const int rs = r[4 * array], r0 = r[0], r1 = r[array], r2 = r[2 * array], r3 = r[3 * array];
            if (PUSH) {
                if (rs && h == 1) {
                    const int fl = min(rs, e);
                    e -= fl;
                    r[4 * array] = rs - fl;
                }
                // Directions in order S, E, N, W; a zero flow changes nothing,
                // and a flow over the band's edge goes by word.
                if (r0 && h == hs + 1) {
                    const int fl = min(r0, e);
                    e -= fl;
                    if (bottom) {
                        r[0] = r0 - fl;
                        flow = fl;
                    } else if (fl) {
                        push_to(fl, r0, r, x + P, r + 2 * array + P);
                    }
                }
                if (r1 && h == he + 1) {
                    const int fl = min(r1, e);
                    e -= fl;
                    if (fl) push_to(fl, r1, r + array, x + 1, r + 3 * array + 1);
                }
                if (r2 && h == hn + 1) {
                    const int fl = min(r2, e);
                    e -= fl;
                    if (top) {
                        r[2 * array] = r2 - fl;
                        flow = fl;
                    } else if (fl) {
                        push_to(fl, r2, r + 2 * array, x - P, r - P);
                    }
                }
                if (r3 && h == hw + 1) {
                    const int fl = min(r3, e);
                    e -= fl;
                    if (fl) push_to(fl, r3, r + 3 * array, x - 1, r + array - 1);
                }
            } else {
                int mh = NP2;
                if (r0) mh = min(mh, hs);
                if (r1) mh = min(mh, he);
                if (r2) mh = min(mh, hn);
                if (r3) mh = min(mh, hw);
                h = rs ? 1 : mh + 1;
                ht[k] = h;
            }
        }
        if (e != e_was) ex[k] = e;
        if (in && edge) box_write(out + 8u * k, (uint64_t)(tag | (uint32_t)h) << 32 | (uint32_t)flow);
        __threadfence_block();
        __syncwarp();
        if (lane == 0) *mine = k == steps - 1 ? kSweepDone : k;
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
                    if ((threadIdx.x >> 5) & 1) sweep<false>(b, threadIdx.x >> 5, tag, p.status);
                    else sweep<true>(b, threadIdx.x >> 5, tag, p.status);
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
    if (C > kMaxBands || (C > 1 && R < 2)) return cudaSuccess;
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
