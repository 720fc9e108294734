// Learning kernel for one GPU, graphs of up to 1,024 nodes and up to 32 classes: the per-graph dependency chain, shortened.
//
// Online learning is sequential over graphs (tm.py:668-747), so what bounds it is how long one graph takes from its
// predecessor's update to its own: evaluation, votes of all clauses, decisions, updates.  One persistent cooperative
// launch works on one graph at a time; a CTA owns a range of clauses for the whole launch.
//
//   Evaluation.  Graphs are kept TRANSPOSED in shared memory: row(l) holds literal l of every node, RW words.  A warp
//   evaluates a clause: groups of lanes take different include words, the lanes of a group the node words of a row (128
//   bits each), and the groups' results are ANDed - 32 / (RW / 4) included literals per step instead of one.  Graphs of
//   one to three nodes are tested row-wise, lane = include word.
//   Messages (depth > 1) are PULLED.  Clauses publish their node words (plain stores); after a grid barrier CTA b makes
//   the message bits 8b .. 8b+7 of every node: it ORs the node words of the clauses whose hypervectors hold a bit of the
//   window (lists per bit, made once), walks the edges once, a packed word each, with the window as one word per node - a rotation by the edge
//   type (kernels.py:581) is a shift of the window - and stores the bits both transposed, the next layer's rows as the
//   evaluation reads them, and node-major for the feedback.  A second barrier, and every CTA copies the rows.  Nothing is
//   merged with atomics: sending source-node marks to shared rows (fit_resident_kernel) took 40,000 cycles per layer on
//   1,000-node graphs with 2,000 clauses, 143 atomics per word.
//   Votes are exchanged with one relaxed atomic and one poll per class: the accumulators only grow, a CTA subtracts what
//   it read two steps before, so nothing is cleared and nothing has to be released.
//   In the shadow of the exchange: node choice, decision uniforms and the first rounds of Type-I masks of every clause
//   (the positions of these draws do not depend on the class sums), and the transposition of the next graph.
//   Feedback and the next graph's first layer are one pass: a clause's warp decides, updates and evaluates.
//
// What bounds it: instructions of few warps.  One epoch and the way back of the state on one B200, ms, here / in
// fit_resident_kernel or fit_kernel: 10,000 Noisy-XOR graphs (one CTA) 57 / 109; 4,000 images x 2,500 clauses 22 / 44; 200
// sequences of 1,000 nodes 7.6 / 26.7; 300 multigraphs x 20,000 clauses 54 / 160, 36 of them in the kernel, half of that for the
// Philox draws and the automata of some 95 clauses per CTA and graph.
//
// State: automaton planes in shared memory while they fit; otherwise (kHybrid) only the include planes, which the
// evaluation reads, and the other planes are read and written in global memory for the clauses that get feedback.
#pragma once
#include <climits>

#include "gtm_device.cuh"
#include "gtm_fit.cuh"

namespace gtm {

// Most threads of a CTA; they set the register budgets.  80 registers for wide layers, whose work items all warps share (300
// multigraphs, 20,000 clauses: 36.3 ms with 24 warps of 80, 37.2 with 32 of 64), 96 for narrow ones, where a warp does
// everything for its clause and there is hardly more than a clause per warp, 64 where many clauses share a CTA's memory.
constexpr int chain_threads(bool hybrid, bool narrow) { return narrow ? (hybrid ? 1024 : 576) : 768; }
constexpr int kChainStateBits = 8;       // state bits of an automaton: constant, or every step of an addition is a predicate of its own
constexpr int kChainStages = 3;          // graphs in shared memory: current, next, next but one (on its way)
constexpr int kChainRowWise = 3;         // graphs of at most this many nodes are evaluated row-wise
constexpr int kChainMaxType = 24;        // largest edge type of a set whose messages are pulled: the window is 8 + 24 bits
constexpr int kChainRec = 40;            // words per clause of a step: chosen, pos (2), taken, -, -, -, -, draws / feedback [32]

constexpr u32 kNoEdge = ~0u;

struct ChainArgs {
    const int *Y;                // [N][K] +-T targets, absolute graph ids
    int64_t first, count;
    int epochs;
    unsigned long long *votes;   // [2][K] accumulators, zero before the launch
    unsigned *barrier;           // arrival counter, zero before the launch
    int *error;
    int *clause_node, *update, *class_sum_tap;       // taps: the last graph's
    unsigned long long *phase_cycles;
    int timers;
    unsigned long long wait_ns;
    int missing;                 // test hook: waits expect this many arrivals more than there are CTAs
    int clauses_per_cta, clause_words;
    int helper;                  // the last warp has no clauses: it stages graphs and exchanges votes
    int solo;                    // one CTA: its barriers replace the grid's, messages stay in shared memory
    int narrow;                  // kNarrow: a clause's masks come from one packed stream (all layers of one probability, up to 32 words)
    int pre_words, spec_rounds;  // narrow: words of that stream kept per clause; rounds made in the exchange's shadow
    int stage_words, stage_nodes, stage_edges;       // room for a staged graph: literal words, nodes, edge rows
    int max_nodes;
    u32 *node_bits;              // [D-1][C][RW] node words of every clause after each layer but the last
    u32 *rows_t;                 // [D-1][32*MW][RW] message rows, transposed
    u32 *rows_n;                 // [D-1][max_nodes][MW] message rows, node-major
    const u32 *packed;           // [edges] source | destination << 10 | type << 20 of every edge row; kNoEdge: malformed
    const int *bit_off;          // clauses whose hypervector holds message bit b: bit_clause[bit_off[b] ..]
    const int2 *bit_clause;      // (clause, b)
    int tmax;                    // largest edge type
    u32 key[20];                 // Philox round keys: operands in the constant bank instead of two additions a round
};

// Four consecutive draws of the stream of clause c (draw_block without recorded draws, which the older kernels serve).
__device__ __forceinline__ uint4 chain_draws(const ChainArgs &a, u32 c, u64 block)
{
    u32 c0 = (u32)block, c1 = (u32)(block >> 32), c2 = c, c3 = 0;
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const u32 lo0 = 0xD2511F53u * c0, hi0 = __umulhi(0xD2511F53u, c0);
        const u32 lo1 = 0xCD9E8D57u * c2, hi1 = __umulhi(0xCD9E8D57u, c2);
        c0 = hi1 ^ c1 ^ a.key[2 * r]; c1 = lo1;
        c2 = hi0 ^ c3 ^ a.key[2 * r + 1]; c3 = lo0;
    }
    return make_uint4(c0, c1, c2, c3);
}

__device__ __forceinline__ u32 chain_draw_at(const ChainArgs &a, u32 c, u64 i)
{
    const uint4 o = chain_draws(a, c, i >> 2);
    const u32 even = (i & 2) ? o.z : o.x, odd = (i & 2) ? o.w : o.y;
    return (i & 1) ? odd : even;
}

// Mask word of a lane in a stretch of 32 words: outcomes [draw <= p] of the 32 draws that start `shift` (0..3) draws into
// Philox block `block` (the lane's own; the next lane's block is 8 further on).  A lane makes the eight blocks of its own
// word, so nothing is packed or exchanged but the `shift` bits that spill into the next word.
__device__ __forceinline__ u32 lane_mask(const ChainArgs &a, int c, u64 block, int shift, u32 below, int lane)
{
    u32 word = 0;
#pragma unroll 2
    for (int q = 0; q < 8; ++q) {
        const uint4 o = chain_draws(a, (u32)c, block + q);
        word >>= 4;                                     // block q ends up at bits 4q .. 4q+3
        if (o.x < below) word |= 1u << 28;
        if (o.y < below) word |= 1u << 29;
        if (o.z < below) word |= 1u << 30;
        if (o.w < below) word |= 1u << 31;
    }
    if (shift == 0) return word;
    u32 next = __shfl_down_sync(kFull, word, 1);
    if (lane == 31) {
        const uint4 o = chain_draws(a, (u32)c, block + 8);
        next = (o.x < below ? 1u : 0u) | (o.y < below ? 2u : 0u) | (o.z < below ? 4u : 0u);
    }
    return __funnelshift_r(word, next, shift);
}

// The same for a lane whose neighbour's word is elsewhere in the stream.
__device__ __forceinline__ u32 own_mask(const ChainArgs &a, int c, u64 block, int shift, u32 below)
{
    u32 word = 0, next = 0;
#pragma unroll 1
    for (int q = 0; q < (shift ? 9 : 8); ++q) {
        const uint4 o = chain_draws(a, (u32)c, block + q);
        const u32 nib = (o.x < below ? 1u : 0u) | (o.y < below ? 2u : 0u) | (o.z < below ? 4u : 0u) | (o.w < below ? 8u : 0u);
        if (q < 8) word |= nib << (4 * q);
        else next = nib;
    }
    return __funnelshift_r(word, next, shift);
}

// Rounds [q0, q1) of a clause's packed stream that starts at Philox block `block0`: words 4q .. 4q+3 of dst.
__device__ __forceinline__ void stream_rounds(const ChainArgs &a, int c, u64 block0, int q0, int q1, u32 below, u32 *dst, int lane)
{
#pragma unroll 2
    for (int q = q0; q < q1; ++q) {
        const uint4 o = chain_draws(a, (u32)c, block0 + (u64)q * 32 + lane);
        u32 w = (o.x < below ? 1u : 0u) | (o.y < below ? 2u : 0u) | (o.z < below ? 4u : 0u) | (o.w < below ? 8u : 0u);
        w <<= 4 * (lane & 7);
        w |= __shfl_xor_sync(kFull, w, 1);
        w |= __shfl_xor_sync(kFull, w, 2);
        w |= __shfl_xor_sync(kFull, w, 4);
        if ((lane & 7) == 0) dst[4 * q + (lane >> 3)] = w;
    }
}

// Position of the (rank+1)-th set bit of a word (it has one).
__device__ __forceinline__ int nth_set_bit(u32 word, int rank, int lane)
{
    return __ffs(__ballot_sync(kFull, ((word >> lane) & 1u) != 0 && __popc(word & ((1u << lane) - 1u)) == rank)) - 1;
}

// Automata of up to 32 words of one clause, a word per lane that has one (`mine`; w, W, lo and inc belong to the word's layer
// and may differ from lane to lane), all classes in order (kernels.py:98-183): planes 0..SB-2 at lo[b * W + w], the include
// plane at inc[w].  `masks(rank)` gives the lane's mask word of the Type-I class of that rank.  Returns the
// change of the lane's include count (bits of `valid`).
template <class Masks>
__device__ __forceinline__ int update_words(int boost, int w, int W, bool mine, u32 *lo, u32 *inc, u32 x, int upd, bool clause_true, bool within,
                                            u32 valid, Masks masks)
{
    constexpr int SB = kChainStateBits;
    u32 pl[SB - 1];
#pragma unroll
    for (int b = 0; b < SB - 1; ++b) pl[b] = mine ? lo[(size_t)b * W + w] : 0u;
    u32 in = mine ? inc[w] : 0u;
    const u32 before = in;
    bool dirty = false;
    int rank = 0;
    // the include plane is the top bit of the counters
    auto add = [&](u32 active) {
        u32 carry = active;
#pragma unroll
        for (int b = 0; b < SB - 1; ++b) { const u32 nx = pl[b] & carry; pl[b] ^= carry; carry = nx; }
        const u32 over = in & carry;
        in ^= carry;
#pragma unroll
        for (int b = 0; b < SB - 1; ++b) pl[b] |= over;
        in |= over;
    };
    auto sub = [&](u32 active) {
        u32 borrow = active;
#pragma unroll
        for (int b = 0; b < SB - 1; ++b) { const u32 nx = ~pl[b] & borrow; pl[b] ^= borrow; borrow = nx; }
        const u32 under = ~in & borrow;
        in ^= borrow;
#pragma unroll
        for (int b = 0; b < SB - 1; ++b) pl[b] &= ~under;
        in &= ~under;
    };
    u32 todo = __ballot_sync(kFull, upd != 0);
    while (todo) {
        const int k = __ffs(todo) - 1;
        todo &= todo - 1;
        const int u = __shfl_sync(kFull, upd, k);
        if (u > 0) {
            const u32 mask = masks(rank);
            ++rank;
            if (clause_true && within) {
                add(boost == 1 ? x : (x & ~mask));
                sub(~x & mask);
            } else {
                sub(mask);
            }
            dirty = true;
        } else if (clause_true) {
            add(~x & ~in);
            dirty = true;
        }
    }
    if (mine && dirty) {
#pragma unroll
        for (int b = 0; b < SB - 1; ++b) lo[(size_t)b * W + w] = pl[b];
        inc[w] = in;
    }
    return mine ? __popc(in & valid) - __popc(before & valid) : 0;
}

// ---------------------------------------------------------------------------------------------- evaluation
// ANDs the rows of the set bits of include word `w` (of a layer of W words over WT source words; MS = 0: layer 0) into r.
template <int RW, class V>
__device__ __forceinline__ void and_included(V &r, u32 iw, int w, const u32 *T, int WT, int MS, int MW, int q)
{
    auto take = [&](const u32 *at, u32 flip) {
        if constexpr (RW == 1) {
            r &= *at ^ flip;
        } else {
            const uint4 x = *reinterpret_cast<const uint4 *>(at);
            r.x &= x.x ^ flip; r.y &= x.y ^ flip; r.z &= x.z ^ flip; r.w &= x.w ^ flip;
        }
    };
    const int step = WT * RW;
    if ((MS & 31) == 0) {
        const bool neg = MS > 0 && w >= MW;                  // a whole word of complements
        const u32 flip = neg ? kFull : 0u;
        const u32 *base = T + (neg ? w - MW : w) * RW + 4 * q;
        while (iw) {
            const int b0 = __ffs(iw) - 1;
            iw &= iw - 1;
            const int b1 = iw ? __ffs(iw) - 1 : b0;
            iw &= iw - 1;
            take(base + b0 * step, flip);
            take(base + b1 * step, flip);
        }
    } else {
        while (iw) {
            const int l = 32 * w + __ffs(iw) - 1;
            iw &= iw - 1;
            const int p = l < MS ? l : l - MS;
            take(T + ((p & 31) * WT + (p >> 5)) * RW + 4 * q, l < MS ? 0u : kFull);
        }
    }
}

// One clause on a transposed graph: nodes[0..RW) (in: the layer below, unless `first`; out: this layer), `type` = the rows
// of the clause's node type.  Returns whether any node is left (warp-uniform).
template <int RW>
__device__ __forceinline__ bool eval_clause_rows(const u32 *T, int WT, const u32 *inc, int W, u32 last_mask, int MS, int MW, const u32 *type,
                                                 u32 *nodes, bool first, int lane)
{
    constexpr int Q = RW == 1 ? 1 : RW / 4;          // lanes of a group
    constexpr int G = 32 / Q;                        // groups
    const int g = lane / Q, q = lane % Q;
    // layers of fewer words than groups: several groups share a word, each takes a run of its bits
    const int wp = W >= G ? G : (W <= 1 ? 1 : 1 << (32 - __clz(W - 1)));
    const int piece_bits = min(32, 32 * wp / G);
    const u32 piece = piece_bits == 32 ? kFull : ((1u << piece_bits) - 1u) << ((g / wp) * piece_bits & 31);
    if constexpr (RW == 1) {
        u32 r = type[0];
        if (!first) r &= nodes[0];
        if (r != 0) {
            u32 acc = kFull;
            for (int w = g & (wp - 1); w < W; w += G) {
                const u32 iw = inc[w] & (w == W - 1 ? last_mask : kFull) & piece;
                and_included<RW>(acc, iw, w, T, WT, MS, MW, 0);
            }
            r &= __reduce_and_sync(kFull, acc);
        }
        if (lane == 0) nodes[0] = r;
        return r != 0;
    } else {
        uint4 r = *reinterpret_cast<const uint4 *>(type + 4 * q);
        if (!first) {
            const uint4 p = *reinterpret_cast<const uint4 *>(nodes + 4 * q);
            r.x &= p.x; r.y &= p.y; r.z &= p.z; r.w &= p.w;
        }
        bool alive = __any_sync(kFull, (r.x | r.y | r.z | r.w) != 0);
        for (int w0 = 0; w0 < W && alive; w0 += G) {
            const int w = w0 + (g & (wp - 1));
            if (w < W) {
                const u32 iw = inc[w] & (w == W - 1 ? last_mask : kFull) & piece;
                and_included<RW>(r, iw, w, T, WT, MS, MW, q);
            }
            __syncwarp();
#pragma unroll
            for (int d = Q; d < 32; d <<= 1) {
                r.x &= __shfl_xor_sync(kFull, r.x, d); r.y &= __shfl_xor_sync(kFull, r.y, d);
                r.z &= __shfl_xor_sync(kFull, r.z, d); r.w &= __shfl_xor_sync(kFull, r.w, d);
            }
            alive = __any_sync(kFull, (r.x | r.y | r.z | r.w) != 0);
        }
        __syncwarp();
        if (lane < Q) *reinterpret_cast<uint4 *>(nodes + 4 * q) = r;
        return alive;
    }
}

// The same on a graph of at most three nodes, row-wise: `row(v, w)` = word w of node v's literal vector of the layer.
template <class Row>
__device__ __forceinline__ bool eval_clause_rowwise(const u32 *inc, int W, u32 last_mask, u32 type, u32 *nodes, bool first, int lane, Row row)
{
    u32 r = type;
    if (!first) r &= nodes[0];
    if (r != 0) {
        u32 fail = 0;                                    // bit v: node v fails on one of this lane's words
        for (int w = lane; w < W; w += 32) {
            const u32 iw = inc[w] & (w == W - 1 ? last_mask : kFull);
#pragma unroll
            for (int v = 0; v < kChainRowWise; ++v)
                if ((r >> v) & 1u) fail |= (iw & ~row(v, w)) != 0 ? 1u << v : 0u;
        }
        r &= ~__reduce_or_sync(kFull, fail);
    }
    if (lane == 0) nodes[0] = r;
    return r != 0;
}

// Rows [v][0..W) of n nodes -> T, by `threads` threads (whole warps): a thread takes 32 nodes x 32 literals; the 32 lanes of a warp take
// 8 words x 4 node words, which keeps reads in 32-byte sectors and the bank conflicts of the stores at eight.
template <int RW>
__device__ __forceinline__ void transpose_rows(const u32 *rows, int n, int W, u32 *T, int thread, int threads)
{
    const int nw = (n + 31) >> 5, wb = (W + 7) >> 3, jb = (nw + 3) >> 2;
    for (int i = thread; i < wb * jb * 32; i += threads) {
        const int b8 = i >> 5, w = (b8 % wb) * 8 + (i & 7), j = (b8 / wb) * 4 + ((i >> 3) & 3);
        if (w >= W || j >= nw) continue;
        u32 r[32];
#pragma unroll
        for (int k = 0; k < 32; ++k) {
            const int v = 32 * j + k;
            r[k] = v < n ? rows[(size_t)v * W + w] : 0u;
        }
        transpose32(r);
#pragma unroll
        for (int b = 0; b < 32; ++b) T[(b * W + w) * RW + j] = r[b];
    }
}

// ------------------------------------------------------------------------------------------------- messages
// Message bits 8*unit .. 8*unit+7 of every node from the node words of layer d's clauses (see the header): for the units of
// this CTA.  All threads; the node words are complete (grid barrier); the rows are complete after another grid barrier.
// s_row [32][RW], s_win / s_dst [32*RW]: scratch.
template <int RW>
__device__ __forceinline__ void pull_messages(const ChainArgs &a, const DevModel &m, const GraphView &gv, const u32 *packed, int edges, const u32 *node_bits, u32 *rows_t,
                                              u32 *rows_n, u32 *s_row, u32 *s_win, u32 *s_dst)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int nw = (gv.n + 31) >> 5, units = (m.MS + 7) >> 3;
    for (int unit = blockIdx.x; unit < units; unit += gridDim.x) {
        const int b0 = 8 * unit, nb = min(8, m.MS - b0), win = nb + a.tmax;
        // (1) node words of the window's bits b0 - tmax .. b0 + nb - 1.  Their clauses are one stretch of the list, or several
        //     where the bits wrap around; groups of RW lanes take entries of it, four loads of node words in flight each.
        u32 ahead[4];                                                   // the thread's first edges, on their way meanwhile
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const int e = threadIdx.x + t * blockDim.x;
            ahead[t] = e < edges ? __ldg(packed + e) : kNoEdge;
        }
        for (int i = threadIdx.x; i < win * RW; i += blockDim.x) s_row[i] = 0;
        __syncthreads();
        const int j = lane % RW, group = warp * (32 / RW) + lane / RW, groups = nwarps * (32 / RW);
        const int start = (((b0 - a.tmax) % m.MS) + m.MS) % m.MS;       // bit of window row 0
        for (int row0 = 0; row0 < win;) {
            const int bit0 = (start + row0) % m.MS, rows = min(win - row0, m.MS - bit0);
            const int lo = __ldg(a.bit_off + bit0), hi = __ldg(a.bit_off + bit0 + rows);
            for (int s0 = lo + group; s0 < hi; s0 += 4 * groups) {
                u32 word[4];
                int row[4];
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    const int s = s0 + t * groups;
                    word[t] = 0;
                    row[t] = 0;
                    if (s < hi) {
                        const int2 entry = __ldg(a.bit_clause + s);     // clause, bit
                        row[t] = row0 + entry.y - bit0;
                        if (j < nw) word[t] = __ldcg(node_bits + (size_t)entry.x * RW + j);
                    }
                }
#pragma unroll
                for (int t = 0; t < 4; ++t)
                    if (word[t]) atomicOr(s_row + row[t] * RW + j, word[t]);
            }
            row0 += rows;
        }
        __syncthreads();
        // (2) the window of every source node as one word
        for (int j = warp; j < nw; j += nwarps) {
            u32 s = 0;
#pragma unroll 4
            for (int i = 0; i < win; ++i) s |= ((s_row[i * RW + j] >> lane) & 1u) << i;
            s_win[32 * j + lane] = s;
            s_dst[32 * j + lane] = 0;
        }
        __syncthreads();
        // (3) bit b of a destination is bit b - t of a source: the window shifted by the edge type
        const u32 keep = (1u << nb) - 1u;
        auto send = [&](u32 e) {
            if (e == kNoEdge) return;
            const u32 v = (s_win[e & 1023u] >> (a.tmax - (int)(e >> 20))) & keep;
            if (v) atomicOr(s_dst + ((e >> 10) & 1023u), v);
        };
#pragma unroll
        for (int t = 0; t < 4; ++t) send(ahead[t]);
        for (int e = threadIdx.x + 4 * blockDim.x; e < edges; e += blockDim.x) send(__ldg(packed + e));
        __syncthreads();
        // (4) out: node-major bytes, and the transposed rows of the unit's bits
        for (int j = warp; j < nw; j += nwarps) {
            const int v = 32 * j + lane;
            const u32 d = s_dst[v];
            if (v < gv.n) reinterpret_cast<unsigned char *>(rows_n + (size_t)v * m.MW)[unit] = (unsigned char)d;
            u32 row = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const u32 b = __ballot_sync(kFull, (d >> i) & 1u);
                if (lane == i) row = b;
            }
            if (lane < nb) rows_t[(size_t)(((b0 & 31) + lane) * m.MW + (b0 >> 5)) * RW + j] = row;
        }
        __syncthreads();
    }
}

// One CTA with the whole model: message rows [v][MW] in shared memory, node-major, from the clauses' marks on the source
// nodes `src` (complete: call after a CTA barrier; the rows are complete on return).  Graphs of a few nodes: a thread per row
// word looks through all edges, so that nothing is cleared first and nothing merged - a barrier instead of three.
__device__ __forceinline__ void solo_messages(const DevModel &m, const GraphView &gv, const u32 *src, u32 *out)
{
    const int n = gv.n, MW = m.MW;
    const bool gather = n <= kChainRowWise;
    if (!gather) {
        for (int i = threadIdx.x; i < n * MW; i += blockDim.x) out[i] = 0;
        __syncthreads();
    }
    for (int i = threadIdx.x; i < n * MW; i += blockDim.x) {
        const int v0 = i / MW, w = i - v0 * MW;
        u32 acc = 0;
        for (int u = gather ? 0 : v0; u < (gather ? n : v0 + 1); ++u) {
            const u32 *row = src + u * MW;
            const u32 e0 = gv.eidx[u] - gv.e_off, deg = gv.degree[u];
            for (u32 k = 0; k < deg && e0 + k < gv.e_cnt; ++k) {
                const u32 dst = gv.edge[2 * (size_t)(e0 + k)], ty = gv.edge[2 * (size_t)(e0 + k) + 1];
                if (gather ? dst != (u32)v0 : dst >= (u32)n) continue;       // malformed edges are ignored
                const u32 v = rotated_word(row, w, ty >= (u32)m.MS ? ty % (u32)m.MS : ty, m.MS, MW);
                if (gather) acc |= v;
                else if (v) atomicOr(out + dst * MW + w, v);
            }
        }
        if (gather) out[i] = acc;
    }
    __syncthreads();
}

// ------------------------------------------------------------------------------------------------ the kernel
// Dynamic shared memory, in words (plan_chain counts the same): [KP] vote partial | [KP] totals | [KP] targets | [KP] thresholds |
// [kChainStages][KP] targets of staged graphs | [4][4] graph sizes | [kChainStages] staged graphs, stage_total each | message
// scratch [msg_words] | T: transposed rows [t_rows][RW] | type rows [kTransposedTypes][max(RW, 4)] | per clause: record
// [kChainRec], mask stream [pre_words], state [clause_words] = draw position (2), include count, its pending change, weights
// [KP], node words [max(RW, 4)], planes (or include planes) of all layers
template <int RW, bool kOneLayer, bool kHybrid, bool kNarrow>
__global__ void __launch_bounds__(chain_threads(kHybrid, kNarrow), 1) fit_chain_kernel(DevModel m_in, DevGraphs g, ChainArgs a)
{
    DevModel m = m_in;
    if (kOneLayer) m.D = 1;
    extern __shared__ __align__(16) u32 s_mem[];
    __shared__ MaskProb s_prob[kMaxDepth];
    __shared__ int s_abort, s_items, s_next_item;
    __shared__ long long s_lap[9];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    constexpr int SB = kChainStateBits;
    const int KP = (m.K + 3) & ~3;
    const bool solo = a.solo != 0;
    int *s_sum = reinterpret_cast<int *>(s_mem), *s_total = s_sum + KP, *s_target = s_total + KP;
    float *s_thr = reinterpret_cast<float *>(s_target + KP);
    int *s_y = s_target + 2 * KP;                                        // [kChainStages][KP]
    int *s_size = s_y + kChainStages * KP;                               // [4][4]: n, first node, first edge row, edge rows
    u32 *s_stage = reinterpret_cast<u32 *>(s_size + 16);
    const int stage_total = (a.stage_words + 3 * a.stage_nodes + 2 * a.stage_edges + 3) & ~3;
    u32 *s_msg = s_stage + kChainStages * stage_total;
    // message scratch: solo [n][MW] marks, [D-1][n][MW] rows, [n][MW] marks; else window rows [32][RW], window words and destinations [32*RW] each
    const int msg_words = kOneLayer ? 0 : solo ? (m.D + 1) * a.max_nodes * m.MW : 96 * RW;
    u32 *s_T = s_msg + ((msg_words + 3) & ~3);
    const int t_rows = 32 * max(m.L0, kOneLayer ? 0 : m.MW);
    u32 *s_types = s_T + (size_t)t_rows * RW;
    u32 *s_clause = s_types + kTransposedTypes * max(RW, 4);
    const int per_clause = kChainRec + a.pre_words + a.clause_words;
    const int clause_warps = nwarps - a.helper, vote_warp = a.helper ? clause_warps : 0;
    const int stage_thread = a.helper ? (int)threadIdx.x - 32 * clause_warps : (int)threadIdx.x, stage_threads = a.helper ? 32 : (int)blockDim.x;
    const int c_lo = min(m.C, (int)blockIdx.x * a.clauses_per_cta), c_hi = min(m.C, c_lo + a.clauses_per_cta), mine = c_hi - c_lo;
    const int clause0 = warp < clause_warps ? warp : mine;               // first of the warp's clauses

    auto record = [&](int i) { return reinterpret_cast<int *>(s_clause + (size_t)i * per_clause); };
    auto stream = [&](int i) { return s_clause + (size_t)i * per_clause + kChainRec; };
    auto state = [&](int i) { return s_clause + (size_t)i * per_clause + kChainRec + a.pre_words; };
    auto weights = [&](int i) { return reinterpret_cast<int *>(state(i) + 4); };
    auto nodes = [&](int i) { return state(i) + 4 + KP; };
    auto layer_words = [&](int l) { return l == 0 ? m.L0 : m.M; };
    // planes of a layer: the include plane always in shared memory, the others there or in global memory
    auto planes = [&](int i, int l) -> u32 * {
        if (kHybrid) return l == 0 ? m.ta0 + (size_t)(c_lo + i) * SB * m.L0 : m.tam + ((size_t)(l - 1) * m.C + c_lo + i) * SB * m.M;
        return nodes(i) + max(RW, 4) + (l == 0 ? 0 : SB * (m.L0 + (l - 1) * m.M));
    };
    auto include = [&](int i, int l) -> u32 * {
        if (kHybrid) return nodes(i) + max(RW, 4) + (l == 0 ? 0 : m.L0 + (l - 1) * m.M);
        return planes(i, l) + (SB - 1) * layer_words(l);
    };
    // solo: the clauses mark one buffer while the other, which the last messages were made from, is cleared
    int turn = 0;
    auto marks = [&](int t) { return s_msg + (size_t)(t ? m.D : 0) * a.max_nodes * m.MW; };
    auto mark = [&](int i, int n) {
        u32 *to = marks(turn);
        for (int j = 0; j < (n + 31) >> 5; ++j)
            if ((nodes(i)[j] >> lane) & 1u)
                for (int b = 0; b < m.MB; ++b) {
                    u32 bit = __ldg(m.hv + (size_t)(c_lo + i) * m.MB + b);
                    if (bit >= (u32)m.MS) bit %= (u32)m.MS;
                    atomicOr(to + (32 * j + lane) * m.MW + (bit >> 5), 1u << (bit & 31));
                }
    };
    auto layer_mask = [&](int l) { return l == 0 ? m.lit_mask : m.msg_mask; };

    // ---- staging of graphs: sizes three steps ahead, arrays two ----
    const u64 steps = (u64)a.epochs * (u64)a.count;
    auto advance = [&](int64_t e) { return e + 1 < a.first + a.count ? e + 1 : a.first; };
    auto fits = [&](const int *sz) { return sz[0] <= a.stage_nodes && sz[0] * m.L0 <= a.stage_words && (kOneLayer || sz[3] <= a.stage_edges); };
    auto fetch_sizes = [&](u64 st, int64_t e) {
        if (stage_thread >= 0 && stage_thread < 4 && st < steps) {
            const u32 *src = stage_thread == 0 ? g.n_nodes : stage_thread == 1 ? g.node_index : stage_thread == 2 ? g.graph_edge0 : g.graph_edges;
            async_copy_word(reinterpret_cast<u32 *>(s_size + (int)(st & 3) * 4 + stage_thread), src + e);
        }
    };
    auto fetch_graph = [&](u64 st, int64_t e, int slot) {               // sizes of step st are there
        if (st >= steps || stage_thread < 0) return;
        if (stage_thread < m.K) async_copy_word(reinterpret_cast<u32 *>(s_y + slot * KP + stage_thread), reinterpret_cast<const u32 *>(a.Y + (size_t)e * m.K + stage_thread));
        const int *sz = s_size + (int)(st & 3) * 4;
        if (!fits(sz)) return;
        const int n = sz[0], base = sz[1], e0 = sz[2], ne = sz[3];
        u32 *x = s_stage + slot * stage_total, *t = x + a.stage_words;
        for (int i = stage_thread; i < n * m.L0; i += stage_threads) async_copy_word(x + i, g.X + (size_t)base * m.L0 + i);
        for (int i = stage_thread; i < n; i += stage_threads) {
            async_copy_word(t + i, g.node_type + base + i);
            if (!kOneLayer) {
                async_copy_word(t + a.stage_nodes + i, g.degree + base + i);
                async_copy_word(t + 2 * a.stage_nodes + i, g.edge_index + base + i);
            }
        }
        if (!kOneLayer)
            for (int i = stage_thread; i < 2 * ne; i += stage_threads) async_copy_word(t + 3 * a.stage_nodes + i, g.edge + 2 * (size_t)e0 + i);
    };
    auto wait_copies = [&]() { asm volatile("cp.async.wait_all;" ::: "memory"); };
    auto view_of = [&](u64 st, int slot) {
        const int *sz = s_size + (int)(st & 3) * 4;
        GraphView gv;
        gv.n = sz[0];
        if (fits(sz)) {
            const u32 *x = s_stage + slot * stage_total, *t = x + a.stage_words;
            gv.X = x; gv.type = t; gv.degree = t + a.stage_nodes; gv.eidx = t + 2 * a.stage_nodes; gv.edge = t + 3 * a.stage_nodes;
            gv.e_off = (u32)sz[2]; gv.e_cnt = (u32)sz[3];
        } else {
            const int base = sz[1];
            gv.X = g.X + (size_t)base * m.L0; gv.type = g.node_type + base; gv.degree = g.degree + base;
            gv.eidx = g.edge_index + base; gv.edge = g.edge; gv.e_off = 0; gv.e_cnt = g.total_edges;
        }
        return gv;
    };
    auto row_wise = [&](int n) { return RW == 1 && n <= kChainRowWise; };
    // transposed rows of the first layer and type rows of a graph
    auto prepare_graph = [&](const GraphView &gv) {
        if (stage_thread < 0) return;
        for (int j = stage_thread >> 5; j < (RW == 1 ? 1 : RW); j += stage_threads >> 5) {
            const int v = 32 * j + lane;
            const u32 ty = v < gv.n ? gv.type[v] : ~0u;
            for (int t = 0; t < g.n_types; ++t) {
                const u32 col = __ballot_sync(kFull, ty == (u32)t);
                if (lane == 0) s_types[t * RW + j] = col;
            }
        }
        if (!row_wise(gv.n)) transpose_rows<RW>(gv.X, gv.n, m.L0, s_T, stage_thread, stage_threads);
    };

    // ---- waits ----
    auto barrier = [&](unsigned nb) {                                   // all CTAs; false once any of them gave up
        __syncthreads();
        if (threadIdx.x == 0) {
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.barrier) : "memory");
            const unsigned want = nb * (gridDim.x + (unsigned)a.missing);
            WaitClock clock;
            while (true) {
                unsigned seen;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(a.barrier) : "memory");
                if ((int)(seen - want) >= 0) break;
                if (clock.expired(a.wait_ns) || ((clock.spins & 63u) == 0 && *(volatile int *)a.error)) { atomicExch(a.error, 1); s_abort = 1; break; }
            }
        }
        __syncthreads();
        return s_abort == 0;
    };

    // ---- first layer of a clause on a graph, and its vote when there is no other layer ----
    int vote = 0;                                                       // lane k: class k's weights of this warp's clauses that are true
    auto first_layer = [&](int i, const GraphView &gv) {
        const int ct = (c_lo + i) % g.n_types;
        const u32 *inc = include(i, 0);
        bool any;
        if (row_wise(gv.n)) any = eval_clause_rowwise(inc, m.L0, m.lit_mask, s_types[ct * RW], nodes(i), true, lane, [&](int v, int w) { return gv.X[v * m.L0 + w]; });
        else any = eval_clause_rows<RW>(s_T, m.L0, inc, m.L0, m.lit_mask, 0, m.MW, s_types + ct * RW, nodes(i), true, lane);
        if (kOneLayer || m.D == 1) { if (any && lane < m.K) vote += weights(i)[lane]; }
        else if (!solo) {
            __syncwarp();
            if (lane < RW) a.node_bits[(size_t)(c_lo + i) * RW + lane] = nodes(i)[lane];
        } else if (any) {
            __syncwarp();
            mark(i, gv.n);
        }
    };

    // ---- state in ----
    if (threadIdx.x < kMaxDepth) s_prob[threadIdx.x] = mask_prob(m_in.p_mask[threadIdx.x]);
    if (threadIdx.x == 0) { s_abort = 0; s_items = 0; s_next_item = 0; }
    if (threadIdx.x < m.K) s_sum[threadIdx.x] = 0;
    if (!kOneLayer && solo) for (int i = threadIdx.x; i < a.max_nodes * m.MW; i += blockDim.x) marks(0)[i] = marks(1)[i] = 0;
    for (int i = clause0; i < mine; i += clause_warps) {
        const int c = c_lo + i;
        u32 *st = state(i);
        if (lane == 0) { *reinterpret_cast<u64 *>(st) = m.draw_pos[c]; st[3] = 0; }
        for (int k = lane; k < m.K; k += 32) weights(i)[k] = m.weights[(size_t)k * m.C + c];
        if (lane < max(RW, 4)) nodes(i)[lane] = 0;
        int n_inc = 0;
        for (int l = 0; l < m.D; ++l) {
            const int W = layer_words(l);
            const u32 *src = l == 0 ? m.ta0 + (size_t)c * SB * W : m.tam + ((size_t)(l - 1) * m.C + c) * SB * W;
            if (kHybrid) src += (size_t)(SB - 1) * W;
            u32 *dst = kHybrid ? include(i, l) : planes(i, l);
            for (int t = lane; t < (kHybrid ? W : SB * W); t += 32) dst[t] = src[t];
            __syncwarp();
            for (int t = lane; t < W; t += 32) n_inc += __popc(include(i, l)[t] & (t == W - 1 ? layer_mask(l) : kFull));
        }
        n_inc = __reduce_add_sync(kFull, n_inc);
        if (lane == 0) st[2] = (u32)n_inc;
    }
    int64_t e1 = advance(a.first), e2 = advance(e1), e3 = advance(e2);     // graphs one, two, three steps ahead
    fetch_sizes(0, a.first); fetch_sizes(1, e1); fetch_sizes(2, e2);
    wait_copies();
    __syncthreads();
    fetch_graph(0, a.first, 0);
    fetch_graph(1, e1, 1);
    wait_copies();
    __syncthreads();
    prepare_graph(view_of(0, 0));
    __syncthreads();
    {
        const GraphView gv = view_of(0, 0);
        for (int i = clause0; i < mine; i += clause_warps) first_layer(i, gv);
    }
    // accumulators only grow: what this CTA read last from each of the two sets (lane k of the voting warp)
    unsigned long long seen_votes[2] = {0, 0};
    unsigned nb = 0;
    const bool timer = a.timers != 0 && blockIdx.x == 0 && threadIdx.x < 32;
    // phase times live in shared memory: as variables they took 20 registers of every thread
    if (timer && lane < 9) s_lap[lane] = lane == 8 ? clock64() : 0;
    __syncwarp();
    auto lap = [&](int phase) {
        if (timer) {
            const long long now = clock64(), before = s_lap[8], sum = s_lap[phase];
            __syncwarp();
            if (lane == 0) { s_lap[phase] = sum + now - before; s_lap[8] = now; }
            __syncwarp();
        }
    };

    GraphView gv = view_of(0, 0);                                       // the current graph
    int slot = 0;                                                       // staging slot of the current graph
    for (u64 step = 0; step < steps; ++step) {
        const int slot1 = slot == 2 ? 0 : slot + 1, slot2 = slot1 == 2 ? 0 : slot1 + 1;
        wait_copies();                                                  // issued a step ago; seen by all after the next barrier
        // ---- message layers ----
        for (int d = 1; d < m.D; ++d) {
            u32 *bits = a.node_bits + (size_t)(d - 1) * m.C * RW, *rows_t = a.rows_t + (size_t)(d - 1) * 32 * m.MW * RW,
                *rows_n = a.rows_n + (size_t)(d - 1) * a.max_nodes * m.MW;
            lap(0);
            if (solo) {
                rows_n = s_msg + (size_t)d * a.max_nodes * m.MW;
                __syncthreads();
                u32 *sent = marks(turn);
                solo_messages(m, gv, sent, rows_n);
                if (!row_wise(gv.n)) { transpose_rows<RW>(rows_n, gv.n, m.MW, s_T, threadIdx.x, blockDim.x); __syncthreads(); }
                turn ^= 1;
                for (int i = threadIdx.x; i < gv.n * m.MW; i += blockDim.x) sent[i] = 0;
                lap(5);
            } else {
                if (!barrier(++nb)) return;
                lap(1);
                pull_messages<RW>(a, m, gv, a.packed + (u32)s_size[(int)(step & 3) * 4 + 2], s_size[(int)(step & 3) * 4 + 3], bits, rows_t, rows_n, s_msg, s_msg + 32 * RW, s_msg + 64 * RW);
                lap(4);
                if (!barrier(++nb)) return;
                lap(1);
                // 32*MW*RW words, a multiple of 128 bytes
                for (int i = threadIdx.x; i < 8 * m.MW * RW; i += blockDim.x) {
                    const unsigned dst = (unsigned)__cvta_generic_to_shared(s_T + 4 * i);
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(rows_t + 4 * i) : "memory");
                }
                wait_copies();
                __syncthreads();
                lap(5);
            }
            const bool last = d == m.D - 1;
            for (int i = clause0; i < mine; i += clause_warps) {
                const int ct = (c_lo + i) % g.n_types;
                const u32 *inc = include(i, d);
                bool any;
                if (solo && row_wise(gv.n))
                    any = eval_clause_rowwise(inc, m.M, m.msg_mask, s_types[ct * RW], nodes(i), false, lane,
                                              [&](int v, int w) { return msg_word(rows_n + v * m.MW, w, m.MS, m.MW); });
                else any = eval_clause_rows<RW>(s_T, m.MW, inc, m.M, m.msg_mask, m.MS, m.MW, s_types + ct * RW, nodes(i), false, lane);
                if (last) { if (any && lane < m.K) vote += weights(i)[lane]; }
                else if (!solo) {
                    __syncwarp();
                    if (lane < RW) bits[(size_t)m.C * RW + (size_t)(c_lo + i) * RW + lane] = nodes(i)[lane];
                } else if (any) {
                    __syncwarp();
                    mark(i, gv.n);
                }
            }
        }
        // ---- votes out ----
        if (lane < m.K && vote != 0) atomicAdd(&s_sum[lane], vote);
        vote = 0;
        __syncthreads();
        lap(0);
        const int *y = s_y + slot * KP;
        const int set = (int)(step & 1);
        if (warp == vote_warp && lane < m.K) {
            const int sum = s_sum[lane];
            s_sum[lane] = 0;
            if (solo) {
                s_total[lane] = sum;
                class_decision_input(m.T, sum, y[lane], s_target + lane, s_thr + lane);
            } else {
                // one word: arrivals in bits 48..63, the partial plus 2^31 (never negative) below
                const unsigned long long word = (1ull << 48) + (1ull << 31) + (unsigned long long)(long long)sum;
                asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(a.votes + set * m.K + lane), "l"(word) : "memory");
            }
        }
        // ---- in the shadow of the exchange: the graph after next, what decisions need besides the class sums, the next graph ----
        fetch_sizes(step + 3, e3);
        fetch_graph(step + 2, e2, slot2);
        for (int i = clause0; i < mine; i += clause_warps) {
            const int c = c_lo + i;
            int *rec = record(i);
            const u32 *nd = nodes(i);
            const u64 pos = *reinterpret_cast<const u64 *>(state(i));
            const u32 draw = chain_draw_at(a, c, pos + lane);
            // one true node, uniformly: the (draw % count)-th set bit in ascending node order (kernels.py:319-349)
            int count, chosen = -1, pc = 0;
            if (RW == 1) count = __popc(nd[0]);
            else { pc = lane < RW ? __popc(nd[lane]) : 0; count = __reduce_add_sync(kFull, pc); }
            if (count > 0) {
                int rank = count == 1 ? 0 : (int)(__shfl_sync(kFull, draw, 0) % (u32)count);
                if (RW == 1) {
                    chosen = nth_set_bit(nd[0], rank, lane);
                } else {
                    int incl = pc;
#pragma unroll
                    for (int d = 1; d < RW; d <<= 1) {
                        const int t = __shfl_up_sync(kFull, incl, d);
                        if (lane >= d) incl += t;
                    }
                    const int src = __ffs(__ballot_sync(kFull, lane < RW && rank >= incl - pc && rank < incl)) - 1;
                    rank -= __shfl_sync(kFull, incl - pc, src);
                    chosen = 32 * src + nth_set_bit(nd[src], rank, lane);
                }
            }
            const u64 after = pos + (count > 0 ? 1 : 0);
            if (lane == 0) { rec[0] = chosen; rec[1] = count > 0; }
            rec[8 + lane] = (int)draw;
            if constexpr (kNarrow) stream_rounds(a, c, (after + (u64)m.K) >> 2, 0, a.spec_rounds, s_prob[0].count, stream(i), lane);
        }
        const bool more = step + 1 < steps;
        const GraphView gn = view_of(step + 1, slot1);
        if (more) prepare_graph(gn);
        lap(6);
        // ---- votes in ----
        if (!solo && warp == vote_warp) {
            bool gave_up = false;
            if (lane < m.K) {
                const unsigned long long want = (unsigned long long)gridDim.x + (unsigned long long)a.missing;
                unsigned long long *acc = a.votes + set * m.K + lane, v, d;
                WaitClock clock;
                while (true) {
                    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(acc) : "memory");
                    d = v - (set ? seen_votes[1] : seen_votes[0]);
                    if ((d >> 48) >= want) break;
                    if (clock.expired(a.wait_ns) || ((clock.spins & 63u) == 0 && *(volatile int *)a.error)) { atomicExch(a.error, 1); gave_up = true; break; }
                }
                if (set) seen_votes[1] = v; else seen_votes[0] = v;
                const int sum = (int)(long long)((d & 0xffffffffffffull) - ((d >> 48) << 31));
                s_total[lane] = sum;
                class_decision_input(m.T, sum, y[lane], s_target + lane, s_thr + lane);
            }
            if (__any_sync(kFull, gave_up) && lane == 0) s_abort = 1;
        }
        __syncthreads();
        if (s_abort) return;
        lap(2);
        // ---- feedback and the next graph's first layer ----
        const bool final_step = !more;
        for (int i = clause0; i < mine; i += clause_warps) {
            const int c = c_lo + i;
            int *rec = record(i);
            u32 *st = state(i);
            int *wgt = weights(i);
            const int chosen = rec[0], taken = rec[1];
            u32 draw = (u32)rec[8 + lane];
            const bool clause_true = chosen >= 0;
            const u64 after = *reinterpret_cast<const u64 *>(st) + taken;
            u64 pos = after;
            // feedback type per class + weight move (kernels.py:351-405), up to 15 classes per pass, one class per lane.  Class k
            // reads its first uniform at offset k + #{j < k : negative target and its first uniform kept it} - the
            // reference's short-circuit order -, the unique fixed point of which is found by re-evaluating all lanes until the set
            // of kept classes stops changing.
            int upd_all = 0;                                            // lane k: feedback type of class k
            for (int kb = 0; kb < m.K; kb += 15) {
                const int kn = min(15, m.K - kb), at = kb == 0 ? taken : 0;
                if (kb > 0) draw = chain_draw_at(a, c, pos + lane);
                const float uni = to_uniform(draw);
                const bool has = lane < kn;
                int w = 0, sign = 1, t = 1;
                float thr = 0.0f;
                if (has) { w = wgt[kb + lane]; sign = w >= 0 ? 1 : -1; t = s_target[kb + lane]; thr = s_thr[kb + lane]; }
                u32 kept = 0, seen;
                int off;
                float u1;
                do {
                    seen = kept;
                    off = lane + __popc(kept & ((1u << lane) - 1u)) + at;
                    u1 = __shfl_sync(kFull, uni, off & 31);
                    kept = __ballot_sync(kFull, has && t == -1 && !(u1 > m.q_keep_f));
                } while (kept != seen);
                const float u2 = __shfl_sync(kFull, uni, (off + 1) & 31);
                // negative target: dropped when the first uniform exceeds q/(K-1), else decided by the second; positive target:
                // decided by its only uniform
                const bool skip = t == -1 ? ((u1 > m.q_keep_f) || (u2 > thr)) : (u1 > thr);
                const int upd = (has && !skip) ? t * sign : 0;
                if (has && upd != 0 && clause_true) {
                    if (upd > 0) { if (abs(w) < INT_MAX) w += sign; }
                    else w -= sign;
                    wgt[kb + lane] = w;
                }
                if (final_step && has) a.update[(size_t)(kb + lane) * m.C + c] = upd;
                const int moved = __shfl_sync(kFull, upd, (lane - kb) & 31);
                if (lane >= kb && lane < kb + kn) upd_all = moved;
                pos += kn + __popc(kept);
            }
            if (final_step && lane == 0) a.clause_node[c] = chosen;
            const u32 positive = __ballot_sync(kFull, upd_all > 0);
            const bool any_feedback = positive != 0 || __ballot_sync(kFull, upd_all < 0 && clause_true) != 0;
            const int npos = __popc(positive);
            const int words_all = m.L0 + (m.D - 1) * m.M;
            if constexpr (kNarrow) {
                if (any_feedback) {
                    const u64 block0 = (after + (u64)m.K) >> 2;
                    const int off0 = (int)(pos - 4 * block0);
                    const bool all_ones = s_prob[0].p >= 1.0f;
                    const int rounds = all_ones ? 0 : (off0 + 32 * npos * words_all + 127) >> 7;
                    u32 *pre = stream(i);
                    const bool packed = 4 * rounds + 1 <= a.pre_words;
                    if (npos > 0 && packed) stream_rounds(a, c, block0, a.spec_rounds, rounds, s_prob[0].count, pre, lane);
                    __syncwarp();
                    const bool within = (int)st[2] <= m.max_included;
                    int change = 0;
                    // the words of all layers, 32 at a time
                    for (int f0 = 0; f0 < words_all; f0 += 32) {
                        int l = 0, w = f0 + lane, W = m.L0;
                        if (!kOneLayer) while (w >= W && l < m.D - 1) { w -= W; W = m.M; ++l; }
                        const int before = f0 + lane - w;                    // words of the layers before
                        const bool in_layer = w < W;
                        if (!in_layer) w = 0;
                        u32 x = 0;
                        if (clause_true && in_layer) {
                            if (l == 0) x = gv.X[(size_t)chosen * m.L0 + w];
                            else if (solo) x = msg_word(s_msg + ((size_t)l * a.max_nodes + chosen) * m.MW, w, m.MS, m.MW);
                            else x = msg_word(a.rows_n + ((size_t)(l - 1) * a.max_nodes + chosen) * m.MW, w, m.MS, m.MW);
                        }
                        const u32 valid = w == W - 1 ? layer_mask(l) : kFull;
                        change += update_words(m.boost, w, W, in_layer, planes(i, l), include(i, l), x, upd_all, clause_true, within, valid, [&](int rank) {
                            if (all_ones || !in_layer) return kFull;
                            const int bit = off0 + 32 * (npos * before + rank * W + w);
                            if (packed) return __funnelshift_r(pre[bit >> 5], pre[(bit >> 5) + 1], bit & 31);
                            // more Type-I classes than the buffer holds: the lane makes its own word
                            const u64 first_draw = 4 * block0 + (u64)(u32)bit;
                            return own_mask(a, c, first_draw >> 2, (int)(first_draw & 3), s_prob[0].count);
                        });
                    }
                    change = __reduce_add_sync(kFull, change);
                    if (lane == 0) st[2] += (u32)change;
                }
                if (lane == 0) *reinterpret_cast<u64 *>(st) = pos + (u64)npos * (u64)words_all * 32u;
                __syncwarp();
                if (more) first_layer(i, gn);
            } else {
                // wide layers: (clause, layer, 32 words) items, handed out to all warps
                if (any_feedback && lane == 0) record(atomicAdd(&s_items, 1))[7] = i;
                if (lane == 0) {
                    rec[2] = (int)(u32)pos; rec[3] = (int)(u32)(pos >> 32);
                    *reinterpret_cast<u64 *>(st) = pos + (u64)npos * (u64)words_all * 32u;
                }
                rec[8 + lane] = upd_all;
            }
        }
        if constexpr (!kNarrow) {
            lap(7);
            __syncthreads();
            const int per0 = (m.L0 + 31) >> 5, perM = (m.M + 31) >> 5, per = per0 + (m.D - 1) * perM, total = s_items * per;
            while (true) {
                int item = 0;
                if (lane == 0) item = atomicAdd(&s_next_item, 1);
                item = __shfl_sync(kFull, item, 0);
                if (item >= total) break;
                const int i = record(item / per)[7], r = item % per;
                const int l = r < per0 ? 0 : 1 + (r - per0) / perM, g0 = 32 * (r < per0 ? r : (r - per0) % perM);
                const int *rec = record(i);
                u32 *st = state(i);
                const int W = layer_words(l), w = g0 + lane, chosen = rec[0], upd = rec[8 + lane];
                const bool clause_true = chosen >= 0;
                const int npos = __popc(__ballot_sync(kFull, upd > 0));
                const u64 pos = (u64)(u32)rec[2] | ((u64)(u32)rec[3] << 32);
                const u64 layer_pos = pos + (l == 0 ? 0u : (u64)npos * (u64)(m.L0 + (l - 1) * m.M) * 32u);
                u32 x = 0;
                if (clause_true && w < W) {
                    if (l == 0) x = gv.X[(size_t)chosen * m.L0 + w];
                    else if (solo) x = msg_word(s_msg + ((size_t)l * a.max_nodes + chosen) * m.MW, w, m.MS, m.MW);
                    else x = msg_word(a.rows_n + ((size_t)(l - 1) * a.max_nodes + chosen) * m.MW, w, m.MS, m.MW);
                }
                const MaskProb mp = s_prob[l];
                int change = update_words(m.boost, w, W, w < W, planes(i, l), include(i, l), x, upd, clause_true, (int)st[2] <= m.max_included,
                                          w == W - 1 ? layer_mask(l) : kFull, [&](int rank) {
                    if (mp.p >= 1.0f) return kFull;
                    const u64 first_draw = layer_pos + (u64)32 * (u64)(rank * W + g0);
                    return lane_mask(a, c_lo + i, (first_draw >> 2) + (u64)8 * lane, (int)(first_draw & 3), mp.count, lane);
                });
                change = __reduce_add_sync(kFull, change);
                if (lane == 0 && change != 0) atomicAdd(reinterpret_cast<int *>(st + 3), change);
            }
            __syncthreads();
            if (threadIdx.x == 0) { s_items = 0; s_next_item = 0; }
            for (int i = clause0; i < mine; i += clause_warps) {
                u32 *st = state(i);
                if (lane == 0) { st[2] += st[3]; st[3] = 0; }
                __syncwarp();
                if (more) first_layer(i, gn);
            }
        }
        if (final_step && blockIdx.x == 0 && threadIdx.x < m.K) a.class_sum_tap[threadIdx.x] = s_total[threadIdx.x];
        lap(3);
        slot = slot1;
        gv = gn;
        e2 = e3; e3 = advance(e3);
    }

    // ---- state out ----
    for (int i = clause0; i < mine; i += clause_warps) {
        const int c = c_lo + i;
        if (lane == 0) m.draw_pos[c] = *reinterpret_cast<u64 *>(state(i));
        for (int k = lane; k < m.K; k += 32) m.weights[(size_t)k * m.C + c] = weights(i)[k];
        for (int l = 0; l < m.D; ++l) {
            const int W = layer_words(l);
            u32 *dst = l == 0 ? m.ta0 + (size_t)c * SB * W : m.tam + ((size_t)(l - 1) * m.C + c) * SB * W;
            if (kHybrid) dst += (size_t)(SB - 1) * W;
            const u32 *src = kHybrid ? include(i, l) : planes(i, l);
            for (int t = lane; t < (kHybrid ? W : SB * W); t += 32) dst[t] = src[t];
        }
    }
    if (timer && lane < 8) a.phase_cycles[lane] = (unsigned long long)s_lap[lane];
}

}  // namespace gtm
