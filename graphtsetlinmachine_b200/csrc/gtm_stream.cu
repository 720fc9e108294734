// Node-stream scoring: the fast path of batched inference for depth-1 models.
//
// Idea.  Layer-0 clause evaluation is a per-node test, so a graph set is one long stream of nodes.  A CTA
// takes a TILE of consecutive graphs (at most TN = 32*TNC nodes), turns the tile's literal rows into the
// transposed form XT[literal][node word] (bit i of word j = literal of node 32j+i) in shared memory, and then
// evaluates a clause on 32 nodes per AND: r = AND over the clause's INCLUDED literals of XT[literal][j].
// That is popcount(include) word operations per 32 nodes instead of 32*ceil(literals/32) for the row-wise
// test, and an empty clause costs nothing (and is true, as in kernels.py:443-460).  Included literals come
// from per-clause lists rebuilt from the include planes whenever the automata changed.
//
// A thread evaluates one clause on FOUR node words at a time (one 128-bit shared load per literal; the eight lanes of
// a wavefront read one row, so the loads are free of bank conflicts for tiles of 32 node words).
//
// Votes are a product: sums[graph][class] = fired[graph][clause] x weight[clause][class] (kernels.py:279-317, unclamped),
// with 0/1 on the left and 32-bit integers on the right, and they run on the tensor cores: the outcomes of 32 clauses on a
// graph are one 32-bit word (32x32 bit transposes in registers), whose bits are spread to bytes with one shift and one AND
// per fragment register, and the weights are cut into signed bytes - as many as the largest weight needs, the sums are exact
// modulo 2^32 like the additions they stand for.  A walk over the fired clauses with one thread per graph, which this
// replaces, took 200 of the 270 us of 120,000 images x 2,500 clauses (20 % of them firing): every fired clause cost a
// gather of its weight row.
//
// A launch works on units of (tile, share of the clauses).  Large sets have enough tiles to fill the chip and take all
// clauses of a tile in one unit; for smaller ones the clauses are split so that even a single graph keeps many CTAs busy.
// The shares of a tile leave their partial sums in global memory and the one that finishes last adds them up.
//
// Derived model data (StreamModel): literal lists (uint16 row numbers, padded to a multiple of 4 with the number of an
// all-ones row) and the weights as tensor-core fragments.
#include "../../include/gtm_b200.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <vector>

#include "gtm_stream.h"

namespace gtm {

constexpr int kStreamThreads = 512;
constexpr int kStreamWarps = kStreamThreads / 32;
constexpr int kStreamCB = 256;          // clauses per vote block
constexpr int kStreamMaxK = 32;
constexpr int kStreamLimbs = 4;         // signed bytes of a weight
constexpr int kStreamMaxTypes = 8;
constexpr int kStreamMaxSplitTiles = 2048;              // launches over more tiles do not split the clauses
constexpr size_t kStreamMaxPart = (size_t)64 << 20;     // bytes of partial sums

// ------------------------------------------------------------------------------------------- list building
// Fragment byte of (clause c, class k): the A operand (16 classes x 32 clauses, s8) of mma.m16n8k32.  The clauses of a
// word are taken in the order that makes the B operand cheap: element 4*t+i of the first (second) half of the k range is
// clause bit 8*i+t (8*i+4+t), so that a B register is (word >> t) & 0x01010101.
__device__ __forceinline__ size_t stream_weight_at(int limb, int c, int k, int kt, int cwords)
{
    const int bit = c & 31, t = bit & 7, i = bit >> 3;
    const int lane = (k & 7) * 4 + (t & 3), reg = ((k & 15) >> 3) + (t >> 2) * 2;
    return ((((size_t)limb * kt + (k >> 4)) * cwords + (c >> 5)) * 32 + lane) * 16 + reg * 4 + i;
}

// One warp per clause: the list of its included literals, and its weights.
__global__ void __launch_bounds__(256) stream_lists_kernel(DevModel m, int *cnt, unsigned short *list, int list_stride, signed char *wf, int kt,
                                                           int *limbs)
{
    const int lane = threadIdx.x & 31, c = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (c >= m.C) return;
    const u32 *inc = m.ta0 + ((size_t)c * m.SB + (m.SB - 1)) * m.L0;
    unsigned short *out = list + (size_t)c * list_stride;
    int n = 0;
    for (int w0 = 0; w0 < m.L0; w0 += 32) {
        const int w = w0 + lane;
        u32 bits = w < m.L0 ? inc[w] & (w == m.L0 - 1 ? m.lit_mask : kFull) : 0u;
        const int mine = __popc(bits);
        int incl = mine;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int t = __shfl_up_sync(kFull, incl, d);
            if (lane >= d) incl += t;
        }
        int at = n + incl - mine;
        while (bits) {
            const int b = __ffs(bits) - 1;
            bits &= bits - 1;
            out[at++] = (unsigned short)(w * 32 + b);
        }
        n += __shfl_sync(kFull, incl, 31);
    }
    const int padded = (n + 3) & ~3;
    if (lane < padded - n) out[n + lane] = (unsigned short)m.literals;     // the all-ones row
    if (lane == 0) cnt[c] = padded;
    const int cwords = (m.C + 31) >> 5;
    int most = 1;
    for (int k = lane; k < m.K; k += 32) {
        int rest = m.weights[(size_t)k * m.C + c];
        for (int l = 0; l < kStreamLimbs; ++l) {
            const int digit = (int)(signed char)(rest & 0xff);
            wf[stream_weight_at(l, c, k, kt, cwords)] = (signed char)digit;
            if (digit != 0) most = max(most, l + 1);
            rest = (int)(((long long)rest - digit) >> 8);
        }
    }
    most = __reduce_max_sync(kFull, most);
    if (lane == 0 && most > 1) atomicMax(limbs, most);
}

// -------------------------------------------------------------------------------------------------- scoring
struct StreamArgs {
    const int *tile_graph;              // first graph of every tile, or NULL: every tile holds graphs_per_tile graphs
    int graphs_per_tile;
    int tile_lo, tile_hi;               // tiles [tile_lo, tile_hi)
    int64_t first, count;               // graphs written: [first, first+count)
    int64_t n_graphs, total_nodes;
    int *class_sums;                    // [count][K]
    unsigned *unit_counter;             // units handed out beyond the first of every CTA, zero before the launch
    int splits;                         // shares of a tile's clauses
    int blocks_per_split;               // clause blocks of a share
    int *part;                          // [splits][n_graphs][K] partial sums (splits > 1)
    int *ticket;                        // [tiles of the launch] shares of a tile that are done (splits > 1), zero before the launch
    int TNC;
    const int *lit_cnt;
    const unsigned short *lit_list;
    int list_stride;
    const signed char *wf;
    const int *limbs;
};

__device__ __forceinline__ uint4 lds128(unsigned addr)
{
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}

// d (16 classes x 8 graphs, s32) += a (16 classes x 32 clauses, s8) * b (32 clauses x 8 graphs, u8)
__device__ __forceinline__ void mma_votes(int (&d)[4], const uint4 &a, u32 b0, u32 b1)
{
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.u8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
                 : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}

// KT: 16-class row blocks of the votes (1: up to 16 classes, 2: up to 32).  NT: 8-graph column blocks per warp, so a tile
// holds at most 8*NT*16 graphs: 1,024 with one row block; with two, 512, which keeps the accumulators in registers at two
// CTAs per SM.
template <int KT, int NT>
__global__ void __launch_bounds__(kStreamThreads, 2) stream_score_kernel(DevModel m, DevGraphs g, StreamArgs a)
{
    extern __shared__ __align__(16) u32 s_dyn[];
    constexpr int CW = kStreamCB / 32;                 // clause words per block
    const int TNC = a.TNC, RS = TNC | 1;               // node words per tile; row stride of RT
    const int rowshift = 31 - __clz(TNC * 4);
    u32 *XT = s_dyn;                                   // [literals+1][TNC]
    u32 *TMV = XT + (size_t)(m.literals + 1) * TNC;    // [n_types][TNC] valid & node type
    u32 *R = TMV + (size_t)g.n_types * TNC;            // [CB][TNC]        node bits per clause; then FW of sets with multi-node graphs
    u32 *RT = R + (size_t)kStreamCB * TNC;             // [CW][32*RS]      clause bits per node: node 32j+b at b*RS + j
    __shared__ int s_unit, s_last;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned xt32 = (unsigned)__cvta_generic_to_shared(XT);
    const unsigned keep = 0xffffu << rowshift;
    const int cwords = (m.C + 31) >> 5;
    const int limbs = max(1, *a.limbs);
    const int units = (a.tile_hi - a.tile_lo) * a.splits;
    const int more = units - (int)gridDim.x;           // units beyond the first of every CTA

    for (int unit = blockIdx.x; unit < units;) {
        const int tile = a.tile_lo + unit / a.splits, split = unit % a.splits;
        const int g0 = a.tile_graph ? a.tile_graph[tile] : (int)min((int64_t)tile * a.graphs_per_tile, a.n_graphs);
        const int g1 = a.tile_graph ? a.tile_graph[tile + 1] : (int)min((int64_t)(tile + 1) * a.graphs_per_tile, a.n_graphs);
        const int node0 = (int)g.node_index[g0];
        const int node1 = g1 < a.n_graphs ? (int)g.node_index[g1] : (int)a.total_nodes;
        const int nn = node1 - node0, ng = g1 - g0;
        const int tnc = (nn + 31) >> 5;                // node words in use
        const int qshift = tnc <= 4 ? 0 : 32 - __clz(((tnc + 3) >> 2) - 1);   // log2 of the quads (128 nodes) looked at
        const int Q = 1 << qshift;

        // ---- the tile's literal rows, transposed in registers: a thread takes 32 nodes x 32 literals ----
        for (int blk = tid; blk < 4 * Q * m.L0; blk += kStreamThreads) {
            const int j = blk / m.L0, w = blk - j * m.L0;
            u32 rows[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                const int v = 32 * j + i;
                rows[i] = v < nn ? __ldg(g.X + (size_t)(node0 + v) * m.L0 + w) : 0u;
            }
            transpose32(rows);
            const int nbits = min(32, m.literals - 32 * w);
#pragma unroll
            for (int b = 0; b < 32; ++b)
                if (b < nbits) XT[(size_t)(32 * w + b) * TNC + j] = rows[b];
        }
        for (int j = tid; j < TNC; j += kStreamThreads) XT[(size_t)m.literals * TNC + j] = kFull;
        for (int j = warp; j < 4 * Q; j += kStreamWarps) {
            const int v = j * 32 + lane;
            const u32 ty = v < nn ? g.node_type[node0 + v] : ~0u;
            for (int t = 0; t < g.n_types; ++t) {
                const u32 col = __ballot_sync(kFull, ty == (u32)t);
                if (lane == 0) TMV[t * TNC + j] = col;
            }
        }
        // how the outcomes of a graph's nodes become outcomes of the graph: single-node graphs are their node; few large
        // graphs are ORed clause by clause along R's words; many small ones node by node along RT's
        const bool single = nn == ng, large = !single && nn >= 8 * ng;

        int acc[KT][NT][4];
#pragma unroll
        for (int kt = 0; kt < KT; ++kt)
#pragma unroll
            for (int t = 0; t < NT; ++t)
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[kt][t][i] = 0;
        __syncthreads();

        const int cb_end = min(m.C, (split + 1) * a.blocks_per_split * kStreamCB);
        for (int cb0 = split * a.blocks_per_split * kStreamCB; cb0 < cb_end; cb0 += kStreamCB) {
            const int cbn = min(kStreamCB, cb_end - cb0), cwn = (cbn + 31) >> 5;
            // ---- evaluation: (clause, 4 node words) per thread; AND the transposed rows of the included literals ----
            for (int idx = tid; idx < cwn * 32 << qshift; idx += kStreamThreads) {
                const int cb = idx >> qshift, quad = idx & (Q - 1);
                uint4 r = make_uint4(0u, 0u, 0u, 0u);              // rows past the last clause stay empty
                if (cb < cbn) {
                    const int c = cb0 + cb;
                    const unsigned xq = xt32 + quad * 16;
                    r = *reinterpret_cast<const uint4 *>(TMV + (c % g.n_types) * TNC + quad * 4);
                    const uint2 *lp = reinterpret_cast<const uint2 *>(a.lit_list + (size_t)c * a.list_stride);
                    const int groups = __ldg(a.lit_cnt + c) >> 2;
#pragma unroll 2
                    for (int q = 0; q < groups; ++q) {
                        const uint2 four = __ldg(lp + q);
                        const uint4 x0 = lds128(xq + ((four.x << rowshift) & keep));
                        const uint4 x1 = lds128(xq + ((four.x >> (16 - rowshift)) & keep));
                        const uint4 x2 = lds128(xq + ((four.y << rowshift) & keep));
                        const uint4 x3 = lds128(xq + ((four.y >> (16 - rowshift)) & keep));
                        r.x &= x0.x & x1.x; r.y &= x0.y & x1.y; r.z &= x0.z & x1.z; r.w &= x0.w & x1.w;
                        r.x &= x2.x & x3.x; r.y &= x2.y & x3.y; r.z &= x2.z & x3.z; r.w &= x2.w & x3.w;
                    }
                }
                *reinterpret_cast<uint4 *>(R + (size_t)cb * TNC + quad * 4) = r;
            }
            __syncthreads();
            const u32 *FW;                             // outcome word of (clause word cw, graph n)
            int fw_cw, fw_lo, fw_hi;                   // at cw * fw_cw + (n & 31) * fw_lo + (n >> 5) * fw_hi
            if (large) {
                FW = RT; fw_cw = ng; fw_lo = 1; fw_hi = 32;
                for (int task = warp; task < cwn * ng; task += kStreamWarps) {
                    const int gl = task / cwn, cw = task - gl * cwn, cb = 32 * cw + lane;
                    const int lo = (int)g.node_index[g0 + gl] - node0, hi = lo + (int)g.n_nodes[g0 + gl];     // slots [lo, hi)
                    const int j0 = lo >> 5, j1 = (hi - 1) >> 5, jn = j1 - j0 + 1;
                    u32 any = 0;
                    // the words of a row are taken in an order that differs from lane to lane: rows are a multiple of four
                    // words apart, the same word of 32 rows would sit in a few banks
                    int j = j0 + lane % jn;
                    for (int s = 0; s < jn; ++s) {
                        u32 mask = kFull;
                        if (j == j0) mask &= kFull << (lo & 31);
                        if (j == j1) mask &= kFull >> (31 - ((hi - 1) & 31));
                        any |= R[(size_t)cb * TNC + j] & mask;
                        j = j == j1 ? j0 : j + 1;
                    }
                    const u32 word = __ballot_sync(kFull, any != 0);
                    if (lane == 0) RT[cw * ng + gl] = word;
                }
            } else {
                // ---- 32 clauses x 32 nodes blocks of R, transposed in registers ----
                FW = RT; fw_cw = 32 * RS; fw_lo = RS; fw_hi = 1;
                for (int blk = tid; blk < cwn * 4 * Q; blk += kStreamThreads) {
                    const int cw = blk >> (qshift + 2), j = blk & (4 * Q - 1);
                    u32 rows[32];
#pragma unroll
                    for (int i = 0; i < 32; ++i) rows[i] = R[(size_t)(32 * cw + i) * TNC + j];
                    transpose32(rows);
#pragma unroll
                    for (int b = 0; b < 32; ++b) RT[(size_t)cw * 32 * RS + b * RS + j] = rows[b];
                }
                if (!single) {
                    __syncthreads();
                    FW = R; fw_cw = ng; fw_lo = 1; fw_hi = 32;
                    for (int i = tid; i < cwn * ng; i += kStreamThreads) {
                        const int cw = i / ng, gl = i - cw * ng;
                        const int lo = (int)g.node_index[g0 + gl] - node0, hi = lo + (int)g.n_nodes[g0 + gl];
                        u32 fired = 0;
                        for (int v = lo; v < hi; ++v) fired |= RT[(size_t)cw * 32 * RS + (v & 31) * RS + (v >> 5)];
                        R[i] = fired;
                    }
                }
            }
            __syncthreads();
            // ---- votes: warp w takes graphs 8*(w + 16t) .. +7 ----
            const int mine = warp * 8 + (lane >> 2), sh = lane & 3;
            for (int l = 0; l < limbs; ++l)
                for (int cw = 0; cw < cwn; ++cw) {
                    uint4 wa[KT];
#pragma unroll
                    for (int kt = 0; kt < KT; ++kt)
                        wa[kt] = __ldg(reinterpret_cast<const uint4 *>(a.wf) + (((size_t)l * KT + kt) * cwords + (cb0 >> 5) + cw) * 32 + lane);
#pragma unroll
                    for (int t = 0; t < NT; ++t) {
                        if (8 * (warp + kStreamWarps * t) >= ng) break;
                        const int n = min(mine + 8 * kStreamWarps * t, ng - 1);     // columns past the last graph repeat it and are not written
                        const u32 word = FW[cw * fw_cw + (n & 31) * fw_lo + (n >> 5) * fw_hi];
                        const u32 b0 = (word >> sh) & 0x01010101u, b1 = (word >> (sh + 4)) & 0x01010101u;
#pragma unroll
                        for (int kt = 0; kt < KT; ++kt) {
                            if (l == 0) {
                                mma_votes(acc[kt][t], wa[kt], b0, b1);
                            } else {
                                int d[4] = {0, 0, 0, 0};
                                mma_votes(d, wa[kt], b0, b1);
#pragma unroll
                                for (int i = 0; i < 4; ++i) acc[kt][t][i] += (int)((u32)d[i] << (8 * l));
                            }
                        }
                    }
                }
            __syncthreads();
        }

        // ---- class sums of the tile's graphs, through shared memory (R and RT are free) ----
        int *sums = reinterpret_cast<int *>(R);
#pragma unroll
        for (int kt = 0; kt < KT; ++kt)
#pragma unroll
            for (int t = 0; t < NT; ++t)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int n = 8 * (warp + kStreamWarps * t) + 2 * (lane & 3) + (i & 1), k = 16 * kt + (lane >> 2) + 8 * (i >> 1);
                    if (n < ng && k < m.K) sums[n * m.K + k] = acc[kt][t][i];
                }
        __syncthreads();
        bool write = true;
        if (a.splits > 1) {
            int *mine = a.part + ((size_t)split * a.n_graphs + g0) * m.K;
            for (int i = tid; i < ng * m.K; i += kStreamThreads) __stcg(mine + i, sums[i]);
            __threadfence();
            __syncthreads();
            if (tid == 0) s_last = atomicAdd(a.ticket + (tile - a.tile_lo), 1) == a.splits - 1;
            __syncthreads();
            write = s_last != 0;
            if (write) {
                __threadfence();
                for (int i = tid; i < ng * m.K; i += kStreamThreads) {
                    int v = sums[i];
                    for (int s = 0; s < a.splits; ++s)
                        if (s != split) v += __ldcg(a.part + ((size_t)s * a.n_graphs + g0) * m.K + i);
                    sums[i] = v;
                }
            }
            // a thread reads below what it has written itself
        }
        if (write)      // only graphs inside the requested range
            for (int i = tid; i < ng * m.K; i += kStreamThreads) {
                const int64_t gi = (int64_t)g0 + i / m.K;
                if (gi >= a.first && gi < a.first + a.count) a.class_sums[((int64_t)g0 - a.first) * m.K + i] = sums[i];
            }
        // ---- next unit ----
        if (more <= 0) break;
        if (tid == 0) s_unit = (int)gridDim.x + (int)atomicAdd(a.unit_counter, 1u);
        __syncthreads();       // s_unit; the shared buffers are reused by the next unit
        unit = s_unit;
    }
}

// ------------------------------------------------------------------------------------------------ host side
static int stream_kt(int K) { return K <= 16 ? 1 : 2; }

static const void *stream_kernel_for(int K)
{
    return stream_kt(K) == 1 ? (const void *)stream_score_kernel<1, 8> : (const void *)stream_score_kernel<2, 4>;
}

static size_t stream_smem_bytes(int literals, int TNC, int n_types)
{
    return ((size_t)(literals + 1 + n_types) * TNC + (size_t)kStreamCB * TNC + (size_t)kStreamCB * (TNC | 1)) * sizeof(u32);
}

// Graphs of a tile: the votes' accumulators hold 1,024 graphs of up to 16 classes or 512 of up to 32, and the class sums
// of a tile leave through the buffers R and RT.
static int stream_max_graphs(int K, int TNC) { return stream_kt(K) == 1 ? std::min(1024, 32 * TNC) : std::min(512, 16 * TNC); }

int stream_model_create(StreamModel *sm, const DevModel &d)
{
    // row numbers are 16 bits; the smallest tile (four node words) has to fit
    if (d.D != 1 || d.K > kStreamMaxK || d.literals > 65534 || stream_smem_bytes(d.literals, 4, kStreamMaxTypes) > 220 * 1024) return GTM_OK;
    sm->list_stride = (d.literals + 3) & ~3;
    const size_t wf = (size_t)kStreamLimbs * stream_kt(d.K) * ((d.C + 31) / 32) * 512;
    GTM_TRY(dev_alloc(&sm->lit_cnt, (size_t)d.C));
    GTM_TRY(dev_alloc(&sm->lit_list, (size_t)d.C * sm->list_stride));
    GTM_TRY(dev_alloc(&sm->wf, wf));
    GTM_TRY(dev_alloc(&sm->limbs, 1));
    GTM_CU(cudaMemset(sm->wf, 0, wf));
    sm->applicable = true;
    return GTM_OK;
}

void stream_model_destroy(StreamModel *sm)
{
    cudaFree(sm->lit_cnt); cudaFree(sm->lit_list); cudaFree(sm->wf); cudaFree(sm->limbs);
    *sm = StreamModel();
}

int stream_model_refresh(StreamModel *sm, const DevModel &d, cudaStream_t s)
{
    if (!sm->applicable) return GTM_OK;
    GTM_CU(cudaMemsetAsync(sm->limbs, 0, sizeof(int), s));
    stream_lists_kernel<<<(d.C + 7) / 8, 256, 0, s>>>(d, sm->lit_cnt, sm->lit_list, sm->list_stride, sm->wf, stream_kt(d.K), sm->limbs);
    GTM_CU(cudaGetLastError());
    return GTM_OK;
}

int stream_data_create(StreamData *sd, const StreamModel &sm, const DevModel &d, const gtm_graphs_view *v, u32 n_min, u32 n_max,
                       int sm_count, cudaStream_t s)
{
    sd->supported = 0;
    if (!sm.applicable) return GTM_OK;
    // Node words of a tile: no more than the set has nodes for (a few graphs are evaluated 128 nodes at a time, and rows
    // of 16 bytes keep the bank conflicts of that small), at most 32 (rows of 128 bytes: none), and as many as let two
    // CTAs share an SM - or one, when only that holds the largest graph.
    const int64_t most = v->max_number_of_graph_nodes;
    int TNC = 0;
    for (int pass = 0; pass < 2 && TNC == 0; ++pass)
        for (int cand = 32; cand >= 4; cand >>= 1) {
            if (cand > 4 && (int64_t)cand * 16 >= v->total_nodes) continue;
            if (most > 32 * cand) break;
            if (stream_smem_bytes(d.literals, cand, kStreamMaxTypes) <= (size_t)(pass == 0 ? 112 : 220) * 1024) { TNC = cand; break; }
        }
    if (TNC == 0) return GTM_OK;
    const size_t smem = stream_smem_bytes(d.literals, TNC, kStreamMaxTypes);
    const void *fn = stream_kernel_for(d.K);
    GTM_CU(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 224 * 1024));      // not the set's own: another set may need more
    int per_sm = 0;
    GTM_CU(cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(&per_sm, fn, kStreamThreads, smem, 0));
    if (per_sm < 1) return GTM_OK;

    // tiling: consecutive graphs while nodes and graphs stay within the tile; sets whose graphs all have one size need no table
    const int TN = TNC * 32, max_graphs = stream_max_graphs(d.K, TNC);
    std::vector<int> &tg = sd->tile_graph_host;
    tg.clear();
    sd->tile_graph = nullptr;
    if (most == 1) n_min = n_max = 1;
    if (n_min > 0 && n_min == n_max) {
        sd->graphs_per_tile = std::min(TN / (int)n_min, max_graphs);
        sd->n_tiles = (int)((v->number_of_graphs + sd->graphs_per_tile - 1) / sd->graphs_per_tile);
    } else {
        sd->graphs_per_tile = 0;
        tg.reserve((size_t)(v->total_nodes / TN) * 2 + 16);
        tg.push_back(0);
        int64_t used = 0;
        for (int64_t gi = 0; gi < v->number_of_graphs; ++gi) {
            const int64_t n = v->number_of_graph_nodes[gi];
            if (used + n > TN || (gi - tg.back()) >= max_graphs) { tg.push_back((int)gi); used = 0; }
            used += n;
        }
        tg.push_back((int)v->number_of_graphs);
        sd->n_tiles = (int)tg.size() - 1;
        GTM_TRY(pool_alloc(&sd->tile_graph, tg.size(), s));
        GTM_CU(cudaMemcpyAsync(sd->tile_graph, tg.data(), tg.size() * sizeof(int), cudaMemcpyHostToDevice, s));
    }
    sd->TNC = TNC;
    sd->grid = sm_count * per_sm;
    sd->total_nodes = v->total_nodes;
    sd->n_graphs = v->number_of_graphs;
    sd->supported = 1;
    return GTM_OK;
}

// s: a stream behind every kernel that reads the tables (the model's, which may not be the one they were made on).
void stream_data_destroy(StreamData *sd, cudaStream_t s)
{
    if (sd->tile_graph) cudaFreeAsync(sd->tile_graph, s);
    sd->tile_graph = nullptr; sd->supported = 0;
}

bool stream_supported(const StreamData &sd, int n_types) { return sd.supported != 0 && n_types <= kStreamMaxTypes; }

// Shares of the clauses for a launch over `tiles` tiles: the number that makes the rounds of units on the chip cheapest, a
// unit costing as much as its clause blocks plus about half a block for the tile's transposition and sums.
static int stream_splits(const StreamData &sd, const DevModel &d, int tiles, int *blocks_per_split)
{
    const int blocks = (d.C + kStreamCB - 1) / kStreamCB;
    *blocks_per_split = blocks;
    int best = 1;
    double best_cost = 1e30;
    if (tiles > kStreamMaxSplitTiles) return 1;
    for (int s = 1; s <= blocks; ++s) {
        const int per = (blocks + s - 1) / s;
        if ((blocks + per - 1) / per != s) continue;                               // the same shares as a smaller number
        if (s > 1 && (size_t)s * sd.n_graphs * d.K * sizeof(int) > kStreamMaxPart) break;
        const double cost = (double)(((int64_t)tiles * s + sd.grid - 1) / sd.grid) * (0.5 + per);
        if (cost < best_cost) { best_cost = cost; best = s; *blocks_per_split = per; }
    }
    return best;
}

static void stream_tiles(const StreamData &sd, int64_t first, int64_t count, int *lo, int *hi)
{
    if (sd.graphs_per_tile > 0) {
        *lo = (int)(first / sd.graphs_per_tile);
        *hi = (int)((first + count + sd.graphs_per_tile - 1) / sd.graphs_per_tile);
    } else {
        const std::vector<int> &tg = sd.tile_graph_host;
        *lo = (int)(std::upper_bound(tg.begin(), tg.end(), (int)first) - tg.begin()) - 1;
        *hi = (int)(std::lower_bound(tg.begin(), tg.end(), (int)(first + count)) - tg.begin());
    }
}

// Scratch of a launch: the unit counter, a ticket per tile when the clauses are split, then the shares' partial sums.
static size_t stream_sync_bytes(int tiles, int splits) { return (((size_t)1 + (splits > 1 ? tiles : 0)) * sizeof(int) + 255) & ~(size_t)255; }

size_t stream_scratch_bytes(const StreamData &sd, const DevModel &d, int64_t first, int64_t count)
{
    int lo, hi, per;
    stream_tiles(sd, first, count, &lo, &hi);
    const int splits = stream_splits(sd, d, hi - lo, &per);
    return stream_sync_bytes(hi - lo, splits) + (splits > 1 ? (size_t)splits * sd.n_graphs * d.K * sizeof(int) : 0);
}

int stream_score(const StreamModel &sm, const StreamData &sd, const DevModel &d, const DevGraphs &dg, int n_types,
                 int64_t first, int64_t count, int *sums_dev, char *scratch, cudaStream_t s)
{
    DevGraphs g = dg;
    g.n_types = n_types;
    StreamArgs a;
    a.tile_graph = sd.tile_graph;
    stream_tiles(sd, first, count, &a.tile_lo, &a.tile_hi);          // tiles that overlap [first, first+count)
    const int tiles = a.tile_hi - a.tile_lo;
    a.splits = stream_splits(sd, d, tiles, &a.blocks_per_split);
    const size_t sync_bytes = stream_sync_bytes(tiles, a.splits);
    a.unit_counter = (unsigned *)scratch; a.ticket = (int *)scratch + 1; a.part = (int *)(scratch + sync_bytes);
    a.graphs_per_tile = sd.graphs_per_tile;
    a.first = first; a.count = count; a.n_graphs = sd.n_graphs; a.total_nodes = sd.total_nodes;
    a.class_sums = sums_dev; a.TNC = sd.TNC;
    a.lit_cnt = sm.lit_cnt; a.lit_list = sm.lit_list; a.list_stride = sm.list_stride;
    a.wf = sm.wf; a.limbs = sm.limbs;
    const int grid = std::max(1, std::min(sd.grid, tiles * a.splits));
    if (a.splits > 1 || tiles > grid) GTM_CU(cudaMemsetAsync(scratch, 0, sync_bytes, s));      // else the kernel reads none of it
    DevModel dm = d;
    void *args[] = {&dm, &g, &a};
    GTM_CU(cudaLaunchKernel(stream_kernel_for(d.K), dim3(grid), dim3(kStreamThreads), args, stream_smem_bytes(d.literals, sd.TNC, n_types), s));
    return GTM_OK;
}

}  // namespace gtm
