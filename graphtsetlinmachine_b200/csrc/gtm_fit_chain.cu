// Launch logic of the learning kernel for one GPU (gtm_fit_chain.cuh).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "gtm_handles.h"
#include "gtm_fit_chain.cuh"

const void *fit_chain_kernel_narrow_rw1(bool one_layer, bool hybrid);
const void *fit_chain_kernel_narrow_rw4(bool one_layer, bool hybrid);
const void *fit_chain_kernel_narrow_rw16(bool one_layer, bool hybrid);
const void *fit_chain_kernel_narrow_rw32(bool one_layer, bool hybrid);
const void *fit_chain_kernel_wide_rw1(bool one_layer, bool hybrid);
const void *fit_chain_kernel_wide_rw4(bool one_layer, bool hybrid);
const void *fit_chain_kernel_wide_rw16(bool one_layer, bool hybrid);
const void *fit_chain_kernel_wide_rw32(bool one_layer, bool hybrid);

static const void *chain_kernel_for(int rw, bool one_layer, bool hybrid, bool narrow)
{
    if (narrow)
        return rw == 1 ? fit_chain_kernel_narrow_rw1(one_layer, hybrid) : rw == 4 ? fit_chain_kernel_narrow_rw4(one_layer, hybrid)
             : rw == 16 ? fit_chain_kernel_narrow_rw16(one_layer, hybrid) : fit_chain_kernel_narrow_rw32(one_layer, hybrid);
    return rw == 1 ? fit_chain_kernel_wide_rw1(one_layer, hybrid) : rw == 4 ? fit_chain_kernel_wide_rw4(one_layer, hybrid)
         : rw == 16 ? fit_chain_kernel_wide_rw16(one_layer, hybrid) : fit_chain_kernel_wide_rw32(one_layer, hybrid);
}

__global__ void largest_edge_type_kernel(const u32 *edge, size_t edges, u32 *out)
{
    u32 most = 0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < edges; i += (size_t)gridDim.x * blockDim.x) most = max(most, edge[2 * i + 1]);
    most = __reduce_max_sync(kFull, most);
    if ((threadIdx.x & 31) == 0 && most > 0) atomicMax(out, most);
}

// Edge rows of graphs of at most 1,024 nodes and edge types below 4,096 as one word each.  The learning kernel walked the
// nodes' row starts, degrees and rows, three dependent loads that a barrier's acquire sends to L2 every time.
__global__ void __launch_bounds__(256) pack_edges_kernel(DevGraphs g, int64_t graphs, u32 *packed)
{
    const int lane = threadIdx.x & 31;
    for (int64_t e = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; e < graphs; e += (gridDim.x * (int64_t)blockDim.x) >> 5) {
        const u32 base = g.node_index[e], n = g.n_nodes[e];
        for (u32 u = lane; u < n; u += 32) {
            const u32 e0 = g.edge_index[base + u], deg = g.degree[base + u];
            for (u32 k = 0; k < deg && e0 + k < g.total_edges; ++k) {
                const u32 dst = g.edge[2 * (size_t)(e0 + k)], ty = g.edge[2 * (size_t)(e0 + k) + 1];
                packed[e0 + k] = dst < n ? u | dst << 10 | ty << 20 : kNoEdge;
            }
        }
    }
}

// Message buffers of a set, its packed edges, the largest edge type, and the clauses of every message bit: made on the first fit.
static int chain_prepare(gtm_model *m, gtm_dataset *ds, int rw)
{
    const DevModel &d = m->dm;
    if (!m->chain_sync) GTM_TRY(dev_alloc(&m->chain_sync, (size_t)2 * d.K + 1));
    if (d.D == 1) return GTM_OK;
    if (!m->hv_lists_valid) {
        std::vector<int> off((size_t)d.MS + 1, 0), list((size_t)2 * d.C * d.MB);
        for (u32 h : m->hv_host) ++off[h % (u32)d.MS + 1];
        for (int b = 0; b < d.MS; ++b) off[(size_t)b + 1] += off[(size_t)b];
        std::vector<int> at(off.begin(), off.end() - 1);
        for (size_t i = 0; i < m->hv_host.size(); ++i) {
            const int bit = (int)(m->hv_host[i] % (u32)d.MS);
            const size_t entry = (size_t)at[(size_t)bit]++;
            list[2 * entry] = (int)(i / (size_t)d.MB);
            list[2 * entry + 1] = bit;
        }
        if (!m->hv_off) {
            GTM_TRY(dev_alloc(&m->hv_off, off.size()));
            GTM_TRY(dev_alloc(&m->hv_clause, list.size()));
        }
        GTM_CU(cudaMemcpyAsync(m->hv_off, off.data(), off.size() * sizeof(int), cudaMemcpyHostToDevice, m->stream));
        GTM_CU(cudaMemcpyAsync(m->hv_clause, list.data(), list.size() * sizeof(int), cudaMemcpyHostToDevice, m->stream));
        GTM_CU(cudaStreamSynchronize(m->stream));
        m->hv_lists_valid = true;
    }
    if (ds->largest_edge_type < 0) {
        u32 *out, most = 0;
        GTM_TRY(pool_alloc(&out, 1, m->stream));
        GTM_CU(cudaMemsetAsync(out, 0, sizeof(u32), m->stream));
        if (ds->total_edges > 0) largest_edge_type_kernel<<<(unsigned)std::min<int64_t>((ds->total_edges + 255) / 256, 1184), 256, 0, m->stream>>>(ds->dg.edge, (size_t)ds->total_edges, out);
        GTM_CU(cudaMemcpyAsync(&most, out, sizeof(u32), cudaMemcpyDeviceToHost, m->stream));
        cudaFreeAsync(out, m->stream);
        GTM_CU(cudaStreamSynchronize(m->stream));
        ds->largest_edge_type = (int)std::min<u32>(most, 1u << 30);
    }
    if (!ds->chain_packed && ds->largest_edge_type <= kChainMaxType) {
        u32 *p;
        GTM_TRY(pool_alloc(&p, (size_t)std::max<int64_t>(1, ds->total_edges), m->stream));
        ds->owned.push_back(p);
        pack_edges_kernel<<<(unsigned)std::min<int64_t>((ds->n_graphs + 7) / 8, 1184), 256, 0, m->stream>>>(ds->dg, ds->n_graphs, p);
        GTM_CU(cudaGetLastError());
        ds->chain_packed = p;
    }
    if (!ds->chain_msg) {
        const size_t bits = (size_t)(d.D - 1) * d.C * rw, rows = (size_t)(d.D - 1) * 32 * d.MW * rw, nodes = (size_t)(d.D - 1) * ds->max_nodes * d.MW;
        const size_t total = ((bits + 63) & ~(size_t)63) + ((rows + 63) & ~(size_t)63) + nodes;
        u32 *p;
        GTM_TRY(pool_alloc(&p, total, m->stream));
        ds->owned.push_back(p);
        GTM_CU(cudaMemsetAsync(p, 0, total * sizeof(u32), m->stream));        // padding bytes of the rows are never written
        ds->chain_bits = p;
        ds->chain_rows_t = p + ((bits + 63) & ~(size_t)63);
        ds->chain_rows_n = ds->chain_rows_t + ((rows + 63) & ~(size_t)63);
        ds->chain_msg = true;
    }
    return GTM_OK;
}

struct ChainPlan { bool ok = false, hybrid = false; int rw = 0, grid = 0, threads = 0; size_t smem = 0; ChainArgs a; };

// Whether one CTA learns the model alone.  It saves the grid-wide steps (one per graph, two per message layer, about 2,000
// cycles each) and the rounds of a few CTAs over many message bits, and pays with more than a clause per warp (16 warps) and
// with graphs that grow.  Measured on one B200, us a graph, one CTA / a CTA per clause:
//   messages, up to 16 clauses: 10 clauses, 12 nodes 10.0 / 12.4; 16 clauses, 90 nodes 11.8 / 11.6; 16 clauses, 200 nodes, 64
//     message bits 13.4 / 12.8, 512 bits 19.8 / 20.3; 16 clauses, 500 nodes 17.2 / 12.9 and 33.9 / 20.3;
//   messages, more clauses: 24 clauses, 3 nodes 11.8 / 10.9, 12 nodes 13.9 / 12.6; 60 clauses, 500 nodes 38.4 / 12.4;
//   the same on graphs of a few nodes when s = 1, which leaves no masks to draw: 20 clauses 8.5 / 11.4, 32 clauses 9.2 / 9.5, 48
//     clauses 11.9 / 9.5;
//   no messages: 4 clauses 3.5 / 3.5 (images), 4.3 / 4.8 (90 nodes); 8 clauses 3.9 / 3.6, 4.6 / 4.8; 32 clauses 8.5 / 3.9, 9.4 / 5.3.
static bool learned_by_one_cta(const DevModel &d, int max_nodes)
{
    if (d.D == 1) return d.C <= 4;
    bool no_masks = true;
    for (int l = 0; l < d.D; ++l) no_masks = no_masks && d.p_mask[l] >= 1.0f;
    if (no_masks && max_nodes <= kChainRowWise) return d.C <= 32;
    return d.C <= 16 && max_nodes <= 256;
}

static ChainPlan plan_chain(const gtm_model *m, const gtm_dataset *ds)
{
    const DevModel &d = m->dm;
    ChainPlan plan;
    memset(&plan.a, 0, sizeof plan.a);
    ChainArgs &a = plan.a;
    plan.rw = ds->max_nodes <= 32 ? 1 : ds->max_nodes <= 128 ? 4 : ds->max_nodes <= 512 ? 16 : 32;
    const int rw = plan.rw, rw4 = std::max(rw, 4), KP = (d.K + 3) & ~3, D1 = d.D - 1;
    const int words_all = d.L0 + D1 * d.M;
    a.max_nodes = ds->max_nodes;
    bool one_p = true;
    for (int l = 1; l < d.D; ++l) one_p = one_p && d.p_mask[l] == d.p_mask[0];
    a.narrow = one_p && d.L0 <= 32 && (d.D == 1 || d.M <= 32);
    if (a.narrow) {
        // The first rounds of the stream are made in the shadow of the vote exchange, for every clause, wanted or not: two of
        // them fit the shadow (4,000 images x 2,500 clauses: 24.1 ms without, 23.9 with two, 24.0 with the three that one class
        // needs; 200 sequences of three layers, 21 rounds: 8.1 ms without or with two, 9.1 with all).  Room for four classes.
        a.spec_rounds = d.p_mask[0] >= 1.0f ? 0 : std::min(2, (d.K + 3 + 32 * words_all + 127) / 128);
        a.pre_words = (std::max(4 * a.spec_rounds, (d.K + 3) / 32 + 1 + std::min(d.K, 4) * words_all) + 4 + 7) & ~3;
    }
    int cpc = m->opt_fit_block_clauses;
    if (cpc <= 0) cpc = learned_by_one_cta(d, ds->max_nodes) ? d.C : (d.C + m->sm_count - 1) / m->sm_count;
    for (int attempt = 0; attempt < 2; ++attempt) {
        const int grid = (d.C + cpc - 1) / cpc;
        const bool solo = grid == 1;
        if (grid > m->sm_count) return plan;
        const int want_warps = a.narrow ? std::max(D1 > 0 && !solo ? 16 : 8, cpc) : 32;
        for (int variant = 0; variant < 4; ++variant) {        // planes resident, then include planes only; with and without staged graphs
            const bool hybrid = variant >= 2, stage = (variant & 1) == 0;
            const int most = chain_threads(hybrid, a.narrow != 0) / 32;
            // Graphs that are tested as they are: a warp without clauses stages them and exchanges the votes (4,000 images x 2,500
            // clauses 24.1 -> 21.6 ms, 10,000 Noisy-XOR graphs 55.8 -> 54.2).  Transposing a graph of 90 nodes took that warp longer
            // than the exchange (700 graphs 15.6 -> 16.0 ms).
            a.helper = a.narrow && want_warps < most && ds->max_nodes <= kChainRowWise;
            const int warps = std::min(want_warps + a.helper, most);
            a.stage_nodes = stage ? std::min(ds->max_nodes, 512) : 0;
            a.stage_words = stage ? (std::min(ds->max_nodes * d.L0, 4096) + 3) & ~3 : 0;
            a.stage_edges = stage && D1 > 0 ? 512 : 0;
            a.clause_words = (4 + KP + rw4 + words_all * (hybrid ? 1 : d.SB) + 3) & ~3;
            const size_t msg = D1 == 0 ? 0 : solo ? (size_t)(d.D + 1) * ds->max_nodes * d.MW : (size_t)96 * rw;
            const size_t words = (size_t)7 * KP + 16 + (size_t)kChainStages * ((a.stage_words + 3 * a.stage_nodes + 2 * a.stage_edges + 3) & ~3) +
                                 ((msg + 3) & ~(size_t)3) + (size_t)32 * std::max(d.L0, D1 > 0 ? d.MW : 0) * rw + (size_t)kTransposedTypes * rw4 +
                                 (size_t)cpc * (kChainRec + a.pre_words + a.clause_words);
            const size_t smem = words * sizeof(u32);
            const void *fn = chain_kernel_for(rw, d.D == 1, hybrid, a.narrow != 0);
            cudaFuncAttributes fa;
            if (cudaFuncGetAttributes(&fa, fn) != cudaSuccess) { cudaGetLastError(); return plan; }
            if (smem + fa.sharedSizeBytes > 227 * 1024 || 32 * warps > fa.maxThreadsPerBlock) continue;
            plan.ok = true; plan.hybrid = hybrid; plan.grid = grid; plan.threads = 32 * warps; plan.smem = smem;
            a.clauses_per_cta = cpc; a.solo = solo;
            return plan;
        }
        if (!solo || m->opt_fit_block_clauses > 0) break;
        cpc = (d.C + m->sm_count - 1) / m->sm_count;           // too much for one CTA: all SMs
    }
    return plan;
}

// Learns with fit_chain_kernel; *done = 0 when it does not cover the model or the set.
int launch_fit_chain(gtm_model *m, gtm_dataset *ds, int n_types, const int *Y_dev, int64_t first, int64_t count, int epochs, int *done)
{
    const DevModel &d = m->dm;
    *done = 0;
    if (d.recorded || d.K > 32 || d.SB != kChainStateBits || ds->max_nodes > 1024 || n_types > kTransposedTypes) return GTM_OK;
    ChainPlan plan = plan_chain(m, ds);
    if (!plan.ok) return GTM_OK;
    GTM_TRY(chain_prepare(m, ds, plan.rw));
    if (d.D > 1 && !plan.a.solo && ds->largest_edge_type > kChainMaxType) return GTM_OK;
    ChainArgs &a = plan.a;
    a.Y = Y_dev; a.first = first; a.count = count; a.epochs = epochs;
    // accumulators, arrival counter and the error word start every launch at zero
    a.votes = m->chain_sync; a.barrier = (unsigned *)(m->chain_sync + 2 * d.K); a.error = (int *)a.barrier + 1;
    GTM_CU(cudaMemsetAsync(m->chain_sync, 0, ((size_t)2 * d.K + 1) * sizeof(unsigned long long), m->stream));
    a.clause_node = m->clause_node; a.update = m->update; a.class_sum_tap = m->class_sum_tap;
    a.phase_cycles = m->phase_cycles; a.timers = m->opt_fit_timers;
    a.wait_ns = (unsigned long long)m->opt_fit_wait_ms * 1000000ull;
    a.missing = m->opt_fit_missing_cta;
    a.node_bits = ds->chain_bits; a.rows_t = ds->chain_rows_t; a.rows_n = ds->chain_rows_n;
    a.packed = ds->chain_packed; a.bit_off = m->hv_off; a.bit_clause = reinterpret_cast<const int2 *>(m->hv_clause); a.tmax = std::max(0, ds->largest_edge_type);
    for (int r = 0; r < 10; ++r) {
        a.key[2 * r] = d.seed_lo + (u32)r * 0x9E3779B9u;
        a.key[2 * r + 1] = d.seed_hi + (u32)r * 0xBB67AE85u;
    }
    DevGraphs g = ds->dg;
    g.n_types = n_types;
    DevModel dm = d;
    const void *fn = chain_kernel_for(plan.rw, d.D == 1, plan.hybrid, plan.a.narrow != 0);
    // the limit belongs to the kernel: set to this plan's size, another model's fit in another thread could lower it before the launch
    cudaFuncAttributes fa;
    GTM_CU(cudaFuncGetAttributes(&fa, fn));
    GTM_CU(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024 - (int)fa.sharedSizeBytes));
    void *args[] = {&dm, &g, &a};
    GTM_CU(cudaLaunchCooperativeKernel(fn, dim3(plan.grid), dim3(plan.threads), args, plan.smem, m->stream));
    *done = 1;
    const int info[6] = {2, plan.grid, plan.rw, plan.hybrid, plan.a.narrow != 0, a.solo != 0};
    memcpy(m->last_fit, info, sizeof info);
    int err = 0;
    GTM_CU(cudaMemcpyAsync(&err, a.error, sizeof(int), cudaMemcpyDeviceToHost, m->stream));
    GTM_CU(cudaStreamSynchronize(m->stream));
    if (err) return fail(GTM_ERR_TIMEOUT, "a bounded wait of the learning kernel (grid barrier or vote exchange) gave up");
    return GTM_OK;
}
