// Host runtime and C ABI (include/gtm_b200.h) of the B200-native Graph Tsetlin Machine engine.
#include "../../include/gtm_b200.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <cmath>
#include <cstring>
#include <new>
#include <string>
#include <vector>

#include "gtm_handles.h"
#include "gtm_kernels.cuh"
#include "gtm_stage.h"

// The general scoring kernel with or without four-at-a-time node words (graph sets with more than 32 nodes per graph).
static const void *score_kernel_for(int max_nodes, int units = 1)
{
    if (units > 1) return (const void *)score_small_graphs_kernel;
    return max_nodes > 32 ? (const void *)score_graphs_kernel<true> : (const void *)score_graphs_kernel<false>;
}

static int bind(gtm_model *m)
{
    if (!m) return fail(GTM_ERR_ARG, "null model handle");
    GTM_CU(cudaSetDevice(m->cfg.device));
    return GTM_OK;
}

static bool is_capturing(cudaStream_t s)
{
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &status) != cudaSuccess) { cudaGetLastError(); return true; }
    return status != cudaStreamCaptureStatusNone;
}

// For calls that return with work in flight: gtm_set_stream orders the next stream behind it.  Work that is recorded into a
// graph is not in flight; its replays are the caller's to order.
static int note_queued(gtm_model *m)
{
    if (is_capturing(m->stream)) return GTM_OK;
    GTM_CU(cudaEventRecord(m->queued, m->stream));
    m->in_flight = true;
    return GTM_OK;
}

// largest float that is <= d
static float float_round_down(double d)
{
    float f = (float)d;
    if ((double)f > d) f = nextafterf(f, -INFINITY);
    return f;
}

static int words_for(int bits) { return (bits - 1) / 32 + 1; }
static u32 tail_mask(int bits) { return (bits % 32) ? ~(0xffffffffu << (bits % 32)) : 0xffffffffu; }
static int layer_words(const gtm_model *m, int layer) { return layer == 0 ? m->dm.L0 : m->dm.M; }
static u32 *layer_planes(const gtm_model *m, int layer)
{
    const DevModel &d = m->dm;
    return layer == 0 ? d.ta0 : d.tam + (size_t)(layer - 1) * d.C * d.SB * d.M;
}

// The host reads and writes callers' arrays itself where the driver once copied all of them: device memory is refused here, as
// the driver refused it.
static int check_on_host(const void *p, const char *what)
{
    cudaPointerAttributes at;
    if (!p) return GTM_OK;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) { cudaGetLastError(); return GTM_OK; }
    return at.type == cudaMemoryTypeDevice ? fail(GTM_ERR_ARG, "%s is in device memory, not in host memory", what) : GTM_OK;
}

// --------------------------------------------------------------------------------------------- library
extern "C" const char *gtm_version(void) { return "gtm_b200 0.1 (sm_100a)"; }
extern "C" const char *gtm_last_error(void) { return gtm_error_text().c_str(); }

extern "C" int gtm_device_count(int *count_out)
{
    if (!count_out) return fail(GTM_ERR_ARG, "count_out is null");
    GTM_CU(cudaGetDeviceCount(count_out));
    return GTM_OK;
}

// Calls without a model, from a thread that may be new to CUDA: on a device that a model lives on, if there is one, instead of
// on device 0, where a context would be made.
static int bind_any()
{
    const int device = stage_device();
    if (device >= 0) GTM_CU(cudaSetDevice(device));
    return GTM_OK;
}

extern "C" int gtm_host_alloc(uint64_t bytes, void **out)
{
    if (!out) return fail(GTM_ERR_ARG, "out is null");
    *out = nullptr;
    GTM_TRY(bind_any());
    GTM_CU(cudaHostAlloc(out, (size_t)std::max<uint64_t>(bytes, 1), cudaHostAllocPortable));
    return GTM_OK;
}

extern "C" int gtm_host_free(void *p)
{
    if (!p) return GTM_OK;
    GTM_TRY(bind_any());
    GTM_CU(cudaFreeHost(p));
    return GTM_OK;
}

// ---------------------------------------------------------------------------------------------- model
extern "C" int gtm_create(const gtm_config *cfg, gtm_model **out)
{
    if (!cfg || !out) return fail(GTM_ERR_ARG, "null argument");
    *out = nullptr;
    if (cfg->number_of_clauses < 1 || cfg->number_of_outputs < 1 || cfg->number_of_literals < 1)
        return fail(GTM_ERR_ARG, "clauses, outputs and literals must be positive");
    if (cfg->number_of_state_bits < 1 || cfg->number_of_state_bits > GTM_MAX_STATE_BITS)
        return fail(GTM_ERR_ARG, "number_of_state_bits must be in 1..%d", GTM_MAX_STATE_BITS);
    if (cfg->depth < 1 || cfg->depth > GTM_MAX_DEPTH) return fail(GTM_ERR_ARG, "depth must be in 1..%d", GTM_MAX_DEPTH);
    if (cfg->T < 1) return fail(GTM_ERR_ARG, "T must be positive");
    if (cfg->depth > 1 && (cfg->message_size < 1 || cfg->message_bits < 1))
        return fail(GTM_ERR_ARG, "message_size and message_bits must be positive when depth > 1");
    for (int d = 0; d < cfg->depth; ++d)
        if (!(cfg->s[d] > 0.0f)) return fail(GTM_ERR_ARG, "s[%d] must be positive", d);
    int ndev = 0;
    GTM_CU(cudaGetDeviceCount(&ndev));
    if (cfg->device < 0 || cfg->device >= ndev) return fail(GTM_ERR_ARG, "device %d out of range (%d visible)", cfg->device, ndev);
    GTM_CU(cudaSetDevice(cfg->device));

    gtm_model *m = new (std::nothrow) gtm_model();
    if (!m) return fail(GTM_ERR_OOM, "host allocation failed");
    m->cfg = *cfg;
    DevModel &d = m->dm;
    memset(&d, 0, sizeof d);
    d.C = cfg->number_of_clauses; d.K = cfg->number_of_outputs; d.literals = cfg->number_of_literals;
    d.SB = cfg->number_of_state_bits; d.boost = cfg->boost_true_positive_feedback; d.T = cfg->T;
    d.max_included = cfg->max_included_literals; d.MS = std::max(1, cfg->message_size);
    d.MB = std::max(1, cfg->message_bits); d.D = cfg->depth;
    d.L0 = words_for(d.literals); d.M = words_for(2 * d.MS); d.MW = words_for(d.MS);
    d.lit_mask = tail_mask(d.literals); d.msg_mask = tail_mask(2 * d.MS);
    for (int i = 0; i < kMaxDepth; ++i) d.s[i] = cfg->s[i];
    d.q_keep = 1.0 * cfg->q / (double)std::max(1, d.K - 1);
    d.q_keep_f = float_round_down(d.q_keep);
    for (int i = 0; i < kMaxDepth; ++i) d.p_mask[i] = cfg->s[i] > 0.0f ? float_round_down(1.0 / (double)cfg->s[i]) : 1.0f;
    d.seed_lo = (u32)cfg->seed; d.seed_hi = (u32)(cfg->seed >> 32);

    cudaDeviceProp prop;
    GTM_CU(cudaGetDeviceProperties(&prop, cfg->device));
    m->sm_count = prop.multiProcessorCount;
    { int st0 = pool_prepare(cfg->device); if (st0 != GTM_OK) { delete m; return st0; } }
    stage_retain(cfg->device);       // given back by gtm_destroy

    int st = GTM_OK;
    st = dev_alloc(&d.ta0, (size_t)d.C * d.SB * d.L0);
    if (st == GTM_OK) st = dev_alloc(&d.tam, (size_t)std::max(1, d.D - 1) * d.C * d.SB * d.M);
    u32 *hv = nullptr;
    if (st == GTM_OK) st = dev_alloc(&d.weights, (size_t)d.K * d.C);
    if (st == GTM_OK) st = dev_alloc(&hv, (size_t)d.C * d.MB);
    if (st == GTM_OK) st = dev_alloc(&d.draw_pos, (size_t)d.C);
    if (st == GTM_OK) st = dev_alloc(&m->clause_node, (size_t)d.C);
    if (st == GTM_OK) st = dev_alloc(&m->update, (size_t)d.K * d.C);
    if (st == GTM_OK) st = dev_alloc(&m->class_sum_tap, (size_t)d.K);
    if (st == GTM_OK) st = dev_alloc(&m->barrier, 1);
    if (st == GTM_OK) st = dev_alloc(&m->error, 1);
    if (st == GTM_OK && cudaMallocHost((void **)&m->score_error, sizeof(int)) != cudaSuccess) { cudaGetLastError(); st = fail(GTM_ERR_OOM, "page-locked host allocation failed"); }
    if (st == GTM_OK) st = dev_alloc(&m->phase_cycles, 8);
    if (st == GTM_OK && cudaEventCreateWithFlags(&m->queued, cudaEventDisableTiming) != cudaSuccess) { cudaGetLastError(); st = fail(GTM_ERR_CUDA, "an event could not be created"); }
    if (st != GTM_OK) { gtm_destroy(m); return st; }
    d.hv = hv;
    m->hv_host.assign((size_t)d.C * d.MB, 0);
    cudaMemset(hv, 0, (size_t)d.C * d.MB * sizeof(u32));
    cudaMemset(d.draw_pos, 0, (size_t)d.C * sizeof(u64));
    cudaMemset(d.weights, 0, (size_t)d.K * d.C * sizeof(int));
    *m->score_error = 0;

    // learning grid: all CTAs must be co-resident (cooperative launch); no more warps than clauses
    st = fit_grid_for_global_state(d, m->sm_count, m->fit_block, &m->fit_grid);
    if (st != GTM_OK) { gtm_destroy(m); return st; }
    st = dev_alloc(&m->exchange, exchange_bytes(1, d.K) / sizeof(unsigned long long) + 1);
    if (st == GTM_OK) st = stream_model_create(&m->sm, d);
    if (st == GTM_OK) st = tile_model_create(&m->tm, d);
    if (st != GTM_OK) { gtm_destroy(m); return fail(st, "device allocation failed"); }
    *out = m;
    return GTM_OK;
}

extern "C" int gtm_destroy(gtm_model *m)
{
    if (!m) return GTM_OK;
    cudaSetDevice(m->cfg.device);
    cudaFree(m->dm.ta0); cudaFree(m->dm.tam);
    cudaFree(m->dm.weights); cudaFree((void *)m->dm.hv); cudaFree(m->dm.draw_pos); cudaFree(m->recorded);
    cudaFree(m->exchange); cudaFree(m->error); cudaFree(m->clause_node); cudaFree(m->update);
    cudaFree(m->class_sum_tap); cudaFree(m->barrier); cudaFree(m->phase_cycles); cudaFree(m->chain_sync); cudaFree(m->hv_off); cudaFree(m->hv_clause);
    stream_model_destroy(&m->sm);
    tile_model_destroy(&m->tm);
    if (m->score_error) cudaFreeHost(m->score_error);
    if (m->queued) cudaEventDestroy(m->queued);
    delete m;
    stage_drop();
    return GTM_OK;
}

extern "C" int gtm_set_stream(gtm_model *m, void *stream)
{
    GTM_TRY(bind(m));
    // Lists, weights and automata are the model's: what is in flight on the old stream makes or reads them.  (The old stream
    // itself may be gone by now, the event is not.)
    if (m->in_flight && (cudaStream_t)stream != m->stream && !is_capturing((cudaStream_t)stream))
        GTM_CU(cudaStreamWaitEvent((cudaStream_t)stream, m->queued, 0));
    m->stream = (cudaStream_t)stream;
    return GTM_OK;
}

extern "C" int gtm_set_option(gtm_model *m, const char *name, int value)
{
    GTM_TRY(bind(m));
    if (!name) return fail(GTM_ERR_ARG, "option name is null");
    if (!strcmp(name, "fit_block_clauses") && value >= 0 && value <= 4096) { m->opt_fit_block_clauses = value; return GTM_OK; }
    if (!strcmp(name, "fit_kernel") && value >= 0 && value <= 2) { m->opt_fit_kernel = value; return GTM_OK; }
    if (!strcmp(name, "score_kernel") && value >= 0 && value <= 3) { m->opt_score_kernel = value; return GTM_OK; }
    if (!strcmp(name, "fit_timers") && value >= 0 && value <= 3) { m->opt_fit_timers = value; return GTM_OK; }
    if (!strcmp(name, "fit_wait_ms") && value >= 1 && value <= 600000) { m->opt_fit_wait_ms = value; return GTM_OK; }
    if (!strcmp(name, "fit_missing_cta") && value >= 0 && value <= 1) { m->opt_fit_missing_cta = value; return GTM_OK; }
    return fail(GTM_ERR_ARG, "unknown option '%s' or value %d out of range", name, value);
}

extern "C" int gtm_init_state(gtm_model *m, int reset_message_layers)
{
    GTM_TRY(bind(m));
    const DevModel &d = m->dm;
    init_weights_kernel<<<(d.C + 255) / 256, 256, 0, m->stream>>>(d);
    for (int l = 0; l < d.D; ++l) {
        if (l > 0 && !reset_message_layers) break;
        const size_t total = (size_t)d.C * d.SB * layer_words(m, l);
        init_planes_kernel<<<(unsigned)std::min<size_t>((total + 255) / 256, 4096), 256, 0, m->stream>>>(layer_planes(m, l), d.C, d.SB, layer_words(m, l));
    }
    GTM_CU(cudaGetLastError());
    GTM_CU(cudaStreamSynchronize(m->stream));
    m->has_state = true;
    m->lists_dirty = true; ++m->state_version;
    return GTM_OK;
}

static int check_layer(gtm_model *m, int layer)
{
    if (layer < 0 || layer >= m->dm.D) return fail(GTM_ERR_ARG, "layer %d out of range (depth %d)", layer, m->dm.D);
    return GTM_OK;
}

extern "C" int gtm_set_ta_state(gtm_model *m, int layer, const uint32_t *ta)
{
    GTM_TRY(bind(m));
    GTM_TRY(check_layer(m, layer));
    if (!ta) return fail(GTM_ERR_ARG, "ta_state is null");
    const DevModel &d = m->dm;
    const int W = layer_words(m, layer);
    const size_t total = (size_t)d.C * d.SB * W;
    u32 *tmp;
    GTM_TRY(pool_alloc(&tmp, total, m->stream));      // stream-ordered: no device-wide synchronisation
    cudaError_t e = cudaMemcpyAsync(tmp, ta, total * sizeof(u32), cudaMemcpyHostToDevice, m->stream);
    if (e == cudaSuccess)
        planes_from_reference_kernel<<<(unsigned)std::min<size_t>((total + 255) / 256, 4096), 256, 0, m->stream>>>(tmp, layer_planes(m, layer), d.C, d.SB, W);
    cudaFreeAsync(tmp, m->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
    GTM_CU(e);
    m->has_state = true;
    m->lists_dirty = true; ++m->state_version;
    return GTM_OK;
}

extern "C" int gtm_get_ta_state(gtm_model *m, int layer, uint32_t *out)
{
    GTM_TRY(bind(m));
    GTM_TRY(check_layer(m, layer));
    if (!out) return fail(GTM_ERR_ARG, "ta_state_out is null");
    GTM_TRY(check_on_host(out, "ta_state_out"));
    const DevModel &d = m->dm;
    const int W = layer_words(m, layer);
    const size_t total = (size_t)d.C * d.SB * W;
    LaneGuard guard;
    GTM_TRY(lane_acquire(m->cfg.device, &guard.lane));
    u32 *tmp;
    GTM_TRY(pool_alloc(&tmp, total, m->stream));
    planes_to_reference_kernel<<<(unsigned)std::min<size_t>((total + 255) / 256, 4096), 256, 0, m->stream>>>(layer_planes(m, layer), tmp, d.C, d.SB, W);
    int st = stage_down(guard.lane, out, tmp, total * sizeof(u32), host_is_pinned(out), m->stream);
    cudaFreeAsync(tmp, m->stream);
    if (st == GTM_OK) st = stage_down_finish(guard.lane);
    if (st != GTM_OK) stage_abandon(guard.lane);
    return st;
}

extern "C" int gtm_set_weights(gtm_model *m, const int32_t *w)
{
    GTM_TRY(bind(m));
    if (!w) return fail(GTM_ERR_ARG, "clause_weights is null");
    GTM_CU(cudaMemcpyAsync(m->dm.weights, w, (size_t)m->dm.K * m->dm.C * sizeof(int), cudaMemcpyHostToDevice, m->stream));
    GTM_CU(cudaStreamSynchronize(m->stream));
    m->lists_dirty = true; ++m->state_version;
    return GTM_OK;
}

extern "C" int gtm_get_weights(gtm_model *m, int32_t *w)
{
    GTM_TRY(bind(m));
    if (!w) return fail(GTM_ERR_ARG, "clause_weights_out is null");
    GTM_CU(cudaMemcpyAsync(w, m->dm.weights, (size_t)m->dm.K * m->dm.C * sizeof(int), cudaMemcpyDeviceToHost, m->stream));
    GTM_CU(cudaStreamSynchronize(m->stream));
    return GTM_OK;
}

extern "C" int gtm_set_hypervectors(gtm_model *m, const uint32_t *hv)
{
    GTM_TRY(bind(m));
    if (!hv) return fail(GTM_ERR_ARG, "hypervectors is null");
    GTM_CU(cudaMemcpyAsync((void *)m->dm.hv, hv, (size_t)m->dm.C * m->dm.MB * sizeof(u32), cudaMemcpyHostToDevice, m->stream));
    GTM_CU(cudaStreamSynchronize(m->stream));
    m->hv_host.assign(hv, hv + (size_t)m->dm.C * m->dm.MB);
    m->hv_lists_valid = false;
    m->lists_dirty = true; ++m->state_version;
    return GTM_OK;
}

extern "C" int gtm_set_draw_positions(gtm_model *m, const uint64_t *pos)
{
    GTM_TRY(bind(m));
    if (!pos) return fail(GTM_ERR_ARG, "positions is null");
    GTM_CU(cudaMemcpyAsync(m->dm.draw_pos, pos, (size_t)m->dm.C * sizeof(u64), cudaMemcpyHostToDevice, m->stream));
    GTM_CU(cudaStreamSynchronize(m->stream));
    return GTM_OK;
}

extern "C" int gtm_get_draw_positions(gtm_model *m, uint64_t *pos)
{
    GTM_TRY(bind(m));
    if (!pos) return fail(GTM_ERR_ARG, "positions_out is null");
    GTM_CU(cudaMemcpyAsync(pos, m->dm.draw_pos, (size_t)m->dm.C * sizeof(u64), cudaMemcpyDeviceToHost, m->stream));
    GTM_CU(cudaStreamSynchronize(m->stream));
    return GTM_OK;
}

extern "C" int gtm_set_recorded_draws(gtm_model *m, const uint32_t *draws, uint64_t per_clause)
{
    GTM_TRY(bind(m));
    GTM_CU(cudaStreamSynchronize(m->stream));
    cudaFree(m->recorded);
    m->recorded = nullptr; m->dm.recorded = nullptr; m->dm.recorded_len = 0;
    if (!draws) return GTM_OK;
    if (per_clause == 0) return fail(GTM_ERR_ARG, "draws_per_clause must be positive");
    const size_t total = (size_t)m->dm.C * per_clause;
    GTM_TRY(dev_alloc(&m->recorded, total));
    GTM_CU(cudaMemcpy(m->recorded, draws, total * sizeof(u32), cudaMemcpyHostToDevice));
    m->dm.recorded = m->recorded;
    m->dm.recorded_len = per_clause;
    return GTM_OK;
}

// --------------------------------------------------------------------------------------------- datasets
template <class T>
static int scratch(gtm_dataset *ds, T **dev, size_t count)
{
    GTM_TRY(pool_alloc(dev, count, ds->model->stream));
    ds->owned.push_back(*dev);
    return GTM_OK;
}

// The graph arrays of a set live in one allocation, in this order, each on a 64-byte boundary; a small set goes up as one
// copy of a host image of it.
struct SetLayout {
    size_t X, node_type, degree, edge_index, edge, node_index, n_nodes, edge0, edges, bytes;
};

static SetLayout set_layout(const gtm_graphs_view *v, int L0)
{
    SetLayout l;
    size_t at = 0;
    auto take = [&](size_t words) { const size_t here = at; at = (at + words * sizeof(u32) + 63) & ~(size_t)63; return here; };
    const size_t nodes = (size_t)v->total_nodes, graphs = (size_t)v->number_of_graphs;
    l.X = take(nodes * L0 + 4);       // the tile kernel fetches literal rows with bulk copies widened to 16-byte boundaries
    l.node_type = take(nodes); l.degree = take(nodes); l.edge_index = take(nodes);
    l.edge = take(2 * (size_t)v->total_edges);
    l.node_index = take(graphs); l.n_nodes = take(graphs); l.edge0 = take(graphs); l.edges = take(graphs);
    l.bytes = at;
    return l;
}

// Host arrays must have the layout that graphs.py produces: node_index and edge_index are exclusive prefix sums of the
// node counts and out-degrees (graphs.py:101-102,127-128), every graph has 1..max_number_of_graph_nodes nodes.  The
// kernels size their scratch rows from max_number_of_graph_nodes and index the arrays with these values, so anything
// else is refused here.  Checks graphs [g_lo, g_hi) and their nodes, and notes what the arrays have in common: constant
// arrays are made on the device instead of being copied.
struct GraphChecks { u32 bad_count = 0, bad_index = 0, bad_edges = 0, n_min = ~0u, n_max = 0, types = 0; };

static void check_graph_span(const gtm_graphs_view *v, int64_t g_lo, int64_t g_hi, GraphChecks *out)
{
    const int64_t N = v->number_of_graphs;
    const u32 max_nodes = (u32)v->max_number_of_graph_nodes;
    GraphChecks c;
    for (int64_t gi = g_lo; gi < g_hi; ++gi) {
        const u32 n = v->number_of_graph_nodes[gi];
        const uint64_t end = (uint64_t)v->node_index[gi] + n;
        const uint64_t want = gi + 1 < N ? (uint64_t)v->node_index[gi + 1] : (uint64_t)v->total_nodes;
        c.bad_count |= (u32)(n - 1u >= max_nodes);
        c.bad_index |= (u32)(end != want);
        c.n_min = std::min(c.n_min, n);
        c.n_max = std::max(c.n_max, n);
    }
    // a span is consistent in itself wherever it starts: its nodes and edges have to lie inside the arrays as well
    const int64_t v_lo = v->node_index[g_lo], v_hi = g_hi < N ? (int64_t)v->node_index[g_hi] : v->total_nodes;
    c.bad_index |= (u32)(v_hi > v->total_nodes);
    if (!c.bad_count && !c.bad_index) {          // node ranges are sound: the span's nodes
        for (int64_t vi = v_lo; vi < v_hi; ++vi) {
            const uint64_t end = (uint64_t)v->edge_index[vi] + v->number_of_graph_node_edges[vi];
            const uint64_t want = vi + 1 < v->total_nodes ? (uint64_t)v->edge_index[vi + 1] : (uint64_t)v->total_edges;
            c.bad_edges |= (u32)(end != want);
        }
        c.bad_edges |= (u32)(v_hi < v->total_nodes && (int64_t)v->edge_index[v_hi] > v->total_edges);
        for (int64_t vi = v_lo; vi < v_hi; ++vi) c.types |= v->node_type[vi];
    }
    *out = c;
}

static int validate_graphs(const gtm_graphs_view *v, int64_t g_lo, int64_t g_hi, GraphChecks *all_out = nullptr)
{
    if (g_lo == 0 && (v->node_index[0] != 0 || v->edge_index[0] != 0)) return fail(GTM_ERR_ARG, "node_index[0] and edge_index[0] must be 0");
    // large sets are checked by the copy threads side by side (the arrays are only read); a thread takes about 2^15 nodes
    const int64_t span = g_hi - g_lo, nodes = span * (v->total_nodes / v->number_of_graphs + 1);
    const int pieces = (int)std::max<int64_t>(1, std::min<int64_t>(std::min<int64_t>(16, span), nodes >> 15));
    struct Job { const gtm_graphs_view *v; int64_t lo, span; int pieces; GraphChecks parts[16]; } job;
    job.v = v; job.lo = g_lo; job.span = span; job.pieces = pieces;
    host_parallel(pieces, [](void *c, int i) {
        Job *j = (Job *)c;
        check_graph_span(j->v, j->lo + j->span * i / j->pieces, j->lo + j->span * (i + 1) / j->pieces, &j->parts[i]);
    }, &job);
    GraphChecks all;
    for (int i = 0; i < pieces; ++i) {
        const GraphChecks &c = job.parts[i];
        all.bad_count |= c.bad_count; all.bad_index |= c.bad_index; all.bad_edges |= c.bad_edges; all.types |= c.types;
        all.n_min = std::min(all.n_min, c.n_min); all.n_max = std::max(all.n_max, c.n_max);
    }
    if (all.bad_count) return fail(GTM_ERR_ARG, "a graph has no nodes or more than max_number_of_graph_nodes = %d", v->max_number_of_graph_nodes);
    if (all.bad_index) return fail(GTM_ERR_ARG, "node_index is not the running sum of number_of_graph_nodes (or exceeds total_nodes)");
    if (all.bad_edges) return fail(GTM_ERR_ARG, "edge_index is not the running sum of number_of_graph_node_edges (or exceeds total_edges)");
    if (all_out) *all_out = all;
    return GTM_OK;
}

static int check_view_on_host(const gtm_graphs_view *v)
{
    GTM_TRY(check_on_host(v->X, "X"));
    GTM_TRY(check_on_host(v->node_type, "node_type"));
    GTM_TRY(check_on_host(v->number_of_graph_node_edges, "number_of_graph_node_edges"));
    GTM_TRY(check_on_host(v->edge_index, "edge_index"));
    GTM_TRY(check_on_host(v->edge, "edge"));
    GTM_TRY(check_on_host(v->node_index, "node_index"));
    return check_on_host(v->number_of_graph_nodes, "number_of_graph_nodes");
}

static int check_view(const gtm_graphs_view *v)
{
    if (!v) return fail(GTM_ERR_ARG, "null argument");
    if (v->number_of_graphs < 1 || v->total_nodes < 1) return fail(GTM_ERR_ARG, "empty graph set");
    if (!v->X || !v->node_type || !v->number_of_graph_node_edges || !v->edge_index || !v->node_index || !v->number_of_graph_nodes)
        return fail(GTM_ERR_ARG, "graph arrays must not be null");
    if (v->total_edges < 0 || (v->total_edges > 0 && !v->edge)) return fail(GTM_ERR_ARG, "edge array is null but total_edges > 0");
    if (v->max_number_of_graph_nodes < 1) return fail(GTM_ERR_ARG, "max_number_of_graph_nodes must be positive");
    if (v->total_nodes >= (int64_t)1 << 31 || v->total_edges >= (int64_t)1 << 31)
        return fail(GTM_ERR_ARG, "graph sets beyond 2^31 nodes or edges are not supported");
    if (v->number_of_graphs > v->total_nodes) return fail(GTM_ERR_ARG, "more graphs than nodes");
    return GTM_OK;
}

extern "C" int gtm_validate_graphs(const gtm_graphs_view *v)
{
    GTM_TRY(check_view(v));
    struct Keep { Keep() { stage_retain(-1); } ~Keep() { stage_drop(); } } keep;      // the copy threads stay while they check
    return validate_graphs(v, 0, v->number_of_graphs);
}

// What the copies of graphs [g0, g1) leave to the device: constant arrays, index arrays of equally large graphs, and the
// edge rows of every graph (first and number; graphs own consecutive CSR rows).
struct RangeFill {
    int64_t g0, g1, v0, v1;
    u32 e0;
    int uniform_n;          // > 0: every graph has this many nodes; node_index and n_nodes are made here
    int no_types;           // every node has type 0
    int no_edges;           // no node has an edge: degree is 0, edge_index is e0
    int next_graph;         // node_index of graph g1 is made too: a tile ends where the next graph's nodes begin
    u32 *node_type, *degree, *edge_index, *node_index, *n_nodes, *graph_edge0, *graph_edges;
};

__global__ void __launch_bounds__(256) fill_range_kernel(RangeFill f)
{
    const int64_t t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
    if (f.no_types)
        for (int64_t i = f.v0 + t0; i < f.v1; i += step) f.node_type[i] = 0;
    if (f.no_edges)
        for (int64_t i = f.v0 + t0; i < f.v1; i += step) { f.degree[i] = 0; f.edge_index[i] = f.e0; }
    for (int64_t gi = f.g0 + t0; gi < f.g1; gi += step) {
        u32 first, n;
        if (f.uniform_n > 0) {
            first = (u32)(f.v0 + (gi - f.g0) * f.uniform_n); n = (u32)f.uniform_n;
            f.node_index[gi] = first;
            f.n_nodes[gi] = n;
        } else {
            first = f.node_index[gi]; n = f.n_nodes[gi];
        }
        const u32 start = f.no_edges ? f.e0 : f.edge_index[first], last = first + n - 1;
        f.graph_edge0[gi] = start;
        f.graph_edges[gi] = f.no_edges ? 0u : f.edge_index[last] + f.degree[last] - start;
    }
    if (f.uniform_n > 0 && f.next_graph && t0 == 0) f.node_index[f.g1] = (u32)f.v1;
}

// Graphs [g0, g1) of the set: copies queued on stream `in`, and the rest of their arrays described for fill_range_kernel.
static int upload_range(gtm_dataset *ds, const gtm_graphs_view *v, StageLane *lane, int64_t g0, int64_t g1, const GraphChecks &facts, cudaStream_t in,
                        RangeFill *fill)
{
    const DevGraphs &dg = ds->dg;
    const int64_t N = v->number_of_graphs;
    const int L0 = ds->model->dm.L0;
    RangeFill f;
    memset(&f, 0, sizeof f);
    f.g0 = g0; f.g1 = g1;
    f.v0 = v->node_index[g0]; f.v1 = g1 < N ? (int64_t)v->node_index[g1] : v->total_nodes;
    f.e0 = v->edge_index[f.v0];
    const int64_t e1 = f.v1 < v->total_nodes ? (int64_t)v->edge_index[f.v1] : v->total_edges;
    f.uniform_n = facts.n_min == facts.n_max ? (int)facts.n_min : 0;
    f.no_types = facts.types == 0;
    f.no_edges = e1 == (int64_t)f.e0;
    f.next_graph = g1 < N;
    f.node_type = const_cast<u32 *>(dg.node_type); f.degree = const_cast<u32 *>(dg.degree); f.edge_index = const_cast<u32 *>(dg.edge_index);
    f.node_index = const_cast<u32 *>(dg.node_index); f.n_nodes = const_cast<u32 *>(dg.n_nodes);
    f.graph_edge0 = const_cast<u32 *>(dg.graph_edge0); f.graph_edges = const_cast<u32 *>(dg.graph_edges);
    *fill = f;
    const bool pinned = host_is_pinned(v->X);
    auto up = [&](const u32 *dst, const u32 *src, size_t first, size_t count, bool pin) {
        return stage_up(lane, const_cast<u32 *>(dst) + first, src + first, count * sizeof(u32), pin, in);
    };
    const size_t v0 = (size_t)f.v0, nodes = (size_t)(f.v1 - f.v0), graphs = (size_t)(g1 - g0);
    GTM_TRY(up(dg.X, v->X, v0 * L0, nodes * L0, pinned));
    if (!f.no_types) GTM_TRY(up(dg.node_type, v->node_type, v0, nodes, host_is_pinned(v->node_type)));
    if (!f.no_edges) {
        GTM_TRY(up(dg.degree, v->number_of_graph_node_edges, v0, nodes, host_is_pinned(v->number_of_graph_node_edges)));
        GTM_TRY(up(dg.edge_index, v->edge_index, v0, nodes, host_is_pinned(v->edge_index)));
        GTM_TRY(up(dg.edge, v->edge, 2 * (size_t)f.e0, 2 * (size_t)(e1 - f.e0), host_is_pinned(v->edge)));
    }
    if (f.uniform_n == 0) {
        GTM_TRY(up(dg.node_index, v->node_index, (size_t)g0, graphs + (g1 < N ? 1 : 0), host_is_pinned(v->node_index)));
        GTM_TRY(up(dg.n_nodes, v->number_of_graph_nodes, (size_t)g0, graphs, host_is_pinned(v->number_of_graph_nodes)));
    }
    return GTM_OK;
}

static int fill_range(const RangeFill &f, cudaStream_t s)
{
    const int64_t items = std::max(f.no_types || f.no_edges ? f.v1 - f.v0 : 0, f.g1 - f.g0);
    fill_range_kernel<<<(unsigned)std::min<int64_t>((items + 255) / 256, 1024), 256, 0, s>>>(f);
    GTM_CU(cudaGetLastError());
    return GTM_OK;
}

// A small set: validated, laid out in page-locked memory as it will lie on the device, one copy.
static int upload_small(gtm_dataset *ds, const gtm_graphs_view *v, StageLane *lane, const SetLayout &l, char *dev, cudaStream_t s)
{
    char *img = lane->small;
    const size_t nodes = (size_t)v->total_nodes, graphs = (size_t)v->number_of_graphs;
    memcpy(img + l.X, v->X, nodes * ds->model->dm.L0 * sizeof(u32));
    memcpy(img + l.node_type, v->node_type, nodes * sizeof(u32));
    memcpy(img + l.degree, v->number_of_graph_node_edges, nodes * sizeof(u32));
    memcpy(img + l.edge_index, v->edge_index, nodes * sizeof(u32));
    if (v->total_edges) memcpy(img + l.edge, v->edge, 2 * (size_t)v->total_edges * sizeof(u32));
    memcpy(img + l.node_index, v->node_index, graphs * sizeof(u32));
    memcpy(img + l.n_nodes, v->number_of_graph_nodes, graphs * sizeof(u32));
    u32 *e0 = (u32 *)(img + l.edge0), *ne = (u32 *)(img + l.edges);
    for (size_t gi = 0; gi < graphs; ++gi) {
        const u32 first = v->node_index[gi], last = first + v->number_of_graph_nodes[gi] - 1;
        e0[gi] = v->edge_index[first];
        ne[gi] = v->edge_index[last] + v->number_of_graph_node_edges[last] - e0[gi];
    }
    GTM_CU(cudaMemcpyAsync(dev, img, l.bytes, cudaMemcpyHostToDevice, s));
    return GTM_OK;
}

enum class SetCopy { whole, in_ranges };        // in_ranges: the caller validates and copies the arrays range by range

// Allocates the set's arrays and plans its scoring; the copies (SetCopy::whole) are queued on the model's stream and may
// still be running when this returns.
static int dataset_build(gtm_model *m, const gtm_graphs_view *v, gtm_dataset *ds, SetCopy copy, StageLane *lane)
{
    const DevModel &d = m->dm;
    cudaStream_t s = m->stream;
    const SetLayout l = set_layout(v, d.L0);
    char *dev;
    GTM_TRY(scratch(ds, &dev, l.bytes));
    DevGraphs &dg = ds->dg;
    dg.X = (u32 *)(dev + l.X); dg.node_type = (u32 *)(dev + l.node_type); dg.degree = (u32 *)(dev + l.degree);
    dg.edge_index = (u32 *)(dev + l.edge_index); dg.edge = (u32 *)(dev + l.edge);
    dg.node_index = (u32 *)(dev + l.node_index); dg.n_nodes = (u32 *)(dev + l.n_nodes);
    dg.graph_edge0 = (u32 *)(dev + l.edge0); dg.graph_edges = (u32 *)(dev + l.edges);
    dg.n_types = 1;
    dg.total_nodes = (u32)v->total_nodes; dg.total_edges = (u32)v->total_edges;
    dg.max_nodes = ds->max_nodes; dg.error = m->score_error;
    if (copy == SetCopy::whole) {
        GraphChecks facts;
        GTM_TRY(validate_graphs(v, 0, v->number_of_graphs, &facts));
        ds->n_min = facts.n_min; ds->n_max = facts.n_max;
        if (l.bytes <= kStageSmall) {
            GTM_TRY(upload_small(ds, v, lane, l, dev, s));
        } else {
            RangeFill f;
            GTM_TRY(upload_range(ds, v, lane, 0, v->number_of_graphs, facts, s, &f));
            GTM_TRY(fill_range(f, s));
        }
    } else if (ds->max_nodes > 1) {                      // not validated yet: the tilings take these only as hints
        u32 lo = ~0u, hi = 0;
        for (int64_t gi = 0; gi < v->number_of_graphs; ++gi) {
            lo = std::min(lo, v->number_of_graph_nodes[gi]);
            hi = std::max(hi, v->number_of_graph_nodes[gi]);
        }
        if (lo >= 1 && hi <= (u32)ds->max_nodes) { ds->n_min = lo; ds->n_max = hi; }
    }

    // general scoring scratch: one slice per resident CTA
    // General scoring kernel, shared memory per CTA: vote partial; for depth > 1 the source-node message bits of a graph
    // (flush_messages) when they are small enough not to cost resident CTAs; for graph sets of 33..1024 nodes per graph the
    // transposed copy of the graph - and then the message bits too (up to 64 KB), in CTAs of 512 threads, one or two per SM.
    const size_t p_words = (size_t)std::max(1, d.D - 1) * ds->max_nodes * d.MW;
    ds->score_part_words = 0;
    ds->score_t_stride = 0;
    ds->score_block = 256;
    ds->score_smem = (size_t)((d.K + 3) & ~3) * sizeof(int);
    const size_t msg_bytes = (size_t)(((ds->max_nodes + 31) & ~31) + kTransposedTypes) * (d.MW | 1) * sizeof(u32);   // padded rows + per-type rows, see ScatterTargets
    {
        const int t_stride = ds->NC | 1;
        const size_t t_bytes = ((size_t)32 * std::max(d.L0, d.MW) + kTransposedTypes) * t_stride * sizeof(u32);
        if (ds->max_nodes > 32 && ds->NC <= 32 && t_bytes <= 96 * 1024) {
            ds->score_t_stride = t_stride;
            ds->score_smem += t_bytes;
            ds->score_block = 512;
        }
    }
    if (d.D > 1 && (msg_bytes <= 8 * 1024 || (ds->score_t_stride > 0 && msg_bytes <= 72 * 1024))) {
        ds->score_part_words = (int)(msg_bytes / sizeof(u32));
        ds->score_smem += msg_bytes;
    }
    // small models on small graphs: a warp per graph, eight graphs per CTA (score_small_graphs_kernel)
    ds->score_units = 1;
    if (ds->max_nodes <= 32 && d.C <= 128) {
        const size_t per_warp = ((size_t)((d.K + 3) & ~3) + ds->score_part_words) * sizeof(int);
        if (8 * per_warp <= 40 * 1024) {
            ds->score_units = 8;
            ds->score_smem = 8 * per_warp;
        }
    }
    ds->cno_stride = (size_t)2 * d.C * ds->NC;
    ds->P_stride = p_words;
    ds->ninc_stride = (size_t)d.C;
    ds->score_sc.NC = ds->NC; ds->score_sc.cno_slots = 2; ds->score_sc.max_nodes = ds->max_nodes;
    ds->score_sc.cno = nullptr;   // allocated on first use of the general kernel (ensure_score_scratch)

    GTM_TRY(stream_data_create(&ds->sd, m->sm, d, v, ds->n_min, ds->n_max, m->sm_count, s));
    // tiles of whole graphs for the tile kernel: deeper models, or sets the node-stream kernel does not cover
    if (d.D > 1 || !ds->sd.supported || m->opt_score_kernel == 3) GTM_TRY(tile_data_create(&ds->td, m->tm, d, v, ds->n_min, ds->n_max, m->sm_count, s));
    return GTM_OK;
}

static int dataset_create(gtm_model *m, const gtm_graphs_view *v, gtm_dataset **out, SetCopy copy, StageLane *lane)
{
    *out = nullptr;
    gtm_dataset *ds = new (std::nothrow) gtm_dataset();
    if (!ds) return fail(GTM_ERR_OOM, "host allocation failed");
    ds->model = m;
    ds->n_graphs = v->number_of_graphs; ds->total_nodes = v->total_nodes; ds->total_edges = v->total_edges;
    ds->max_nodes = v->max_number_of_graph_nodes;
    ds->NC = words_for(ds->max_nodes);
    const int st = dataset_build(m, v, ds, copy, lane);
    if (st != GTM_OK) {
        cudaStreamSynchronize(m->stream);               // nothing may still be reading the host arrays when the call returns
        gtm_dataset_destroy(ds);
        return st;
    }
    *out = ds;
    return GTM_OK;
}

extern "C" int gtm_dataset_create(gtm_model *m, const gtm_graphs_view *v, gtm_dataset **out)
{
    GTM_TRY(bind(m));
    if (!v || !out) return fail(GTM_ERR_ARG, "null argument");
    *out = nullptr;
    GTM_TRY(check_view(v));
    GTM_TRY(check_view_on_host(v));
    LaneGuard guard;
    GTM_TRY(lane_acquire(m->cfg.device, &guard.lane));
    GTM_TRY(dataset_create(m, v, out, SetCopy::whole, guard.lane));
    const cudaError_t e = cudaStreamSynchronize(m->stream);
    if (e != cudaSuccess) { gtm_dataset_destroy(*out); *out = nullptr; }
    GTM_CU(e);
    return GTM_OK;
}

extern "C" int gtm_dataset_destroy(gtm_dataset *ds)
{
    if (!ds) return GTM_OK;
    cudaSetDevice(ds->model->cfg.device);
    for (void *p : ds->owned) cudaFreeAsync(p, ds->model->stream);        // in stream order, behind the kernels that use them
    if (ds->Y) cudaFree(ds->Y);
    stream_data_destroy(&ds->sd, ds->model->stream);
    tile_data_destroy(&ds->td, ds->model->stream);
    if (ds->comm.block) cudaStreamSynchronize(ds->model->stream);
    fit_comm_release(ds);
    delete ds;
    return GTM_OK;
}

// Scratch of the learning kernels (every layer kept), made when the set is first learned from or evaluated by a tap.
int ensure_fit_scratch(gtm_dataset *ds)
{
    if (ds->fit_sc.cno) return GTM_OK;
    const DevModel &d = ds->model->dm;
    const size_t p_words = (size_t)std::max(1, d.D - 1) * ds->max_nodes * d.MW;
    ds->fit_sc.NC = ds->NC; ds->fit_sc.cno_slots = d.D; ds->fit_sc.max_nodes = ds->max_nodes;
    u32 *cno;
    GTM_TRY(scratch(ds, &cno, (size_t)d.D * d.C * ds->NC));
    GTM_TRY(scratch(ds, &ds->fit_sc.n_inc, (size_t)d.C));
    GTM_TRY(scratch(ds, &ds->P_pair[0], p_words));
    GTM_TRY(scratch(ds, &ds->P_pair[1], p_words));
    GTM_TRY(scratch(ds, &ds->Q_pair[0], p_words));
    GTM_TRY(scratch(ds, &ds->Q_pair[1], p_words));
    GTM_TRY(scratch(ds, &ds->rank_barrier, 64));
    ds->fit_sc.P = ds->P_pair[0];
    ds->fit_sc.cno = cno;
    return GTM_OK;
}

// ---------------------------------------------------------------------------------------------- scoring
static int check_range(gtm_model *m, gtm_dataset *ds, int n_types, int64_t first, int64_t count)
{
    if (!ds || ds->model != m) return fail(GTM_ERR_ARG, "dataset does not belong to this model");
    if (!m->has_state) return fail(GTM_ERR_STATE, "model has no state: call gtm_init_state or gtm_set_ta_state first");
    if (n_types < 1) return fail(GTM_ERR_ARG, "number_of_node_types must be positive");
    if (first < 0 || count < 0 || first + count > ds->n_graphs)
        return fail(GTM_ERR_ARG, "graph range [%lld, %lld) outside the set of %lld graphs", (long long)first,
                    (long long)(first + count), (long long)ds->n_graphs);
    return GTM_OK;
}

// What the word that scoring kernels raise means to the caller (page-locked host memory that the device writes; the
// stream has been waited for).  Cleared once it was seen.
static int score_flag_status(gtm_model *m)
{
    const int flag = *(volatile int *)m->score_error;
    if (flag == 0) return GTM_OK;
    *(volatile int *)m->score_error = 0;
    if (flag == 2) return fail(GTM_ERR_TIMEOUT, "a scoring kernel gave up waiting for a bulk copy into shared memory; the class sums are not valid");
    return fail(GTM_ERR_ARG, "a scoring kernel skipped a malformed graph (node count or node range out of bounds)");
}

// Launch shape and scratch of the general scoring kernel, made on its first use.
static int ensure_score_scratch(gtm_dataset *ds)
{
    if (ds->score_sc.cno) return GTM_OK;
    const void *fn = score_kernel_for(ds->max_nodes, ds->score_units);
    if (ds->score_smem > 48 * 1024) GTM_CU(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 224 * 1024));   // not the set's own: another set may need more
    int per_sm = 0;
    GTM_CU(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, ds->score_block, ds->score_smem));
    ds->score_grid = (int)std::max<int64_t>(1, std::min<int64_t>((int64_t)ds->model->sm_count * std::max(1, per_sm), ds->n_graphs));
    const size_t slices = (size_t)ds->score_grid * ds->score_units;     // one slice per graph in flight
    u32 *cno;
    GTM_TRY(scratch(ds, &cno, ds->cno_stride * slices));
    GTM_TRY(scratch(ds, &ds->score_sc.P, ds->P_stride * slices));
    GTM_TRY(scratch(ds, &ds->score_sc.n_inc, ds->ninc_stride * slices));
    ds->score_sc.cno = cno;
    return GTM_OK;
}

static int launch_score_general(gtm_model *m, gtm_dataset *ds, int n_types, int64_t first, int64_t count,
                                int *sums_dev, int *clause_out_dev, int *node_out_dev = nullptr, int node_stride = 0)
{
    GTM_TRY(ensure_score_scratch(ds));
    DevGraphs g = ds->dg;
    g.n_types = n_types;
    ScoreArgs a;
    a.first = first; a.count = count; a.class_sums = sums_dev; a.clause_outputs = clause_out_dev;
    a.node_outputs = node_out_dev; a.node_stride = node_stride;
    a.cno_stride = ds->cno_stride; a.P_stride = ds->P_stride; a.ninc_stride = ds->ninc_stride;
    a.part_words = ds->score_part_words; a.t_stride = ds->score_t_stride;
    const int grid = (int)std::min<int64_t>(ds->score_grid, (count + ds->score_units - 1) / ds->score_units);
    {
        DevModel dm = m->dm;
        EvalScratch sc = ds->score_sc;
        void *args[] = {&dm, &g, &sc, &a};
        GTM_CU(cudaLaunchKernel(score_kernel_for(ds->max_nodes, ds->score_units), dim3(grid), dim3(ds->score_block), args, ds->score_smem, m->stream));
    }
    GTM_CU(cudaGetLastError());
    return GTM_OK;
}

static int refresh_lists(gtm_model *m)
{
    if (!m->lists_dirty) return GTM_OK;
    GTM_TRY(stream_model_refresh(&m->sm, m->dm, m->stream));
    m->lists_dirty = false;
    return GTM_OK;
}

static int refresh_tile_lists(gtm_model *m)
{
    if (m->tile_lists_version == m->state_version) return GTM_OK;
    GTM_TRY(tile_model_refresh(&m->tm, m->dm, m->stream));
    m->tile_lists_version = m->state_version;
    return GTM_OK;
}

static bool scores_by_stream(gtm_model *m, gtm_dataset *ds, int n_types)
{
    return (m->opt_score_kernel == 0 || m->opt_score_kernel == 2) && stream_supported(ds->sd, n_types);
}

// The option that forces the tile kernel stands for tiles of several graphs and one pass of the votes, and is an error beyond.
// So are tiles that a set got for its first transform: the option is to be set before the set is made.
static bool scores_by_tile(gtm_model *m, gtm_dataset *ds, int n_types)
{
    if (!tile_supported(ds->td, n_types)) return false;
    return m->opt_score_kernel == 0 || (m->opt_score_kernel == 3 && !ds->td.span && m->dm.K <= 16 && !ds->tiles_tried);
}

// One launch of a tiled kernel; clause_out_dev: the tile kernel only.  Its scratch belongs to the launch alone: kept with the
// model or the set, launches on two streams would share it.
static int launch_score_tiled(gtm_model *m, gtm_dataset *ds, bool by_stream, int n_types, int64_t first, int64_t count, int *sums_dev,
                              int *clause_out_dev, char *scratch, cudaStream_t s)
{
    if (by_stream) return stream_score(m->sm, ds->sd, m->dm, ds->dg, n_types, first, count, sums_dev, scratch, s);
    return tile_score(m->tm, ds->td, m->dm, ds->dg, n_types, first, count, sums_dev, clause_out_dev, m->score_error, scratch, s);
}

static size_t tiled_scratch_bytes(const gtm_model *m, const gtm_dataset *ds, bool by_stream, int64_t first, int64_t count)
{
    return by_stream ? stream_scratch_bytes(ds->sd, m->dm, first, count) : tile_scratch_bytes(ds->td, m->dm, first, count);
}

// The same on the model's stream, with lists and scratch: the lane's for a call that waits for its kernels, and else, without a
// lane, a block from the memory pool in stream order.
static int score_tiled(gtm_model *m, gtm_dataset *ds, bool by_stream, int n_types, int64_t first, int64_t count, int *sums_dev,
                       int *clause_out_dev, StageLane *lane)
{
    GTM_TRY(by_stream ? refresh_lists(m) : refresh_tile_lists(m));
    const size_t need = tiled_scratch_bytes(m, ds, by_stream, first, count);
    if (lane) {
        GTM_TRY(lane_scratch(lane, 0, need));
        return launch_score_tiled(m, ds, by_stream, n_types, first, count, sums_dev, clause_out_dev, lane->scratch[0], m->stream);
    }
    char *scratch;
    GTM_TRY(pool_alloc(&scratch, need, m->stream));
    const int st = launch_score_tiled(m, ds, by_stream, n_types, first, count, sums_dev, clause_out_dev, scratch, m->stream);
    cudaFreeAsync(scratch, m->stream);
    return st;
}

static int score_device(gtm_model *m, gtm_dataset *ds, int n_types, int64_t first, int64_t count, int32_t *sums_dev, StageLane *lane)
{
    GTM_TRY(bind(m));
    GTM_TRY(check_range(m, ds, n_types, first, count));
    if (count == 0) return GTM_OK;
    if (!sums_dev) return fail(GTM_ERR_ARG, "class_sums_device is null");
    if (m->opt_score_kernel == 2 && !stream_supported(ds->sd, n_types))
        return fail(GTM_ERR_ARG, "the node-stream scoring kernel does not cover this model / graph set");
    if (m->opt_score_kernel == 3 && !scores_by_tile(m, ds, n_types))
        return fail(GTM_ERR_ARG, "the tile scoring kernel does not cover this model / graph set");
    const bool by_stream = scores_by_stream(m, ds, n_types);
    if (by_stream || scores_by_tile(m, ds, n_types)) return score_tiled(m, ds, by_stream, n_types, first, count, sums_dev, nullptr, lane);
    return launch_score_general(m, ds, n_types, first, count, sums_dev, nullptr);
}

extern "C" int gtm_score_device(gtm_model *m, gtm_dataset *ds, int n_types, int64_t first, int64_t count,
                                int32_t *sums_dev)
{
    GTM_TRY(score_device(m, ds, n_types, first, count, sums_dev, nullptr));
    return note_queued(m);
}

// Scoring of graphs [first, first+count) into host memory by a tiled kernel, pipelined: chunks of whole tiles are scored
// on two streams in turn, so that one chunk's last tiles and the next one's first share the chip, and class sums go back
// on a copy stream meanwhile.  With `v` (and the whole set as the range) the set's arrays go up too, chunk by chunk on
// another copy stream - a chunk is the literal rows, per-node arrays and edge rows of a contiguous range of graphs -, each
// validated just before it is copied and scored when it has landed.
static int score_in_chunks(gtm_model *m, gtm_dataset *ds, const gtm_graphs_view *v, bool by_stream, int n_types, int64_t first, int64_t count,
                           int32_t *out, StageLane *lane)
{
    const DevModel &d = m->dm;
    const int64_t n = ds->n_graphs;
    const int uniform_gpt = by_stream ? ds->sd.graphs_per_tile : ds->td.graphs_per_tile;
    const std::vector<int> &table = by_stream ? ds->sd.tile_graph_host : ds->td.tile_graph_host;
    const int all_tiles = by_stream ? ds->sd.n_tiles : ds->td.n_tiles;
    auto tile_first = [&](int t) -> int64_t {           // first graph of tile t
        if (t >= all_tiles) return n;
        return uniform_gpt > 0 ? std::min<int64_t>((int64_t)t * uniform_gpt, n) : (int64_t)table[(size_t)t];
    };
    auto tile_of = [&](int64_t g) -> int {
        return uniform_gpt > 0 ? (int)(g / uniform_gpt) : (int)(std::upper_bound(table.begin(), table.end(), (int)g) - table.begin()) - 1;
    };
    const int t_lo = tile_of(first), t_hi = tile_of(first + count - 1) + 1, tiles = t_hi - t_lo;
    // Chunks of a quarter of the range, and of 1 to 8 MB where arrays go up: little of the copies is left uncovered and the
    // per-chunk work of the host stays small.  The tile kernel takes a tile per CTA: whole half-waves of them, two chunks
    // side by side fill the chip.
    int chunk_tiles = (tiles + 3) / 4;
    if (v) {
        const size_t tile_bytes = std::max<size_t>(1, set_layout(v, d.L0).bytes / (size_t)all_tiles);
        chunk_tiles = (int)std::max<size_t>(((size_t)1 << 20) / tile_bytes, std::min<size_t>((size_t)chunk_tiles, ((size_t)8 << 20) / tile_bytes)) + 1;
    }
    if (!by_stream) chunk_tiles = (chunk_tiles + m->sm_count - 1) / m->sm_count * m->sm_count;
    const bool pinned_out = host_is_pinned(out);
    auto chunk_lo = [&](int t0) { return std::max(first, tile_first(t0)); };
    auto chunk_hi = [&](int t0) { return std::min(first + count, tile_first(t0 + chunk_tiles)); };
    int *dev = nullptr;
    auto body = [&]() -> int {
        GTM_TRY(by_stream ? refresh_lists(m) : refresh_tile_lists(m));
        size_t need = 0;
        for (int t0 = t_lo; t0 < t_hi; t0 += chunk_tiles)
            if (chunk_hi(t0) > chunk_lo(t0)) need = std::max(need, tiled_scratch_bytes(m, ds, by_stream, chunk_lo(t0), chunk_hi(t0) - chunk_lo(t0)));
        for (int i = 0; i < (chunk_tiles < tiles ? 2 : 1); ++i) GTM_TRY(lane_scratch(lane, i, need));
        GTM_TRY(pool_alloc(&dev, (size_t)count * d.K, m->stream));
        GTM_CU(cudaEventRecord(lane->event[0], m->stream));       // allocations, tile tables and literal lists are in stream order
        GTM_CU(cudaStreamWaitEvent(lane->in, lane->event[0], 0));
        GTM_CU(cudaStreamWaitEvent(lane->aux, lane->event[0], 0));
        int turn = 0;
        for (int t0 = t_lo; t0 < t_hi; t0 += chunk_tiles, turn ^= 1) {
            const int64_t g0 = chunk_lo(t0), g1 = chunk_hi(t0);
            if (g1 <= g0) continue;
            const size_t cnt = (size_t)(g1 - g0), at = (size_t)(g0 - first) * d.K;
            cudaStream_t cs = turn ? lane->aux : m->stream;
            if (v) {
                GraphChecks facts;
                RangeFill f;
                GTM_TRY(validate_graphs(v, g0, g1, &facts));      // overlaps the copies of the chunks before
                GTM_TRY(upload_range(ds, v, lane, g0, g1, facts, lane->in, &f));
                GTM_CU(cudaEventRecord(lane->event[1], lane->in));
                GTM_CU(cudaStreamWaitEvent(cs, lane->event[1], 0));
                GTM_TRY(fill_range(f, cs));
            }
            GTM_TRY(launch_score_tiled(m, ds, by_stream, n_types, g0, (int64_t)cnt, dev + at, nullptr, lane->scratch[turn], cs));
            GTM_CU(cudaEventRecord(lane->event[2], cs));
            GTM_CU(cudaStreamWaitEvent(lane->back, lane->event[2], 0));
            GTM_TRY(stage_down(lane, out + at, dev + at, cnt * d.K * sizeof(int), pinned_out, lane->back));
        }
        GTM_CU(cudaEventRecord(lane->event[1], lane->aux));       // everything that used the set is in the order of the model's stream
        GTM_CU(cudaStreamWaitEvent(m->stream, lane->event[1], 0));
        GTM_TRY(stage_down_finish(lane));
        if (v) GTM_CU(cudaStreamSynchronize(lane->in));
        GTM_CU(cudaStreamSynchronize(m->stream));
        return score_flag_status(m);
    };
    const int st = body();
    if (st != GTM_OK) {                                           // nothing may still be reading the host arrays when the call returns
        stage_abandon(lane);
        cudaStreamSynchronize(m->stream);
    }
    if (dev) cudaFreeAsync(dev, m->stream);
    return st;
}

// Class sums of graphs [first, first+count) into host memory; waits for them.
static int score_to_host(gtm_model *m, gtm_dataset *ds, int n_types, int64_t first, int64_t count, int32_t *out, StageLane *lane)
{
    const size_t bytes = (size_t)count * m->dm.K * sizeof(int);
    // a few results: the kernel writes them to page-locked host memory itself, which takes less than starting a copy
    if (bytes <= 16 * 1024) {
        int *direct = (int *)(lane->small + kStageSmall);
        GTM_TRY(score_device(m, ds, n_types, first, count, direct, lane));
        GTM_CU(cudaStreamSynchronize(m->stream));
        GTM_TRY(score_flag_status(m));
        memcpy(out, direct, bytes);
        return GTM_OK;
    }
    // results whose way back (50 GB/s) is worth hiding behind the kernel
    if (bytes >= 512 * 1024) {
        const bool by_stream = scores_by_stream(m, ds, n_types);
        if (by_stream || scores_by_tile(m, ds, n_types)) return score_in_chunks(m, ds, nullptr, by_stream, n_types, first, count, out, lane);
    }
    int *dev;
    GTM_TRY(pool_alloc(&dev, (size_t)count * m->dm.K, m->stream));
    int st = score_device(m, ds, n_types, first, count, dev, lane);
    if (st == GTM_OK) st = stage_down(lane, out, dev, bytes, host_is_pinned(out), m->stream);
    cudaFreeAsync(dev, m->stream);
    if (st == GTM_OK) st = stage_down_finish(lane);
    if (st != GTM_OK) { stage_abandon(lane); cudaStreamSynchronize(m->stream); return st; }
    GTM_CU(cudaStreamSynchronize(m->stream));
    return score_flag_status(m);
}

extern "C" int gtm_score(gtm_model *m, gtm_dataset *ds, int n_types, int64_t first, int64_t count, int32_t *out)
{
    GTM_TRY(bind(m));
    GTM_TRY(check_range(m, ds, n_types, first, count));
    if (count == 0) return GTM_OK;
    if (!out) return fail(GTM_ERR_ARG, "class_sums_out is null");
    GTM_TRY(check_on_host(out, "class_sums_out"));
    LaneGuard guard;
    GTM_TRY(lane_acquire(m->cfg.device, &guard.lane));
    return score_to_host(m, ds, n_types, first, count, out, guard.lane);
}

// Upload and scoring of a whole host graph set in one call.  A small set is one copy, one kernel and one wait; larger sets
// that a tiled kernel covers are pipelined; other sets take gtm_dataset_create followed by gtm_score.
// The dataset stays valid for later calls either way.
extern "C" int gtm_dataset_create_scored(gtm_model *m, const gtm_graphs_view *v, int n_types, int32_t *out,
                                         gtm_dataset **dataset_out)
{
    GTM_TRY(bind(m));
    if (!v || !out || !dataset_out) return fail(GTM_ERR_ARG, "null argument");
    *dataset_out = nullptr;
    if (!m->has_state) return fail(GTM_ERR_STATE, "model has no state: call gtm_init_state or gtm_set_ta_state first");
    if (n_types < 1) return fail(GTM_ERR_ARG, "number_of_node_types must be positive");
    GTM_TRY(check_view(v));
    GTM_TRY(check_view_on_host(v));
    GTM_TRY(check_on_host(out, "class_sums_out"));
    LaneGuard guard;
    GTM_TRY(lane_acquire(m->cfg.device, &guard.lane));
    // what a tiled kernel may cover; stream_supported / tile_supported decide once the tiles are made
    const bool pipelined = m->opt_score_kernel != 1 && n_types <= 8 && v->max_number_of_graph_nodes <= 1024 &&
                           (m->sm.applicable || m->tm.applicable) && set_layout(v, m->dm.L0).bytes > kStageSmall;
    gtm_dataset *ds = nullptr;
    GTM_TRY(dataset_create(m, v, &ds, pipelined ? SetCopy::in_ranges : SetCopy::whole, guard.lane));
    const bool by_stream = pipelined && scores_by_stream(m, ds, n_types);
    const bool by_tile = pipelined && !by_stream && scores_by_tile(m, ds, n_types);
    int st;
    if (by_stream || by_tile) {
        st = score_in_chunks(m, ds, v, by_stream, n_types, 0, ds->n_graphs, out, guard.lane);
    } else {
        if (pipelined) {   // the arrays were not copied, but no tiled kernel turned out to cover the set
            gtm_dataset_destroy(ds);
            ds = nullptr;
            GTM_TRY(dataset_create(m, v, &ds, SetCopy::whole, guard.lane));
        }
        st = score_to_host(m, ds, n_types, 0, ds->n_graphs, out, guard.lane);
        if (st != GTM_OK) cudaStreamSynchronize(m->stream);
    }
    if (st != GTM_OK) { gtm_dataset_destroy(ds); return st; }
    *dataset_out = ds;
    return GTM_OK;
}

// Tiles of a set that was made without them: sets of models without message layers that the node-stream kernel scores.
static int ensure_tiles(gtm_model *m, gtm_dataset *ds)
{
    if (ds->td.supported || ds->tiles_tried || !m->tm.applicable) return GTM_OK;
    std::vector<u32> nodes;
    gtm_graphs_view v;
    memset(&v, 0, sizeof v);
    v.number_of_graphs = ds->n_graphs;
    v.max_number_of_graph_nodes = ds->max_nodes;
    if (ds->n_min != ds->n_max || ds->n_max == 0) {                       // ragged: the packing goes by the graphs' sizes
        nodes.resize((size_t)ds->n_graphs);
        GTM_CU(cudaMemcpyAsync(nodes.data(), ds->dg.n_nodes, nodes.size() * sizeof(u32), cudaMemcpyDeviceToHost, m->stream));
        GTM_CU(cudaStreamSynchronize(m->stream));
        v.number_of_graph_nodes = nodes.data();
    }
    GTM_TRY(tile_data_create(&ds->td, m->tm, m->dm, &v, ds->n_min, ds->n_max, m->sm_count, m->stream));
    GTM_CU(cudaStreamSynchronize(m->stream));                             // the packing's host arrays go out of scope
    ds->tiles_tried = true;
    return GTM_OK;
}

// clause outputs per graph and / or per node; results land in host arrays
static int transform_common(gtm_model *m, gtm_dataset *ds, int n_types, int64_t first, int64_t count, int32_t *clause_out,
                            int32_t *node_out, int node_stride, int32_t *sums_out)
{
    GTM_TRY(bind(m));
    GTM_TRY(check_range(m, ds, n_types, first, count));
    if (count == 0) return GTM_OK;
    GTM_TRY(check_on_host(clause_out, "clause_outputs_out"));
    GTM_TRY(check_on_host(node_out, "node_outputs_out"));
    GTM_TRY(check_on_host(sums_out, "class_sums_out"));
    int *sums_dev = nullptr, *co_dev = nullptr, *no_dev = nullptr;
    const size_t n_sums = (size_t)count * m->dm.K, n_co = (size_t)count * m->dm.C, n_no = n_co * (size_t)node_stride;
    LaneGuard guard;
    GTM_TRY(lane_acquire(m->cfg.device, &guard.lane));
    int st = pool_alloc(&sums_dev, n_sums, m->stream);
    if (st == GTM_OK && clause_out) st = pool_alloc(&co_dev, n_co, m->stream);
    if (st == GTM_OK && node_out) st = pool_alloc(&no_dev, n_no, m->stream);
    if (st == GTM_OK) {
        // clause outputs of whole graphs come out of the tile kernel too; outputs per node only out of the general one
        if (!node_out && clause_out && m->opt_score_kernel != 1) st = ensure_tiles(m, ds);
        if (st == GTM_OK && !node_out && clause_out && m->opt_score_kernel != 1 && tile_supported(ds->td, n_types)) {
            st = score_tiled(m, ds, false, n_types, first, count, sums_dev, co_dev, guard.lane);
        } else if (st == GTM_OK) {
            st = launch_score_general(m, ds, n_types, first, count, sums_dev, co_dev, no_dev, node_stride);
        }
    }
    auto down = [&](int32_t *host, const int *dev, size_t n) {
        if (st == GTM_OK && host) st = stage_down(guard.lane, host, dev, n * sizeof(int), host_is_pinned(host), m->stream);
    };
    down(sums_out, sums_dev, n_sums);
    down(clause_out, co_dev, n_co);
    down(node_out, no_dev, n_no);
    if (sums_dev) cudaFreeAsync(sums_dev, m->stream);
    if (co_dev) cudaFreeAsync(co_dev, m->stream);
    if (no_dev) cudaFreeAsync(no_dev, m->stream);
    if (st == GTM_OK) st = stage_down_finish(guard.lane);
    if (st != GTM_OK) stage_abandon(guard.lane);
    const cudaError_t e = cudaStreamSynchronize(m->stream);
    if (st != GTM_OK) return st;
    GTM_CU(e);
    return score_flag_status(m);
}

extern "C" int gtm_transform(gtm_model *m, gtm_dataset *ds, int n_types, int64_t first, int64_t count,
                             int32_t *clause_out, int32_t *sums_out)
{
    return transform_common(m, ds, n_types, first, count, clause_out, nullptr, 0, sums_out);
}

extern "C" int gtm_transform_nodewise(gtm_model *m, gtm_dataset *ds, int n_types, int64_t first, int64_t count,
                                      int node_stride, int32_t *node_out, int32_t *sums_out)
{
    if (!node_out) return fail(GTM_ERR_ARG, "node_outputs_out is null");
    if (!ds || node_stride < ds->max_nodes) return fail(GTM_ERR_ARG, "node_stride must be at least the largest graph's node count");
    return transform_common(m, ds, n_types, first, count, nullptr, node_out, node_stride, sums_out);
}

// --------------------------------------------------------------------------------------------- learning
extern "C" int gtm_fit(gtm_model *m, gtm_dataset *ds, int n_types, const int32_t *Y, int64_t first, int64_t count, int epochs)
{
    GTM_TRY(bind(m));
    GTM_TRY(check_range(m, ds, n_types, first, count));
    if (!Y) return fail(GTM_ERR_ARG, "encoded_Y is null");
    if (epochs < 0) return fail(GTM_ERR_ARG, "epochs must not be negative");
    if (count == 0 || epochs == 0) return GTM_OK;
    const size_t need = (size_t)ds->n_graphs * m->dm.K;
    if (ds->Y_capacity < need) {
        cudaFree(ds->Y); ds->Y = nullptr; ds->Y_capacity = 0;
        GTM_TRY(dev_alloc(&ds->Y, need));
        ds->Y_capacity = need;
    }
    GTM_CU(cudaMemcpyAsync(ds->Y + (size_t)first * m->dm.K, Y + (size_t)first * m->dm.K,
                           (size_t)count * m->dm.K * sizeof(int), cudaMemcpyHostToDevice, m->stream));
    m->lists_dirty = true; ++m->state_version;
    return launch_fit(m, ds, n_types, ds->Y, first, count, epochs, 0);
}

// ------------------------------------------------------------------------------------------------- taps
extern "C" int gtm_debug_evaluate(gtm_model *m, gtm_dataset *ds, int n_types, int64_t graph, int path,
                                  uint32_t *cno_out, uint32_t *msg_out, int32_t *n_inc_out, int32_t *class_sum_out)
{
    GTM_TRY(bind(m));
    GTM_TRY(check_range(m, ds, n_types, graph, 1));
    const DevModel &d = m->dm;
    GTM_TRY(ensure_fit_scratch(ds));
    std::vector<u32> nn(1), ni(1);
    GTM_CU(cudaMemcpy(nn.data(), ds->dg.n_nodes + graph, sizeof(u32), cudaMemcpyDeviceToHost));
    const int n = (int)nn[0], words = (n + 31) / 32;
    if (path == 1) {
        GTM_TRY(launch_fit(m, ds, n_types, nullptr, graph, 1, 1, 1));
        if (cno_out)
            for (int l = 0; l < d.D; ++l)
                GTM_CU(cudaMemcpy2D(cno_out + (size_t)l * d.C * words, words * sizeof(u32),
                                    ds->fit_sc.cno + (size_t)l * d.C * ds->NC, ds->NC * sizeof(u32),
                                    words * sizeof(u32), d.C, cudaMemcpyDeviceToHost));
        if (msg_out && d.D > 1) {
            u32 *tmp;
            GTM_TRY(dev_alloc(&tmp, (size_t)n * d.M));
            for (int l = 0; l < d.D - 1; ++l) {
                expand_messages_kernel<<<64, 256, 0, m->stream>>>(ds->P_pair[0] + (size_t)l * ds->max_nodes * d.MW, tmp, n, d.MS, d.MW, d.M);
                cudaMemcpyAsync(msg_out + (size_t)l * n * d.M, tmp, (size_t)n * d.M * sizeof(u32), cudaMemcpyDeviceToHost, m->stream);
            }
            cudaError_t e = cudaStreamSynchronize(m->stream);
            cudaFree(tmp);
            GTM_CU(e);
        }
        if (n_inc_out) GTM_CU(cudaMemcpy(n_inc_out, ds->fit_sc.n_inc, (size_t)d.C * sizeof(int), cudaMemcpyDeviceToHost));
        if (class_sum_out) GTM_CU(cudaMemcpy(class_sum_out, m->class_sum_tap, (size_t)d.K * sizeof(int), cudaMemcpyDeviceToHost));
        return GTM_OK;
    }
    if (path == 0) {
        // general scoring kernel with a one-CTA grid and every layer kept (scratch of the learning kernel)
        DevGraphs g = ds->dg;
        g.n_types = n_types;
        int *sums;
        GTM_TRY(dev_alloc(&sums, (size_t)d.K));
        ScoreArgs a;
        a.first = graph; a.count = 1; a.class_sums = sums; a.clause_outputs = nullptr; a.node_outputs = nullptr; a.node_stride = 0;
        a.cno_stride = a.P_stride = a.ninc_stride = 0;
        a.part_words = 0; a.t_stride = 0;
        EvalScratch sc = ds->fit_sc;
        sc.P = ds->P_pair[0];
        score_graphs_kernel<true><<<1, 256, (size_t)d.K * sizeof(int), m->stream>>>(d, g, sc, a);
        cudaError_t e = cudaStreamSynchronize(m->stream);
        if (e == cudaSuccess && class_sum_out) e = cudaMemcpy(class_sum_out, sums, (size_t)d.K * sizeof(int), cudaMemcpyDeviceToHost);
        cudaFree(sums);
        GTM_CU(e);
        if (cno_out)
            for (int l = 0; l < d.D; ++l)
                GTM_CU(cudaMemcpy2D(cno_out + (size_t)l * d.C * words, words * sizeof(u32),
                                    ds->fit_sc.cno + (size_t)l * d.C * ds->NC, ds->NC * sizeof(u32),
                                    words * sizeof(u32), d.C, cudaMemcpyDeviceToHost));
        if (msg_out && d.D > 1) {
            u32 *tmp;
            GTM_TRY(dev_alloc(&tmp, (size_t)n * d.M));
            for (int l = 0; l < d.D - 1; ++l) {
                expand_messages_kernel<<<64, 256, 0, m->stream>>>(ds->P_pair[0] + (size_t)l * ds->max_nodes * d.MW, tmp, n, d.MS, d.MW, d.M);
                cudaMemcpyAsync(msg_out + (size_t)l * n * d.M, tmp, (size_t)n * d.M * sizeof(u32), cudaMemcpyDeviceToHost, m->stream);
            }
            e = cudaStreamSynchronize(m->stream);
            cudaFree(tmp);
            GTM_CU(e);
        }
        if (n_inc_out) GTM_CU(cudaMemcpy(n_inc_out, ds->fit_sc.n_inc, (size_t)d.C * sizeof(int), cudaMemcpyDeviceToHost));
        return GTM_OK;
    }
    return fail(GTM_ERR_ARG, "path must be 0 (scoring kernel) or 1 (learning kernel)");
}

// Eight independent chains of three-input logic operations per thread, all in registers.
__global__ void __launch_bounds__(256) logic_op_rate_kernel(int iterations, u32 seed, u32 *sink)
{
    u32 x[8], a = seed ^ (threadIdx.x * 2654435761u), b = seed + blockIdx.x * 40503u;
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = a * (2 * i + 3) + b;
    for (int it = 0; it < iterations; ++it) {
#pragma unroll
        for (int r = 0; r < 8; ++r) {
#pragma unroll
            for (int i = 0; i < 8; ++i)                                       // one LOP3 each (bitwise select), chains independent of one another
                asm volatile("lop3.b32 %0, %0, %1, %2, 0xCA;" : "+r"(x[i]) : "r"(a), "r"(b));
        }
    }
    u32 v = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) v ^= x[i];
    if (v == 0x12345u) sink[0] = v;                                           // keeps the chains alive
}

extern "C" int gtm_debug_logic_op_rate(gtm_model *m, double *tera_ops_per_second_out)
{
    if (!m || !tera_ops_per_second_out) return fail(GTM_ERR_ARG, "null argument");
    GTM_TRY(bind(m));
    u32 *sink = nullptr;
    GTM_TRY(dev_alloc(&sink, 1));
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    const int iterations = 4096, grid = m->sm_count * 16;
    float ms = 0.0f;
    for (int rep = 0; rep < 3; ++rep) {          // the last repetition is the one reported
        cudaEventRecord(e0, m->stream);
        logic_op_rate_kernel<<<grid, 256, 0, m->stream>>>(iterations, 1u + rep, sink);
        cudaEventRecord(e1, m->stream);
        cudaEventSynchronize(e1);
        cudaEventElapsedTime(&ms, e0, e1);
    }
    cudaError_t e = cudaGetLastError();
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(sink);
    GTM_CU(e);
    *tera_ops_per_second_out = (double)grid * 256.0 * iterations * 64.0 / (ms * 1e-3) / 1e12;
    return GTM_OK;
}

extern "C" int gtm_debug_fit_phase_cycles(gtm_model *m, uint64_t *cycles_out)
{
    GTM_TRY(bind(m));
    if (!cycles_out) return fail(GTM_ERR_ARG, "cycles_out is null");
    GTM_CU(cudaStreamSynchronize(m->stream));
    GTM_CU(cudaMemcpy(cycles_out, m->phase_cycles, 8 * sizeof(uint64_t), cudaMemcpyDeviceToHost));
    return GTM_OK;
}

extern "C" int gtm_debug_last_fit_kernel(gtm_model *m, int32_t *info_out)
{
    GTM_TRY(bind(m));
    if (!info_out) return fail(GTM_ERR_ARG, "info_out is null");
    memcpy(info_out, m->last_fit, sizeof m->last_fit);
    return GTM_OK;
}

extern "C" int gtm_debug_last_feedback(gtm_model *m, int32_t *clause_node_out, int32_t *update_out)
{
    GTM_TRY(bind(m));
    GTM_CU(cudaStreamSynchronize(m->stream));
    if (clause_node_out) GTM_CU(cudaMemcpy(clause_node_out, m->clause_node, (size_t)m->dm.C * sizeof(int), cudaMemcpyDeviceToHost));
    if (update_out) GTM_CU(cudaMemcpy(update_out, m->update, (size_t)m->dm.K * m->dm.C * sizeof(int), cudaMemcpyDeviceToHost));
    return GTM_OK;
}

// ------------------------------------------------------------------------- scoring with built-in scratch
// Scratch of gtm_score_static_scratch: lives in the library image, so every GPU that loads the library holds these
// GTM_STATIC_SCRATCH_BYTES until the process exits.  In host code the name below is only a stand-in for the
// symbol, not a device address; the address is looked up once per device (g_static_scratch_addr).
static __device__ __align__(256) unsigned int g_static_scratch[GTM_STATIC_SCRATCH_BYTES / sizeof(unsigned int)];
static unsigned int *g_static_scratch_addr[64];

extern "C" int gtm_score_static_scratch(gtm_model *m, const gtm_graphs_view *v, int n_types, int64_t first, int64_t count,
                                        int32_t *sums_dev)
{
    GTM_TRY(bind(m));
    if (!v) return fail(GTM_ERR_ARG, "device_graphs is null");
    if (!m->has_state) return fail(GTM_ERR_STATE, "model has no state: call gtm_init_state or gtm_set_ta_state first");
    if (n_types < 1) return fail(GTM_ERR_ARG, "number_of_node_types must be positive");
    if (first < 0 || count < 0 || first + count > v->number_of_graphs)
        return fail(GTM_ERR_ARG, "graph range [%lld, %lld) outside the set of %lld graphs", (long long)first,
                    (long long)(first + count), (long long)v->number_of_graphs);
    if (count == 0) return GTM_OK;
    if (!sums_dev || !v->X || !v->node_type || !v->number_of_graph_node_edges || !v->edge_index || !v->node_index ||
        !v->number_of_graph_nodes || (v->total_edges > 0 && !v->edge))
        return fail(GTM_ERR_ARG, "device arrays must not be null");
    if (v->max_number_of_graph_nodes < 1) return fail(GTM_ERR_ARG, "max_number_of_graph_nodes must be positive");
    if (v->total_nodes < 1 || v->total_nodes >= (int64_t)1 << 31 || v->total_edges < 0 || v->total_edges >= (int64_t)1 << 31)
        return fail(GTM_ERR_ARG, "total_nodes must be in 1..2^31-1 and total_edges in 0..2^31-1");
    // layer-0 rows of a multiple of four words are read with 128-bit loads; every array is read as 32-bit words
    if ((m->dm.L0 & 3) == 0 && ((uintptr_t)v->X & 15) != 0)
        return fail(GTM_ERR_ARG, "X must be 16-byte aligned when a literal row is a multiple of 16 bytes (it is %d bytes here)", m->dm.L0 * 4);
    {
        const void *arrays[] = {v->X, v->node_type, v->number_of_graph_node_edges, v->edge_index, v->edge, v->node_index,
                                v->number_of_graph_nodes, sums_dev};
        for (const void *p : arrays)
            if (((uintptr_t)p & 3) != 0) return fail(GTM_ERR_ARG, "device arrays must be 4-byte aligned");
    }
    const int dev = m->cfg.device;
    if (dev >= 64) return fail(GTM_ERR_ARG, "device ordinal %d beyond the 64 this entry point keeps an address for", dev);

    const DevModel &d = m->dm;
    const int NC = words_for(v->max_number_of_graph_nodes);
    const size_t cno_words = (size_t)2 * d.C * NC;
    const size_t p_words = (size_t)std::max(1, d.D - 1) * v->max_number_of_graph_nodes * d.MW;
    const size_t per_cta = cno_words + p_words + (size_t)d.C;                       // words of scratch one CTA needs
    const size_t capacity = GTM_STATIC_SCRATCH_BYTES / sizeof(unsigned int);
    if (per_cta > capacity)
        return fail(GTM_ERR_ARG,
                    "model and graph sizes need %zu bytes of scratch per thread block; the built-in scratch holds %u bytes "
                    "(use gtm_dataset_create + gtm_score_device for this size)", per_cta * sizeof(unsigned int),
                    (unsigned)GTM_STATIC_SCRATCH_BYTES);

    // first call on this device: resolve the device address of the built-in array (this device is current)
    if (!g_static_scratch_addr[dev]) {
        unsigned int *addr = nullptr;
        GTM_CU(cudaGetSymbolAddress((void **)&addr, g_static_scratch));
        g_static_scratch_addr[dev] = addr;
    }
    unsigned int *scratch_base = g_static_scratch_addr[dev];

    const int64_t fit_ctas = (int64_t)(capacity / per_cta);
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(std::min<int64_t>(count, fit_ctas), (int64_t)m->sm_count * 4));

    DevGraphs g;
    memset(&g, 0, sizeof g);
    g.X = v->X; g.node_type = v->node_type; g.degree = v->number_of_graph_node_edges; g.edge_index = v->edge_index;
    g.edge = v->edge; g.node_index = v->node_index; g.n_nodes = v->number_of_graph_nodes;
    g.n_types = n_types;
    // the arrays are in device memory and cannot be checked here: the kernel skips graphs that would leave them or the
    // scratch slice and raises the word that gtm_check_skipped_graphs reads
    g.total_nodes = (u32)v->total_nodes; g.total_edges = (u32)v->total_edges;
    g.max_nodes = v->max_number_of_graph_nodes; g.error = m->score_error;
    EvalScratch sc;
    sc.cno = scratch_base;
    sc.P = scratch_base + cno_words;
    sc.n_inc = reinterpret_cast<int *>(scratch_base + cno_words + p_words);
    sc.NC = NC; sc.cno_slots = 2; sc.max_nodes = v->max_number_of_graph_nodes;
    ScoreArgs a;
    a.first = first; a.count = count; a.class_sums = sums_dev; a.clause_outputs = nullptr; a.node_outputs = nullptr; a.node_stride = 0;
    a.cno_stride = a.P_stride = a.ninc_stride = per_cta;                             // one contiguous slice per CTA
    a.part_words = 0; a.t_stride = 0;
    score_graphs_kernel<true><<<grid, 256, (size_t)d.K * sizeof(int), m->stream>>>(d, g, sc, a);
    GTM_CU(cudaGetLastError());
    return note_queued(m);
}

extern "C" int gtm_check_skipped_graphs(gtm_model *m, int *skipped_out)
{
    GTM_TRY(bind(m));
    if (!skipped_out) return fail(GTM_ERR_ARG, "skipped_out is null");
    GTM_CU(cudaStreamSynchronize(m->stream));
    const int flag = *(volatile int *)m->score_error;
    if (flag == 2) return score_flag_status(m);
    *(volatile int *)m->score_error = 0;
    *skipped_out = flag == 1;
    return GTM_OK;
}
