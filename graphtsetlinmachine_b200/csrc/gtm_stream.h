// Node-stream scoring (gtm_stream.cu): types and entry points used by the host runtime.
#pragma once
#include <vector>

#include "gtm_device.cuh"
#include "gtm_host.cuh"

namespace gtm {

struct StreamModel {
    bool applicable = false;
    int *lit_cnt = nullptr;             // [C]   list lengths (multiples of 4)
    unsigned short *lit_list = nullptr; // [C][list_stride] row numbers of the included literals
    int list_stride = 0;
    signed char *wf = nullptr;          // weights as tensor-core fragments, see stream_weight_at
    int *limbs = nullptr;               // signed bytes that the largest weight needs
};

struct StreamData {
    int supported = 0;
    int TNC = 0;                        // node words per tile
    int n_tiles = 0;
    int *tile_graph = nullptr;          // [n_tiles+1] first graph of every tile (NULL for sets of equally large graphs)
    int graphs_per_tile = 0;            // > 0: every tile holds this many graphs
    std::vector<int> tile_graph_host;
    int grid = 0;
    int64_t total_nodes = 0, n_graphs = 0;
};


int stream_model_create(StreamModel *sm, const DevModel &d);
void stream_model_destroy(StreamModel *sm);
int stream_model_refresh(StreamModel *sm, const DevModel &d, cudaStream_t s);
int stream_data_create(StreamData *sd, const StreamModel &sm, const DevModel &d, const gtm_graphs_view *v, u32 n_min, u32 n_max,
                       int sm_count, cudaStream_t s);
void stream_data_destroy(StreamData *sd, cudaStream_t s);
bool stream_supported(const StreamData &sd, int n_types);
// Bytes of scratch (256-byte aligned device memory, no contents expected) that a launch over graphs [first, first+count)
// needs.  The scratch belongs to one launch: launches on different streams share nothing.
size_t stream_scratch_bytes(const StreamData &sd, const DevModel &d, int64_t first, int64_t count);
int stream_score(const StreamModel &sm, const StreamData &sd, const DevModel &d, const DevGraphs &dg, int n_types,
                 int64_t first, int64_t count, int *sums_dev, char *scratch, cudaStream_t s);

}  // namespace gtm
