// plan_emu.cpp — TEST INFRASTRUCTURE ONLY: the host plans that need no CUDA.
#include <cstddef>

#include "batch_plan.h"
#include "hostio.h"
#include "slice.h"

extern "C" {

double plan_slice_us(int64_t terms, int shots) { return ksim::slice_item_us(terms, shots); }
double plan_record_us(double stream_bytes, int64_t shots) { return ksim::record_item_us(stream_bytes, shots); }

int plan_tile_ok(int S, int shots, int threads) { return ksim::slice_tile_ok(S, shots, threads) ? 1 : 0; }

// Chunk boundaries of a host call; returns how many.
int plan_host_call(int64_t B, int64_t in_row, int64_t out_row, int sliced, int64_t n_terms, int64_t n_graphs,
                   int64_t sms, int64_t *out, int max)
{
    const ksim::HostCall c = {B, in_row, out_row, sliced != 0, n_terms, n_graphs, sms};
    const std::vector<int64_t> b = ksim::host_call_bounds(c);
    for (size_t i = 0; i < b.size() && (int)i < max; ++i) out[i] = b[i];
    return (int)b.size();
}
int plan_host_ramp(int64_t B, int64_t row, int64_t *out, int max)
{
    const std::vector<int64_t> b = ksim::host_chunk_bounds(B, row);
    for (size_t i = 0; i < b.size() && (int)i < max; ++i) out[i] = b[i];
    return (int)b.size();
}

}  // extern "C"
