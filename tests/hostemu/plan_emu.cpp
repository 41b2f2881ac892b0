// plan_emu.cpp — TEST INFRASTRUCTURE ONLY: the host plans that need no CUDA.
#include "batch_plan.h"

extern "C" {

double plan_slice_us(int64_t terms, int shots) { return ksim::slice_item_us(terms, shots); }
double plan_record_us(double stream_bytes, int64_t shots) { return ksim::record_item_us(stream_bytes, shots); }

}  // extern "C"
