// Real-space passes of the chain sweeps, complex64 (split_passes.cuh).
#define FTSP_SPLIT_INSTANCES
#include "split_passes.cuh"

namespace ftsp {
FTSP_SPLIT_REAL_ALL(template, float)
}  // namespace ftsp
