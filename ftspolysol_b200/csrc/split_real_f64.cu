// Real-space passes of the chain sweeps, complex128 (split_passes.cuh).
#define FTSP_SPLIT_INSTANCES
#include "split_passes.cuh"

namespace ftsp {
FTSP_SPLIT_REAL_ALL(template, double)
}  // namespace ftsp
