// Run-time passes of the grids without split passes, complex64 (passes.cuh).
#define FTSP_LINE_INSTANCES
#include "engine.cuh"

namespace ftsp {
FTSP_LINE_ALL(template, float)
}  // namespace ftsp
