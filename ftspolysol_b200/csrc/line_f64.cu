// Run-time passes of the grids without split passes, complex128 (passes.cuh).
#define FTSP_LINE_INSTANCES
#include "engine.cuh"

namespace ftsp {
FTSP_LINE_ALL(template, double)
}  // namespace ftsp
