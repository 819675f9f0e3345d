// paths_nee.cu — the path kernel (paths.cuh) with next-event estimation.
#include "paths.cuh"

namespace solrt {

solrt_status launch_paths_nee(Context& ctx, uint32_t kind, const PathArgs& a) { return launch_paths_any<true>(ctx, kind, a); }

}  // namespace solrt
