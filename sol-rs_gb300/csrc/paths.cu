// paths.cu — the path kernel (paths.cuh) without next-event estimation.
#include "paths.cuh"

namespace solrt {

solrt_status launch_paths(Context& ctx, uint32_t kind, const PathArgs& a) { return launch_paths_any<false>(ctx, kind, a); }

}  // namespace solrt
