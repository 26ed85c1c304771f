// Row-accumulate kernels for fp32 (TF32) tiles.
#include "rowacc.cuh"

namespace vb {

template int launch_rowacc<VOID_KIND_TF32>(const RowaccLaunch&);

}  // namespace vb
