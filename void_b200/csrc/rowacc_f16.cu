// Row-accumulate kernels for fp16 and bf16 tiles.
#include "rowacc.cuh"

namespace vb {

template int launch_rowacc<VOID_KIND_F16>(const RowaccLaunch&);

}  // namespace vb
