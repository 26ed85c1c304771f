// Row-accumulate kernels for FP8 E4M3 tiles.
#include "rowacc.cuh"

namespace vb {

template int launch_rowacc<VOID_KIND_F8E4M3>(const RowaccLaunch&);

}  // namespace vb
