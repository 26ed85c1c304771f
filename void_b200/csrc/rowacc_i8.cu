// Row-accumulate kernels for INT8 tiles.
#include "rowacc.cuh"

namespace vb {

template int launch_rowacc<VOID_KIND_I8>(const RowaccLaunch&);

}  // namespace vb
