// The row-owning decode kernel for 4-bit weights.
#include "qmv_rows.cuh"

namespace b200q {
namespace rows {
template int launch_rows<4>(const RowsPlan& pl, cudaStream_t st);
}
}  // namespace b200q
