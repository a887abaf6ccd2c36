// The row-owning decode kernel for 5-bit weights.
#include "qmv_rows.cuh"

namespace b200q {
namespace rows {
template int launch_rows<5>(const RowsPlan& pl, cudaStream_t st);
}
}  // namespace b200q
