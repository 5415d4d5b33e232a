// Instances of the streaming matvec: integer grids of 2, 3 and 5 to 8 bits; f16 activations.
#include "gemv_stream.cuh"

namespace mkb {
namespace stream {
template int dispatch_raw<X_F16>(const StreamArgs&, const StreamPlan&, cudaStream_t, int*);
}  // namespace stream
}  // namespace mkb
