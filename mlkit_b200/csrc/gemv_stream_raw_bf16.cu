// Instances of the streaming matvec: integer grids of 2, 3 and 5 to 8 bits; bf16 activations.
#include "gemv_stream.cuh"

namespace mkb {
namespace stream {
template int dispatch_raw<X_BF16>(const StreamArgs&, const StreamPlan&, cudaStream_t, int*);
}  // namespace stream
}  // namespace mkb
