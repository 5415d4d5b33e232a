// Instances of the streaming matvec: integer grids of 4 bits, one, two or four scale groups per 128 codes, with and without offsets; bf16 activations.
#include "gemv_stream.cuh"

namespace mkb {
namespace stream {
template int dispatch_raw4<X_BF16>(const StreamArgs&, const StreamPlan&, cudaStream_t, int*);
}  // namespace stream
}  // namespace mkb
