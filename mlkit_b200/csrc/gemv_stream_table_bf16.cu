// Instances of the streaming matvec: table codecs of 3 and 4 bits; bf16 activations.
#include "gemv_stream.cuh"

namespace mkb {
namespace stream {
template int dispatch_table<X_BF16>(const StreamArgs&, const StreamPlan&, cudaStream_t, int*);
}  // namespace stream
}  // namespace mkb
