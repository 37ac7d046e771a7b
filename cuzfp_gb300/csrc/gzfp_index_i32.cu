// Parallel block index of general-mode streams of int32_t fields.
#include "gzfp_index.cuh"

namespace gzfp {

template cudaError_t launch_index_fill<int32_t>(int, const IndexJob&, const IndexLists&,
                                            const IndexState*, bool, int, cudaStream_t);
template cudaError_t launch_index_sample<int32_t>(int, const IndexJob&, IndexState*, uint64_t, int,
                                              cudaStream_t);

}  // namespace gzfp
