// Streaming stage kernels for FP16 storage.
#include "stage_stream.cuh"

namespace cgfdm {

STREAM_INSTANTIATE(__half)

#if STREAM_PART == 0

template cudaError_t launch_stage_stream_batch<__half>(const StageArgs<__half> *,
                                                       const void *const *, int, int *, int *,
                                                       StreamPair, int *);
template bool stage_stream_supported<__half>();
template int encode_stream_maps<__half>(const __half *, const __half *, const __half *,
                                        const __half *, const __half *,
                                        const Layout &, void *);
template cudaError_t launch_stage_stream<__half>(const StageArgs<__half> &, const void *, int *,
                                                 int *, StreamPair, cudaEvent_t, int *, int);

#endif

}  // namespace cgfdm
