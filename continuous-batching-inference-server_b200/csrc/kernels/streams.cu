// Streams that nobody else holds.  (Those of a pool are handed out in turn: two holders may have the same one, and what one
// launches on it while the other captures ends up in the other's graph.)
#include "common.cuh"

CBIS_EXPORT int cbis_stream_create(void** stream) {
  return (int)cudaStreamCreateWithFlags(reinterpret_cast<cudaStream_t*>(stream), cudaStreamNonBlocking);
}

CBIS_EXPORT int cbis_stream_destroy(void* stream) { return (int)cudaStreamDestroy((cudaStream_t)stream); }
