// The plain sort's kernels and launch logic for 8-byte keys with items (all three key orders).
#define HPCS_INSTANTIATE_SORTS
#include "sort_host.cuh"

namespace hpcs {
template int enqueue_sort<uint64_t, KIND_UNSIGNED, uint32_t>(hpcs_ctx*, uint64_t*, uint32_t*, int64_t, cudaStream_t);
template int enqueue_sort<uint64_t, KIND_SIGNED, uint32_t>(hpcs_ctx*, uint64_t*, uint32_t*, int64_t, cudaStream_t);
template int enqueue_sort<uint64_t, KIND_FLOAT, uint32_t>(hpcs_ctx*, uint64_t*, uint32_t*, int64_t, cudaStream_t);
}  // namespace hpcs
