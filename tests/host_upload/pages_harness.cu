/*
 * pages_harness.cu -- TEST INFRASTRUCTURE ONLY.
 *
 * harness.cu with fn_download's page touching in sight; every pointer passes
 * for pageable memory.  For tests/test_download_pages_host.py.
 */
static cudaError_t hp_attributes(cudaPointerAttributes* a, const void*) {
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
#define cudaPointerGetAttributes hp_attributes
#include "harness.cu"

HU_API void hp_touch(void* buffer, size_t bytes) { touch_pages(buffer, bytes); }
