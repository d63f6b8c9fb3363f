// A host stand-in for libhdc_gb300 behind dropin/gpu_dropin.cpp: "device" memory with a limit, a search that reports every
// query's first database entries, and a status word, so that the drop-in's handling of both can be checked without a GPU.
// argv: bytes that may be allocated, the status word.  Prints the workspace that the search was given.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <stdexcept>

#include "GPU.cuh"
#include "hdc_gb300.h"

namespace {
size_t limit_bytes = 0, used = 0;
int word = 0;
constexpr size_t kFull = (size_t)1 << 30, kLeast = 4096;
}  // namespace

struct hdc_context {};

extern "C" {
const char* hdc_last_error(void) { return "stub"; }
int hdc_context_create(int, int, int, int, hdc_context** out) {
    *out = new hdc_context;
    return HDC_OK;
}
int hdc_device_alloc(size_t bytes, void** out) {
    *out = nullptr;
    if (used + bytes > limit_bytes) return HDC_ERR_NOMEM;
    used += bytes;
    *out = std::malloc(bytes < 4096 ? 4096 : bytes);
    return HDC_OK;
}
int hdc_device_free(void* p) {
    std::free(p);
    return HDC_OK;
}
int hdc_copy(void* dst, const void* src, size_t bytes, int, void*) {
    std::memcpy(dst, src, bytes);
    return HDC_OK;
}
int hdc_stream_sync(void*) { return HDC_OK; }
int hdc_norms(hdc_context*, const void*, int, int64_t, int64_t*, int32_t*, void*) { return HDC_OK; }
int64_t hdc_num_windows(const hdc_context*, int64_t) { return 0; }
int hdc_encode_windows(hdc_context*, const char*, const int64_t*, const int64_t*, int64_t, int64_t, int16_t*, void*) {
    return HDC_OK;
}
size_t hdc_search_workspace_bytes(const hdc_context*, int64_t, int64_t, int) { return kFull; }
size_t hdc_search_workspace_min_bytes(const hdc_context*, int64_t, int64_t, int) { return kLeast; }
int hdc_search_plain(hdc_context*, const int16_t*, const int64_t*, int64_t nq, int32_t, const int16_t*, const int64_t*,
                     int64_t, int32_t, int k, int, float* score, int32_t* idx, double*, int64_t*, void* work,
                     size_t work_bytes, void*) {
    std::printf("work %zu\n", work ? work_bytes : 0);
    for (int64_t i = 0; i < nq * k; ++i) {
        score[i] = 0.5f;
        idx[i] = (int32_t)(i % k);
    }
    return HDC_OK;
}
int hdc_context_status(hdc_context*, int* status) {
    *status = word;
    return HDC_OK;
}
}

int main(int argc, char** argv) {
    if (argc != 3) return 2;
    limit_bytes = std::strtoull(argv[1], nullptr, 10);
    word = std::atoi(argv[2]);
    HV_16 a(HV_DIM, 1), b(HV_DIM, 2);
    std::vector<HV_16*> db = {&a, &b};
    try {
        auto r = cosine_search({&b}, db, 1);
        std::printf("found %d\n", (int)(r.at(&b).at(0).second == &a));
    } catch (const std::exception& e) {
        std::printf("threw %s\n", e.what());
    }
    return 0;
}
