// A scene is compiled while another thread captures a stream of its own: the
// compile succeeds, waits for nothing that the capture is part of, and the
// capture comes to its end.
#include <cuda_runtime_api.h>

#include <cstdio>
#include <thread>
#include <vector>

#include "fake_cudart.h"
#include "tpdsplat.h"

#define CHECK(x)                                                        \
    do {                                                                \
        if (!(x)) return std::printf("line %d: %s\n", __LINE__, #x), 1; \
    } while (0)

int main() {
    tpd_settings s;
    tpd_settings_init(&s);
    tpd_engine* e = nullptr;
    CHECK(tpd_create(&s, &e) == TPD_OK);
    const unsigned n = 1000;
    std::vector<float> records(n * 60, 0.5f), p(n * 59, 0.5f);
    float view[16] = {1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 1};
    cudaStream_t other;
    cudaStreamCreateWithFlags(&other, cudaStreamNonBlocking);
    for (int again = 0; again < 2; ++again) {  // new buffers, then kept ones
        for (int params = 0; params < 2; ++params) {
            cudaGraph_t graph = nullptr;
            std::thread([&] { cudaStreamBeginCapture(other, cudaStreamCaptureModeThreadLocal); }).join();
            const int rc = params ? tpd_compile_params_device(e, &p[0], &p[n * 3], &p[n * 6], &p[n * 10], &p[n * 11], n)
                                  : tpd_compile(e, records.data(), n, nullptr, 1);
            cudaError_t end = cudaErrorUnknown;
            std::thread([&] { end = cudaStreamEndCapture(other, &graph); }).join();
            CHECK(rc == TPD_OK);
            CHECK(end == cudaSuccess && graph);
            CHECK(fake::device_syncs == 0);
            cudaGraphDestroy(graph);
            CHECK(tpd_set_camera(e, view, view, 320, 200) == TPD_OK);
            CHECK(tpd_raster_frame(e, nullptr) == TPD_OK);
        }
    }
    cudaStreamDestroy(other);
    tpd_destroy(e);
    CHECK(fake::sizes().empty());
    std::puts("ok");
    return 0;
}
