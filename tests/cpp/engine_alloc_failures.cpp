// Every allocation of a session fails once, in turn. A call that reports the
// failure is made again; afterwards the engine must hold what an engine holds
// whose allocations all succeeded: no buffer may be missing behind a size that
// says it is there.
#include <algorithm>
#include <cstdio>
#include <functional>
#include <iterator>
#include <vector>

#include "fake_cudart.h"
#include "tpdsplat.h"

namespace {

std::vector<float> records(5000 * 60, 0.5f), params(5000 * 59, 0.5f);
std::vector<unsigned> entity(5000, 1u);
std::vector<float> image(3840u * 2160u * 4u), gradient(1024u * 608u * 3u);

tpd_view view(unsigned w, unsigned h) {
    tpd_view v = {};
    for (int k = 0; k < 4; ++k) v.view[5 * k] = v.proj[5 * k] = 1.f;
    v.width = w;
    v.height = h;
    return v;
}

int look(tpd_engine* e, unsigned w, unsigned h, unsigned views = 1) {
    const tpd_view v[2] = {view(w, h), view(w, h)};
    return tpd_set_views(e, v, views);
}

int compile_params(tpd_engine* e, unsigned n) {
    const float* p = params.data();
    return tpd_compile_params_device(e, p, p + 3 * n, p + 6 * n, p + 10 * n, p + 11 * n, n);
}

// The buffers of small and large scenes, of one and several entities, of small
// images, of images blended by list length, of strips, of several views, of
// the backward, of pipelined renders and of read-back.
std::vector<std::function<int(tpd_engine*)>> session() {
    const float eye[16] = {1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 1};
    std::vector<float> m(eye, eye + 16);
    return {
        [](tpd_engine* e) { return tpd_compile(e, records.data(), 1000, nullptr, 1); },
        [](tpd_engine* e) { return look(e, 320, 200); },
        [](tpd_engine* e) { return tpd_raster_frame(e, nullptr); },
        [](tpd_engine* e) { return look(e, 800, 608); },
        [](tpd_engine* e) { return tpd_raster_frame(e, nullptr); },
        [](tpd_engine* e) { return tpd_render_async(e, image.data(), TPD_IMAGE_RGBA8, 0); },
        [](tpd_engine* e) { return tpd_wait_render(e, nullptr); },
        [](tpd_engine* e) { return tpd_compile(e, records.data(), 5000, entity.data(), 3); },
        [m](tpd_engine* e) { return tpd_set_transform(e, 1, m.data()); },
        [](tpd_engine* e) { return look(e, 1024, 608, 2); },
        [](tpd_engine* e) { return tpd_raster_frame(e, nullptr); },
        [](tpd_engine* e) { return tpd_render_async(e, image.data(), TPD_IMAGE_RGB32F, 0); },
        [](tpd_engine* e) { return tpd_wait_render(e, nullptr); },
        [](tpd_engine* e) { return tpd_read_buffer(e, TPD_BUF_KEYS, image.data(), 0, 8, 0); },
        [](tpd_engine* e) { return compile_params(e, 5000); },
        [](tpd_engine* e) { return look(e, 1024, 608); },
        [](tpd_engine* e) { return tpd_raster_frame(e, nullptr); },
        [](tpd_engine* e) {
            return tpd_backward(e, gradient.data(), nullptr, nullptr, nullptr, nullptr, nullptr);
        },
        [](tpd_engine* e) { return look(e, 3840, 2160); },
        [](tpd_engine* e) { return tpd_raster_frame(e, nullptr); },
        [](tpd_engine* e) { return tpd_read_image(e, image.data(), TPD_IMAGE_RGBA8, 0); },
        [](tpd_engine* e) { return compile_params(e, 1000); },
        [](tpd_engine* e) { return tpd_raster_frame(e, nullptr); },
    };
}

}  // namespace

int main() {
    std::vector<std::multiset<size_t>> whole;  // the buffers after each call of the session without failures
    const auto steps = session();
    for (long k = -1;; ++k) {
        fake::fail_at = k;
        fake::failed = 0;
        tpd_settings s;
        tpd_settings_init(&s);
        tpd_engine* e = nullptr;
        bool reported = false;
        if (tpd_create(&s, &e) != TPD_OK) {
            reported = true;
            if (tpd_create(&s, &e) != TPD_OK) return std::printf("allocation %ld: create\n", k), 1;
        }
        for (size_t i = 0; i < steps.size(); ++i) {
            int rc = steps[i](e);
            if (rc != TPD_OK) {
                if (fake::failed == 0) return std::printf("step %zu: status %d without a failure\n", i, rc), 1;
                reported = true;
                rc = steps[i](e);
            }
            if (rc != TPD_OK)
                return std::printf("allocation %ld: step %zu: status %d (%s)\n", k, i, rc, tpd_last_error(e)), 1;
            const std::multiset<size_t> have = fake::sizes();
            if (k < 0) {
                whole.push_back(have);
            } else if (reported && have != whole[i]) {
                std::multiset<size_t> lack;
                std::set_difference(whole[i].begin(), whole[i].end(), have.begin(), have.end(),
                                    std::inserter(lack, lack.end()));
                std::printf("allocation %ld: step %zu: %zu buffers of %zu, lacking", k, i, have.size(), whole[i].size());
                for (size_t b : lack) std::printf(" %zu", b);
                return std::puts(" bytes"), 1;
            }
        }
        tpd_destroy(e);
        if (!fake::sizes().empty()) return std::printf("allocation %ld: buffers left behind\n", k), 1;
        if (k >= 0 && fake::failed == 0) break;  // past the last allocation
    }
    std::puts("ok");
    return 0;
}
