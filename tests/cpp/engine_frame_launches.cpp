// The kernels that a frame launches, for frames whose sorts and blends have different forms: a
// line "views n width height key_sort_lookback sort_ctas_per_sm launches" each.
#include <cstdio>
#include <vector>

#include "fake_cudart.h"
#include "tpdsplat.h"

int main() {
    std::vector<float> records(60 * 60000, 0.5f);
    const unsigned sizes[][2] = {{201, 151}, {256, 256}, {801, 603}, {1280, 720}, {1920, 1080}, {4112, 64}};
    for (const unsigned lookback : {0u, 1u})
        for (const unsigned ctas : {0u, 2u})
            for (const unsigned views : {1u, 2u, 9u})
                for (const unsigned n : {1000u, 6200u, 60000u})
                    for (const auto& size : sizes) {
                        tpd_settings s;
                        tpd_settings_init(&s);
                        s.use_graph = 0;
                        s.key_sort_lookback = lookback;
                        s.sort_ctas_per_sm = ctas;
                        tpd_engine* e = nullptr;
                        std::vector<tpd_view> v(views);
                        for (auto& x : v) {
                            x = tpd_view{};
                            x.width = size[0];
                            x.height = size[1];
                        }
                        if (tpd_create(&s, &e) != TPD_OK || tpd_compile(e, records.data(), n, nullptr, 1) != TPD_OK ||
                            tpd_set_views(e, v.data(), views) != TPD_OK)
                            return std::puts("set-up failed"), 1;
                        const long before = fake::launches;
                        if (tpd_raster_frame(e, nullptr) != TPD_OK) return std::puts("frame failed"), 1;
                        std::printf("%u %u %u %u %u %u %ld\n", views, n, size[0], size[1], lookback, ctas,
                                    fake::launches - before);
                        tpd_destroy(e);
                    }
    std::puts("ok");
    return 0;
}
