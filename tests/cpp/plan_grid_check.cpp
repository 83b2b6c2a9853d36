// The bound on the items of a device-built field grid does not wrap around 2^32 (element counts as plan_grid
// sees them, not elements): larger fields are built on the host.
#include <cstdio>
#include <string>
#include <vector>

#include "csp_scene.h"

using namespace csp;

int main() {
    // twenty flat mirrors in a row and a receiver
    std::vector<csp_element> el(21);
    for (size_t i = 0; i < el.size(); ++i) {
        csp_element e{};
        e.origin[0] = 15.0 * (double)i;
        e.aim_point[0] = e.origin[0];
        e.aim_point[2] = 1.0;
        e.aperture = CSP_APERTURE_RECTANGLE;
        e.surface = CSP_SURFACE_FLAT;
        e.width = e.height = 10.0;
        e.reflectivity = 1.0;
        el[i] = e;
    }
    HostScene s;
    std::string err;
    GridStats stats;
    if (build_elements(el.data(), (uint32_t)el.size(), s, err, &stats) != CSP_OK) return 2;
    HostGrid g;
    plan_grid(s, stats, g);
    bool ok = g.valid && g.on_device && field_items(s, g) <= g.cap_items && field_items(s, g) >= 20;
    // many small boxes and some of the largest ratio that the device takes: up to 6 x 6 cells a box
    stats.max = 10.0f;
    stats.min = 1.0f;
    for (const uint32_t n : {100000000u, 119304647u, 119304648u, 200000000u}) {
        stats.n = n;
        stats.sum = (double)n * (10.0 / (1.4 * 4.0));
        plan_grid(s, stats, g);
        const bool fits = n <= 119304647u;  // 36 n < 2^32
        ok = ok && g.valid && g.on_device == fits && (!fits || g.cap_items == 36u * n);
        std::printf("%u %d %u\n", n, (int)g.on_device, g.cap_items);
    }
    std::puts(ok ? "OK" : "FAIL");
    return ok ? 0 : 1;
}
