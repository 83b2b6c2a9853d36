// rsqrt_near_1 against 1.0f / sqrtf for every float it is used for, and normalize_unit against
// normalize at and beyond the edges of that range (infinities, NaN and zero among them).
#include <cmath>
#include <cstdio>
#include <cstring>
#include <utility>

#include "csp_math.cuh"

int main() {
    long bad = 0;
    for (int k = -2048; k < 2048; ++k) {
        const float x = csp::u2f((uint32_t)(0x3f800000 + k));
        if (csp::f2u(csp::rsqrt_near_1(x)) != csp::f2u(1.0f / std::sqrt(x))) ++bad;
    }
    // vectors of every squared length around the range, and of any other
    for (int k = -6000; k < 6000; ++k) {
        const float s = std::sqrt(csp::u2f((uint32_t)(0x3f800000 + k)));
        const float3 a = csp::f3(s, 0.f, 0.f), b = csp::f3(0.6f * s, 0.f, 0.8f * s);
        for (float3 v : {a, b}) {
            const float3 p = csp::normalize_unit(v), q = csp::normalize(v);
            if (std::memcmp(&p, &q, sizeof p)) ++bad;
        }
    }
    for (float s : {0.f, 1e-30f, 1e-3f, 0.5f, 2.f, 1e10f, 3e38f, INFINITY, -INFINITY, NAN}) {
        const float3 p = csp::normalize_unit(csp::f3(s, s, 1e-3f * s)), q = csp::normalize(csp::f3(s, s, 1e-3f * s));
        for (auto pq : {std::make_pair(p.x, q.x), std::make_pair(p.y, q.y), std::make_pair(p.z, q.z)})
            if (!(pq.first == pq.second || (std::isnan(pq.first) && std::isnan(pq.second)))) ++bad;
    }
    std::printf("%ld mismatches\n", bad);
    return bad ? 1 : 0;
}
