// A shadow flux where the process can make no thread (linked with the library's objects and the fake CUDA
// runtime). Exits 0 if the call comes back with success.
#include <cerrno>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <pthread.h>
#include <vector>

#include "dsmc_cuda.h"

extern "C" int pthread_create(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *) noexcept {
    return EAGAIN;
}

int main() {
    const int side = 60;   // a wavy sheet of 2 x 60 x 60 triangles
    std::vector<double> spot, normal;
    std::vector<int32_t> facet;
    for (int i = 0; i <= side; i++)
        for (int j = 0; j <= side; j++) spot.insert(spot.end(), {1.0 * i, 1.0 * j, std::sin(0.3 * i) * std::cos(0.2 * j)});
    for (int i = 0; i < side; i++)
        for (int j = 0; j < side; j++) {
            const int32_t a = i * (side + 1) + j, b = a + side + 1;
            facet.insert(facet.end(), {a, b, a + 1, a + 1, b, b + 1});
            normal.insert(normal.end(), {0.0, 0.0, 1.0, 0.0, 0.0, 1.0});
        }
    const int nface = 2 * side * side;
    std::vector<double> F(nface);
    dsmc_ctx *c = nullptr;
    if (dsmc_ctx_create(0, &c) != DSMC_OK) return 2;
    const int rc = dsmc_shadow_flux_host(c, (side + 1) * (side + 1), spot.data(), nface, facet.data(), normal.data(),
                                         0.1, 1, 1, F.data());
    if (rc != DSMC_OK) std::fprintf(stderr, "%s\n", dsmc_last_error(c));
    dsmc_ctx_destroy(c);
    return rc == DSMC_OK ? 0 : 1;
}
