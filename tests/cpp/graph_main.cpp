// Counts the CUDA graphs a program launches per als_iterate call.  Linked from the library's
// objects with --wrap=cudaGraphLaunch.  argv: precision solve use_graph, then the calls' epoch counts; prints
// the launches of each call on a line of its own, then whether the factors equal those of the same
// epochs on a handle without graphs.
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "als_gb300.h"

static int launches = 0;
extern "C" int __real_cudaGraphLaunch(void *exec, void *stream);
extern "C" int __wrap_cudaGraphLaunch(void *exec, void *stream) {
    ++launches;
    return __real_cudaGraphLaunch(exec, stream);
}

#define CHECK(x)                                                                  \
    do {                                                                          \
        if ((x) != ALS_OK) {                                                      \
            std::fprintf(stderr, "%s: %s\n", #x, als_last_error(nullptr));        \
            return 1;                                                             \
        }                                                                         \
    } while (0)

int main(int argc, char **argv) {
    if (argc < 5) return 2;
    const int m = 300, n = 200, per = 20;
    std::vector<int32_t> ptr(m + 1), idx;
    std::vector<float> val;
    for (int u = 0; u < m; ++u) {
        ptr[u + 1] = ptr[u] + per;
        for (int k = 0; k < per; ++k) {
            idx.push_back(k * 10 + (u * 7 + k) % 10);
            val.push_back(1.f + (float)((u + 3 * k) % 5));
        }
    }
    const als_csr_view csr = {m, n, (int64_t)idx.size(), ptr.data(), idx.data(), val.data()};
    als_config cfg;
    als_config_default(&cfg);
    cfg.f = 24;
    cfg.precision = std::atoi(argv[1]);
    cfg.solve_type = std::atoi(argv[2]);
    std::vector<float> U[2], V[2];
    for (int run = 0; run < 2; ++run) {
        cfg.use_graph = run == 0 ? std::atoi(argv[3]) : 0;
        als_handle *h = nullptr;
        CHECK(als_create(&cfg, &csr, nullptr, nullptr, &h));
        CHECK(als_init_factors(h));
        for (int k = 4; k < argc; ++k) {
            launches = 0;
            CHECK(als_iterate(h, std::atoi(argv[k])));
            double ms[4];
            CHECK(als_get_stage_ms(h, ms));
            if (run == 0) std::printf("%d %d\n", launches, ms[0] > 0.0 && ms[1] > 0.0 ? 1 : 0);
        }
        U[run].resize((size_t)m * cfg.f);
        V[run].resize((size_t)n * cfg.f);
        CHECK(als_get_factors(h, U[run].data(), V[run].data()));
        CHECK(als_destroy(h));
    }
    std::printf("%s\n", std::memcmp(U[0].data(), U[1].data(), U[0].size() * sizeof(float)) == 0 &&
                                std::memcmp(V[0].data(), V[1].data(), V[0].size() * sizeof(float)) == 0
                            ? "equal" : "differ");
    return 0;
}
