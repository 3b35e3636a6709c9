// Host check of the launch wrapper (sparse-eigs-mex_b200/csrc/launch.h) against
// a stand-in for the runtime's launch call: what the call refuses is returned
// to the caller, kept -- the first one -- until it is asked for, and kept per
// host thread; a failed synchronisation comes before it.
#include "launch.h"

#include <cstdio>
#include <thread>

namespace spx {
Counters &counters() {
    static Counters c;
    return c;
}
}  // namespace spx

static cudaError_t answer = cudaSuccess;
static int chained = 0;
extern "C" cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *cfg, const void *, void **) {
    chained = (int)cfg->numAttrs;
    return answer;
}

static void kernel(int, const double *) {}

#define CHECK(x) if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; }

int main() {
    const double *p = nullptr;
    CHECK(spx::launch_chained(kernel, 1, 32, 0, nullptr, 1, p) == cudaSuccess && chained == 1);
    CHECK(spx::launch_plain(kernel, 1, 32, 0, nullptr, 1, p) == cudaSuccess && chained == 0);
    CHECK(spx::launch_result(cudaSuccess) == cudaSuccess);
    answer = cudaErrorInvalidValue;
    CHECK(spx::launch_chained(kernel, 1, 32, 1 << 20, nullptr, 1, p) == cudaErrorInvalidValue);
    answer = cudaErrorInvalidConfiguration;
    CHECK(spx::launch_plain(kernel, 1, 32, 1 << 20, nullptr, 1, p) == cudaErrorInvalidConfiguration);
    answer = cudaSuccess;
    CHECK(spx::launch_chained(kernel, 1, 32, 0, nullptr, 1, p) == cudaSuccess);
    cudaError_t other = cudaErrorUnknown;
    std::thread([&] { other = spx::launch_result(cudaSuccess); }).join();
    CHECK(other == cudaSuccess);
    CHECK(spx::launch_result(cudaSuccess) == cudaErrorInvalidValue);
    CHECK(spx::launch_result(cudaSuccess) == cudaSuccess);
    answer = cudaErrorInvalidValue;
    spx::launch_chained(kernel, 1, 32, 0, nullptr, 1, p);
    CHECK(spx::launch_result(cudaErrorLaunchFailure) == cudaErrorLaunchFailure);
    CHECK(spx::launch_result(cudaSuccess) == cudaSuccess);
    CHECK(spx::counters().launches == 6);
    puts("ok");
    return 0;
}
