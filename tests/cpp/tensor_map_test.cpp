// get_encode_fn from several threads at once, against a lookup that takes its time: every one of them gets the function.
#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstring>
#include <thread>
#include <vector>

#include "tensor_map.h"

static std::atomic<int> lookups{0};
static int marker;

extern "C" cudaError_t CUDARTAPI cudaGetDriverEntryPoint(const char* symbol, void** fn, unsigned long long,
                                                         cudaDriverEntryPointQueryResult* res) {
    lookups++;
    std::this_thread::sleep_for(std::chrono::milliseconds(100));
    *fn = std::strcmp(symbol, "cuTensorMapEncodeTiled") == 0 ? &marker : nullptr;
    *res = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
extern "C" cudaError_t CUDARTAPI cudaGetLastError() { return cudaSuccess; }

int main() {
    std::atomic<int> good{0};
    std::vector<std::thread> threads;
    for (int i = 0; i < 8; i++)
        threads.emplace_back([&] { good += reinterpret_cast<void*>(b200f::get_encode_fn()) == &marker ? 1 : 0; });
    for (auto& t : threads) t.join();
    std::printf("%d of 8 threads, %d lookups\n", good.load(), lookups.load());
    return good == 8 && lookups == 1 ? 0 : 1;
}
