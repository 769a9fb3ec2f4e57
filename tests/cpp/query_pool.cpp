// Host checks of the ray-query workers (albedo_b200/csrc/query_pool.cpp) against a
// stand-in for the CUDA runtime: device memory is host memory, work on the
// workers' streams runs when it is enqueued, work on the default stream when
// something waits for it.
//
// Arguments: the name of a check. Prints what it finds.
#include "../../albedo_b200/csrc/query_pool.hpp"

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <mutex>
#include <string>
#include <vector>

namespace fake {

std::mutex mutex;
// Work queued on the default stream.
std::vector<std::function<void()>> default_stream;

} // namespace fake

extern "C" {

cudaError_t cudaGetDevice(int* device)
{
    *device = 0;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaGetLastError() { return cudaSuccess; }

cudaError_t cudaMalloc(void** p, size_t bytes)
{
    *p = std::malloc(bytes);
    return cudaSuccess;
}
cudaError_t cudaFree(void* p)
{
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t bytes) { return cudaMalloc(p, bytes); }
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* stream, unsigned int)
{
    *stream = reinterpret_cast<cudaStream_t>(std::malloc(1));
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t stream)
{
    std::free(stream);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t stream)
{
    if (stream == nullptr || stream == cudaStreamLegacy) {
        const std::lock_guard lock{fake::mutex};
        for (const auto& work : fake::default_stream) {
            work();
        }
        fake::default_stream.clear();
    }
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* to, const void* from, size_t bytes, cudaMemcpyKind, cudaStream_t)
{
    std::memcpy(to, from, bytes);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* to, int value, size_t bytes, cudaStream_t)
{
    std::memset(to, value, bytes);
    return cudaSuccess;
}

} // extern "C"

namespace {

using namespace albedo_b200;

// A stand-in for a query: 2 v + 1 of each 4-byte input, nothing for negative ones.
cudaError_t twicePlusOne(void* const* in, void* const* out, int count, cudaStream_t)
{
    for (int i = 0; i < count; ++i) {
        const int v = static_cast<const int*>(in[0])[i];
        if (v >= 0) {
            static_cast<int*>(out[0])[i] = 2 * v + 1;
        }
    }
    return cudaSuccess;
}

std::vector<int> numbers(std::size_t count)
{
    std::vector<int> v(count);
    for (std::size_t i = 0; i < count; ++i) {
        v[i] = i % 7 == 3 ? -1 : static_cast<int>(i);
    }
    return v;
}

std::size_t wrongAnswers(const std::vector<int>& in, const int* out)
{
    std::size_t wrong = 0;
    for (std::size_t i = 0; i < in.size(); ++i) {
        wrong += out[i] != (in[i] < 0 ? 0 : 2 * in[i] + 1) ? 1 : 0;
    }
    return wrong;
}

void run(const std::vector<int>& in, std::vector<int>& out)
{
    const QueryInput inputs[]{{in.data(), sizeof(int)}};
    const QueryOutput outputs[]{{out.data(), sizeof(int)}};
    runQueries(static_cast<std::int64_t>(in.size()), inputs, outputs, twicePlusOne);
}

// Inputs that work on the default stream is still to fill when the call is made.
void order()
{
    for (const std::size_t count : {std::size_t{1}, std::size_t{1000}, std::size_t{300'007}}) {
        const std::vector<int> wanted = numbers(count);
        std::vector<int> in(count, 5);
        std::vector<int> out(count, 5);
        fake::default_stream.push_back([&] { in = wanted; });
        run(in, out);
        std::printf("order count=%zu wrong=%zu\n", count, wrongAnswers(wanted, out.data()));
    }
}

} // namespace

int main(int argc, char** argv)
{
    const std::map<std::string, void (*)()> checks{{"order", order}};
    const auto check = checks.find(argc > 1 ? argv[1] : "");
    if (check == checks.end()) {
        return 2;
    }
    retainQueryBuffers(0);
    check->second();
    releaseQueryBuffers(0);
    return 0;
}
