// Host checks of the ray-query workers (albedo_b200/csrc/query_pool.cpp) against a
// stand-in for the CUDA runtime: device memory is host memory, work on the
// workers' streams runs when it is enqueued, work on the default stream when
// something waits for it. Allocations and streams belong to the context that is
// current in the thread that makes them, and device memory may be short.
//
// Arguments: the name of a check. Prints what it finds.
#include "../../albedo_b200/csrc/query_pool.hpp"

#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <limits>
#include <map>
#include <mutex>
#include <new>
#include <stdexcept>
#include <string>
#include <vector>

namespace fake {

std::mutex mutex;
// Work queued on the default stream.
std::vector<std::function<void()>> default_stream;

// Contexts 1 (the device's primary one, always active) and up; 0: none.
thread_local std::uintptr_t current{0};
std::atomic<int> used_elsewhere{0}; // pointers and streams used in another context than their own

std::uintptr_t useCurrent()
{
    if (current == 0) {
        current = 1;
    }
    return current;
}

// What is allocated, by address: its context, kind and size.
struct Made {
    std::uintptr_t context;
    std::string kind;
    std::size_t bytes;
};
std::map<const void*, Made> made;
std::size_t device_limit{std::numeric_limits<std::size_t>::max()};
thread_local cudaError_t last_error{cudaSuccess};

void* make(const char* kind, std::size_t bytes)
{
    void* p = std::malloc(bytes);
    const std::lock_guard lock{mutex};
    made[p] = {useCurrent(), kind, bytes};
    return p;
}
cudaError_t unmake(const char* kind, void* p)
{
    if (p == nullptr) {
        static_cast<void>(useCurrent());
        return cudaSuccess;
    }
    const std::lock_guard lock{mutex};
    const auto found = made.find(p);
    if (found == made.end() || found->second.kind != kind) {
        std::abort();
    }
    made.erase(found);
    std::free(p);
    return cudaSuccess;
}
// Counts a use of `p`, or of the allocation `p` points into, in another context.
void use(const void* p)
{
    const std::lock_guard lock{mutex};
    auto found = made.upper_bound(p);
    if (found == made.begin() || (--found)->second.context != useCurrent()) {
        ++used_elsewhere;
    }
}
// Copies and clears on each stream since something last waited for it.
std::map<cudaStream_t, int> pending;

void enqueue(cudaStream_t stream)
{
    use(stream);
    const std::lock_guard lock{mutex};
    ++pending[stream];
}
int inFlight()
{
    const std::lock_guard lock{mutex};
    int n = 0;
    for (const auto& [stream, count] : pending) {
        n += count;
    }
    return n;
}
std::size_t alive()
{
    const std::lock_guard lock{mutex};
    return made.size();
}

CUresult ctxGetCurrent(CUcontext* context)
{
    *context = reinterpret_cast<CUcontext>(current);
    return CUDA_SUCCESS;
}
CUresult ctxSetCurrent(CUcontext context)
{
    current = reinterpret_cast<std::uintptr_t>(context);
    return CUDA_SUCCESS;
}
CUresult ctxGetId(CUcontext context, unsigned long long* id)
{
    *id = 100 + reinterpret_cast<std::uintptr_t>(context);
    return CUDA_SUCCESS;
}
CUresult ctxGetDevice(CUdevice* device)
{
    *device = 0;
    return CUDA_SUCCESS;
}
CUresult primaryState(CUdevice, unsigned int*, int* active)
{
    *active = 1;
    return CUDA_SUCCESS;
}
CUresult primaryRetain(CUcontext* context, CUdevice)
{
    *context = reinterpret_cast<CUcontext>(1);
    return CUDA_SUCCESS;
}
CUresult primaryRelease(CUdevice) { return CUDA_SUCCESS; }

} // namespace fake

extern "C" {

cudaError_t cudaGetDriverEntryPointByVersion(const char* name, void** function, unsigned int, unsigned long long,
                                             cudaDriverEntryPointQueryResult* found)
{
    const std::map<std::string, void*> functions{
        {"cuCtxGetCurrent", reinterpret_cast<void*>(fake::ctxGetCurrent)},
        {"cuCtxSetCurrent", reinterpret_cast<void*>(fake::ctxSetCurrent)},
        {"cuCtxGetId", reinterpret_cast<void*>(fake::ctxGetId)},
        {"cuCtxGetDevice", reinterpret_cast<void*>(fake::ctxGetDevice)},
        {"cuDevicePrimaryCtxGetState", reinterpret_cast<void*>(fake::primaryState)},
        {"cuDevicePrimaryCtxRetain", reinterpret_cast<void*>(fake::primaryRetain)},
        {"cuDevicePrimaryCtxRelease", reinterpret_cast<void*>(fake::primaryRelease)}};
    const auto at = functions.find(name);
    *function = at == functions.end() ? nullptr : at->second;
    *found = *function == nullptr ? cudaDriverEntryPointSymbolNotFound : cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* device)
{
    *device = 0;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int)
{
    fake::current = 1;
    return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaGetLastError()
{
    const cudaError_t e = fake::last_error;
    fake::last_error = cudaSuccess;
    return e;
}

cudaError_t cudaMalloc(void** p, size_t bytes)
{
    std::size_t used = 0;
    {
        const std::lock_guard lock{fake::mutex};
        for (const auto& [at, m] : fake::made) {
            used += m.kind == "device" ? m.bytes : 0;
        }
    }
    if (bytes > fake::device_limit || used > fake::device_limit - bytes) {
        fake::last_error = cudaErrorMemoryAllocation;
        return cudaErrorMemoryAllocation;
    }
    *p = fake::make("device", bytes);
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) { return fake::unmake("device", p); }
cudaError_t cudaMallocHost(void** p, size_t bytes)
{
    *p = fake::make("pinned", bytes);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { return fake::unmake("pinned", p); }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* stream, unsigned int)
{
    *stream = reinterpret_cast<cudaStream_t>(fake::make("stream", 1));
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t stream) { return fake::unmake("stream", stream); }
cudaError_t cudaStreamSynchronize(cudaStream_t stream)
{
    if (stream == nullptr || stream == cudaStreamLegacy) {
        const std::lock_guard lock{fake::mutex};
        for (const auto& work : fake::default_stream) {
            work();
        }
        fake::default_stream.clear();
    } else {
        fake::use(stream);
        const std::lock_guard lock{fake::mutex};
        fake::pending[stream] = 0;
    }
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* to, const void* from, size_t bytes, cudaMemcpyKind, cudaStream_t stream)
{
    fake::use(to);
    fake::use(from);
    fake::enqueue(stream);
    std::memcpy(to, from, bytes);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* to, int value, size_t bytes, cudaStream_t stream)
{
    fake::use(to);
    fake::enqueue(stream);
    std::memset(to, value, bytes);
    return cudaSuccess;
}

} // extern "C"

namespace {

using namespace albedo_b200;

// A stand-in for a query: 2 v + 1 of each 4-byte input, nothing for negative ones.
cudaError_t twicePlusOne(void* const* in, void* const* out, int count, cudaStream_t stream)
{
    fake::use(in[0]);
    fake::use(out[0]);
    fake::use(stream);
    for (int i = 0; i < count; ++i) {
        const int v = static_cast<const int*>(in[0])[i];
        if (v >= 0) {
            static_cast<int*>(out[0])[i] = 2 * v + 1;
        }
    }
    return cudaGetLastError(); // as a launch reports what went wrong before it
}

SlotPool* kept = nullptr; // of the scene that main() holds

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
    runQueries(kept, static_cast<std::int64_t>(in.size()), inputs, outputs, twicePlusOne);
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

// Calls in the primary context, in one of the program's own and in the primary
// one again: everything is used where it was made, the caller's context stays, and
// what is kept is kept in the primary one.
void context()
{
    for (const std::uintptr_t own : {1, 7, 1}) {
        fake::current = own;
        SlotPool* const before = kept;
        kept = retainQueryBuffers();
        const std::vector<int> in = numbers(300'007);
        std::vector<int> out(in.size(), 5);
        run(in, out);
        releaseQueryBuffers(kept);
        kept = before;
        std::printf("context own=%d after=%d wrong=%zu elsewhere=%d kept_elsewhere=%d\n", static_cast<int>(own),
                    static_cast<int>(fake::current), wrongAnswers(in, out.data()), fake::used_elsewhere.load(),
                    [] {
                        int n = 0;
                        for (const auto& [p, m] : fake::made) {
                            n += m.context != 1 ? 1 : 0;
                        }
                        return n;
                    }());
    }
}

// With the last scene gone nothing is left; a scene of the program's own context
// has no share.
void scenes()
{
    const std::vector<int> in = numbers(300'007);
    std::vector<int> out(in.size(), 5);
    run(in, out);
    releaseQueryBuffers(retainQueryBuffers());
    const bool still = fake::alive() > 0;
    fake::current = 7;
    std::printf("scenes kept=%d own_share=%d\n", still ? 1 : 0, retainQueryBuffers() != nullptr ? 1 : 0);
}

// Device memory for nothing, for a small slot, for one slot and for three of those
// a call would use, and without a limit; ten calls each.
void memory()
{
    const std::vector<int> in = numbers(300'007);
    for (const std::size_t limit : {std::size_t{0}, std::size_t{100'000}, std::size_t{3'000'000},
                                    std::size_t{9'000'000}, std::numeric_limits<std::size_t>::max()}) {
        fake::device_limit = limit;
        for (int k = 0; k < 10; ++k) {
            std::vector<int> out(in.size(), 5);
            bool refused = false;
            try {
                run(in, out);
            } catch (const std::bad_alloc&) {
                refused = true;
            }
            std::printf("memory limit=%zu refused=%d wrong=%zu error=%d\n", limit, refused ? 1 : 0,
                        refused ? std::size_t{0} : wrongAnswers(in, out.data()), static_cast<int>(cudaGetLastError()));
        }
    }
}

// Outputs over the inputs, in place and shifted either way, and two outputs over each other.
void overlap()
{
    for (const std::size_t count : {std::size_t{1}, std::size_t{20'000}, std::size_t{300'007}}) {
        const std::vector<int> in = numbers(count);
        for (const std::size_t before : {std::size_t{0}, std::size_t{1}, count / 2}) {
            for (const std::size_t behind : {std::size_t{0}, std::size_t{1}, count / 2}) {
                std::vector<int> both(count + before + behind);
                std::copy(in.begin(), in.end(), both.begin() + static_cast<std::ptrdiff_t>(before));
                int* const results = both.data() + behind;
                const QueryInput inputs[]{{both.data() + before, sizeof(int)}};
                const QueryOutput outputs[]{{results, sizeof(int)}};
                runQueries(kept, static_cast<std::int64_t>(count), inputs, outputs, twicePlusOne);
                std::printf("overlap count=%zu wrong=%zu\n", count, wrongAnswers(in, results));
            }
        }
        // The second output, 12 bytes a ray, ends up whole, the first where it reaches beyond it.
        std::vector<int> both(4 * count);
        const QueryInput inputs[]{{in.data(), sizeof(int)}};
        const QueryOutput outputs[]{{both.data() + 3 * count - count / 2, sizeof(int)}, {both.data(), 3 * sizeof(int)}};
        runQueries(kept, static_cast<std::int64_t>(count), inputs, outputs,
                   [](void* const* i, void* const* o, int n, cudaStream_t stream) {
                       for (int k = 0; k < 3 * n; ++k) {
                           static_cast<int*>(o[1])[k] = -7;
                       }
                       return twicePlusOne(i, o, n, stream);
                   });
        std::size_t wrong = 0;
        for (std::size_t k = 0; k < 3 * count; ++k) {
            wrong += both[k] != -7 ? 1 : 0;
        }
        for (std::size_t k = count / 2; k < count; ++k) {
            const int v = in[k];
            wrong += both[3 * count - count / 2 + k] != (v < 0 ? 0 : 2 * v + 1) ? 1 : 0;
        }
        std::printf("overlap count=%zu wrong=%zu\n", count, wrong);
    }
}

// Launches that fail, the first, a later one and all of them; then a call that does not.
void failure()
{
    const std::vector<int> in = numbers(300'007);
    for (const int bad : {0, 5, -1, 1000}) {
        std::vector<int> out(in.size(), 5);
        const QueryInput inputs[]{{in.data(), sizeof(int)}};
        const QueryOutput outputs[]{{out.data(), sizeof(int)}};
        std::atomic<int> launches{0};
        bool failed = false;
        try {
            runQueries(kept, static_cast<std::int64_t>(in.size()), inputs, outputs,
                       [&](void* const* i, void* const* o, int n, cudaStream_t stream) {
                           const int k = launches++;
                           return k == bad || bad < 0 ? cudaErrorLaunchFailure : twicePlusOne(i, o, n, stream);
                       });
        } catch (const std::runtime_error&) {
            failed = true;
        }
        std::printf("failure bad=%d failed=%d flight=%d wrong=%zu\n", bad, failed ? 1 : 0, fake::inFlight(),
                    failed ? std::size_t{0} : wrongAnswers(in, out.data()));
    }
}

} // namespace

int main(int argc, char** argv)
{
    const std::map<std::string, void (*)()> checks{{"order", order}, {"context", context}, {"scenes", scenes},
                                                      {"memory", memory}, {"overlap", overlap}, {"failure", failure}};
    const auto check = checks.find(argc > 1 ? argv[1] : "");
    if (check == checks.end()) {
        return 2;
    }
    kept = retainQueryBuffers();
    check->second();
    releaseQueryBuffers(kept);
    std::printf("end left=%zu\n", fake::alive());
    return 0;
}
