// Worker buffers of host-array ray queries, and the chunk loop.
#include "query_pool.hpp"

#include <cuda.h>

#include <algorithm>
#include <array>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <exception>
#include <format>
#include <map>
#include <memory>
#include <mutex>
#include <new>
#include <stdexcept>
#include <thread>
#include <vector>

namespace albedo_b200 {

namespace {

// Rays of a chunk: a call is split into kMaxWorkers chunks, of no fewer rays
// than make a full wave of threads worth launching and no more than a worker's
// buffers hold (2.8 MB pinned and as much device memory, 22 MB of each per
// device at most).
constexpr std::int64_t kMinChunk{16384};
constexpr std::int64_t kMaxChunk{32768};
constexpr std::size_t kMaxWorkers{8};
constexpr std::size_t kArrayAlign{256};
// Rays of the slot that serves a call where memory is short (90 KB of each).
constexpr std::int64_t kFewRays{1024};

void cudaCheck(cudaError_t e, const char* what)
{
    if (e == cudaErrorMemoryAllocation) {
        throw std::bad_alloc{};
    }
    if (e != cudaSuccess) {
        throw std::runtime_error{std::format("{}: {}", what, cudaGetErrorString(e))};
    }
}

// The driver's context functions. The library links the runtime alone, which
// hands out the driver's entry points.
template <typename Function>
Function driverFunction(const char* name)
{
    void* function{nullptr};
    cudaDriverEntryPointQueryResult found{};
    cudaCheck(cudaGetDriverEntryPointByVersion(name, &function, 12000, cudaEnableDefault, &found), name);
    if (found != cudaDriverEntryPointSuccess || function == nullptr) {
        throw std::runtime_error{std::format("{} is not in the driver", name)};
    }
    return reinterpret_cast<Function>(function);
}

struct Driver {
    decltype(&cuCtxGetCurrent) current{driverFunction<decltype(&cuCtxGetCurrent)>("cuCtxGetCurrent")};
    decltype(&cuCtxSetCurrent) makeCurrent{driverFunction<decltype(&cuCtxSetCurrent)>("cuCtxSetCurrent")};
    decltype(&cuCtxGetId) id{driverFunction<decltype(&cuCtxGetId)>("cuCtxGetId")};
    decltype(&cuCtxGetDevice) device{driverFunction<decltype(&cuCtxGetDevice)>("cuCtxGetDevice")};
    decltype(&cuDevicePrimaryCtxGetState) primaryState{
        driverFunction<decltype(&cuDevicePrimaryCtxGetState)>("cuDevicePrimaryCtxGetState")};
    decltype(&cuDevicePrimaryCtxRetain) retainPrimary{
        driverFunction<decltype(&cuDevicePrimaryCtxRetain)>("cuDevicePrimaryCtxRetain")};
    decltype(&cuDevicePrimaryCtxRelease) releasePrimary{
        driverFunction<decltype(&cuDevicePrimaryCtxRelease)>("cuDevicePrimaryCtxRelease")};
};

const Driver& driver()
{
    static const Driver functions;
    return functions;
}

void driverCheck(CUresult e, const char* what)
{
    if (e != CUDA_SUCCESS) {
        throw std::runtime_error{std::format("{}: driver error {}", what, static_cast<int>(e))};
    }
}

// The context that is current in the calling thread: a scene's tables are there,
// and so are a call's streams and buffers. It need not be its device's primary
// one, which is what the runtime makes current in a thread that has none.
CUcontext currentContext()
{
    CUcontext context{nullptr};
    driverCheck(driver().current(&context), "current context");
    if (context == nullptr) {
        cudaCheck(cudaFree(nullptr), "current context");
        driverCheck(driver().current(&context), "current context");
    }
    return context;
}

bool isPrimary(CUcontext context)
{
    CUdevice device{};
    unsigned int flags{0};
    int active{0};
    driverCheck(driver().device(&device), "context device");
    driverCheck(driver().primaryState(device, &flags, &active), "primary context");
    if (active == 0) {
        return false;
    }
    CUcontext primary{nullptr};
    driverCheck(driver().retainPrimary(&primary, device), "primary context");
    driverCheck(driver().releasePrimary(device), "primary context");
    return primary == context;
}

// One worker's stream, pinned buffer and device buffer, for `rays` rays.
struct Slot {
    cudaStream_t stream{nullptr};
    char* pinned{nullptr};
    char* device{nullptr};
    std::int64_t rays{0};

    Slot() = default;
    Slot(const Slot&) = delete;
    Slot& operator=(const Slot&) = delete;
    // Throws std::bad_alloc where there is no memory for it; the thread's CUDA
    // error state is then clear again.
    void allocate(std::int64_t count)
    {
        const std::size_t bytes{static_cast<std::size_t>(count) * kMaxQueryRayBytes +
                                2 * kMaxQueryArrays * kArrayAlign};
        const auto need = [](cudaError_t e, const char* what) {
            if (e == cudaErrorMemoryAllocation) {
                static_cast<void>(cudaGetLastError());
            }
            cudaCheck(e, what);
        };
        if (stream == nullptr) {
            need(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking), "query stream");
        }
        void* p{nullptr};
        if (pinned == nullptr) {
            need(cudaMallocHost(&p, bytes), "query staging");
            pinned = static_cast<char*>(p);
        }
        need(cudaMalloc(&p, bytes), "query buffers");
        device = static_cast<char*>(p);
        rays = count;
    }
    ~Slot()
    {
        if (device != nullptr) {
            cudaFree(device);
        }
        if (pinned != nullptr) {
            cudaFreeHost(pinned);
        }
        if (stream != nullptr) {
            cudaStreamDestroy(stream);
        }
    }
};

} // namespace

struct SlotPool {
    std::mutex mutex;
    std::condition_variable freed;
    std::vector<std::unique_ptr<Slot>> idle;
    std::size_t made{0};
    int scenes{0};

    // Slots are put back from destructors, which must not allocate.
    SlotPool() { idle.reserve(kMaxWorkers); }

    // A slot for the caller of a query: waits for one while all are in use, and
    // takes a small one where there is no memory for a whole one.
    std::unique_ptr<Slot> take()
    {
        {
            std::unique_lock lock{mutex};
            freed.wait(lock, [&] { return !idle.empty() || made < kMaxWorkers; });
            if (!idle.empty()) {
                return takeIdle();
            }
            ++made;
        }
        try {
            std::unique_ptr<Slot> slot{std::make_unique<Slot>()};
            try {
                slot->allocate(kMaxChunk);
            } catch (const std::bad_alloc&) {
                slot->allocate(kFewRays);
            }
            return slot;
        } catch (...) {
            drop();
            throw;
        }
    }
    // A slot for a helper thread, or none: where all are in use or there is no
    // memory for one, the other workers do its share.
    std::unique_ptr<Slot> tryTake()
    {
        {
            const std::lock_guard lock{mutex};
            if (!idle.empty()) {
                return takeIdle();
            }
            if (made == kMaxWorkers) {
                return nullptr;
            }
            ++made;
        }
        try {
            std::unique_ptr<Slot> slot{std::make_unique<Slot>()};
            slot->allocate(kMaxChunk);
            return slot;
        } catch (const std::bad_alloc&) {
            drop();
            return nullptr;
        } catch (...) {
            drop();
            throw;
        }
    }
    // Puts a slot back; a small one, and any with no scene left in the context, is
    // given up.
    void give(std::unique_ptr<Slot> slot)
    {
        {
            const std::lock_guard lock{mutex};
            if (scenes > 0 && slot->rays == kMaxChunk) {
                idle.push_back(std::move(slot));
                freed.notify_one();
                return;
            }
        }
        slot.reset();
        drop();
    }

private:
    std::unique_ptr<Slot> takeIdle()
    {
        std::unique_ptr<Slot> slot{std::move(idle.back())};
        idle.pop_back();
        return slot;
    }
    void drop()
    {
        const std::lock_guard lock{mutex};
        --made;
        freed.notify_one();
    }
};

namespace {

// The slots kept in a primary context, by the driver's id for it, which no other
// context of the process has, before or after.
SlotPool& keptSlots(std::uint64_t context)
{
    static std::mutex table_mutex;
    // Never destroyed: freeing device memory from a static destructor at exit
    // would run after the CUDA runtime has shut down.
    static auto* table{new std::map<std::uint64_t, std::unique_ptr<SlotPool>>};
    const std::lock_guard lock{table_mutex};
    std::unique_ptr<SlotPool>& entry{(*table)[context]};
    if (!entry) {
        entry = std::make_unique<SlotPool>();
    }
    return *entry;
}

// A slot held by a worker.
class HeldSlot {
public:
    HeldSlot(SlotPool& pool, std::unique_ptr<Slot> slot) : pool_{pool}, slot_{std::move(slot)} {}
    ~HeldSlot() { pool_.give(std::move(slot_)); }
    HeldSlot(const HeldSlot&) = delete;
    HeldSlot& operator=(const HeldSlot&) = delete;
    Slot& operator*() const { return *slot_; }

private:
    SlotPool& pool_;
    std::unique_ptr<Slot> slot_;
};

std::size_t aligned(std::size_t n) { return (n + kArrayAlign - 1) & ~(kArrayAlign - 1); }

// Queries [first, first + n) of the call through one slot: inputs lie at the
// slot's start, outputs behind them, each array on its own 256-byte boundary.
void runChunk(const Slot& slot, std::size_t first, std::size_t n, std::span<const QueryInput> inputs,
              std::span<const QueryOutput> outputs, const QueryLaunch& launch)
{
    std::array<void*, kMaxQueryArrays> device_in{};
    std::array<void*, kMaxQueryArrays> device_out{};
    std::size_t at{0};
    for (std::size_t i{0}; i < inputs.size(); ++i) {
        const std::size_t bytes{n * inputs[i].ray_bytes};
        std::memcpy(slot.pinned + at, static_cast<const char*>(inputs[i].host) + first * inputs[i].ray_bytes, bytes);
        device_in[i] = slot.device + at;
        at += aligned(bytes);
    }
    const std::size_t results{at};
    cudaCheck(cudaMemcpyAsync(slot.device, slot.pinned, results, cudaMemcpyHostToDevice, slot.stream), "upload");
    for (std::size_t i{0}; i < outputs.size(); ++i) {
        device_out[i] = slot.device + at;
        at += aligned(n * outputs[i].ray_bytes);
    }
    // What a query leaves unwritten (a miss) is zero.
    cudaCheck(cudaMemsetAsync(slot.device + results, 0, at - results, slot.stream), "query buffers");
    cudaCheck(launch(device_in.data(), device_out.data(), static_cast<int>(n), slot.stream), "query launch");
    cudaCheck(cudaMemcpyAsync(slot.pinned + results, slot.device + results, at - results, cudaMemcpyDeviceToHost,
                              slot.stream),
              "download");
    cudaCheck(cudaStreamSynchronize(slot.stream), "queries");
    at = results;
    for (const QueryOutput& out : outputs) {
        const std::size_t bytes{n * out.ray_bytes};
        if (out.host != nullptr) {
            std::memcpy(static_cast<char*>(out.host) + first * out.ray_bytes, slot.pinned + at, bytes);
        }
        at += aligned(bytes);
    }
}

// Whether an output of the call shares memory with another of its arrays.
bool arraysOverlap(std::size_t count, std::span<const QueryInput> inputs, std::span<const QueryOutput> outputs)
{
    const auto shared = [&](const QueryOutput& a, const void* host, std::size_t ray_bytes) {
        const auto at{reinterpret_cast<std::uintptr_t>(a.host)};
        const auto other{reinterpret_cast<std::uintptr_t>(host)};
        return a.host != nullptr && host != nullptr && at < other + count * ray_bytes &&
               other < at + count * a.ray_bytes;
    };
    for (std::size_t i{0}; i < outputs.size(); ++i) {
        for (const QueryInput& in : inputs) {
            if (shared(outputs[i], in.host, in.ray_bytes)) {
                return true;
            }
        }
        for (std::size_t k{i + 1}; k < outputs.size(); ++k) {
            if (shared(outputs[i], outputs[k].host, outputs[k].ray_bytes)) {
                return true;
            }
        }
    }
    return false;
}

// A call whose outputs lie over its inputs or each other reads every input before
// it writes a result and writes its outputs whole, one after the other; its chunks,
// which run beside each other, work on copies.
void runOnCopies(SlotPool* kept, std::int64_t count, std::span<const QueryInput> inputs,
                 std::span<const QueryOutput> outputs, const QueryLaunch& launch)
{
    const auto n{static_cast<std::size_t>(count)};
    std::vector<std::vector<char>> memory;
    std::vector<QueryInput> in{inputs.begin(), inputs.end()};
    for (QueryInput& i : in) {
        const char* const host{static_cast<const char*>(i.host)};
        i.host = memory.emplace_back(host, host + n * i.ray_bytes).data();
    }
    std::vector<QueryOutput> out{outputs.begin(), outputs.end()};
    for (QueryOutput& o : out) {
        if (o.host != nullptr) {
            o.host = memory.emplace_back(n * o.ray_bytes).data();
        }
    }
    runQueries(kept, count, in, out, launch);
    for (std::size_t i{0}; i < outputs.size(); ++i) {
        if (outputs[i].host != nullptr) {
            std::memcpy(outputs[i].host, out[i].host, n * outputs[i].ray_bytes);
        }
    }
}

} // namespace

void runQueries(SlotPool* kept, std::int64_t count, std::span<const QueryInput> inputs,
                std::span<const QueryOutput> outputs, const QueryLaunch& launch)
{
    if (count < 0) {
        throw std::bad_alloc{};
    }
    if (count == 0) {
        return;
    }
    std::size_t ray_bytes{0};
    for (const QueryInput& in : inputs) {
        ray_bytes += in.ray_bytes;
    }
    for (const QueryOutput& out : outputs) {
        ray_bytes += out.ray_bytes;
    }
    if (ray_bytes > kMaxQueryRayBytes || inputs.size() > kMaxQueryArrays || outputs.size() > kMaxQueryArrays) {
        throw std::logic_error{"a query takes more bytes a ray than a worker's buffers hold"};
    }
    // The caller's arrays may still be filled, or read, by work on the default
    // stream (and the streams that order themselves with it): pinned or managed
    // memory takes asynchronous copies and kernels. The workers read and write the
    // arrays on the host, so that work has to be over first (under 2 us where there
    // is none).
    cudaCheck(cudaStreamSynchronize(cudaStreamLegacy), "queries");
    if (arraysOverlap(static_cast<std::size_t>(count), inputs, outputs)) {
        return runOnCopies(kept, count, inputs, outputs, launch);
    }
    SlotPool calls_own;
    SlotPool& pool{kept != nullptr ? *kept : calls_own};
    const std::int64_t share{(count + static_cast<std::int64_t>(kMaxWorkers) - 1) /
                             static_cast<std::int64_t>(kMaxWorkers)};
    const std::int64_t chunk{std::clamp(share, kMinChunk, kMaxChunk)};
    const std::int64_t chunks{(count + chunk - 1) / chunk};
    std::atomic<std::int64_t> next{0};
    const auto work = [&](const Slot& slot) {
        for (std::int64_t c{next++}; c < chunks; c = next++) {
            const std::int64_t end{std::min((c + 1) * chunk, count)};
            for (std::int64_t first{c * chunk}; first < end; first += slot.rays) {
                const std::int64_t n{std::min(slot.rays, end - first)};
                try {
                    runChunk(slot, static_cast<std::size_t>(first), static_cast<std::size_t>(n), inputs, outputs,
                             launch);
                } catch (...) {
                    // What failed may have left copies in flight that use the buffers.
                    cudaStreamSynchronize(slot.stream);
                    throw;
                }
            }
        }
    };
    const std::size_t cores{std::max<std::size_t>(1, std::thread::hardware_concurrency())};
    const std::size_t workers{std::min({kMaxWorkers, cores, static_cast<std::size_t>(chunks)})};
    const CUcontext context{workers > 1 ? currentContext() : nullptr};
    std::vector<std::exception_ptr> failed(workers);
    const auto guarded = [&](std::size_t k, const auto& body) {
        try {
            body();
        } catch (...) {
            failed[k] = std::current_exception();
            next = chunks;
        }
    };
    // The caller has a slot before there are helpers, so the call waits for no
    // other slot and fails for want of memory only where nothing can run.
    const HeldSlot own{pool, pool.take()};
    const auto help = [&](std::size_t k) {
        guarded(k, [&] {
            if (next >= chunks) {
                return;
            }
            driverCheck(driver().makeCurrent(context), "current context");
            if (std::unique_ptr<Slot> slot{pool.tryTake()}) {
                const HeldSlot held{pool, std::move(slot)};
                work(*held);
            }
        });
    };
    {
        std::vector<std::jthread> helpers;
        helpers.reserve(workers - 1);
        try {
            for (std::size_t k{1}; k < workers; ++k) {
                helpers.emplace_back(help, k);
            }
        } catch (const std::system_error&) {
            // Fewer threads than asked for: the ones that started share the chunks.
        }
        guarded(0, [&] { work(*own); });
    }
    for (const std::exception_ptr& e : failed) {
        if (e) {
            std::rethrow_exception(e);
        }
    }
}

SlotPool* retainQueryBuffers()
{
    const CUcontext context{currentContext()};
    if (!isPrimary(context)) {
        return nullptr;
    }
    unsigned long long id{0};
    driverCheck(driver().id(context, &id), "context id");
    SlotPool& pool{keptSlots(id)};
    const std::lock_guard lock{pool.mutex};
    ++pool.scenes;
    return &pool;
}

void releaseQueryBuffers(SlotPool* kept)
{
    if (kept == nullptr) {
        return;
    }
    std::array<std::unique_ptr<Slot>, kMaxWorkers> given;
    {
        const std::lock_guard lock{kept->mutex};
        if (--kept->scenes > 0) {
            return;
        }
        std::move(kept->idle.begin(), kept->idle.end(), given.begin());
        kept->made -= kept->idle.size();
        kept->idle.clear();
        kept->freed.notify_all();
    }
}

} // namespace albedo_b200
