// Ray queries from host arrays: chunks of rays staged through pinned memory by
// a few threads, each with a stream and buffers of its own.
//
// A query call moves 24 to 28 bytes a ray in and 4 to 56 out. Through pageable
// copies one thread of the driver stages all of it, before and after the
// kernel, into device buffers allocated for the call. Here each worker copies
// a chunk into its pinned buffer, enqueues upload, kernel and download on its
// stream, waits, and copies the chunk's results out, so that the host copies of
// several chunks, the transfers and the kernels overlap, and nothing is
// allocated after the first calls.
// Measured on 16 host cores, from and to pageable arrays, instanced trefoils, ms
// (pageable copies and per-call buffers -> this): 1,000,003 any-hit queries 4.89
// -> 1.61, 1,000 of them 0.13 -> 0.07; closest hits with their geometry 262,144
// 7.37 -> 2.38, 10,000 0.385 -> 0.180, 100 0.200 -> 0.092; 1,048,576 without 8.09 ->
// 2.68. The first call of a size pays about a millisecond for each worker's buffers.
#pragma once

#include <cuda_runtime_api.h>

#include <cstddef>
#include <cstdint>
#include <functional>
#include <span>

namespace albedo_b200 {

struct QueryInput {
    const void* host;
    std::size_t ray_bytes;
};

// `host` may be null: the values are computed and dropped.
struct QueryOutput {
    void* host;
    std::size_t ray_bytes;
};

constexpr std::size_t kMaxQueryArrays{8};
// Bytes a ray may take over all inputs and outputs of one call.
constexpr std::size_t kMaxQueryRayBytes{84};

// Enqueues the queries of one chunk: device arrays in the order of the call's
// inputs and outputs.
using QueryLaunch =
    std::function<cudaError_t(void* const* inputs, void* const* outputs, int count, cudaStream_t stream)>;

// A context's slots (a worker's stream and buffers each): at most eight, made as
// they are needed.
struct SlotPool;

// A scene came to the calling thread's current context: the slots kept for queries
// there, until the last scene leaves it. They are kept in a device's primary
// context alone; a context that a program made may be destroyed while scenes of it
// are alive, and its streams with it. Null elsewhere: a call has its own.
SlotPool* retainQueryBuffers();
void releaseQueryBuffers(SlotPool* kept);

// Runs `count` queries in the calling thread's current context, that of the scene
// that holds `kept`, after the work that the default stream held when the call was
// made, and returns when every result is in its host array. Safe from several
// threads. Throws std::bad_alloc, or std::runtime_error for any other CUDA failure.
void runQueries(SlotPool* kept, std::int64_t count, std::span<const QueryInput> inputs,
                std::span<const QueryOutput> outputs, const QueryLaunch& launch);

} // namespace albedo_b200
