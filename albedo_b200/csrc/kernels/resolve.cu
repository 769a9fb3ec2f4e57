// The film's resolve: per-pixel FP64 accumulators to 8-bit sRGB, 3 bytes a pixel,
// rows from the top — the bytes the reference's writePpm writes for
// PixelBuffer::average (image/ppm.cpp:22-33, image/pixel_buffer.cpp:37-45,
// color/srgb.cpp:18-36).
//
// The byte is that of sum / count in FP64, correctly rounded as on the host. It
// comes from the host's tables: 255 thresholds (the smallest double of each
// byte, found with the reference's own transfer function) and a start byte per
// bucket of doubles (exponent and top 7 mantissa bits) that holds at most one
// threshold. One table read and one comparison settle a channel (the tiled
// kernel packs both tables into one 64-bit entry per bucket), so the result is
// the reference's byte exactly and the kernel evaluates no power function; and
// where a quotient good to 2^-44 is not next to a decision it stands for the
// exact one. A pure stream: 32 bytes read and 3 written per pixel, the reads as
// one coalesced 256-bit load per pixel; 3840x2160 takes 51.6 us among other
// launches, 86% of the measured copy bandwidth, and 54.3 by itself.
#include "launch.hpp"

#include <algorithm>
#include <cstdint>

namespace albedo_b200 {

namespace {

// The tiled kernel: one block of 24 warps per SM, four pixels a lane in flight
// (4 KB a warp, 96 KB an SM). Every block packs the tables into shared memory
// first, from constant-bank reads that differ per lane, so fewer and wider
// blocks start sooner: among other launches 3840x2160 51.6 us, against 55.7 for four
// blocks of 256 threads and 67.8 for eight (1920x1080 18.5, 24.0 and 30.8).
constexpr int kTileThreads{768};
constexpr int kTileBlocksPerSm{1};
constexpr int kResolveGroup{4};
// The kernel for any alignment.
constexpr int kAnyThreads{256};
constexpr int kAnyBlocksPerSm{6};

__device__ __forceinline__ unsigned int srgbByteOf(double v, double lowest, double highest, const double* lower,
                                                   const unsigned char* start)
{
    // Without branches: NaN, zero and negative averages fail `in_range` (byte
    // 0); 1.0 and above pass `saturated` (byte 255). Between them v lies in a
    // bucket, since lower[1] > 2^-13 and lower[255] <= 1; outside, the bucket
    // and the start byte are clamped so every table read stays in bounds, and
    // the selects discard what they give. The bucket is the high word of v
    // shifted right by kResolveBucketShift - 32.
    const bool in_range{v >= lowest};
    const bool saturated{v >= highest};
    const int bucket{min(max((__double2hiint(v) >> (kResolveBucketShift - 32)) -
                                 static_cast<int>(kResolveBucketBase),
                             0),
                         kResolveBuckets - 1)};
    const unsigned int b{min(static_cast<unsigned int>(start[bucket]), 254u)};
    const unsigned int byte{b + (v >= lower[b + 1] ? 1u : 0u)};
    return saturated ? 255u : (in_range ? byte : 0u);
}

// PixelBuffer::average (image/pixel_buffer.cpp:37-45): the count is unsigned.
struct Divisor {
    unsigned long long count;
    double reciprocal;  // 2^-k when count = 2^k, else 0
};

__device__ __forceinline__ Divisor divisorOf(unsigned long long count)
{
    const bool power_of_two{count != 0 && (count & (count - 1)) == 0};
    const long long k{63 - __clzll(static_cast<long long>(count))};
    return {count, power_of_two ? __longlong_as_double((1023 - k) << 52) : 0.0};
}

__device__ __forceinline__ double averageOf(double sum, const Divisor& d)
{
    if (d.count == 0) {
        return 0.0;
    }
    return d.reciprocal != 0.0 ? sum * d.reciprocal : sum / static_cast<double>(d.count);
}

// The tables into shared memory; every thread takes part.
__device__ __forceinline__ void loadTables(const SrgbThresholds& table, double* lower, unsigned char* start)
{
    for (int i{static_cast<int>(threadIdx.x)}; i < 256; i += blockDim.x) {
        lower[i] = table.lower[i];
    }
    for (int i{static_cast<int>(threadIdx.x)}; i < kResolveBuckets; i += blockDim.x) {
        start[i] = table.start[i];
    }
    __syncthreads();
}

// One pixel's accumulator in one 256-bit load (sm_100 global vector load), marked
// streaming: each accumulator is read once. The address is 32-byte aligned.
__device__ __forceinline__ void loadPixel(const PixelAccum* a, double& r, double& g, double& b,
                                          unsigned long long& count)
{
    double c;
    asm("ld.global.cs.v4.f64 {%0, %1, %2, %3}, [%4];"
                 : "=d"(r), "=d"(g), "=d"(b), "=d"(c)
                 : "l"(a));
    count = static_cast<unsigned long long>(__double_as_longlong(c));
}

constexpr int kResolveWarps{kTileThreads / 32};
constexpr int kTilePixels{32 * kResolveGroup};
constexpr int kTileBytes{3 * kTilePixels};  // 96 * kResolveGroup: whole 16-byte units

// The tiled kernel's form of the tables: one 64-bit entry per bucket, read with
// one shared-memory load: the bucket's start byte s, and of the threshold
// lower[s + 1], when it lies in the bucket, the top 32 of its
// kResolveBucketShift low bits (kNoCut when it does not). Doubles of one bucket
// share their high bits, so comparing these "cuts" compares the values to 2^-39.
constexpr unsigned int kNoCut{0xFFFFFFFFu};
constexpr int kCutShift{kResolveBucketShift - 32};

__device__ __forceinline__ unsigned int cutOf(double v)
{
    return __funnelshift_r(static_cast<unsigned int>(__double2loint(v)),
                           static_cast<unsigned int>(__double2hiint(v)), kCutShift);
}

__device__ __forceinline__ void packBuckets(const SrgbThresholds& table, uint2* packed)
{
    for (int k{static_cast<int>(threadIdx.x)}; k < kResolveBuckets; k += blockDim.x) {
        const unsigned int s{table.start[k]};
        unsigned int cut{kNoCut};
        if (s < 255) {
            const double t{table.lower[s + 1]};
            if ((__double_as_longlong(t) >> kResolveBucketShift) == kResolveBucketBase + k) {
                cut = cutOf(t);
            }
        }
        packed[k] = make_uint2(cut, s);
    }
    __syncthreads();
}

// An average to within 2^-44 without a division: the FP32 reciprocal of the
// count (2^-22) and one Newton step in FP64 (2^-44), then one product a channel.
struct NearDivisor {
    double reciprocal;
};

__device__ __forceinline__ NearDivisor nearDivisorOf(unsigned long long count)
{
    // Counts below 2^32 (nearly all) convert with one instruction.
    const unsigned int low{static_cast<unsigned int>(count)};
    const bool wide{(count >> 32) != 0};
    const double c{wide ? static_cast<double>(count) : static_cast<double>(low)};
    const double r{static_cast<double>(__frcp_rn(static_cast<float>(c)))};
    // No samples: the average is zero.
    return {count == 0 ? 0.0 : fma(r, fma(-c, r, 1.0), r)};
}

// The byte of an average known to 2^-44. `unsure` is set when a threshold, or
// the edge of the bucket (beyond which one may lie), is within 2^-39 of it: then
// the caller divides. Every other average's byte is that of the exact one.
__device__ __forceinline__ unsigned int srgbByteNear(double v, double lowest, double highest, const uint2* packed,
                                                     bool& unsure)
{
    const bool in_range{v >= lowest};
    const bool saturated{v >= highest};
    const int bucket{min(max((__double2hiint(v) >> (kResolveBucketShift - 32)) -
                                 static_cast<int>(kResolveBucketBase),
                             0),
                         kResolveBuckets - 1)};
    const uint2 entry{packed[bucket]};
    const unsigned int cut{cutOf(v)};
    // Only from just below the first threshold to just above the last one
    // (black and saturated averages, exact zeros and ones among them, are sure).
    const int first{__double2hiint(lowest) - 1};
    const int span{__double2hiint(highest) + 1 - first};
    const bool near_range{static_cast<unsigned int>(__double2hiint(v) - first) <= static_cast<unsigned int>(span)};
    unsure |= near_range && (cut + 1u <= 1u || cut - entry.x + 1u <= 2u);
    const unsigned int byte{entry.y + (cut > entry.x ? 1u : 0u)};
    return saturated ? 255u : (in_range ? byte : 0u);
}

// One warp tile into the warp's stage: lane l resolves pixels l, l + 32, ...
// of the tile's n. FULL tiles (n == kTilePixels) need no bounds tests, so the
// loads and the byte computations run as straight-line code the compiler can
// interleave.
//
// Three correctly rounded FP64 divisions a pixel bounded the kernel; a quotient
// to 2^-44 decides the byte of all but about one average in 2^30. 3840x2160,
// half the pixels of 36 samples and half of 64: 71.8 -> 55.7 us.
template <bool FULL>
__device__ __forceinline__ void resolveTile(const PixelAccum* tile, int n, int lane, unsigned char* stage,
                                            double lowest, double highest, const uint2* packed,
                                            const SrgbThresholds& table)
{
    double r[kResolveGroup], g[kResolveGroup], b[kResolveGroup];
    unsigned long long count[kResolveGroup];
#pragma unroll
    for (int j{0}; j < kResolveGroup; ++j) {
        const int q{lane + 32 * j};
        r[j] = g[j] = b[j] = 0.0;
        count[j] = 0;
        if (FULL || q < n) {
            loadPixel(tile + q, r[j], g[j], b[j], count[j]);
        }
    }
#pragma unroll
    for (int j{0}; j < kResolveGroup; ++j) {
        const int q{lane + 32 * j};
        if (FULL || q < n) {
            const NearDivisor d{nearDivisorOf(count[j])};
            bool unsure{false};
            unsigned int br{srgbByteNear(r[j] * d.reciprocal, lowest, highest, packed, unsure)};
            unsigned int bg{srgbByteNear(g[j] * d.reciprocal, lowest, highest, packed, unsure)};
            unsigned int bb{srgbByteNear(b[j] * d.reciprocal, lowest, highest, packed, unsure)};
            if (unsure) {
                const Divisor exact{divisorOf(count[j])};
                br = srgbByteOf(averageOf(r[j], exact), lowest, highest, table.lower, table.start);
                bg = srgbByteOf(averageOf(g[j], exact), lowest, highest, table.lower, table.start);
                bb = srgbByteOf(averageOf(b[j], exact), lowest, highest, table.lower, table.start);
            }
            stage[3 * q + 0] = static_cast<unsigned char>(br);
            stage[3 * q + 1] = static_cast<unsigned char>(bg);
            stage[3 * q + 2] = static_cast<unsigned char>(bb);
        }
    }
}

// Accumulators 32-byte aligned and output 16-byte aligned. Each warp resolves
// tiles of kTilePixels pixels: lane l takes pixels l, l + 32, ..., so each of
// its kResolveGroup loads is one coalesced 1 KB read across the warp. The bytes
// are transposed through the warp's shared-memory stage and leave as coalesced
// 16-byte stores.
__global__ void __launch_bounds__(kTileThreads, kTileBlocksPerSm)
    resolveSrgbTiles(const PixelAccum* __restrict__ accum, long long pixels, unsigned char* __restrict__ out,
                     const __grid_constant__ SrgbThresholds table)
{
    __shared__ uint2 packed[kResolveBuckets];
    __shared__ __align__(16) unsigned char stage[kResolveWarps][kTileBytes];
    packBuckets(table, packed);
    const double lowest{table.lower[1]};
    const double highest{table.lower[255]};
    const int lane{static_cast<int>(threadIdx.x) & 31};
    const int warp{static_cast<int>(threadIdx.x) >> 5};
    unsigned char* my_stage{stage[warp]};

    const long long tiles{(pixels + kTilePixels - 1) / kTilePixels};
    const long long warps_total{static_cast<long long>(gridDim.x) * kResolveWarps};
    for (long long t{static_cast<long long>(blockIdx.x) * kResolveWarps + warp}; t < tiles; t += warps_total) {
        const long long first{t * kTilePixels};
        const int n{static_cast<int>(min(static_cast<long long>(kTilePixels), pixels - first))};
        if (n == kTilePixels) {
            resolveTile<true>(accum + first, n, lane, my_stage, lowest, highest, packed, table);
        } else {
            resolveTile<false>(accum + first, n, lane, my_stage, lowest, highest, packed, table);
        }
        __syncwarp();
        unsigned char* dst{out + 3 * first};
        if (n == kTilePixels) {
            for (int i{lane}; i < kTileBytes / 16; i += 32) {
                __stcs(reinterpret_cast<uint4*>(dst) + i, reinterpret_cast<const uint4*>(my_stage)[i]);
            }
        } else {
            for (int i{lane}; i < 3 * n; i += 32) {
                dst[i] = my_stage[i];
            }
        }
        __syncwarp();
    }
}

// Any other alignment (accumulators at least 8-byte aligned): one pixel per
// thread per turn, 8-byte loads and byte stores.
__global__ void __launch_bounds__(kAnyThreads) resolveSrgbAnyAlignment(const PixelAccum* __restrict__ accum,
                                                                            long long pixels,
                                                                            unsigned char* __restrict__ out,
                                                                            SrgbThresholds table)
{
    __shared__ double lower[256];
    __shared__ unsigned char start[kResolveBuckets];
    loadTables(table, lower, start);
    const double lowest{lower[1]};
    const double highest{lower[255]};
    const long long stride{static_cast<long long>(gridDim.x) * blockDim.x};
    for (long long p{static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x}; p < pixels; p += stride) {
        const PixelAccum* a{accum + p};
        const Divisor d{divisorOf(static_cast<unsigned long long>(__ldcs(&a->count)))};
        out[3 * p + 0] = static_cast<unsigned char>(srgbByteOf(averageOf(__ldcs(&a->r), d), lowest, highest, lower,
                                                               start));
        out[3 * p + 1] = static_cast<unsigned char>(srgbByteOf(averageOf(__ldcs(&a->g), d), lowest, highest, lower,
                                                               start));
        out[3 * p + 2] = static_cast<unsigned char>(srgbByteOf(averageOf(__ldcs(&a->b), d), lowest, highest, lower,
                                                               start));
    }
}

} // namespace

cudaError_t launchResolveSrgb(const PixelAccum* accum, long long pixels, unsigned char* out,
                              const SrgbThresholds& table, cudaStream_t stream)
{
    if (pixels <= 0) {
        return cudaSuccess;
    }
    int device{0};
    int sms{0};
    cudaError_t e{cudaGetDevice(&device)};
    if (e == cudaSuccess) {
        e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    }
    if (e != cudaSuccess) {
        return e;
    }
    // A grid-stride stream, one wave of resident blocks: all of them keep
    // loads in flight, enough to saturate HBM.
    const bool tiled{(reinterpret_cast<std::uintptr_t>(accum) & 31) == 0 &&
                     (reinterpret_cast<std::uintptr_t>(out) & 15) == 0};
    const auto kernel{tiled ? resolveSrgbTiles : resolveSrgbAnyAlignment};
    const int per_sm{tiled ? kTileBlocksPerSm : kAnyBlocksPerSm};
    const int threads{tiled ? kTileThreads : kAnyThreads};
    const long long per_block{tiled ? static_cast<long long>(kTilePixels) * kResolveWarps : kAnyThreads};
    const long long wanted{(pixels + per_block - 1) / per_block};
    const int blocks{static_cast<int>(std::min(wanted, static_cast<long long>(per_sm) * sms))};
    kernel<<<blocks, threads, 0, stream>>>(accum, pixels, out, table);
    return cudaGetLastError();
}

} // namespace albedo_b200
