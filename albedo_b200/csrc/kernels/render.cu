// The plain per-pixel megakernel and the ray-query kernels.
//
// renderPixel (render/render_image.cpp:27-44): each pixel owns one PCG32 stream
// and draws its n x n stratified samples from it in row-major order, so one
// thread runs one pixel's samples serially. Blocks cover tiles of 128 pixels
// (16 x 8 by default; fewer pixels for small images) so a warp's camera rays start
// coherent. The traversal stack of every thread sits in shared memory: STACK
// child references of 4 bytes, or STACK entries of 8 bytes in the counting
// kernels.
#include "estimator.cuh"

#include <type_traits>

namespace albedo_b200 {

namespace {

constexpr int kBlock = kTraceBlock;
constexpr int kTileW = 16; // default tile: 16 x 8 pixels
// Resident blocks per SM the megakernel's register budget is sized for: 3 (168
// registers a thread). The path estimator is also compiled for 4 (128 registers,
// lean); chooseBlocksPerSm says when each is taken for a scene that has not been
// tuned.
#ifndef ALBEDO_MEGA_BLOCKS_PER_SM
#define ALBEDO_MEGA_BLOCKS_PER_SM 3
#endif
constexpr int kMegaBlocksPerSm = ALBEDO_MEGA_BLOCKS_PER_SM;

// Pixels a block renders: warp_pixels in each of its four warps.
__host__ __device__ inline int blockPixels(const RenderArgs& args) { return kBlock / 32 * args.warp_pixels; }

// Width of a block's tile: the shape's for full warps, near-square for fewer
// pixels (8 x 8, 8 x 4, 4 x 4, 4 x 2, 2 x 2).
__host__ __device__ inline int tileWidth(const RenderArgs& args)
{
    if (args.warp_pixels == 32) {
        return args.tile_width > 0 ? args.tile_width : kTileW;
    }
    return args.warp_pixels >= 8 ? 8 : (args.warp_pixels >= 2 ? 4 : 2);
}

// Per-pixel running sums: FP64, or FP32 with Kahan compensation.
template <int ACC>
struct PixelSums;

// reset() zeroes them.
template <>
struct PixelSums<kAccumulateFp64> {
    double r, g, b;
    ALB_DEV void reset() { r = g = b = 0.0; }
    ALB_DEV void add(float3 v)
    {
        r += v.x;
        g += v.y;
        b += v.z;
    }
    ALB_DEV double3 total() const { return make_double3(r, g, b); }
};

template <>
struct PixelSums<kAccumulateKahan> {
    float r, g, b;
    float cr, cg, cb;
    ALB_DEV void reset() { r = g = b = cr = cg = cb = 0.0f; }
    // Kahan 1965: c carries the low-order part lost by the previous addition.
    static ALB_DEV void kahan(float& sum, float& c, float v)
    {
        const float y = __fsub_rn(v, c);
        const float t = __fadd_rn(sum, y);
        c = __fsub_rn(__fsub_rn(t, sum), y);
        sum = t;
    }
    ALB_DEV void add(float3 v)
    {
        kahan(r, cr, v.x);
        kahan(g, cg, v.y);
        kahan(b, cb, v.z);
    }
    ALB_DEV double3 total() const
    {
        return make_double3(static_cast<double>(r) - cr, static_cast<double>(g) - cg, static_cast<double>(b) - cb);
    }
};

// A path's state kept in shared memory by the lean variants: 23 words a thread
// (an odd stride, so a warp's accesses to one field hit 32 different banks).
struct alignas(4) SharedPath {
    PathState p;
    float pad;
};
static_assert(sizeof(SharedPath) % 8 == 4, "odd word stride");

// Stack entry type: the child reference alone (4 bytes), but for the counting
// kernels, whose counts are those of a traversal that drops popped entries
// beyond the current hit (8 bytes: reference and entry distance).
template <bool COUNT>
using StackEntry = std::conditional_t<COUNT, uint2, unsigned>;

// INL: 0 = both queries call the shared out-of-line traversal, 1 = both are
// inlined, 2 = the closest-hit query is inlined and the shadow query calls the
// out-of-line copy (a smaller kernel than 1, no register saves around the
// per-bounce call). LEAN: the path's state between bounces lives in shared
// memory rather than registers, so fewer registers carry state across the
// traversal and more blocks fit an SM.
template <int STACK, int EST, bool COUNT = false, int MINB = kMegaBlocksPerSm, int ACC = kAccumulateFp64,
          int INL = 0, bool LEAN = false>
__global__ void __launch_bounds__(kBlock, MINB) megakernel(const DevScene scene, const DevCamera camera,
                                                          const RenderArgs args, PixelAccum* accum,
                                                          unsigned int* error_flag,
                                                          unsigned long long* totals = nullptr)
{
    using Entry = StackEntry<COUNT>;
    extern __shared__ uint2 stack_memory[];
    Entry* const stack = reinterpret_cast<Entry*>(stack_memory);
    TraversalCounts counts{0, 0, 0, 0, 0, 0};
    const TraceContext<INL != 0, COUNT, INL == 1, Entry, EST == kEstimatorPath> ctx{
        TraceStack<Entry>::of(stack + threadIdx.x, STACK), error_flag, COUNT ? &counts : nullptr};
    int x, y, slot;
    const int lanes = args.warp_pixels;
    const int lane = static_cast<int>(threadIdx.x) & 31;
    if (lane >= lanes) {
        return;
    }
    const int place = (static_cast<int>(threadIdx.x) >> 5) * lanes + lane;
    if (args.pixels != nullptr) {
        slot = blockIdx.x * blockPixels(args) + place;
        if (slot >= args.pixel_count) {
            return;
        }
        x = args.pixels[slot].x;
        y = args.pixels[slot].y;
    } else {
        const int tile_w = tileWidth(args);
        const int tile_h = blockPixels(args) / tile_w;
        const int tiles_x = (args.width + tile_w - 1) / tile_w;
        x = (blockIdx.x % tiles_x) * tile_w + place % tile_w;
        y = (blockIdx.x / tiles_x) * tile_h + place / tile_w;
        if (x >= args.width || y >= args.height) {
            return;
        }
        slot = y * args.width + x;
    }
    Pcg32 g = pixelGenerator(args.seed, static_cast<std::uint32_t>(x), static_cast<std::uint32_t>(y),
                             static_cast<std::uint32_t>(args.width));
    const int n = args.samples_per_axis;
    const float inv_n = 1.0f / static_cast<float>(n);
    const float width = static_cast<float>(args.width);
    const float height = static_cast<float>(args.height);
    PixelSums<ACC> sums;
    sums.reset();
    // Sums of squared samples (for two-sample tests) go straight to memory, one
    // read-modify-write per sample, only when asked for: no registers carry them
    // through the traversal calls of an ordinary render.
    double* const squares = args.sum_squares != nullptr ? args.sum_squares + 3 * slot : nullptr;
    // One bounce per iteration: a lane whose path ends starts the pixel's next
    // sample at once (drawing its jitter next from the same stream, as the
    // reference does), so a warp waits for the longest pixel, not the longest
    // path of every sample.
    const int total = n * n;
    int sample = 0;
    PathState local_path;
    PathState* path_ptr = &local_path;
    if constexpr (LEAN) {
        __shared__ SharedPath shared_paths[kBlock];
        path_ptr = &shared_paths[threadIdx.x].p;
    }
    PathState& path = *path_ptr;
    startSample(camera, path, g, x, y, 0, n, inv_n, width, height);
    for (;;) {
        if (estimatorBounce<EST>(scene, ctx, path, g, args)) {
            continue;
        }
        const float3 L = path.result;
        sums.add(L);
        if (squares != nullptr) {
            squares[0] += static_cast<double>(L.x) * L.x;
            squares[1] += static_cast<double>(L.y) * L.y;
            squares[2] += static_cast<double>(L.z) * L.z;
        }
        if (++sample == total) {
            break;
        }
        startSample(camera, path, g, x, y, sample, n, inv_n, width, height);
    }
    PixelAccum& a = accum[slot];
    const double3 total_sum = sums.total();
    a.r += total_sum.x;
    a.g += total_sum.y;
    a.b += total_sum.z;
    a.count += static_cast<long long>(n) * n;
    if constexpr (COUNT) {
        atomicAdd(totals + 0, counts.boxes);
        atomicAdd(totals + 1, counts.triangles);
        atomicAdd(totals + 2, counts.spheres);
        atomicAdd(totals + 3, counts.instances);
        atomicAdd(totals + 4, counts.rays);
        atomicAdd(totals + 5, counts.reference_boxes);
    }
}

// Closest-hit queries of given rays, counting their traversal work into
// totals[0..5] (as the counting megakernel does). Not used for timing.
template <int STACK>
__global__ void __launch_bounds__(kBlock) traceCountKernel(const DevScene scene, const float* rays, int count,
                                                           float t_min, float t_max, unsigned int* error_flag,
                                                           unsigned long long* totals)
{
    extern __shared__ uint2 stack[];
    const int i = blockIdx.x * kBlock + threadIdx.x;
    if (i >= count) {
        return;
    }
    TraversalCounts counts{0, 0, 0, 0, 0, 0};
    const float3 o = mk(rays[6 * i], rays[6 * i + 1], rays[6 * i + 2]);
    const float3 d = mk(rays[6 * i + 3], rays[6 * i + 4], rays[6 * i + 5]);
    TraceHit hit;
    float tmax = t_max;
    static_cast<void>(traceScene<false, false, true>(scene, o, d, t_min, tmax, SkipRule::none(), hit,
                                                     TraceStack<uint2>::of(stack + threadIdx.x, STACK), error_flag,
                                                     &counts));
    atomicAdd(totals + 0, counts.boxes);
    atomicAdd(totals + 1, counts.triangles);
    atomicAdd(totals + 2, counts.spheres);
    atomicAdd(totals + 3, counts.instances);
    atomicAdd(totals + 4, counts.rays);
    atomicAdd(totals + 5, counts.reference_boxes);
}

// The ray a thread of a query kernel takes when `lanes` lanes of each warp take
// one (-1: none).
ALB_DEV int queryRay(int count, int lanes)
{
    const int lane = static_cast<int>(threadIdx.x) & 31;
    const int i = (static_cast<int>(blockIdx.x) * (kBlock / 32) + (static_cast<int>(threadIdx.x) >> 5)) * lanes + lane;
    return lane < lanes && i < count ? i : -1;
}

template <int STACK>
__global__ void __launch_bounds__(kBlock) traceKernel(const DevScene scene, const float* rays, int count, int lanes,
                                                      float t_min, float t_max, TraceOutputs out,
                                                      unsigned int* error_flag)
{
    extern __shared__ unsigned ref_stack[];
    const int i = queryRay(count, lanes);
    if (i < 0) {
        return;
    }
    const float3 o = mk(rays[6 * i], rays[6 * i + 1], rays[6 * i + 2]);
    const float3 d = mk(rays[6 * i + 3], rays[6 * i + 4], rays[6 * i + 5]);
    TraceHit hit;
    float tmax = t_max;
    const bool found = traceScene<false>(scene, o, d, t_min, tmax, SkipRule::none(), hit,
                                         TraceStack<unsigned>::of(ref_stack + threadIdx.x, STACK), error_flag);
    out.hit[i] = found ? 1 : 0;
    if (!found) {
        return;
    }
    Surface sf;
    resolveHit(scene, o, d, hit, sf);
    out.t[i] = static_cast<float>(refinedDistance(scene, o, d, hit));
    out.object[i] = static_cast<int>(sf.object_id);
    out.triangle[i] = -1;
    const DevObject obj = scene.objects[hit.obj_pos];
    if (obj.kind == kObjInstance) {
        out.triangle[i] = static_cast<int>(__float_as_uint(scene.triangles[hit.tri_pos].v0w));
    }
    if (out.point != nullptr) {
        out.point[3 * i] = sf.p.x;
        out.point[3 * i + 1] = sf.p.y;
        out.point[3 * i + 2] = sf.p.z;
        out.normal[3 * i] = sf.n.x;
        out.normal[3 * i + 1] = sf.n.y;
        out.normal[3 * i + 2] = sf.n.z;
        out.shading_normal[3 * i] = sf.ns.x;
        out.shading_normal[3 * i + 1] = sf.ns.y;
        out.shading_normal[3 * i + 2] = sf.ns.z;
        out.front[i] = sf.front ? 1 : 0;
    }
}

template <int STACK>
__global__ void __launch_bounds__(kBlock) occludedKernel(const DevScene scene, const float* rays, const float* t_max,
                                                         int count, int lanes, int* occluded_out,
                                                         unsigned int* error_flag)
{
    extern __shared__ unsigned ref_stack[];
    const int i = queryRay(count, lanes);
    if (i < 0) {
        return;
    }
    const float3 o = mk(rays[6 * i], rays[6 * i + 1], rays[6 * i + 2]);
    const float3 d = mk(rays[6 * i + 3], rays[6 * i + 4], rays[6 * i + 5]);
    TraceHit hit;
    float tmax = t_max[i];
    occluded_out[i] = traceScene<true>(scene, o, d, 0.0f, tmax, SkipRule::none(), hit,
                                       TraceStack<unsigned>::of(ref_stack + threadIdx.x, STACK), error_flag)
                          ? 1
                          : 0;
}

constexpr std::size_t stackBytes(int stack, std::size_t entry_bytes)
{
    return static_cast<std::size_t>(stack) * kBlock * entry_bytes;
}

constexpr int kCountEntry = static_cast<int>(sizeof(StackEntry<true>));

int megaBlocks(const RenderArgs& args)
{
    if (args.pixels != nullptr) {
        return (args.pixel_count + blockPixels(args) - 1) / blockPixels(args);
    }
    const int tile_w = tileWidth(args);
    const int tile_h = blockPixels(args) / tile_w;
    return ((args.width + tile_w - 1) / tile_w) * ((args.height + tile_h - 1) / tile_h);
}

// The smallest power of two (32 at most) of items a warp for which `items` take
// no more than `warps_per_sm` warps on every SM of the current device.
cudaError_t spreadOver(int warps_per_sm, long long items, int& lanes)
{
    int device = 0;
    int sms = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e == cudaSuccess) {
        e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    }
    const long long warps = static_cast<long long>(sms) * warps_per_sm;
    lanes = 1;
    while (lanes < 32 && items > warps * lanes) {
        lanes *= 2;
    }
    return e;
}

long long imagePixels(const RenderArgs& args)
{
    return args.pixels != nullptr ? args.pixel_count : static_cast<long long>(args.width) * args.height;
}

// How many lanes of a warp take a pixel (RenderArgs::warp_pixels): 32, or fewer
// for an image too small to fill the GPU with full warps. A pixel's samples run
// in sequence on its lane, so a small image takes as long as its slowest warps,
// and a warp of divergent lanes takes several times as long as one lane alone:
// spreading the pixels over the idle warp slots shortens each warp's chain. The
// smallest power of two is taken whose warps are at most 12 per SM, the resident
// warps of the default shape (3 blocks of 4), or 3 per SM for scenes of spheres
// with hardly any triangle, whose short queries leave less divergence to save
// and whose FP64 sphere tests cost a warp the same for one lane as for 32.
//
// Measured, 9 samples, depth 10, full warps -> this rule, in ms (trefoils of
// 12,288 triangles / 20,480-triangle icosphere / soup of 30,000):
//   64x36 4.04 / 3.60 / 5.72 -> 1.79 / 1.65 / 1.87
//   96x54 4.18 / 4.28 / 7.21 -> 2.44 / 2.26 / 3.08
//   128x72 4.16 / 4.68 / 7.83 -> 3.03 / 3.17 / 4.41
//   192x108 4.54 / 5.00 / 8.37 -> 4.56 / 4.35 / 6.36
// From 256x144 on full warps win for some of them (trefoils 5.48, and 6.21 at
// 16 pixels a warp). Sphere room: 32x18 1.54 -> 0.66, 64x36 1.79 -> 1.26, 96x54
// 1.86 -> 1.60; at 128x72 full warps, 1.87, beat 16 pixels a warp, 1.95.
cudaError_t chooseWarpPixels(const DevScene& scene, RenderArgs& args)
{
    constexpr std::uint32_t kFewTriangles = 256;
    return spreadOver(scene.triangle_count < kFewTriangles ? 3 : 12, imagePixels(args), args.warp_pixels);
}

// The register budget of a path-estimator launch that names none: 4 blocks per SM
// (lean) for images of many waves of warps, 3 otherwise. Four resident warps a
// scheduler hide more of a query's dependent fetches than three, but each warp then
// takes longer over its pixels' samples, which run in sequence. With many waves the
// longer chains of a few pixels are overlapped by other warps; with few, the launch
// waits for them. A mesh whose queries enter many nodes (overlapping boxes:
// RenderArgs::mesh_steps) waits longest on memory and gains from fewer waves on.
//
// Measured, lean over 3 blocks per SM: 1920x1080, 36 waves of the 3-block shape, in
// 25 scenes of 5 to 1.31M triangles and one to seven materials, 2 and 3 samples an
// axis, 0.84 (200,003-triangle soup) to 0.98 (instances of gold and rough glass);
// 1440x810, 20 waves: 0.90 to 1.01; 1280x720, 16 waves: 0.84 to 1.02; 960x540, 9
// waves: 0.89 to 1.05; 640x360, 4 waves: up to 1.11. Soups of 20,000 to 300,000
// triangles (mesh_steps 43 to 221) take 0.80 to 0.92 from 800x450, 6.3 waves, on,
// but up to 1.06 at 640x360. Closed surfaces of 1,280 to 1.31M triangles (12 to 24)
// scatter between 0.92 and 1.08 at 800x450. The costliest mesh decides, however small:
// soups of 20,000 and 200,000 triangles and a tenth to half the size of the trefoils
// or the icosphere beside them take 0.92 to 0.99 from 800x450 on; beside the
// icosphere and as large as it, 1.10 at 800x450 and 0.94 to 0.99 at 960x540.
constexpr int kDefaultWarpsPerSm = kMegaBlocksPerSm * kBlock / 32;

constexpr int defaultBlocksPerSm(long long pixels, int sms, int warp_pixels, float mesh_steps)
{
    constexpr int kManyWaves = 20;
    constexpr int kCostlyMeshWaves = 6;
    constexpr float kCostlyMeshSteps = 40.0f;
    const int waves = mesh_steps >= kCostlyMeshSteps ? kCostlyMeshWaves : kManyWaves;
    const long long full = static_cast<long long>(sms) * kDefaultWarpsPerSm * warp_pixels * waves;
    return pixels >= full ? 4 : kMegaBlocksPerSm;
}

// Both sides of each limit, for 148 SMs (12 x 32 x 148 = 56,832 pixels a wave).
static_assert(kMegaBlocksPerSm != 3 ||
              (defaultBlocksPerSm(20 * 56832 - 1, 148, 32, 39.9f) == 3 &&
               defaultBlocksPerSm(20 * 56832, 148, 32, 0.0f) == 4 &&
               defaultBlocksPerSm(6 * 56832 - 1, 148, 32, 40.0f) == 3 &&
               defaultBlocksPerSm(6 * 56832, 148, 32, 40.0f) == 4 &&
               defaultBlocksPerSm(6 * 56832, 148, 32, 39.9f) == 3 && defaultBlocksPerSm(1, 148, 1, 200.0f) == 3));

cudaError_t chooseBlocksPerSm(RenderArgs& args)
{
    if (args.blocks_per_sm != 0 || args.estimator != kEstimatorPath) {
        return cudaSuccess;
    }
    int device = 0;
    int sms = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e == cudaSuccess) {
        e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    }
    args.blocks_per_sm = defaultBlocksPerSm(imagePixels(args), sms, args.warp_pixels, args.mesh_steps);
    return e;
}

// Ray queries spread likewise, over 8 warps per SM (a staged call runs up to eight
// chunks beside each other): 1,000 any-hit queries of the trefoils from host
// arrays 0.081 -> 0.072 ms, 100,000 0.353 -> 0.331.
constexpr int kQueryWarpsPerSm = 8;

int queryBlocks(int count, int lanes)
{
    const int per_block = kBlock / 32 * lanes;
    return (count + per_block - 1) / per_block;
}

// Launches `kernel` over `blocks` blocks with a STACK-entry shared-memory stack
// of ENTRY-byte entries.
template <int STACK, int ENTRY = static_cast<int>(sizeof(unsigned)), typename Kernel, typename... Args>
cudaError_t launchStacked(Kernel kernel, int blocks, cudaStream_t stream, Args... args)
{
    if (blocks == 0) {
        return cudaSuccess;
    }
    const cudaError_t e = allowStackMemory(kernel, STACK, ENTRY);
    if (e != cudaSuccess) {
        return e;
    }
    kernel<<<blocks, kBlock, stackBytes(STACK, ENTRY), stream>>>(args...);
    return cudaGetLastError();
}

} // namespace

cudaError_t launchMegakernelCounting(const DevScene& scene, const DevCamera& camera, const RenderArgs& render,
                                     PixelAccum* accum, unsigned int* error_flag, int stack_capacity,
                                     unsigned long long* totals, cudaStream_t stream)
{
    RenderArgs args = render;
    args.warp_pixels = 32;
    return withStack(stack_capacity, [&](auto size) {
        constexpr int S = decltype(size)::value;
        return launchStacked<S, kCountEntry>(megakernel<S, kEstimatorPath, true>, megaBlocks(args), stream, scene, camera, args,
                                accum, error_flag, totals);
    });
}

int stackCapacityFor(std::uint32_t stack_need)
{
    if (stack_need <= 32u) {
        return 32;
    }
    if (stack_need <= 48u) {
        return 48;
    }
    if (stack_need <= 64u) {
        return 64;
    }
    return 0;
}

// Path-estimator megakernel of the shape `args` names: blocks_per_sm 3 (state
// in registers) or 4 (lean: state in shared memory), and how its traversal is placed (inline_traversal).
template <int S, int ACC>
cudaError_t launchPathMegakernel(const DevScene& scene, const DevCamera& camera, const RenderArgs& args,
                                 PixelAccum* accum, unsigned int* error_flag, cudaStream_t stream)
{
    unsigned long long* no_totals = nullptr;
    const int blocks = megaBlocks(args);
    if (args.blocks_per_sm == 4) {
        if (args.inline_traversal == 1) {
            return launchStacked<S>(megakernel<S, kEstimatorPath, false, 4, ACC, 1, true>, blocks, stream,
                                            scene, camera, args, accum, error_flag, no_totals);
        }
        return launchStacked<S>(megakernel<S, kEstimatorPath, false, 4, ACC, 0, true>, blocks, stream, scene,
                                        camera, args, accum, error_flag, no_totals);
    }
    if (args.inline_traversal == 1) {
        return launchStacked<S>(megakernel<S, kEstimatorPath, false, kMegaBlocksPerSm, ACC, 1>, blocks, stream, scene,
                                camera, args, accum, error_flag, no_totals);
    }
    if (args.inline_traversal == 2) {
        return launchStacked<S>(megakernel<S, kEstimatorPath, false, kMegaBlocksPerSm, ACC, 2>, blocks, stream, scene,
                                camera, args, accum, error_flag, no_totals);
    }
    return launchStacked<S>(megakernel<S, kEstimatorPath, false, kMegaBlocksPerSm, ACC>, blocks, stream, scene, camera,
                            args, accum, error_flag, no_totals);
}

cudaError_t launchMegakernel(const DevScene& scene, const DevCamera& camera, const RenderArgs& render,
                             PixelAccum* accum, unsigned int* error_flag, int stack_capacity, cudaStream_t stream)
{
    RenderArgs args = render;
    cudaError_t chosen = chooseWarpPixels(scene, args);
    if (chosen == cudaSuccess) {
        chosen = chooseBlocksPerSm(args);
    }
    if (chosen != cudaSuccess) {
        return chosen;
    }
    return withStack(stack_capacity, [&](auto size) {
        constexpr int S = decltype(size)::value;
        unsigned long long* no_totals = nullptr;
        switch (args.estimator) {
        case kEstimatorScatterOnly:
            return launchStacked<S>(megakernel<S, kEstimatorScatterOnly>, megaBlocks(args), stream, scene, camera,
                                    args, accum, error_flag, no_totals);
        case kEstimatorNormals:
            return launchStacked<S>(megakernel<S, kEstimatorNormals>, megaBlocks(args), stream, scene, camera, args,
                                    accum, error_flag, no_totals);
        default:
            if (args.accumulation == kAccumulateKahan) {
                return launchPathMegakernel<S, kAccumulateKahan>(scene, camera, args, accum, error_flag, stream);
            }
            return launchPathMegakernel<S, kAccumulateFp64>(scene, camera, args, accum, error_flag, stream);
        }
    });
}

cudaError_t launchTrace(const DevScene& scene, const float* rays, int count, float t_min, float t_max,
                        const TraceOutputs& out, unsigned int* error_flag, int stack_capacity, cudaStream_t stream)
{
    int lanes = 32;
    if (const cudaError_t e = spreadOver(kQueryWarpsPerSm, count, lanes); e != cudaSuccess) {
        return e;
    }
    return withStack(stack_capacity, [&](auto size) {
        constexpr int S = decltype(size)::value;
        return launchStacked<S>(traceKernel<S>, queryBlocks(count, lanes), stream, scene, rays, count, lanes, t_min,
                                t_max, out, error_flag);
    });
}

cudaError_t launchTraceCounting(const DevScene& scene, const float* rays, int count, float t_min, float t_max,
                                unsigned int* error_flag, int stack_capacity, unsigned long long* totals,
                                cudaStream_t stream)
{
    return withStack(stack_capacity, [&](auto size) {
        constexpr int S = decltype(size)::value;
        return launchStacked<S, kCountEntry>(traceCountKernel<S>, (count + kBlock - 1) / kBlock, stream, scene, rays, count, t_min,
                                t_max, error_flag, totals);
    });
}

cudaError_t launchOccluded(const DevScene& scene, const float* rays, const float* t_max, int count, int* occluded_out,
                           unsigned int* error_flag, int stack_capacity, cudaStream_t stream)
{
    int lanes = 32;
    if (const cudaError_t e = spreadOver(kQueryWarpsPerSm, count, lanes); e != cudaSuccess) {
        return e;
    }
    return withStack(stack_capacity, [&](auto size) {
        constexpr int S = decltype(size)::value;
        return launchStacked<S>(occludedKernel<S>, queryBlocks(count, lanes), stream, scene, rays, t_max, count, lanes,
                                occluded_out, error_flag);
    });
}

} // namespace albedo_b200
