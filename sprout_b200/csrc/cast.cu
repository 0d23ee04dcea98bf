// GPU ray cast: closest hit and any hit over the 8-wide quantized BVH built in bvh8.cpp.
//
// Kernel design (sm_100a):
//  * Persistent warps with dynamic ray fetch: each warp keeps 32 rays in flight.  Its lanes walk
//    together (gpu::warp_step) until Refill_threshold of them have finished; those answer their
//    rays and fetch new ones, so lanes stay busy although ray costs differ by orders of magnitude.
//  * A fetched ray is first tested against the tree's padded scene box (gpu::enters_box, in
//    double precision); one that misses it is answered at once, without the 8-child test of the
//    root node.  Where most rays miss it, a second form of the kernel fetches and tests 64 rays
//    at a time with all lanes (choose_kernel).
//  * A batch with at most a ray for each resident lane is dealt out in fixed shares of 32 rays a
//    warp: no work counter, so no memset before the kernel.
//  * Rays are loaded with evict-first hints and results stored with streaming stores, so the
//    512 MiB of benchmark rays do not push the tree (83 MB) out of L2.
//  * Traversal, triangle test and hit definition: traverse.cuh.
//
// What bounds it, and what it measured (B200; before: every lane stepping by itself through
// 80-byte nodes, one launch form).  On 4,194,301 short any-hit rays from the surface of 1,048,576
// triangles 9.8 of 32 lanes were busy and the ALU pipe 70 % (29 warp instructions a step); together
// 18.9 lanes are, the ALU pipe is at 51 %, and what is left is the latency of dependent node loads
// (5.8 stalls an instruction, 31 warps an SM) and L1's one tag look-up a cycle for each lane's line
// (62 % of its rate).  Casts one after another on a stream, us:
//   16,777,216 incoherent closest-hit rays, 1,048,576 triangles: 2,540 -> 1,205
//   those 4,194,301 any-hit rays: 2,600 -> 1,265 (1,300 with a wait after each)
//   360,000 primary rays, 65,536 triangles: 253 -> 125
//   4,099 any-hit rays: 37 -> 23 (38 -> 27 with a wait after each)
// Tried and not kept: ray batches copied to shared memory ahead of use (cp.async, one batch ahead:
// 1,250, 1,360 and 170 us on the first three, for claimed batches wait while other warps run dry);
// the closest hit's barycentrics recomputed at the end instead of carried (1 % slower).
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cstring>
#include <mutex>
#include <string>
#include <type_traits>

#include "bvh8.hpp"
#include "common.hpp"
#include "traverse.cuh"

namespace {

using namespace spb;

// Launch shape: 128-thread blocks, registers bounded so that SPB_CAST_MIN_BLOCKS blocks fit on
// an SM (8: 64 registers, 32 warps; 9 spill in the walk and are 3-12 % slower, 7 are 2-7 % slower
// on the large batches); a warp refills once Refill_threshold of its lanes are idle (4 and 12 are
// 1-4 % slower).
#ifndef SPB_CAST_REFILL
#define SPB_CAST_REFILL 8
#endif
#ifndef SPB_CAST_MIN_BLOCKS
#define SPB_CAST_MIN_BLOCKS 8
#endif
constexpr int      Block            = 128;
constexpr uint32_t Refill_threshold = SPB_CAST_REFILL;
#if SPB_CAST_MIN_BLOCKS > 0
#define SPB_CAST_BOUNDS __launch_bounds__(Block, SPB_CAST_MIN_BLOCKS)
#else
#define SPB_CAST_BOUNDS __launch_bounds__(Block)
#endif
constexpr uint32_t Full_mask        = 0xFFFFFFFFu;
constexpr uint32_t Waiting          = 64;  // rays a warp of the sparse form fetches together

// Counter slots (2 words each: work counter, overflow count).  Slot 0 serves the device
// entry points, slots 1 to 3 the three streams of the host pipeline.
constexpr uint32_t Num_counter_slots = 4;
// After them, one word a slot: the form of kernel its cast takes (choose_kernel).
constexpr uint32_t Num_counter_words = 3 * Num_counter_slots;

// From this many rays on, a cast chooses between the two forms of the kernel.  The choice costs
// two launches (about 8 us); at 2^20 rays a cast takes 70 us or more, and the sparse form saves a
// quarter where it is the better one.
constexpr uint32_t Choose_rays = 1u << 20;
constexpr uint32_t Probes      = 256;

// Answers a ray that misses the scene box.
template <bool Any_hit>
__device__ __forceinline__ void answer_miss(uint32_t i, float t, uint32_t* ids, float* ts, float2* uvs,
                                            uint8_t* occluded) {
    if (Any_hit) {
        __stcs(occluded + i, uint8_t(0));
    } else {
        __stcs(ids + i, gpu::Miss);
        __stcs(ts + i, t);
        if (uvs) {
            __stcs(uvs + i, make_float2(0.f, 0.f));
        }
    }
}

// Chooses the form of a large cast: *sparse = 1 if most of Probes rays spread over the batch miss
// the scene box.  One block of Probes threads.  The sparse form against the dense one, closest hits
// of incoherent rays around 1,048,576 triangles, us at 2^20 / 2^24 rays: 28 % entering 215 / 1,216
// against 232 / 1,617, half 240 / 1,932 against 252 / 2,267, three quarters 275 / 2,822 against
// 274 / 3,009, all 380 / 4,156 against 354 / 4,158 (its queue takes registers from the walk; 4,194,301
// any-hit rays that all enter: 1,320 against 1,265).  Half is thus on the safe side of the line at
// every size.
__global__ void choose_kernel(float4 const* __restrict__ rays, uint32_t num_rays, float3 scene_lo, float3 scene_hi,
                              uint32_t* __restrict__ sparse) {
    uint32_t const i = uint32_t(uint64_t(threadIdx.x) * num_rays / Probes);
    gpu::Ray_state r;
    gpu::Traversal tv;
    gpu::start_ray(r, tv, __ldg(rays + 2 * size_t(i)), __ldg(rays + 2 * size_t(i) + 1));
    int const entering = __syncthreads_count(gpu::enters_box(r, scene_lo, scene_hi));
    if (threadIdx.x == 0) {
        *sparse = 2 * entering < int(Probes) ? 1u : 0u;
    }
}

// Waiting rays from index base on, two a lane: those that enter the scene box are put into the
// warp's queue, the others answered.  Returns how many entered.  Out of line: its registers must
// not add to those of the walk.
template <bool Any_hit>
__device__ __noinline__ uint32_t fetch_sparse(float4 const* rays, uint32_t base, uint32_t num_rays, float3 scene_lo,
                                              float3 scene_hi, uint32_t* queue, uint32_t* ids, float* ts,
                                              float2* uvs, uint8_t* occluded) {
    constexpr uint32_t Each   = Waiting / 32;
    uint32_t const     lane   = threadIdx.x & 31u;
    uint32_t           queued = 0;
    float4             o[Each], d[Each];
#pragma unroll
    for (uint32_t h = 0; h < Each; ++h) {
        size_t const i = min(base + 32 * h + lane, num_rays - 1);
        o[h]           = __ldcs(rays + 2 * i);
        d[h]           = __ldcs(rays + 2 * i + 1);
    }
#pragma unroll
    for (uint32_t h = 0; h < Each; ++h) {
        uint32_t const i     = base + 32 * h + lane;
        bool           enter = false;
        if (i < num_rays) {
            gpu::Ray_state r;
            gpu::Traversal tv;
            gpu::start_ray(r, tv, o[h], d[h]);
            enter = gpu::enters_box(r, scene_lo, scene_hi);
            if (!enter) {
                answer_miss<Any_hit>(i, r.tbest, ids, ts, uvs, occluded);
            }
        }
        uint32_t const mask = __ballot_sync(Full_mask, enter);
        if (enter) {
            queue[queued + __popc(mask & ((1u << lane) - 1u))] = i;
        }
        queued += __popc(mask);
    }
    __syncwarp();
    return queued;
}

// Stats: also count, per ray, the node and triangle steps of its traversal (summed per warp
// into stats[0] and stats[1]); the counting variant is only launched by spb_cast_stats_device.
// work: the work counter, or null for fixed shares.  form (may be null): the form chosen for the
// cast; the other one has nothing to do.
template <bool Any_hit, bool Sparse, bool Stats = false>
__global__ void SPB_CAST_BOUNDS
    cast_kernel(Wide_node const* __restrict__ nodes, float4 const* __restrict__ triangles,
                float4 const* __restrict__ rays, uint32_t num_rays, uint32_t* __restrict__ ids,
                float* __restrict__ ts, float2* __restrict__ uvs, uint8_t* __restrict__ occluded,
                uint32_t* __restrict__ work, uint32_t const* __restrict__ form,
                uint32_t* __restrict__ overflow, float hit_margin,
                float3 scene_lo, float3 scene_hi, unsigned long long* __restrict__ stats) {
    if (form && (*form != 0) != Sparse) {
        return;
    }
    uint32_t const lane = threadIdx.x & 31u;
    uint32_t const lt   = (1u << lane) - 1u;

    gpu::Ray_state r;
    gpu::Traversal tv;
    uint2          stack[gpu::Stack_size];
    uint32_t       ray       = gpu::Miss;  // the lane's ray, until its result is written
    bool           active    = false;
    bool           exhausted = false;
    uint32_t       node_steps = 0;
    uint32_t       tri_steps  = 0;

    // Takes `count` ray indices for the warp.
    auto const take = [&](uint32_t count) {
        uint32_t base = (blockIdx.x * (Block / 32) + threadIdx.x / 32) * 32u;
        if (work) {
            if (lane == 0) {
                base = atomicAdd(work, count);
            }
            base = __shfl_sync(Full_mask, base, 0);
        }
        exhausted = !work || uint64_t(base) + count >= num_rays;
        return base;
    };

    __shared__ uint32_t waiting[Sparse ? Block / 32 : 1][Waiting];
    uint32_t            queued = 0;  // Sparse: the warp's fetched rays that wait for a lane
    while (true) {
        uint32_t idle = __ballot_sync(Full_mask, !active);
        while ((!exhausted || queued != 0) && __popc(idle) >= int(Refill_threshold)) {
            uint32_t const want = __popc(idle);
            if constexpr (Sparse) {
                uint32_t const  rank  = __popc(idle & lt);
                uint32_t* const queue = waiting[threadIdx.x / 32];
                if (queued == 0) {
                    queued = fetch_sparse<Any_hit>(rays, take(Waiting), num_rays, scene_lo, scene_hi, queue, ids, ts,
                                                   uvs, occluded);
                }
                uint32_t const given = min(queued, want);
                if (!active && rank < given) {
                    ray = queue[queued - 1u - rank];
                    gpu::start_ray(r, tv, __ldcs(rays + 2 * size_t(ray)), __ldcs(rays + 2 * size_t(ray) + 1));
                    active = true;
                }
                queued -= given;
                __syncwarp();
            } else {
                uint32_t const i = take(want) + __popc(idle & lt);
                if (!active && i < num_rays) {
                    gpu::start_ray(r, tv, __ldcs(rays + 2 * size_t(i)), __ldcs(rays + 2 * size_t(i) + 1));
                    active = gpu::enters_box(r, scene_lo, scene_hi);
                    if (active) {
                        ray = i;
                    } else {
                        answer_miss<Any_hit>(i, r.tbest, ids, ts, uvs, occluded);
                    }
                }
            }
            idle = __ballot_sync(Full_mask, !active);
        }
        if (idle == Full_mask) {
            break;
        }
        // The lanes walk until enough are idle for a refill, or with no rays left until all are.
        int const floor = exhausted && queued == 0 ? 0 : 32 - int(Refill_threshold);
        do {
            if constexpr (Stats) {
                if (active) {
                    tri_steps += tv.tri_group.y != 0;
                    node_steps += (tv.tri_group.y & (tv.tri_group.y - 1)) == 0 &&
                                  ((tv.group.y & 0xFF000000u) || tv.sp > 0);
                }
            }
            if (gpu::warp_step<Any_hit>(active, r, tv, stack, nodes, triangles, hit_margin, overflow)) {
                active = false;
            }
        } while (__popc(__ballot_sync(Full_mask, active)) > floor);
        if (!active && ray != gpu::Miss) {
            if (Any_hit) {
                __stcs(occluded + ray, uint8_t(r.best_id != gpu::Miss ? 1 : 0));
            } else {
                __stcs(ids + ray, r.best_id);
                __stcs(ts + ray, r.tbest);
                if (uvs) {
                    __stcs(uvs + ray, make_float2(r.u, r.v));
                }
            }
            ray = gpu::Miss;
        }
    }
    if constexpr (Stats) {
        unsigned long long n = node_steps;
        unsigned long long t = tri_steps;
        for (int o = 16; o > 0; o >>= 1) {
            n += __shfl_down_sync(Full_mask, n, o);
            t += __shfl_down_sync(Full_mask, t, o);
        }
        if (lane == 0) {
            atomicAdd(stats + 0, n);
            atomicAdd(stats + 1, t);
        }
    }
}

struct Pipeline {
    static constexpr uint64_t Chunk   = 1ull << 20;  // most rays per chunk
    static constexpr int      Streams = 3;

    cudaStream_t streams[Streams] = {};
    float4*      rays[Streams]    = {};
    uint32_t*    ids[Streams]     = {};
    float*       ts[Streams]      = {};
    float2*      uvs[Streams]     = {};
    uint8_t*     occ[Streams]     = {};
    bool         ready      = false;
};

}  // namespace

struct spb_tree {
    int           device     = 0;
    int           num_sms    = 0;
    int           grid_hit   = 0;
    int           grid_any   = 0;
    spb::Wide_node* d_nodes  = nullptr;
    float4*       d_tris     = nullptr;
    uint32_t*     d_counters = nullptr;
    unsigned long long* d_stats = nullptr;  // node steps, triangle steps (spb_cast_stats_device)
    bool          built      = false;
    float         hit_margin = 0.f;
    float3        scene_lo   = {0.f, 0.f, 0.f};  // Wide_bvh::scene_lo / scene_hi
    float3        scene_hi   = {0.f, 0.f, 0.f};
    spb_tree_info info{};
    Pipeline      pipe;
    cudaStream_t  last_stream = nullptr;
};

namespace {

int32_t cuda_fail(cudaError_t e, char const* what) {
    return spb::fail(SPB_ERROR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

#define SPB_CUDA(call)                          \
    do {                                        \
        cudaError_t const e_ = (call);          \
        if (e_ != cudaSuccess) {                \
            return cuda_fail(e_, #call);        \
        }                                       \
    } while (0)

class Device_scope {
  public:
    explicit Device_scope(int device) {
        cudaGetDevice(&previous_);
        if (previous_ != device) {
            cudaSetDevice(device);
        }
        device_ = device;
    }
    ~Device_scope() {
        if (previous_ != device_) {
            cudaSetDevice(previous_);
        }
    }

  private:
    int previous_ = 0;
    int device_   = 0;
};

void free_pipeline(Pipeline& p) {
    for (int s = 0; s < Pipeline::Streams; ++s) {
        cudaFree(p.rays[s]);
        cudaFree(p.ids[s]);
        cudaFree(p.ts[s]);
        cudaFree(p.uvs[s]);
        cudaFree(p.occ[s]);
        if (p.streams[s]) {
            cudaStreamDestroy(p.streams[s]);
        }
    }
    p = Pipeline();
}

int32_t ensure_pipeline(spb_tree* tree) {
    Pipeline& p = tree->pipe;
    if (p.ready) {
        return SPB_OK;
    }
    for (int s = 0; s < Pipeline::Streams; ++s) {
        SPB_CUDA(cudaStreamCreateWithFlags(&p.streams[s], cudaStreamNonBlocking));
        SPB_CUDA(cudaMalloc(&p.rays[s], Pipeline::Chunk * 32));
        SPB_CUDA(cudaMalloc(&p.ids[s], Pipeline::Chunk * 4));
        SPB_CUDA(cudaMalloc(&p.ts[s], Pipeline::Chunk * 4));
        SPB_CUDA(cudaMalloc(&p.uvs[s], Pipeline::Chunk * 8));
        SPB_CUDA(cudaMalloc(&p.occ[s], Pipeline::Chunk));
    }
    p.ready = true;
    return SPB_OK;
}

// Blocks of a cast of n rays, of at most `full`.  With a ray or less for each of their lanes the
// warps take fixed shares of 32 rays (fixed), otherwise they take rays from the work counter.
int launch_shape(uint32_t n, int full, bool& fixed) {
    uint64_t const need = (uint64_t(n) + Block - 1) / Block;
    fixed               = need <= uint64_t(full);
    return fixed ? int(need) : full;
}

int32_t launch(spb_tree* tree, bool any_hit, uint32_t slot, float4 const* rays, uint32_t n,
               uint32_t* ids, float* ts, float2* uvs, uint8_t* occ, cudaStream_t stream) {
    uint32_t* const counters = tree->d_counters + 2 * slot;
    bool            fixed    = false;
    int const       grid     = launch_shape(n, any_hit ? tree->grid_any : tree->grid_hit, fixed);
    uint32_t* const work     = fixed ? nullptr : counters;
    if (work) {
        SPB_CUDA(cudaMemsetAsync(work, 0, sizeof(uint32_t), stream));
    }
    auto const cast = [&](auto Any_hit, auto Sparse, uint32_t const* form) {
        cast_kernel<decltype(Any_hit)::value, decltype(Sparse)::value><<<grid, Block, 0, stream>>>(
            tree->d_nodes, tree->d_tris, rays, n, ids, ts, uvs, occ, work, form, counters + 1, tree->hit_margin,
            tree->scene_lo, tree->scene_hi, nullptr);
    };
    uint32_t const* form = nullptr;
    // (The sparse form takes more rays at a time than a fixed share holds: it needs the counter.)
    if (work && n >= Choose_rays) {
        uint32_t* const chosen = tree->d_counters + 2 * Num_counter_slots + slot;
        choose_kernel<<<1, Probes, 0, stream>>>(rays, n, tree->scene_lo, tree->scene_hi, chosen);
        form = chosen;
        any_hit ? cast(std::true_type(), std::true_type(), form) : cast(std::false_type(), std::true_type(), form);
    }
    any_hit ? cast(std::true_type(), std::false_type(), form) : cast(std::false_type(), std::false_type(), form);
    SPB_CUDA(cudaGetLastError());
    return SPB_OK;
}

void release_device(spb_tree* tree) {
    cudaFree(tree->d_nodes);
    cudaFree(tree->d_tris);
    tree->d_nodes = nullptr;
    tree->d_tris  = nullptr;
    tree->built   = false;
}

}  // namespace

extern "C" SPB_API int32_t spb_tree_create(spb_tree** out) {
    spb::clear_error();
    if (!out) {
        return spb::fail(SPB_ERROR_ARGUMENT, "spb_tree_create: out is null");
    }
    *out = nullptr;
    auto* tree = new spb_tree;
    cudaError_t e = cudaGetDevice(&tree->device);
    if (e == cudaSuccess) {
        e = cudaDeviceGetAttribute(&tree->num_sms, cudaDevAttrMultiProcessorCount, tree->device);
    }
    int per_sm_hit = 0;
    int per_sm_any = 0;
    if (e == cudaSuccess) {
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_hit, cast_kernel<false, false>, Block,
                                                          0);
    }
    if (e == cudaSuccess) {
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_any, cast_kernel<true, false>, Block,
                                                          0);
    }
    if (e == cudaSuccess) {
        e = cudaMalloc(&tree->d_counters, Num_counter_words * sizeof(uint32_t));
    }
    if (e == cudaSuccess) {
        e = cudaMemset(tree->d_counters, 0, Num_counter_words * sizeof(uint32_t));
    }
    if (e == cudaSuccess) {
        e = cudaMalloc(&tree->d_stats, 2 * sizeof(unsigned long long));
    }
    if (e != cudaSuccess) {
        cudaFree(tree->d_stats);
        cudaFree(tree->d_counters);
        delete tree;
        return cuda_fail(e, "spb_tree_create");
    }
    tree->grid_hit = std::max(1, per_sm_hit) * tree->num_sms;
    tree->grid_any = std::max(1, per_sm_any) * tree->num_sms;
    *out           = tree;
    return SPB_OK;
}

extern "C" SPB_API int32_t spb_tree_release(spb_tree* tree) {
    spb::clear_error();
    if (!tree) {
        return spb::fail(SPB_ERROR_ARGUMENT, "spb_tree_release: tree is null");
    }
    {
        Device_scope scope(tree->device);
        cudaDeviceSynchronize();
        release_device(tree);
        free_pipeline(tree->pipe);
        cudaFree(tree->d_counters);
        cudaFree(tree->d_stats);
    }
    delete tree;
    return SPB_OK;
}

extern "C" SPB_API int32_t spb_tree_build(spb_tree* tree, uint32_t num_vertices,
                                          uint32_t num_triangles, float const* positions,
                                          uint32_t const* indices, uint32_t num_threads) {
    spb::clear_error();
    if (!tree || !positions || !indices) {
        return spb::fail(SPB_ERROR_ARGUMENT, "spb_tree_build: null argument");
    }
    if (num_triangles == 0 || num_vertices == 0) {
        return spb::fail(SPB_ERROR_ARGUMENT, "spb_tree_build: empty mesh");
    }
    Device_scope scope(tree->device);

    auto const     t0 = std::chrono::steady_clock::now();
    spb::Wide_bvh  bvh;
    std::string    error;
    if (!spb::build_wide_bvh(num_vertices, num_triangles, positions, indices,
                             spb::resolve_threads(num_threads), bvh, error)) {
        return spb::fail(SPB_ERROR_ARGUMENT, "spb_tree_build: %s", error.c_str());
    }

    SPB_CUDA(cudaDeviceSynchronize());
    release_device(tree);
    size_t const node_bytes = bvh.nodes.size() * sizeof(spb::Wide_node);
    size_t const tri_bytes  = bvh.triangles.size() * sizeof(spb::Wide_triangle);
    SPB_CUDA(cudaMalloc(&tree->d_nodes, node_bytes));
    SPB_CUDA(cudaMalloc(&tree->d_tris, tri_bytes));
    SPB_CUDA(cudaMemcpy(tree->d_nodes, bvh.nodes.data(), node_bytes, cudaMemcpyHostToDevice));
    SPB_CUDA(cudaMemcpy(tree->d_tris, bvh.triangles.data(), tri_bytes, cudaMemcpyHostToDevice));

    auto const t1 = std::chrono::steady_clock::now();

    tree->info.num_triangles = num_triangles;
    tree->info.num_nodes     = uint32_t(bvh.nodes.size());
    tree->info.num_leaves    = bvh.num_leaves;
    tree->info.max_depth     = bvh.max_depth;
    tree->info.device_bytes  = node_bytes + tri_bytes;
    tree->info.build_seconds = std::chrono::duration<double>(t1 - t0).count();
    tree->info.sah_cost      = bvh.sah_cost;
    tree->hit_margin         = bvh.hit_margin;
    tree->scene_lo           = make_float3(bvh.scene_lo[0], bvh.scene_lo[1], bvh.scene_lo[2]);
    tree->scene_hi           = make_float3(bvh.scene_hi[0], bvh.scene_hi[1], bvh.scene_hi[2]);
    tree->built              = true;
    return SPB_OK;
}

extern "C" SPB_API int32_t spb_tree_info_get(spb_tree const* tree, spb_tree_info* info) {
    spb::clear_error();
    if (!tree || !info) {
        return spb::fail(SPB_ERROR_ARGUMENT, "spb_tree_info_get: null argument");
    }
    *info = tree->info;
    return SPB_OK;
}

namespace {

int32_t check_cast(spb_tree* tree, float const* rays, uint64_t n, bool outputs_ok,
                   char const* who) {
    if (!tree) {
        return spb::fail(SPB_ERROR_ARGUMENT, "%s: tree is null", who);
    }
    if (!tree->built) {
        return spb::fail(SPB_ERROR_STATE, "%s: tree has not been built", who);
    }
    if (n > SPB_MAX_RAYS_PER_CALL) {
        return spb::fail(SPB_ERROR_ARGUMENT, "%s: %llu rays exceed the per-call limit", who,
                         (unsigned long long)n);
    }
    if (n > 0 && (!rays || !outputs_ok)) {
        return spb::fail(SPB_ERROR_ARGUMENT, "%s: null buffer", who);
    }
    return SPB_OK;
}

}  // namespace

extern "C" SPB_API int32_t spb_intersect_device(spb_tree* tree, float const* rays,
                                                uint64_t num_rays, uint32_t* ids, float* ts,
                                                float* uvs, void* stream) {
    spb::clear_error();
    if (int32_t const s = check_cast(tree, rays, num_rays, ids && ts, "spb_intersect_device")) {
        return s;
    }
    if (num_rays == 0) {
        return SPB_OK;
    }
    Device_scope scope(tree->device);
    tree->last_stream = static_cast<cudaStream_t>(stream);
    return launch(tree, false, 0, reinterpret_cast<float4 const*>(rays), uint32_t(num_rays), ids,
                  ts, reinterpret_cast<float2*>(uvs), nullptr, tree->last_stream);
}

extern "C" SPB_API int32_t spb_intersect_p_device(spb_tree* tree, float const* rays,
                                                  uint64_t num_rays, uint8_t* occluded,
                                                  void* stream) {
    spb::clear_error();
    if (int32_t const s = check_cast(tree, rays, num_rays, occluded != nullptr,
                                     "spb_intersect_p_device")) {
        return s;
    }
    if (num_rays == 0) {
        return SPB_OK;
    }
    Device_scope scope(tree->device);
    tree->last_stream = static_cast<cudaStream_t>(stream);
    return launch(tree, true, 0, reinterpret_cast<float4 const*>(rays), uint32_t(num_rays),
                  nullptr, nullptr, nullptr, occluded, tree->last_stream);
}

extern "C" SPB_API int32_t spb_cast_stats_device(spb_tree* tree, float const* rays,
                                                 uint64_t num_rays, uint32_t* ids, float* ts,
                                                 void* stream, uint64_t* node_steps,
                                                 uint64_t* triangle_steps) {
    spb::clear_error();
    if (int32_t const s = check_cast(tree, rays, num_rays, ids && ts && node_steps && triangle_steps,
                                     "spb_cast_stats_device")) {
        return s;
    }
    if (!node_steps || !triangle_steps) {
        return spb::fail(SPB_ERROR_ARGUMENT, "spb_cast_stats_device: null counter");
    }
    *node_steps     = 0;
    *triangle_steps = 0;
    if (num_rays == 0) {
        return SPB_OK;
    }
    Device_scope       scope(tree->device);
    cudaStream_t const st = static_cast<cudaStream_t>(stream);
    tree->last_stream     = st;
    uint32_t* counters    = tree->d_counters;
    SPB_CUDA(cudaMemsetAsync(counters, 0, sizeof(uint32_t), st));
    SPB_CUDA(cudaMemsetAsync(tree->d_stats, 0, 2 * sizeof(unsigned long long), st));
    uint32_t const n    = uint32_t(num_rays);
    int const      grid = std::max(1, std::min(tree->grid_hit, int((uint64_t(n) + Block - 1) / Block)));
    cast_kernel<false, false, true><<<grid, Block, 0, st>>>(
        tree->d_nodes, tree->d_tris,
        reinterpret_cast<float4 const*>(rays), n, ids, ts, nullptr, nullptr, counters, nullptr,
        counters + 1, tree->hit_margin, tree->scene_lo, tree->scene_hi, tree->d_stats);
    SPB_CUDA(cudaGetLastError());
    unsigned long long host[2] = {0, 0};
    SPB_CUDA(cudaMemcpyAsync(host, tree->d_stats, sizeof(host), cudaMemcpyDeviceToHost, st));
    SPB_CUDA(cudaStreamSynchronize(st));
    *node_steps     = host[0];
    *triangle_steps = host[1];
    return SPB_OK;
}

namespace {

// Whether host memory is page-locked or otherwise known to CUDA (copies from and to other memory,
// pageable, are not asynchronous).
bool page_locked(void const* p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type != cudaMemoryTypeUnregistered;
}

int32_t cast_host(spb_tree* tree, bool any_hit, float const* rays, uint64_t n, uint32_t* ids,
                  float* ts, float* uvs, uint8_t* occ) {
    Device_scope scope(tree->device);
    if (int32_t const s = ensure_pipeline(tree)) {
        return s;
    }
    Pipeline& p = tree->pipe;
    // Chunks, so that the copies in, the casts and the copies out overlap.  From page-locked memory
    // an eighth of the batch at a time: the call then takes little more than its copies in.  Chunks
    // below 65,536 rays would not fill the GPU.  Three streams: with two, a chunk's copy in waits for
    // the copy out before last.  (1,000,003 rays, 262,144 triangles: 997 us in one chunk, 763 in
    // eight.)
    //
    // Copies to and from pageable memory keep the calling thread, so rays in such memory are cast in
    // halves of at least 131,072 (each further chunk costs more than the cast it hides: 2,520 us in
    // eighths, 2,150 in halves, 2,210 in one chunk), and a chunk's results go out to such memory only
    // when the next chunk's cast is under way (lag), or the thread would wait for the cast as well.
    // Eighths without lag, as from page-locked memory, -> this: closest hits of 1,000,003 pageable rays
    // 3,300 -> 2,100 us, of 300,000 1,200 -> 680; of page-locked rays to pageable results 2,090 -> 1,260
    // and 930 -> 520 us.
    uint64_t chunk = n;
    uint64_t lag   = 0;
    if (n > 65536) {
        bool const     locked = page_locked(rays);
        uint64_t const parts  = locked ? 8 : 2;
        uint64_t const part   = (n / parts + 32767) / 32768 * 32768;
        chunk                 = std::clamp<uint64_t>(part, locked ? 65536 : 131072, Pipeline::Chunk);
        bool const results    = any_hit ? page_locked(occ)
                                        : page_locked(ids) && page_locked(ts) && (!uvs || page_locked(uvs));
        lag                   = results ? 0 : 1;
    }
    auto const copy_out = [&](uint64_t c) -> int32_t {
        int const          s     = int(c % Pipeline::Streams);
        uint64_t const     first = c * chunk;
        uint64_t const     count = std::min<uint64_t>(chunk, n - first);
        cudaStream_t const st    = p.streams[s];
        if (any_hit) {
            SPB_CUDA(cudaMemcpyAsync(occ + first, p.occ[s], count, cudaMemcpyDeviceToHost, st));
            return SPB_OK;
        }
        SPB_CUDA(cudaMemcpyAsync(ids + first, p.ids[s], count * 4, cudaMemcpyDeviceToHost, st));
        SPB_CUDA(cudaMemcpyAsync(ts + first, p.ts[s], count * 4, cudaMemcpyDeviceToHost, st));
        if (uvs) {
            SPB_CUDA(cudaMemcpyAsync(uvs + 2 * first, p.uvs[s], count * 8, cudaMemcpyDeviceToHost, st));
        }
        return SPB_OK;
    };
    uint64_t const chunks = (n + chunk - 1) / chunk;
    for (uint64_t c = 0; c < chunks + lag; ++c) {
        if (c < chunks) {
            int const          s     = int(c % Pipeline::Streams);
            uint64_t const     first = c * chunk;
            uint64_t const     count = std::min<uint64_t>(chunk, n - first);
            cudaStream_t const st    = p.streams[s];
            SPB_CUDA(cudaMemcpyAsync(p.rays[s], rays + 8 * first, count * 32, cudaMemcpyHostToDevice, st));
            if (int32_t const r = launch(tree, any_hit, 1 + uint32_t(s), p.rays[s], uint32_t(count), p.ids[s],
                                         p.ts[s], uvs ? p.uvs[s] : nullptr, p.occ[s], st)) {
                return r;
            }
        }
        if (c >= lag) {
            if (int32_t const r = copy_out(c - lag)) {
                return r;
            }
        }
    }
    for (cudaStream_t const st : p.streams) {
        SPB_CUDA(cudaStreamSynchronize(st));
    }
    tree->last_stream = p.streams[Pipeline::Streams - 1];
    return SPB_OK;
}

}  // namespace

extern "C" SPB_API int32_t spb_intersect_host(spb_tree* tree, float const* rays,
                                              uint64_t num_rays, uint32_t* ids, float* ts,
                                              float* uvs) {
    spb::clear_error();
    if (int32_t const s = check_cast(tree, rays, num_rays, ids && ts, "spb_intersect_host")) {
        return s;
    }
    if (num_rays == 0) {
        return SPB_OK;
    }
    return cast_host(tree, false, rays, num_rays, ids, ts, uvs, nullptr);
}

extern "C" SPB_API int32_t spb_intersect_p_host(spb_tree* tree, float const* rays,
                                                uint64_t num_rays, uint8_t* occluded) {
    spb::clear_error();
    if (int32_t const s = check_cast(tree, rays, num_rays, occluded != nullptr,
                                     "spb_intersect_p_host")) {
        return s;
    }
    if (num_rays == 0) {
        return SPB_OK;
    }
    return cast_host(tree, true, rays, num_rays, nullptr, nullptr, nullptr, occluded);
}

extern "C" SPB_API int32_t spb_tree_status(spb_tree* tree, uint32_t* overflowed_rays) {
    spb::clear_error();
    if (!tree || !overflowed_rays) {
        return spb::fail(SPB_ERROR_ARGUMENT, "spb_tree_status: null argument");
    }
    Device_scope scope(tree->device);
    SPB_CUDA(cudaDeviceSynchronize());
    uint32_t host[2 * Num_counter_slots];
    SPB_CUDA(cudaMemcpy(host, tree->d_counters, sizeof(host), cudaMemcpyDeviceToHost));
    *overflowed_rays = 0;
    for (uint32_t slot = 0; slot < Num_counter_slots; ++slot) {
        *overflowed_rays += host[2 * slot + 1];
    }
    return SPB_OK;
}

// ---- Closest hit without any device allocation ------------------------------------------
//
// Some callers cannot call cudaMalloc: a cudaMalloc may synchronize the whole device and may
// fail once device memory is exhausted, so a frame loop with a fixed time budget, or a host
// application whose own allocator owns all device memory, must not allocate on the way to a
// cast.  spb_intersect_host allocates device staging buffers on its first call;
// spb_intersect_host_static instead stages rays and results in the file-scope array below,
// which every GPU that loads this library holds until the process exits.

namespace {

constexpr uint64_t Static_max_rays      = SPB_STATIC_MAX_RAYS;
constexpr size_t   Static_counter_bytes = 256;  // work counter, padded
constexpr size_t   Static_scratch_bytes = Static_counter_bytes + Static_max_rays * (32 + 4 + 4);
constexpr int      Static_max_devices   = 64;

__device__ __align__(256) unsigned char g_static_scratch[Static_scratch_bytes];

// The array's device address per device, with the id of the CUDA context it was looked up in:
// a context created after a cudaDeviceReset may place the array elsewhere, so the address is
// looked up again whenever the current context's id differs from the cached one.
struct Static_address {
    unsigned char*     address    = nullptr;
    unsigned long long context_id = 0;
};

std::mutex     g_static_mutex;
Static_address g_static_address[Static_max_devices];

using Ctx_get_current = CUresult(CUDAAPI*)(CUcontext*);
using Ctx_get_id      = CUresult(CUDAAPI*)(CUcontext, unsigned long long*);

// Id of the calling thread's current context (0 if the driver cannot tell, in which case the
// address is looked up on every call).
unsigned long long current_context_id() {
    static Ctx_get_current get_current = nullptr;
    static Ctx_get_id      get_id      = nullptr;
    static bool const      resolved    = [] {
        void* a = nullptr;
        void* b = nullptr;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &a, cudaEnableDefault) == cudaSuccess &&
            cudaGetDriverEntryPoint("cuCtxGetId", &b, cudaEnableDefault) == cudaSuccess) {
            get_current = reinterpret_cast<Ctx_get_current>(a);
            get_id      = reinterpret_cast<Ctx_get_id>(b);
        }
        return true;
    }();
    (void)resolved;
    CUcontext          ctx = nullptr;
    unsigned long long id  = 0;
    if (get_current && get_id && get_current(&ctx) == CUDA_SUCCESS && ctx &&
        get_id(ctx, &id) == CUDA_SUCCESS) {
        return id;
    }
    return 0;
}

// Device address of g_static_scratch on the current device, looked up once per device and
// context (the host-side symbol g_static_scratch itself is not a device address).
int32_t static_scratch(int device, unsigned char** out) {
    if (device < 0 || device >= Static_max_devices) {
        return spb::fail(SPB_ERROR_STATE, "spb_intersect_host_static: device %d not supported",
                         device);
    }
    unsigned long long const    context = current_context_id();
    std::lock_guard<std::mutex> lock(g_static_mutex);
    Static_address&             cached = g_static_address[device];
    if (!cached.address || context == 0 || cached.context_id != context) {
        void*             ptr = nullptr;
        cudaError_t const e   = cudaGetSymbolAddress(&ptr, g_static_scratch);
        if (e != cudaSuccess) {
            return cuda_fail(e, "cudaGetSymbolAddress(g_static_scratch)");
        }
        cached.address    = static_cast<unsigned char*>(ptr);
        cached.context_id = context;
    }
    *out = cached.address;
    return SPB_OK;
}

}  // namespace

extern "C" SPB_API int32_t spb_intersect_host_static(spb_tree* tree, float const* rays,
                                                     uint64_t num_rays, uint32_t* ids,
                                                     float* ts) {
    spb::clear_error();
    if (int32_t const s = check_cast(tree, rays, num_rays, ids && ts,
                                     "spb_intersect_host_static")) {
        return s;
    }
    if (num_rays > Static_max_rays) {
        return spb::fail(SPB_ERROR_ARGUMENT,
                         "spb_intersect_host_static: %llu rays exceed the static scratch limit "
                         "of %llu rays per call",
                         (unsigned long long)num_rays, (unsigned long long)Static_max_rays);
    }
    if (num_rays == 0) {
        return SPB_OK;
    }
    Device_scope scope(tree->device);
    unsigned char* base = nullptr;
    if (int32_t const s = static_scratch(tree->device, &base)) {
        return s;
    }
    auto* work   = reinterpret_cast<uint32_t*>(base);
    auto* d_rays = reinterpret_cast<float4*>(base + Static_counter_bytes);
    auto* d_ids  = reinterpret_cast<uint32_t*>(base + Static_counter_bytes + Static_max_rays * 32);
    auto* d_ts   = reinterpret_cast<float*>(base + Static_counter_bytes + Static_max_rays * 36);
    uint32_t const n = uint32_t(num_rays);

    // The array keeps the previous call's contents: the work counter must start at zero.
    // Stack overflows (none for trees this library builds) are counted in the tree's own
    // counter, as spb_intersect_host counts them, and reported by spb_tree_status.
    bool      fixed = false;
    int const grid  = launch_shape(n, tree->grid_hit, fixed);
    if (!fixed) {
        SPB_CUDA(cudaMemsetAsync(work, 0, sizeof(uint32_t), nullptr));
    }
    SPB_CUDA(cudaMemcpyAsync(d_rays, rays, size_t(n) * 32, cudaMemcpyHostToDevice, nullptr));
    cast_kernel<false, false><<<grid, Block, 0, nullptr>>>(tree->d_nodes,
                                                    tree->d_tris, d_rays, n, d_ids, d_ts, nullptr,
                                                    nullptr, fixed ? nullptr : work, nullptr, tree->d_counters + 1,
                                                    tree->hit_margin, tree->scene_lo, tree->scene_hi, nullptr);
    SPB_CUDA(cudaGetLastError());
    SPB_CUDA(cudaMemcpyAsync(ids, d_ids, size_t(n) * 4, cudaMemcpyDeviceToHost, nullptr));
    SPB_CUDA(cudaMemcpyAsync(ts, d_ts, size_t(n) * 4, cudaMemcpyDeviceToHost, nullptr));
    SPB_CUDA(cudaStreamSynchronize(nullptr));
    return SPB_OK;
}
