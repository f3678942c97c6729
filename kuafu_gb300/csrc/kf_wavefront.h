// kf_wavefront.h — device data views and kernel launchers of the wavefront path tracer.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "kf_device.cuh"

namespace kf {

constexpr int kMaxLightSlots = 1 + KF_MAX_POINT_LIGHTS + KF_MAX_ACTIVE_LIGHTS; // 41

// Everything a kernel needs to read about one scene (device pointers).
struct SceneDev {
    const float4* verts;             // 3 float4 per vertex (kf_vertex, 48 B)
    const uint32_t* indices;         // 3 per triangle, geometry-local vertex indices
    const uint32_t* matidx;          // material index per triangle
    const uint4* geom;               // per geometry {vertex_offset, tri_offset, num_tris, flags}
    const kf_material_gpu* materials;
    const InstanceRec* inst;
    const Node4* blas_nodes;
    const Tri* tris;
    const Node4* tlas_nodes;
    const uint32_t* tlas_inst;
    const kf_dir_light_ubo* dlight;
    const kf_point_lights_ubo* plights;
    const kf_active_lights_ubo* alights;
    const uint4* tex_info;           // per texture {texel offset, width, height, srgb}
    const uchar4* texels;
    const float* srgb_decode;        // 256 entries
    const float4* env;               // environment cube map: 6 faces of env_size^2 texels (null = none)
    uint32_t env_size;
    uint32_t num_instances;
    uint32_t has_tlas;
    uint32_t num_textures;
    uint32_t num_slots;              // shadow-ray light slots in use
    uint8_t slot_group[kMaxLightSlots]; // 0 directional, 1 point, 2 active
    uint8_t slot_index[kMaxLightSlots];
};

// Per-frame constants, resident in device memory so a captured graph can replay them.
struct FrameDev {
    kf_camera_ubo cam;
    kf_push_constants pc;
    uint32_t width, height, npix, seed;
    uint32_t frame, camera_index, pad0, pad1;
};

constexpr uint32_t kNoRoot = 0xFFFFFFFFu;

// One view of a batched launch: its frame constants, where its paths start in the
// batch's path space, and what of its scene the kernels need beyond the shared
// (concatenated) geometry / BVH pools: TLAS root, light slots, environment, AOVs.
struct ItemDev {
    FrameDev f;
    uint64_t path_start;
    uint32_t block_start;     // first block of the item in the batched resolve (kResolvePix pixels each)
    uint32_t spp;
    uint32_t root;            // TLAS root node in the batch's node pool (kNoRoot: nothing to hit)
    uint32_t num_slots;
    uint8_t slot_group[kMaxLightSlots];
    uint8_t slot_index[kMaxLightSlots];
    uint16_t pad;
    const kf_dir_light_ubo* dlight;
    const kf_point_lights_ubo* plights;
    const kf_active_lights_ubo* alights;
    const float4* env;
    uint32_t env_size;
    uint32_t inst_base;       // first instance of the item's scene in the batch's instance pool
    uint32_t geom_base;       // first geometry of the item's scene in the batch's geometry pool
    uint32_t pad3;
    float4* albedo;
    float4* normal;
    float* depth;
    uint4* seg;
    float4* accum;            // resolve targets
    dbl4* sum64;
    uchar4* bgra;
};

// Batch description handed to the kernels (items == nullptr: a single-view frame).
struct BatchDev {
    const ItemDev* items;
    uint32_t num_items;
    uint32_t pad;
};

// Counters of one bounce, cleared once per chunk for all its bounces: a row per depth, so that
// no launch waits for a clear between bounces.
constexpr int kCounterRow = 8; // [0] rays queued, [1] rays that hit, [2] / [3] fetch cursors (closest / shadow),
                               // [4] finished blocks of k_paths
constexpr int kSlotRow = 64;   // shadow rays queued per light slot

// Per-chunk wavefront state. A path's number within its view is pixel * spp + sample: a pixel's
// samples are neighbours in the radiance buffer as they are in the ray queues, so a warp's
// radiance accesses fall into a few lines. Everything a bounce hands from kernel to kernel is
// stored in queue order (rays) or hit-list order (hits) and read coalesced. Before, throughput,
// radiance, requests, contributions and visibility were indexed by a sample-major path number,
// which put a warp's 32 accesses into 32 lines: a Cornell room of 256 x 256 at 64 spp takes 3.49
// instead of 4.57 ms (no NEE there: its three kernels and records, a quarter of that frame, are
// skipped), the 256-icosphere frame at 1080p, 8 spp, 21.8 instead of 22.7 ms.
struct WaveDev {
    float4* q_o[2];       // ray queue: origin.xyz + path id bits
    float4* q_d[2];       // ray queue: direction.xyz + throughput.x
    float2* q_w[2];       // ray queue: throughput.yz (not written for camera rays: 1)
    uint32_t* counters;   // kCounterRow words per depth
    float4* hit;          // t, u, v, primitive bits
    uint32_t* hit_inst;   // instance, or all ones on a miss (apart: k_miss reads this word of every ray only)
    uint32_t* sel;        // queue positions of this bounce's rays that hit
    uint32_t* scount;     // kSlotRow words per depth: slot j's shadow rays, at sq_o/sq_d[j * chunk_cap + k]
    uint32_t nslot;       // light slots of the launch, each with a shadow queue (scount entries)
    uint32_t lit;         // some view of the launch has a light slot (else no NEE is recorded)
    float4* nee_w;        // per hit: throughput that scales this bounce's NEE + path id and flag bits
    float4* nee_in;       // per hit, 5 arrays of chunk_cap: what k_nee needs of k_shade's shading
    uint64_t* req;        // per hit: shadow slots requested this bounce (bit j = slot j)
    float4* contrib;      // [slot][hit] light contribution
    uint8_t* vis;         // [slot][hit] 1 = unoccluded
    float4* sq_o;         // shadow queue: origin.xyz + tmax
    float4* sq_d;         // shadow queue: direction.xyz + (slot << 26 | hit) bits
    float4* radiance;     // per global path (frame): accumulated `color`
    kf_hit* primary;      // per global path, debug (may be null)
    float4* albedo;       // per pixel AOVs
    float4* normal;
    float* depth;
    uint4* seg;           // per pixel {instance, geometry, material, primitive} of sample 0's first hit
    unsigned long long* stats; // [0] primary, [1] extension, [2] shadow, [3] nodes, [4] tris, [5] inst
    uint16_t* path_item;       // batched launch: item of each path of the chunk
    uint16_t* hit_item;        // batched launch: item of each hit
    uint32_t chunk_cap;
    uint32_t pad; // no padding bytes: a captured launch is known by this struct's
};

// Every launcher takes the batch description b: b.items == nullptr renders the single
// view of f with the scene's own TLAS and lights; otherwise f is unused and each path
// takes its frame constants, TLAS root, lights and AOV targets from its item.
void launch_raygen(const FrameDev* f, const BatchDev& b, const WaveDev& w, uint64_t chunk_start, uint32_t chunk_n,
                   cudaStream_t st);
// Every path of a launch of n paths (one chunk), from raygen to the end of the path. sms: SMs of
// the GPU. The wavefront is faster from more than kPathsMax paths on, or kPathsMaxLit where some
// view has lights to sample.
constexpr uint64_t kPathsMax = 163840, kPathsMaxLit = 16384;
void launch_paths(const SceneDev& s, const FrameDev* f, const BatchDev& b, const WaveDev& w, uint32_t n,
                  uint32_t max_depth, uint32_t sms, cudaStream_t st);
// The rest of every path of bounce `depth` of a chunk (its closest hits found, the NEE of the
// bounces before gathered), if there are few enough of them; the bounce's queue is then empty.
void launch_tail(const SceneDev& s, const FrameDev* f, const BatchDev& b, const WaveDev& w, int cur, uint32_t depth,
                 uint64_t chunk_start, uint32_t max_depth, uint32_t sms, cudaStream_t st);
void launch_extend(const SceneDev& s, const FrameDev* f, const BatchDev& b, const WaveDev& w, int cur,
                   uint32_t depth, uint64_t chunk_start, uint32_t grid, bool count_mode, cudaStream_t st);
// k_miss ends the paths whose ray missed and lists the others in w.sel; k_shade shades those.
void launch_shade(const SceneDev& s, const FrameDev* f, const BatchDev& b, const WaveDev& w, int cur,
                  uint32_t depth, uint64_t chunk_start, uint32_t grid, cudaStream_t st);
void launch_miss(const SceneDev& s, const FrameDev* f, const BatchDev& b, const WaveDev& w, int cur,
                 uint32_t depth, uint64_t chunk_start, uint32_t grid, cudaStream_t st);
// Light samples (shadow queues, contributions, NEE requests) of the hits k_shade shaded.
void launch_nee(const SceneDev& s, const FrameDev* f, const BatchDev& b, const WaveDev& w, uint32_t depth,
                uint64_t chunk_start, uint32_t grid, cudaStream_t st);
void launch_shadow(const SceneDev& s, const BatchDev& b, const WaveDev& w, uint32_t depth, uint32_t grid,
                   bool count_mode, cudaStream_t st);
// Persistent traversal with dynamic ray fetch (closest hit, or shadow rays when `shadow`).
// refill_below (1..32) and steps (1..64): the warp scheduling of the persistent kernel.
void launch_trace_dyn(const SceneDev& s, const FrameDev* f, const BatchDev& b, const WaveDev& w, int cur,
                      uint32_t depth, uint64_t chunk_start, bool shadow, uint32_t grid, bool count_mode,
                      uint32_t refill_below, uint32_t steps, cudaStream_t st);
// resident blocks per SM of the persistent traversal kernel's variants: shadow rays, camera rays
// (depth 0) and later closest-hit rays
// rays a block of it takes at least (a launch has no more blocks than that gives work)
constexpr uint32_t kTraceMinBlockRays = 16;
enum class TraceKind { shadow, camera, bounce };
uint32_t trace_dyn_blocks_per_sm(TraceKind kind);
void launch_gather(const SceneDev& s, const BatchDev& b, const WaveDev& w, uint32_t depth, uint64_t chunk_start,
                   uint32_t grid, cudaStream_t st);
// Per-pixel mean, running mean, FP64 sum and the BGRA frame of one view.
constexpr uint32_t kResolvePix = 256; // pixels per block
void launch_resolve(const FrameDev* f, const float4* radiance, uint32_t npix, uint32_t spp, float4* accum,
                    dbl4* sum64, uchar4* bgra, cudaStream_t st);
// The same for every view of a batch in one launch (blocks: the items' resolve blocks in all).
void launch_resolve_batch(const BatchDev& b, const float4* radiance, uint32_t blocks, cudaStream_t st);
// Paths first .. first + n - 1 of a per-path buffer (`words` float4 each) in sample-major order, as
// downloads have them: dst[k] = src[pix * spp + sample] with sample * npix + pix = first + k.
void launch_sample_major(const float4* src, uint32_t npix, uint32_t spp, uint32_t words, uint64_t first, uint32_t n,
                         float4* dst, cudaStream_t st);
void launch_srgb(const float4* img, uint32_t npix, uchar4* out, cudaStream_t st);
void upload_srgb_thresholds(const float* thresh256);
void launch_relmse(const float4* x, const float4* ref, uint64_t n, double eps, double* partial, uint32_t blocks,
                   double* out, cudaStream_t st);

} // namespace kf
