// Batched uneven workload: device structures shared by batch.cu (kernel) and
// batch_api.cu (host object).
#pragma once
#include <algorithm>
#include <vector>

#include "photon_trace.cuh"

namespace sc {

constexpr uint32_t kBatchPrims = 4;
constexpr uint32_t kBatchPlanes = 16;
// Per-warp dirty masks up to this many words live in shared memory (a 1024x1024
// film has 16384 tiles = 512 words); larger films mark their tiles with red.or.
constexpr uint32_t kBatchMaskWords = 512;

// What one warp stages for its current job (byte image copied as 16-byte words).
struct alignas(16) BatchSlotImage {
    PhotonParams p;
    alignas(16) sc_primitive prims[kBatchPrims];
    sc_plane planes[kBatchPlanes];
    sc_material mats[kBatchPrims];
};

struct alignas(16) BatchJobDev {
    BatchSlotImage slot_image;
    uint32_t* flags;
    uint32_t mask_words;
};

struct WorkItem { uint32_t job, begin, count; };

// Appends the work items of photons [begin, begin + count) of job `job` to `out`.
// `left`: photons of the whole launch not yet cut, this job's included; `warps`:
// warps that share the launch.  An item is at most `chunk` photons and at most an
// even share of what is left (half of one while shares are large), but not below
// kMinChunk: large items keep a warp on one film, small ones at the end let the
// warps finish together, and a launch of few photons is spread over all warps.
// Fixed items left most warps idle where there were fewer items than warps.
// Measured against fixed items: 256 scenes, chunk 8192 21.1 -> 19.3 ms; 16 scenes
// of up to 2^20 photons 3.5 -> 0.66 ms; 40 served requests (chunk 2048) 163 -> 122
// ms.  Half shares throughout: 19.3, 0.77, 130; whole ones: 19.6, 0.66, 122.
constexpr uint32_t kMinChunk = 64;
inline void cut_items(std::vector<WorkItem>& out, uint32_t job, uint32_t begin, uint32_t count, uint32_t chunk,
                      uint64_t& left, uint32_t warps) {
    while (count) {
        uint64_t share = left / std::max(warps, 1u) + 31u;
        if (share >= 1024u) share /= 2u;
        const uint32_t n = std::min({count, chunk, std::max(kMinChunk, (uint32_t)std::min<uint64_t>(share, chunk) & ~31u)});
        out.push_back(WorkItem{job, begin, n});
        begin += n;
        count -= n;
        left -= n;
    }
}

// `block`: threads per CTA, 128 or 256 (one shared-memory job slot per warp).
// `ff`: some job uses free-flight sampling (the kernel built with it).
size_t batch_smem(uint32_t mask_words_max, uint32_t block = 256);
int batch_occupancy(int agg, int minb, uint32_t mask_words_max, uint32_t block = 256, bool ff = false);
cudaError_t launch_batch(const BatchJobDev* jobs, const WorkItem* items, uint32_t n_items, uint32_t* counter,
                         const float* cmf, uint32_t mask_words_max, int agg, int minb, uint32_t grid,
                         cudaStream_t s, uint32_t block = 256, bool ff = false);

}  // namespace sc
