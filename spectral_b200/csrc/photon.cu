// Forward photon emitter / tracer with point-estimator haze splatting.
//
// One photon per lane, in groups (photon_trace.cuh), restating render_volumetric_scene_point
// (spectral-core/src/volume.rs:99-168) and its GPU mirror
// (spectral-gpu/src/shaders/volume.wgsl:542-647): emission from the beam
// aperture, hero wavelength, up to max_bounces segments, 4 uniform haze samples
// per segment connected to the camera (HG phase x transmittance / d^2), then the
// Fresnel / refract / TIR scatter at the hit.  The RNG stream is consumed in
// exactly the reference order, so paths are bit-identical to the CPU crate.
//
// Splats land in a 64-bit fixed-point film with red.global.add.u64; the film is
// tile-major (8x8 pixel tiles) and every touched tile raises a dirty flag so the
// drain/reduce pass reads only tiles that received light.
#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>
#include <set>
#include <tuple>
#include <utility>

#include "photon_trace.cuh"

namespace sc {

namespace {

// Byte offset of the warps' parked photons: after scene records, CMF table and
// the dirty mask, rounded up to 16 bytes.
__host__ __device__ __forceinline__ size_t park_offset(const PhotonParams& p, uint32_t mask_words) {
    const size_t b = p.n_prims * sizeof(sc_primitive) + p.n_planes * sizeof(sc_plane) +
                     p.n_mats * sizeof(sc_material) + 3 * kTableN * sizeof(float) + mask_words * sizeof(uint32_t);
    return (b + 15u) & ~size_t(15);
}

// 256 threads per CTA; MINB CTAs per SM bound the registers (4: 64 registers, spectral
// films without spills, XYZ films with 24 B, with the cache 38 B; 5: 48 registers, 140 B
// and 240 to 300 B, more warps in flight).
// FF: built with free-flight sampling (estimator 3) as well.  EXACT: haze
// samples in the CPU crate's operation order.  CACHE: built with the shared-memory
// cell cache.  chunk: photons of each warp.  cached: slots of
// the cache, 0: none (CACHE only; launches without it take the kernel without it: XYZ,
// dsotm 640x360, 2^14 photons 32.8 -> 30.3 us, rainbow 25.9 -> 24.0).
template <bool SPEC, int AGG, int MINB, bool FF, bool EXACT = false, bool CACHE = false>
__global__ void __launch_bounds__(256, MINB) photon_kernel(const PhotonParams p, uint32_t mask_words, uint32_t chunk,
                                                           uint32_t cached) {
    extern __shared__ __align__(16) unsigned char smem[];
    const float* cmf;
    uint32_t* smask;
    const SceneView S = load_scene(p, smem, &cmf, &smask, mask_words);
    CellCacheOf<SPEC> cells(smem + park_offset(p, mask_words) + 8 * sizeof(ParkedPhotons<SPEC>), cached);
    CellCacheOf<SPEC>* cache = CACHE && cached ? &cells : nullptr;
    if (cache) {
        cache->clear();
        __syncthreads();
    }
    // one chunk of the launch's photons per warp; CTAs start in launch order, so
    // the photons in flight stay close in it (the wavelength-ordered dispatch
    // relies on that)
    const uint32_t warp = threadIdx.x >> 5;
    const uint64_t base = (uint64_t)(blockIdx.x * (blockDim.x >> 5) + warp) * chunk;
    if (base < p.photon_count) {
        const uint32_t b0 = (uint32_t)base;
        trace_group_range<SPEC, AGG, FF, true, EXACT>(
            p, S, cmf, min(chunk, p.photon_count - b0),
            [&](uint32_t k) { return p.photon_base + (p.order ? p.order[b0 + k] : b0 + k); }, smask,
            reinterpret_cast<ParkedPhotons<SPEC>*>(smem + park_offset(p, mask_words))[warp], cache);
    }
    if (cache) {
        __syncthreads();
        cache->flush(p.film);
    }
    if (smask) {  // publish this CTA's dirty tiles
        __syncthreads();
        for (uint32_t w = threadIdx.x; w < mask_words; w += blockDim.x)
            if (smask[w]) atomicOr(p.flags + w, smask[w]);
    }
}

// Instrumented pass: same transport, no film writes; sums the per-photon work
// counters into out[0..3] = photons, segments, in-frame samples, scatters.
__global__ void __launch_bounds__(256) photon_count_kernel(const PhotonParams p, unsigned long long* out) {
    extern __shared__ __align__(16) unsigned char smem[];
    const float* cmf;
    const SceneView S = load_scene(p, smem, &cmf);
    unsigned long long seg = 0, spl = 0, sca = 0, ph = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < p.photon_count; i += gridDim.x * blockDim.x) {
        PhotonCounts c = {0u, 0u, 0u};
        trace_photon<false>(p, S, p.photon_base + i, &c);
        seg += c.segments; spl += c.splats; sca += c.scatters; ++ph;
    }
    for (int o = 16; o > 0; o >>= 1) {
        seg += __shfl_xor_sync(0xffffffffu, seg, o);
        spl += __shfl_xor_sync(0xffffffffu, spl, o);
        sca += __shfl_xor_sync(0xffffffffu, sca, o);
        ph += __shfl_xor_sync(0xffffffffu, ph, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(out, ph); atomicAdd(out + 1, seg); atomicAdd(out + 2, spl); atomicAdd(out + 3, sca);
    }
}

__global__ void __launch_bounds__(256) photon_debug_kernel(const PhotonParams p) {
    extern __shared__ __align__(16) unsigned char smem[];
    const float* cmf;
    const SceneView S = load_scene(p, smem, &cmf);
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < p.photon_count) trace_photon<true>(p, S, i);
}

// Surface rim pass (spectral-gpu/src/shaders/volume.wgsl:668-703 and its CPU
// oracle cpu_surface_rim, spectral-gpu/src/vol_photons.rs:1517-1538): one camera
// primary ray per pixel, nearest hit, rim = (1 - |n.d|)^2, tinted constant XYZ.
__global__ void __launch_bounds__(256) rim_kernel(const RimParams p) {
    extern __shared__ __align__(16) unsigned char smem[];
    sc_primitive* sp = reinterpret_cast<sc_primitive*>(smem);
    sc_plane* spl = reinterpret_cast<sc_plane*>(sp + p.n_prims);
    sc_material* sm = reinterpret_cast<sc_material*>(spl + p.n_planes);
    const uint32_t tid = threadIdx.y * blockDim.x + threadIdx.x, nt = blockDim.x * blockDim.y;
    for (uint32_t i = tid; i < p.n_prims; i += nt) sp[i] = p.prims[i];
    for (uint32_t i = tid; i < p.n_planes; i += nt) spl[i] = p.planes[i];
    for (uint32_t i = tid; i < p.n_mats; i += nt) sm[i] = p.mats[i];
    __syncthreads();
    const uint32_t px = blockIdx.x * blockDim.x + threadIdx.x, py = blockIdx.y * blockDim.y + threadIdx.y;
    if (px >= p.width || py >= p.height) return;
    SceneView S;
    S.prims = sp; S.planes = spl; S.mats = sm; S.n_prims = p.n_prims;
    const float s = ((float)px + 0.5f) / (float)p.width;
    const float t = 1.0f - ((float)py + 0.5f) / (float)p.height;
    const f3 o = ld3(p.cam.origin), d = primary_dir(p.cam, s, t);
    Hit h;
    uint32_t mi;
    const size_t i = (size_t)py * p.width + px;
    float x = 0.f, y = 0.f, z = 0.f;
    if (scene_hit(S, o, d, h, mi)) {
        const float c = fminf(fmaxf(fabsf(dot(h.normal, d)), 0.0f), 1.0f);
        const float rim = (1.0f - c) * (1.0f - c);
        x = 0.015f + rim * 0.45f; y = 0.02f + rim * 0.5f; z = 0.04f + rim * 0.6f;
    }
    p.out[3 * i] = x; p.out[3 * i + 1] = y; p.out[3 * i + 2] = z;
}

__global__ void rng_draws_kernel(uint32_t key, uint32_t seed, uint32_t n, uint32_t* out) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    Rng r = Rng::make(key, seed);
    for (uint32_t i = 0; i < n; ++i) out[i] = r.u32();
}

// ---------------------------------------------------------------------------
// Wavelength-ordered dispatch.  Photons of random wavelengths traced together
// touch the sectors of all bins of every pixel they reach, and a spectral film
// larger than L2 misses on most of its atomics.  Tracing the photons of a launch
// in order of their film bin keeps the photons in flight within a few bins: a few
// sectors for every four pixels are live at a time.  The photons and their paths are the
// same and the film is a sum of exact integers, so the image is bit-identical.
// Counting sort of the launch's photons by key (kOrderKeys groups of
// consecutive bins): per-CTA key histograms of contiguous photon chunks
// (key-major), one exclusive scan, then a scatter that stages 2048 photons at a
// time in shared memory so that each key's run is written contiguously.
constexpr uint32_t kOrderKeys = 16;
constexpr uint32_t kOrderTile = 2048;  // photons per scatter step: 8 per thread

// Sort key of photon `idx`: the group of its film bin (its third draw, as in
// the transport).
__device__ __forceinline__ uint32_t photon_key(const PhotonParams& p, uint32_t idx) {
    Rng r = Rng::make(idx, p.seed);
    r.state += 2u;  // the two aperture draws
    const float lambda = p.lambda_min + p.lambda_range * r.f32();
    const float fb = (lambda - p.bin_min) * p.bin_inv_width;
    const int bi = (int)fb;
    const uint32_t bin = fb < 0.0f ? 0u : (bi >= (int)p.bins ? p.bins - 1u : (uint32_t)bi);
    return p.bins <= kOrderKeys ? bin : bin * kOrderKeys / p.bins;
}

__global__ void __launch_bounds__(256) order_count_kernel(const PhotonParams p, uint32_t per_cta,
                                                          uint32_t* __restrict__ hist) {
    __shared__ uint32_t h[kOrderKeys];
    const uint32_t K = min(p.bins, kOrderKeys);
    if (threadIdx.x < K) h[threadIdx.x] = 0u;
    __syncthreads();
    const uint32_t i0 = blockIdx.x * per_cta, i1 = min(i0 + per_cta, p.photon_count);
    for (uint32_t i = i0 + threadIdx.x; i < i1; i += blockDim.x) atomicAdd(&h[photon_key(p, p.photon_base + i)], 1u);
    __syncthreads();
    if (threadIdx.x < K) hist[threadIdx.x * gridDim.x + blockIdx.x] = h[threadIdx.x];
}

// In-place exclusive scan of n counts by one CTA of 1024 threads.
__global__ void __launch_bounds__(1024) order_scan_kernel(uint32_t* __restrict__ a, uint32_t n) {
    __shared__ uint32_t part[1024];
    const uint32_t t = threadIdx.x, per = (n + 1023u) / 1024u;
    const uint32_t lo = min(t * per, n), hi = min(lo + per, n);
    uint32_t sum = 0;
    for (uint32_t i = lo; i < hi; ++i) sum += a[i];
    part[t] = sum;
    __syncthreads();
    for (uint32_t off = 1; off < 1024u; off <<= 1) {
        const uint32_t v = t >= off ? part[t - off] : 0u;
        __syncthreads();
        part[t] += v;
        __syncthreads();
    }
    uint32_t run = t ? part[t - 1] : 0u;
    for (uint32_t i = lo; i < hi; ++i) {
        const uint32_t c = a[i];
        a[i] = run;
        run += c;
    }
}

// Blocks of 256 threads.
__global__ void __launch_bounds__(256) order_scatter_kernel(const PhotonParams p, uint32_t per_cta,
                                                            const uint32_t* __restrict__ offsets,
                                                            uint32_t* __restrict__ order) {
    __shared__ uint32_t cur[kOrderKeys], cnt[kOrderKeys], toff[kOrderKeys];
    __shared__ uint32_t stage[kOrderTile];
    __shared__ uint8_t skey[kOrderTile];
    const uint32_t tid = threadIdx.x, K = min(p.bins, kOrderKeys);
    if (tid < K) cur[tid] = offsets[tid * gridDim.x + blockIdx.x];
    const uint32_t i0 = blockIdx.x * per_cta, i1 = min(i0 + per_cta, p.photon_count);
    for (uint32_t t0 = i0; t0 < i1; t0 += kOrderTile) {
        if (tid < K) cnt[tid] = 0u;
        __syncthreads();
        uint32_t key[8], rank[8];
#pragma unroll
        for (uint32_t j = 0; j < 8u; ++j) {
            const uint32_t i = t0 + j * 256u + tid;
            key[j] = i < i1 ? photon_key(p, p.photon_base + i) : 0xFFu;
            rank[j] = key[j] != 0xFFu ? atomicAdd(&cnt[key[j]], 1u) : 0u;  // rank within the tile's key run
        }
        __syncthreads();
        if (tid == 0) {
            uint32_t sum = 0;
            for (uint32_t k = 0; k < K; ++k) { toff[k] = sum; sum += cnt[k]; }
        }
        __syncthreads();
#pragma unroll
        for (uint32_t j = 0; j < 8u; ++j) {
            if (key[j] != 0xFFu) {
                const uint32_t pos = toff[key[j]] + rank[j];
                stage[pos] = t0 + j * 256u + tid;
                skey[pos] = (uint8_t)key[j];
            }
        }
        __syncthreads();
        const uint32_t n = min(kOrderTile, i1 - t0);
        for (uint32_t q = tid; q < n; q += 256u) {
            const uint32_t k = skey[q];
            order[cur[k] + (q - toff[k])] = stage[q];
        }
        __syncthreads();
        if (tid < K) cur[tid] += cnt[tid];
    }
}

__global__ void glass_n_kernel(uint32_t glass, const float* __restrict__ lambda_nm, uint32_t n,
                               float* __restrict__ out) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        out[i] = glass_n(glass, lambda_nm[i]);
}

}  // namespace

cudaError_t launch_glass_n(uint32_t glass, const float* lambda_nm, uint32_t n, float* out, cudaStream_t s) {
    const uint32_t need = (n + 255u) / 256u, grid = need < 148u * 16u ? need : 148u * 16u;
    glass_n_kernel<<<grid, 256, 0, s>>>(glass, lambda_nm, n, out);
    return cudaGetLastError();
}

cudaError_t launch_rng_draws(uint32_t key, uint32_t seed, uint32_t n, uint32_t* out, cudaStream_t s) {
    rng_draws_kernel<<<1, 32, 0, s>>>(key, seed, n, out);
    return cudaGetLastError();
}

size_t scene_smem_bytes(uint32_t n_prims, uint32_t n_planes, uint32_t n_mats) {
    return n_prims * sizeof(sc_primitive) + n_planes * sizeof(sc_plane) + n_mats * sizeof(sc_material) +
           3 * kTableN * sizeof(float);
}

using PhotonKernelFn = void (*)(const PhotonParams, uint32_t, uint32_t, uint32_t);

// `cached`: the launch takes the cell cache (the kernels built with it).
template <bool SPEC>
static PhotonKernelFn photon_fn(const LaunchShape& s, bool cached, bool ff, bool exact) {
    // haze samples in the reference's operation order, and free-flight launches: plain
    // atomics, 4 CTAs per SM
    if (exact) {
        if (ff) return cached ? photon_kernel<SPEC, 0, 4, true, true, true> : photon_kernel<SPEC, 0, 4, true, true>;
        return cached ? photon_kernel<SPEC, 0, 4, false, true, true> : photon_kernel<SPEC, 0, 4, false, true>;
    }
    if (ff) return cached ? photon_kernel<SPEC, 0, 4, true, false, true> : photon_kernel<SPEC, 0, 4, true>;
    if (s.aggregate) return s.minb >= 5 ? photon_kernel<SPEC, 1, 5, false> : photon_kernel<SPEC, 1, 4, false>;
    if (cached) return photon_kernel<SPEC, 0, 4, false, false, true>;  // 4 or 3 CTAs per SM (cache_slots)
    return s.minb >= 5 ? photon_kernel<SPEC, 0, 5, false> : photon_kernel<SPEC, 0, 4, false>;
}
static PhotonKernelFn photon_fn(const LaunchShape& s, bool spec, bool cached, bool ff, bool exact = false) {
    return spec ? photon_fn<true>(s, cached, ff, exact) : photon_fn<false>(s, cached, ff, exact);
}
// Shared memory beyond scene + mask: the parked photons of 8 warps.
static size_t park_bytes(bool spec) {
    return 16 + 8 * (spec ? sizeof(ParkedPhotons<true>) : sizeof(ParkedPhotons<false>));
}
void set_haze_consts(PhotonParams& p) {
    const double pi = 3.14159265358979323846;
    const double g = p.g;
    p.hz_w = (float)p.width;
    p.hz_h = (float)p.height;
    p.hz_hw = 0.5f * p.hz_w;
    p.hz_hh = 0.5f * p.hz_h;
    p.hz_sx = (float)((double)p.width / (double)p.proj.vw);
    p.hz_sy = (float)(-(double)p.height / (double)p.proj.vh);
    p.hz_k = (float)((double)p.sigma_s * (double)p.scale * 0.25 * (1.0 - g * g) / (4.0 * pi));
    p.hz_kiso = (float)((double)p.sigma_s * (double)p.scale * 0.25 / (4.0 * pi));
    p.hz_kexp = (float)(-(double)p.sigma_t * 1.4426950408889634);  // -sigma_t log2(e)
    p.hz_inv_sigma_t = p.sigma_t > 0.0f ? (float)(1.0 / (double)p.sigma_t) : 0.0f;
    p.hz_g2 = (float)(1.0 + g * g);
    p.hz_m2g = (float)(-2.0 * g);
}

void allow_max_smem(const void* fn) {
    static std::mutex mu;
    static std::set<std::pair<int, const void*>> done;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(mu);
    if (done.count({dev, fn})) return;
    cudaFuncAttributes at;
    int optin = 0;
    if (cudaFuncGetAttributes(&at, fn) != cudaSuccess ||
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
        cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)at.sharedSizeBytes) !=
            cudaSuccess) {
        cudaGetLastError();  // a launch that needs more then reports it
        return;
    }
    done.insert({dev, fn});
}

int occupancy_blocks(const void* fn, int block, size_t smem) {
    static std::mutex mu;
    static std::map<std::tuple<int, const void*, int, size_t>, int> cache;
    int dev = 0;
    cudaGetDevice(&dev);
    if (smem > 48 * 1024) allow_max_smem(fn);
    std::lock_guard<std::mutex> lk(mu);
    const auto key = std::make_tuple(dev, fn, block, smem);
    auto it = cache.find(key);
    if (it != cache.end()) return it->second;
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, block, smem) != cudaSuccess) return 1;
    n = n > 0 ? n : 1;
    cache.emplace(key, n);
    return n;
}

int photon_occupancy_blocks(const LaunchShape& shape, bool spectral, size_t smem) {
    return occupancy_blocks(reinterpret_cast<const void*>(photon_fn(shape, spectral, false, false)),
                            (int)shape.block, smem + park_bytes(spectral));
}

uint32_t photon_mask_words(const PhotonParams& p) {
    if (!p.flags) return 0u;
    const uint32_t tiles = p.tiles_x * ((p.height + 7u) / 8u);
    const uint32_t words = (tiles + 31u) / 32u;
    return words <= kMaxSmemMaskWords ? words : 0u;
}

// An attribute of the current device, read once per device (0 if unknown).
static uint32_t device_attribute(cudaDeviceAttr which) {
    static std::mutex mu;
    static std::map<std::pair<int, int>, uint32_t> cache;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(mu);
    const auto key = std::make_pair(dev, (int)which);
    auto it = cache.find(key);
    if (it != cache.end()) return it->second;
    int v = 0;
    cudaDeviceGetAttribute(&v, which, dev);
    cache.emplace(key, (uint32_t)(v > 0 ? v : 0));
    return (uint32_t)(v > 0 ? v : 0);
}
static size_t l2_bytes() { return device_attribute(cudaDevAttrL2CacheSize); }
static uint32_t sm_count() { return std::max(device_attribute(cudaDevAttrMultiProcessorCount), 1u); }

// About the pixels that the samples of the first segments share: they lie along the
// beam, the frame's height times the beam's width in pixels, seen from the camera at
// the beam's start (negative: behind the camera).
static float beam_pixels(const PhotonParams& p) {
    const f3 c = sub(add(p.corner, mul(add(p.bu, p.bv), 0.5f)), p.proj.o);
    const float depth = -dot(c, p.proj.w) / length(p.proj.w);
    const f3 across = cross(p.bdir, p.proj.w);  // on screen, square to the beam
    const float l = length(across);
    float width = length(p.bu) + length(p.bv);
    if (l > 1e-3f * length(p.bdir) * length(p.proj.w)) width = (fabsf(dot(p.bu, across)) + fabsf(dot(p.bv, across))) / l;
    if (!(depth > 0.0f)) return -1.0f;
    return (1.0f + width / depth * (float)p.height / p.proj.vh) * (float)p.height;
}

// Whether a launch takes the wavelength-ordered dispatch: point / isotropic
// estimators on a spectral film, at least 2^16 photons to amortise the sort, a
// memory pool for its scratch, and (order 1; order 2 orders every such launch) more of
// the film touched than L2 holds: a film larger than L2, a beam whose own pixels
// (beam_pixels) have more bytes of bins than L2, and at least two L2s of sectors hit
// (about 10 samples a photon, 32 bytes each).  Photons in the order of their bins
// add to the same lines at the same time, so where L2 holds what they touch the order
// costs.  Not ordered against ordered: rainbow 1920x1080x64 (342 MB under the beam) 2^19
// photons 426 and 437 us, 2^20 523 and 520, 2^22 941 and 818, 2^26 8.2 and 6.6 ms; prism
// 1024x1024x32 (2 MB) 2^20 190 and 218 us, 2^24 2.07 and 3.64 ms; dsotm 1600x1200x32 2^24
// 1.88 and 2.03 ms; 300,000 free-flight photons at 1001x563x31 88 and 114 us.
static bool ordered_dispatch(const PhotonParams& p, const LaunchShape& shape) {
    if (shape.order == 0 || !shape.pool || p.bins == 0u || p.channels != p.bins || p.order ||
        p.photon_count < (1u << 16))
        return false;
    if (shape.order >= 2) return true;
    const size_t film = (size_t)p.tiles_x * ((p.height + 7u) / 8u) * kTilePixels * p.channels * 8u, l2 = l2_bytes();
    return film > l2 && (double)beam_pixels(p) * p.channels * 8.0 > (double)l2 && p.photon_count * 320ull >= 2ull * l2;
}

static cudaError_t launch_photons_in(const PhotonParams& p, const LaunchShape& shape, cudaStream_t s);

cudaError_t launch_photons(const PhotonParams& p, const LaunchShape& shape, cudaStream_t s) {
    if (p.photon_count == 0) return cudaSuccess;
    if (!ordered_dispatch(p, shape)) return launch_photons_in(p, shape, s);
    const uint32_t grid = 148u * 4u;  // sort CTAs, each a contiguous chunk of the launch's photons
    const uint32_t per_cta = (p.photon_count + grid - 1u) / grid;
    const uint32_t keys = p.bins < kOrderKeys ? p.bins : kOrderKeys;
    const size_t words = (size_t)p.photon_count + (size_t)keys * grid;
    uint32_t* buf = nullptr;
    if (cudaMallocFromPoolAsync(reinterpret_cast<void**>(&buf), words * sizeof(uint32_t), shape.pool, s) !=
        cudaSuccess) {
        cudaGetLastError();  // no room for the sort: trace in launch order (same image)
        return launch_photons_in(p, shape, s);
    }
    uint32_t* order = buf;
    uint32_t* hist = buf + p.photon_count;
    order_count_kernel<<<grid, 256, 0, s>>>(p, per_cta, hist);
    order_scan_kernel<<<1, 1024, 0, s>>>(hist, keys * grid);
    order_scatter_kernel<<<grid, 256, 0, s>>>(p, per_cta, hist, order);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) {
        PhotonParams q = p;
        q.order = order;
        e = launch_photons_in(q, shape, s);
    }
    const cudaError_t f = cudaFreeAsync(buf, s);
    return e != cudaSuccess ? e : f;
}

// Whether the cell cache pays: the launch is not small (2^14 photons take as long
// with it as without: clearing and flushing it is 3 us), and the 32 * chunk
// first-segment samples of a CTA share cells (beam_pixels).  Measured at 640x360 (2
// to 3 pixels wide) without and with it: XYZ, 2^16 photons 88 -> 55 us (prism), 2^20
// 933 -> 385, 2^22 3243 -> 1300; dsotm 800x800, 4M photons 1161 -> 800; 8 bins, 2^20
// 265 -> 216 (16 bins take 175 without it).  The rainbow's beam (205 pixels): XYZ 2^20
// 330 -> 278 us (0.055 samples a cell), 2 bins 188 -> 163 (0.028), but 4 bins 108 -> 146
// (0.014): the line lies at 0.02.  At 0.05 for launches of less than 2^16 photons, whose
// one CTA an SM does not hide the clearing and flushing (XYZ, 2^15 photons, rainbow
// 256x256 (0.027) 26.5 and 30.9 us, 160x160 (0.07) 32.3 and 30.2, 128x128 (0.11) 36.3
// and 30.1), and for photons of one segment, whose samples no surface gathers (rainbow
// XYZ, 2^18 (0.028) 38.2 and 40.3, 2^20 (0.055) 124 and 116).  A z-buffer takes samples
// away: 0.055 then lose (148 -> 201), 4 still win (prism 995 -> 464); and without a scene
// they spread over all of the beam (XYZ, 95 pixels wide, 2^20 (0.1) 65 and 81, 2^21
// (0.2) 129 and 139): 0.4.
static bool cache_pays(const PhotonParams& p, uint32_t cells_per_pixel, uint32_t chunk, float pixels) {
    if (p.photon_count < (1u << 15)) return false;
    // keys are 32-bit cell indices below CellCache::kFree; films of one to seven rows
    // or columns have up to eight times their pixels in padded cells
    const uint64_t tiles = (uint64_t)p.tiles_x * ((p.height + 7u) / 8u);
    if (tiles * kTilePixels * cells_per_pixel > 0xFFFFFFFFull) return false;
    // 8 warps of at most 256 photons, 4 samples a segment
    if (8ull * 256ull * 4ull * p.max_bounces > kCacheDeposits) return false;
    if (!(pixels > 0.0f)) return false;
    const float line = p.zbuf || p.n_prims == 0u ? 0.4f
                       : p.photon_count < (1u << 16) || p.max_bounces == 1u ? 0.05f : 0.02f;
    return 32.0f * (float)chunk >= line * pixels * (float)cells_per_pixel;
}
// Slots of the cell cache beside `smem` bytes of a CTA (228 KB per SM, 1 KB of each
// CTA taken): what lets 4 CTAs share an SM, or for XYZ films 3, where the hot cells
// (about 2.5 for each pixel of the beam) find a slot then but not among 4 CTAs, and
// where chunks are long, or the beam is very wide, and they do neither way.  4 against 3
// CTAs, 2^20 photons: 1 to 8 bins 217 and 249 us, dsotm XYZ 256x256 205 and 242, 800x800
// 239 and 281; prism 640x360 XYZ 415 and 384 (2^22: 1388 and 1296), dsotm 1600x1200 2^22
// 955 and 900.  Very wide (rainbow XYZ 640x360, hot 100 n): 2^18 88 and 85 us, 2^19 155
// and 144, 2^20 282 and 254, 2^21 535 and 464 (256x256, 50 n: 2^17 55 and 57, 2^18 88 and
// 85, 2^20 277 and 250); no beam between 8 and 50 n was measured.  Launches of
// 32 photons a warp clear and flush 2048 at most (2^16 photons: 42 us against 44).
static uint32_t cache_slots(bool spec, size_t smem, uint32_t chunk, float pixels) {
    const size_t slot = spec ? CellCacheOf<true>::kSlotBytes : CellCacheOf<false>::kSlotBytes;
    auto fit = [&](uint32_t ctas) {
        const size_t room = (228u * 1024u) / ctas - 1024u;
        return room > smem ? (uint32_t)((room - smem) / slot) : 0u;
    };
    uint32_t n = fit(4);
    const float hot = 2.5f * pixels;
    if (!spec && hot > (float)n && (hot <= (float)fit(3) || chunk >= 256u || hot > 16.0f * (float)n)) n = fit(3);
    for (uint32_t ctas = 3; n < 1024u && ctas >= 1u; --ctas) n = fit(ctas);  // a large mask
    return std::min(n, chunk <= 32u ? 2048u : 8192u);
}

static cudaError_t launch_photons_in(const PhotonParams& p0, const LaunchShape& shape, cudaStream_t s) {
    PhotonParams p = p0;
    set_haze_consts(p);
    const bool exact = p.haze_exact != 0u;
    const uint32_t mw = photon_mask_words(p);
    const bool spec = p.channels != 3u || p.bins != 0u, few = !spec || p.channels <= kCacheBins;  // cells per pixel
    // 32 photons for each warp while the GPU holds all of them; then about two
    // chunks for each warp that it holds, 64 to 256 photons: the hardware starts
    // the next CTA where one has ended.  One CTA per resident slot with its share
    // of the photons ended unevenly (rainbow, 2^26 photons: 8.3 ms against 6.75,
    // SMs idle 18 % of it); longer chunks do so again (512: 6.79 ms, 2048: 6.98),
    // shorter ones pay for each warp's last photons and each CTA's setup (2^26
    // photons in chunks of 64: 7.35 ms; 2^20 photons, 64 bins: 64 187 us, 128 169).
    const uint64_t held = shape.grid * 8ull, per = p.photon_count / (2ull * held);
    uint32_t chunk = p.photon_count <= 32ull * held
                         ? 32u
                         : (uint32_t)(per < 64u ? 64u : per > 256u ? 256u : (per + 31u) & ~31ull);
    const float pixels = beam_pixels(p);
    const bool cached = few && (exact || shape.aggregate == 0) && cache_pays(p, spec ? p.channels : 1u, chunk, pixels);
    size_t smem = park_offset(p, mw) + park_bytes(spec);
    const uint32_t slots = cached ? cache_slots(spec, smem, chunk, pixels) : 0u;
    smem += slots * (size_t)(spec ? CellCacheOf<true>::kSlotBytes : CellCacheOf<false>::kSlotBytes);
    const PhotonKernelFn fn = photon_fn(shape, spec, slots != 0u, free_flight(p), exact);
    if (smem > 48 * 1024) allow_max_smem(reinterpret_cast<const void*>(fn));
    // a launch of less than one and a half rounds of CTAs is spread over one (dsotm
    // 400x300, 2^18 photons: 107 -> 90 us); with more rounds, chunks that are no multiple
    // of 32 cost what the even end saves (prism, 2^20 photons: 169 us against 182)
    const uint64_t resident = (uint64_t)sm_count() * (uint32_t)occupancy_blocks(reinterpret_cast<const void*>(fn), 256, smem);
    if (chunk > 32u && chunk <= 128u && 2ull * (p.photon_count / (8ull * chunk)) < 3ull * resident)
        chunk = std::max(32u, (uint32_t)((p.photon_count - 1u) / (8ull * resident) + 1u));
    const uint32_t grid = (uint32_t)((p.photon_count - 1u) / (8ull * chunk) + 1u);
    fn<<<grid, 256, smem, s>>>(p, mw, chunk, slots);
    return cudaGetLastError();
}

cudaError_t launch_photon_debug(const PhotonParams& p, cudaStream_t s) {
    if (p.photon_count == 0) return cudaSuccess;
    const size_t smem = scene_smem_bytes(p.n_prims, p.n_planes, p.n_mats);
    photon_debug_kernel<<<(p.photon_count + 255) / 256, 256, smem, s>>>(p);
    return cudaGetLastError();
}

cudaError_t launch_photon_count(const PhotonParams& p0, unsigned long long* out, uint32_t grid, cudaStream_t s) {
    if (p0.photon_count == 0) return cudaSuccess;
    PhotonParams p = p0;
    set_haze_consts(p);
    const size_t smem = scene_smem_bytes(p.n_prims, p.n_planes, p.n_mats);
    const uint32_t need = (p.photon_count + 255) / 256;
    photon_count_kernel<<<need < grid ? need : grid, 256, smem, s>>>(p, out);
    return cudaGetLastError();
}

cudaError_t launch_rim(const RimParams& p, cudaStream_t s) {
    const size_t smem = p.n_prims * sizeof(sc_primitive) + p.n_planes * sizeof(sc_plane) + p.n_mats * sizeof(sc_material);
    dim3 block(16, 16), grid((p.width + 15) / 16, (p.height + 15) / 16);
    rim_kernel<<<grid, block, smem, s>>>(p);
    return cudaGetLastError();
}

}  // namespace sc
