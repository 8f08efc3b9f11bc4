// Film kernels: sensor reduction / drain, exposure, tonemap, Gaussian gather,
// and the synthetic atomic-film splat.
#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>
#include <tuple>

#include "internal.h"

namespace sc {

namespace {

constexpr int kReduceThreads = 256;

// One film tile (64 pixels x C channels of int64) is staged into shared memory
// with 16-byte coalesced loads, optionally zeroed behind the load (drain), then
// reduced per pixel: XYZ film (no bin weights) -> value / 2^scale; spectral film -> sum over bins
// of count * bin-averaged CMF (f64 accumulation, fixed order per pixel).
// Tiles whose dirty flag is clear are never read: their pixels are written as 0.
//
// Software pipeline: a CTA walks its tiles keeping the next tile's first
// 8 x 256 16-byte vectors (a whole tile up to 64 channels) in registers, so
// those loads are in flight while the current tile is reduced out of shared
// memory.
struct TileRef {
    ReduceParams p;
    uint32_t tile;
    bool valid, dirty, keep;  // keep: never drained (an accumulating film)
};

__device__ __forceinline__ TileRef tile_ref(const ReduceParams& p, uint32_t tile, bool valid, bool keep = false) {
    TileRef t;
    t.p = p;
    t.tile = tile;
    t.valid = valid;
    t.keep = keep;
    t.dirty = valid && (p.flags == nullptr || ((p.flags[tile >> 5] >> (tile & 31u)) & 1u));
    return t;
}

constexpr uint32_t kPrefetch = 8;  // 16-byte vectors per thread held across a tile

__device__ __forceinline__ void prefetch_tile(const TileRef& t, ulonglong2 (&v)[kPrefetch]) {
    if (!t.dirty) return;
    const ulonglong2* src = reinterpret_cast<const ulonglong2*>(t.p.film + (size_t)t.tile * kTilePixels * t.p.channels);
    const uint32_t n2 = kTilePixels * t.p.channels / 2u;
#pragma unroll
    for (uint32_t k = 0; k < kPrefetch; ++k) {
        const uint32_t i = threadIdx.x + k * blockDim.x;
        if (i < n2) v[k] = __ldcs(src + i);
    }
}

// Registers (and any vectors beyond them) into shared memory; zero the film
// behind the copy when draining.
__device__ __forceinline__ void stage_tile(const TileRef& t, const ulonglong2 (&v)[kPrefetch], bool drain,
                                           unsigned long long* sm) {
    if (!t.dirty) return;
    ulonglong2* src = reinterpret_cast<ulonglong2*>(t.p.film + (size_t)t.tile * kTilePixels * t.p.channels);
    ulonglong2* dst = reinterpret_cast<ulonglong2*>(sm);
    const uint32_t n2 = kTilePixels * t.p.channels / 2u;
    const ulonglong2 zero = make_ulonglong2(0ull, 0ull);
#pragma unroll
    for (uint32_t k = 0; k < kPrefetch; ++k) {
        const uint32_t i = threadIdx.x + k * blockDim.x;
        if (i < n2) {
            dst[i] = v[k];
            if (drain) __stcs(src + i, zero);
        }
    }
    for (uint32_t i = threadIdx.x + kPrefetch * blockDim.x; i < n2; i += blockDim.x) {  // > 64 channels
        dst[i] = __ldcs(src + i);
        if (drain) __stcs(src + i, zero);
    }
}

// Per-pixel reduction of a staged tile (or zeros for a clean one).
__device__ __forceinline__ void reduce_staged(const TileRef& t, bool drain, const unsigned long long* sm,
                                              double* part) {
    const ReduceParams& p = t.p;
    const uint32_t C = p.channels, tile = t.tile;
    const uint32_t tx = tile % p.tiles_x, ty = tile / p.tiles_x;
    const uint32_t tid = threadIdx.x;
    if (!t.dirty || p.binw == nullptr) {  // clean, or an XYZ film (one of three bins has weights)
        for (uint32_t i = tid; i < kTilePixels * 3u; i += blockDim.x) {
            const uint32_t l = i / 3u, c = i % 3u;
            const uint32_t px = tx * 8u + (l & 7u), py = ty * 8u + (l >> 3);
            if (px < p.width && py < p.height)
                p.xyz[((size_t)py * p.width + px) * 3u + c] =
                    t.dirty ? (float)((double)(long long)sm[c * (uint32_t)kTilePixels + film_local(l, l >> 3)] *
                                      p.inv_scale)
                            : 0.0f;
        }
    } else {
        // 4 threads per pixel, each a contiguous quarter of the bins (a warp reads 32
        // cells of one bin side by side); partials are summed in quarter order so the result does
        // not depend on timing.
        const uint32_t l = tid & 63u, q = tid >> 6;
        if (q < 4u) {
            const uint32_t b0 = q * C / 4u, b1 = (q + 1u) * C / 4u;
            double x = 0.0, y = 0.0, z = 0.0;
            for (uint32_t b = b0; b < b1; ++b) {
                const double v = (double)(long long)sm[b * (uint32_t)kTilePixels + l];
                x += v * (double)p.binw[b];
                y += v * (double)p.binw[C + b];
                z += v * (double)p.binw[2u * C + b];
            }
            double* o = part + (q * 64u + film_local_pixel(l)) * 3u;
            o[0] = x; o[1] = y; o[2] = z;
        }
        __syncthreads();
        if (tid < 64u) {
            const uint32_t px = tx * 8u + (tid & 7u), py = ty * 8u + (tid >> 3);
            if (px < p.width && py < p.height) {
                float* o = p.xyz + ((size_t)py * p.width + px) * 3u;
                for (uint32_t c = 0; c < 3u; ++c) {
                    const double s = ((part[tid * 3u + c] + part[(64u + tid) * 3u + c]) + part[(128u + tid) * 3u + c]) +
                                     part[(192u + tid) * 3u + c];
                    o[c] = (float)(s * p.inv_scale);
                }
            }
        }
    }
    if (drain && t.dirty && p.flags && tid == 0) atomicAnd(p.flags + (tile >> 5), ~(1u << (tile & 31u)));
}

// The pipelined walk over this CTA's tiles; `at(k)` gives its k-th tile.
template <bool DRAIN, class At>
__device__ __forceinline__ void reduce_walk(At at, unsigned long long* sm, double* part) {
    ulonglong2 v[kPrefetch];
    TileRef cur = at(0u);
    prefetch_tile(cur, v);
    for (uint32_t k = 0; cur.valid; ++k) {
        stage_tile(cur, v, DRAIN && !cur.keep, sm);
        __syncthreads();
        const TileRef nxt = at(k + 1u);
        prefetch_tile(nxt, v);  // in flight while this tile is reduced
        reduce_staged(cur, DRAIN && !cur.keep, sm, part);
        __syncthreads();
        cur = nxt;
    }
}

template <bool DRAIN>
__global__ void __launch_bounds__(kReduceThreads, 3) reduce_kernel(const ReduceParams p) {
    extern __shared__ __align__(16) unsigned char smem[];
    double* part = reinterpret_cast<double*>(smem);
    unsigned long long* sm = reinterpret_cast<unsigned long long*>(smem + 4 * 64 * 3 * sizeof(double));
    const uint32_t ntiles = p.tiles_x * p.tiles_y;
    reduce_walk<DRAIN>(
        [&](uint32_t k) {
            const uint32_t tile = blockIdx.x + k * gridDim.x;
            return tile_ref(p, tile < ntiles ? tile : 0u, tile < ntiles);
        },
        sm, part);
}

// The sum of several films (one per GPU of a split scene: this GPU's own and
// its peers', read over NVLink) reduced for a range of tiles.  Each tile is
// staged as the exact int64 sum of the films' cells, then reduced by the
// single-film code, so a band equals the same band of the summed film's
// image.  The films are read, not drained; every tile counts as lit.
__global__ void __launch_bounds__(kReduceThreads, 3) reduce_peers_kernel(const ReduceParams p, const PeerFilms pf,
                                                                         uint32_t tile_begin, uint32_t tile_end) {
    extern __shared__ __align__(16) unsigned char smem[];
    double* part = reinterpret_cast<double*>(smem);
    unsigned long long* sm = reinterpret_cast<unsigned long long*>(smem + 4 * 64 * 3 * sizeof(double));
    const uint32_t n2 = kTilePixels * p.channels / 2u;
    for (uint32_t tile = tile_begin + blockIdx.x; tile < tile_end; tile += gridDim.x) {
        const size_t off2 = (size_t)tile * kTilePixels * p.channels / 2u;
        for (uint32_t i = threadIdx.x; i < n2; i += blockDim.x) {
            ulonglong2 acc = make_ulonglong2(0ull, 0ull);
            for (uint32_t f = 0; f < pf.n; ++f) {
                const ulonglong2 v = __ldcs(reinterpret_cast<const ulonglong2*>(pf.film[f]) + off2 + i);
                acc.x += v.x;
                acc.y += v.y;
            }
            reinterpret_cast<ulonglong2*>(sm)[i] = acc;
        }
        __syncthreads();
        reduce_staged(tile_ref(p, tile, true), false, sm, part);
        __syncthreads();
    }
}

// Many films, step 1: one CTA per dirty-mask word (32 tiles), a warp for each of
// their 8 pixel rows.  Clean tiles get zeros in the image, 16 bytes a lane where the
// rows allow it; dirty ones go to the list (one atomic per word), and when draining
// the word is cleared.  Words are numbered over all films (FilmDesc::word_begin), so
// a CTA finds its film by a binary search.  Bound: the zeros' stores (256 films of
// 67 M pixels: 392 us, 2 TB/s) or, for a server step's few hundred words, one word's
// chain of stores: 6.7 us, against 20 with one warp per word, tile after tile.
template <bool DRAIN>
__global__ void __launch_bounds__(256) reduce_scan_kernel(const FilmDesc* __restrict__ descs, uint32_t n_films,
                                                          uint32_t total_words, DirtyTile* __restrict__ list,
                                                          uint32_t* __restrict__ count) {
    const uint32_t lane = threadIdx.x & 31u, row = threadIdx.x >> 5;
    for (uint32_t w = blockIdx.x; w < total_words; w += gridDim.x) {
        uint32_t lo = 0, hi = n_films;
        while (hi - lo > 1u) {
            const uint32_t mid = (lo + hi) >> 1;
            if (descs[mid].word_begin <= w) lo = mid; else hi = mid;
        }
        const FilmDesc& d = descs[lo];
        const uint32_t wl = w - d.word_begin, first = wl * 32u, tiles = d.tiles_x * d.tiles_y;
        const uint32_t bits = d.flags[wl];
        const uint32_t valid = tiles - first >= 32u ? 0xFFFFFFFFu : (1u << (tiles - first)) - 1u;
        __syncthreads();  // every warp has read the word
        if (row == 0u) {
            const uint32_t dirty = bits & valid;
            if (dirty) {
                uint32_t base = 0;
                if (lane == 0) base = atomicAdd(count, (uint32_t)__popc(dirty));
                base = __shfl_sync(0xffffffffu, base, 0);
                if ((dirty >> lane) & 1u) list[base + __popc(dirty & ((1u << lane) - 1u))] = DirtyTile{lo, first + lane};
                if (DRAIN && !d.keep && lane == 0) d.flags[wl] = 0u;
            }
        }
        const uint32_t clean = valid & ~bits, row_floats = 3u * d.width;
        if (!clean) continue;
        // this warp's row of the 32 tiles: 6 vectors of 4 floats each
        for (uint32_t j = lane; j < 32u * 6u; j += 32u) {
            const uint32_t k = j / 6u, t = first + k;
            if (!((clean >> k) & 1u)) continue;
            const uint32_t ty = t / d.tiles_x, tx = t - ty * d.tiles_x, py = ty * 8u + row;
            const uint32_t col = tx * 24u + (j - 6u * k) * 4u;
            if (py >= d.height || col >= row_floats) continue;
            float* o = d.xyz + (size_t)py * row_floats + col;
            if (col + 4u <= row_floats && (reinterpret_cast<uintptr_t>(o) & 15u) == 0u) {
                *reinterpret_cast<float4*>(o) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            } else {
                for (uint32_t c = 0; c < 4u && col + c < row_floats; ++c) o[c] = 0.0f;
            }
        }
    }
}

// Many films, step 2: the listed dirty tiles through the pipelined walk.
template <bool DRAIN>
__global__ void __launch_bounds__(kReduceThreads, 3) reduce_list_kernel(const FilmDesc* __restrict__ descs,
                                                                     const DirtyTile* __restrict__ list,
                                                                     const uint32_t* __restrict__ count) {
    extern __shared__ __align__(16) unsigned char smem[];
    double* part = reinterpret_cast<double*>(smem);
    unsigned long long* sm = reinterpret_cast<unsigned long long*>(smem + 4 * 64 * 3 * sizeof(double));
    const uint32_t n = *count;
    reduce_walk<DRAIN>(
        [&](uint32_t k) {
            const uint32_t i = blockIdx.x + k * gridDim.x;
            ReduceParams p;
            if (i >= n) {
                p = ReduceParams{};
                return tile_ref(p, 0u, false);
            }
            const DirtyTile e = list[i];
            const FilmDesc& d = descs[e.film];
            p.film = d.film; p.flags = nullptr; p.xyz = d.xyz; p.width = d.width; p.height = d.height;
            p.tiles_x = d.tiles_x; p.tiles_y = d.tiles_y; p.channels = d.channels; p.binw = d.binw;
            p.inv_scale = d.inv_scale;
            return tile_ref(p, e.tile, true, d.keep != 0u);
        },
        sm, part);
}

__global__ void composite_max_y_kernel(const float* __restrict__ xyz, const float* __restrict__ surface,
                                       uint32_t n, uint32_t* out_bits) {
    float m = 0.0f;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float y = xyz[3u * i + 1u] + (surface ? surface[3u * i + 1u] : 0.0f);
        m = fmaxf(m, y);
    }
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0 && m > 0.0f) atomicMax(out_bits, __float_as_uint(m));
}

// Radix select of the k-th smallest composited luminance (values >= 0, so the
// IEEE bit patterns order like the floats) in three passes of 11, 11 and 10 bits.
// The CTA that finishes a pass last picks the digit that holds k, so a pass is one
// launch.  Lanes that share the first lane's digit (mostly the black pixels') count
// it once.  At 800x800 a call with its read-back takes 53 us (four passes of 8 bits,
// with a launch for each pick by one thread: 93).
// work: [0, 2048) histogram, then the digits found, k among their values, the
// result's bits, CTAs done; zero at the first pass, the histogram zero after each.
constexpr uint32_t kSelectBins = 2048, kSelectPrefix = kSelectBins, kSelectK = kSelectBins + 1,
                   kSelectDone = kSelectBins + 3;
static_assert(kSelectResult == kSelectBins + 2 && kSelectWords == kSelectBins + 4, "work layout");
template <int PASS>
__global__ void __launch_bounds__(256) select_kernel(const float* __restrict__ xyz, const float* __restrict__ surface,
                                                     uint32_t n, uint32_t k0, uint32_t* work) {
    constexpr int kShift = PASS == 0 ? 21 : PASS == 1 ? 10 : 0, kBits = PASS == 2 ? 10 : 11;
    __shared__ uint32_t hist[kSelectBins];
    __shared__ uint32_t warp_sum[8];
    __shared__ bool last;
    const uint32_t tid = threadIdx.x, lane = tid & 31u;
    for (uint32_t i = tid; i < kSelectBins; i += blockDim.x) hist[i] = 0u;
    __syncthreads();
    const uint32_t prefix = PASS ? work[kSelectPrefix] : 0u;
    for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
        const uint32_t i = base + tid;
        bool counts = i < n;
        uint32_t digit = 0;
        if (counts) {
            const float y = fmaxf(xyz[3u * (size_t)i + 1u] + (surface ? surface[3u * (size_t)i + 1u] : 0.0f), 0.0f);
            const uint32_t bits = __float_as_uint(y);
            if (PASS) counts = (bits >> (kShift + kBits)) == (prefix >> (kShift + kBits));
            digit = (bits >> kShift) & ((1u << kBits) - 1u);
        }
        const unsigned any = __ballot_sync(0xffffffffu, counts);
        if (!any) continue;
        const int src = __ffs(any) - 1;
        const uint32_t common = __shfl_sync(0xffffffffu, digit, src);
        const unsigned same = __ballot_sync(0xffffffffu, counts && digit == common);
        if ((int)lane == src) atomicAdd(&hist[common], (uint32_t)__popc(same));
        if (counts && digit != common) atomicAdd(&hist[digit], 1u);
    }
    __syncthreads();
    for (uint32_t i = tid; i < kSelectBins; i += blockDim.x)
        if (hist[i]) atomicAdd(&work[i], hist[i]);
    __threadfence();
    __syncthreads();
    if (tid == 0) last = atomicAdd(&work[kSelectDone], 1u) == gridDim.x - 1u;
    __syncthreads();
    if (!last) return;
    __threadfence();
    constexpr uint32_t kPer = kSelectBins / 256;  // digits of each thread
    uint32_t c[kPer], sum = 0;
#pragma unroll
    for (uint32_t j = 0; j < kPer; ++j) {
        c[j] = __ldcg(&work[tid * kPer + j]);
        work[tid * kPer + j] = 0u;
        sum += c[j];
    }
    uint32_t upto = sum;  // inclusive prefix over the threads
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, upto, o);
        if ((int)lane >= o) upto += v;
    }
    if (lane == 31u) warp_sum[tid >> 5] = upto;
    __syncthreads();
    for (uint32_t w = 0; w < (tid >> 5); ++w) upto += warp_sum[w];
    const uint32_t k = PASS ? work[kSelectK] : k0;
    uint32_t below = upto - sum;
    __syncthreads();  // every thread has read k
    if (below <= k && k < upto) {
        uint32_t j = 0;
#pragma unroll
        for (uint32_t q = 0; q + 1u < kPer; ++q)
            if (j == q && below + c[q] <= k) { below += c[q]; ++j; }
        const uint32_t found = prefix | ((tid * kPer + j) << kShift);
        work[kSelectPrefix] = found;
        work[kSelectK] = k - below;
        if (PASS == 2) work[kSelectResult] = found;
    }
    if (tid == 0) work[kSelectDone] = 0u;
}

__global__ void to_rgb8_kernel(const float* __restrict__ xyz, const float* __restrict__ surface, uint32_t n,
                               float exposure, uint8_t* out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float c[3];
    for (int k = 0; k < 3; ++k) c[k] = xyz[3u * i + k] + (surface ? surface[3u * i + k] : 0.0f);
    // xyz_to_linear_srgb + tonemap_to_u8 (spectral-core/src/cie.rs:121-144)
    const float lin[3] = {3.2406f * c[0] - 1.5372f * c[1] - 0.4986f * c[2],
                          -0.9689f * c[0] + 1.8758f * c[1] + 0.0415f * c[2],
                          0.0557f * c[0] - 0.2040f * c[1] + 1.0570f * c[2]};
    for (int k = 0; k < 3; ++k) {
        const float v = fmaxf(lin[k] * exposure, 0.0f);
        const float mapped = v / (1.0f + v);
        float gm = mapped <= 0.0031308f ? 12.92f * mapped : 1.055f * powf(mapped, 1.0f / 2.4f) - 0.055f;
        gm = fminf(fmaxf(gm, 0.0f), 1.0f);
        const float q = gm * 255.0f + 0.5f;
        out[3u * i + k] = (uint8_t)(q >= 255.0f ? 255.0f : q);
    }
}

// Viewer reconstruction (spectral-viewer/src/main.rs:132-173): normalized
// Gaussian gather, radius kradius, sigma max(kradius/2, 0.5), scaled by k, plus
// the rim surface, XYZ -> linear sRGB, Reinhard, gamma 1/2.2, RGBA8.
__global__ void gather_kernel(const float* __restrict__ xyz, const float* __restrict__ surface, uint32_t w,
                              uint32_t h, float k, float kradius, float exposure, uint8_t* out) {
    const uint32_t px = blockIdx.x * blockDim.x + threadIdx.x, py = blockIdx.y * blockDim.y + threadIdx.y;
    if (px >= w || py >= h) return;
    const int radius = (int)kradius;
    const float sigma = fmaxf(kradius * 0.5f, 0.5f);
    const float inv2s2 = 1.0f / (2.0f * sigma * sigma);
    float acc[3] = {0.f, 0.f, 0.f}, wsum = 0.0f;
    for (int dy = -radius; dy <= radius; ++dy)
        for (int dx = -radius; dx <= radius; ++dx) {
            const int sx = (int)px + dx, sy = (int)py + dy;
            if (sx >= 0 && sx < (int)w && sy >= 0 && sy < (int)h) {
                const size_t si = (size_t)sy * w + sx;
                const float g = expf(-(float)(dx * dx + dy * dy) * inv2s2);
                for (int c = 0; c < 3; ++c) acc[c] = acc[c] + xyz[3 * si + c] * g;
                wsum = wsum + g;
            }
        }
    const size_t i = (size_t)py * w + px;
    const float kk = k / fmaxf(wsum, 1e-6f);
    float comp[3];
    for (int c = 0; c < 3; ++c) comp[c] = (acc[c] * kk + (surface ? surface[3 * i + c] : 0.0f)) * exposure;
    const float lin[3] = {3.2406f * comp[0] - 1.5372f * comp[1] - 0.4986f * comp[2],
                          -0.9689f * comp[0] + 1.8758f * comp[1] + 0.0415f * comp[2],
                          0.0557f * comp[0] - 0.2040f * comp[1] + 1.0570f * comp[2]};
    const float inv_gamma = (float)(1.0 / 2.2);
    for (int c = 0; c < 3; ++c) {
        const float tt = lin[c] / (1.0f + lin[c]);
        float v = powf(fmaxf(tt, 0.0f), inv_gamma);
        v = fminf(fmaxf(v, 0.0f), 1.0f);
        out[4 * i + c] = (uint8_t)(v * 255.0f + 0.5f);
    }
    out[4 * i + 3] = 255;
}

// Synthetic splat (spectral-gpu/src/shaders/vol_splat.wgsl:34-55): one thread
// per splat, a hashed pixel, XYZ in [0,2), x4096 truncated, three u32 atomics.
__global__ void synthetic_splat_kernel(uint32_t* film, uint32_t w, uint32_t h, uint32_t seed, uint32_t n) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    Rng r = Rng::make(t, seed);
    const uint32_t idx = r.u32() % (w * h);
    const float x = r.f32() * 2.0f, y = r.f32() * 2.0f, z = r.f32() * 2.0f;
    atomicAdd(film + 3u * idx, (uint32_t)(fmaxf(x, 0.0f) * 4096.0f));
    atomicAdd(film + 3u * idx + 1u, (uint32_t)(fmaxf(y, 0.0f) * 4096.0f));
    atomicAdd(film + 3u * idx + 2u, (uint32_t)(fmaxf(z, 0.0f) * 4096.0f));
}
// AtomicFilm::resolve (spectral-gpu/src/film.rs:218-224), on the device.
__global__ void atomic_resolve_kernel(uint32_t* film, float* accum, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const uint32_t v = film[i];
        film[i] = 0u;
        accum[i] += (float)v / 4096.0f;
    }
}

size_t reduce_smem(uint32_t channels) {
    return 4 * 64 * 3 * sizeof(double) + (size_t)kTilePixels * channels * sizeof(unsigned long long);
}

}  // namespace

// Resident CTAs of a reduce kernel on the current device for `smem` bytes of
// dynamic shared memory, worked out once per (device, kernel, size) (raising
// the kernel's shared-memory limit on the way) and then served from a table.
static uint32_t reduce_grid(const void* fn, int which, size_t smem) {
    static std::mutex mu;
    static std::map<std::tuple<int, int, size_t>, uint32_t> cache;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(mu);
    const auto key = std::make_tuple(dev, which, smem);
    auto it = cache.find(key);
    if (it != cache.end()) return it->second;
    int sms = 148, per_sm = 1;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (smem > 48 * 1024) allow_max_smem(fn);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kReduceThreads, smem);
    const uint32_t grid = (uint32_t)sms * (uint32_t)(per_sm > 0 ? per_sm : 1);
    cache.emplace(key, grid);
    return grid;
}

cudaError_t launch_reduce(const ReduceParams& p, bool drain, cudaStream_t s) {
    const size_t smem = reduce_smem(p.channels);
    const uint32_t ntiles = p.tiles_x * p.tiles_y;
    const void* fn = drain ? reinterpret_cast<const void*>(&reduce_kernel<true>)
                           : reinterpret_cast<const void*>(&reduce_kernel<false>);
    uint32_t grid = reduce_grid(fn, drain ? 1 : 0, smem);
    if (grid > ntiles) grid = ntiles;
    if (grid == 0) return cudaSuccess;
    if (drain) reduce_kernel<true><<<grid, kReduceThreads, smem, s>>>(p);
    else reduce_kernel<false><<<grid, kReduceThreads, smem, s>>>(p);
    return cudaGetLastError();
}

cudaError_t launch_reduce_peers(const ReduceParams& p, const PeerFilms& films, uint32_t tile_begin, uint32_t tile_end,
                                cudaStream_t s) {
    if (tile_end <= tile_begin || films.n == 0) return cudaSuccess;
    const size_t smem = reduce_smem(p.channels);
    uint32_t grid = reduce_grid(reinterpret_cast<const void*>(&reduce_peers_kernel), 2, smem);
    if (grid > tile_end - tile_begin) grid = tile_end - tile_begin;
    reduce_peers_kernel<<<grid, kReduceThreads, smem, s>>>(p, films, tile_begin, tile_end);
    return cudaGetLastError();
}

cudaError_t launch_reduce_many(const FilmDesc* descs, uint32_t n_films, uint32_t total_words, bool drain,
                               uint32_t max_channels, DirtyTile* list, uint32_t* count, cudaStream_t s) {
    if (total_words == 0 || n_films == 0) return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(count, 0, sizeof(uint32_t), s);
    if (e != cudaSuccess) return e;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const uint32_t cap = (uint32_t)sms * 8u, sgrid = total_words < cap ? total_words : cap;
    if (drain) reduce_scan_kernel<true><<<sgrid, 256, 0, s>>>(descs, n_films, total_words, list, count);
    else reduce_scan_kernel<false><<<sgrid, 256, 0, s>>>(descs, n_films, total_words, list, count);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    const size_t smem = reduce_smem(max_channels);
    const void* fn = drain ? reinterpret_cast<const void*>(&reduce_list_kernel<true>)
                           : reinterpret_cast<const void*>(&reduce_list_kernel<false>);
    const uint32_t grid = reduce_grid(fn, drain ? 3 : 2, smem);
    if (drain) reduce_list_kernel<true><<<grid, kReduceThreads, smem, s>>>(descs, list, count);
    else reduce_list_kernel<false><<<grid, kReduceThreads, smem, s>>>(descs, list, count);
    return cudaGetLastError();
}

cudaError_t launch_composite_max_y(const float* xyz, const float* surface, uint32_t n, uint32_t* out_bits,
                                   cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(out_bits, 0, sizeof(uint32_t), s);
    if (e != cudaSuccess) return e;
    uint32_t grid = (n + 255) / 256;
    if (grid > 1184) grid = 1184;
    if (grid == 0) grid = 1;
    composite_max_y_kernel<<<grid, 256, 0, s>>>(xyz, surface, n, out_bits);
    return cudaGetLastError();
}

cudaError_t launch_composite_select(const float* xyz, const float* surface, uint32_t n, uint32_t k, uint32_t* work,
                                    cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(work, 0, kSelectWords * sizeof(uint32_t), s);
    if (e != cudaSuccess) return e;
    // two CTAs per SM, at least 1024 pixels each: every CTA adds its digits to one histogram
    const uint32_t need = (n + 1023u) / 1024u, grid = need < 296u ? std::max(need, 1u) : 296u;
    select_kernel<0><<<grid, 256, 0, s>>>(xyz, surface, n, k, work);
    select_kernel<1><<<grid, 256, 0, s>>>(xyz, surface, n, k, work);
    select_kernel<2><<<grid, 256, 0, s>>>(xyz, surface, n, k, work);
    return cudaGetLastError();
}

cudaError_t launch_to_rgb8(const float* xyz, const float* surface, uint32_t n, float exposure, uint8_t* out,
                           cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    to_rgb8_kernel<<<(n + 255) / 256, 256, 0, s>>>(xyz, surface, n, exposure, out);
    return cudaGetLastError();
}

cudaError_t launch_gather_rgba8(const float* xyz, const float* surface, uint32_t w, uint32_t h, float k,
                                float kradius, float exposure, uint8_t* out, cudaStream_t s) {
    dim3 block(16, 16), grid((w + 15) / 16, (h + 15) / 16);
    gather_kernel<<<grid, block, 0, s>>>(xyz, surface, w, h, k, kradius, exposure, out);
    return cudaGetLastError();
}

cudaError_t launch_synthetic_splat(uint32_t* film, uint32_t w, uint32_t h, uint32_t seed, uint32_t n,
                                   cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    synthetic_splat_kernel<<<(n + 255) / 256, 256, 0, s>>>(film, w, h, seed, n);
    return cudaGetLastError();
}

cudaError_t launch_atomic_resolve(uint32_t* film, float* accum, size_t n, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    size_t grid = (n + 255) / 256;
    if (grid > 4096) grid = 4096;
    atomic_resolve_kernel<<<(unsigned)grid, 256, 0, s>>>(film, accum, n);
    return cudaGetLastError();
}

// Bin-averaged colour matching: for bin b of [lambda_min, lambda_max), the mean
// of the clamped table lerp over 16 sub-bin midpoints (what a photon drawn
// uniformly inside the bin would deposit on average).
void bin_weights(const float* tables, uint32_t bins, float lambda_min, float lambda_max, float* out) {
    const double width = ((double)lambda_max - (double)lambda_min) / (double)bins;
    for (uint32_t b = 0; b < bins; ++b) {
        double acc[3] = {0.0, 0.0, 0.0};
        for (int j = 0; j < 16; ++j) {
            const float nm = (float)((double)lambda_min + width * ((double)b + ((double)j + 0.5) / 16.0));
            for (int c = 0; c < 3; ++c) acc[c] += (double)tab_sample(tables + c * kTableN, nm);
        }
        for (int c = 0; c < 3; ++c) out[c * bins + b] = (float)(acc[c] / 16.0);
    }
}

Proj make_proj(const sc_camera& c) { return proj_make(c); }

}  // namespace sc
