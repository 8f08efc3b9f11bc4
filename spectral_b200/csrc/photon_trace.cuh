// Per-photon transport shared by the plain photon kernel (photon.cu) and the
// batched persistent kernel (batch.cu): emission, bounce loop, haze samples and
// the fixed-point film deposit.  See photon.cu for the reference it restates.
#pragma once
#include "internal.h"

namespace sc {

constexpr float kInv4Pi = 1.0f / (4.0f * 3.14159265358979323846f);

// Stage the scene records and the CMF table in shared memory; when `mask_words`
// is non-zero a zeroed dirty-tile bitmask of that many words follows them.
__device__ __forceinline__ SceneView load_scene(const PhotonParams& p, unsigned char* smem, const float** cmf_out,
                                                uint32_t** mask_out = nullptr, uint32_t mask_words = 0) {
    sc_primitive* sp = reinterpret_cast<sc_primitive*>(smem);
    sc_plane* spl = reinterpret_cast<sc_plane*>(sp + p.n_prims);
    sc_material* sm = reinterpret_cast<sc_material*>(spl + p.n_planes);
    float* scmf = reinterpret_cast<float*>(sm + p.n_mats);
    uint32_t* mask = reinterpret_cast<uint32_t*>(scmf + 3 * kTableN);
    for (uint32_t i = threadIdx.x; i < p.n_prims; i += blockDim.x) sp[i] = p.prims[i];
    for (uint32_t i = threadIdx.x; i < p.n_planes; i += blockDim.x) spl[i] = p.planes[i];
    for (uint32_t i = threadIdx.x; i < p.n_mats; i += blockDim.x) sm[i] = p.mats[i];
    for (uint32_t i = threadIdx.x; i < 3u * kTableN; i += blockDim.x) scmf[i] = p.cmf[i];
    for (uint32_t i = threadIdx.x; i < mask_words; i += blockDim.x) mask[i] = 0u;
    __syncthreads();
    *cmf_out = scmf;
    if (mask_out) *mask_out = mask_words ? mask : nullptr;
    SceneView S;
    S.prims = sp; S.planes = spl; S.mats = sm; S.n_prims = p.n_prims;
    return S;
}

__device__ __forceinline__ void red_u64(unsigned long long* a, unsigned long long v) {
    if (v) atomicAdd(a, v);
}

// Exact segmented sum of 64-bit values over the lanes of `peers` using three
// 26-bit chunks (no chunk sum can overflow 32 bits for <= 32 lanes).
__device__ __forceinline__ unsigned long long peer_sum64(unsigned peers, unsigned long long v) {
    unsigned c0 = (unsigned)(v & 0x3FFFFFFull);
    unsigned c1 = (unsigned)((v >> 26) & 0x3FFFFFFull);
    unsigned c2 = (unsigned)(v >> 52);
    unsigned s0 = __reduce_add_sync(peers, c0);
    unsigned s1 = __reduce_add_sync(peers, c1);
    unsigned s2 = __reduce_add_sync(peers, c2);
    return (unsigned long long)s0 + ((unsigned long long)s1 << 26) + ((unsigned long long)s2 << 52);
}

// Dirty-tile bitmask: bits go to this CTA's shared-memory copy (flushed to the
// global mask when the CTA finishes) or, for films whose mask does not fit,
// straight to the global mask with a fire-and-forget red.or.
__device__ __forceinline__ void mark_tile(const PhotonParams& p, uint32_t* smask, uint32_t tile) {
    if (!p.flags) return;
    const uint32_t w = tile >> 5, bit = 1u << (tile & 31u);
    if (smask) {
        if (!(smask[w] & bit)) atomicOr(smask + w, bit);
    } else {
        atomicOr(p.flags + w, bit);
    }
}

// Where the mask is: its shared-memory address, or kMaskGlobal (the global mask only)
// or kMaskNone, worked out once for a segment's samples; and the bit of a tile in the
// shared one, in bit 0.
constexpr uint32_t kMaskGlobal = 0xFFFFFFFEu, kMaskNone = 0xFFFFFFFFu;
__device__ __forceinline__ uint32_t mask_address(const PhotonParams& p, const uint32_t* smask) {
    return !p.flags ? kMaskNone : smask ? (uint32_t)__cvta_generic_to_shared(smask) : kMaskGlobal;
}
__device__ __forceinline__ uint32_t mask_bit(uint32_t mask, uint32_t tile) {
    uint32_t w;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w) : "r"(mask + ((tile >> 5) << 2)));
    return w >> (tile & 31u);
}

// Film access of one photon: its bin's cells of tile 0, the cells of a tile, tiles
// per row.
struct FilmView {
    unsigned long long* cell0;
    uint32_t tile_cells, tiles_x;
    // `pixel`: tile << 6 | film_local()
    __device__ __forceinline__ unsigned long long* cell(uint32_t pixel) const {
        return cell0 + (size_t)(pixel >> 6) * tile_cells + (pixel & 63u);
    }
};
template <bool SPEC>
__device__ __forceinline__ FilmView film_view(const PhotonParams& p, uint32_t bin) {
    FilmView v;
    v.cell0 = p.film + (SPEC ? bin * kTilePixels : 0u);
    v.tile_cells = (SPEC ? p.channels : 3u) * kTilePixels;
    v.tiles_x = p.tiles_x;
    return v;
}

// Shared-memory sums of the film cells a CTA deposits to most often, for films
// with few cells per pixel: the photons of a narrow beam meet in a few hundred
// pixels, and every photon of the launch adds to the same cells of each.  A cell (the
// three values of an XYZ pixel, the one of a spectral film's pixel and bin) takes the
// slot its hash names if that is free; others go straight to the film.  A sum is a
// 32-bit word per value and a count of its carries (XYZ: 10 bits of one word each):
// one shared atomic per value, and a second one only where a word wraps.  Values
// below 2^22 stay exact over kCacheDeposits deposits (2^9 carries); launches whose
// CTAs could make more do without.  (Two words per value, both added to: 8 bins 237
// us against 216, dsotm 256x256 XYZ 235 against 205 for 2^20 photons.)
// V: values per cell.
constexpr uint64_t kCacheDeposits = 1u << 19;
template <int V>
struct CellCache {
    static constexpr uint32_t kFree = 0xFFFFFFFFu, kSlotBytes = 4u * (V + 2u);
    uint32_t slots;
    uint32_t* key;  // slots: the cell's position in the film (XYZ: its pixel, tile-major), or free
    uint32_t* sum;  // V x slots: low words of the values
    uint32_t* carry;
    __device__ __forceinline__ CellCache(void* at, uint32_t n)
        : slots(n), key(static_cast<uint32_t*>(at)), sum(key + n), carry(sum + V * n) {}
    __device__ __forceinline__ void clear() {
        for (uint32_t i = threadIdx.x; i < slots; i += blockDim.x) key[i] = kFree;
        for (uint32_t i = threadIdx.x; i < (V + 1u) * slots; i += blockDim.x) sum[i] = 0u;  // and the carries
    }
    // Adds the sums to the film.
    __device__ __forceinline__ void flush(unsigned long long* film) const {
        for (uint32_t i = threadIdx.x; i < slots; i += blockDim.x) {
            if (key[i] == kFree) continue;
            unsigned long long* cell = V == 1 ? film + key[i]
                                              : film + (size_t)(key[i] >> 6) * (V * kTilePixels) + (key[i] & 63u);
#pragma unroll
            for (int k = 0; k < V; ++k) {
                const uint32_t c = V == 1 ? carry[i] : (carry[i] >> (10 * k)) & 1023u;
                red_u64(cell + k * kTilePixels, (unsigned long long)sum[k * slots + i] | ((unsigned long long)c << 32));
            }
        }
    }
    // Whether the values went into the cache.
    __device__ __forceinline__ bool add(uint32_t k, const unsigned long long (&v)[V]) {
        unsigned long long any = 0;
#pragma unroll
        for (int c = 0; c < V; ++c) any |= v[c];
        if (any >> 22) return false;
        const uint32_t slot = __umulhi(k * 0x9E3779B1u, slots);
        uint32_t t = key[slot];
        if (t == kFree) t = atomicCAS(&key[slot], kFree, k);
        if (t != k && t != kFree) return false;
        uint32_t wrapped = 0;
#pragma unroll
        for (int c = 0; c < V; ++c) {
            const uint32_t x = (uint32_t)v[c], old = atomicAdd(&sum[c * slots + slot], x);
            if (old + x < old) wrapped |= 1u << (10 * c);
        }
        if (wrapped) atomicAdd(&carry[slot], wrapped);
        return true;
    }
};
// Spectral films of up to this many bins may go through the cache (2^20 photons of
// the narrow prism beam without and with it: 1 bin 469 -> 216 us, 4 bins 353 -> 219, 8
// bins 265 -> 216; 16 bins take 175 without it).
constexpr uint32_t kCacheBins = 8;
// No cache (a null pointer of it): films of many bins, and small launches.
template <bool SPEC> using CellCacheOf = CellCache<SPEC ? 1 : 3>;

template <bool SPEC>
__device__ __forceinline__ bool cache_take(CellCacheOf<SPEC>& cache, const PhotonParams& p, uint32_t pixel,
                                           const unsigned long long* cell, unsigned long long v0,
                                           unsigned long long v1, unsigned long long v2) {
    if constexpr (SPEC) return cache.add((uint32_t)(cell - p.film), {v0});  // below 2^32 - 1: cache_pays()
    else return cache.add(pixel, {v0, v1, v2});
}

// Deposit one haze sample.  AGG=1 merges lanes of the warp that hit the same
// film cell before issuing the atomic.
// `scale`: the film's 2^k, or 1 when `contrib` carries it already.
template <bool SPEC, int AGG>
__device__ __forceinline__ void deposit(const PhotonParams& p, const FilmView& fv, uint32_t* smask, bool ok,
                                        uint32_t px, uint32_t py, float contrib, float cx, float cy, float cz,
                                        float scale, CellCacheOf<SPEC>* cache = nullptr) {
    unsigned long long* cell = nullptr;
    uint32_t tile = 0, pixel = 0;
    unsigned long long v0 = 0, v1 = 0, v2 = 0;
    if (ok) {
        tile = film_tile(px, py, fv.tiles_x);
        pixel = (tile << 6) | film_local(px, py);  // below 2^32
        cell = fv.cell(pixel);
        if (SPEC) {
            v0 = to_fixed(contrib, scale);
        } else {
            v0 = to_fixed(cx * contrib, scale);
            v1 = to_fixed(cy * contrib, scale);
            v2 = to_fixed(cz * contrib, scale);
        }
    }
    if (AGG == 0) {
        if (!ok) return;
        mark_tile(p, smask, tile);
        if (cache && cache_take<SPEC>(*cache, p, pixel, cell, v0, v1, v2)) return;
        red_u64(cell, v0);
        if (!SPEC) { red_u64(cell + kTilePixels, v1); red_u64(cell + 2 * kTilePixels, v2); }
        return;
    }
    const unsigned mask = __activemask();
    const unsigned peers = __match_any_sync(mask, reinterpret_cast<unsigned long long>(cell));  // null: not in frame
    if (!ok) return;
    const unsigned lane = threadIdx.x & 31u;
    if (peers != (1u << lane)) {
        v0 = peer_sum64(peers, v0);
        if (!SPEC) { v1 = peer_sum64(peers, v1); v2 = peer_sum64(peers, v2); }
        if ((int)lane != __ffs(peers) - 1) return;
    }
    mark_tile(p, smask, tile);
    red_u64(cell, v0);
    if (!SPEC) { red_u64(cell + kTilePixels, v1); red_u64(cell + 2 * kTilePixels, v2); }
}

__device__ __forceinline__ void record_pair(sc_debug_photon* rec, uint32_t pair, f3 o, f3 d) {
    if (pair >= 9u) return;
    float* q = rec->states[2 * pair];
    q[0] = o.x; q[1] = o.y; q[2] = o.z; q[3] = 0.0f;
    q = rec->states[2 * pair + 1];
    q[0] = d.x; q[1] = d.y; q[2] = d.z; q[3] = 0.0f;
}

// Work counters of one photon (instrumented launches only): segments traced,
// haze samples that land in frame (= film splats), dielectric/diffuse scatters.
struct PhotonCounts { uint32_t segments, splats, scatters; };

// Free-flight sampling (estimator 3, no counterpart in the reference): the
// haze sample distance follows the free-flight density sigma_t exp(-sigma_t t)
// restricted to the segment, t = -log(1 - u (1 - exp(-sigma_t seg))) / sigma_t,
// and the sample is weighted by 1 / pdf(t) = (1 - exp(-sigma_t seg)) /
// (sigma_t exp(-sigma_t t)) instead of the uniform estimator's seg: the same
// single-scatter integral, with samples denser where the beam enters.  With
// sigma_t = 0 it is the uniform estimator.
// FF: free-flight distances (estimator 3 with sigma_t > 0).  Kernels are built
// with or without free-flight support (FFOK); launches of the uniform
// estimators take the kernels without it, whose code is the uniform path only.
__host__ __device__ __forceinline__ bool free_flight(const PhotonParams& p) {
    return p.estimator == 3u && p.sigma_t > 0.0f;
}
template <bool FF>
__device__ __forceinline__ float haze_distance(const PhotonParams& p, float u, float seg) {
    if (!FF) return u * seg;
    return -log1pf(u * expm1f(-p.sigma_t * seg)) / p.sigma_t;
}
template <bool FF>
__device__ __forceinline__ float haze_span(const PhotonParams& p, float dist, float seg) {
    if (!FF) return seg;
    return -expm1f(-p.sigma_t * seg) / (p.sigma_t * expf(-p.sigma_t * dist));
}

// One point-estimator haze sample at distance `dist` along a segment
// (spectral-core/src/volume.rs:130-150): camera projection, z-test, HG phase x
// transmittance / d^2 x seg/4 (x 1/pdf / 4 for free-flight samples).  Returns
// whether the sample lands in frame; `contrib`, px, py are its weight and pixel.
template <bool FF>
__device__ __forceinline__ bool haze_sample(const PhotonParams& p, f3 o, f3 d, float dist, float seg, float power,
                                            uint32_t& px, uint32_t& py, float& contrib) {
    const f3 q = add(o, mul(d, dist));
    float s, t;
    bool ok = project(p.proj, q, s, t);
    contrib = 0.0f;
    px = py = 0u;
    if (ok) {
        px = min((uint32_t)(s * (float)p.width), p.width - 1u);
        py = min((uint32_t)((1.0f - t) * (float)p.height), p.height - 1u);
        if (FF || p.estimator != 1u) {  // point estimators (the beam estimator has its own kernel)
            const f3 to = sub(p.proj.o, q);
            const float dd = fmaxf(length(to), 1e-3f);
            if (p.zbuf && !(dd < p.zbuf[py * p.width + px])) {
                ok = false;
            } else {
                // g == 0: phase_hg is exactly 1/(4 pi) (pow(1, 1.5) == 1), so the
                // direction to the camera is not needed.
                const float phase = p.g == 0.0f ? kInv4Pi : phase_hg(p.g, dot(d, vdiv(to, dd)));
                const float trans = expf(-p.sigma_t * dd);
                contrib = power * p.sigma_s * phase * trans / (dd * dd) * haze_span<FF>(p, dist, seg) / 4.0f;
            }
        } else {
            contrib = power * p.sigma_s * seg / 4.0f * kInv4Pi;
        }
    }
    return ok;
}

// ---------------------------------------------------------------------------
// Fast haze samples.  Only the transport (intersection, Fresnel / refract /
// TIR, Sellmeier) decides a photon's path; the haze samples only weight film
// deposits, so they need the film's accuracy (0.5 % relative L1), not the CPU
// crate's operation order.  Along a segment q(t) = o + d t, with D = o - o_cam
// and the camera basis (u, v, w, |horizontal|, |vertical|):
//   depth  c(t)     = D.w + (d.w) t                  (in front: c < -1e-6)
//   column s(t) * W = W/2 + (a0 + a1 t) / -c(t),  a = (D.u, d.u) * W / |horizontal|
//   row (1-t') * H  = H/2 + (b0 + b1 t) / -c(t),  b = (D.v, d.v) * -H / |vertical|
//   distance^2      = h2 + (s0 + s1 t)^2,  s1 = |d|, s0 = -|d| t*, t* = -D.d / |d|^2,
//                     h2 = |D + d t*|^2 (squared distance of closest approach: a sum of
//                     two non-negative terms, so no cancellation near the camera)
//   d . (to camera) / distance = -s1 (s0 + s1 t) / distance
// so a sample costs three fused multiply-adds for the projection, one
// reciprocal, one reciprocal square root and one exp2 (PTX approximations),
// and the constant factor k = power sigma_s seg / 4 * 2^scale * HG numerator
// is formed once per segment.  The HG denominator power 1.5 is r^3 with
// r = rsqrt(max(1 + g^2 - 2 g cos, 1e-6)).
__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rsqrt_approx(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Per-segment constants.  `segs` is seg * 2^-24 for the uniform estimator
// (t = (draw >> 8) * segs, the same product the reference rounds) and
// expm1(-sigma_t seg) for free-flight distances.
struct HazeSeg { float c0, c1, a0, a1, b0, b1, s0, s1, h2, k, segs; };

// Dot product with fused multiply-adds (haze constants only: the transport
// keeps the reference's separate multiplies and adds).
__device__ __forceinline__ float fdot(f3 a, f3 b) { return __fmaf_rn(a.z, b.z, __fmaf_rn(a.y, b.y, a.x * b.x)); }

template <bool FF>
__device__ __forceinline__ HazeSeg haze_setup(const PhotonParams& p, f3 o, f3 d, float seg, float power) {
    const Proj& P = p.proj;
    const f3 D = sub(o, P.o);
    HazeSeg h;
    h.c0 = fdot(D, P.w);
    h.c1 = fdot(d, P.w);
    h.a0 = fdot(D, P.u) * p.hz_sx;
    h.a1 = fdot(d, P.u) * p.hz_sx;
    h.b0 = fdot(D, P.v) * p.hz_sy;
    h.b1 = fdot(d, P.v) * p.hz_sy;
    const float e2 = fdot(d, d);
    const float r2 = rsqrt_approx(e2);                 // 1 / |d|
    const float tstar = -fdot(D, d) * (r2 * r2);
    const f3 m = mk(__fmaf_rn(d.x, tstar, D.x), __fmaf_rn(d.y, tstar, D.y), __fmaf_rn(d.z, tstar, D.z));
    h.h2 = fdot(m, m);
    h.s1 = e2 * r2;                                    // |d|
    h.s0 = -h.s1 * tstar;
    if (FF) {
        const float em = expm1f(-p.sigma_t * seg);
        h.segs = em;
        h.k = power * (-em * p.hz_inv_sigma_t) * p.hz_k;  // 1/pdf numerator (1 - e^-sigma_t seg) / sigma_t
    } else {
        h.segs = seg * (1.0f / 16777216.0f);
        h.k = power * seg * (p.estimator == 1u ? p.hz_kiso : p.hz_k);
    }
    return h;
}

// What every sample of a segment reads of the launch's parameters, loaded once
// per segment: the parameters may live in shared memory, where the compiler has
// to load them again after every film atomic.
struct HazeView {
    float hw, hh, w, h, kexp;
    uint32_t width, height;
};
__device__ __forceinline__ HazeView haze_view(const PhotonParams& p) {
    HazeView v;
    v.hw = p.hz_hw; v.hh = p.hz_hh; v.w = p.hz_w; v.h = p.hz_h; v.kexp = p.hz_kexp;
    v.width = p.width; v.height = p.height;
    return v;
}
// One haze sample of a segment from its 24-bit draw; returns whether it lands
// in frame (and is not occluded), with its pixel and its scaled weight.
template <bool FF>
__device__ __forceinline__ bool haze_fast(const PhotonParams& p, const HazeView& v, const HazeSeg& h, uint32_t draw24,
                                          uint32_t& px, uint32_t& py, float& contrib) {
    float t;
    if (FF) t = -log1pf((float)draw24 * (1.0f / 16777216.0f) * h.segs) * p.hz_inv_sigma_t;
    else t = (float)draw24 * h.segs;
    const float c = __fmaf_rn(h.c1, t, h.c0);
    const float rc = rcp_approx(-c);
    const float x = __fmaf_rn(__fmaf_rn(h.a1, t, h.a0), rc, v.hw);
    const float y = __fmaf_rn(__fmaf_rn(h.b1, t, h.b0), rc, v.hh);
    contrib = 0.0f;
    px = py = 0u;
    if (!(c < -1e-6f && x >= 0.0f && x < v.w && y > 0.0f && y <= v.h)) return false;
    px = min((uint32_t)x, v.width - 1u);
    py = min((uint32_t)y, v.height - 1u);
    if (!FF && p.estimator == 1u) {  // isotropic estimator: no transmittance, no 1/d^2, no z-test
        contrib = h.k;
        return true;
    }
    const float q = __fmaf_rn(h.s1, t, h.s0);
    const float dd2 = fmaxf(__fmaf_rn(q, q, h.h2), 1e-6f);
    const float r = rsqrt_approx(dd2);
    const float dd = dd2 * r;
    if (p.zbuf && !(dd < p.zbuf[py * v.width + px])) return false;
    float w = h.k * ex2_approx(v.kexp * (FF ? dd - t : dd)) * (r * r);
    if (p.g != 0.0f) {
        const float den = fmaxf(__fmaf_rn(p.hz_m2g, -(h.s1 * q) * r, p.hz_g2), 1e-6f);
        const float rr = rsqrt_approx(den);
        w *= rr * rr * rr;
    }
    contrib = w;
    return true;
}

// Photon-level splat payload: CMF of the photon's wavelength (XYZ film) or its bin.
__device__ __forceinline__ void photon_payload(const PhotonParams& p, const float* cmf, float lambda, float& cx,
                                               float& cy, float& cz, uint32_t& bin, bool spec) {
    if (spec) {
        float fb = (lambda - p.bin_min) * p.bin_inv_width;
        int bi = (int)fb;
        bin = fb < 0.0f ? 0u : (bi >= (int)p.bins ? p.bins - 1u : (uint32_t)bi);
    } else {
        cx = tab_sample(cmf, lambda);
        cy = tab_sample(cmf + kTableN, lambda);
        cz = tab_sample(cmf + 2 * kTableN, lambda);
    }
}

// One photon on its own: recorded (DEBUG: its states, no samples) or counted (its
// samples that land in frame, no film).
template <bool DEBUG>
__device__ __forceinline__ void trace_photon(const PhotonParams& p, const SceneView& S, uint32_t idx,
                                             PhotonCounts* cnt = nullptr) {
    Rng r = Rng::make(idx, p.seed);
    const float r1 = r.f32();
    const float r2 = r.f32();
    f3 o = add(add(p.corner, mul(p.bu, r1)), mul(p.bv, r2));
    const float lambda = p.lambda_min + p.lambda_range * r.f32();
    f3 d = p.bdir;
    float power = 1.0f;
    uint32_t n_glass = 0xFFFFFFFFu;
    float n_cached = 1.0f;
    sc_debug_photon* rec = nullptr;
    uint32_t pairs = 1;
    if (DEBUG) {
        rec = p.debug + idx;
        rec->lambda = lambda;
        rec->pad0 = rec->pad1 = 0u;
        record_pair(rec, 0, o, d);
    }
    for (uint32_t b = 0; b < p.max_bounces; ++b) {
        Hit h;
        uint32_t mi = 0;
        const bool any = scene_hit(S, o, d, h, mi);
        const float seg = any ? h.t : p.max_dist;
        if (DEBUG) {
            r.state += 4u;  // the segment's 4 distance draws
        } else {
            ++cnt->segments;
            const bool ff = free_flight(p);
            const HazeSeg hz = ff ? haze_setup<true>(p, o, d, seg, power) : haze_setup<false>(p, o, d, seg, power);
            const HazeView hv = haze_view(p);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t draw24 = r.u32() >> 8;
                uint32_t px, py;
                float contrib;
                const bool ok = ff ? haze_fast<true>(p, hv, hz, draw24, px, py, contrib)
                                   : haze_fast<false>(p, hv, hz, draw24, px, py, contrib);
                if (ok) ++cnt->splats;
            }
        }
        if (!any) break;
        const sc_material& m = S.mats[mi];
        // n(lambda) depends only on the photon's wavelength and the glass: the f64
        // Sellmeier sum runs once per photon and glass, not once per hit.
        float nh = 1.0f;
        if (m.kind == 1u) {
            if (m.glass != n_glass) { n_cached = glass_n(m.glass, p.spectral ? lambda : 550.0f); n_glass = m.glass; }
            nh = n_cached;
        }
        f3 nd;
        float w;
        if (!DEBUG) ++cnt->scatters;
        scatter(m, d, h, nh, r, nd, w);
        power *= w;
        o = h.point;
        d = nd;
        if (DEBUG) { record_pair(rec, pairs, o, d); ++pairs; }
    }
    if (DEBUG) rec->num_states = pairs < 9u ? pairs : 9u;
}

// The four haze samples of a segment into the film.  With plain atomics and the
// point estimators, all four are worked out before the first deposit, without a
// branch, so that their chains of approximations overlap: batch pass 22.3 -> 20.5 ms
// against sample by sample.  (Not with a z-buffer: a sample that is occluded ends
// there.)  Nearly every deposit is below 2^23 quanta and takes the short rounding:
// prism, 2^20 photons 174.5 -> 169.5 us, batch pass 19.3 -> 18.9 ms.  It holds for
// weights that are not negative, as to_fixed() clamps them: a segment's constant
// weight carries their sign (sigma_s, 1 - g^2, a reflectance or a length below zero).
// TOGETHER: the four tiles are tested together (they are lit but for a launch's first
// photons): 300,000 free-flight photons 114.4 -> 112.0 us, rainbow 6.66 -> 6.59 ms; the
// batch kernel, which keeps its parameters in shared memory, has no registers for it
// (18.9 -> 22.6 ms).
// G: g != 0.  FF: free-flight distances.
template <bool SPEC, bool G, bool FF, bool TOGETHER>
__device__ __forceinline__ void haze_four(const PhotonParams& p, const HazeSeg& h, Rng& r, float cx, float cy, float cz,
                                          uint32_t bin, uint32_t* smask, CellCacheOf<SPEC>* cache) {
    const HazeView v = haze_view(p);
    const FilmView fv = film_view<SPEC>(p, bin);
    const float hk = SPEC ? fmaxf(h.k, 0.0f) : h.k;  // NaN: 0, as to_fixed() has it
    uint32_t pixel[4];
    float weight[4];  // -1: not in frame
#pragma unroll
    for (int k = 0; k < 4; ++k) {  // the arithmetic of haze_fast
        const float draw = (float)(r.u32() >> 8);
        float t;
        if (FF) t = -log1pf(draw * (1.0f / 16777216.0f) * h.segs) * p.hz_inv_sigma_t;
        else t = draw * h.segs;
        const float c = __fmaf_rn(h.c1, t, h.c0);
        const float rc = rcp_approx(-c);
        const float x = __fmaf_rn(__fmaf_rn(h.a1, t, h.a0), rc, v.hw);
        const float y = __fmaf_rn(__fmaf_rn(h.b1, t, h.b0), rc, v.hh);
        const bool ok = c < -1e-6f && x >= 0.0f && x < v.w && y > 0.0f && y <= v.h;
        const uint32_t px = min((uint32_t)x, v.width - 1u), py = min((uint32_t)y, v.height - 1u);
        const float q = __fmaf_rn(h.s1, t, h.s0);
        const float dd2 = fmaxf(__fmaf_rn(q, q, h.h2), 1e-6f);
        const float rd = rsqrt_approx(dd2);
        const float dd = dd2 * rd;
        float w = hk * ex2_approx(v.kexp * (FF ? dd - t : dd)) * (rd * rd);
        if (G) {
            const float den = fmaxf(__fmaf_rn(p.hz_m2g, -(h.s1 * q) * rd, p.hz_g2), 1e-6f);
            const float rr = rsqrt_approx(den);
            w *= rr * rr * rr;
        }
        weight[k] = ok ? w : -1.0f;
        pixel[k] = (film_tile(px, py, fv.tiles_x) << 6) | film_local(px, py);  // in the film, ok or not
    }
    if (TOGETHER) {
        const uint32_t mask = mask_address(p, smask);
        uint32_t lit = mask == kMaskNone ? 1u : 0u;
        if (mask < kMaskGlobal) {
            lit = 1u;
#pragma unroll
            for (int k = 0; k < 4; ++k) lit &= mask_bit(mask, pixel[k] >> 6) | (weight[k] == -1.0f ? 1u : 0u);
        }
        if (!(lit & 1u)) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (weight[k] != -1.0f) mark_tile(p, smask, pixel[k] >> 6);
        }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (weight[k] != -1.0f) {
            if (!TOGETHER) mark_tile(p, smask, pixel[k] >> 6);
            unsigned long long* cell = fv.cell(pixel[k]);
            if (SPEC) {
                if (!cache && weight[k] < 8388608.0f) {  // to_fixed without its tests: nearly every deposit
                    atomicAdd(cell, (unsigned long long)(__float_as_uint(weight[k] + 8388608.0f) - 0x4B000000u));
                    continue;
                }
                const unsigned long long x = to_fixed(weight[k], 1.0f);
                if (!cache || !cache_take<SPEC>(*cache, p, pixel[k], cell, x, 0ull, 0ull)) red_u64(cell, x);
            } else {
                const unsigned long long x = to_fixed(cx * weight[k], 1.0f), y = to_fixed(cy * weight[k], 1.0f),
                                         z = to_fixed(cz * weight[k], 1.0f);
                if (!cache || !cache_take<SPEC>(*cache, p, pixel[k], cell, x, y, z)) {
                    red_u64(cell, x);
                    red_u64(cell + kTilePixels, y);
                    red_u64(cell + 2 * kTilePixels, z);
                }
            }
        }
    }
}

// Photons set aside by a warp of the grouped transport: 32 at most.
template <bool SPEC>
struct alignas(16) ParkedPhotons {
    float f[9][32];                // ox oy oz dx dy dz lambda power n(lambda)
    uint32_t rng[32], bounce[32];
    uint32_t meta[32];             // glass of n + 1 (0: none yet) | bin << 16
    float c[SPEC ? 1 : 3][32];     // XYZ films: CMF of lambda
};
// Live lanes below which a warp parks or refills.  16, 20, 24, 28, 32: rainbow, 2^26 photons
// 7.04, 6.89, 6.73, 6.68, 6.68 ms; batch pass 19.05, 19.03, 19.01, 18.99, 19.11; prism,
// 2^20 photons 169 us with each.
constexpr int kGroupLive = 24;

// One photon per lane over positions [0, count) of a range (photon id = id(k)),
// in groups.  All 32 lanes of the warp start photons together, so emission, the
// film payload and the f64 index of the first glass hit run converged, and trace
// them bounce by bounce.  Photons of a beam mostly end after the same number of
// segments; when fewer than kGroupLive lanes are left, the live photons are
// parked in shared memory and the lanes start the next 32, or take up parked
// photons once these make a full warp.  The photons, their draws and their
// samples are those of one photon after the other, so the film is too.
// EXACT: haze samples in the CPU crate's operation order (haze_sample), otherwise
// the fast ones.
template <bool SPEC, int AGG, bool FFOK, bool TOGETHER, bool EXACT, class Id>
__device__ __forceinline__ void trace_group_range(const PhotonParams& p, const SceneView& S, const float* cmf,
                                                  uint32_t count, Id id, uint32_t* smask, ParkedPhotons<SPEC>& park,
                                                  CellCacheOf<SPEC>* cache = nullptr) {
    const uint32_t lane = threadIdx.x & 31u;
    const unsigned below = (1u << lane) - 1u;
    const bool ff = FFOK && free_flight(p);
    if (p.max_bounces == 0u) return;
    Rng r;
    r.state = 0u;
    f3 o = mk(0.f, 0.f, 0.f), d = p.bdir;
    float lambda = 0.0f, power = 1.0f, cx = 0.f, cy = 0.f, cz = 0.f;
    uint32_t bin = 0, bounce = 0, n_glass = 0xFFFFFFFFu;
    float n_cached = 1.0f;
    bool alive = false;
    uint32_t next = 0, parked = 0;  // the same in every lane
    for (;;) {
        const unsigned live = __ballot_sync(0xffffffffu, alive);
        const uint32_t n = __popc(live);
        if (n < (uint32_t)kGroupLive) {
            if (next < count && parked + n < 32u) {
                // park the live photons, start the next group
                if (alive) {
                    const uint32_t q = parked + __popc(live & below);
                    park.f[0][q] = o.x; park.f[1][q] = o.y; park.f[2][q] = o.z;
                    park.f[3][q] = d.x; park.f[4][q] = d.y; park.f[5][q] = d.z;
                    park.f[6][q] = lambda; park.f[7][q] = power; park.f[8][q] = n_cached;
                    park.rng[q] = r.state;
                    park.bounce[q] = bounce;
                    park.meta[q] = (n_glass <= 3u ? n_glass + 1u : 0u) | (bin << 16);
                    if (!SPEC) { park.c[0][q] = cx; park.c[SPEC ? 0 : 1][q] = cy; park.c[SPEC ? 0 : 2][q] = cz; }
                }
                parked += n;
                const uint32_t k = next + lane;
                next += 32u;
                alive = k < count;
                if (alive) {
                    r = Rng::make(id(k), p.seed);
                    const float r1 = r.f32();
                    const float r2 = r.f32();
                    o = add(add(p.corner, mul(p.bu, r1)), mul(p.bv, r2));
                    d = p.bdir;
                    lambda = p.lambda_min + p.lambda_range * r.f32();
                    photon_payload(p, cmf, lambda, cx, cy, cz, bin, SPEC);
                    power = 1.0f;
                    bounce = 0;
                    n_glass = 0xFFFFFFFFu;
                }
            } else if (parked) {
                // idle lanes take up parked photons
                __syncwarp();
                const uint32_t take = min(parked, 32u - n);
                const uint32_t rank = __popc(~live & below);
                if (!alive && rank < take) {
                    const uint32_t q = parked - 1u - rank;
                    o = mk(park.f[0][q], park.f[1][q], park.f[2][q]);
                    d = mk(park.f[3][q], park.f[4][q], park.f[5][q]);
                    lambda = park.f[6][q]; power = park.f[7][q]; n_cached = park.f[8][q];
                    r.state = park.rng[q];
                    const uint32_t m = park.meta[q];
                    bounce = park.bounce[q];
                    n_glass = (m & 0xFFFFu) - 1u;
                    bin = m >> 16;
                    if (!SPEC) { cx = park.c[0][q]; cy = park.c[SPEC ? 0 : 1][q]; cz = park.c[SPEC ? 0 : 2][q]; }
                    alive = true;
                }
                parked -= take;
                __syncwarp();
            } else if (n == 0u) {
                break;
            }
        }
        if (alive) {
            Hit h;
            uint32_t mi = 0;
            const bool any = scene_hit(S, o, d, h, mi);
            const float seg = any ? h.t : p.max_dist;
            if constexpr (EXACT) {
                const FilmView fv = film_view<SPEC>(p, bin);
#pragma unroll 1
                for (int k = 0; k < 4; ++k) {
                    const float u = r.f32();
                    const float dist = ff ? haze_distance<true>(p, u, seg) : haze_distance<false>(p, u, seg);
                    uint32_t px, py;
                    float contrib;
                    const bool ok = ff ? haze_sample<true>(p, o, d, dist, seg, power, px, py, contrib)
                                       : haze_sample<false>(p, o, d, dist, seg, power, px, py, contrib);
                    deposit<SPEC, AGG>(p, fv, smask, ok, px, py, contrib, cx, cy, cz, p.scale, cache);
                }
            } else {
                const HazeSeg hz = ff ? haze_setup<true>(p, o, d, seg, power) : haze_setup<false>(p, o, d, seg, power);
                if (AGG == 0 && FFOK && ff && !p.zbuf) {
                    haze_four<SPEC, true, FFOK, TOGETHER>(p, hz, r, cx, cy, cz, bin, smask, cache);
                } else if (AGG == 0 && !ff && !p.zbuf && p.estimator != 1u) {
                    if (p.g == 0.0f) haze_four<SPEC, false, false, TOGETHER>(p, hz, r, cx, cy, cz, bin, smask, cache);
                    else haze_four<SPEC, true, false, TOGETHER>(p, hz, r, cx, cy, cz, bin, smask, cache);
                } else {
                    const HazeView hv = haze_view(p);
                    const FilmView fv = film_view<SPEC>(p, bin);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const uint32_t draw24 = r.u32() >> 8;
                        uint32_t px, py;
                        float contrib;
                        const bool ok = ff ? haze_fast<true>(p, hv, hz, draw24, px, py, contrib)
                                           : haze_fast<false>(p, hv, hz, draw24, px, py, contrib);
                        deposit<SPEC, AGG>(p, fv, smask, ok, px, py, contrib, cx, cy, cz, 1.0f, cache);
                    }
                }
            }
            ++bounce;
            if (!any || bounce >= p.max_bounces) {
                alive = false;  // escaped, or its last segment: no scatter needed
            } else {
                const sc_material& m = S.mats[mi];
                float nh = 1.0f;
                if (m.kind == 1u) {
                    if (m.glass != n_glass) {
                        n_cached = glass_n(m.glass, p.spectral ? lambda : 550.0f);
                        n_glass = m.glass;
                    }
                    nh = n_cached;
                }
                f3 nd;
                float w;
                scatter(m, d, h, nh, r, nd, w);
                power *= w;
                o = h.point;
                d = nd;
            }
        }
    }
}

}  // namespace sc
