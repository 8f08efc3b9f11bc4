// Wavefront hero-wavelength camera path tracer.
//
// Restates CpuTracer::sample_pixel / accumulate (spectral-core/src/tracer.rs:44-141;
// GPU mirror spectral-gpu/src/shaders/trace.wgsl:419-537) as a wavefront:
//   generate  one path per (pixel, sample): stream key mix2(pixel, sample index),
//             jittered primary ray, hero-comb wavelength draw (spectrum.rs:20-32);
//   intersect nearest scene hit (+ the optional spherical emitter) per ray,
//             in the kernel that shades it (primary rays where they are made;
//             later rays as the next bounce reads them from the dense queue);
//   shade     background / emission at termination, Fresnel / refract / TIR or
//             Lambertian scatter, dispersion collapse to the hero lane, optional
//             Russian roulette; each warp collects its survivors in shared memory
//             and queues them 32 at a time;
//   tail      the paths alive after the compacted bounces finish in one launch,
//             idle lanes taking new paths from the queue;
//   accumulate each pixel's samples summed in sample order (the CPU's order), so
//             the image is deterministic and, for scenes without Lambertian
//             surfaces, bit-identical to the CPU tracer.
// Queue counts stay on the device: the launch sequence of an accumulate call is
// fixed, needs no host synchronisation and is replayed from a CUDA graph.
//
// Bound: instruction issue (the stages' queues take 1 to 1.5 TB/s).  accumulate(64)
// at 1280x720 of the prism on its floor 4.54 -> 3.05 ms, accumulate(4) at 333x187 of
// glass under a sky 75 -> 54 us, from warps that compact and refill by themselves
// (barriers were 30 to 60 % of the stage stalls), combs without radiance left out,
// four table columns in one row, and quotients by constants as products.
#include <algorithm>

#include "internal.h"
#include "tracer.h"

namespace sc {

namespace {

constexpr int kShadeThreads = 256;
// Shade and tail CTAs resident per SM: 5 (48 registers, small spills).
constexpr int kStageCtasPerSm = 5;
constexpr float kLambdaMin = 380.0f, kLambdaRange = 350.0f;

struct TracerSmem {
    TracerParams p;
    float4 table[kTableN + 1];  // x, y, z and illuminant of a row; the last row twice
    alignas(16) sc_primitive prims[SC_MAX_PRIMS];
    sc_material mats[SC_MAX_PRIMS];
    float4 bounds[SC_MAX_PRIMS];
};

// Stage params, scene records and sensor tables in shared memory.  Planes live
// after the fixed part (dynamic size).
__device__ __forceinline__ SceneView load_tracer(const TracerParams* gp, TracerSmem& s, sc_plane* planes) {
    const uint32_t tid = threadIdx.x;
    if (tid == 0) s.p = *gp;
    const float* tab = gp->tables;
    const float* ill = tab + (gp->illuminant == 1u ? 4 : 3) * kTableN;
    for (uint32_t i = tid; i <= (uint32_t)kTableN; i += blockDim.x) {
        const uint32_t k = min(i, (uint32_t)kTableN - 1u);
        s.table[i] = make_float4(tab[k], tab[kTableN + k], tab[2 * kTableN + k], ill[k]);
    }
    __syncthreads();
    for (uint32_t i = tid; i < s.p.n_prims; i += blockDim.x) s.prims[i] = s.p.prims[i];
    for (uint32_t i = tid; i < s.p.n_mats; i += blockDim.x) s.mats[i] = s.p.mats[i];
    for (uint32_t i = tid; i < s.p.n_prims; i += blockDim.x) s.bounds[i] = s.p.bounds[i];
    for (uint32_t i = tid; i < s.p.n_planes; i += blockDim.x) planes[i] = s.p.planes[i];
    __syncthreads();
    SceneView S;
    S.prims = s.prims; S.planes = planes; S.mats = s.mats; S.n_prims = s.p.n_prims;
    return S;
}

__device__ __forceinline__ float lane_lambda(float u, int k) {
    // SpectralSample::from_hero_u: (u*RANGE + k*RANGE/4).rem_euclid(RANGE).  For
    // 0 <= x < 2 RANGE (u is a draw, in [0, 1)) the remainder is x or x - RANGE,
    // which is exact there (RANGE <= x < 2 RANGE).
    const float x = u * kLambdaRange + (float)k * (kLambdaRange / 4.0f);
    return kLambdaMin + (x >= kLambdaRange ? x - kLambdaRange : x);
}

// x / (1 / 350), correctly rounded: the product with the reciprocal (350 is that
// of the rounded 1 / 350), corrected by its fused remainder (Brisebarre, Muller and
// Raina, "Accelerating correctly rounded floating-point division when the divisor is
// known in advance"; all mantissas compared with the quotient).  Where the
// remainder could underflow or the product overflow: the division.
__device__ __forceinline__ float over_pdf(float x) {
    const float pdf = 1.0f / kLambdaRange;
    if (!(x > 1e-25f && x < 1e25f)) return x / pdf;
    const float q = x * kLambdaRange;
    return __fmaf_rn(__fmaf_rn(-pdf, q, x), kLambdaRange, q);
}

// XYZ of a terminated comb whose lanes carry radiance rad_k = tp_k * e * S(lambda_k).
// `valid`: 4 lanes, or 1 after a dispersive hit (dividing by either is scaling by
// a power of two).  A comb of 1 lane has no radiance in the others: they are not
// worked out (unless e is infinite: 0 * inf).  The four table columns lie in one
// row, so a lane costs two 16-byte loads and one division by 5.
__device__ __forceinline__ void comb_xyz(const TracerSmem& s, float u, float tp, uint32_t valid, float e,
                                         float out[3]) {
    const bool one = valid == 1u;
    const int lanes = one && fabsf(e) < __int_as_float(0x7f800000) ? 1 : 4;
    const float inv_valid = one ? 1.0f : 0.25f;
    float x = 0.0f, y = 0.0f, z = 0.0f;
#pragma unroll 1
    for (int k = 0; k < lanes; ++k) {
        const float f = tab_position(lane_lambda(u, k));
        const int i = (int)f;
        const float frac = f - (float)i;
        const float4 a = s.table[i], b = s.table[i + 1];
        const float tk = k == 0 || !one ? tp : 0.0f;
        const float wk = over_pdf(tk * e * (a.w + (b.w - a.w) * frac)) * inv_valid;
        x += (a.x + (b.x - a.x) * frac) * wk;
        y += (a.y + (b.y - a.y) * frac) * wk;
        z += (a.z + (b.z - a.z) * frac) * wk;
    }
    out[0] = x; out[1] = y; out[2] = z;
}

// Whether a ray certainly misses a bounding sphere (centre, radius^2 in b):
// the origin is outside it and the line's closest approach at t >= 0 is
// outside it.  The sphere is inflated on the host (1 % + 1e-3) far beyond the
// rounding of these products; origins farther than 100 radii are not culled
// (the products would cancel), so a culled solid is one that solid_hit would
// not hit either.
__device__ __forceinline__ bool misses_bound(float4 b, f3 o, f3 d) {
    if (!(b.w < __int_as_float(0x7f800000))) return false;
    const f3 oc = mk(b.x - o.x, b.y - o.y, b.z - o.z);
    const float l2 = dot(oc, oc);
    if (!(l2 > b.w) || l2 > 1e4f * b.w) return false;
    const float bb = dot(oc, d);
    if (bb <= 0.0f) return true;  // moving away from the centre, from outside
    return (l2 - b.w) * dot(d, d) > bb * bb;
}

// Scene::intersect (scene_hit) skipping convex solids whose bounding sphere
// the ray misses: the same nearest hit, fewer plane tests.
__device__ __forceinline__ bool scene_hit_bounded(const TracerSmem& s, const SceneView& S, f3 o, f3 d, Hit& best,
                                                  uint32_t& mat) {
    bool any = false;
    float closest = __int_as_float(0x7f800000);
    for (uint32_t i = 0; i < S.n_prims; ++i) {
        const float4 ball = reinterpret_cast<const float4*>(S.prims)[2 * i];
        const uint4 meta = reinterpret_cast<const uint4*>(S.prims)[2 * i + 1];  // first plane, planes, kind, material
        if (meta.z == 1u && misses_bound(s.bounds[i], o, d)) continue;
        Hit h;
        bool ok = meta.z == 0u ? sphere_hit(mk(ball.x, ball.y, ball.z), ball.w, o, d, 1e-3f, closest, h)
                : (meta.z == 1u ? solid_hit(S, meta.x, meta.y, o, d, 1e-3f, closest, h) : false);
        if (ok) { closest = h.t; best = h; mat = meta.w; any = true; }
    }
    return any;
}

// Nearest hit of one ray: scene records and the optional emitter sphere.
// info = material | front_face << 16 | kind << 24 (0 miss, 1 surface, 2 emitter).
__device__ __forceinline__ void trace_hit(const TracerSmem& s, const SceneView& S, f3 o, f3 d, float& t, f3& n,
                                          uint32_t& info) {
    Hit h;
    uint32_t mi = 0;
    const bool any = scene_hit_bounded(s, S, o, d, h, mi);
    uint32_t kind = any ? 1u : 0u;
    t = any ? h.t : __int_as_float(0x7f800000);
    if (s.p.em_radius > 0.0f) {
        Hit he;
        if (sphere_hit(s.p.em_center, s.p.em_radius, o, d, 1e-3f, t, he)) { kind = 2u; t = he.t; }
    }
    n = h.normal;
    info = mi | (((any && h.front_face) ? 1u : 0u) << 16) | (kind << 24);
}

// State of one path between bounces (the ray queue's fields).
struct PathState {
    f3 o, d;
    float tp, u;
    uint32_t rs, id, flags;  // RNG state, path id, valid lanes | depth << 8
};

__device__ __forceinline__ PathState read_path(const RayQueue& q, uint32_t i) {
    PathState P;
    P.o = mk(q.ox[i], q.oy[i], q.oz[i]);
    P.d = mk(q.dx[i], q.dy[i], q.dz[i]);
    P.tp = q.tp[i]; P.u = q.u[i]; P.rs = q.rng[i]; P.id = q.id[i]; P.flags = q.flags[i];
    return P;
}

// Shade one path at `bounce` given its hit: background / emission ends the
// path (`lit`: with a radiance, in xyz; a path that meets none, as under a black
// sky, has no comb to sum); a surface scatters it (Fresnel / refract / TIR or
// Lambertian, dispersion collapse, Russian roulette).  Returns whether the path
// continues.
__device__ __forceinline__ bool shade_path(const TracerSmem& s, const SceneView& S, uint32_t bounce, PathState& P,
                                           float t, f3 n, uint32_t info, bool& lit, float xyz[3]) {
    const uint32_t kind = info >> 24;
    uint32_t valid = P.flags & 0xFFu;
    lit = false;
    if (kind != 1u) {
        float e;
        if (kind == 0u) e = s.p.background + ((s.p.has_horizon && P.d.y > 0.0f) ? s.p.horizon : 0.0f);
        else e = s.p.em_scale;
        lit = e != 0.0f || !(fabsf(P.tp) < __int_as_float(0x7f800000));
        if (lit) comb_xyz(s, P.u, P.tp, valid, e, xyz);
        return false;
    }
    const sc_material& m = S.mats[info & 0xFFFFu];
    Hit h;
    h.t = t;
    h.point = add(P.o, mul(P.d, t));
    h.normal = n;
    h.front_face = ((info >> 16) & 1u) != 0u;
    const float nh = m.kind == 1u ? glass_n(m.glass, s.p.spectral ? lane_lambda(P.u, 0) : 550.0f) : 1.0f;
    Rng r;
    r.state = P.rs;
    f3 nd;
    float w;
    scatter(m, P.d, h, nh, r, nd, w);
    P.tp *= w;
    if (m.kind == 1u && valid > 1u) valid = 1u;
    const uint32_t depth = bounce + 1u;
    bool survive = depth < s.p.max_depth;
    if (s.p.rr_start && depth >= s.p.rr_start) {
        const float qv = fminf(P.tp, 0.95f);
        if (!(r.f32() < qv)) survive = false;
        else P.tp = P.tp / qv;
    }
    P.o = h.point; P.d = nd; P.rs = r.state;
    P.flags = valid | (depth << 8);
    return survive;
}

// n / d and its remainder for a d whose `inv` = floor((2^32 - 1) / d) is known: the
// high word of n * inv is the quotient or one less.
struct FastDiv {
    uint32_t d, inv;
    __device__ __forceinline__ explicit FastDiv(uint32_t v) : d(v), inv(0xFFFFFFFFu / v) {}
    __device__ __forceinline__ uint32_t operator()(uint32_t n, uint32_t& rem) const {
        uint32_t q = __umulhi(n, inv);
        rem = n - q * d;
        if (rem >= d) { ++q; rem -= d; }
        return q;
    }
};

// Survivors of a warp on their way into the next ray queue: a ring of 64 in shared
// memory.  Full groups of 32 go out with one atomic and whole 128-byte lines, and
// no warp waits for another one of its CTA (compacting per CTA cost three barriers
// a bounce: 30 % of the stalls).
struct PathRing {
    float f[8][64];
    uint32_t u[3][64];
};
__device__ __forceinline__ void ring_write(const PathRing& ring, uint32_t head, uint32_t n, const RayQueue& out,
                                           uint32_t* count, uint32_t lane) {
    uint32_t g = 0;
    if (lane == 0) g = atomicAdd(count, n);
    g = __shfl_sync(0xffffffffu, g, 0) + lane;
    if (lane >= n) return;
    const uint32_t j = (head + lane) & 63u;
    out.ox[g] = ring.f[0][j]; out.oy[g] = ring.f[1][j]; out.oz[g] = ring.f[2][j];
    out.dx[g] = ring.f[3][j]; out.dy[g] = ring.f[4][j]; out.dz[g] = ring.f[5][j];
    out.tp[g] = ring.f[6][j]; out.u[g] = ring.f[7][j];
    out.rng[g] = ring.u[0][j]; out.id[g] = ring.u[1][j]; out.flags[g] = ring.u[2][j];
}

// One compacted bounce: each path's ray is intersected and shaded here, and the
// survivors are compacted into the next ray queue (no hit queue: the bounce that
// reads a ray intersects it, from the dense queue).
// GEN: the first bounce with no queue in: each path's primary ray is made here
// (stream key mix2(pixel, sample index), jittered through the pixel, hero-comb
// draw), intersected in place and shaded.  Paths of a wave are numbered
// sample-major (path i = sample s of wave pixel j with i = s * n_pixels + j):
// neighbouring threads trace neighbouring pixels, and the per-pixel sums read
// the results coalesced.  counts[1..] are zero at entry.
template <bool GEN>
__global__ void __launch_bounds__(kShadeThreads, kStageCtasPerSm) tr_shade(const TracerParams* __restrict__ gp, uint32_t bounce,
                                                          RayQueue q, RayQueue out,
                                                          uint32_t* counts, float* result, uint32_t first_pixel,
                                                          uint32_t n_pixels, uint32_t n_paths,
                                                          const uint32_t* __restrict__ base) {
    __shared__ TracerSmem s;
    __shared__ PathRing rings[kShadeThreads / 32];
    extern __shared__ __align__(16) unsigned char dyn[];
    if (GEN && blockIdx.x == 0 && threadIdx.x == 0) counts[0] = n_paths;
    const uint32_t n = GEN ? n_paths : counts[bounce];
    if (blockIdx.x * blockDim.x >= n) return;  // nothing queued for this CTA (late bounces)
    const SceneView S = load_tracer(gp, s, reinterpret_cast<sc_plane*>(dyn));
    const uint32_t lane = threadIdx.x & 31u;
    PathRing& ring = rings[threadIdx.x >> 5];
    const uint32_t b0 = GEN ? *base : 0u;
    const FastDiv per_sample(n_pixels), per_row(s.p.width);
    uint32_t head = 0, held = 0;  // the same in every lane
    for (uint32_t tile = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); tile < n; tile += gridDim.x * blockDim.x) {
        const uint32_t i = tile + lane;
        bool survive = false, lit = false;
        PathState P;
        float xyz[3] = {0.0f, 0.0f, 0.0f};
        if (i < n) {
            if (GEN) {
                uint32_t j, px;
                const uint32_t smp = per_sample(i, j), pixel = first_pixel + j, py = per_row(pixel, px);
                Rng r = Rng::make(mix2(pixel, b0 + smp), s.p.seed);
                const float fs = ((float)px + r.f32()) / (float)s.p.width;
                const float ft = 1.0f - ((float)py + r.f32()) / (float)s.p.height;
                P.u = r.f32();
                P.o = ld3(s.p.cam.origin);
                P.d = primary_dir(s.p.cam, fs, ft);
                P.rs = r.state; P.tp = 1.0f; P.id = i; P.flags = 4u;
            } else {
                P = read_path(q, i);
            }
            float t;
            f3 nrm;
            uint32_t info;
            trace_hit(s, S, P.o, P.d, t, nrm, info);
            survive = shade_path(s, S, GEN ? 0u : bounce, P, t, nrm, info, lit, xyz);
            if (GEN || lit) {
                float* o = result + 3 * (size_t)P.id;
                o[0] = xyz[0]; o[1] = xyz[1]; o[2] = xyz[2];
            }
        }
        const unsigned ball = __ballot_sync(0xffffffffu, survive);
        if (survive) {
            const uint32_t j = (head + held + __popc(ball & ((1u << lane) - 1u))) & 63u;
            ring.f[0][j] = P.o.x; ring.f[1][j] = P.o.y; ring.f[2][j] = P.o.z;
            ring.f[3][j] = P.d.x; ring.f[4][j] = P.d.y; ring.f[5][j] = P.d.z;
            ring.f[6][j] = P.tp; ring.f[7][j] = P.u;
            ring.u[0][j] = P.rs; ring.u[1][j] = P.id; ring.u[2][j] = P.flags;
        }
        held += __popc(ball);
        __syncwarp();
        if (held >= 32u) {
            ring_write(ring, head, 32u, out, counts + bounce + 1, lane);
            head += 32u;
            held -= 32u;
            __syncwarp();
        }
    }
    if (held) ring_write(ring, head, held, out, counts + bounce + 1, lane);
}

// The bounces after the compacted ones in one launch: each lane keeps a path in
// registers until it ends, and a warp with fewer than kTailLive paths claims new
// ones from the queue for its idle lanes (counter counts[max_depth + 1], zero
// at entry), whatever bounces the others are at.  Warps
// stay full without waiting for one another.  The same hit and shade code, so the
// image is unchanged.  Segments after each path's first tail bounce are added to
// counts[first + 1].  (16, 20, 24, 28, 32 lanes: accumulate(64) with its read-back 3.83,
// 3.82 to 3.87, 3.76 to 3.80, 3.80, 3.85 to 3.91 ms.)
constexpr uint32_t kTailLive = 24;
__global__ void __launch_bounds__(256, kStageCtasPerSm) tr_tail(const TracerParams* __restrict__ gp, uint32_t first,
                                                                RayQueue q, uint32_t* counts, float* result) {
    __shared__ TracerSmem s;
    extern __shared__ __align__(16) unsigned char dyn[];
    const uint32_t n = counts[first];
    if (blockIdx.x * blockDim.x >= n) return;
    const SceneView S = load_tracer(gp, s, reinterpret_cast<sc_plane*>(dyn));
    uint32_t* claim = counts + s.p.max_depth + 1;
    const uint32_t lane = threadIdx.x & 31u;
    // A claim is a quarter of a warp's share, 32 to 256 paths: one per refill made the
    // warps queue up at the counter (all bounces but the first here, 1280x720, 64 spp:
    // 4.29 ms).
    const uint32_t share = n / (4u * gridDim.x * (blockDim.x >> 5));
    const uint32_t step = share < 32u ? 32u : share > 256u ? 256u : share & ~31u;
    uint32_t segs = 0, next = 0, end = 0;  // next, end: what is left of the claim, the same in every lane
    bool alive = false, more = true;
    PathState P;
    for (;;) {
        const unsigned live = __ballot_sync(0xffffffffu, alive);
        const uint32_t m = __popc(live);
        if (more && m < kTailLive) {
            if (next == end) {
                uint32_t at = 0;
                if (lane == 0) at = atomicAdd(claim, step);
                next = min(__shfl_sync(0xffffffffu, at, 0), n);
                end = next + min(step, n - next);
                more = next < n;
            }
            const uint32_t i = next + __popc(~live & ((1u << lane) - 1u));
            if (!alive && i < end) {
                P = read_path(q, i);
                alive = true;
            }
            next = min(next + 32u - m, end);
        } else if (m == 0u) {
            break;
        }
        if (alive) {
            const uint32_t b = (P.flags >> 8) & 0xFFu;  // the bounce this path is at
            float t, xyz[3];
            f3 nrm;
            uint32_t info;
            bool lit;
            trace_hit(s, S, P.o, P.d, t, nrm, info);
            if (b > first) ++segs;  // counts[first] already holds the first tail bounce's rays
            alive = shade_path(s, S, b, P, t, nrm, info, lit, xyz);
            if (lit) {
                float* o = result + 3 * (size_t)P.id;
                o[0] = xyz[0]; o[1] = xyz[1]; o[2] = xyz[2];
            }
        }
    }
    for (int o = 16; o > 0; o >>= 1) segs += __shfl_xor_sync(0xffffffffu, segs, o);
    if (lane == 0 && segs) atomicAdd(counts + first + 1, segs);
}

// Per-pixel sample sum in sample order (tracer.rs:121-135), added to the running
// sum.  One thread per (pixel, channel) of the wave: consecutive threads read
// consecutive floats of each sample (coalesced), and each adds its samples in
// sample order.
__global__ void __launch_bounds__(256) tr_accumulate(uint32_t first_pixel, uint32_t n_pixels, uint32_t spp,
                                                     const float* __restrict__ result, float* sum,
                                                     const uint32_t* __restrict__ counts, uint32_t max_depth,
                                                     unsigned long long* segments) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j == 0) {
        unsigned long long t = 0;
        for (uint32_t b = 0; b < max_depth; ++b) t += counts[b];
        atomicAdd(segments, t);  // both wave chains add here
    }
    const uint32_t n = 3u * n_pixels;
    if (j >= n) return;
    float a = 0.0f;
#pragma unroll 16
    for (uint32_t s = 0; s < spp; ++s) a += result[(size_t)s * n + j];  // loads run ahead; adds in sample order
    sum[3u * (size_t)first_pixel + j] += a;
}

// AccumBuffer::mean (spectral-core/src/lib.rs:16-20): each sum divided by the
// sample count (an IEEE division, as the host would do it).
__global__ void __launch_bounds__(256) tr_mean(const float* __restrict__ sum, float* __restrict__ out, size_t n,
                                               float count) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        out[i] = sum[i] / count;
}

}  // namespace

cudaError_t launch_tracer_mean(const float* sum, float* out, size_t n, float count, int sms, cudaStream_t st) {
    const size_t blocks = std::min<size_t>((n + 255) / 256, (size_t)sms * 8);
    if (blocks == 0) return cudaSuccess;
    tr_mean<<<(unsigned)blocks, 256, 0, st>>>(sum, out, n, count);
    return cudaGetLastError();
}

size_t tracer_dyn_smem(uint32_t n_planes) { return (size_t)(n_planes ? n_planes : 1u) * sizeof(sc_plane); }

int tracer_grid(int sms) {
    int a = 0, b = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, tr_tail, 256, tracer_dyn_smem(SC_MAX_PLANES));
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, tr_shade<false>, kShadeThreads,
                                                  tracer_dyn_smem(SC_MAX_PLANES));
    int c = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&c, tr_shade<true>, kShadeThreads,
                                                  tracer_dyn_smem(SC_MAX_PLANES));
    int k = a < b ? a : b;
    k = k < c ? k : c;
    return sms * (k > 0 ? k : 1);
}

cudaError_t launch_tracer_wave(const TracerParams* d_params, const TracerLaunch& L, uint32_t first_pixel,
                               uint32_t n_pixels, cudaStream_t st) {
    const uint32_t n_paths = n_pixels * L.spp;
    const size_t dyn = tracer_dyn_smem(L.n_planes);
    // wavefront with compaction for the first bounces, then the tail in place;
    // the first bounce makes, intersects and shades the primary rays in one kernel
    // (where the caller does not say: two, or one for waves that the tail's warps
    // hold with few refills.  accumulate(64) at 1280x720, waves of 2^22 paths: one 3.28
    // ms, two 3.05, three 3.06; accumulate(4) at 333x187: 54, 60, 64 us.  One and two by
    // the wave's paths: the prism on its floor under a black sky 2^18 54 and 60 us, 2^19
    // 75 and 72, 2^20 102 and 98, 2^21 178 and 171, 2^22 285 and 274, under a bright one
    // 2^20 106 and 108, 2^21 197 and 188; glass under a sky, whose paths end after fewer
    // bounces, 2^20 92 and 98, 2^22 239 and 251)
    const uint32_t want = L.wave_bounces ? L.wave_bounces : n_paths <= (1u << 20) ? 1u : 2u;
    const uint32_t wave_bounces = L.max_depth < want ? L.max_depth : want;
    // bounce b intersects and shades the rays of bounce b and queues its
    // compacted survivors (ray queues alternate)
    for (uint32_t b = 0; b < wave_bounces; ++b) {
        const RayQueue& in = (b & 1u) ? L.qb : L.qa;
        const RayQueue& out = (b & 1u) ? L.qa : L.qb;
        if (b == 0) {
            // the first bounce makes its primary rays itself: no queue in; later
            // bounces (and the tail's claim counter) count from zero
            cudaError_t e = cudaMemsetAsync(L.counts + 1, 0, (L.max_depth + 1) * sizeof(uint32_t), st);
            if (e != cudaSuccess) return e;
            tr_shade<true><<<L.grid, kShadeThreads, dyn, st>>>(d_params, 0u, in, out, L.counts, L.result, first_pixel,
                                                              n_pixels, n_paths, L.d_base);
        } else {
            tr_shade<false><<<L.grid, kShadeThreads, dyn, st>>>(d_params, b, in, out, L.counts, L.result, 0u, 1u, 0u,
                                                               L.d_base);
        }
    }
    if (L.max_depth > wave_bounces)
        tr_tail<<<L.grid, 256, dyn, st>>>(d_params, wave_bounces, (wave_bounces & 1u) ? L.qb : L.qa, L.counts,
                                          L.result);
    tr_accumulate<<<(3 * n_pixels + 255) / 256, 256, 0, st>>>(first_pixel, n_pixels, L.spp, L.result, L.sum, L.counts,
                                                               L.max_depth, L.segments);
    return cudaGetLastError();
}

}  // namespace sc
