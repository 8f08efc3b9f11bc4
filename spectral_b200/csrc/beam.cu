// Photon-beam estimator: render_volumetric_scene + splat_transverse
// (spectral-core/src/volume.rs:170-329).
//
// Same emission and bounce loop as the point estimator, but no per-segment
// distance draws: every segment (including the escaping one, length max_dist)
// is marched in M = ceil(2 x projected pixel length) + 1 deterministic steps
// (ceil(80 x length) when an end point is off frame; 1 <= M <= 4096).  Each step
// at distance (k + 1/2) * len / M is connected to the camera with the point
// estimator's weight (HG phase x transmittance / d^2) times the step length, and
// deposited over a tent footprint whose radius is the projected beam radius
// 0.03 (clamped to [1.5, 24] px, 1 px when the offset point leaves the frame);
// the tent weights are renormalised over the covered pixels, so a footprint
// clipped by the frame edge keeps its energy.
//
// GPU shape.  A photon has up to max_bounces segments of up to 4096 steps each,
// so per-photon work varies by three orders of magnitude.  Each warp traces a
// small group of photons (one per lane) and only records segments (origin,
// direction, step length, power, M) in a per-warp shared-memory buffer; when the
// buffer fills (and when the group is done) the warp marches all buffered steps
// as one flat list: 32 steps at a time are set up one per lane (step t found by a
// binary search over the buffer's prefix sums of M; the step's own lane adds up
// its tent sum, row by row like the reference), then splatted in march order
// through a window of pixels that the lanes hold in registers (window_march).
// Film width and height are below 2^16 (corners are packed into one word).
//
// Bound: instruction issue (0.71 of the issue slots at 24 warps per SM, which
// registers limit: 80, with 202 B of spills; 4 CTAs per SM spill more and are 4-8 %
// slower on most films).  Of
// the 38 ms that 2^18 photons take on the 800x800 XYZ film, the setup of the
// 470 M steps is 13 ms and the windows are the rest, ~75 warp instructions for
// each of the 279 M steps in frame.  Splatting step by step over each box, with
// one atomic per cell for every one or two steps, took 164-168 ms: 446 warp
// instructions per step.
//
// |d| is d2 * rsqrt(d2) (within 2 ulp), |d| / r a multiply by 1/r, the tent's
// two sums and the deposit's rounding are fused, and the HG power 1.5 is
// x * sqrt(x), so a deposit can differ from the reference's in the last few bits.
#include "photon_trace.cuh"

namespace sc {

namespace {

constexpr float kBeamRadius = 0.03f;  // R_BEAM (volume.rs:172)
constexpr uint32_t kMaxSteps = 4096u;

struct BeamSeg { f3 o, d; float ds, power; uint32_t m, lane; };
// One march step ready to splat, in the order the warp reads it (four 16-byte
// broadcasts; what the packed arithmetic takes is stored twice): footprint
// centre (y negated) and -1 / radius in pixels, 1 / tent sum over the box, and
// the step's colour (XYZ film) or weight and bin (spectral film) times the
// film's fixed-point scale (a power of two: exact, so a pixel's deposit
// fixed_scaled(c * w) is to_fixed(c_unscaled * w, scale)).  The footprint box is
// [x0, x0 + bw) x [y0, y0 + bh).
struct alignas(16) StepRec {
    float cx;
    uint32_t x0y0;        // x0 | y0 << 16
    float ncy[2], nir[2], inv_wsum[2], c0[2], c1[2], c2[2];
    uint32_t bin;
    uint32_t box;         // bw | bh << 16 (<= 50); 0: whole colour on the centre pixel
};
static_assert(sizeof(StepRec) == 64, "step record layout");
// How a step is splatted (the setup's verdict, kept by its lane): not in frame;
// by the 8x8 or the 16x16 window; on its own (a larger box, one at kWindowEnd, a deposit
// of 2^23 quanta or more, or an empty tent).
enum : uint32_t { kStepNone = 0u, kStepWin8 = 1u, kStepWin16 = 2u, kStepAlone = 3u };
// Boxes of the windows' steps start below this column and row, so two of them differ by
// less than 2^16 - 16 and window_march can compare their corners modulo 2^16 (only a
// film of more than 65,520 pixels on a side has others; they go on their own).
constexpr int kWindowEnd = 65536 - 16;
constexpr uint32_t kBeamSegs = 64;
struct alignas(16) BeamWarpSmem {
    BeamSeg seg[kBeamSegs];
    uint32_t start[kBeamSegs + 4];  // exclusive prefix of m; start[kBeamSegs] = total
    float4 payload[32];             // per-lane CMF (x, y, z) and bin of its photon
    StepRec step[32];               // 32 march steps set up for splatting
};

// Work counters of an instrumented launch: segments, march steps, steps in
// frame (and not occluded), footprint pixels deposited.
struct BeamCounts { unsigned long long segments, steps, in_frame, deposits; };

__host__ __device__ __forceinline__ size_t beam_offset(const PhotonParams& p, uint32_t mask_words) {
    const size_t b = p.n_prims * sizeof(sc_primitive) + p.n_planes * sizeof(sc_plane) +
                     p.n_mats * sizeof(sc_material) + 3 * kTableN * sizeof(float) + mask_words * sizeof(uint32_t);
    return (b + 15u) & ~size_t(15);
}

// March count of one segment (volume.rs:255-266).
__device__ __forceinline__ uint32_t march_count(const PhotonParams& p, f3 o, f3 d, float seg) {
    const f3 pend = add(o, mul(d, seg));
    float s0, t0, s1, t1;
    float mf;
    uint32_t extra;
    if (project(p.proj, o, s0, t0) && project(p.proj, pend, s1, t1)) {
        const float dx = (s1 - s0) * (float)p.width;
        const float dy = (t1 - t0) * (float)p.height;
        mf = ceilf(sqrtf(dx * dx + dy * dy) * 2.0f);
        extra = 1u;
    } else {
        mf = ceilf(seg * 80.0f);
        extra = 0u;
    }
    if (!(mf > 0.0f)) mf = 0.0f;
    mf = fminf(mf, (float)kMaxSteps);
    const uint32_t m = (uint32_t)mf + extra;
    return m < 1u ? 1u : (m > kMaxSteps ? kMaxSteps : m);
}

// Tent weight max(1 - |d| / r, 0); the division is a multiply by 1/r (within
// an ulp of the reference's quotient), both sums fused multiply-adds.
__device__ __forceinline__ float tent(float dx2, float dy, float inv_r) {
    const float d2 = __fmaf_rn(dy, dy, dx2);
    const float d = d2 > 0.0f ? d2 * rsqrtf(d2) : 0.0f;  // |d| within 2 ulp
    return fmaxf(__fmaf_rn(-d, inv_r, 1.0f), 0.0f);
}

// Two f32 operations in one instruction, each rounded as on its own (a packed
// multiply whose only use is a packed add is fused by the assembler: such pairs
// are written as fma2).
__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// Two tents (the arithmetic of tent()): a squared distance of 0 is raised to
// 1e-35, whose tent is 1 as well.
__device__ __forceinline__ uint64_t tent2(uint64_t dx2, uint64_t dy, uint64_t nir, uint64_t one) {
    float a, b;
    unpack2(fma2(dy, dy, dx2), a, b);
    a = fmaxf(a, 1e-35f);
    b = fmaxf(b, 1e-35f);
    unpack2(fma2(mul2(pack2(a, b), pack2(rsqrt_approx(a), rsqrt_approx(b))), nir, one), a, b);
    return pack2(fmaxf(a, 0.0f), fmaxf(b, 0.0f));
}

// Fixed-point value of an already scaled deposit: the same integer as
// to_fixed(x, scale) for y = x * scale (scale a power of two), with the common case
// (0 <= y < 2^23, by its bits) in two ALU operations.
__device__ __forceinline__ unsigned long long fixed_scaled(float y) {
    if (__float_as_uint(y) < 0x4B000000u) return (unsigned long long)(__float_as_uint(y + 8388608.0f) - 0x4B000000u);
    return to_fixed(y, 1.0f);
}

// Dirty bits of the tiles under a footprint box, set by the step's own lane
// during the setup (most are already set, and mark_tile reads before it
// writes): its corners' tiles when it spans at most 2 tiles per axis, else
// every tile.
__device__ __forceinline__ void mark_box(const PhotonParams& p, uint32_t* smask, int x0, int y0, int x1, int y1) {
    const int tx0 = x0 >> 3, ty0 = y0 >> 3, tx1 = x1 >> 3, ty1 = y1 >> 3;
    if (tx1 - tx0 <= 1 && ty1 - ty0 <= 1) {
        mark_tile(p, smask, (uint32_t)(ty0 * (int)p.tiles_x + tx0));
        mark_tile(p, smask, (uint32_t)(ty0 * (int)p.tiles_x + tx1));
        mark_tile(p, smask, (uint32_t)(ty1 * (int)p.tiles_x + tx0));
        mark_tile(p, smask, (uint32_t)(ty1 * (int)p.tiles_x + tx1));
    } else {
        for (int ty = ty0; ty <= ty1; ++ty)
            for (int tx = tx0; tx <= tx1; ++tx) mark_tile(p, smask, (uint32_t)(ty * (int)p.tiles_x + tx));
    }
}

// The pixel that takes the whole colour of a step whose tent sum is 0.
__device__ __forceinline__ uint32_t centre_pixel(float c, uint32_t n) {
    return (uint32_t)min(max((int)roundf(c), 0), (int)n - 1);
}

// Per-step setup (volume.rs:268-300), one lane per step: the step point, its
// projection, z-test, camera-connection weight and projected beam radius.
template <bool SPEC, bool COUNT>
__device__ __forceinline__ uint32_t beam_step(const PhotonParams& p, uint32_t* smask, const BeamSeg& B, float4 pay,
                                              uint32_t k, StepRec& R, BeamCounts& cnt) {
    const float dist = ((float)k + 0.5f) * B.ds;
    const f3 q = add(B.o, mul(B.d, dist));
    float s, t;
    if (!project(p.proj, q, s, t)) return kStepNone;
    const uint32_t px = min((uint32_t)(s * (float)p.width), p.width - 1u);
    const uint32_t py = min((uint32_t)((1.0f - t) * (float)p.height), p.height - 1u);
    const f3 to = sub(p.proj.o, q);
    const float dd = fmaxf(length(to), 1e-3f);
    if (p.zbuf && !(dd < p.zbuf[py * p.width + px])) return kStepNone;
    if (COUNT) ++cnt.in_frame;
    const f3 view = vdiv(to, dd);
    // phase_hg with den^1.5 as den * sqrt(den)
    const float den = fmaxf(1.0f + p.g * p.g - 2.0f * p.g * dot(B.d, view), 1e-6f);
    const float phase = (1.0f - p.g * p.g) / (4.0f * 3.14159265358979323846f * (den * sqrtf(den)));
    const float trans = expf(-p.sigma_t * dd);
    const float weight = B.power * p.sigma_s * phase * trans / (dd * dd) * B.ds;
    f3 perp = mk(-view.z, 0.0f, view.x);  // view x (0, 1, 0)
    if (dot(perp, perp) < 1e-8f) perp = mk(0.0f, view.z, -view.y);  // view x (1, 0, 0)
    perp = mul(normalize(perp), kBeamRadius);
    float s2, t2, radius = 1.0f;
    if (project(p.proj, add(q, perp), s2, t2)) {
        const float dpx = (s2 - s) * (float)p.width, dpy = (t2 - t) * (float)p.height;
        radius = fminf(fmaxf(sqrtf(dpx * dpx + dpy * dpy), 1.5f), 24.0f);
    }
    // splat_transverse (volume.rs:174-186): centre, radius and box in pixels
    const float cx = s * (float)p.width - 0.5f, cy = (1.0f - t) * (float)p.height - 0.5f;
    const float r = fmaxf(radius, 0.5f), inv_r = 1.0f / r;
    int x0 = (int)fmaxf(floorf(cx - r), 0.0f), x1 = min(max((int)ceilf(cx + r), 0), (int)p.width - 1);
    int y0 = (int)fmaxf(floorf(cy - r), 0.0f), y1 = min(max((int)ceilf(cy + r), 0), (int)p.height - 1);
    // the box's outer columns and rows lie at least r away unless the film clips
    // it: their tents are 0, so they are left out (r_out: beyond any rounding)
    const float r_out = r * 1.00001f;
    x0 += cx - (float)x0 > r_out;
    x1 -= (float)x1 - cx > r_out;
    y0 += cy - (float)y0 > r_out;
    y1 -= (float)y1 - cy > r_out;
    const uint32_t bw = (uint32_t)max(x1 - x0 + 1, 0), bh = (uint32_t)max(y1 - y0 + 1, 0);
    float c0, c1 = 0.0f, c2 = 0.0f;
    if (SPEC) { c0 = weight * p.scale; }
    else { c0 = pay.x * weight * p.scale; c1 = pay.y * weight * p.scale; c2 = pay.z * weight * p.scale; }
    // the tent sum over the box, row by row as the reference adds it
    float wsum = 0.0f;
    if (bw <= 8u) {  // two columns at a time; those beyond the box far away: tent 0
        const uint64_t nir = pack2(-inv_r, -inv_r), one = pack2(1.0f, 1.0f);
        uint64_t dx2[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float a = (float)(x0 + 2 * k) - cx, b = (float)(x0 + 2 * k + 1) - cx;
            dx2[k] = pack2(x0 + 2 * k <= x1 ? a * a : 1e30f, x0 + 2 * k + 1 <= x1 ? b * b : 1e30f);
        }
        for (int py = y0; py <= y1; ++py) {
            const float dy = (float)py - cy;
            const uint64_t dy2 = pack2(dy, dy);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (2u * k < bw) {
                    float a, b;
                    unpack2(tent2(dx2[k], dy2, nir, one), a, b);
                    wsum += a;
                    wsum += b;
                }
            }
        }
    } else {
        for (int py = y0; py <= y1; ++py) {
            const float dy = (float)py - cy;
            for (int px = x0; px <= x1; ++px) {
                const float dx = (float)px - cx;
                wsum += tent(dx * dx, dy, inv_r);
            }
        }
    }
    const bool lit = wsum > 0.0f;
    if (!COUNT) {
        if (lit) mark_box(p, smask, x0, y0, x1, y1);
        else mark_tile(p, smask, film_tile(centre_pixel(cx, p.width), centre_pixel(cy, p.height), p.tiles_x));
    }
    const float inv = lit ? 1.0f / wsum : 0.0f;
    R.cx = cx;
    R.x0y0 = (uint32_t)x0 | ((uint32_t)y0 << 16);
    R.ncy[0] = R.ncy[1] = -cy;
    R.nir[0] = R.nir[1] = -inv_r;
    R.inv_wsum[0] = R.inv_wsum[1] = inv;
    R.c0[0] = R.c0[1] = c0;
    R.c1[0] = R.c1[1] = c1;
    R.c2[0] = R.c2[1] = c2;
    R.bin = __float_as_uint(pay.w);
    R.box = lit ? bw | (bh << 16) : 0u;
    // every tent is at most 1, so no deposit of the step reaches 2^23 quanta
    // where this holds (and the colours are not negative or NaN)
    const bool small = lit && c0 >= 0.0f && c1 >= 0.0f && c2 >= 0.0f &&
                       fmaxf(c0, fmaxf(c1, c2)) * inv < 8388000.0f;
    const uint32_t side = x0 < kWindowEnd && y0 < kWindowEnd ? max(bw, bh) : 17u;
    return small && side <= 8u ? kStepWin8 : (small && side <= 16u ? kStepWin16 : kStepAlone);
}

// Add one footprint pixel's share (w = tent / wsum) to the film.
template <bool SPEC>
__device__ __forceinline__ void deposit_pixel(const PhotonParams& p, uint32_t px, uint32_t py, const StepRec& R,
                                              float w) {
    unsigned long long* c = p.film + film_cell(px, py, p.tiles_x, SPEC ? p.channels : 3u, SPEC ? R.bin : 0u);
    if (SPEC) {
        red_u64(c, fixed_scaled(R.c0[0] * w));
    } else {
        red_u64(c, fixed_scaled(R.c0[0] * w));
        red_u64(c + kTilePixels, fixed_scaled(R.c1[0] * w));
        red_u64(c + 2 * kTilePixels, fixed_scaled(R.c2[0] * w));
    }
}

// The march steps of records [0, n), whose boxes are at most N x N pixels,
// deposited through a sliding window.  The footprint of a march moves
// by about half a pixel per step, so a pixel takes part in ten or so consecutive
// steps.  Each lane holds the fixed-point sums of N * N / 32 pixels in registers:
// the pixels of its residue class (x mod N, y mod N) inside an N x N window that
// holds the step's box.  The window moves only when a box leaves it (and then as
// far as the box allows, in the direction of the march), and only the pixels that
// leave the window are added to the film: one atomic per cell and visit instead of
// one per cell and step or two.  The film's sums do not depend on the order.  Pixels of the window
// outside the footprint have tent 0, and so have those outside the film, which
// are placed far away.
//
// A deposit y in [0, 2^23) is rounded by adding 2^23: the sum's bits are
// 0x4B000000 + the integer.  The sums add those bits as they are, and the bias
// (the same for all pixels: one 0x4B000000 per step) comes off when a pixel
// leaves: 32 steps of integers below 2^23 fit 32 bits.
template <bool SPEC, int N>
__device__ __forceinline__ void window_march(const PhotonParams& p, const BeamWarpSmem& ws, uint32_t n,
                                             uint32_t lane) {
    constexpr int P = N * N / 32, ROWS = 32 / N, CH = SPEC ? 1 : 3;
    constexpr float kFar = 1e15f;
    const uint32_t lx = lane & (N - 1), ly = lane / N;
    uint32_t acc[P][CH], bias = 0u;
#pragma unroll
    for (int k = 0; k < P; ++k)
#pragma unroll
        for (int c = 0; c < CH; ++c) acc[k][c] = 0u;
    const uint64_t one = pack2(1.0f, 1.0f), magic = pack2(8388608.0f, 8388608.0f);
    uint32_t wxy = 0u, bin = 0u;  // window corner x | y << 16, bin of its sums (spectral films)
    uint32_t px = 0u, py[P];      // this lane's pixels
    float fpx = 0.0f;
    uint64_t fpy[P / 2];
#pragma unroll
    for (int k = 0; k < P; ++k) py[k] = 0u;
#pragma unroll
    for (int k = 0; k < P / 2; ++k) fpy[k] = 0ull;
    // The k-th pixel's sums to the film.
    auto leave = [&](int k) {
        bool any = false;
#pragma unroll
        for (int c = 0; c < CH; ++c) any |= acc[k][c] != bias;
        if (any) {
            unsigned long long* cell = p.film + film_cell(px, py[k], p.tiles_x, SPEC ? p.channels : 3u, SPEC ? bin : 0u);
#pragma unroll
            for (int c = 0; c < CH; ++c) {
                atomicAdd(cell + c * kTilePixels, (unsigned long long)(acc[k][c] - bias));
                acc[k][c] = bias;
            }
        }
    };
    for (uint32_t j = 0; j < n; ++j) {
        const bool open = j != 0u;
        const ulonglong2* rec = reinterpret_cast<const ulonglong2*>(&ws.step[j]);
        const ulonglong2 q0 = rec[0], q1 = rec[1], q2 = rec[2], q3 = rec[3];
        const uint32_t xy = (uint32_t)(q0.x >> 32), nbin = (uint32_t)q3.y, box = (uint32_t)(q3.y >> 32);
        // the box lies in the window where both halves of xy - wxy are within
        // [0, N - side]: neither they nor the slack left have a sign bit (corners
        // differ by less than 2^16 - N: kWindowEnd)
        const uint32_t at = xy - wxy, slack = (uint32_t)(N | (N << 16)) - box - at;
        if (((at | slack) & 0x80008000u) || !open || (SPEC && nbin != bin)) {
            const uint32_t x0 = xy & 0xFFFFu, y0 = xy >> 16, bw = box & 0xFFFFu, bh = box >> 16;
            uint32_t wx = wxy & 0xFFFFu, wy = wxy >> 16;
            if (!open || x0 + bw > wx + N) wx = x0;
            else if (x0 < wx) wx = x0 + bw > N ? x0 + bw - N : 0u;
            if (!open || y0 + bh > wy + N) wy = y0;
            else if (y0 < wy) wy = y0 + bh > N ? y0 + bh - N : 0u;
            const uint32_t npx = wx + ((lx - wx) & (N - 1));
            const bool column = npx != px || (SPEC && nbin != bin);
            uint32_t npy[P];
#pragma unroll
            for (int k = 0; k < P; ++k) {
                npy[k] = wy + ((ly + (uint32_t)(k * ROWS) - wy) & (N - 1));
                if (open && (column || npy[k] != py[k])) leave(k);
                py[k] = npy[k];
            }
            wxy = wx | (wy << 16);
            bin = nbin;
            px = npx;
            fpx = px < p.width ? (float)px : kFar;
#pragma unroll
            for (int k = 0; k < P / 2; ++k)
                fpy[k] = pack2(py[2 * k] < p.height ? (float)py[2 * k] : kFar,
                               py[2 * k + 1] < p.height ? (float)py[2 * k + 1] : kFar);
        }
        const float dx = fpx - __uint_as_float((uint32_t)q0.x), dx2 = dx * dx;
        const uint64_t dx22 = pack2(dx2, dx2);
#pragma unroll
        for (int k = 0; k < P / 2; ++k) {
            const uint64_t w = mul2(tent2(dx22, add2(fpy[k], q0.y), q1.x, one), q1.y);
            float a, b;
            unpack2(fma2(q2.x, w, magic), a, b);
            acc[2 * k][0] += __float_as_uint(a);
            acc[2 * k + 1][0] += __float_as_uint(b);
            if (!SPEC) {
                unpack2(fma2(q2.y, w, magic), a, b);
                acc[2 * k][CH - 2] += __float_as_uint(a);
                acc[2 * k + 1][CH - 2] += __float_as_uint(b);
                unpack2(fma2(q3.x, w, magic), a, b);
                acc[2 * k][CH - 1] += __float_as_uint(a);
                acc[2 * k + 1][CH - 1] += __float_as_uint(b);
            }
        }
        bias += 0x4B000000u;
    }
#pragma unroll
    for (int k = 0; k < P; ++k) leave(k);
}

// splat_transverse (volume.rs:174-218) by the whole warp, its tent sum already
// known: lanes cover the footprint box (rows packed 32 / width at a time, or
// 32-column chunks of one row for boxes wider than 32) and deposit their pixels'
// renormalised shares (the step's lane marked the tiles under the box).
template <bool SPEC, bool COUNT>
__device__ __forceinline__ void splat_warp(const PhotonParams& p, const StepRec& R, uint32_t lane, BeamCounts& cnt) {
    const float cx = R.cx, cy = -R.ncy[0];
    if (R.box == 0u) {  // empty tent sum: the whole colour to the centre pixel
        if (lane == 0) {
            if (COUNT) { ++cnt.deposits; return; }
            deposit_pixel<SPEC>(p, centre_pixel(cx, p.width), centre_pixel(cy, p.height), R, 1.0f);
        }
        return;
    }
    const int x0 = (int)(R.x0y0 & 0xFFFFu), y0 = (int)(R.x0y0 >> 16);
    const int bw = (int)(R.box & 0xFFFFu), bh = (int)(R.box >> 16), rows = bw <= 32 ? 32 / bw : 1;
    const int x1 = x0 + bw - 1, y1 = y0 + bh - 1;
    const float inv_r = -R.nir[0], inv = R.inv_wsum[0];
    const int lrow = bw <= 32 ? (int)lane / bw : 0;
    const int lcol = (int)lane - lrow * bw;
    if (lrow >= rows) return;
    const int chunks = bw <= 32 ? 1 : (bw + 31) / 32;
    for (int ch = 0; ch < chunks; ++ch) {
        const int px = x0 + ch * 32 + lcol;
        if (px > x1) break;
        const float dx = (float)px - cx, dx2 = dx * dx;
        for (int py = y0 + lrow; py <= y1; py += rows) {
            const float w = tent(dx2, (float)py - cy, inv_r) * inv;
            if (w > 0.0f) {
                if (COUNT) ++cnt.deposits;
                else deposit_pixel<SPEC>(p, (uint32_t)px, (uint32_t)py, R, w);
            }
        }
    }
}

// March every step of the n buffered segments as one flat list: 32 steps at a
// time are set up one per lane, then splatted one at a time by the whole warp.
template <bool SPEC, bool COUNT>
__device__ __forceinline__ void beam_flush(const PhotonParams& p, BeamWarpSmem& ws, uint32_t n, uint32_t* smask,
                                           BeamCounts& cnt) {
    const uint32_t lane = threadIdx.x & 31u;
    __syncwarp();
    const uint32_t m0 = lane < n ? ws.seg[lane].m : 0u;
    const uint32_t m1 = lane + 32u < n ? ws.seg[lane + 32u].m : 0u;
    uint32_t i0 = m0, i1 = m1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t a = __shfl_up_sync(0xffffffffu, i0, o), b = __shfl_up_sync(0xffffffffu, i1, o);
        if ((int)lane >= o) { i0 += a; i1 += b; }
    }
    const uint32_t tot0 = __shfl_sync(0xffffffffu, i0, 31), tot1 = __shfl_sync(0xffffffffu, i1, 31);
    ws.start[lane] = i0 - m0;
    ws.start[lane + 32u] = tot0 + i1 - m1;
    if (lane == 0) ws.start[kBeamSegs] = tot0 + tot1;
    __syncwarp();
    const uint32_t total = tot0 + tot1;
    if (COUNT && lane == 0) { cnt.segments += n; cnt.steps += total; }
    for (uint32_t t0 = 0; t0 < total; t0 += 32u) {
        const uint32_t t = t0 + lane;
        uint32_t how = kStepNone;
        StepRec R;
        if (t < total) {
            uint32_t lo = 0, hi = n;  // start[lo] <= t < start[hi]
            while (hi - lo > 1u) {
                const uint32_t mid = (lo + hi) >> 1;
                if (ws.start[mid] <= t) lo = mid; else hi = mid;
            }
            const BeamSeg B = ws.seg[lo];
            how = beam_step<SPEC, COUNT>(p, smask, B, ws.payload[B.lane], t - ws.start[lo], R, cnt);
        }
        // records: the windows' steps first, in march order, then the others
        const unsigned win16 = COUNT ? 0u : __ballot_sync(0xffffffffu, how == kStepWin16);
        const unsigned win = COUNT ? 0u : win16 | __ballot_sync(0xffffffffu, how == kStepWin8);
        const unsigned alone = __ballot_sync(0xffffffffu, how != kStepNone) & ~win;
        const uint32_t n_win = __popc(win), n_all = n_win + __popc(alone);
        const unsigned below = (1u << lane) - 1u;
        if (how != kStepNone)
            ws.step[(win >> lane) & 1u ? __popc(win & below) : n_win + __popc(alone & below)] = R;
        __syncwarp();
        if (!COUNT) {
            // one window size per 32 steps, the larger where any step needs it
            if (win16) window_march<SPEC, 16>(p, ws, n_win, lane);
            else if (win) window_march<SPEC, 8>(p, ws, n_win, lane);
        }
        for (uint32_t j = n_win; j < n_all; ++j) splat_warp<SPEC, COUNT>(p, ws.step[j], lane, cnt);
        __syncwarp();
    }
}

// 32 photons of one warp (lane = photon): transport with segments recorded,
// then marched by beam_flush.
template <bool SPEC, bool COUNT>
__device__ __forceinline__ void trace_beam_warp(const PhotonParams& p, const SceneView& S, const float* cmf,
                                                uint32_t idx, bool valid, uint32_t* smask, BeamWarpSmem& ws,
                                                BeamCounts& cnt) {
    const uint32_t lane = threadIdx.x & 31u;
    Rng r = Rng::make(idx, p.seed);
    const float r1 = r.f32();
    const float r2 = r.f32();
    f3 o = add(add(p.corner, mul(p.bu, r1)), mul(p.bv, r2));
    const float lambda = p.lambda_min + p.lambda_range * r.f32();
    float cx = 0.0f, cy = 0.0f, cz = 0.0f;
    uint32_t bin = 0;
    photon_payload(p, cmf, lambda, cx, cy, cz, bin, SPEC);
    ws.payload[lane] = make_float4(cx, cy, cz, __uint_as_float(bin));
    f3 d = p.bdir;
    float power = 1.0f;
    bool alive = valid;
    uint32_t n = 0, n_glass = 0xFFFFFFFFu;
    float n_cached = 1.0f;
    for (uint32_t b = 0;; ++b) {
        const unsigned live = b < p.max_bounces ? __ballot_sync(0xffffffffu, alive) : 0u;
        // one flush site (keeps beam_flush inlined): when the buffer cannot take
        // another 32 segments, and once when the 32 photons are done
        if (n > kBeamSegs - 32u || (!live && n)) {
            beam_flush<SPEC, COUNT>(p, ws, n, smask, cnt);
            n = 0;
        }
        if (!live) break;
        Hit h;
        uint32_t mi = 0;
        bool any = false;
        if (alive) {
            any = scene_hit(S, o, d, h, mi);
            const float seg = any ? h.t : p.max_dist;
            const uint32_t m = march_count(p, o, d, seg);
            BeamSeg& B = ws.seg[n + __popc(live & ((1u << lane) - 1u))];
            B.o = o; B.d = d; B.ds = seg / (float)m; B.power = power; B.m = m; B.lane = lane;
        }
        n += __popc(live);
        if (alive) {
            if (any) {
                const sc_material& mt = S.mats[mi];
                float nh = 1.0f;
                if (mt.kind == 1u) {
                    if (mt.glass != n_glass) {
                        n_cached = glass_n(mt.glass, p.spectral ? lambda : 550.0f);
                        n_glass = mt.glass;
                    }
                    nh = n_cached;
                }
                f3 nd;
                float w;
                scatter(mt, d, h, nh, r, nd, w);
                power *= w;
                o = h.point;
                d = nd;
            } else {
                alive = false;
            }
        }
    }
}

template <bool SPEC>
__global__ void __launch_bounds__(256, 3) beam_kernel(const PhotonParams p, uint32_t mask_words) {
    extern __shared__ __align__(16) unsigned char smem[];
    const float* cmf;
    uint32_t* smask;
    const SceneView S = load_scene(p, smem, &cmf, &smask, mask_words);
    BeamWarpSmem* ws = reinterpret_cast<BeamWarpSmem*>(smem + beam_offset(p, mask_words));
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    BeamCounts cnt = {0, 0, 0, 0};
    // The whole warp marches, however few photons it traced, so a warp takes
    // groups small enough for each to have about 8 of them (up to 32 photons):
    // with 32 a launch of 2^18 photons was 2.3 groups per warp, a third of the
    // last round idle, and one of 1500 photons ran on 47 warps.
    const uint32_t group = min(32u, max(1u, p.photon_count / (warps * 8u)));
    for (uint64_t at = (uint64_t)(blockIdx.x * (blockDim.x >> 5) + warp) * group; at < p.photon_count;
         at += (uint64_t)warps * group) {
        const uint32_t base = (uint32_t)at;
        trace_beam_warp<SPEC, false>(p, S, cmf, p.photon_base + base + lane,
                                     lane < group && lane < p.photon_count - base, smask, ws[warp], cnt);
    }
    if (smask) {
        __syncthreads();
        for (uint32_t w = threadIdx.x; w < mask_words; w += blockDim.x)
            if (smask[w]) atomicOr(p.flags + w, smask[w]);
    }
}

// Instrumented pass: same transport and march, no film writes; sums the work
// counters into out[0..4] = photons, segments, steps, in-frame steps, deposits.
__global__ void __launch_bounds__(256, 3) beam_count_kernel(const PhotonParams p, unsigned long long* out) {
    extern __shared__ __align__(16) unsigned char smem[];
    const float* cmf;
    const SceneView S = load_scene(p, smem, &cmf);
    BeamWarpSmem* ws = reinterpret_cast<BeamWarpSmem*>(smem + beam_offset(p, 0));
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    BeamCounts cnt = {0, 0, 0, 0};
    unsigned long long ph = 0;
    for (uint32_t base = (blockIdx.x * (blockDim.x >> 5) + warp) * 32u; base < p.photon_count; base += warps * 32u) {
        trace_beam_warp<false, true>(p, S, cmf, p.photon_base + base + lane, base + lane < p.photon_count, nullptr,
                                        ws[warp], cnt);
        ph += base + lane < p.photon_count;
    }
    unsigned long long v[5] = {ph, cnt.segments, cnt.steps, cnt.in_frame, cnt.deposits};
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        for (int o = 16; o > 0; o >>= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
        if (lane == 0 && v[i]) atomicAdd(out + i, v[i]);
    }
}

using BeamKernelFn = void (*)(const PhotonParams, uint32_t);

BeamKernelFn beam_fn(bool spec) { return spec ? beam_kernel<true> : beam_kernel<false>; }

size_t beam_smem(const PhotonParams& p, uint32_t mask_words) {
    return beam_offset(p, mask_words) + 8 * sizeof(BeamWarpSmem);
}

}  // namespace

int beam_occupancy_blocks(const LaunchShape& shape, bool spectral, size_t smem) {
    return occupancy_blocks(reinterpret_cast<const void*>(beam_fn(spectral)), (int)shape.block,
                            smem + 16 + 8 * sizeof(BeamWarpSmem));
}

cudaError_t launch_beam_count(const PhotonParams& p, unsigned long long* out, uint32_t grid, cudaStream_t s) {
    if (p.photon_count == 0) return cudaSuccess;
    const uint32_t need = (p.photon_count + 255u) / 256u;
    const size_t smem = beam_smem(p, 0);
    if (smem > 48 * 1024)
        allow_max_smem(reinterpret_cast<const void*>(beam_count_kernel));
    beam_count_kernel<<<need < grid ? need : grid, 256, smem, s>>>(p, out);
    return cudaGetLastError();
}

cudaError_t launch_beam(const PhotonParams& p, const LaunchShape& shape, cudaStream_t s) {
    if (p.photon_count == 0) return cudaSuccess;
    const uint32_t mw = photon_mask_words(p);
    const bool spec = p.channels != 3u || p.bins != 0u;
    const uint32_t need = (p.photon_count - 1u) / 8u + 1u;  // at least one photon per warp
    const uint32_t grid = need < shape.grid ? need : shape.grid;
    const size_t smem = beam_smem(p, mw);  // the scene may have grown since the film was created
    if (smem > 48 * 1024) allow_max_smem(reinterpret_cast<const void*>(beam_fn(spec)));
    beam_fn(spec)<<<grid, 256, smem, s>>>(p, mw);
    return cudaGetLastError();
}

}  // namespace sc
