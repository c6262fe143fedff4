// render.cu -- the per-sample path loop: pathTrace and the pixel loop of the reference
// (src/main.cpp:69-204, 323-365), with a counter-based per-pixel RNG instead of the one global
// std::mt19937 stream, and the material extensions the benchmark scenes need (per-triangle
// albedo, emitters, mirrors; the reference has albedo 0.8 and no emitters).
//
// One persistent kernel (k_paths) traces every (pixel, sample) path: a warp's lanes hold 32 paths
// at different bounces, walk the tree and test leaves together (trace_warp.cuh), and lanes whose
// ray is done are shaded together -- emission, next direction, roulette -- and go on with their next
// ray or a new path. Each path's radiance goes to a buffer, and k_sum adds a pixel's samples in
// sample order (the reference's loop order), so images do not depend on the schedule.
// RT_RENDER_PLAIN and RT_RENDER_WAVEFRONT differ in nothing but the paths per launch
// (rt_wavefront_params). Scenes of a batched build (rt_render_batch) are rendered by the same
// launch: a path starts at its scene's root with that scene's camera and seed.
//
// Why not queues of rays between a trace and a shade kernel per bounce, as before: every such
// step lasts at least as long as its longest ray (0.3-0.6 ms), which was more than half of the
// time of a 1080p image at 8 bounces; and why not a thread per pixel: a 256 x 256 image fills
// 0.4 of the chip that way.
//
// Random numbers: Philox4x32-10 (Salmon et al., SC'11) keyed by (seed, 0x5EED), counter
// (pixel, sample, 0, 0) for the pixel jitter and (pixel, sample, bounce + 1, 0) for the
// bounce's direction and Russian roulette draws.
//
// Adjoint (no counterpart in the reference): gradients of sum(dL/dI * I) with respect to the
// albedo used at each triangle and each material's emission, by path-replay backpropagation
// (Vicini, Speierer, Jakob: "Path Replay Backpropagation", SIGGRAPH 2021). Per sample, a first
// pass computes the path's radiance L and keeps its triangles; a second pass follows them (or
// re-traces a long path from the same counter-based random numbers), and at vertex k the radiance still to
// come, L - sum_{i<=k} T_i E_i, divided by the albedo there is dL/dalbedo_k. One path per thread
// is kept at a time, so memory stays O(pixels). Russian-roulette probabilities are held constant.
#include "trace_warp.cuh"

#include <algorithm>
#include <cstring>
#include <mutex>
#include <vector>

namespace rtb
{

// camera basis and RNG key of one scene (src/main.cpp:43-83)
struct Cam
{
    float    pos[3], fwd[3], right[3], up[3];
    float    th;
    uint32_t seed;
};

namespace
{

struct RP
{
    uint32_t W, H, spp, max_bounce;
    int32_t  rr_after;
    uint32_t env_kind;
    float    env[3];
    Cam      cam;
    uint32_t sample_offset;
    uint32_t env_w, env_h;
    const float* env_map;
};

__device__ __forceinline__ uint4 philox(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3, uint32_t k0, uint32_t k1)
{
#pragma unroll
    for (int r = 0; r < 10; r++)
    {
        const uint32_t lo0 = 0xD2511F53u * c0, hi0 = __umulhi(0xD2511F53u, c0);
        const uint32_t lo1 = 0xCD9E8D57u * c2, hi1 = __umulhi(0xCD9E8D57u, c2);
        const uint32_t n0 = hi1 ^ c1 ^ k0, n1 = lo1, n2 = hi0 ^ c3 ^ k1, n3 = lo0;
        c0 = n0; c1 = n1; c2 = n2; c3 = n3;
        k0 += 0x9E3779B9u; k1 += 0xBB67AE85u;
    }
    return make_uint4(c0, c1, c2, c3);
}
__device__ __forceinline__ float u01(uint32_t x) { return (float)(x >> 8) * (1.0f / 16777216.0f); }

// Shading inputs (all optional): materials, the material of each baked triangle, and an RGB
// albedo per baked triangle that replaces the material's.
struct Shade
{
    const rt_material* mats;
    const uint32_t*    mot;
    const float*       talb;
    uint32_t           n_mats;
};

struct Surf
{
    f3       albedo, emission;
    uint32_t kind, mat;
};

__device__ __forceinline__ Surf surface(const Shade& S, uint32_t tri)
{
    Surf r;
    r.albedo = mk3(0.8f, 0.8f, 0.8f);
    r.emission = mk3(0.f, 0.f, 0.f);
    r.kind = 0; r.mat = 0;
    if (S.mats)
    {
        const uint32_t m = min(S.mot ? S.mot[tri] : 0u, S.n_mats - 1u);
        const rt_material M = S.mats[m];
        r.albedo = mk3(M.albedo[0], M.albedo[1], M.albedo[2]);
        r.emission = mk3(M.emission[0], M.emission[1], M.emission[2]);
        r.kind = M.kind; r.mat = m;
    }
    if (S.talb) { r.albedo = mk3(S.talb[3 * tri], S.talb[3 * tri + 1], S.talb[3 * tri + 2]); }
    return r;
}

constexpr float kPi = 3.14159265358979323846f;

// primaryRay, src/main.cpp:69-83
__device__ __forceinline__ void primary(const RP& P, const Cam& C, uint32_t x, uint32_t y, uint32_t pix, uint32_t sidx,
                                        f3& o, f3& d)
{
    const uint4 r = philox(pix, sidx, 0u, 0u, C.seed, 0x5EEDu);
    const float aspect = (float)P.W / (float)P.H;
    const float u = (((float)x + u01(r.x)) / (float)P.W * 2.f - 1.f) * aspect;
    const float v = ((float)y + u01(r.y)) / (float)P.H * 2.f - 1.f;
    const f3 fwd = mk3(C.fwd[0], C.fwd[1], C.fwd[2]);
    const f3 rgt = mk3(C.right[0], C.right[1], C.right[2]);
    const f3 up = mk3(C.up[0], C.up[1], C.up[2]);
    o = mk3(C.pos[0], C.pos[1], C.pos[2]);
    d = norm3(add3(add3(fwd, muls(rgt, u * C.th)), muls(up, v * C.th)));
}

// background (src/main.cpp:162-173); env_kind 2: IBL::sample (main.cpp:107-117), the
// nearest texel of an equirectangular map
__device__ __forceinline__ f3 environment(const RP& P, f3 d)
{
    if (P.env_kind == 0)
    {
        const float t = d.y * 0.5f + 0.5f;
        return add3(muls(mk3(1.0f, 1.0f, 1.0f), 1.f - t), muls(mk3(0.5f, 0.7f, 1.0f), t));
    }
    if (P.env_kind == 2)
    {
        const float phi = atan2f(d.z, d.x);
        const float y = d.y < -1.f ? -1.f : (1.f < d.y ? 1.f : d.y);  // std::clamp
        const float theta = acosf(y);
        const float u = (phi + kPi) / (2.f * kPi);
        const float v = theta / kPi;
        const int px = min((int)(u * (float)P.env_w), (int)P.env_w - 1);
        const int py = min((int)(v * (float)P.env_h), (int)P.env_h - 1);
        const float* p = P.env_map + ((size_t)py * P.env_w + px) * 3;
        return mk3(__ldg(p), __ldg(p + 1), __ldg(p + 2));
    }
    return mk3(P.env[0], P.env[1], P.env[2]);
}

// One bounce at a hit (src/main.cpp:178-200) after the emission of the surface was added:
// the next direction (cosine hemisphere about the shading normal, or the mirror direction),
// throughput update and Russian roulette. Returns false when roulette ends the path.
__device__ __forceinline__ bool scatter(const RP& P, uint32_t seed, const Surf& sf, f3 n, f3 din, uint32_t pix,
                                        uint32_t sidx, uint32_t bounce, f3& tp, f3& dout)
{
    const uint4 r = philox(pix, sidx, bounce + 1u, 0u, seed, 0x5EEDu);
    if (sf.kind == 1)
    {
        dout = sub3(din, muls(n, 2.f * dot3(din, n)));
    }
    else
    {
        // sampleCosineHemisphere + toWorld, src/main.cpp:123-141
        const float u1 = u01(r.x), u2 = u01(r.y);
        const float rr = sqrtf(u1);
        const float theta = 2.f * kPi * u2;
        const f3 ld = mk3(rr * cosf(theta), sqrtf(std_max(0.f, 1.f - u1)), rr * sinf(theta));
        const f3 axis = fabsf(n.x) < 0.9f ? mk3(1.f, 0.f, 0.f) : mk3(0.f, 1.f, 0.f);
        const f3 t = norm3(cross3(n, axis));
        const f3 b = cross3(n, t);
        dout = add3(add3(muls(t, ld.x), muls(n, ld.y)), muls(b, ld.z));
    }
    tp = mul3(tp, sf.albedo);
    if (P.rr_after >= 0 && (int32_t)bounce > P.rr_after)
    {
        const float p = std_max(std_max(tp.x, tp.y), tp.z);
        if (u01(r.z) > p) { return false; }
        tp = divs(tp, p);
    }
    return true;
}

// Shades a traced ray of a path: adds the emission (or background) it reached to `sum` and, where the
// path goes on, makes its next ray r0 = {o, tmin}, r1 = {d, tmax}. sf: the surface hit.
__device__ __forceinline__ bool shade(const TraceCtx& T, const RP& P, const Shade& sh, uint32_t seed, uint32_t pix, uint32_t sidx,
                                      uint32_t bounce, bool hit, float t, float4 uvt, f3 o, f3 d, f3& tp, f3& sum, Surf& sf,
                                      float4& r0, float4& r1)
{
    if (!hit)
    {
        sum = add3(sum, mul3(tp, environment(P, d)));
        return false;
    }
    const uint32_t tri = __float_as_uint(uvt.z);
    sf = surface(sh, tri);
    sum = add3(sum, mul3(tp, sf.emission));
    const f3 n = hit_normal(T, tri, uvt.x, uvt.y);
    f3 nd;
    if (!scatter(P, seed, sf, n, d, pix, sidx, bounce, tp, nd) || bounce >= P.max_bounce) { return false; }
    const f3 no = add3(o, muls(d, t));
    r0 = make_float4(no.x, no.y, no.z, 1e-4f);
    r1 = make_float4(nd.x, nd.y, nd.z, bits2f(0x7f800000u));
    return true;
}

// Pixels of an image in tiles of 32: 8 x 4 (neighbouring lanes start with neighbouring pixels), or one
// pixel wide or high where that takes fewer items (a very narrow or low image would take up to
// eight times its pixels).
struct Tiles
{
    uint32_t lw, tiles_x;  // log2 of a tile's width, tiles in a row
    uint64_t items;        // all tiles' pixels
};

Tiles make_tiles(uint32_t w, uint32_t h)
{
    Tiles best{ 0, 0, ~0ull };
    for (const uint32_t lw : { 3u, 0u, 5u })
    {
        const uint64_t tx = ((uint64_t)w + (1u << lw) - 1) >> lw, ty = ((uint64_t)h + (32u >> lw) - 1) >> (5 - lw);
        if (tx * ty * 32 < best.items) { best = Tiles{ lw, (uint32_t)tx, tx * ty * 32 }; }
    }
    return best;
}

// What one launch of k_paths works on. Items are numbered sample by sample, scene by scene and tile by
// tile; items of a tile that lie outside the image are skipped.
struct PathJob
{
    RP               P;
    Shade            sh;
    const Cam*       cams;     // per scene (nullptr: P.cam)
    const TraceRoot* roots;    // per scene (nullptr: the handle's root)
    uint32_t         S;        // scenes
    uint32_t         tile_lw, tiles_x, scene_items;
    uint32_t         sample0;  // sample of item 0, from P.sample_offset
    uint32_t         first, n; // this launch's items
    float*           rad;      // radiance per path: [sample - sample0][scene][pixel][3]
    float*           rgb;      // the images (OWN)
    float*           rgb2;
};

// Shared memory of one warp's paths.
struct PathShare
{
    WarpShare w;
    float4    tp[32];  // throughput, image pixel (scene * W * H + pixel)
    float4    sum[32]; // radiance so far, sample
};
// The radiance of every path. OWN: a lane takes whole pixels, adds their samples to the images itself,
// in the order and with the roundings of k_sum, and needs no memory besides: for renders that may not
// have any, and single samples (run_paths). Small Cornell box, 4 bounces: 256 x 256 x 16 4.2 ms against 1.5, where its
// pixels leave half of the lanes idle, 1080p x 16 39 against 29 ms.
template <int STK, bool OWN>
__global__ void __launch_bounds__(256, 4)
k_paths(const TraceCtx T, const __grid_constant__ PathJob J, uint32_t* __restrict__ counter, int per_warp)
{
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr unsigned FULL = 0xffffffffu;
    PathShare& S = reinterpret_cast<PathShare*>(smem)[threadIdx.x >> 5];
    const int lane = (int)(threadIdx.x & 31u);
    const unsigned lanes = per_warp >= 32 ? FULL : (1u << per_warp) - 1u;
    const int refill = per_warp >= 32 ? REFILL : (per_warp + 1) / 2;
    const bool odd_tree = *T.odd != 0u;
    const uint32_t npix = J.P.W * J.P.H;
    LaneTrace<0, STK> L;
    uint2 stk[STK];
    L.live = false;
    bool pending = false, more = true;  // this lane has a ray (to shade when it is done); items are left
    uint64_t own = 0, own_step = 0;     // OWN: the lane's pixel (an item of one sample), the way to its next
    uint32_t smp = 0;                   // OWN: its sample
    if (OWN)
    {
        const uint32_t wpb = blockDim.x >> 5;
        own_step = (uint64_t)gridDim.x * wpb * (uint32_t)per_warp;
        own = ((uint64_t)blockIdx.x * wpb + (threadIdx.x >> 5)) * (uint32_t)per_warp + (uint32_t)lane;
        if (lane >= per_warp) { own = J.n; }
    }
    // the first ray of sample s of an item of one sample; false where the item lies outside the image
    auto begin = [&](uint32_t item, uint32_t s, float4& r0, float4& r1) -> bool {
        const uint32_t sc = item / J.scene_items;
        const uint32_t q = item - sc * J.scene_items, tile = q >> 5, ty = tile / J.tiles_x;
        const uint32_t lw = J.tile_lw, p = q & 31u;
        const uint32_t x = ((tile - ty * J.tiles_x) << lw) + (p & ((1u << lw) - 1u)), y = (ty << (5u - lw)) + (p >> lw);
        if (x >= J.P.W || y >= J.P.H) { return false; }
        const uint32_t pix = y * J.P.W + x, sidx = J.P.sample_offset + J.sample0 + s;
        f3 o, d;
        primary(J.P, J.cams ? J.cams[sc] : J.P.cam, x, y, pix, sidx, o, d);
        r0 = make_float4(o.x, o.y, o.z, 1e-3f);
        r1 = make_float4(d.x, d.y, d.z, bits2f(0x7f800000u));
        S.tp[lane] = make_float4(1.f, 1.f, 1.f, __uint_as_float(sc * npix + pix));
        S.sum[lane] = make_float4(0.f, 0.f, 0.f, __uint_as_float(sidx));
        return true;
    };
    for (;;)
    {
        // lanes whose ray is done are shaded, and those whose path is done get a new one, once enough
        // of them wait; when no paths are left, once half of the lanes still at work do
        const unsigned idle = __ballot_sync(FULL, !L.live) & lanes;
        const unsigned takers = OWN ? __ballot_sync(FULL, own < J.n) : more ? lanes : __ballot_sync(FULL, pending);
        if (OWN) { more = takers == lanes; }
        const int serve = more ? refill : (__popc(takers) + 1) / 2;
        if (__popc(idle & takers) >= serve)
        {
            const bool mine = (idle >> lane) & 1u;
            bool go = false;  // r0, r1: the lane's next ray
            float4 r0 = make_float4(0.f, 0.f, 0.f, 0.f), r1 = r0;
            uint32_t bounce = 0;
            // shade what the finished rays hit
            if (mine && pending)
            {
                pending = false;
                const float4 a = S.w.a[lane], b = S.w.b[lane], h = S.w.hit[lane], ts = S.tp[lane], ss = S.sum[lane];
                f3 tp = mk3(ts.x, ts.y, ts.z), sum = mk3(ss.x, ss.y, ss.z);
                const uint32_t gpix = __float_as_uint(ts.w), sidx = __float_as_uint(ss.w);
                const uint32_t sc = gpix / npix;
                bounce = (uint32_t)S.w.id[lane];
                Surf sf;
                go = shade(T, J.P, J.sh, J.cams ? J.cams[sc].seed : J.P.cam.seed, gpix - sc * npix, sidx, bounce, L.hit, L.best, h,
                           mk3(a.x, a.y, a.z), mk3(b.x, b.y, b.z), tp, sum, sf, r0, r1);
                if (go)
                {
                    S.tp[lane] = make_float4(tp.x, tp.y, tp.z, ts.w);
                    S.sum[lane] = make_float4(sum.x, sum.y, sum.z, ss.w);
                    bounce++;
                }
                else if (OWN)
                {
                    const float fs = (float)J.P.spp;
                    const bool end = smp + 1u == J.P.spp;
#pragma unroll
                    for (int c = 0; c < 3; c++)
                    {
                        const float v = get3(sum, c);
                        float* p = J.rgb + 3 * (size_t)gpix + c;
                        const float a = (smp ? *p : 0.f) + v;
                        *p = end ? a / fs : a;
                        if (J.rgb2)
                        {
                            float* p2 = J.rgb2 + 3 * (size_t)gpix + c;
                            const float a2 = (smp ? *p2 : 0.f) + v * v;
                            *p2 = end ? a2 / fs : a2;
                        }
                    }
                    smp = end ? 0u : smp + 1u;
                    if (end) { own += own_step; }
                }
                else
                {
                    const size_t at = 3 * ((size_t)(sidx - J.P.sample_offset - J.sample0) * J.S * npix + gpix);
                    J.rad[at] = sum.x; J.rad[at + 1] = sum.y; J.rad[at + 2] = sum.z;
                }
            }
            // new paths for the others
            const bool want = mine && !go;
            if (OWN)
            {
                if (want)
                {
                    while (own < J.n && !(go = begin((uint32_t)own, smp, r0, r1))) { own += own_step; }
                    bounce = 0;
                }
            }
            else
            {
                const unsigned wants = __ballot_sync(FULL, want);
                if (more && wants)
                {
                    uint32_t base = 0;
                    if (lane == 0) { base = atomicAdd(counter, (uint32_t)__popc(wants)); }
                    base = __shfl_sync(FULL, base, 0);
                    if (base + (uint32_t)__popc(wants) >= J.n) { more = false; }
                    const uint32_t g = base + (uint32_t)__popc(wants & ((1u << lane) - 1u));
                    if (want && g < J.n)
                    {
                        const uint32_t G = J.first + g, per_sample = J.scene_items * J.S, s = G / per_sample;
                        go = begin(G - s * per_sample, s, r0, r1);
                        bounce = 0;
                    }
                }
            }
            if (go)
            {
                const TraceRoot* R = T.root;
                if (J.roots) { R = J.roots + __float_as_uint(S.tp[lane].w) / npix; }
                L.start(S.w, *R, r0, r1, odd_tree);
                S.w.id[lane] = bounce;
                pending = true;
            }
            __syncwarp();
            if ((OWN || !more) && !__any_sync(FULL, pending)) { break; }
            continue;
        }
        warp_walk<0, STK>(L, stk, T, takers, serve);
        warp_leaves<0, STK>(L, stk, T, S.w);
    }
}

constexpr uint32_t NO_TRI = 0xFFFFFFFFu;
constexpr uint32_t REC_BOUNCES = 64;  // triangles of a path that are kept

// The radiance of one sample of one pixel (primaryRay + pathTrace). REC: rec[] gets the triangles
// of the path, and NO_TRI after its last where it ends before max_bounce.
template <bool REC>
__device__ __forceinline__ f3 path_sample(const TraceCtx& T, const RP& P, const Shade& S, uint32_t x, uint32_t y,
                                          uint32_t pix, uint32_t sidx, uint32_t (&rec)[REC_BOUNCES])
{
    f3 o, d;
    primary(P, P.cam, x, y, pix, sidx, o, d);
    float tmin = 1e-3f;
    f3 tp = mk3(1.f, 1.f, 1.f), L = mk3(0.f, 0.f, 0.f);
    for (uint32_t bounce = 0; bounce <= P.max_bounce; bounce++)
    {
        const THit H = trace_ray(T, o, d, tmin, bits2f(0x7f800000u));
        if (REC) { rec[bounce] = H.hit ? H.tri : NO_TRI; }
        if (!H.hit)
        {
            L = add3(L, mul3(tp, environment(P, d)));
            break;
        }
        const Surf sf = surface(S, H.tri);
        L = add3(L, mul3(tp, sf.emission));
        if (REC && bounce == P.max_bounce) { break; }
        const f3 n = hit_normal(T, H.tri, H.u, H.v);
        f3 nd;
        if (!scatter(P, P.cam.seed, sf, n, d, pix, sidx, bounce, tp, nd))
        {
            if (REC) { rec[bounce + 1] = NO_TRI; }
            break;
        }
        o = add3(o, muls(d, H.t));
        d = nd;
        tmin = 1e-4f;
    }
    return L;
}

// dst[3 key + c] += v.c for every lane with `valid`, lanes of the warp with equal keys summed
// first so each distinct key costs one set of atomics per warp. All 32 lanes must call it.
__device__ __forceinline__ void warp_add3(float* __restrict__ dst, uint32_t key, bool valid, f3 v)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t k = valid ? key : 0xFFFFFFFFu;
    const uint32_t peers = __match_any_sync(0xFFFFFFFFu, k);
    bool pending = valid && __popc(peers) > 1;
    if (valid && !pending)
    {
        atomicAdd(&dst[3 * (size_t)key], v.x); atomicAdd(&dst[3 * (size_t)key + 1], v.y); atomicAdd(&dst[3 * (size_t)key + 2], v.z);
    }
    uint32_t pend = __ballot_sync(0xFFFFFFFFu, pending);
    while (pend)
    {
        const int ldr = __ffs(pend) - 1;
        const uint32_t lk = __shfl_sync(0xFFFFFFFFu, k, ldr);
        const bool in = pending && k == lk;
        float sx = in ? v.x : 0.f, sy = in ? v.y : 0.f, sz = in ? v.z : 0.f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
        {
            sx += __shfl_xor_sync(0xFFFFFFFFu, sx, o);
            sy += __shfl_xor_sync(0xFFFFFFFFu, sy, o);
            sz += __shfl_xor_sync(0xFFFFFFFFu, sz, o);
        }
        if ((int)lane == ldr)
        {
            atomicAdd(&dst[3 * (size_t)key], sx); atomicAdd(&dst[3 * (size_t)key + 1], sy); atomicAdd(&dst[3 * (size_t)key + 2], sz);
        }
        if (in) { pending = false; }
        pend = __ballot_sync(0xFFFFFFFFu, pending);
    }
}

// Path-replay adjoint, one thread per pixel. Lanes run the replay's bounce loop in step so the
// gradient adds can be combined per warp; pixels whose dL/dI is zero are skipped.
//
// REC: the forward pass keeps the triangles of its path, and the replay needs no more: throughput and
// gradients follow from them (roulette's survivors are the paths with a next triangle). Without it
// the replay traces the path again, which half of the time went to: 512 x 512 x 32, 50,000
// triangles, 4 bounces 106 -> 54 ms, 200,000 triangles, 5 bounces 201 -> 101 ms. Paths of more than
// REC_BOUNCES bounces are traced twice.
//
// Why a thread per pixel, per-lane traversal and five blocks per SM: a material's emission gradient
// is one 32-bit sum of millions of terms, off by 1.5e-4 from the exact one at 512 x 512 x 32, and
// where it ends up depends on which tiles are at work together. With this schedule it is 0.3-1.2e-5 (1.9e-5
// at most) from the paths traced twice, whose runs differ by 0.3-1.1e-5; warps that trace together as the renderer's do (31 ms) move it by 0.5-4e-5,
// paths traced by k_paths and replayed by a kernel of their own (35 ms) or other numbers of blocks by up to 3e-4.
template <bool REC>
__global__ void __launch_bounds__(128, REC ? 5 : 1)
k_adjoint(TraceCtx T, RP P, Shade S, const float* __restrict__ dimg, float* __restrict__ g_alb, float* __restrict__ g_em)
{
    const uint32_t x = blockIdx.x * 16 + (threadIdx.x & 15);
    const uint32_t y = blockIdx.y * 8 + (threadIdx.x >> 4);
    const bool in_img = x < P.W && y < P.H;
    const uint32_t pix = in_img ? y * P.W + x : 0u;
    const float fs = (float)P.spp;
    f3 dl = mk3(0.f, 0.f, 0.f);
    if (in_img) { dl = mk3(dimg[3 * pix] / fs, dimg[3 * pix + 1] / fs, dimg[3 * pix + 2] / fs); }
    const bool act = in_img && (dl.x != 0.f || dl.y != 0.f || dl.z != 0.f);
    if (!__any_sync(0xFFFFFFFFu, act)) { return; }
    uint32_t rec[REC_BOUNCES];
    for (uint32_t s = 0; s < P.spp; s++)
    {
        const uint32_t sidx = P.sample_offset + s;
        f3 Ltot = mk3(0.f, 0.f, 0.f);
        if (act) { Ltot = path_sample<REC>(T, P, S, x, y, pix, sidx, rec); }
        // replay
        f3 o = mk3(0.f, 0.f, 0.f), d = mk3(0.f, 0.f, 1.f);
        if (!REC && act) { primary(P, P.cam, x, y, pix, sidx, o, d); }
        float tmin = 1e-3f;
        f3 tp = mk3(1.f, 1.f, 1.f), Ssum = mk3(0.f, 0.f, 0.f);
        bool alive = act;
        for (uint32_t bounce = 0; bounce <= P.max_bounce; bounce++)
        {
            if (!__any_sync(0xFFFFFFFFu, alive)) { break; }
            bool hv = false;
            uint32_t tri = 0, mat = 0;
            f3 ga = mk3(0.f, 0.f, 0.f), ge = mk3(0.f, 0.f, 0.f);
            if (alive)
            {
                THit H;
                if (REC) { tri = rec[bounce]; }
                else
                {
                    H = trace_ray(T, o, d, tmin, bits2f(0x7f800000u));
                    tri = H.hit ? H.tri : NO_TRI;
                }
                if (tri == NO_TRI) { alive = false; }
                else
                {
                    const Surf sf = surface(S, tri);
                    hv = true; mat = sf.mat;
                    ge = mul3(dl, tp);
                    Ssum = add3(Ssum, mul3(tp, sf.emission));
                    const f3 rest = sub3(Ltot, Ssum);
                    ga = mk3(sf.albedo.x != 0.f ? dl.x * rest.x / sf.albedo.x : 0.f,
                             sf.albedo.y != 0.f ? dl.y * rest.y / sf.albedo.y : 0.f,
                             sf.albedo.z != 0.f ? dl.z * rest.z / sf.albedo.z : 0.f);
                    if (REC)
                    {
                        tp = mul3(tp, sf.albedo);
                        if (P.rr_after >= 0 && (int32_t)bounce > P.rr_after) { tp = divs(tp, std_max(std_max(tp.x, tp.y), tp.z)); }
                    }
                    else
                    {
                        const f3 n = hit_normal(T, tri, H.u, H.v);
                        f3 nd;
                        if (!scatter(P, P.cam.seed, sf, n, d, pix, sidx, bounce, tp, nd) || bounce >= P.max_bounce)
                        {
                            alive = false;
                        }
                        o = add3(o, muls(d, H.t));
                        d = nd;
                        tmin = 1e-4f;
                    }
                }
            }
            if (g_alb) { warp_add3(g_alb, tri, hv, ga); }
            if (g_em) { warp_add3(g_em, mat, hv && S.mats != nullptr, ge); }
        }
    }
}

// Adds the samples of every pixel channel in sample order: acc (+)= rad[0 .. n), and their squares;
// the last call divides by the sample count.
__global__ void __launch_bounds__(256)
k_sum(const float* __restrict__ rad, uint64_t channels, uint32_t n, bool start, bool end, float spp, float* __restrict__ rgb,
      float* __restrict__ rgb2)
{
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < channels; i += (uint64_t)gridDim.x * blockDim.x)
    {
        float acc = start ? 0.f : rgb[i], acc2 = start || !rgb2 ? 0.f : rgb2[i];
#pragma unroll 4
        for (uint32_t s = 0; s < n; s++)
        {
            const float v = __ldcs(&rad[(uint64_t)s * channels + i]);
            acc += v;
            acc2 += v * v;
        }
        rgb[i] = end ? acc / spp : acc;
        if (rgb2) { rgb2[i] = end ? acc2 / spp : acc2; }
    }
}

Cam make_cam(const rt_render_cfg& c)
{
    Cam C;
    for (int k = 0; k < 3; k++) { C.pos[k] = c.cam_pos[k]; C.fwd[k] = c.cam_fwd[k]; C.right[k] = c.cam_right[k]; C.up[k] = c.cam_up[k]; }
    C.th = c.tan_half_fov_y;
    C.seed = c.seed;
    return C;
}

RP make_rp(const rt_render_cfg& c, const rt_shading& sh)
{
    RP P;
    std::memset(&P, 0, sizeof(P));
    P.env_map = sh.env_map; P.env_w = sh.env_w; P.env_h = sh.env_h;
    P.W = c.width; P.H = c.height; P.spp = c.spp; P.max_bounce = c.max_bounce; P.rr_after = c.rr_after;
    P.env_kind = c.env_kind;
    for (int k = 0; k < 3; k++) { P.env[k] = c.env_color[k]; }
    P.cam = make_cam(c);
    P.sample_offset = c.sample_offset;
    return P;
}

constexpr uint32_t MAX_WAVEFRONT_BOUNCE = 62;

rt_wavefront_params default_params()
{
    rt_wavefront_params W;
    W.trace_block = 256;
    W.chunk_paths = 1u << 25;
    W.stack_depth = 64;
    W.shade_block = 256;
    return W;
}

int check_params(const rt_wavefront_params& W)
{
    if (W.trace_block == 0 || W.trace_block % 32 || W.trace_block > 256) { return fail(RT_E_INVALID, "trace_block must be 32..256, a multiple of 32"); }
    if (W.shade_block == 0 || W.shade_block % 32 || W.shade_block > 1024) { return fail(RT_E_INVALID, "shade_block must be 32..1024, a multiple of 32"); }
    if (W.chunk_paths < 1024 || W.chunk_paths > (1u << 26)) { return fail(RT_E_INVALID, "chunk_paths must be in [1024, 2^26]"); }
    if (W.stack_depth != 32 && W.stack_depth != 64) { return fail(RT_E_INVALID, "stack_depth must be 32 or 64"); }
    return RT_OK;
}

using PathFn = void (*)(TraceCtx, PathJob, uint32_t*, int);

int launch_paths(PathFn fn, const TraceCtx& T, const PathJob& J, uint32_t* counter, uint32_t block, cudaStream_t st)
{
    const size_t smem = (size_t)(block / 32) * sizeof(PathShare);
    const int per_sm = blocks_per_sm(reinterpret_cast<const void*>(fn), (int)block, smem);
    // few items are spread over the resident warps (as few rays are by trace)
    const uint64_t warps = (uint64_t)device_sm_count() * (uint64_t)per_sm * (block / 32);
    const uint64_t per_warp = std::min<uint64_t>(32, (J.n + warps - 1) / warps);
    const uint64_t grid = std::min<uint64_t>((uint64_t)device_sm_count() * (uint64_t)per_sm,
                                             (J.n + per_warp * (block / 32) - 1) / (per_warp * (block / 32)));
    if (counter) { RT_CUDA(cudaMemsetAsync(counter, 0, 4, st)); }
    fn<<<(uint32_t)grid, block, smem, st>>>(T, J, counter, (int)per_warp);
    count_launch();
    return check_launch("paths");
}

// Renders J's scenes. Samples are taken in groups
// whose paths fit W.chunk_paths (at least one sample of every pixel), each group launched in pieces
// of at most that many paths. The call's scratch: the radiance of a group's paths, the cameras and the item
// counter. Where the device has no memory for it, smaller groups give the same image, and at last a
// lane per pixel does.
int run_paths(const rt_bvh* B, PathJob J, const Cam* h_cams, const rt_wavefront_params& W, float* rgb, float* rgb2,
              cudaStream_t st)
{
    const uint64_t npix = (uint64_t)J.P.W * J.P.H;
    const Tiles tiles = make_tiles(J.P.W, J.P.H);
    if (tiles.items > 0xffffffffull / J.S) { return fail(RT_E_CAPACITY, "more than 2^32 pixels"); }
    J.tile_lw = tiles.lw;
    J.tiles_x = tiles.tiles_x;
    J.scene_items = (uint32_t)tiles.items;
    const uint64_t per_sample = tiles.items * J.S;
    const TraceCtx T = make_trace_ctx(B);
    auto own_pixels = [&]() {
        J.rgb = rgb; J.rgb2 = rgb2;
        J.n = (uint32_t)per_sample;
        return launch_paths(k_paths<STACK, true>, T, J, nullptr, W.trace_block, st);
    };
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    RT_CUDA(cudaStreamIsCapturing(st, &cs));
    if (cs != cudaStreamCaptureStatusNone)
    {
        if (h_cams) { return fail(RT_E_INVALID, "a render of several scenes cannot be captured"); }
        // A captured render is one kernel node: memory nodes would keep the caller from using the
        // graph as a child or twice at a time.
        return own_pixels();
    }
    // (Asked for in every call: a warm-up also loads the kernel that a captured call launches.)
    // One sample of an image that the chip holds at once: the lanes own their pixels just as well, and that
    // needs one launch instead of two, a clear and scratch.
    const uint64_t warps = (uint64_t)device_sm_count() *
                           blocks_per_sm(reinterpret_cast<const void*>(k_paths<STACK, true>), (int)W.trace_block,
                                         (W.trace_block / 32) * sizeof(PathShare)) * (W.trace_block / 32);
    if (J.P.spp == 1 && !h_cams && per_sample <= warps * 32) { return own_pixels(); }
    // cameras, item counter, radiance
    const uint64_t cam_bytes = h_cams ? (J.S * sizeof(Cam) + 255) / 256 * 256 : 0, head = cam_bytes + 256;
    uint64_t group = std::max<uint64_t>(1, std::min<uint64_t>(W.chunk_paths / per_sample, J.P.spp));
    CallScratch scratch;
    int missing = 0;
    while ((missing = scratch.get(head + group * npix * J.S * 12, st)) != 0 && group > 0) { group /= 2; }
    if (missing && h_cams) { return missing; }
    if (h_cams)
    {
        // (an upload from pageable memory has left the host array when cudaMemcpyAsync returns)
        RT_CUDA(cudaMemcpyAsync(scratch.as<void>(), h_cams, J.S * sizeof(Cam), cudaMemcpyHostToDevice, st));
        J.cams = scratch.as<Cam>();
    }
    if (group == 0) { return own_pixels(); }
    uint32_t* counter = reinterpret_cast<uint32_t*>(scratch.as<char>() + cam_bytes);
    J.rad = reinterpret_cast<float*>(scratch.as<char>() + head);
    const PathFn fn = W.stack_depth < 64 ? k_paths<32, false> : k_paths<STACK, false>;
    const uint64_t channels = npix * J.S * 3;
    for (uint64_t s0 = 0; s0 < J.P.spp; s0 += group)
    {
        const uint64_t ns = std::min<uint64_t>(group, J.P.spp - s0), all = ns * per_sample;
        const uint64_t piece = std::min<uint64_t>(std::max<uint64_t>(W.chunk_paths, 1), 1ull << 30);
        J.sample0 = (uint32_t)s0;
        for (uint64_t g = 0; g < all; g += piece)
        {
            J.first = (uint32_t)g;
            J.n = (uint32_t)std::min<uint64_t>(piece, all - g);
            if (int e = launch_paths(fn, T, J, counter, W.trace_block, st)) { return e; }
        }
        const uint64_t blocks = (channels + W.shade_block - 1) / W.shade_block;
        k_sum<<<(uint32_t)std::min<uint64_t>(blocks, 1u << 20), W.shade_block, 0, st>>>(J.rad, channels, (uint32_t)ns, s0 == 0,
                                                                                  s0 + ns == J.P.spp, (float)J.P.spp, rgb, rgb2);
        count_launch();
        if (int e = check_launch("sample sums")) { return e; }
    }
    return RT_OK;
}

// A valid parameter set for a render of this handle: the tuned one, else the defaults (with the
// stack the tree needs). A larger job than the tuning's has no measurement of its own launches: it takes
// the default's at least.
rt_wavefront_params pick_params(const rt_bvh* B, const rt_wavefront_params* W, const rt_render_cfg& c, uint32_t S)
{
    if (W) { return *W; }
    rt_wavefront_params P = default_params();
    if (B->wf_tuned_valid)
    {
        const uint32_t chunk = P.chunk_paths;
        P = B->wf_tuned;
        if (make_tiles(c.width, c.height).items * S * c.spp > B->wf_tuned_paths) { P.chunk_paths = std::max(P.chunk_paths, chunk); }
    }
    return P;
}

} // namespace

int render(const rt_bvh* B, const rt_render_cfg& cfg, const rt_shading& sh, int mode, float* rgb, float* rgb2,
           cudaStream_t st)
{
    if (mode != RT_RENDER_PLAIN && mode != RT_RENDER_WAVEFRONT) { return fail(RT_E_INVALID, "unknown render mode"); }
    if (mode == RT_RENDER_WAVEFRONT && cfg.max_bounce > MAX_WAVEFRONT_BOUNCE) { return fail(RT_E_INVALID, "max_bounce must be below 63 for the wavefront"); }
    PathJob J{};
    J.P = make_rp(cfg, sh);
    J.S = 1;
    J.sh = Shade{ sh.mats, sh.mat_of_tri, sh.tri_albedo, sh.n_mats };
    rt_wavefront_params W = mode == RT_RENDER_WAVEFRONT ? pick_params(B, nullptr, cfg, 1) : default_params();
    W.stack_depth = 64;  // tuned for a batch; a plain handle keeps the full stack
    return run_paths(B, J, nullptr, W, rgb, rgb2, st);
}

int render_batch(rt_bvh* B, const rt_render_cfg* cfgs, uint32_t S, const rt_shading& sh, const rt_wavefront_params* params,
                 float* rgb, float* rgb2, cudaStream_t st)
{
    const rt_render_cfg& c0 = cfgs[0];
    if (c0.max_bounce > MAX_WAVEFRONT_BOUNCE) { return fail(RT_E_INVALID, "max_bounce must be below 63 for the wavefront"); }
    const rt_wavefront_params W = pick_params(B, params, c0, S);
    if (int e = check_params(W)) { return e; }
    if (W.stack_depth < 64)
    {
        uint32_t depth = 0;
        if (int e = tree_depth(B, st, &depth)) { return e; }
        if (depth + 1 > W.stack_depth) { return fail(RT_E_INVALID, "stack_depth is smaller than the tree needs"); }
    }
    std::vector<Cam> cams(S);
    for (uint32_t s = 0; s < S; s++) { cams[s] = make_cam(cfgs[s]); }
    PathJob J{};
    J.P = make_rp(c0, sh);
    J.S = S;
    J.sh = Shade{ sh.mats, sh.mat_of_tri, sh.tri_albedo, sh.n_mats };
    J.roots = S > 1 ? B->scene_roots.as<TraceRoot>() : nullptr;  // one scene: the whole tree
    return run_paths(B, J, S > 1 ? cams.data() : nullptr, W, rgb, rgb2, st);
}

int autotune_wavefront(rt_bvh* B, const rt_render_cfg* cfgs, uint32_t S, const rt_shading& sh, rt_wavefront_params* best,
                       float* scratch_rgb, cudaStream_t st)
{
    uint32_t depth = 0;
    if (int e = tree_depth(B, st, &depth)) { return e; }
    const uint32_t chunks[] = { 1u << 20, 1u << 21, 1u << 22, 1u << 23, 1u << 24, 1u << 25 };
    // trial renders with enough samples per pixel that the largest chunk fills (a one-sample
    // trial of a small image cannot tell the chunk sizes apart), at most the configs' own
    const uint64_t items = make_tiles(cfgs[0].width, cfgs[0].height).items * S, largest = chunks[5];
    std::vector<rt_render_cfg> c1(cfgs, cfgs + S);
    for (auto& c : c1)
    {
        c.spp = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((largest + items - 1) / items, c.spp));
        c.sample_offset = 0;
    }
    // chunks that hold the whole trial launch the same: the smallest of them stands for all, the default's too
    uint32_t whole = 0;
    while (chunks[whole] < items * c1[0].spp && whole < 5) { whole++; }
    cudaEvent_t a, b;
    RT_CUDA(cudaEventCreate(&a));
    RT_CUDA(cudaEventCreate(&b));
    int err = RT_OK;
    auto time = [&](const rt_wavefront_params& W) {  // the faster of two runs
        float best_ms = 1e30f;
        for (int rep = 0; rep < 2 && !err; rep++)
        {
            if (cudaEventRecord(a, st) != cudaSuccess) { err = fail(RT_E_CUDA, "event"); break; }
            err = render_batch(B, c1.data(), S, sh, &W, scratch_rgb, nullptr, st);
            if (err) { break; }
            if (cudaEventRecord(b, st) != cudaSuccess || cudaEventSynchronize(b) != cudaSuccess) { err = fail(RT_E_CUDA, "event"); break; }
            float ms = 0.f;
            cudaEventElapsedTime(&ms, a, b);
            best_ms = std::min(best_ms, ms);
        }
        return best_ms;
    };
    rt_wavefront_params bw = default_params();
    bw.chunk_paths = chunks[whole];
    const rt_wavefront_params dw = bw;
    time(bw);
    const float default_ms = time(bw);
    float best_ms = default_ms;
    auto trial = [&](const rt_wavefront_params& W) {
        if (err || std::memcmp(&W, &dw, sizeof(W)) == 0) { return; }
        const float ms = time(W);
        if (!err && ms < best_ms) { best_ms = ms; bw = W; }
    };
    // the block and the stack at the default's chunk, then the chunk
    for (const uint32_t stack : { 32u, 64u })
    {
        for (const uint32_t block : { 64u, 128u, 256u })
        {
            rt_wavefront_params W = dw;
            W.trace_block = block; W.stack_depth = stack;
            if (stack == 64 || depth + 1 <= stack) { trial(W); }
        }
    }
    const rt_wavefront_params shape = bw;
    for (uint32_t k = 0; k < whole; k++)
    {
        rt_wavefront_params W = shape;
        W.chunk_paths = chunks[k];
        trial(W);
    }
    if (best_ms > 0.98f * default_ms) { bw = dw; }  // (closer times are the runs' own spread)
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    if (err) { return err; }
    B->wf_tuned = bw;
    B->wf_tuned_paths = c1[0].spp < cfgs[0].spp ? ~0ull : items * cfgs[0].spp;
    B->wf_tuned_valid = true;
    if (best) { *best = bw; }
    return RT_OK;
}

int adjoint(const rt_bvh* B, const rt_render_cfg& cfg, const rt_shading& sh, const float* d_rgb, float* g_alb,
            float* g_em, cudaStream_t st)
{
    const TraceCtx T = make_trace_ctx(B);
    const RP P = make_rp(cfg, sh);
    const Shade S{ sh.mats, sh.mat_of_tri, sh.tri_albedo, sh.n_mats };
    const dim3 grid((cfg.width + 15) / 16, (cfg.height + 7) / 8);
    const auto fn = cfg.max_bounce < REC_BOUNCES ? k_adjoint<true> : k_adjoint<false>;
    fn<<<grid, 128, 0, st>>>(T, P, S, d_rgb, g_alb, sh.mats ? g_em : nullptr);
    count_launch();
    return check_launch("adjoint");
}

} // namespace rtb
