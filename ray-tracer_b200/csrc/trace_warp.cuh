// trace_warp.cuh -- bvh::trace (src/bvh/bvh_traverse.cpp:91-178) for the rays of a warp: lanes walk
// inner nodes on their own and test leaves together.
//
// What bounded the per-lane loops this replaces: issue slots with 5 of 32 lanes busy (incoherent
// rays of a warp stand at different leaves of different sizes and finish after very different
// numbers of steps). Here
//  * the (ray, triangle) pairs of all leaves the lanes stand at are dealt out to the 32 lanes, one
//    pair each, in lane order and leaf order (warp_leaves): neighbouring lanes read neighbouring
//    triangles;
//  * the inner-node loop stops once fewer than WALK_MIN lanes still walk and others wait at a leaf
//    or for a new ray;
//  * finished lanes take new rays once REFILL of them are idle.
// Every ray still sees the reference's nodes, leaves and triangles in the reference's order with the
// same best distance at each test, so hits are the reference's bit for bit: a leaf's accepted
// triangles reach their ray's lane in leaf order and pass the strict "t < best" there.
// 2,097,152 incoherent rays, 1M-triangle soup: LBVH (leaf 16) 15.7 -> 6.5 ms, SAH (leaf 4)
// 11.4 -> 6.0 ms; 1080p primary plus shadow rays, 1M triangles, hybrid tree: 3.07 -> 1.96 ms.
//
// The rest of the time goes to L1 (node and triangle fetches, stacks: 60-78 % of its wavefronts)
// and issue slots (49-74 %) with 17-21 lanes busy. Hence the 8-byte stack entries (16 bytes: 8.2 ms on the
// SAH tree -- the stacks of an SM alone filled its L1), the top entry kept in registers, nodes
// fetched with two 256-bit loads, and rays and hits kept in shared memory rather than in
// registers (64 registers, four blocks of 256 threads per SM; 80 registers 5-10 % slower). Slower too:
// both planes of an axis in Blackwell's packed f32x2 arithmetic (2-5 %: six more registers), triangles
// in pair records tested with it (3-8 %, and 30 % with a filter before the exact test).
#pragma once

#include "trace_core.cuh"

namespace rtb
{

// the halves of a 64-bit register pair
__device__ __forceinline__ void unpack2(unsigned long long r, float& a, float& b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r));
}

// 256-bit read-only load (p: 32-byte aligned)
struct quad64 { unsigned long long x, y, z, w; };
__device__ __forceinline__ quad64 ldg256(const void* p)
{
    quad64 r;
    asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(r.x), "=l"(r.y), "=l"(r.z), "=l"(r.w) : "l"(p));
    return r;
}

// Shared memory of one warp: its lanes' rays and hits, and the leaves they stand at.
struct WarpShare
{
    float4   a[32];   // o.xyz, tmin
    float4   b[32];   // d.xyz, tmax
    float4   hit[32]; // u, v, triangle of the closest hit so far
    uint4    leaf[32];// first triangle - first pair, lane, best distance
    uint64_t id[32];  // the caller's ray index
};

// Lanes below which the inner-node loop stops for waiting lanes, and idle lanes of 32 at which new
// rays are taken. Both optima are flat: WALK_MIN 8-16 and REFILL 12-20 are within 3 % on LBVH,
// hybrid and SAH trees; 4 and 24 cost 5-8 %.
constexpr int WALK_MIN = 12;
constexpr int REFILL = 16;
// Leaves are tested lane by lane instead of pair by pair when the longest one would leave the warp
// at least DIRECT_NUM / 32 busy: the ray is at hand and hits stay in the lane. (Rare: with it off,
// nothing measured changes by more than 1 %.)
constexpr uint32_t DIRECT_NUM = 24;
constexpr uint32_t SHARE_MAX = 1u << 20;  // leaves above this are always tested lane by lane

// One lane's traversal state. A stack entry is {child, entry distance}: an inner child by its node
// index, a leaf by LEAF_BIT | parent node << 1 | right, whose range is read again when it is
// popped (so node indices stay below 2^30: 120 GB of nodes).
template <int MODE, int STK>
struct LaneTrace
{
    float    ox, oy, oz, ix, iy, iz;  // o and 1 / d
    float    tmin, best;
    uint32_t ref, cnt;                // the node or leaf the lane stands at
    uint32_t tref;                    // the top stack entry (stk[1 .. top - 1] holds those below)
    float    ttn;
    int      top;
    uint32_t steps;
    bool     live, hit, overflow, odd;

    // r0, r1: o and tmin, d and tmax. odd_tree: boxes may hold NaN.
    __device__ __forceinline__ void start(WarpShare& S, const TraceRoot& R, float4 r0, float4 r1, bool odd_tree)
    {
        const int lane = (int)(threadIdx.x & 31u);
        S.a[lane] = r0;
        S.b[lane] = r1;
        tmin = r0.w; best = r1.w;
        hit = false; overflow = false; top = 0; steps = 0;
        const f3 o = mk3(r0.x, r0.y, r0.z), d = mk3(r1.x, r1.y, r1.z);
        const f3 inv = mk3(1.f / d.x, 1.f / d.y, 1.f / d.z);
        // With finite o, d and 1 / d and boxes without NaN no slab distance is NaN, and min / max
        // instructions give what the reference's std::min / std::max do; other rays take ray_box.
        const float inf = bits2f(0x7f800000u);
        odd = odd_tree || !(fabsf(inv.x) < inf && fabsf(inv.y) < inf && fabsf(inv.z) < inf && fabsf(o.x) < inf &&
                            fabsf(o.y) < inf && fabsf(o.z) < inf && fabsf(d.x) < inf && fabsf(d.y) < inf && fabsf(d.z) < inf) ||
              tmin != tmin || best != best;
        ref = R.ref; cnt = R.cnt;
        live = ray_box(o, inv, tmin, best, R.box[0], R.box[1], R.box[2], R.box[3], R.box[4], R.box[5]) < best;
        ox = o.x; oy = o.y; oz = o.z; ix = inv.x; iy = inv.y; iz = inv.z;
    }

    // The next stack entry whose entry distance is below best, or none. (All entries pass unless
    // best shrank since they were pushed, so this rarely loops.)
    __device__ __forceinline__ void pop(uint2 (&stk)[STK], const rt_gnode* __restrict__ gn)
    {
        live = false;
        while (top > 0)
        {
            ref = tref;
            const bool ok = ttn < best;
            if (--top > 0)
            {
                const uint2 e = stk[top];
                tref = e.x; ttn = __uint_as_float(e.y);
            }
            if (ok) { live = true; break; }
        }
        cnt = 0u;
        if (live && (ref & LEAF_BIT))
        {
            const uint32_t* w = reinterpret_cast<const uint32_t*>(&gn[(ref & ~LEAF_BIT) >> 1].d) + (ref & 1u);
            ref = __ldg(w);
            cnt = __ldg(w + 2);
        }
    }

    // One inner node: both children's boxes, the nearer child next, the farther one on the stack.
    __device__ __forceinline__ void step(uint2 (&stk)[STK], const rt_gnode* __restrict__ gn)
    {
        const quad64 A = ldg256(gn + ref), B = ldg256(reinterpret_cast<const char*>(gn + ref) + 32);
        uint32_t lref, rref, lcnt, rcnt;
        asm("mov.b64 {%0, %1}, %2;" : "=r"(lref), "=r"(rref) : "l"(B.z));
        asm("mov.b64 {%0, %1}, %2;" : "=r"(lcnt), "=r"(rcnt) : "l"(B.w));
        const float inf = bits2f(0x7f800000u);
        float tl, tr;
        if (odd)
        {
            float l0, l1, l2, l3, l4, l5, r0, r1, r2, r3, r4, r5;
            unpack2(A.x, l0, l3); unpack2(A.y, l1, l4); unpack2(A.z, l2, l5);
            unpack2(A.w, r0, r3); unpack2(B.x, r1, r4); unpack2(B.y, r2, r5);
            const f3 o = mk3(ox, oy, oz), inv = mk3(ix, iy, iz);
            tl = ray_box(o, inv, tmin, best, l0, l1, l2, l3, l4, l5);
            tr = ray_box(o, inv, tmin, best, r0, r1, r2, r3, r4, r5);
        }
        else
        {
            // rayAABB (bvh_traverse.cpp:22-41)
            auto slab = [&](unsigned long long bx, unsigned long long by, unsigned long long bz) {
                float x0, x1, y0, y1, z0, z1;
                unpack2(bx, x0, x1); unpack2(by, y0, y1); unpack2(bz, z0, z1);
                x0 = (x0 - ox) * ix; x1 = (x1 - ox) * ix;
                y0 = (y0 - oy) * iy; y1 = (y1 - oy) * iy;
                z0 = (z0 - oz) * iz; z1 = (z1 - oz) * iz;
                const float tn = fmaxf(fmaxf(fmaxf(fminf(x0, x1), fminf(y0, y1)), fminf(z0, z1)), tmin);
                const float tf = fminf(fminf(fminf(fmaxf(x0, x1), fmaxf(y0, y1)), fmaxf(z0, z1)), best);
                return tn <= tf ? tn : inf;
            };
            tl = slab(A.x, A.y, A.z);
            tr = slab(A.w, B.x, B.y);
        }
        const bool left = tl <= tr;  // left first on ties
        const float nt = left ? tl : tr, ft = left ? tr : tl;
        if (nt < best)  // (the farther child is hit only if the nearer one is)
        {
            const uint32_t fref = left ? rref : lref, fcnt = left ? rcnt : lcnt;
            const uint32_t at = LEAF_BIT | (ref << 1) | (left ? 1u : 0u);
            ref = left ? lref : rref;
            cnt = left ? lcnt : rcnt;
            if (ft < best)
            {
                // (the reference's 64-entry stack holds the nearer child too; alone it always fits)
                if (top + 1 >= STK) { overflow = true; live = false; return; }
                stk[top++] = make_uint2(tref, __float_as_uint(ttn));
                tref = (fcnt & LEAF_BIT) ? at : fref;
                ttn = ft;
            }
        }
        else { pop(stk, gn); }
    }
};

template <int MODE>
__device__ __forceinline__ bool test_triangle(const float4* __restrict__ tp, uint32_t ti, float4 ra, float4 rb, float& t,
                                              float& u, float& v)
{
    const float4 p0 = __ldg(&tp[3 * (size_t)ti]), p1 = __ldg(&tp[3 * (size_t)ti + 1]), p2 = __ldg(&tp[3 * (size_t)ti + 2]);
    const f3 v0 = mk3(p0.x, p0.y, p0.z), v1 = mk3(p0.w, p1.x, p1.y), v2 = mk3(p1.z, p1.w, p2.x);
    const f3 o = mk3(ra.x, ra.y, ra.z), d = mk3(rb.x, rb.y, rb.z);
    return (MODE & 2) ? ray_tri_watertight(o, d, ra.w, rb.w, v0, v1, v2, t, u, v)
                      : ray_tri(o, d, ra.w, rb.w, v0, v1, v2, t, u, v);
}

// Tests the leaves that lanes stand at (bvh_traverse.cpp:112-142) and moves those lanes on. All 32
// lanes call it.
template <int MODE, int STK>
__device__ __forceinline__ void warp_leaves(LaneTrace<MODE, STK>& L, uint2 (&stk)[STK], const TraceCtx& T, WarpShare& S)
{
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = (int)(threadIdx.x & 31u);
    const bool leaf = L.live && (L.cnt & LEAF_BIT);
    const uint32_t cnt = leaf ? (L.cnt & ~LEAF_BIT) : 0u;
    const uint32_t longest = __reduce_max_sync(FULL, cnt);
    bool accepted = false;
    if (longest > 0u)
    {
        const bool share = longest <= SHARE_MAX;
        const uint32_t pairs = share ? __reduce_add_sync(FULL, cnt) : 0u;
        if (!share || longest * DIRECT_NUM <= pairs)
        {
            for (uint32_t k = 0; k < cnt; k++)
            {
                float t, u, v;
                if (test_triangle<MODE>(T.tp, L.ref + k, S.a[lane], S.b[lane], t, u, v) && t < L.best)
                {
                    L.best = t;
                    S.hit[lane] = make_float4(u, v, __uint_as_float(L.ref + k), 0.f);
                    L.hit = accepted = true;
                    if (MODE & 1) { break; }
                }
            }
            __syncwarp();
        }
        else
        {
            // pairs are numbered lane by lane; start = this lane's first
            uint32_t start = cnt;
#pragma unroll
            for (int s = 1; s < 32; s <<= 1)
            {
                const uint32_t x = __shfl_up_sync(FULL, start, s);
                if (lane >= s) { start += x; }
            }
            start -= cnt;
            const unsigned below = (1u << lane) - 1u, upto = below | (1u << lane);
            const unsigned have = __ballot_sync(FULL, cnt > 0u);
            if (cnt > 0u)
            {
                S.leaf[__popc(have & below)] = make_uint4(L.ref - start, (uint32_t)lane, __float_as_uint(L.best), 0u);
            }
            __syncwarp();
            int before = 0;  // leaves that start before this round's pairs
            for (uint32_t base = 0; base < pairs; base += 32)
            {
                // the pairs at which leaves start in this round tell each lane its pair's leaf
                const bool here = cnt > 0u && start - base < 32u;
                const unsigned marks = __reduce_or_sync(FULL, here ? 1u << (start - base) : 0u);
                const int r = before + __popc(marks & upto) - 1;
                before += __popc(marks);
                const uint32_t p = base + (uint32_t)lane;
                float t = 0.f, u = 0.f, v = 0.f;
                uint32_t ti = 0, own = 0;
                bool acc = false;
                if (p < pairs)
                {
                    const uint4 lf = S.leaf[r];
                    own = lf.y;
                    ti = lf.x + p;
                    acc = test_triangle<MODE>(T.tp, ti, S.a[own], S.b[own], t, u, v) && t < __uint_as_float(lf.z);
                }
                // accepted hits to their rays' lanes, in leaf order
                for (unsigned am = __ballot_sync(FULL, acc); am; am &= am - 1u)
                {
                    const int s = __ffs((int)am) - 1;
                    const uint32_t to = __shfl_sync(FULL, own, s), is = __shfl_sync(FULL, ti, s);
                    const float ts = __shfl_sync(FULL, t, s), us = __shfl_sync(FULL, u, s), vs = __shfl_sync(FULL, v, s);
                    if ((uint32_t)lane == to && ts < L.best && !((MODE & 1) && accepted))
                    {
                        L.best = ts;
                        S.hit[lane] = make_float4(us, vs, __uint_as_float(is), 0.f);
                        L.hit = accepted = true;
                    }
                }
            }
            __syncwarp();
        }
    }
    if (leaf)
    {
        if ((MODE & 1) && accepted) { L.live = false; } else { L.pop(stk, T.gn); }
    }
}

// Walks inner nodes until every live lane stands at a leaf, or few lanes walk and others wait at a
// leaf or, `serve` or more of `takers`, to be served by the caller (a new ray).
template <int MODE, int STK>
__device__ __forceinline__ void warp_walk(LaneTrace<MODE, STK>& L, uint2 (&stk)[STK], const TraceCtx& T, unsigned takers,
                                          int serve)
{
    constexpr unsigned FULL = 0xffffffffu;
    for (uint32_t it = 0; it < 1024u; it++)
    {
        const bool walk = L.live && !(L.cnt & LEAF_BIT);
        const unsigned walking = __ballot_sync(FULL, walk);
        if (walking == 0u) { break; }
        if (it > 0 && __popc(walking) < WALK_MIN)
        {
            const unsigned live = __ballot_sync(FULL, L.live);
            if (live != walking || __popc(takers & ~live) >= serve) { break; }
        }
        if (walk)
        {
            L.step(stk, T.gn);
            L.steps++;
        }
        __syncwarp();
    }
    // A validated BVH is a DAG with children after parents; the cap only bounds the work a
    // malformed one could cause. (Only the lane's own nodes count, not its waits for others.)
    if (L.live && L.steps > MAX_POPS) { L.overflow = true; L.live = false; }
}

} // namespace rtb
