// traverse.cu -- closest-hit / any-hit ray traversal: bvh::trace (src/bvh/bvh_traverse.cpp:91-246)
// for batches of rays on the GPU.
//
// Layout: the .bvh node array is re-laid as 64-byte two-child nodes (rt_gnode: both children's
// boxes and references, two 256-bit loads per visited inner node) and a 48-byte triangle
// position record per baked triangle (three 128-bit loads per triangle test). Node indices are
// those of the .bvh array, so the traversal visits exactly the reference's nodes.
//
// Equivalence with the reference loop: the reference pops a node and re-tests its box against
// the current best t (bvh_traverse.cpp:104-110); here the stack keeps the entry distance tNear
// computed when the node was pushed. The slab interval's far end depends on the best t only
// through min(tFar, bestT), so "rayAABB(node, bestT) >= bestT" holds exactly when
// tNear >= bestT (also with the NaN slabs of axis-parallel rays: tNear, and whether tFar is NaN,
// do not depend on bestT). Children are tested and pushed in the reference's order (far child
// first, the left child first on ties, :143-174) and triangles are tested in leaf order with the
// strict "t < bestT" update (:112-142), so the first triangle at the minimal distance wins as
// in the reference and hits carry identical triangle indices (trace_warp.cuh).
//
// The kernel is persistent: warps claim rays from a global counter as their lanes finish, and
// test leaves together (trace_warp.cuh).
#include "trace_warp.cuh"

#include <algorithm>
#include <mutex>
#include <vector>

namespace rtb
{

namespace
{

constexpr int TBLK = 128;

// Also validates the structure before any traversal may run on it: children of node i have
// larger indices (DFS pre-order, so no cycles) inside the array, leaf ranges inside the
// triangle array. A violation sets ST_CAPACITY and the handle is refused.
// d_counts (optional) holds {nodes, triangles} on the device (a build that has not synchronised);
// thread 0 also writes the traversal entry record of node 0.
__global__ void k_make_gnodes(const rt_bvh_node* __restrict__ nodes, uint32_t n_nodes, uint32_t n_tris,
                              const uint32_t* __restrict__ d_counts, rt_gnode* __restrict__ gn, TraceRoot* __restrict__ root,
                              uint32_t* __restrict__ odd, uint32_t* __restrict__ status)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (d_counts) { n_nodes = d_counts[0]; n_tris = d_counts[1]; }
    if (i >= n_nodes) { return; }
    const rt_bvh_node nd = nodes[i];
    if (i == 0)
    {
        TraceRoot r;
        for (int k = 0; k < 3; k++) { r.box[k] = nd.bmin[k]; r.box[3 + k] = nd.bmax[k]; }
        r.ref = nd.is_leaf ? nd.a : 0u;
        r.cnt = nd.is_leaf ? (LEAF_BIT | nd.b) : 0u;
        *root = r;
    }
    if (nd.is_leaf)
    {
        if ((uint64_t)nd.a + nd.b > n_tris) { atomicOr(status, ST_CAPACITY); }
        return;
    }
    if (nd.a <= i || nd.b <= i || nd.a >= n_nodes || nd.b >= n_nodes)
    {
        atomicOr(status, ST_CAPACITY);
        gn[i] = rt_gnode{ make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f),
                          make_uint4(0u, 0u, LEAF_BIT, LEAF_BIT) };
        return;
    }
    const rt_bvh_node l = nodes[nd.a], r = nodes[nd.b];
    rt_gnode g;
    g.a = make_float4(l.bmin[0], l.bmax[0], l.bmin[1], l.bmax[1]);
    g.b = make_float4(l.bmin[2], l.bmax[2], r.bmin[0], r.bmax[0]);
    g.c = make_float4(r.bmin[1], r.bmax[1], r.bmin[2], r.bmax[2]);
    g.d = make_uint4(l.is_leaf ? l.a : nd.a, r.is_leaf ? r.a : nd.b, l.is_leaf ? (LEAF_BIT | l.b) : 0u,
                     r.is_leaf ? (LEAF_BIT | r.b) : 0u);
    gn[i] = g;
    // a NaN plane makes the traversal take the general box test
    bool nan = false;
    for (int k = 0; k < 3; k++) { nan |= l.bmin[k] != l.bmin[k] || l.bmax[k] != l.bmax[k] || r.bmin[k] != r.bmin[k] || r.bmax[k] != r.bmax[k]; }
    if (nan) { *odd = 1u; }
}

__global__ void k_make_tripos(const rt_triangle* __restrict__ tris, uint32_t n, const uint32_t* __restrict__ d_counts,
                              const rt_vertex* __restrict__ v, float4* __restrict__ tp)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (d_counts) { n = d_counts[1]; }
    if (i >= n) { return; }
    const rt_triangle t = tris[i];
    const rt_vertex a = v[t.v[0]], b = v[t.v[1]], c = v[t.v[2]];
    tp[3 * i + 0] = make_float4(a.x, a.y, a.z, b.x);
    tp[3 * i + 1] = make_float4(b.y, b.z, c.x, c.y);
    tp[3 * i + 2] = make_float4(c.z, 0.f, 0.f, 0.f);
}

// Entry record of each scene root of a batched build; d_counts[0] = node count. A root
// outside the node array (a record the build did not write) sets ST_CAPACITY.
__global__ void k_scene_roots(const rt_bvh_node* __restrict__ nodes, const uint32_t* __restrict__ info, uint32_t S,
                              const uint32_t* __restrict__ d_counts, TraceRoot* __restrict__ out,
                              uint32_t* __restrict__ status)
{
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= S) { return; }
    if (info[4 * s] >= d_counts[0])
    {
        atomicOr(status, ST_CAPACITY);
        out[s] = TraceRoot{ { 0.f, 0.f, 0.f, 0.f, 0.f, 0.f }, 0u, LEAF_BIT };
        return;
    }
    const rt_bvh_node nd = nodes[info[4 * s]];
    TraceRoot r;
    for (int k = 0; k < 3; k++) { r.box[k] = nd.bmin[k]; r.box[3 + k] = nd.bmax[k]; }
    r.ref = nd.is_leaf ? nd.a : info[4 * s];
    r.cnt = nd.is_leaf ? (LEAF_BIT | nd.b) : 0u;
    out[s] = r;
}

// Tree depth: parent links (children of node i have larger indices), then every leaf counts
// its ancestors (bounded by the node count).
__global__ void k_parents(const rt_bvh_node* __restrict__ nodes, uint32_t n, uint32_t* __restrict__ par)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) { return; }
    if (i == 0) { par[0] = 0xffffffffu; }
    const rt_bvh_node nd = nodes[i];
    if (!nd.is_leaf && nd.a < n && nd.b < n) { par[nd.a] = i; par[nd.b] = i; }
}
__global__ void k_depth(const rt_bvh_node* __restrict__ nodes, uint32_t n, const uint32_t* __restrict__ par,
                        uint32_t* __restrict__ depth)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || !nodes[i].is_leaf) { return; }
    uint32_t d = 0;
    for (uint32_t p = par[i]; p != 0xffffffffu && d < n; p = par[p]) { d++; }
    atomicMax(depth, d);
}

// The hit record of a finished ray.
__device__ __forceinline__ void write_hit(const TraceCtx& T, float4* __restrict__ hits, uint64_t ri, bool hit, bool overflow,
                                          float t, float u, float v, uint32_t tri, uint32_t* __restrict__ status)
{
    float4 h0 = make_float4(0.f, 0.f, 0.f, 0.f), h1 = make_float4(0.f, 0.f, 0.f, 0.f);
    uint32_t flags = 0;
    if (hit)
    {
        const f3 nrm = hit_normal(T, tri, u, v);
        h0 = make_float4(t, u, v, __uint_as_float(tri));
        h1 = make_float4(nrm.x, nrm.y, nrm.z, 0.f);
        flags = RT_HIT_FLAG_HIT;
    }
    if (overflow) { flags |= RT_HIT_FLAG_OVERFLOW; *static_cast<volatile uint32_t*>(status) = ST_STACK; }
    h1.w = __uint_as_float(flags);
    hits[2 * ri] = h0;
    hits[2 * ri + 1] = h1;
}

// rt_ray records in, rt_hit records out (two 128-bit accesses each). A warp holds at most `per_warp`
// rays at a time; without a counter it traces those of its own index only. status: a word of the host's.
template <int MODE>
__global__ void __launch_bounds__(256, 4)
k_trace(TraceCtx T, const float4* __restrict__ rays, float4* __restrict__ hits, uint64_t n,
        unsigned long long* __restrict__ counter, uint32_t* __restrict__ status, int per_warp)
{
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr unsigned FULL = 0xffffffffu;
    WarpShare& S = reinterpret_cast<WarpShare*>(smem)[threadIdx.x >> 5];
    const int lane = (int)(threadIdx.x & 31u);
    const unsigned lanes = per_warp >= 32 ? FULL : (1u << per_warp) - 1u;
    const int refill = per_warp >= 32 ? REFILL : (per_warp + 1) / 2;
    const bool odd_tree = *T.odd != 0u;
    LaneTrace<MODE, STACK> L;
    uint2 stk[STACK];
    L.live = false;
    bool pending = false, more = true;  // this lane has a result to write; rays are left
    for (;;)
    {
        const unsigned idle = __ballot_sync(FULL, !L.live) & lanes;
        if (idle == lanes || (more && __popc(idle) >= refill))
        {
            if (!L.live && pending)
            {
                pending = false;
                const float4 h = S.hit[lane];
                write_hit(T, hits, S.id[lane], L.hit, L.overflow, L.best, h.x, h.y, __float_as_uint(h.z), status);
            }
            if (!more) { break; }
            unsigned long long base = 0;
            if (counter)
            {
                if (lane == 0) { base = atomicAdd(counter, (unsigned long long)__popc(idle)); }
                base = __shfl_sync(FULL, base, 0);
                if (base + __popc(idle) >= n) { more = false; }
            }
            else
            {
                base = ((uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * (uint64_t)per_warp;
                more = false;
            }
            if ((idle >> lane) & 1u)
            {
                const uint64_t ri = base + __popc(idle & ((1u << lane) - 1u));
                if (ri < n)
                {
                    const float4 r0 = rays[2 * ri], r1 = rays[2 * ri + 1];
                    L.start(S, *T.root, r0, r1, odd_tree);
                    S.id[lane] = ri;
                    pending = true;
                }
            }
            __syncwarp();
            continue;
        }
        warp_walk<MODE, STACK>(L, stk, T, more ? lanes : 0u, refill);
        warp_leaves<MODE, STACK>(L, stk, T, S);
    }
}

// The 8-wide layout's kernel: each warp claims 32 rays at a time until the batch is exhausted; without a
// counter it traces the `per_warp` of its own index.
template <int MODE>
__global__ void __launch_bounds__(256)
k_trace_wide(TraceCtx T, const float4* __restrict__ rays, float4* __restrict__ hits, uint64_t n,
             unsigned long long* __restrict__ counter, uint32_t* __restrict__ status, int per_warp)
{
    const int lane = threadIdx.x & 31;
    const TraceRoot R = *T.root;
    for (bool more = true; more; more = counter != nullptr)
    {
        unsigned long long base = ((uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * (uint64_t)per_warp;
        if (counter)
        {
            if (lane == 0) { base = atomicAdd(counter, 32ull); }
            base = __shfl_sync(0xffffffffu, base, 0);
        }
        if (base >= n) { return; }
        const uint64_t ri = base + (uint64_t)lane;
        if (ri >= n || lane >= per_warp) { continue; }
        const float4 r0 = rays[2 * ri], r1 = rays[2 * ri + 1];
        const THit H = trace_ray_wide<MODE, STACK>(T, R, mk3(r0.x, r0.y, r0.z), mk3(r1.x, r1.y, r1.z), r0.w, r1.w);
        write_hit(T, hits, ri, H.hit, H.overflow, H.t, H.u, H.v, H.tri, status);
    }
}

using TraceFn = void (*)(TraceCtx, const float4*, float4*, uint64_t, unsigned long long*, uint32_t*, int);

TraceFn trace_fn(uint32_t flags, bool wide)
{
    switch (flags & 3u)
    {
    case 0: return wide ? k_trace_wide<0> : k_trace<0>;
    case 1: return wide ? k_trace_wide<1> : k_trace<1>;
    case 2: return wide ? k_trace_wide<2> : k_trace<2>;
    default: return wide ? k_trace_wide<3> : k_trace<3>;
    }
}

// Resident blocks per SM, per device, kernel variant and block size.
std::mutex g_occ_mu;
struct OccKey { const void* fn; int device, block, v; };
std::vector<OccKey> g_occ;

} // namespace

int blocks_per_sm(const void* fn, int block, size_t smem)
{
    int device = 0;
    cudaGetDevice(&device);
    std::lock_guard<std::mutex> lk(g_occ_mu);
    for (const OccKey& k : g_occ)
    {
        if (k.fn == fn && k.device == device && k.block == block) { return k.v; }
    }
    int v = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, fn, block, smem) != cudaSuccess) { cudaGetLastError(); v = 1; }
    if (v < 1) { v = 1; }
    g_occ.push_back(OccKey{ fn, device, block, v });
    return v;
}

TraceCtx make_trace_ctx(const rt_bvh* B)
{
    TraceCtx T;
    T.gn = B->gnodes.as<rt_gnode>();
    T.tp = B->tripos.as<float4>();
    T.tris = B->tris.as<rt_triangle>();
    T.verts = B->verts.as<rt_vertex>();
    T.root = B->rootbuf.as<TraceRoot>();
    T.odd = reinterpret_cast<const uint32_t*>(T.root + 1);
    T.ww = B->trace_ww ? 1u : 0u;
    T.wn = B->wnodes.as<rt_wnode>();
    T.wid = B->wid.as<uint32_t>();
    return T;
}

int launch_traversal_layout(rt_bvh* B, cudaStream_t st, uint32_t max_nodes, uint32_t max_tris, const uint32_t* d_counts,
                            uint32_t* vstatus, bool tripos_ready, bool gnodes_ready)
{
    if (B->gnodes.ensure((size_t)max_nodes * sizeof(rt_gnode)) || B->tripos.ensure((size_t)(max_tris ? max_tris : 1) * 48) ||
        B->rootbuf.ensure(ROOT_RECORD_BYTES))
    {
        return RT_E_CUDA;
    }
    if (!gnodes_ready)
    {
        uint32_t* odd = reinterpret_cast<uint32_t*>(B->rootbuf.as<TraceRoot>() + 1);  // zeroed by the caller
        k_make_gnodes<<<(max_nodes + 255) / 256, 256, 0, st>>>(B->nodes.as<rt_bvh_node>(), max_nodes, max_tris, d_counts,
                                                               B->gnodes.as<rt_gnode>(), B->rootbuf.as<TraceRoot>(), odd, vstatus);
        count_launch();
    }
    if (max_tris && !tripos_ready)
    {
        k_make_tripos<<<(max_tris + 255) / 256, 256, 0, st>>>(B->tris.as<rt_triangle>(), max_tris, d_counts,
                                                              B->verts.as<rt_vertex>(), B->tripos.as<float4>());
        count_launch();
    }
    return check_launch("traversal layout");
}

int make_traversal_layout(rt_bvh* B, cudaStream_t st)
{
    if (B->n_nodes == 0) { return fail(RT_E_EMPTY, "empty BVH"); }
    if (B->trace_status.ensure(64) || B->rootbuf.ensure(ROOT_RECORD_BYTES)) { return RT_E_CUDA; }
    RT_CUDA(cudaMemsetAsync(B->rootbuf.as<TraceRoot>() + 1, 0, 4, st));
    uint32_t* vstatus = B->trace_status.as<uint32_t>() + 12;
    RT_CUDA(cudaMemsetAsync(vstatus, 0, 4, st));
    if (int e = launch_traversal_layout(B, st, B->n_nodes, B->n_tris, nullptr, vstatus)) { return e; }
    uint32_t vs = 0;
    RT_CUDA(cudaMemcpyAsync(&vs, vstatus, 4, cudaMemcpyDeviceToHost, st));
    RT_CUDA(cudaStreamSynchronize(st));
    if (vs) { return fail(RT_E_FORMAT, "BVH structure check failed (child or triangle index out of range)"); }
    return RT_OK;
}

int launch_scene_roots(rt_bvh* B, uint32_t S, const uint32_t* d_counts, uint32_t* status, cudaStream_t st)
{
    k_scene_roots<<<(S + 127) / 128, 128, 0, st>>>(B->nodes.as<rt_bvh_node>(), B->scene_info.as<uint32_t>(), S, d_counts,
                                                   B->scene_roots.as<TraceRoot>(), status);
    count_launch();
    return check_launch("scene roots");
}

int tree_depth(rt_bvh* B, cudaStream_t st, uint32_t* depth)
{
    if (B->depth) { *depth = B->depth; return RT_OK; }
    const uint32_t n = B->n_nodes;
    DevBuf tmp;
    if (tmp.ensure((size_t)n * 4 + 16)) { return RT_E_CUDA; }
    uint32_t* par = tmp.as<uint32_t>();
    uint32_t* d = par + n;
    int e = RT_OK;
    if (cudaMemsetAsync(d, 0, 4, st) != cudaSuccess) { e = fail(RT_E_CUDA, "memset"); }
    if (!e)
    {
        k_parents<<<(n + 255) / 256, 256, 0, st>>>(B->nodes.as<rt_bvh_node>(), n, par);
        k_depth<<<(n + 255) / 256, 256, 0, st>>>(B->nodes.as<rt_bvh_node>(), n, par, d);
        count_launch(2);
        e = check_launch("depth");
    }
    uint32_t v = 0;
    if (!e && (cudaMemcpyAsync(&v, d, 4, cudaMemcpyDeviceToHost, st) != cudaSuccess || cudaStreamSynchronize(st) != cudaSuccess))
    {
        e = fail(RT_E_CUDA, "depth readback");
    }
    tmp.release();
    if (e) { return e; }
    B->depth = v;
    *depth = v;
    return RT_OK;
}

int trace(const rt_bvh* B, const rt_ray* d_rays, rt_hit* d_hits, uint64_t n, uint32_t flags, cudaStream_t st,
          uint32_t* status)
{
    if (n == 0) { return RT_OK; }
    if (((uintptr_t)d_rays & 15) || ((uintptr_t)d_hits & 15)) { return fail(RT_E_INVALID, "rays/hits must be 16-byte aligned"); }
    const TraceFn fn = trace_fn(flags, B->trace_wide);
    constexpr uint64_t WPB = TBLK / 32;
    const size_t smem = B->trace_wide ? 0 : WPB * sizeof(WarpShare);
    uint64_t grid = (uint64_t)device_sm_count() * (uint64_t)blocks_per_sm(reinterpret_cast<const void*>(fn), TBLK, smem);
    // Few rays are spread over the resident warps, down to one ray per warp: the lanes without
    // a ray still test its leaves' triangles. Every warp then has its rays at once, so they are
    // assigned by index: no counter to clear before the launch and to wait for at its start.
    const uint64_t warps = grid * WPB;
    const bool few = n <= warps * 32;
    const uint64_t per_warp = few ? std::max<uint64_t>(1, (n + warps - 1) / warps) : 32;
    grid = std::min(grid, (n + per_warp * WPB - 1) / (per_warp * WPB));
    // The counter is the call's own: calls on a handle may run at the same time.
    CallScratch counter;
    if (!few)
    {
        if (int e = counter.get(8, st)) { return e; }
        RT_CUDA(cudaMemsetAsync(counter.as<void>(), 0, 8, st));
    }
    const TraceCtx T = make_trace_ctx(B);
    fn<<<(uint32_t)grid, TBLK, smem, st>>>(T, reinterpret_cast<const float4*>(d_rays), reinterpret_cast<float4*>(d_hits), n,
                                           counter.as<unsigned long long>(), status, (int)per_warp);
    count_launch();
    return check_launch("trace");
}

} // namespace rtb
