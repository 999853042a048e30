// Contact phase kernels: narrow phase, manifold compaction, warm-start hash, sleeping-island wake, solver graph
// colouring, the sequential-impulse solver, islands and sleep flags, and work-list rebuilds. Reference routines are
// cited per kernel (paths relative to PhysicsSimulation-Agony/PS_AGONY2D/).
#include "ag2d_solver.cuh"

namespace ag2d {

__device__ __forceinline__ ColliderView collider_view(const DeviceWorld& w, uint32_t c)
{
    ColliderView v;
    const float4 p = w.cpose[c];
    v.pos = V2{p.x, p.y};
    v.c = p.z;
    v.s = p.w;
    const uint32_t packed = w.cshape[c];
    v.type = shape_type(packed);
    const uint32_t si = shape_index(packed);
    v.r = 0.0f; v.hw = 0.0f; v.hh = 0.0f; v.verts = nullptr; v.normals = nullptr; v.nv = 0;
    if (v.type == SHAPE_CIRCLE) {
        v.r = w.circleRadius[si];
    } else if (v.type == SHAPE_BOX) {
        const float2 h = w.boxHalf[si];
        v.hw = h.x; v.hh = h.y;
    } else if (v.type == SHAPE_CAPSULE) {
        const float2 h = w.boxHalf[si];   // capsules share the table: (half length, radius)
        v.hw = h.x; v.r = h.y;
    } else {
        const uint32_t off = w.polyOffset[si];
        v.verts = w.polyVerts + off;
        v.normals = w.polyNormals + off;
        v.nv = w.polyCount[si];
    }
    return v;
}

// ---------------------------------------------------------------------------------------------------------------
// Narrow phase: NarrowPhaseCollisionDetector::processPairs orientation (NarrowPhaseCollisionDetector.cpp:649-668:
// lower shape type first, equal types put the higher collider index first) and the shape-pair method. One thread
// per candidate pair writes the pair's manifold slot and a hit flag; a scan then compacts hits in pair order.
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void write_slot(const Contact& ct, uint32_t a, uint32_t b, Manifold* slot)
{
    Manifold m;
    m.a = a; m.b = b; m.nx = ct.n.x; m.ny = ct.n.y; m.depth = ct.depth; m.count = ct.count;
    m.id0 = ct.id[0]; m.px0 = ct.p[0].x; m.py0 = ct.p[0].y;
    if (ct.count > 1) { m.id1 = ct.id[1]; m.px1 = ct.p[1].x; m.py1 = ct.p[1].y; }
    else { m.id1 = 0; m.px1 = 0.0f; m.py1 = 0.0f; }
    m.jn0 = 0.0f; m.jt0 = 0.0f; m.jn1 = 0.0f; m.jt1 = 0.0f;
    *slot = m;
}

// The warm start of new manifold 'm' (index o of the step's list): its pair's impulses and colour of the last step. True
// when it took an impulse.
__device__ __forceinline__ bool warm_take(const WarmTable& t, Manifold& m, uint32_t o)
{
    const unsigned long long key = pair_key(m.a, m.b);
    const WarmRegion r = warm_region(t, m.a);
    uint32_t idx = NO_COLOR;
    if (r.size) {
        uint32_t s = r.home(key);
        for (uint32_t probes = 0; probes < r.size; probes++) {
            const unsigned long long k = t.keys[s];
            if (k == key) { idx = t.vals[s]; break; }
            if (k == ~0ull) break;
            s = r.next(s);
        }
    }
    if (t.hint) t.hint[o] = (idx != NO_COLOR && t.prevColor) ? t.prevColor[idx & ~WARM_CACHED] : NO_COLOR;
    if (idx == NO_COLOR || !(idx & WARM_CACHED)) return false;
    const Manifold p = t.prev[idx & ~WARM_CACHED];
    if (p.a != m.a || p.b != m.b) return false;
    bool any = false;
    for (uint32_t k = 0; k < m.count; k++) {
        const uint32_t id = k == 0 ? m.id0 : m.id1;
        float jn, jt;
        if (p.count > 0 && id == p.id0) { jn = p.jn0; jt = p.jt0; }
        else if (p.count > 1 && id == p.id1) { jn = p.jn1; jt = p.jt1; }
        else continue;
        if (k == 0) { m.jn0 = jn; m.jt0 = jt; } else { m.jn1 = jn; m.jt1 = jt; }
        any = true;
    }
    return any;
}

// Marks the islands of a manifold's sleeping bodies to wake. Island ids are body indices (the island's root);
// anything else is ignored rather than written.
__device__ __forceinline__ void mark_wakes(const DeviceWorld& w, const Manifold& m, uint32_t* wakeIsland)
{
    const uint32_t bA = w.cbody[m.a], bB = w.cbody[m.b];
    if (w.bstate[bA] == STATE_SLEEPING && w.sleepIsland[bA] < w.nBodies) wakeIsland[w.sleepIsland[bA]] = 1u;
    if (w.bstate[bB] == STATE_SLEEPING && w.sleepIsland[bB] < w.nBodies) wakeIsland[w.sleepIsland[bB]] = 1u;
}

// Narrow phase with the manifold compaction fused in. Blocks take tiles of consecutive pairs in ticket order (tileState
// and the ticket counter zeroed before the launch); in a tile each warp takes perWarp pairs (at most 32), one per
// lane. Pairs of other shape types run one per lane; the warp's polygon-polygon pairs search their axes four at a time,
// one per group of NARROW_GROUP lanes (collide_polygon_polygon_group), and are then clipped one per lane. A group's
// search takes about 1.5 us, so a step with few pairs spreads them over more warps (perWarp 4 is one search a warp)
// and one with many keeps every lane of the one-per-lane parts busy. Each pair's manifold goes to its slot in shared
// memory; the tile's hits are then counted (warp ballots, then a scan of the warps' counts), its output offset
// comes from the decoupled look-back over the preceding tiles, and the hit pairs' manifolds are copied straight to
// their places: manifolds come out in pair order. The last tile writes the manifold count. Launched with a
// multiple of 32 threads (at most 1024) and NARROW_SMEM_PER_THREAD bytes of dynamic shared memory per thread.
// LANES: a warp with more than NARROW_LANES_PAIRS polygon pairs searches and clips them one a lane
// (collide_polygon_polygon_lane) in place of the groups' rounds: 3.7 M polygon pairs (2.7 M manifolds) 1,255 -> 830 us, a
// third of the instructions. Bound now by latency: 32 warps an SM, most stalls at the tile's barriers and on loads (24
// warps with more registers: 863; normals loaded one an axis: 905; tiles of 128 pairs: 979).
template <bool LANES>
__global__ void __launch_bounds__(LANES ? NARROW_LANES_THREADS : 512, LANES ? 4 : 2) k_narrow(DeviceWorld w, const uint2* pairs, const uint32_t* nPairs,
                         uint32_t pairCap, Manifold* out, uint32_t manifoldCap,
                         uint32_t* nOut, StepCounters* counters, uint32_t* tileState,
                         uint32_t* tileCounter, uint32_t perWarp, WarmTable warm,
                         uint32_t* wakeIsland)
{
    chain_begin();
    extern __shared__ __align__(16) unsigned char narrowSmem[];
    // [blockDim] manifold slots, [blockDim] hit flags, then per group A's vertices and B's (in A's frame).
    Manifold* const slot = reinterpret_cast<Manifold*>(narrowSmem);
    uint32_t* const hitS = reinterpret_cast<uint32_t*>(narrowSmem + blockDim.x * sizeof(Manifold));
    V2* const tiles = reinterpret_cast<V2*>(narrowSmem + blockDim.x * (sizeof(Manifold) + sizeof(uint32_t)));
    __shared__ uint32_t warpBase[32];
    __shared__ uint32_t tileSlot, tileBase;
    const uint32_t n = min(*nPairs, pairCap);
    if (n == 0) {
        if (blockIdx.x == 0 && threadIdx.x == 0) { *nOut = 0u; counters->manifolds = 0u; }
        return;
    }
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nWarps = blockDim.x >> 5;
    const uint32_t tilePairs = nWarps * perWarp;
    const uint32_t tiles_n = (n + tilePairs - 1) / tilePairs;
    const uint32_t group = lane / NARROW_GROUP, gl = lane % NARROW_GROUP;
    const uint32_t gmask = ((1u << NARROW_GROUP) - 1u) << (group * NARROW_GROUP);
    V2* const sA = tiles + (threadIdx.x / NARROW_GROUP) * 2 * MAX_POLYGON_VERTICES;
    V2* const sB = sA + MAX_POLYGON_VERTICES;
    const uint32_t warpFirst = warp * 32;
    while (true) {
        if (threadIdx.x == 0) tileSlot = atomicAdd(tileCounter, 1u);
        __syncthreads();
        const uint32_t tile = tileSlot;
        if (tile >= tiles_n) return;
        const uint32_t p = tile * tilePairs + warp * perWarp + lane;
        const bool valid = lane < perWarp && p < n;
        uint32_t a = 0, b = 0;
        bool pp = false;
        hitS[threadIdx.x] = 0u;
        if (valid) {
            a = pairs[p].x;
            b = pairs[p].y;
            const uint32_t ta = shape_type(w.cshape[a]), tb = shape_type(w.cshape[b]);
            if (ta > tb || (ta == tb && b > a)) { const uint32_t t = a; a = b; b = t; }
            pp = ta == SHAPE_POLYGON && tb == SHAPE_POLYGON;
            if (!pp) {
                const ColliderView A = collider_view(w, a), B = collider_view(w, b);
                Contact ct;
                if (collide(A, B, ct)) {
                    hitS[threadIdx.x] = 1u;
                    write_slot(ct, a, b, slot + threadIdx.x);
                }
            }
        }
        const uint32_t polygons = __ballot_sync(0xffffffffu, pp);
        bool alone = false;   // searched by its own lane
        if (LANES && pp && __popc(polygons) > NARROW_LANES_PAIRS) {
            const ColliderView A = collider_view(w, a), B = collider_view(w, b);
            if (max(A.nv, B.nv) <= SAT_LANE_VERTICES) {
                alone = true;
                float depth;
                uint32_t edges;
                Contact ct;
                if (collide_polygon_polygon_lane(A, B, depth, edges) &&
                    collide_polygon_polygon_clip(A, B, depth, edges, ct)) {
                    hitS[threadIdx.x] = 1u;
                    write_slot(ct, a, b, slot + threadIdx.x);
                }
            }
        }
        uint32_t todo = LANES ? __ballot_sync(0xffffffffu, pp && !alone) : polygons;
        while (todo) {
            // Group g takes the g-th remaining polygon-polygon lane; its leader writes that pair's slot and flag.
            uint32_t pick = todo;
            for (uint32_t k = 0; k < group && pick; k++) pick &= pick - 1;
            const bool has = pick != 0;
            const uint32_t src = has ? uint32_t(__ffs(pick) - 1) : 0u;
            const uint32_t ga = __shfl_sync(0xffffffffu, a, src), gb = __shfl_sync(0xffffffffu, b, src);
            for (uint32_t k = 0; k < 32 / NARROW_GROUP && todo; k++) todo &= todo - 1;
            if (has) {
                const ColliderView A = collider_view(w, ga), B = collider_view(w, gb);
                float depth;
                uint32_t edges;
                const bool h = collide_polygon_polygon_group(A, B, depth, edges, gl, gmask, sA, sB);
                if (gl == 0 && h) {
                    hitS[warpFirst + src] = 1u;
                    slot[warpFirst + src].depth = depth;
                    slot[warpFirst + src].id0 = edges;
                }
                __syncwarp(gmask);   // the group's tiles are reused by its next pair
            }
        }
        __syncwarp();
        if (pp && !alone && hitS[threadIdx.x]) {
            const ColliderView A = collider_view(w, a), B = collider_view(w, b);
            Contact ct;
            if (collide_polygon_polygon_clip(A, B, slot[threadIdx.x].depth, slot[threadIdx.x].id0, ct))
                write_slot(ct, a, b, slot + threadIdx.x);
            else
                hitS[threadIdx.x] = 0u;
        }
        const bool h = hitS[threadIdx.x] != 0u;
        // Output offsets: the tile's hits in pair order after those of the preceding tiles.
        const uint32_t hits = __ballot_sync(0xffffffffu, h);
        if (lane == 0) warpBase[warp] = __popc(hits);
        __syncthreads();
        if (warp == 0) {
            const uint32_t c = lane < nWarps ? warpBase[lane] : 0u;
            uint32_t incl = c;
            for (uint32_t o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            const uint32_t aggregate = __shfl_sync(0xffffffffu, incl, 31);
            if (lane < nWarps) warpBase[lane] = incl - c;
            volatile uint32_t* state = tileState;
            uint32_t prefix = 0;
            if (tile == 0) {
                if (lane == 0) state[0] = (2u << 30) | aggregate;
            } else {
                if (lane == 0) state[tile] = (1u << 30) | aggregate;
                prefix = scan_lookback(tile, tileState, &counters->status);
                if (lane == 0) state[tile] = (2u << 30) | (prefix + aggregate);
            }
            if (lane == 0) {
                tileBase = prefix;
                if (tile == tiles_n - 1) {
                    const uint32_t total = prefix + aggregate;
                    counters->manifolds = total;
                    *nOut = min(total, manifoldCap);
                    if (total > manifoldCap) atomicOr(&counters->status, STATUS_MANIFOLD_OVERFLOW);
                }
            }
        }
        __syncthreads();
        if (h) {
            const uint32_t o = tileBase + warpBase[warp] + __popc(hits & ((1u << lane) - 1u));
            if (o < manifoldCap) {
                if (warm.keys && warm_take(warm, slot[threadIdx.x], o)) atomicAdd(&counters->warmHits, 1u);
                if (wakeIsland) mark_wakes(w, slot[threadIdx.x], wakeIsland);
                out[o] = slot[threadIdx.x];
            }
        }
        __syncthreads();   // tileSlot, tileBase, warpBase, the slots and the vertex tiles are reused by the next tile
    }
}

cudaError_t narrow_init()
{
    return cudaFuncSetAttribute(k_narrow<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                int(512 * NARROW_SMEM_PER_THREAD));
}

cudaError_t launch_narrow(bool chained, uint32_t blocks, uint32_t threads, cudaStream_t stream, DeviceWorld w, const uint2* pairs,
                   const uint32_t* nPairs, uint32_t pairCap, Manifold* out, uint32_t manifoldCap, uint32_t* nOut,
                   StepCounters* counters, uint32_t* tileState, uint32_t* tileCounter, uint32_t perWarp, bool lanes,
                   WarmTable warm, uint32_t* wakeIsland)
{
    return chain_launch(chained, lanes && threads <= NARROW_LANES_THREADS ? k_narrow<true> : k_narrow<false>, blocks, threads,
                        size_t(threads) * NARROW_SMEM_PER_THREAD, stream, w, pairs, nPairs, pairCap, out, manifoldCap,
                        nOut, counters, tileState, tileCounter, perWarp, warm, wakeIsland);
}

__global__ void k_warm_insert(WarmTable t) { warm_insert(t); }

// ---------------------------------------------------------------------------------------------------------------
// Wake: every sleeping body in a manifold wakes its whole island (ObjectManager::wakeIslandsOfContacts,
// SimulationImpl/ObjectManager.h:139-157; wakeOne resets the sleep timer, ObjectManager.cpp:1344-1361).
// ---------------------------------------------------------------------------------------------------------------
__global__ void k_wake(DeviceWorld w, const Manifold* __restrict__ m, const uint32_t* __restrict__ nM,
                       uint32_t* __restrict__ wakeIsland, StepCounters* counters)
{
    const uint32_t n = *nM;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        mark_wakes(w, m[i], wakeIsland);
}

__global__ void k_wake_apply(DeviceWorld w, const uint32_t* wakeIsland, StepCounters* counters)
{
    chain_begin();
    uint32_t woke = 0;
    for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b < w.nBodies; b += gridDim.x * blockDim.x) {
        if (w.bstate[b] == STATE_SLEEPING && w.sleepIsland[b] < w.nBodies && wakeIsland[w.sleepIsland[b]]) {
            w.bstate[b] = STATE_DYNAMIC;
            w.sleepTimer[b] = 0.0f;
            if (w.worldDirty) w.worldDirty[w.bodyWorld[b]] = 1u;
            woke++;
        }
    }
    for (int o = 16; o > 0; o >>= 1) woke += __shfl_xor_sync(0xffffffffu, woke, o);
    if ((threadIdx.x & 31) == 0 && woke) {
        atomicAdd(&counters->woke, woke);
        counters->topoDirty = 1u;
    }
}

// ---------------------------------------------------------------------------------------------------------------
// Colouring + solve entry points (ag2d_solver.cuh). Two manifolds conflict when they share a body with non-zero
// inverse mass (static bodies are never written; the reference's planner makes the same exception:
// Solving/SolvingPlanner.cpp:85-88). Colours are independent sets, so solving colour after colour equals a
// sequential Gauss-Seidel sweep in colour-major order.
// ---------------------------------------------------------------------------------------------------------------

// A body's state and its version in one 16-byte word, read and written whole: a reader that sees the version it waits
// for has the state that goes with it, without fences.
__device__ __forceinline__ float4 flow_load(const float4* p)
{
    unsigned long long lo, hi;
    asm volatile("{\n\t.reg .b128 d;\n\tld.relaxed.gpu.global.b128 d, [%2];\n\tmov.b128 {%0, %1}, d;\n\t}"
                 : "=l"(lo), "=l"(hi) : "l"(p) : "memory");
    return make_float4(__uint_as_float(uint32_t(lo)), __uint_as_float(uint32_t(lo >> 32)),
                       __uint_as_float(uint32_t(hi)), __uint_as_float(uint32_t(hi >> 32)));
}
__device__ __forceinline__ void flow_store(float4* p, const float4& v)
{
    const unsigned long long lo = uint64_t(__float_as_uint(v.x)) | uint64_t(__float_as_uint(v.y)) << 32;
    const unsigned long long hi = uint64_t(__float_as_uint(v.z)) | uint64_t(__float_as_uint(v.w)) << 32;
    asm volatile("{\n\t.reg .b128 s;\n\tmov.b128 s, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], s;\n\t}"
                 :: "l"(p), "l"(lo), "l"(hi) : "memory");
}

// One end of a constraint in the dataflow: waits until its body's version is 'need' (a body without a version, of
// infinite mass, is always ready). Polled by a whole warp; false when the wait ran out somewhere on the grid, or when a
// body is past the version waited for, which then never comes.
struct FlowEnd {
    const float4* at;   // null: nothing to wait for
    uint32_t need;
};
__device__ __forceinline__ bool flow_wait(const FlowEnd& a, const FlowEnd& b, float4& va, float4& vb,
                                          const volatile uint32_t* status, uint32_t* statusOut)
{
    bool ra = a.at == nullptr, rb = b.at == nullptr;
    for (uint32_t spins = 0;; spins++) {
        uint32_t gap = 0;   // updates still missing on the body that lacks most
        if (!ra) {
            va = flow_load(a.at);
            gap = a.need - __float_as_uint(va.w);
            ra = gap == 0;
        }
        if (!rb) {
            vb = flow_load(b.at);
            const uint32_t missing = b.need - __float_as_uint(vb.w);
            rb = missing == 0;
            gap = max(gap, missing);
        }
        gap = __reduce_max_sync(0xffffffffu, gap);
        if (gap == 0) return true;
        if (int32_t(gap) < 0) { atomicOr(statusOut, STATUS_SOLVER_STATE); return false; }
        // The missing updates follow one another, half a microsecond each at least: a warp that lacks several sleeps
        // instead of loading the L2 with its polls (all waiting warps polling: 2.5 us a hop).
        if (gap > 1u) __nanosleep(min(gap - 1u, 8u) * 300u);
        if ((spins & 1023u) == 1023u) {
            const bool gone = (*status & (STATUS_BARRIER_TIMEOUT | STATUS_SOLVER_STATE)) != 0;
            if (__any_sync(0xffffffffu, gone)) return false;
            if (spins > SPIN_LIMIT) { atomicOr(statusOut, STATUS_BARRIER_TIMEOUT); return false; }
        }
    }
}

// Whether slot c holds a record to solve. Every slot below a colour's end has one, made by the lane that reads it, with
// bodies of the world; any other is reported as what it is and skipped, and the waits on it end.
__device__ __forceinline__ bool flow_live(uint32_t c, const Constraint& k, uint32_t nBodies, uint32_t* status)
{
    if (c == 0xFFFFFFFFu) return false;
    if (k.bodyA < nBodies && k.bodyB < nBodies) return true;
    atomicOr(status, STATUS_SOLVER_STATE);
    return false;
}

// From a body's byte pair (rank, degree less one): the version its constraint waits for in pass p, and whether the
// constraint is the body's last one.
__device__ __forceinline__ uint32_t flow_need(uint32_t pass, uint32_t pair)
{
    return pass * (((pair >> 8) & 255u) + 1u) + (pair & 255u);
}
__device__ __forceinline__ bool flow_last(uint32_t pair) { return (pair & 255u) == ((pair >> 8) & 255u); }

// Islands' union-find in global memory (see k_island_union): links the bodies of one pair if both are dynamic.
__device__ __forceinline__ uint32_t uf_find(uint32_t* parent, uint32_t x)
{
    uint32_t p = __ldcg(parent + x);
    while (p != x) {
        const uint32_t gp = __ldcg(parent + p);
        if (gp != p) atomicCAS(parent + x, p, gp);   // path halving, benign races
        x = p;
        p = gp;
    }
    return x;
}
__device__ __forceinline__ void uf_link(const DeviceWorld& w, uint32_t* parent, uint32_t a, uint32_t b)
{
    if (w.bstate[a] != STATE_DYNAMIC || w.bstate[b] != STATE_DYNAMIC) return;
    for (uint32_t tries = 0; tries < 1u << 20; tries++) {
        uint32_t ra = uf_find(parent, a), rb = uf_find(parent, b);
        if (ra == rb) break;
        if (ra < rb) { const uint32_t t = ra; ra = rb; rb = t; }   // link the larger root under the smaller
        if (atomicCAS(parent + ra, ra, rb) == ra) break;
    }
}

// Walks a warp's items of one pass: the manifolds in colour-major order, every colour padded to whole warps, chunk q
// of 32 to warp q modulo the warps. A chunk has one colour, so its lanes never wait for one another.
struct FlowWalk {
    const uint32_t* start;    // colour starts (shared memory)
    const uint32_t* chunk;    // first chunk of every colour (shared memory), [ncol] = the chunk count
    uint32_t col;
    __device__ __forceinline__ void seek(uint32_t q) { while (q >= chunk[col + 1]) col++; }
    // This lane's slot of chunk q, or ~0u past the colour's end.
    __device__ __forceinline__ uint32_t slot(uint32_t q) const
    {
        const uint32_t c = start[col] + (q - chunk[col]) * 32u + (threadIdx.x & 31u);
        return c < start[col + 1] ? c : 0xFFFFFFFFu;
    }
};

// Colouring and solve of a large single world on a cooperative grid. The passes have no barriers: a body's constraints
// act on it in colour order, pass after pass, so its k-th update must follow its (k - 1)-th and nothing else. Every
// body carries a version (the updates made so far) in the same 16-byte word as its velocity, and a constraint, the
// r-th of the d around a body (both from the body's masks of colours), waits in pass p for version p d + r of each of
// its moving bodies. Warps take the constraints in colour order within a pass and the passes in order, all warps are
// resident, so the oldest unfinished constraint can always run. Velocity passes (warm start first) and position passes
// touch different state and run on warps of their own. The order of the updates of every body is that of the
// colour-major sweep, so the results are the same bit for bit.
// Bound: the chain of updates along the contacts (a pass costs about one hop a colour, a hop one L2 round trip for
// the store, half a poll and the arithmetic). With a grid barrier a colour instead, and on the sixteen SMs that one
// thread-block cluster has, a pass over the pile of 100,000 bodies (128,000 manifolds, 14 colours) took 8 us a colour.
// Colours beyond the 64 first-fit ones, which a body with that many contacts brings, have masks of their own, filled
// only then. With a grid barrier a colour instead, 7,200 compound bodies of 16 boxes (53,000 manifolds, 108 colours) took
// 5,528 us a solve, 1,793 here. Only a colouring with a tail is solved that way.
__global__ void __launch_bounds__(FLOW_THREADS, 1)
k_color_solve_flow(DeviceWorld w, Manifold* m, const uint32_t* nM, SolveScratch s, FlowScratch f, uint32_t velIters,
                   uint32_t posIters, uint32_t* bar, StepCounters* counters)
{
    const uint32_t rank = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t size = gridDim.x * blockDim.x;
    const uint32_t n = *nM;
    if (n == 0) return;
    const GlobalBodies B{w.bvel, w.bpos, s.bodyMax, s.bodyMask};
    const GridSync sync{bar, &counters->status};
    uint32_t ncol = 0;
    if (!color_manifolds(w, B, m, n, s, rank, size, sync, &counters->colors, &counters->status, ncol)) return;
    if (ncol > TAIL_COLOR) {   // a tail: no order by colours
        if (f.parent)
            for (uint32_t i = rank; i < n; i += size) uf_link(w, f.parent, w.cbody[m[i].a], w.cbody[m[i].b]);
        solve_colored(w, B, m, n, s, ncol, velIters, posIters, rank, size, sync);
        return;
    }
    if (ncol > 64u) {   // the colours above the first-fit ones, around each body
        for (uint32_t i = rank; i < FLOW_HIGH * w.nBodies; i += size) f.high[i] = 0ull;
        if (!sync()) return;
        for (uint32_t i = rank; i < n; i += size) {
            const uint32_t c = s.color[i] & COLOR_MASK;
            if (c < 64u) continue;
            const uint2 q = s.pairBodies[i];
            for (const uint32_t b : {q.x, q.y})
                if (b & PAIR_DYNAMIC)
                    atomicOr(f.high + FLOW_HIGH * (b & PAIR_BODY) + (c >> 6) - 1u, 1ull << (c & 63u));
        }
        if (!sync()) return;
    }
    __shared__ uint32_t start[MAX_COLORS + 1], chunk[MAX_COLORS + 1];
    for (uint32_t c = threadIdx.x; c <= ncol; c += blockDim.x) start[c] = __ldcg(s.colorStart + c);
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t run = 0;
        for (uint32_t c = 0; c < ncol; c++) { chunk[c] = run; run += (start[c + 1] - start[c] + 31u) >> 5; }
        chunk[ncol] = run;
    }
    __syncthreads();
    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t chunks = chunk[ncol];
    const volatile uint32_t* status = &counters->status;
    // Records of every manifold, before any velocity changes, each by the thread that solves it, and the bodies' words
    // at version 0.
    if (warp < FLOW_VEL_WARPS) {
        FlowWalk walk{start, chunk, 0};
        for (uint32_t q = warp * gridDim.x + blockIdx.x; q < chunks; q += FLOW_VEL_WARPS * gridDim.x) {
            walk.seek(q);
            const uint32_t c = walk.slot(q);
            if (c == 0xFFFFFFFFu) continue;
            const uint32_t mi = __ldcg(s.order + c);
            Constraint k;
            prep_constraint(w, B, m[mi], mi, k);
            // A movable body's byte pair: this colour's rank among those around it, and their number less one.
            auto place = [&](uint32_t b) {
                const unsigned long long below = (1ull << (walk.col & 63u)) - 1ull, first = __ldcg(s.bodyMask + b);
                uint32_t r = __popcll(walk.col < 64u ? first & below : first), d = __popcll(first);
                if (ncol > 64u)
                    for (uint32_t j = 0; j < FLOW_HIGH; j++) {
                        const unsigned long long mask = __ldcg(f.high + FLOW_HIGH * b + j);
                        const uint32_t word = walk.col >> 6;   // 0: the first-fit colours
                        if (j + 1u < word) r += __popcll(mask);
                        else if (j + 1u == word) r += __popcll(mask & below);
                        d += __popcll(mask);
                    }
                return r | (d - 1u) << 8;
            };
            uint32_t ranks = 0;
            if (k.imA > 0.0f) ranks |= place(k.bodyA);
            if (k.imB > 0.0f) ranks |= place(k.bodyB) << 16;
            k.pad = __uint_as_float(ranks);
            f.cons[c] = k;
            f.posA[c] = make_float4(k.nx, k.ny, k.penBase, __uint_as_float(ranks));
            f.posB[c] = make_float4(k.imA, k.imB, __uint_as_float(k.bodyA), __uint_as_float(k.bodyB));
        }
    }
    for (uint32_t b = rank; b < w.nBodies; b += size) {
        const float4 v = w.bvel[b], p = w.bpos[b];
        f.vel[b] = make_float4(v.x, v.y, v.z, 0.0f);
        f.pos[b] = make_float4(p.x, p.y, 0.0f, 0.0f);
    }
    if (!sync()) return;
    if (warp < FLOW_VEL_WARPS) {
        const uint32_t q0 = warp * gridDim.x + blockIdx.x, qStep = FLOW_VEL_WARPS * gridDim.x;
        if (q0 >= chunks) return;
        const bool one = q0 + qStep >= chunks;   // one chunk: its records stay in registers
        FlowWalk walk{start, chunk, 0};
        walk.seek(q0);
        uint32_t c = walk.slot(q0);
        Constraint k, nxt;
        if (c != 0xFFFFFFFFu) k = f.cons[c];
        for (uint32_t pass = 0; pass <= velIters; pass++) {
            for (uint32_t q = q0; q < chunks; q += qStep) {
                // The next record is fetched while this one waits for its bodies.
                uint32_t cNext = c;
                if (!one) {
                    uint32_t qn = q + qStep;
                    if (qn >= chunks) { qn = q0; walk.col = 0; }
                    walk.seek(qn);
                    cNext = walk.slot(qn);
                    if (cNext != 0xFFFFFFFFu) nxt = f.cons[cNext];
                }
                const bool live = flow_live(c, k, w.nBodies, &counters->status);
                const BlockMatrix bm = block_matrix(k);   // needs no body: done before the wait
                const uint32_t ranks = live ? __float_as_uint(k.pad) : 0u;
                const bool mA = live && k.imA > 0.0f, mB = live && k.imB > 0.0f;
                const FlowEnd a{mA ? f.vel + k.bodyA : nullptr, flow_need(pass, ranks)};
                const FlowEnd b{mB ? f.vel + k.bodyB : nullptr, flow_need(pass, ranks >> 16)};
                float4 vA = make_float4(0.0f, 0.0f, 0.0f, 0.0f), vB = vA;
                if (live && !mA) vA = w.bvel[k.bodyA];
                if (live && !mB) vB = w.bvel[k.bodyB];
                if (!flow_wait(a, b, vA, vB, status, &counters->status)) return;
                if (live) {
                    vA.w = k.imA;
                    vB.w = k.imB;
                    if (pass == 0) {
                        warm_solve(k, vA, vB);
                    } else {
                        velocity_solve(k, bm, vA, vB);
                        if (!one) *reinterpret_cast<float4*>(&f.cons[c].jn0) = make_float4(k.jn0, k.jt0, k.jn1, k.jt1);
                    }
                    if (mA) {
                        flow_store(f.vel + k.bodyA, make_float4(vA.x, vA.y, vA.z, __uint_as_float(a.need + 1u)));
                        if (pass == velIters && flow_last(ranks)) w.bvel[k.bodyA] = vA;
                    }
                    if (mB) {
                        flow_store(f.vel + k.bodyB, make_float4(vB.x, vB.y, vB.z, __uint_as_float(b.need + 1u)));
                        if (pass == velIters && flow_last(ranks >> 16)) w.bvel[k.bodyB] = vB;
                    }
                    if (pass == velIters) {
                        Manifold& d = m[k.manifold];
                        d.jn0 = k.jn0; d.jt0 = k.jt0; d.jn1 = k.jn1; d.jt1 = k.jt1;
                    }
                }
                if (!one) { k = nxt; c = cNext; }
            }
        }
    } else {
        const uint32_t q0 = (warp - FLOW_VEL_WARPS) * gridDim.x + blockIdx.x, qStep = FLOW_POS_WARPS * gridDim.x;
        for (uint32_t pass = 0; pass < posIters; pass++) {
            FlowWalk walk{start, chunk, 0};
            for (uint32_t q = q0; q < chunks; q += qStep) {
                walk.seek(q);
                const uint32_t c = walk.slot(q);
                Constraint k;
                uint32_t ranks = 0;
                k.imA = k.imB = 0.0f;
                if (c != 0xFFFFFFFFu) {
                    const float4 r0 = __ldcg(f.posA + c), r1 = __ldcg(f.posB + c);
                    k.nx = r0.x; k.ny = r0.y; k.penBase = r0.z; ranks = __float_as_uint(r0.w);
                    k.imA = r1.x; k.imB = r1.y; k.bodyA = __float_as_uint(r1.z); k.bodyB = __float_as_uint(r1.w);
                }
                const bool live = flow_live(c, k, w.nBodies, &counters->status);
                const bool mA = live && k.imA > 0.0f, mB = live && k.imB > 0.0f;
                const FlowEnd a{mA ? f.pos + k.bodyA : nullptr, flow_need(pass, ranks)};
                const FlowEnd b{mB ? f.pos + k.bodyB : nullptr, flow_need(pass, ranks >> 16)};
                float4 pA = make_float4(0.0f, 0.0f, 0.0f, 0.0f), pB = pA;
                if (live && !mA) pA = w.bpos[k.bodyA];
                if (live && !mB) pB = w.bpos[k.bodyB];
                if (!flow_wait(a, b, pA, pB, status, &counters->status)) return;
                if (live) {
                    position_solve(k, pA, pB);
                    if (mA) {
                        flow_store(f.pos + k.bodyA, make_float4(pA.x, pA.y, 0.0f, __uint_as_float(a.need + 1u)));
                        if (pass + 1u == posIters && flow_last(ranks))
                            *reinterpret_cast<float2*>(w.bpos + k.bodyA) = make_float2(pA.x, pA.y);
                    }
                    if (mB) {
                        flow_store(f.pos + k.bodyB, make_float4(pB.x, pB.y, 0.0f, __uint_as_float(b.need + 1u)));
                        if (pass + 1u == posIters && flow_last(ranks >> 16))
                            *reinterpret_cast<float2*>(w.bpos + k.bodyB) = make_float2(pB.x, pB.y);
                    }
                }
            }
        }
        // The position warps are done before the velocity warps: the islands are linked meanwhile.
        if (f.parent)
            for (uint32_t i = q0 * 32u + (threadIdx.x & 31u); i < n; i += qStep * 32u)
                uf_link(w, f.parent, w.cbody[m[i].a], w.cbody[m[i].b]);
    }
}

// Union-find over a parent array in shared or global memory (generic addressing; volatile reads see other SMs'
// links), linking the larger root under the smaller, so every island's root is its smallest body index whatever
// the order of the links (IslandManager's islands, the same roots k_island_union gives).
__device__ __forceinline__ uint32_t team_find(uint32_t* par, uint32_t x)
{
    volatile uint32_t* p = par;
    uint32_t px = p[x];
    for (uint32_t guard = 0; px != x && guard < (1u << 20); guard++) {
        const uint32_t gp = p[px];
        if (gp != px) p[x] = gp;   // path halving: x is no root, and any ancestor is a good parent
        x = px;
        px = gp;
    }
    return x;
}
__device__ __forceinline__ void team_union(uint32_t* par, uint32_t a, uint32_t b)
{
    for (uint32_t tries = 0; tries < (1u << 20); tries++) {
        uint32_t ra = team_find(par, a), rb = team_find(par, b);
        if (ra == rb) return;
        if (ra < rb) { const uint32_t t = ra; ra = rb; rb = t; }
        if (atomicCAS(par + ra, ra, rb) == ra) return;
    }
}

// A single world in one CTA: bodies in shared memory (colouring words first, SharedBodies lazy), then its islands.
template <uint32_t THREADS>
__global__ void __launch_bounds__(THREADS, 1) k_color_solve_block(BlockSolve a)
{
    chain_begin();
    extern __shared__ float4 teamCache[];
    __shared__ uint32_t colorCount[COLOR_SLOTS];
    __shared__ uint32_t colorStart[MAX_COLORS + 1];
    const DeviceWorld& w = a.w;
    const uint32_t n = *a.nM, nb = w.nBodies;
    uint32_t* par = reinterpret_cast<uint32_t*>(teamCache);
    if (n > 0) {
        float4* vel = teamCache;
        float4* pos = teamCache + a.bodyCap;
        auto* maxW = reinterpret_cast<unsigned long long*>(teamCache);
        unsigned long long* maskW = maxW + a.bodyCap;
        for (uint32_t i = threadIdx.x; i < nb; i += THREADS) {
            maxW[i] = 0ull;
            maskW[i] = 0ull;
        }
        __syncthreads();
        SharedBodies sb{vel, pos, maxW, maskW, 0u};
        sb.count = nb;
        sb.gvel = w.bvel;
        sb.gpos = w.bpos;
        SolveScratch s = a.s;
        s.colorCount = colorCount;
        s.colorStart = colorStart;
        const bool solved = color_and_solve<BlockSync, SharedBodies>(w, sb, a.m, n, s, a.velIters, a.posIters,
                                                                     threadIdx.x, THREADS, BlockSync{},
                                                                     &a.counters->colors, &a.counters->status);
        __syncthreads();
        if (!solved) {   // the step is redone or fails: the bodies stay as they were, every one its own island
            for (uint32_t i = threadIdx.x; i < nb; i += THREADS) {
                a.ufParent[i] = i;
                a.ufFlag[i] = 1u;
            }
            return;
        }
        for (uint32_t i = threadIdx.x; i < nb; i += THREADS) {
            w.bvel[i] = vel[i];
            w.bpos[i] = pos[i];
        }
        const uint32_t colors = min(__ldcg(&a.counters->colors), MAX_COLORS);
        for (uint32_t c = threadIdx.x; c <= colors; c += THREADS) a.s.colorStart[c] = colorStart[c];
        __syncthreads();
    }
    for (uint32_t i = threadIdx.x; i < nb; i += THREADS) par[i] = i;
    __syncthreads();
    for (uint32_t j = threadIdx.x; j < n; j += THREADS) {
        const uint2 q = a.s.pairBodies[j];
        const uint32_t x = q.x & PAIR_BODY, y = q.y & PAIR_BODY;
        if (w.bstate[x] == STATE_DYNAMIC && w.bstate[y] == STATE_DYNAMIC) team_union(par, x, y);
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < nb; i += THREADS) {
        a.ufParent[i] = team_find(par, i);
        a.ufFlag[i] = 1u;
    }
}

cudaError_t block_solver_init()
{
    const int bytes = int(team_smem_bytes(BLOCK_SOLVE_BODIES, 0));
    for (const void* k : {reinterpret_cast<const void*>(k_color_solve_block<128>),
                          reinterpret_cast<const void*>(k_color_solve_block<512>),
                          reinterpret_cast<const void*>(k_color_solve_block<1024>)}) {
        const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_color_solve_block(uint32_t perColor, cudaStream_t stream, const BlockSolve& a)
{
    const size_t smem = team_smem_bytes(a.bodyCap, 0);
    // The threads that a colour's steps use, for each one more is slower at the barriers: 122 manifolds in 7 colours take
    // 48 us with 128 threads and 51 with 512, 157 in 5: 52 and 49; 554 in 7: 63 with 512 and 66 with 1,024, 2,086 in 36:
    // 385 and 410, 1,042 in 7: 93 and 91, 3,301 in 9: 202 and 187.
    if (perColor <= 24) return chain_launch(true, k_color_solve_block<128>, 1, 128, smem, stream, a);
    if (perColor <= 128) return chain_launch(true, k_color_solve_block<512>, 1, 512, smem, stream, a);
    return chain_launch(true, k_color_solve_block<1024>, 1, 1024, smem, stream, a);
}

// Batched worlds: each CTA takes the next team of consecutive worlds, whose manifolds are one contiguous range of
// the world-grouped list, and colours + solves that range as one problem (the worlds share no body, so their
// colour classes simply merge). Priorities are world-local indices: every world gets the colouring, hence the
// solving order, it has when stepped on its own, whichever team it is in. A team whose bodies fit the dynamic
// shared memory (bodyCap bodies) keeps their velocities, poses and colouring words there. The solver is bound by
// load latency and barriers, so what counts is how many teams an SM holds at once: the colouring words share the
// body cache when the records stay in global memory (32 B of shared memory a body), and the unpipelined variant is
// held to 64 registers a thread (1024 threads an SM).
template <uint32_t THREADS, bool PIPELINED>
__global__ void __launch_bounds__(THREADS, PIPELINED ? 1 : 1024 / THREADS) k_color_solve_teams(TeamLaunch a)
{
    chain_begin();
    // [bodyCap] velocities, [bodyCap] poses, then 2 x [bodyCap] u64 colouring words, overwritten after colouring by
    // the constraint records (team_smem_bytes).
    extern __shared__ float4 teamCache[];
    __shared__ uint32_t colorCount[COLOR_SLOTS];
    __shared__ uint32_t colorStart[MAX_COLORS + 1];
    __shared__ uint32_t item;
    const DeviceWorld& w = a.w;
    Manifold* m = a.m;
    uint32_t* prio = const_cast<uint32_t*>(a.s.prio);
    while (true) {
        if (threadIdx.x == 0) item = atomicAdd(a.nextTeam, 1u);
        __syncthreads();
        const uint32_t k = item;
        __syncthreads();
        if (k >= a.teams) return;
        const uint32_t t = a.teamOrder[k];
        const uint32_t w0 = a.teamWorld[t], w1 = a.teamWorld[t + 1];
        const uint32_t lo = a.manSeg[w0], hi = a.manSeg[w1];
        if (hi <= lo) continue;
        for (uint32_t i = lo + threadIdx.x; i < hi; i += THREADS)
            prio[i] = priority_hash(i - a.manSeg[w.bodyWorld[w.cbody[m[i].a]]]);
        const SolveScratch ls{a.s.color + lo, a.s.order + lo, a.s.bodyMax, a.s.bodyMask, colorCount, colorStart,
                              a.s.cons.from(lo), prio + lo, a.s.listA + lo, a.s.listB + lo, a.s.pairBodies + lo,
                              a.s.hint ? a.s.hint + lo : nullptr};
        const uint32_t b0 = w.worldBodyStart[w0], nb = w.worldBodyStart[w1] - b0;
        if (nb <= a.bodyCap) {
            float4* vel = teamCache;
            float4* pos = teamCache + a.bodyCap;
            // No records on chip: the colouring words sit where the body cache goes and the bodies are loaded after
            // colouring (SharedBodies, lazy). Otherwise the bodies are loaded now and the words follow them.
            const bool lazy = a.consCap == 0;
            auto* maxW = reinterpret_cast<unsigned long long*>(lazy ? teamCache : teamCache + 2 * a.bodyCap);
            unsigned long long* maskW = maxW + a.bodyCap;
            for (uint32_t i = threadIdx.x; i < nb; i += THREADS) {
                if (!lazy) {
                    vel[i] = w.bvel[b0 + i];
                    pos[i] = w.bpos[b0 + i];
                }
                maxW[i] = 0ull;
                maskW[i] = 0ull;
            }
            __syncthreads();
            ConsSmem cs;
            cs.q = teamCache + 2 * a.bodyCap;
            cs.cap = a.consCap;
            cs.base = b0;
            SharedBodies sb{vel, pos, maxW, maskW, b0};
            if (lazy) { sb.count = nb; sb.gvel = w.bvel; sb.gpos = w.bpos; }
            const bool solved = color_and_solve<BlockSync, SharedBodies, PIPELINED>(
                w, sb, m + lo, hi - lo, ls, a.velIters, a.posIters, threadIdx.x, THREADS, BlockSync{},
                &a.counters->colors, &a.counters->status, cs);
            __syncthreads();
            // A team that gave up (its status bit is set and the step is redone or fails) leaves the bodies alone:
            // a lazy cache may still hold colouring words.
            if (solved) {
                for (uint32_t i = threadIdx.x; i < nb; i += THREADS) {
                    w.bvel[b0 + i] = vel[i];
                    w.bpos[b0 + i] = pos[i];
                }
            }
            if (solved && a.ufParent) {
                // The team's islands, in the shared memory the body cache used: links between two dynamic bodies.
                __syncthreads();
                uint32_t* par = reinterpret_cast<uint32_t*>(teamCache);
                for (uint32_t i = threadIdx.x; i < nb; i += THREADS) par[i] = i;
                __syncthreads();
                const uint2* pb = a.s.pairBodies + lo;
                for (uint32_t j = threadIdx.x; j < hi - lo; j += THREADS) {
                    const uint2 q = pb[j];
                    if ((q.x & PAIR_DYNAMIC) && (q.y & PAIR_DYNAMIC))
                        team_union(par, (q.x & PAIR_BODY) - b0, (q.y & PAIR_BODY) - b0);
                }
                __syncthreads();
                for (uint32_t i = threadIdx.x; i < nb; i += THREADS) a.ufParent[b0 + i] = b0 + team_find(par, i);
            }
        } else {
            __syncthreads();
            const bool solved = color_and_solve<BlockSync, GlobalBodies, PIPELINED>(
                w, GlobalBodies{w.bvel, w.bpos, a.s.bodyMax, a.s.bodyMask}, m + lo, hi - lo, ls, a.velIters,
                a.posIters, threadIdx.x, THREADS, BlockSync{}, &a.counters->colors, &a.counters->status);
            if (solved && a.ufParent) {
                __syncthreads();
                const uint2* pb = a.s.pairBodies + lo;
                for (uint32_t j = threadIdx.x; j < hi - lo; j += THREADS) {
                    const uint2 q = pb[j];
                    if ((q.x & PAIR_DYNAMIC) && (q.y & PAIR_DYNAMIC))
                        team_union(a.ufParent, q.x & PAIR_BODY, q.y & PAIR_BODY);
                }
            }
        }
        __syncthreads();
    }
}

template <uint32_t THREADS, bool PIPELINED>
static cudaError_t team_occupancy(uint32_t bodyCap, uint32_t consCap, int* out)
{
    cudaError_t e = cudaFuncSetAttribute(k_color_solve_teams<THREADS, PIPELINED>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, int(TEAM_SMEM_MAX));
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(out, k_color_solve_teams<THREADS, PIPELINED>, THREADS,
                                                         team_smem_bytes(bodyCap, consCap));
}

cudaError_t team_solver_blocks_per_sm(uint32_t threads, bool pipelined, uint32_t bodyCap, uint32_t consCap, int* out)
{
    switch (threads) {
    case 64: return pipelined ? team_occupancy<64, true>(bodyCap, consCap, out) : team_occupancy<64, false>(bodyCap, consCap, out);
    case 128: return pipelined ? team_occupancy<128, true>(bodyCap, consCap, out) : team_occupancy<128, false>(bodyCap, consCap, out);
    case 256: return pipelined ? team_occupancy<256, true>(bodyCap, consCap, out) : team_occupancy<256, false>(bodyCap, consCap, out);
    case 512: return pipelined ? team_occupancy<512, true>(bodyCap, consCap, out) : team_occupancy<512, false>(bodyCap, consCap, out);
    default: return cudaErrorInvalidValue;
    }
}

template <uint32_t THREADS>
static cudaError_t launch_teams(bool chained, bool pipelined, uint32_t grid, size_t smem, cudaStream_t stream,
                                const TeamLaunch& a)
{
    return chain_launch(chained, pipelined ? k_color_solve_teams<THREADS, true> : k_color_solve_teams<THREADS, false>,
                        grid, THREADS, smem, stream, a);
}

cudaError_t launch_color_solve_teams(bool chained, uint32_t threads, bool pipelined, uint32_t grid, cudaStream_t stream,
                                     const TeamLaunch& a)
{
    const size_t smem = team_smem_bytes(a.bodyCap, a.consCap);
    if (smem > TEAM_SMEM_MAX) return cudaErrorInvalidValue;
    switch (threads) {
    case 64: return launch_teams<64>(chained, pipelined, grid, smem, stream, a);
    case 128: return launch_teams<128>(chained, pipelined, grid, smem, stream, a);
    case 256: return launch_teams<256>(chained, pipelined, grid, smem, stream, a);
    case 512: return launch_teams<512>(chained, pipelined, grid, smem, stream, a);
    default: return cudaErrorInvalidValue;
    }
}

// ---------------------------------------------------------------------------------------------------------------
// Islands and sleep (IslandManager.cpp:7-116, ObjectManager::updateSleeping ObjectManager.cpp:1438-1491).
// Union-find over manifolds whose bodies are both dynamic, linking the larger root under the smaller (the root is
// the island's smallest body index: a deterministic island id). A body is quiet when |v| + |w| * boundRadius is at
// most the speed threshold; its timer accumulates while quiet. An island sleeps when every member is quiet and has
// been for the time threshold.
// ---------------------------------------------------------------------------------------------------------------
__global__ void k_island_init(DeviceWorld w, uint32_t* __restrict__ parent, uint32_t* __restrict__ flag)
{
    for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b < w.nBodies; b += gridDim.x * blockDim.x) {
        parent[b] = b;
        flag[b] = 1u;
    }
}

__global__ void k_island_union(DeviceWorld w, const Manifold* __restrict__ m, const uint32_t* __restrict__ nM,
                               uint32_t* __restrict__ parent)
{
    const uint32_t n = *nM;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uf_link(w, parent, w.cbody[m[i].a], w.cbody[m[i].b]);
    }
}

// The active body constraints' links (Simulation.cpp:338-341: islandManager.step over each system's active edges).
__global__ void k_island_union_edges(DeviceWorld w, const uint2* __restrict__ edges, uint32_t n,
                                     uint32_t* __restrict__ parent)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uf_link(w, parent, edges[i].x, edges[i].y);
    }
}

__global__ void k_island_quiet(DeviceWorld w, uint32_t* parent, uint32_t* flag, float dt,
                               float speedThreshold, float timeThreshold)
{
    chain_begin();
    for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b < w.nBodies; b += gridDim.x * blockDim.x) {
        if (w.bstate[b] != STATE_DYNAMIC) continue;
        const float4 v = w.bvel[b];
        const float speed = sqrtf(v.x * v.x + v.y * v.y) + fabsf(v.z) * w.boundRadius[b];
        const bool quiet = speed <= speedThreshold;
        const float timer = (w.sleepTimer[b] + dt) * float(quiet);
        w.sleepTimer[b] = timer;
        if (!(quiet && timer >= timeThreshold)) atomicAnd(flag + uf_find(parent, b), 0u);
    }
}

// Last thing of a step: see StepEnd. Called by every thread of the launch's blocks, after their own work.
__device__ __forceinline__ void step_end(const StepEnd& e, StepCounters* counters)
{
    if (!e.host) return;
    __shared__ bool last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(e.done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    constexpr uint32_t WORDS = sizeof(StepCounters) / sizeof(uint32_t);
    if (threadIdx.x < WORDS)
        reinterpret_cast<volatile uint32_t*>(e.host)[threadIdx.x] =
            __ldcg(reinterpret_cast<const uint32_t*>(counters) + threadIdx.x);
    if (threadIdx.x == 0 && __ldcg(&counters->status) == 0u) *e.nPrev = __ldcg(e.nManifolds);
    __threadfence_system();
}

__global__ void k_island_sleep(DeviceWorld w, uint32_t* parent, const uint32_t* flag,
                               StepCounters* counters, StepEnd end)
{
    chain_begin();
    uint32_t slept = 0;
    for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b < w.nBodies; b += gridDim.x * blockDim.x) {
        if (w.bstate[b] != STATE_DYNAMIC) continue;
        const uint32_t root = uf_find(parent, b);
        if (__ldcg(flag + root)) {
            w.bstate[b] = STATE_SLEEPING;
            w.sleepIsland[b] = root;
            w.sleepTimer[b] = 0.0f;
            if (w.worldDirty) w.worldDirty[w.bodyWorld[b]] = 1u;
            slept++;
        }
    }
    for (int o = 16; o > 0; o >>= 1) slept += __shfl_xor_sync(0xffffffffu, slept, o);
    if ((threadIdx.x & 31) == 0 && slept) {
        atomicAdd(&counters->slept, slept);
        counters->topoDirty = 1u;
    }
    step_end(end, counters);
}

// Work-list flags from body states: dynamic bodies, dynamic colliders, static + sleeping colliders.
__global__ void k_state_flags(const uint8_t* __restrict__ bstate, const uint32_t* __restrict__ cbody,
                              uint32_t nBodies, uint32_t nColliders, uint32_t* __restrict__ bodyDyn,
                              uint32_t* __restrict__ colDyn, uint32_t* __restrict__ colOther,
                              uint32_t* __restrict__ sleeping)
{
    const uint32_t stride = gridDim.x * blockDim.x;
    bool any = false;
    for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b < nBodies; b += stride) {
        bodyDyn[b] = bstate[b] == STATE_DYNAMIC;
        any |= bstate[b] == STATE_SLEEPING;
    }
    if (any) *sleeping = 1u;
    for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < nColliders; c += stride) {
        const uint8_t st = bstate[cbody[c]];
        colDyn[c] = st == STATE_DYNAMIC;
        colOther[c] = st == STATE_STATIC || st == STATE_SLEEPING;   // destroyed bodies' colliders: neither
    }
}

// Signed distance from a query circle's centre to one collider, as NarrowPhaseCollisionDetector::
// findCollisionsInCircle (NarrowPhaseCollisionDetector.cpp:153-270) computes it: circle - centre distance minus the
// radius; box - the exact box distance field in the box frame; polygon - distance to the support edge's closest
// point (findSupportEdge / closestPointOnSegment, HelperMethods.h:73-109), or the (negative) separation inside.
// False where the reference skips the collider or the distance is not below the query radius.
__device__ __forceinline__ bool circle_contact(const ColliderView& B, V2 pos, float radius, float& sdf)
{
    if (B.type == SHAPE_CIRCLE) {
        const V2 delta = B.pos - pos;
        const float distSq = dot(delta, delta);
        const float radiusSum = B.r + radius;
        if (radiusSum <= 0.0f || distSq >= radiusSum * radiusSum) return false;
        sdf = sqrtf(distSq) - B.r;
    } else {
        const V2 right = V2{B.c, B.s}, up = V2{-B.s, B.c};
        const V2 d = pos - B.pos;
        const V2 loc = V2{dot(d, right), dot(d, up)};
        if (B.type == SHAPE_CAPSULE) {
            // Closest point of the core to the query centre (NarrowPhaseCollisionDetector.cpp:245-262).
            const V2 axis = V2{B.c, B.s};
            const float t = clamp_value(dot(d, axis), -B.hw, B.hw);
            const V2 delta = d - axis * t;
            const float distSquared = dot(delta, delta);
            const float radiusSum = B.r + radius;
            if (radiusSum <= 0.0f || distSquared >= radiusSum * radiusSum) return false;
            sdf = sqrtf(distSquared) - B.r;
        } else if (B.type == SHAPE_BOX) {
            const float dx = fabsf(loc.x) - B.hw, dy = fabsf(loc.y) - B.hh;
            const float maxD = rfmaxf(dx, dy);
            if (maxD > 0.0f && maxD >= radius) return false;
            const float ex = rfmaxf(0.0f, dx), ey = rfmaxf(0.0f, dy);
            const float outside = sqrtf(ex * ex + ey * ey);
            const float inside = rfminf(0.0f, maxD);
            sdf = inside + outside;
        } else {
            float maxSep = -FLT_MAX;
            uint32_t edge = 0;
            for (uint32_t i = 0; i < B.nv; i++) {
                const float sep = dot(ld2(B.normals, i), loc - ld2(B.verts, i));
                if (sep > radius) return false;
                if (sep > maxSep) { maxSep = sep; edge = i; }
            }
            if (maxSep >= ZERO_DIVISION_BOUNDARY) {
                const V2 a = ld2(B.verts, edge), b = ld2(B.verts, next_index(edge, B.nv));
                const V2 ab = b - a;
                const float denom = dot(ab, ab);
                V2 q = a;
                if (denom >= ZERO_DIVISION_BOUNDARY_SQUARED) {
                    const float t = dot(loc - a, ab) / denom;
                    q = a + ab * rfminf(rfmaxf(t, 0.0f), 1.0f);
                }
                const V2 e = loc - q;
                sdf = sqrtf(dot(e, e));
            } else {
                sdf = maxSep;
            }
        }
    }
    return sdf < radius;
}

// ---------------------------------------------------------------------------------------------------------------
// Spatial query (BroadPhaseCollisionDetector::queryCollidersInShape, BroadPhaseCollisionDetector.h:189-203;
// BvhTree::queryCollidersInShape, BvhTree.h:110-192): a collider is found when its body's tree (dynamic, static
// or sleeping) is selected and its AABB passes the query shape's leaf test (QueryShapes.h): strict overlap for an
// AABB (AABBQuery::simdOverlap), closest-point squared distance within the squared radius for a circle
// (CircleQuery::simdOverlap, radius clamped at 0). With 'contacts' the circle query's colliders that the circle itself
// touches (circle_contact, the radius as given), with their signed distances.
// Test and compaction in one launch: blocks take tiles of blockDim.x colliders in ticket order, count their hits and
// place them after the preceding tiles' by decoupled look-back, so the indices come out ascending. The first hostCap
// results go straight to page-locked memory with the count. The states of the next query's tiles are cleared here.
// Bound: 24 bytes a collider read; a query of a few thousand colliders is the launch and the wait for it. As a flag
// pass, a scan with its clear, a scatter and two copies back it took 47 us on 20,000 colliders.
// ---------------------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(QUERY_SELECT_THREADS) k_query_select(DeviceWorld w, QuerySelect q)
{
    __shared__ uint32_t warpBase[QUERY_SELECT_THREADS / 32];
    __shared__ uint32_t tileSlot, tileBase;
    const uint32_t n = w.nColliders, tiles = (n + QUERY_SELECT_THREADS - 1) / QUERY_SELECT_THREADS;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t* const ticket = q.tileState + tiles;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i <= tiles; i += gridDim.x * blockDim.x) q.nextState[i] = 0u;
    const float r = rfmaxf(0.0f, q.shape.z);
    const float rr = r * r;
    while (true) {
        if (threadIdx.x == 0) tileSlot = atomicAdd(ticket, 1u);
        __syncthreads();
        const uint32_t tile = tileSlot;
        if (tile >= tiles) return;
        const uint32_t c = tile * QUERY_SELECT_THREADS + threadIdx.x;
        bool hit = false;
        float sdf = 0.0f;
        if (c < n) {
            const uint8_t st = w.bstate[w.cbody[c]];
            const uint32_t tree = st == STATE_DYNAMIC ? 1u : (st == STATE_STATIC ? 2u : (st == STATE_SLEEPING ? 4u : 0u));
            if (q.trees & tree) {
                const float4 b = w.caabb[c];
                if (q.kind == QUERY_SELECT_AABB) {
                    hit = b.x < q.shape.z && b.z > q.shape.x && b.y < q.shape.w && b.w > q.shape.y;
                } else {
                    const float dx = rfmaxf(b.x - q.shape.x, rfmaxf(0.0f, q.shape.x - b.z));
                    const float dy = rfmaxf(b.y - q.shape.y, rfmaxf(0.0f, q.shape.y - b.w));
                    hit = (dx * dx + dy * dy) <= rr;
                    if (hit && q.kind == QUERY_SELECT_CONTACTS)
                        hit = circle_contact(collider_view(w, c), V2{q.shape.x, q.shape.y}, q.shape.z, sdf);
                }
            }
        }
        const uint32_t hits = __ballot_sync(0xffffffffu, hit);
        if (lane == 0) warpBase[warp] = __popc(hits);
        __syncthreads();
        if (warp == 0) {
            const uint32_t count = lane < QUERY_SELECT_THREADS / 32 ? warpBase[lane] : 0u;
            uint32_t incl = count;
            for (uint32_t o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            const uint32_t aggregate = __shfl_sync(0xffffffffu, incl, 31);
            if (lane < QUERY_SELECT_THREADS / 32) warpBase[lane] = incl - count;
            volatile uint32_t* state = q.tileState;
            uint32_t prefix = 0;
            if (tile > 0) {
                if (lane == 0) state[tile] = (1u << 30) | aggregate;
                prefix = scan_lookback(tile, q.tileState, q.status);
            }
            if (lane == 0) {
                state[tile] = (2u << 30) | (prefix + aggregate);
                tileBase = prefix;
                if (tile == tiles - 1) {
                    q.host[0] = prefix + aggregate;
                    q.host[1] = *static_cast<volatile uint32_t*>(q.status) & STATUS_LOOKBACK_TIMEOUT;
                }
            }
        }
        __syncthreads();
        if (hit) {
            const uint32_t o = tileBase + warpBase[warp] + __popc(hits & ((1u << lane) - 1u));
            q.list[o] = c;
            if (q.kind == QUERY_SELECT_CONTACTS) q.dist[o] = sdf;
            if (o < q.hostCap) {
                q.host[2 + o] = c;
                if (q.kind == QUERY_SELECT_CONTACTS) q.host[2 + q.hostCap + o] = __float_as_uint(sdf);
            }
        }
        __syncthreads();   // tileSlot, tileBase and warpBase are reused by the next tile
    }
}

__global__ void k_scatter_list(const uint32_t* __restrict__ flag, const uint32_t* __restrict__ offset, uint32_t n,
                               uint32_t* __restrict__ list)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        if (flag[i]) list[offset[i]] = i;
}

}  // namespace ag2d
