// Kernel declarations and launch constants for the collision/contact pipeline.
#pragma once

#include "ag2d_math.cuh"
#include "ag2d_world.cuh"

namespace ag2d {

constexpr uint32_t SORT_THREADS = 256;
// Keys a thread of the sort: few while that leaves an SM at most a few tiles, many above (fewer tiles to look back over).
constexpr uint32_t SORT_ITEMS_SMALL = 4, SORT_ITEMS_LARGE = 16;
constexpr uint32_t SORT_SMALL_MAX = 300000;
constexpr uint32_t SCAN_THREADS = 256;
constexpr uint32_t SCAN_ITEMS = 8;
constexpr uint32_t SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;
constexpr int QUERY_STACK = 64;
constexpr uint32_t QUERY_STASH = 16;   // pair partners a query keeps from its counting traversal
constexpr uint32_t MAX_COLORS = 256;
constexpr uint32_t NO_COLOR = 0xFFFFFFFFu;

// Traversal record of an internal node: both children's AABBs, their child codes (internal node index, or ~leaf)
// and the last leaf of each child's range, so that a traversal step is one 48-byte load.
struct alignas(16) NodeRec {
    float4 box[2];
    int2 child;
    int2 last;
};
static_assert(sizeof(NodeRec) == 48, "NodeRec is 48 bytes");

// Warm start: the previous step's manifolds in an open-addressing table keyed by the unordered collider pair, those
// with a non-zero impulse on an active contact flagged (bit 31 of the value: the reference caches only these,
// rebuildContactCache, NarrowPhaseCollisionDetector.cpp:272-297; makePairKey .h:216-219); each new manifold of the
// same ordered pair takes the flagged manifold's impulses of the contacts with equal ids (finalizeResults,
// :749-766). Every new manifold whose pair was there also takes that manifold's colour as its colouring hint.
// One region of the table per world of a batch, [2 seg[w], 2 seg[w + 1]) for the world's seg[w + 1] - seg[w] previous
// manifolds (seg: the previous list's world starts), so a probe stays in its world's few kilobytes and hits in cache;
// a single world (seg null) uses the whole power-of-two table. Which region holds a pair changes nothing but where
// it is found.
constexpr uint32_t WARM_CACHED = 0x80000000u;   // the manifold had a non-zero impulse
struct WarmTable {
    unsigned long long* keys;   // all ones: empty; null: no warm start
    uint32_t* vals;
    uint32_t capacity;
    const uint32_t* seg;
    const uint32_t* colWorld;
    const Manifold* prev;
    const uint32_t* nPrev;
    const uint32_t* prevColor;   // or null
    uint32_t* hint;              // colouring hints of the new manifolds out, or null
    uint32_t* status;
};

// Read-only view of one LBVH over n leaves in sorted order. A single tree has n - 1 internal nodes and root 0; a
// world-segmented tree (sortedWorld non-null) holds one tree per world segment [segStart[w], segStart[w + 1]),
// rooted at internal node segStart[w].
struct TreeView {
    int n;
    const int2* child;
    const float4* nodeAabb;
    const float4* leafAabb;       // AABBs in sorted (leaf) order
    const uint32_t* vals;         // collider index of each leaf
    const uint32_t* sortedWorld;  // world of each leaf, or null (one world)
    const uint32_t* segStart;     // [worlds + 1] segment starts, or null (one world)
    const NodeRec* rec;           // traversal records of the internal nodes
};

// Spatial kernels (k_spatial.cu).
struct IntegrateParams {
    float dt, gx, gy;
    float dampHalf;   // damping^(dt/2), or >= 1 when damping is off
};
__global__ void k_integrate(DeviceWorld w, const uint32_t* dynBody, const uint8_t* dynSimd, uint32_t nDyn,
                            IntegrateParams ip, uint32_t phase);
// A 16-byte aligned buffer to fill with a value, or (iota) with its indices.
struct FillRegion {
    uint32_t* p;
    uint32_t words, value, iota;
};
constexpr uint32_t MAX_FILLS = 12;
struct StepBegin {
    DeviceWorld w;
    float4 *snapVel, *snapPos;
    float2* snapRot;
    float *snapWrap, *snapTimer;
    uint8_t* snapState;
    uint32_t* snapIsland;
    const uint32_t* dynBody;   // the dynamic bodies
    const uint8_t* dynSimd;
    uint32_t nDyn;
    uint32_t both;             // both halves of the integration, else the first
    IntegrateParams ip;
    float4* copyDst;           // collider poses to save (or bring back) for continuous collision
    const float4* copySrc;
    uint32_t copyCount;
    uint32_t fills;
    FillRegion fill[MAX_FILLS];
    const uint32_t* nIsle;
    StepCounters* counters;
};
// A chain of kernels on one stream: launched with chain_launch, a kernel's blocks may be placed while its predecessor
// still runs, and chain_begin, the first thing they do, waits for its end (and for its writes). Kernels of a small step
// run about ten microseconds and the gaps between them up to a third of that. Unchained against chained, a step of 64
// bodies 98 and 90 us; of n bodies in flight: 5,000: 112 and 105, 20,000: 130 and 110, 40,000: 134 and 114, 80,000: 148 and
// 132; of n still falling into a pile: 20,000: 236 and 215, 80,000: 277 and 256; a detection pass over n: 20,000: 115 and
// 112, 60,000: 131 and 127. Large kernels lose more to the waiting blocks than the gaps cost: a pass over 80,000: 138 and 145,
// over a million: 465 and 489, a step of 100,000 bodies piled up: 900 and 937. Engines of up to CHAIN_COLLIDERS are
// chained, half of the 60,000 up to which nothing measured loses.
// Such a kernel takes no pointer as __restrict__ and reads nothing through __ldg that an earlier kernel of the chain
// writes: those loads may move ahead of the wait and need not see the writes.
constexpr uint32_t CHAIN_COLLIDERS = 32768;
__device__ __forceinline__ void chain_begin()
{
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
template <class... P, class... A>
inline cudaError_t chain_launch(bool chained, void (*kernel)(P...), uint32_t blocks, uint32_t threads, size_t smem,
                                cudaStream_t stream, A... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = chained ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
__global__ void k_step_begin(StepBegin a);
__global__ void k_collider_pose(DeviceWorld w, const uint32_t* list, const uint8_t* listSimd, uint32_t n,
                                const uint32_t* worldMask, WarmTable insert);
__global__ void k_bounds_init(uint32_t* bounds, uint32_t worlds);
__global__ void k_bounds(const float4* aabb, const uint32_t* list, uint32_t n, const uint32_t* colWorld,
                         uint32_t* bounds, float4* parts, uint32_t* clear, uint32_t clearWords);
__global__ void k_count_world(const uint32_t* list, uint32_t n, const uint32_t* elemWorld, uint32_t* counts);
__global__ void k_simd_flags(const uint32_t* list, uint32_t n, const uint32_t* offsets, uint32_t nElems,
                             const uint32_t* elemWorld, const uint32_t* worldStart, uint32_t worlds, uint8_t* simd);
__global__ void k_morton(const float4* aabb, const uint32_t* list, uint32_t n, const uint32_t* colWorld,
                         const uint32_t* bounds, const float4* parts, uint32_t nParts, uint32_t* keys, uint32_t* vals,
                         uint32_t* keyOf, uint32_t* hist, uint32_t* done);
__global__ void k_world_keys(const uint32_t* vals, uint32_t n, const uint32_t* colWorld, uint32_t* keys, uint32_t* hist,
                             uint32_t* done);
__global__ void k_seg_starts(const uint32_t* offsets, const uint32_t* worldStart, uint32_t worlds, uint32_t nElems,
                             const uint32_t* total, uint32_t* segStart);
__global__ void k_manifold_segments(const Manifold* m, const uint32_t* nM, const uint32_t* cbody,
                                    const uint32_t* bodyWorld, uint32_t worlds, uint32_t* segStart);
__global__ void k_tree_gather(const uint32_t* vals, uint32_t n, const uint32_t* keyOf, const uint32_t* colWorld,
                              const float4* caabb, uint32_t* sortedKey, uint32_t* sortedWorld, float4* leafAabb);
// Host side: tiles of a sort pass over n keys, and one pass. digitBase: the digits' exclusive scan; tileState [tiles x
// 256] and tileCounter zeroed before the launch.
uint32_t sort_tiles(uint32_t n);
cudaError_t launch_sort_pass(const uint32_t* keysIn, const uint32_t* valsIn, uint32_t* keysOut, uint32_t* valsOut,
                             uint32_t n, uint32_t shift, const uint32_t* digitBase, uint32_t* tileState,
                             uint32_t* tileCounter, uint32_t* status, bool chained, cudaStream_t stream);
// Trees of up to TREE_SEGMENT_MAX leaves are built by one CTA each (k_tree_segments), in size classes.
constexpr uint32_t TREE_SEGMENT_MAX = 16384;
// A single tree of more leaves is built by the whole GPU in eight launches: 75 us at 6,000 and 77 at 8,000 leaves,
// where one CTA takes 85 and 113 (57 at 4,000).
constexpr uint32_t TREE_SINGLE_MAX = 5120;
struct TreeBuild {
    const float4* caabb;
    const uint32_t* list;       // colliders, world-grouped
    const uint32_t* segStart;   // [worlds + 1], or null: one segment of n
    uint32_t worlds, n;
    uint32_t *vals, *keys;      // sorted colliders and their Morton keys
    uint32_t* sortedWorld;      // or null
    float4* leafAabb;
    float4* nodeAabb;           // or null: the boxes in the records are enough for the pair query
    int2* child;                // or null, likewise
    NodeRec* rec;
    float4* meet;               // [2 x leaves] meeting boxes of the largest class
    bool chained;               // one class: launched ahead of its predecessor's end (chain_launch)
};
// Host side: builds every segment's tree; 'largest' bounds the segment sizes (at most TREE_SEGMENT_MAX); *launches: the
// kernels launched.
cudaError_t launch_tree_segments(const TreeBuild& t, uint32_t largest, uint32_t sms, cudaStream_t stream,
                                 uint32_t* launches);
// Host side: raises the builders' dynamic shared-memory limit (once per device).
cudaError_t tree_segments_init();
__global__ void k_lbvh_build(const uint32_t* keys, const uint32_t* sortedWorld, const uint32_t* segStart, int n,
                             const uint32_t* vals, const float4* caabb, float4* leafAabb, int2* child, int* parent, int* leafParent, float4* meet, NodeRec* rec);
__global__ void k_lbvh_refit(int n, const int2* child, const int* parent, const int* leafParent,
                             const float4* leafAabb, float4* nodeAabb, float4* meet, NodeRec* rec);
// Empty marker of a refit meeting slot (min x bits): a NaN no arithmetic produces.
constexpr uint32_t MEET_EMPTY = 0xFFFFFFFFu;
// Pair query: every candidate pair of the dynamic colliders, in query-rank order, into pairs; *total = the count.
// tileState [tiles + 1] and tileCounter zeroed before the launch (tiles: blockDim.x queries each).
constexpr uint32_t QUERY_MAX_THREADS = 256;
__global__ void k_query(TreeView dyn, TreeView other, const uint32_t* cbody, uint2* pairs, uint32_t pairCap,
                        uint32_t* total, uint32_t* status, uint32_t* tileState, uint32_t* tileCounter);
__global__ void k_ccd_sweep(DeviceWorld w, const uint32_t* dynCol, uint32_t n, TreeView other, const float4* prevPos,
                            const float4* prevPose, const float* minExtent, uint32_t* hitTime, uint32_t* status);
__global__ void k_ccd_shift_colliders(DeviceWorld w, const uint32_t* dynCol, uint32_t n, const float4* prevPos,
                                      const uint32_t* hitTime);
__global__ void k_ccd_shift_bodies(DeviceWorld w, const uint32_t* dynBody, uint32_t n, const float4* prevPos,
                                   uint32_t* hitTime, StepCounters* counters);
// Decoupled look-back over tiles taken in ticket order: tile t publishes flag << 30 | value in tileState[t] (flag 1:
// its aggregate, 2: its inclusive prefix) and sums its predecessors' values, read by the calling warp 32 at a time,
// nearest first, up to the nearest inclusive prefix. A tile only waits on tiles with smaller tickets, all held by
// running blocks, so the waits end; each is still bounded by SPIN_LIMIT (then STATUS_LOOKBACK_TIMEOUT is set and the
// partial sum returned). Called by one full warp; returns the exclusive prefix of tile 'tile' (> 0).
__device__ __forceinline__ uint32_t scan_lookback(uint32_t tile, uint32_t* tileState, uint32_t* status)
{
    const uint32_t lane = threadIdx.x & 31;
    volatile uint32_t* state = tileState;
    uint32_t prefix = 0, spins = 0;
    int32_t t = int32_t(tile) - 1;
    while (t >= 0) {
        const int32_t idx = t - int32_t(lane);
        const uint32_t sv = idx >= 0 ? state[idx] : (2u << 30);
        const uint32_t flag = sv >> 30;
        const uint32_t inc = __ballot_sync(0xffffffffu, flag == 2u);
        const uint32_t window = inc ? (((inc & (0u - inc)) << 1) - 1u) : 0xffffffffu;   // lanes up to the nearest
        if (__ballot_sync(0xffffffffu, flag == 0u) & window) {                             // inclusive prefix
            if (++spins > SPIN_LIMIT) {
                if (lane == 0) atomicOr(status, STATUS_LOOKBACK_TIMEOUT);
                break;
            }
            continue;
        }
        uint32_t v = ((window >> lane) & 1u) ? (sv & 0x3FFFFFFFu) : 0u;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        prefix += v;
        if (inc) break;
        t -= 32;
    }
    return prefix;
}

// Contact-cache key of an unordered collider pair, and the region of the table that holds it.
__device__ __forceinline__ unsigned long long pair_key(uint32_t a, uint32_t b)
{
    const uint32_t lo = a < b ? a : b, hi = a < b ? b : a;
    return (static_cast<unsigned long long>(lo) << 32) | hi;
}
struct WarmRegion {
    uint32_t base, size;   // size 0: the world had no manifolds
    __device__ __forceinline__ uint32_t home(unsigned long long key) const
    {
        return base + uint32_t(((key * 0x9E3779B97F4A7C15ull) >> 32) % size);
    }
    __device__ __forceinline__ uint32_t next(uint32_t s) const { return s + 1 == base + size ? base : s + 1; }
};
__device__ __forceinline__ WarmRegion warm_region(const WarmTable& t, uint32_t a)
{
    if (!t.seg) return WarmRegion{0u, t.capacity};
    const uint32_t wd = t.colWorld[a];
    const uint32_t lo = t.seg[wd], hi = t.seg[wd + 1];
    if (hi < lo || 2ull * hi > t.capacity) return WarmRegion{0u, 0u};   // not a valid segmentation: no region
    return WarmRegion{2u * lo, 2u * (hi - lo)};
}
// Puts the previous manifolds into the (empty) table, grid-stride over all threads of the launch.
__device__ __forceinline__ void warm_insert(const WarmTable& t)
{
    const uint32_t n = *t.nPrev;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint2 pair = *reinterpret_cast<const uint2*>(&t.prev[i].a);
        const uint32_t count = t.prev[i].count;
        const float4 j = *reinterpret_cast<const float4*>(&t.prev[i].jn0);
        uint32_t mask = uint32_t(j.x != 0.0f) | uint32_t(j.y != 0.0f) << 1 | uint32_t(j.z != 0.0f) << 2 |
                        uint32_t(j.w != 0.0f) << 3;
        mask &= (1u << (2u * count)) - 1u;
        const unsigned long long key = pair_key(pair.x, pair.y);
        const WarmRegion r = warm_region(t, pair.x);
        if (r.size == 0) { atomicOr(t.status, STATUS_HASH_FULL); continue; }   // cannot happen: m is in its world
        uint32_t s = r.home(key);
        uint32_t probes = 0;
        for (;;) {
            const unsigned long long old = atomicCAS(t.keys + s, ~0ull, key);
            if (old == ~0ull || old == key) { t.vals[s] = i | (mask ? WARM_CACHED : 0u); break; }
            s = r.next(s);
            if (++probes >= r.size) { atomicOr(t.status, STATUS_HASH_FULL); break; }
        }
    }
}

// Exclusive scan of in[0, min(n, *nDev)) into out (nDev may be null), total = the sum (may be null).
__global__ void k_scan(const uint32_t* in, uint32_t* out, uint32_t n, const uint32_t* nDev, uint32_t* total,
                       uint32_t* tileState, uint32_t* tileCounter, uint32_t* status);

// Contact kernels (k_contact.cu).
// Per thread: a 64-byte manifold slot, a hit flag and its share of its group's vertex tiles (100 bytes).
constexpr uint32_t NARROW_SMEM_PER_THREAD =
    uint32_t(sizeof(Manifold) + sizeof(uint32_t) + 2 * MAX_POLYGON_VERTICES * sizeof(V2) / NARROW_GROUP);
// Narrow phase + manifold compaction: manifolds of the hit pairs, in pair order, into out; tileState [tiles + 1] and
// tileCounter zeroed before the launch (tiles: blockDim.x / 32 x perWarp pairs each, perWarp at most 32).
// The narrow phase; lanes: polygon pairs one a lane where a warp has enough of them (blocks of up to
// NARROW_LANES_THREADS).
constexpr uint32_t NARROW_LANES_THREADS = 256;   // largest block of the one-pair-a-lane form
// Polygon pairs of a warp from which on each takes its own lane: the lanes together cost what about three rounds of the
// groups (four pairs each) do.
constexpr int NARROW_LANES_PAIRS = 10;
// Host side: raises the narrow phase's dynamic shared-memory limit (once per device).
cudaError_t narrow_init();
cudaError_t launch_narrow(bool chained, uint32_t blocks, uint32_t threads, cudaStream_t stream, DeviceWorld w, const uint2* pairs,
                   const uint32_t* nPairs, uint32_t pairCap, Manifold* out, uint32_t manifoldCap, uint32_t* nOut,
                   StepCounters* counters, uint32_t* tileState, uint32_t* tileCounter, uint32_t perWarp, bool lanes,
                   WarmTable warm, uint32_t* wakeIsland);
__global__ void k_warm_insert(WarmTable t);
__global__ void k_wake(DeviceWorld w, const Manifold* m, const uint32_t* nM, uint32_t* wakeIsland,
                       StepCounters* counters);
__global__ void k_wake_apply(DeviceWorld w, const uint32_t* wakeIsland, StepCounters* counters);
__global__ void k_island_init(DeviceWorld w, uint32_t* parent, uint32_t* flag);
__global__ void k_island_union(DeviceWorld w, const Manifold* m, const uint32_t* nM, uint32_t* parent);
__global__ void k_island_quiet(DeviceWorld w, uint32_t* parent, uint32_t* flag, float dt, float speedThreshold,
                               float timeThreshold);
// The end of a step on the device, by the last block of its last kernel: the warm-start count (a step without error
// bits becomes the next one's source) and the counters written to page-locked host memory. done: blocks finished,
// zeroed before the launch; null host: not the end of a step.
struct StepEnd {
    StepCounters* host;
    uint32_t* done;
    const uint32_t* nManifolds;
    uint32_t* nPrev;
};
__global__ void k_island_sleep(DeviceWorld w, uint32_t* parent, const uint32_t* flag, StepCounters* counters,
                               StepEnd end);
__global__ void k_state_flags(const uint8_t* bstate, const uint32_t* cbody, uint32_t nBodies, uint32_t nColliders,
                              uint32_t* bodyDyn, uint32_t* colDyn, uint32_t* colOther, uint32_t* sleeping);
__global__ void k_scatter_list(const uint32_t* flag, const uint32_t* offset, uint32_t n, uint32_t* list);

// Sleeping-island manifold store (k_islands.cu): restore at wake, move at sleep.
__global__ void k_isle_stage_flags(DeviceWorld w, const Manifold* isle, const uint32_t* isleId, const uint32_t* nIsle,
                                   const uint32_t* wakeIsland, uint32_t* flag);
__global__ void k_isle_stage_list(DeviceWorld w, const Manifold* isle, const uint32_t* nIsle, const uint32_t* flag,
                                  const uint32_t* off, uint32_t* list, uint32_t* listWorld);
__global__ void k_isle_append(Manifold* cur, const uint32_t* nCur, uint32_t cap, uint32_t* hint, const Manifold* isle,
                              const uint32_t* list, const uint32_t* nList, uint32_t* status);
__global__ void k_isle_merge(DeviceWorld w, const Manifold* cur, const uint32_t* hint, const uint32_t* nCur,
                             const uint32_t* seg, const Manifold* isle, const uint32_t* list,
                             const uint32_t* listWorld, const uint32_t* nList, uint32_t cap, Manifold* out,
                             uint32_t* outHint, uint32_t* status);
__global__ void k_isle_count(uint32_t* nCur, const uint32_t* nStage, const uint32_t* nList, uint32_t cap,
                             StepCounters* counters);
__global__ void k_isle_keep_flags(DeviceWorld w, const Manifold* isle, const uint32_t* isleId, const uint32_t* nIsle,
                                  const uint32_t* wakeIsland, uint32_t checkAlive, uint32_t* keep);
__global__ void k_isle_move_flags(DeviceWorld w, const Manifold* m, const uint32_t* nM, uint32_t* stay,
                                  uint32_t* move, uint32_t* moveIsland);
__global__ void k_isle_sleep_worlds(DeviceWorld w, const Manifold* isle, const uint32_t* nIsle, const uint32_t* keep,
                                    const uint32_t* keepOff, const Manifold* m, const uint32_t* nM,
                                    const uint32_t* move, const uint32_t* moveOff, uint32_t* keepWorld,
                                    uint32_t* moveWorld);
__global__ void k_isle_store_scatter(DeviceWorld w, const Manifold* isle, const uint32_t* isleId,
                                     const uint32_t* nIsle, const uint32_t* keep, const uint32_t* keepOff,
                                     const uint32_t* nKeep, const Manifold* m, const uint32_t* nM,
                                     const uint32_t* move, const uint32_t* moveOff, const uint32_t* nMove,
                                     const uint32_t* moveIsland, const uint32_t* keepWorld, const uint32_t* moveWorld,
                                     Manifold* isleOut, uint32_t* isleIdOut);
__global__ void k_isle_store_count(const uint32_t* nKeep, const uint32_t* nMove, uint32_t* nIsle);
__global__ void k_isle_append_moved(const Manifold* m, const uint32_t* nM, const uint32_t* move,
                                    const uint32_t* moveOff, const uint32_t* moveIsland, const uint32_t* nIsle,
                                    Manifold* isle, uint32_t* isleId);
__global__ void k_isle_add_count(uint32_t* nIsle, const uint32_t* nMove);
__global__ void k_isle_list_scatter(const Manifold* m, const uint32_t* color, const uint32_t* nM,
                                    const uint32_t* stay, const uint32_t* stayOff, Manifold* out,
                                    uint32_t* colorOut);
// Spatial queries: kind, the box (min x, min y, max x, max y) or circle (x, y, radius), tree selection; tileState
// [tiles + 1] (tiles of QUERY_SELECT_THREADS colliders, then the ticket counter) clear, nextState cleared for the next
// query; results to list / dist and the first hostCap of them to page-locked host: {count, timeout, indices, distances}.
constexpr uint32_t QUERY_SELECT_THREADS = 256;
enum QuerySelectKind : uint32_t { QUERY_SELECT_AABB = 0, QUERY_SELECT_CIRCLE = 1, QUERY_SELECT_CONTACTS = 2 };
struct QuerySelect {
    uint32_t kind, trees;
    float4 shape;
    uint32_t* tileState;
    uint32_t* nextState;
    uint32_t* list;
    float* dist;
    uint32_t* host;
    uint32_t hostCap;
    uint32_t* status;
};
__global__ void k_query_select(DeviceWorld w, QuerySelect q);

// Body constraints (k_joints.cu): springs (kind 0), revolute (1), prismatic (2) and slider (3) joints and motors
// (4), the reference's ConstraintType order, each kind's active
// constraints in rec[k] grouped by level (level l: [levelStart[k][l], levelStart[k][l + 1])), solver data in
// data[k], the motors' accumulated impulses by dense index in motorImpulse. One CTA of JOINT_THREADS threads.
constexpr uint32_t JOINT_KINDS_DEVICE = 5;
constexpr uint32_t JOINT_THREADS = 1024;
// The dataflow schedule (k_joints_flow): the bodies that active constraints name, with how many constraints of each type
// act on them (dynamic bodies), and per constraint its bodies in that list and its rank among its type's on each.
struct JointBody {
    uint32_t body;
    uint16_t degree[JOINT_KINDS_DEVICE];
    uint16_t moves;
};
static_assert(sizeof(JointBody) == 16, "JointBody is 16 bytes");
struct JointFlow {
    uint16_t a, b, rankA, rankB;
};
constexpr uint32_t JOINT_FLOW_BODY_BYTES = sizeof(float4) + sizeof(JointBody) + sizeof(float2);
constexpr uint32_t JOINT_FLOW_BODIES = 5600;   // 40 B of shared memory each
struct JointLaunch {
    const JointRec* rec[JOINT_KINDS_DEVICE];
    const JointFlow* flow[JOINT_KINDS_DEVICE];
    const JointBody* body;
    uint32_t bodies;
    uint32_t* status;
    JointData* data[JOINT_KINDS_DEVICE];
    const uint32_t* levelStart[JOINT_KINDS_DEVICE];
    uint32_t count[JOINT_KINDS_DEVICE];
    uint32_t levels[JOINT_KINDS_DEVICE];
    uint32_t iterations[JOINT_KINDS_DEVICE];
    uint32_t maxIterations;
    float dt;
    float* motorImpulse;
};
__global__ void k_joints(DeviceWorld w, JointLaunch L);
__global__ void k_joints_flow(DeviceWorld w, JointLaunch L);
// Host side: raises the dataflow kernel's dynamic shared-memory limit (once per device).
cudaError_t joints_init();
// Island links of the active constraints' body pairs (edges[i] = {a, b}), as k_island_union links manifolds.
__global__ void k_island_union_edges(DeviceWorld w, const uint2* edges, uint32_t n, uint32_t* parent);

// Collision events (k_events.cu): the events of the manifolds in man[0, min(*nMan, manCap)) whose colliders opted
// in (cev), appended to ring (counters->events counts them all; STATUS_EVENT_OVERFLOW when more than ringCap).
// Launched with a multiple of 32 threads a block, before the solver changes the velocities.
__global__ void k_collision_events(DeviceWorld w, const ColliderEvent* cev, const Manifold* man,
                                   const uint32_t* nMan, uint32_t manCap, EventRecord* ring, uint32_t ringCap,
                                   StepCounters* counters);

// Batch repacking (k_repack.cu). A segment copies 'count' elements from [src, ...) of the current array (fromNew
// 0), or from the staged section of joining world 'src' (fromNew 1), to [dst, ...) of the new array; the deltas
// shift the indices stored in the elements (new start - source start of that kind of element in the segment's
// world; a staged world's indices start at 0).
struct GatherSeg {
    uint32_t dst, src, count, fromNew;
    int32_t dBody, dCol, dCircle, dBox, dPoly, dVert, dMat, pad;
};
enum GatherMode : uint32_t {
    GATHER_PLAIN = 0, GATHER_ISLAND, GATHER_BODY, GATHER_SHAPE, GATHER_MATERIAL, GATHER_VERTEX
};
template <class T>
cudaError_t launch_gather(T* dst, const T* srcOld, const T* srcNew, const GatherSeg* segs, uint32_t nsegs,
                          uint32_t total, uint32_t mode, uint32_t grid, cudaStream_t stream,
                          const unsigned long long* sections, uint32_t nsec, uint32_t section);
__global__ void k_world_of(const uint32_t* starts, uint32_t worlds, uint32_t n, uint32_t* out);
__global__ void k_fill_u32(uint32_t* out, uint32_t n, uint32_t value);
// Host reads: how k_extract packs a field (EXTRACT_DIRECT fields are copied as they lie).
enum ExtractKind : uint32_t {
    EXTRACT_DIRECT = 0, EXTRACT_F4_COMP, EXTRACT_F4_XYZ, EXTRACT_F2_COMP, EXTRACT_U8_U32, EXTRACT_ISLAND
};
struct SectionCopy {
    uint8_t* dst;
    const uint8_t* src;
    uint64_t bytes;
};
struct SectionCopies {
    uint32_t count;
    SectionCopy c[32];
};
__global__ void k_copy_sections(SectionCopies a);
__global__ void k_extract(const void* src, uint32_t lo, uint32_t n, uint32_t kind, uint32_t comp, uint32_t bias,
                          void* out);

}  // namespace ag2d
