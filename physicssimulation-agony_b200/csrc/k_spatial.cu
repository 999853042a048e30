// Spatial phase kernels: integration, collider poses + AABBs, Morton keys, onesweep radix sort, Karras LBVH build
// and refit, and the candidate-pair query. Reference routines cited per kernel (paths relative to
// PhysicsSimulation-Agony/PS_AGONY2D/).
#include <algorithm>

#include "ag2d_ccd.cuh"
#include "ag2d_kernels.cuh"

namespace ag2d {

// ---------------------------------------------------------------------------------------------------------------
// Integration: Integrator::integratePhase1/2_VelocityVerlet + dampAngularVelocities (Integration/Integrator.cpp:
// 140-299, call order Simulation.cpp:392-407), wrapBodyRotations (LeftOutFunctions.cpp:13-60) and
// computeRotationCosSin (Integrator.cpp:301-311), fused per dynamic body. Elementwise: HBM-bound at 40 B/body.
// ---------------------------------------------------------------------------------------------------------------
// phase: 3 both halves; 1 the first (half kick and damping: Integrator::integratePhase1_VelocityVerlet +
// dampAngularVelocities); 2 the second (position step, half kick, damping, wrap, cos/sin). The body constraints
// run between the two (Simulation.cpp:399-404).
__device__ __forceinline__ void integrate_kick(float4& v, const float4& p, bool simd, float gdx, float gdy,
                                               float dampHalf /* damping^(dt/2), or >= 1 when damping is off */)
{
    const bool movable = v.w != 0.0f;
    const bool angMovable = p.w != 0.0f;
    if (simd) { v.x += movable ? gdx : 0.0f; v.y += movable ? gdy : 0.0f; }
    else { v.x += gdx * float(movable); v.y += gdy * float(movable); }
    if (dampHalf < 1.0f) {
        const float nv = v.z * dampHalf;
        if (simd) v.z = angMovable ? nv : v.z;
        else { const float m = float(angMovable); v.z = m * nv + (1.0f - m) * v.z; }
    }
}

// The second half; wrap holds the body's wrap count in and out.
__device__ __forceinline__ void integrate_move(const DeviceWorld& w, uint32_t b, float4 v, float4 p, float wrap, bool simd,
                                               const IntegrateParams& ip)
{
    p.x = v.x * ip.dt + p.x;
    p.y = v.y * ip.dt + p.y;
    p.z = v.z * ip.dt + p.z;
    const float halfDT = ip.dt * 0.5f;
    integrate_kick(v, p, simd, ip.gx * halfDT, ip.gy * halfDT, ip.dampHalf);
    float wraps;
    p.z = wrap_angle(p.z, simd, wraps);
    w.wrapCount[b] = wrap + wraps;
    float c, s;
    fast_cos_sin(p.z, simd, c, s);
    w.bvel[b] = v;
    w.bpos[b] = p;
    w.brot[b] = make_float2(c, s);
}

__global__ void k_integrate(DeviceWorld w, const uint32_t* dynBody, const uint8_t* dynSimd,
                            uint32_t nDyn, IntegrateParams ip, uint32_t phase)
{
    chain_begin();
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < nDyn; k += gridDim.x * blockDim.x) {
        const uint32_t b = dynBody[k];
        const bool simd = dynSimd ? dynSimd[k] != 0 : k < (nDyn & ~7u);
        float4 v = w.bvel[b];
        const float4 p = w.bpos[b];
        const float halfDT = ip.dt * 0.5f;
        if (phase & 1u) integrate_kick(v, p, simd, ip.gx * halfDT, ip.gy * halfDT, ip.dampHalf);
        if (phase & 2u) integrate_move(w, b, v, p, w.wrapCount[b], simd, ip);
        else w.bvel[b] = v;
    }
}

// The start of a step in one launch: the body state saved (a step that overflows a buffer is redone from it), wrap
// counts cleared, the integration (both halves, or the first when body constraints follow), the step's counters reset
// and every buffer that the step's kernels expect cleared. As separate copies, clears and kernels these were twenty
// operations of two to three microseconds each, most of a small world's step; by bytes it is one pass over the bodies.
__global__ void k_step_begin(StepBegin a)
{
    const DeviceWorld& w = a.w;
    const uint32_t first = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    if (first == 0) {
        StepCounters c = {};
        c.stored = *a.nIsle;
        *a.counters = c;
    }
    // Bodies that are not dynamic (the dynamic ones are the list's, below).
    for (uint32_t b = first; b < w.nBodies; b += stride) {
        const uint8_t st = w.bstate[b];
        a.snapState[b] = st;
        a.snapTimer[b] = w.sleepTimer[b];
        a.snapIsland[b] = w.sleepIsland[b];
        if (st == STATE_DYNAMIC) continue;
        a.snapVel[b] = w.bvel[b];
        a.snapPos[b] = w.bpos[b];
        a.snapRot[b] = w.brot[b];
        a.snapWrap[b] = w.wrapCount[b];
        w.wrapCount[b] = 0.0f;
    }
    const float halfDT = a.ip.dt * 0.5f;
    for (uint32_t k = first; k < a.nDyn; k += stride) {
        const uint32_t b = a.dynBody[k];
        const bool simd = a.dynSimd ? a.dynSimd[k] != 0 : k < (a.nDyn & ~7u);
        float4 v = w.bvel[b];
        const float4 p = w.bpos[b];
        a.snapVel[b] = v;
        a.snapPos[b] = p;
        a.snapRot[b] = w.brot[b];
        a.snapWrap[b] = w.wrapCount[b];
        integrate_kick(v, p, simd, a.ip.gx * halfDT, a.ip.gy * halfDT, a.ip.dampHalf);
        if (a.both) {
            integrate_move(w, b, v, p, 0.0f, simd, a.ip);
        } else {
            w.bvel[b] = v;
            w.wrapCount[b] = 0.0f;
        }
    }
    for (uint32_t i = first; i < a.copyCount; i += stride) a.copyDst[i] = a.copySrc[i];
    for (uint32_t f = 0; f < a.fills; f++) {
        const FillRegion r = a.fill[f];
        if (r.iota) {
            for (uint32_t i = first; i < r.words; i += stride) r.p[i] = i;
            continue;
        }
        const uint32_t quads = r.words / 4;
        uint4* const q = reinterpret_cast<uint4*>(r.p);
        for (uint32_t i = first; i < quads; i += stride) q[i] = make_uint4(r.value, r.value, r.value, r.value);
        if (first < r.words - 4 * quads) r.p[4 * quads + first] = r.value;
    }
}

// ---------------------------------------------------------------------------------------------------------------
// Collider world pose and AABB: computeColliderWorldPositions/Rotations (Simulation.cpp:673-736) and the shape
// AABB builders (SimulationImpl/ColliderAABBBuilder.cpp:8-136). 'list' selects the colliders with their SIMD-path
// flags (the k-th collider of its world's pass takes the reference's SIMD path iff k < (count & ~7)); null = every
// collider, classified by its index within its world's collider range (the reference's live-range pass), or only
// those of the worlds set in 'worldMask'.
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ float4 collider_aabb(const DeviceWorld& w, uint32_t c, float x, float y, float cs, float sn)
{
    const uint32_t packed = w.cshape[c];
    const uint32_t si = shape_index(packed);
    switch (shape_type(packed)) {
    case SHAPE_CIRCLE: {
        const float r = w.circleRadius[si];
        return make_float4(x - r, y - r, x + r, y + r);
    }
    case SHAPE_BOX: {
        const float2 h = w.boxHalf[si];
        const float ac = fabsf(cs), as = fabsf(sn);
        const float ex = ac * h.x + as * h.y;
        const float ey = as * h.x + ac * h.y;
        return make_float4(x - ex, y - ey, x + ex, y + ey);
    }
    case SHAPE_CAPSULE: {   // buildCapsuleAABBs (ColliderAABBBuilder.cpp:138-175): (half length, radius)
        const float2 h = w.boxHalf[si];
        const float ex = fabsf(cs) * h.x + h.y;
        const float ey = fabsf(sn) * h.x + h.y;
        return make_float4(x - ex, y - ey, x + ex, y + ey);
    }
    default: {
        const uint32_t off = w.polyOffset[si], nv = w.polyCount[si];
        float mnx = FLT_MAX, mny = FLT_MAX, mxx = -FLT_MAX, mxy = -FLT_MAX;
        for (uint32_t k = 0; k < nv; k++) {
            const float2 v = w.polyVerts[off + k];
            const float wx = cs * v.x - sn * v.y;
            const float wy = sn * v.x + cs * v.y;
            mnx = rfminf(mnx, wx); mxx = rfmaxf(mxx, wx);
            mny = rfminf(mny, wy); mxy = rfmaxf(mxy, wy);
        }
        return make_float4(x + mnx, y + mny, x + mxx, y + mxy);
    }
    }
}

// insert: the warm-start table filled beside the poses (one launch for two passes that touch nothing in common), or a
// table without keys.
__global__ void k_collider_pose(DeviceWorld w, const uint32_t* list, const uint8_t* listSimd,
                                uint32_t n, const uint32_t* worldMask, WarmTable insert)
{
    chain_begin();
    if (insert.keys) warm_insert(insert);
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const uint32_t c = list ? list[k] : k;
        if (worldMask && !worldMask[w.colWorld[c]]) continue;
        bool simd;
        if (list) {
            simd = listSimd ? listSimd[k] != 0 : k < (n & ~7u);
        } else if (w.colWorld) {
            const uint32_t wd = w.colWorld[c];
            const uint32_t lo = w.worldColStart[wd], hi = w.worldColStart[wd + 1];
            simd = (c - lo) < ((hi - lo) & ~7u);
        } else {
            simd = k < (n & ~7u);
        }
        const uint32_t b = w.cbody[c];
        const float4 off = w.coff[c];
        const float4 bp = w.bpos[b];
        const float2 br = w.brot[b];
        const float x = bp.x + (off.x * br.x - off.y * br.y);
        const float y = bp.y + (off.x * br.y + off.y * br.x);
        float wraps;
        const float rot = wrap_angle(bp.z + off.z, simd, wraps);
        float cs, sn;
        fast_cos_sin(rot, simd, cs, sn);
        w.cpose[c] = make_float4(x, y, cs, sn);
        w.cworldRot[c] = rot;
        w.caabb[c] = collider_aabb(w, c, x, y, cs, sn);
    }
}

// ---------------------------------------------------------------------------------------------------------------
// Tree bounds: the union of the AABBs of one tree's colliders (BvhTree::gatherCentroids, BvhTree.cpp:148-188).
// min/max are order-independent, so a block reduction plus ordered-integer atomics gives the sequential result
// (up to the sign of a zero bound).
// ---------------------------------------------------------------------------------------------------------------
// The union of a block's boxes (blocks of at most 32 warps), valid in thread 0.
__device__ __forceinline__ float4 block_bounds(float mnx, float mny, float mxx, float mxy)
{
    for (int o = 16; o > 0; o >>= 1) {
        mnx = fminf(mnx, __shfl_xor_sync(0xffffffffu, mnx, o));
        mny = fminf(mny, __shfl_xor_sync(0xffffffffu, mny, o));
        mxx = fmaxf(mxx, __shfl_xor_sync(0xffffffffu, mxx, o));
        mxy = fmaxf(mxy, __shfl_xor_sync(0xffffffffu, mxy, o));
    }
    __shared__ float4 part[32];
    const uint32_t warp = threadIdx.x >> 5, warps = (blockDim.x + 31) >> 5;
    if ((threadIdx.x & 31) == 0) part[warp] = make_float4(mnx, mny, mxx, mxy);
    __syncthreads();
    float4 r = part[0];
    if (threadIdx.x == 0)
        for (uint32_t k = 1; k < warps; k++) {
            const float4 q = part[k];
            r = make_float4(fminf(r.x, q.x), fminf(r.y, q.y), fmaxf(r.z, q.z), fmaxf(r.w, q.w));
        }
    return r;
}

// One world: every block leaves the bounds of its colliders in parts[block] (k_morton's blocks reduce them). Several
// worlds: 4 ordered words each; a warp whose lanes all belong to one world reduces first and issues one atomic per
// word, a warp that straddles worlds issues per-lane atomics. The sort's words are cleared beside it.
__global__ void k_bounds(const float4* aabb, const uint32_t* list, uint32_t n,
                         const uint32_t* colWorld, uint32_t* bounds,
                         float4* parts, uint32_t* clear, uint32_t clearWords)
{
    chain_begin();
    const uint32_t stride = gridDim.x * blockDim.x;
    const uint32_t base0 = blockIdx.x * blockDim.x;
    for (uint32_t i = base0 + threadIdx.x; i < clearWords; i += stride) clear[i] = 0u;
    if (!colWorld) {
        float mnx = FLT_MAX, mny = FLT_MAX, mxx = -FLT_MAX, mxy = -FLT_MAX;
        for (uint32_t k = base0 + threadIdx.x; k < n; k += stride) {
            const float4 a = aabb[list ? list[k] : k];
            mnx = fminf(mnx, a.x); mny = fminf(mny, a.y); mxx = fmaxf(mxx, a.z); mxy = fmaxf(mxy, a.w);
        }
        const float4 r = block_bounds(mnx, mny, mxx, mxy);
        if (threadIdx.x == 0)   // a block that saw no collider leaves neutral bounds
            parts[blockIdx.x] = r.x <= r.z ? r : make_float4(FLT_MAX, FLT_MAX, -FLT_MAX, -FLT_MAX);
        return;
    }
    for (uint32_t base = base0; base < n; base += stride) {
        const uint32_t k = base + threadIdx.x;
        const bool valid = k < n;
        const uint32_t c = valid ? (list ? list[k] : k) : 0u;
        const float4 a = valid ? aabb[c] : make_float4(FLT_MAX, FLT_MAX, -FLT_MAX, -FLT_MAX);
        const uint32_t wd = valid ? (colWorld ? colWorld[c] : 0u) : 0xFFFFFFFFu;
        const uint32_t active = __ballot_sync(0xffffffffu, valid);
        const uint32_t firstLane = __ffs(active) - 1;
        const uint32_t w0 = __shfl_sync(0xffffffffu, wd, firstLane);
        const bool uniform = __all_sync(0xffffffffu, !valid || wd == w0);
        if (uniform) {
            float mnx = a.x, mny = a.y, mxx = a.z, mxy = a.w;
            for (int o = 16; o > 0; o >>= 1) {
                mnx = fminf(mnx, __shfl_xor_sync(0xffffffffu, mnx, o));
                mny = fminf(mny, __shfl_xor_sync(0xffffffffu, mny, o));
                mxx = fmaxf(mxx, __shfl_xor_sync(0xffffffffu, mxx, o));
                mxy = fmaxf(mxy, __shfl_xor_sync(0xffffffffu, mxy, o));
            }
            if ((threadIdx.x & 31) == firstLane && active) {
                uint32_t* b = bounds + 4 * w0;
                atomicMin(b + 0, float_to_ordered(mnx));
                atomicMin(b + 1, float_to_ordered(mny));
                atomicMax(b + 2, float_to_ordered(mxx));
                atomicMax(b + 3, float_to_ordered(mxy));
            }
        } else if (valid) {
            uint32_t* b = bounds + 4 * wd;
            atomicMin(b + 0, float_to_ordered(a.x));
            atomicMin(b + 1, float_to_ordered(a.y));
            atomicMax(b + 2, float_to_ordered(a.z));
            atomicMax(b + 3, float_to_ordered(a.w));
        }
    }
}

__global__ void k_bounds_init(uint32_t* bounds, uint32_t worlds)
{
    for (uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w < worlds; w += gridDim.x * blockDim.x) {
        bounds[4 * w + 0] = float_to_ordered(FLT_MAX);
        bounds[4 * w + 1] = float_to_ordered(FLT_MAX);
        bounds[4 * w + 2] = float_to_ordered(-FLT_MAX);
        bounds[4 * w + 3] = float_to_ordered(-FLT_MAX);
    }
}

// Elements per world of a work list (for the per-world segment offsets of a tree or a manifold list).
__global__ void k_count_world(const uint32_t* __restrict__ list, uint32_t n, const uint32_t* __restrict__ elemWorld,
                              uint32_t* __restrict__ counts)
{
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x)
        atomicAdd(counts + elemWorld[list ? list[k] : k], 1u);
}

// SIMD-path flag of each work-list entry: the rank of its element among its world's listed elements, against that
// world's (count & ~7). 'offsets' is the exclusive scan of the list flags over all elements, 'worldStart' the
// first element index of each world.
__global__ void k_simd_flags(const uint32_t* __restrict__ list, uint32_t n, const uint32_t* __restrict__ offsets,
                             uint32_t nElems, const uint32_t* __restrict__ elemWorld,
                             const uint32_t* __restrict__ worldStart, uint32_t worlds, uint8_t* __restrict__ simd)
{
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const uint32_t w = elemWorld[list[k]];
        const uint32_t firstElem = worldStart[w], endElem = worldStart[w + 1];
        const uint32_t lo = offsets[firstElem];
        const uint32_t hi = endElem < nElems ? offsets[endElem] : n;
        simd[k] = (k - lo) < ((hi - lo) & ~7u) ? 1u : 0u;
    }
}

// ---------------------------------------------------------------------------------------------------------------
// Morton keys: transformCentroids + computeMortonCodes (BvhTree.cpp:191-280). 2 x centroid scaled into [0, 65535]
// per axis by the tree bounds, truncated, bits interleaved (y in the odd bits): a 32-bit key.
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t morton_key(const float4& a, float bminX, float bminY, float bmaxX, float bmaxY)
{
    const float kEps = 1e-5f;
    const float maxX = rfmaxf(bmaxX, bminX + kEps);
    const float maxY = rfmaxf(bmaxY, bminY + kEps);
    const float clampMax = 65535.0f;
    const float scaleX = clampMax / (maxX - bminX);
    const float scaleY = clampMax / (maxY - bminY);
    const float negScaledMinX = -bminX * scaleX;
    const float negScaledMinY = -bminY * scaleY;
    const float halfScaleX = scaleX * 0.5f;
    const float halfScaleY = scaleY * 0.5f;
    const float cx = a.x + a.z;
    const float cy = a.y + a.w;
    float tx = cx * halfScaleX + negScaledMinX;
    float ty = cy * halfScaleY + negScaledMinY;
    tx = tx < 0.0f ? 0.0f : (tx > clampMax ? clampMax : tx);
    ty = ty < 0.0f ? 0.0f : (ty > clampMax ? clampMax : ty);
    return (part1by1(uint32_t(ty)) << 1) | part1by1(uint32_t(tx));
}

// Keys of a radix sort's digit histograms, counted in shared memory ('sh', zeroed, 4 x 256) by blocks of 256 threads and
// added to 'hist' at the end; the last block to finish turns each histogram into its exclusive scan.
__device__ __forceinline__ void digits_count(uint32_t* sh, uint32_t k)
{
    atomicAdd(&sh[0 * 256 + (k & 0xFF)], 1u);
    atomicAdd(&sh[1 * 256 + ((k >> 8) & 0xFF)], 1u);
    atomicAdd(&sh[2 * 256 + ((k >> 16) & 0xFF)], 1u);
    atomicAdd(&sh[3 * 256 + (k >> 24)], 1u);
}
__device__ __forceinline__ void digits_end(const uint32_t* sh, uint32_t* hist, uint32_t* done)
{
    __shared__ uint32_t warpSum[8], lastBlock;
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    __syncthreads();
    for (uint32_t i = t; i < 4 * 256; i += 256)
        if (sh[i]) atomicAdd(&hist[i], sh[i]);
    __threadfence();
    __syncthreads();
    if (t == 0) lastBlock = atomicAdd(done, 1u) == gridDim.x - 1 ? 1u : 0u;
    __syncthreads();
    if (!lastBlock) return;
    __threadfence();
    for (uint32_t j = 0; j < 4; j++) {
        const uint32_t v = __ldcg(hist + j * 256 + t);
        uint32_t incl = v;
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += x;
        }
        if (lane == 31) warpSum[warp] = incl;
        __syncthreads();
        for (uint32_t k = 0; k < warp; k++) incl += warpSum[k];
        hist[j * 256 + t] = incl - v;
        __syncthreads();
    }
}

// Morton keys with the digit histograms of their sort (blocks of 256 threads). One world: the bounds are the union of
// parts[0, nParts), reduced by every block.
__global__ void __launch_bounds__(256) k_morton(const float4* aabb, const uint32_t* list,
                                                uint32_t n, const uint32_t* colWorld,
                                                const uint32_t* bounds,
                                                const float4* parts, uint32_t nParts,
                                                uint32_t* keys, uint32_t* vals,
                                                uint32_t* keyOf, uint32_t* hist, uint32_t* done)
{
    chain_begin();
    __shared__ uint32_t sh[4 * 256];
    __shared__ float4 whole;
    for (uint32_t i = threadIdx.x; i < 4 * 256; i += 256) sh[i] = 0;
    if (!colWorld) {
        float mnx = FLT_MAX, mny = FLT_MAX, mxx = -FLT_MAX, mxy = -FLT_MAX;
        for (uint32_t k = threadIdx.x; k < nParts; k += 256) {
            const float4 a = parts[k];
            mnx = fminf(mnx, a.x); mny = fminf(mny, a.y); mxx = fmaxf(mxx, a.z); mxy = fmaxf(mxy, a.w);
        }
        const float4 r = block_bounds(mnx, mny, mxx, mxy);
        if (threadIdx.x == 0) whole = r;
    }
    __syncthreads();
    for (uint32_t k = blockIdx.x * 256 + threadIdx.x; k < n; k += gridDim.x * 256) {
        const uint32_t c = list ? list[k] : k;
        float4 b;
        if (colWorld) {
            const uint32_t* const words = bounds + 4 * colWorld[c];
            b = make_float4(ordered_to_float(words[0]), ordered_to_float(words[1]), ordered_to_float(words[2]),
                            ordered_to_float(words[3]));
        } else {
            b = whole;
        }
        const uint32_t key = morton_key(aabb[c], b.x, b.y, b.z, b.w);
        keys[k] = key;
        vals[k] = c;
        if (keyOf) keyOf[c] = key;
        digits_count(sh, key);
    }
    digits_end(sh, hist, done);
}

// After the Morton passes: the world id of each sorted element becomes the key of the next (stable) passes, so the
// final order is by (world, Morton key) with ties in collider order.
__global__ void __launch_bounds__(256) k_world_keys(const uint32_t* __restrict__ vals, uint32_t n,
                                                    const uint32_t* __restrict__ colWorld,
                                                    uint32_t* __restrict__ keys, uint32_t* hist, uint32_t* done)
{
    __shared__ uint32_t sh[4 * 256];
    for (uint32_t i = threadIdx.x; i < 4 * 256; i += 256) sh[i] = 0;
    __syncthreads();
    for (uint32_t i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) {
        const uint32_t wd = colWorld[vals[i]];
        keys[i] = wd;
        digits_count(sh, wd);
    }
    digits_end(sh, hist, done);
}

// First index of every world's segment of a world-grouped list: segStart[w] = offsets[worldStart[w]] (the exclusive
// scan of the list flags over the elements), segStart[worlds] = the list length.
__global__ void k_seg_starts(const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ worldStart,
                             uint32_t worlds, uint32_t nElems, const uint32_t* __restrict__ total,
                             uint32_t* __restrict__ segStart)
{
    for (uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w <= worlds; w += gridDim.x * blockDim.x) {
        const uint32_t e = worldStart[w];
        segStart[w] = (w == worlds || e >= nElems) ? *total : offsets[e];
    }
}

// Segment starts of the world-grouped manifold list (world of body a, non-decreasing): the thread at each world
// change fills the starts of every world in the gap, so worlds without manifolds get empty segments.
__global__ void k_manifold_segments(const Manifold* m, const uint32_t* nM,
                                    const uint32_t* cbody, const uint32_t* bodyWorld,
                                    uint32_t worlds, uint32_t* segStart)
{
    chain_begin();
    const uint32_t n = *nM;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i <= n; i += gridDim.x * blockDim.x) {
        const int prev = i == 0 ? -1 : int(bodyWorld[cbody[m[i - 1].a]]);
        const int cur = i == n ? int(worlds) : int(bodyWorld[cbody[m[i].a]]);
        for (int w = prev + 1; w <= cur; w++) segStart[w] = i;
    }
}

// Sorted-order gathers for the trees of several worlds: Morton key (after the world passes), world id and AABB of every
// leaf.
__global__ void k_tree_gather(const uint32_t* __restrict__ vals, uint32_t n, const uint32_t* __restrict__ keyOf,
                              const uint32_t* __restrict__ colWorld, const float4* __restrict__ caabb,
                              uint32_t* __restrict__ sortedKey, uint32_t* __restrict__ sortedWorld,
                              float4* __restrict__ leafAabb)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t c = vals[i];
        sortedKey[i] = keyOf[c];
        sortedWorld[i] = colWorld[c];
        leafAabb[i] = caabb[c];
    }
}

// ---------------------------------------------------------------------------------------------------------------
// Onesweep LSD radix sort of (key, value) pairs, 8-bit digits, stable: the same permutation as
// BvhTree::sortByMortonCodes (BvhTree.cpp:282-354). The kernel that makes the keys counts all four digits; then per
// digit one kernel ranks a tile (per warp, striped so ranks follow input order), resolves the tile's global digit
// offsets by decoupled look-back over the preceding tiles, reorders the tile in shared memory and writes each digit's
// run contiguously.
// ---------------------------------------------------------------------------------------------------------------
// The lanes of a full warp that hold the same 8-bit digit as this one (among the valid): one ballot a bit. match.any
// serves one distinct value after the other, and the digits of a warp mostly differ: with it the ranking of 2,000 keys
// in one CTA took 4,100 cycles a pass.
__device__ __forceinline__ uint32_t digit_peers(uint32_t d, bool valid)
{
    uint32_t peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
    for (uint32_t b = 0; b < 8; b++) {
        const bool bit = (d >> b) & 1u;
        const uint32_t with = __ballot_sync(0xffffffffu, bit);
        peers &= bit ? with : ~with;
    }
    return peers;
}

template <uint32_t SORT_ITEMS>
__global__ void __launch_bounds__(SORT_THREADS) k_sort_pass(
    const uint32_t* keysIn, const uint32_t* valsIn, uint32_t* keysOut,
    uint32_t* valsOut, uint32_t n, uint32_t shift, const uint32_t* digitBase,
    uint32_t* tileState, uint32_t* tileCounter, uint32_t* status)
{
    chain_begin();
    constexpr uint32_t WARPS = SORT_THREADS / 32, SORT_TILE = SORT_THREADS * SORT_ITEMS;
    __shared__ uint32_t warpHist[WARPS][256];
    __shared__ uint32_t digitStart[256];     // exclusive scan of the tile's digit counts
    __shared__ uint32_t globalBase[256];     // global output position of the tile's first key of each digit
    __shared__ uint32_t smKey[SORT_TILE];
    __shared__ uint32_t smVal[SORT_TILE];
    __shared__ uint32_t tileSlot;

    if (threadIdx.x == 0) tileSlot = atomicAdd(tileCounter, 1u);   // tiles start in order: look-back progresses
    for (uint32_t i = threadIdx.x; i < WARPS * 256; i += SORT_THREADS) (&warpHist[0][0])[i] = 0;
    __syncthreads();
    const uint32_t tile = tileSlot;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t segBase = tile * SORT_TILE + warp * (SORT_ITEMS * 32);
    const uint32_t ltMask = (1u << lane) - 1u;

    uint32_t key[SORT_ITEMS], val[SORT_ITEMS], rank[SORT_ITEMS];
#pragma unroll
    for (uint32_t k = 0; k < SORT_ITEMS; k++) {
        const uint32_t idx = segBase + k * 32 + lane;
        const bool valid = idx < n;
        key[k] = valid ? keysIn[idx] : 0u;
        val[k] = valid ? valsIn[idx] : 0u;
        const uint32_t d = (key[k] >> shift) & 0xFFu;
        const uint32_t peers = digit_peers(d, valid);
        const uint32_t before = __popc(peers & ltMask);
        uint32_t base = 0;
        if (valid) base = warpHist[warp][d];
        __syncwarp();
        if (valid && before == 0) warpHist[warp][d] = base + __popc(peers);
        __syncwarp();
        rank[k] = base + before;
    }
    __syncthreads();

    // Per digit (one thread each): warp offsets within the tile, the tile aggregate, look-back.
    {
        const uint32_t d = threadIdx.x;
        uint32_t running = 0;
#pragma unroll
        for (uint32_t wi = 0; wi < WARPS; wi++) {
            const uint32_t c = warpHist[wi][d];
            warpHist[wi][d] = running;
            running += c;
        }
        volatile uint32_t* state = tileState;
        if (tile == 0) {
            state[d] = (2u << 30) | running;
            globalBase[d] = digitBase[d];
        } else {
            state[tile * 256 + d] = (1u << 30) | running;
            uint32_t prefix = 0;
            int32_t t = int32_t(tile) - 1;
            uint32_t spins = 0;
            // Look back over a window of LOOKBACK predecessors per round trip: their states are loaded together,
            // then summed newest first up to the first inclusive prefix; a tile not yet published restarts the
            // window at that tile. Tile 0 always publishes an inclusive prefix, so the walk ends there at the latest.
            // Only a window that makes no progress counts towards the spin limit.
            constexpr int32_t LOOKBACK = 8;
            bool done = false;
            while (!done && t >= 0) {
                uint32_t s[LOOKBACK];
#pragma unroll
                for (int32_t j = 0; j < LOOKBACK; j++) s[j] = t - j >= 0 ? state[(t - j) * 256 + d] : (2u << 30);
#pragma unroll
                for (int32_t j = 0; j < LOOKBACK; j++) {
                    const uint32_t flag = s[j] >> 30;
                    if (flag == 0) break;   // not published yet: reload from tile t
                    prefix += s[j] & 0x3FFFFFFFu;
                    t--;
                    if (flag == 2) { done = true; break; }
                }
                if (!done && t >= 0 && (s[0] >> 30) == 0 && ++spins > SPIN_LIMIT) {
                    atomicOr(status, STATUS_LOOKBACK_TIMEOUT);
                    break;
                }
            }
            __threadfence();
            state[tile * 256 + d] = (2u << 30) | (prefix + running);
            globalBase[d] = digitBase[d] + prefix;
        }
        digitStart[d] = running;   // scanned below
    }
    __syncthreads();
    // Exclusive scan of the 256 digit counts (digitStart holds counts).
    if (threadIdx.x < 32) {
        uint32_t local[8];
        uint32_t sum = 0;
#pragma unroll
        for (uint32_t j = 0; j < 8; j++) { local[j] = digitStart[lane * 8 + j]; sum += local[j]; }
        uint32_t incl = sum;
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        uint32_t excl = incl - sum;
#pragma unroll
        for (uint32_t j = 0; j < 8; j++) { digitStart[lane * 8 + j] = excl; excl += local[j]; }
    }
    __syncthreads();
#pragma unroll
    for (uint32_t k = 0; k < SORT_ITEMS; k++) {
        const uint32_t idx = segBase + k * 32 + lane;
        if (idx < n) {
            const uint32_t d = (key[k] >> shift) & 0xFFu;
            const uint32_t pos = digitStart[d] + warpHist[warp][d] + rank[k];
            smKey[pos] = key[k];
            smVal[pos] = val[k];
        }
    }
    __syncthreads();
    const uint32_t tileBase = tile * SORT_TILE;
    const uint32_t tileN = n - tileBase < SORT_TILE ? n - tileBase : SORT_TILE;
    for (uint32_t i = threadIdx.x; i < tileN; i += SORT_THREADS) {
        const uint32_t k = smKey[i];
        const uint32_t d = (k >> shift) & 0xFFu;
        const uint32_t dst = globalBase[d] + (i - digitStart[d]);
        keysOut[dst] = k;
        valsOut[dst] = smVal[i];
    }
}

uint32_t sort_tiles(uint32_t n)
{
    const uint32_t tile = SORT_THREADS * (n <= SORT_SMALL_MAX ? SORT_ITEMS_SMALL : SORT_ITEMS_LARGE);
    return (n + tile - 1) / tile;
}

cudaError_t launch_sort_pass(const uint32_t* keysIn, const uint32_t* valsIn, uint32_t* keysOut, uint32_t* valsOut,
                             uint32_t n, uint32_t shift, const uint32_t* digitBase, uint32_t* tileState,
                             uint32_t* tileCounter, uint32_t* status, bool chained, cudaStream_t stream)
{
    return chain_launch(chained, n <= SORT_SMALL_MAX ? k_sort_pass<SORT_ITEMS_SMALL> : k_sort_pass<SORT_ITEMS_LARGE>, sort_tiles(n),
                        SORT_THREADS, 0, stream, keysIn, valsIn, keysOut, valsOut, n, shift, digitBase, tileState,
                        tileCounter, status);
}

// ---------------------------------------------------------------------------------------------------------------
// Karras LBVH over sorted keys (leaf = one collider). Internal node i spans [first, last] of the sorted order and
// splits at the highest differing bit; equal keys are ordered by index (key ++ index), as the reference's stable
// sort orders them. Children: >= 0 internal node, < 0 leaf ~rank. Worlds are independent segments [lo, hi) of the
// sorted order (sorted by world first): keys outside the segment count as unrelated (delta -1), so one build makes
// every world's tree, rooted at internal node lo.
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ int lbvh_delta(const uint32_t* keys, int lo, int hi, int i, int j)
{
    if (j < lo || j >= hi) return -1;
    const uint32_t a = keys[i], b = keys[j];
    if (a != b) return __clz(a ^ b);
    // Index tie-break on segment-relative positions: a world's tree does not depend on where its segment starts.
    return 32 + __clz(uint32_t(i - lo) ^ uint32_t(j - lo));
}

// Internal node i of a tree with prefix lengths delta(i, j) (-1 outside the segment): its range and split.
struct KarrasNode {
    int first, last, gamma;
};
template <class Delta>
__device__ __forceinline__ KarrasNode karras_node(int i, Delta delta)
{
    const int d = (delta(i, i + 1) - delta(i, i - 1)) >= 0 ? 1 : -1;
    const int dmin = delta(i, i - d);
    int lmax = 2;
    while (delta(i, i + lmax * d) > dmin) lmax <<= 1;
    int l = 0;
    for (int t = lmax >> 1; t >= 1; t >>= 1)
        if (delta(i, i + (l + t) * d) > dmin) l += t;
    const int j = i + l * d;
    const int dnode = delta(i, j);
    int s = 0, t = l;
    do {
        t = (t + 1) >> 1;
        if (delta(i, i + (s + t) * d) > dnode) s += t;
    } while (t > 1);
    return KarrasNode{i < j ? i : j, i < j ? j : i, i + s * d + (d < 0 ? -1 : 0)};
}

// sortedWorld/segStart null: one segment [0, n), and the leaf boxes are gathered beside the build.
__global__ void k_lbvh_build(const uint32_t* keys, const uint32_t* sortedWorld,
                             const uint32_t* segStart, int n, const uint32_t* vals,
                             const float4* caabb, float4* leafAabb,
                             int2* child, int* parent, int* leafParent,
                             float4* meet, NodeRec* rec)
{
    chain_begin();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int lo = 0, hi = n;
        if (!sortedWorld) leafAabb[i] = caabb[vals[i]];
        if (sortedWorld) {
            const uint32_t wd = sortedWorld[i];
            lo = int(segStart[wd]);
            hi = int(segStart[wd + 1]);
        }
        if (hi - lo == 1) leafParent[i] = -1;
        if (i >= hi - 1) continue;
        meet[i] = make_float4(__uint_as_float(MEET_EMPTY), 0.0f, 0.0f, 0.0f);
        if (i == lo) parent[i] = -1;
        const KarrasNode k = karras_node(i, [&](int a, int b) { return lbvh_delta(keys, lo, hi, a, b); });
        const int first = k.first, last = k.last, gamma = k.gamma;
        const int left = (first == gamma) ? ~gamma : gamma;
        const int right = (last == gamma + 1) ? ~(gamma + 1) : gamma + 1;
        child[i] = make_int2(left, right);
        rec[i].child = make_int2(left, right);
        rec[i].last = make_int2(gamma, last);
        if (left < 0) leafParent[~left] = i; else parent[left] = i;
        if (right < 0) leafParent[~right] = i; else parent[right] = i;
    }
}

// Swaps a box into a node's meeting slot with one 16-byte atomic and returns what was there.
__device__ __forceinline__ float4 exchange_box(float4* slot, float4 v)
{
    const unsigned long long lo = uint64_t(__float_as_uint(v.x)) | uint64_t(__float_as_uint(v.y)) << 32;
    const unsigned long long hi = uint64_t(__float_as_uint(v.z)) | uint64_t(__float_as_uint(v.w)) << 32;
    unsigned long long rlo, rhi;
    asm volatile("{\n\t.reg .b128 d, s;\n\tmov.b128 s, {%2, %3};\n\t"
                 "atom.relaxed.gpu.global.exch.b128 d, [%4], s;\n\tmov.b128 {%0, %1}, d;\n\t}"
                 : "=l"(rlo), "=l"(rhi) : "l"(lo), "l"(hi), "l"(slot) : "memory");
    return make_float4(__uint_as_float(uint32_t(rlo)), __uint_as_float(uint32_t(rlo >> 32)),
                       __uint_as_float(uint32_t(rhi)), __uint_as_float(uint32_t(rhi >> 32)));
}

// ---------------------------------------------------------------------------------------------------------------
// The whole tree of a segment in one CTA: bounds, Morton keys, sort, leaf gather and the nodes with their boxes, over
// every world segment [segStart[w], segStart[w + 1]) of a world-grouped list (or the one segment [0, n)) whose size is
// in (minSize, maxSize], maxSize at most THREADS x E. The results are those of the kernels above and below run one
// after the other.
// Sort: four 8-bit radix passes in shared memory, ranked per warp as k_sort_pass ranks a tile, so equal keys keep their
// list order.
// Nodes: bottom up from the leaves. A subtree over [l, r] is the left child of the node that splits after r when the
// keys r and r + 1 share more bits than l - 1 and l do, else the right child of the one that splits after l - 1. Both
// children leave their boxes at the split; the second one to arrive there (a meeting word) takes the whole range and
// carries on. The records are written afterwards, split by split; a node is numbered as Karras numbers it (r as a left
// child, l as a right child, the root 0).
// Bound: shared-memory latency and instruction issue of one CTA. One launch a size class in place of seven or more over
// all segments (bounds, keys, sort, gather, build, refit, their clears), which took 460 us a step on 4,096 worlds and 70
// to 95 us on one world of 64 to 2,048 colliders; now 250 and 16 to 40. Cycles at 2,000 leaves: sort 15,700, nodes and
// boxes 22,000, records 6,200. With a bitonic network and Karras's searches in shared memory it was 32,000 for the
// sort, 21,000 for the nodes and 29,000 for the boxes; the network in registers and shuffles took 20,700.
// ---------------------------------------------------------------------------------------------------------------
// Acquire-release fence of the CTA's memory order (__threadfence_block is the sequentially consistent one).
__device__ __forceinline__ void fence_cta() { asm volatile("fence.acq_rel.cta;" ::: "memory"); }

template <uint32_t THREADS, uint32_t E, bool MEET_SHARED>
struct TreeSmem {
    static constexpr uint32_t WARPS = THREADS / 32, CAP = THREADS * E;
    // The sort's words, and (MEET_SHARED) over them the boxes of both children of every split.
    static constexpr size_t SORT = (WARPS + 1) * 256 * sizeof(uint32_t) + CAP * (sizeof(uint32_t) + sizeof(uint16_t));
    __host__ __device__ static constexpr size_t front(uint32_t maxSize)
    {
        return MEET_SHARED && size_t(maxSize) * 32 > SORT ? size_t(maxSize) * 32 : SORT;
    }
    // Behind them the meeting words and the bits shared by each split's two keys.
    __host__ __device__ static constexpr size_t bytes(uint32_t maxSize) { return front(maxSize) + 5 * size_t(maxSize) + 16; }
};

template <uint32_t THREADS, uint32_t E, bool MEET_SHARED>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS) k_tree_segments(TreeBuild t, uint32_t minSize, uint32_t maxSize)
{
    if (t.chained) {
        chain_begin();
    } else {
        // The classes work on different segments: the next class's launch need not wait for this one.
        asm volatile("griddepcontrol.launch_dependents;");
    }
    using Smem = TreeSmem<THREADS, E, MEET_SHARED>;
    constexpr uint32_t WARPS = Smem::WARPS;
    extern __shared__ float4 treeTile[];
    __shared__ float4 part[WARPS];
    uint32_t* const hist = reinterpret_cast<uint32_t*>(treeTile);        // [WARPS][256]
    uint32_t* const digit = hist + WARPS * 256;                          // [256]
    uint32_t* const sortKey = digit + 256;                               // [CAP]
    uint16_t* const sortPos = reinterpret_cast<uint16_t*>(sortKey + Smem::CAP);   // [CAP]
    uint32_t* const met = reinterpret_cast<uint32_t*>(reinterpret_cast<unsigned char*>(treeTile) + Smem::front(maxSize));
    uint8_t* const shared = reinterpret_cast<uint8_t*>(met + maxSize);
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t ltMask = (1u << lane) - 1u;
    for (uint32_t w = blockIdx.x; w < t.worlds; w += gridDim.x) {
        const uint32_t lo = t.segStart ? t.segStart[w] : 0u, n = t.segStart ? t.segStart[w + 1] - lo : t.n;
        if (n <= minSize || n > maxSize) continue;
        const uint32_t* const list = t.list + lo;
        // Bounds of the segment's boxes.
        float4 bb = make_float4(FLT_MAX, FLT_MAX, -FLT_MAX, -FLT_MAX);
        for (uint32_t i = threadIdx.x; i < n; i += THREADS) {
            const float4 a = t.caabb[__ldg(list + i)];
            bb = make_float4(fminf(bb.x, a.x), fminf(bb.y, a.y), fmaxf(bb.z, a.z), fmaxf(bb.w, a.w));
        }
        for (int o = 16; o > 0; o >>= 1) {
            bb.x = fminf(bb.x, __shfl_xor_sync(0xffffffffu, bb.x, o));
            bb.y = fminf(bb.y, __shfl_xor_sync(0xffffffffu, bb.y, o));
            bb.z = fmaxf(bb.z, __shfl_xor_sync(0xffffffffu, bb.z, o));
            bb.w = fmaxf(bb.w, __shfl_xor_sync(0xffffffffu, bb.w, o));
        }
        if (lane == 0) part[warp] = bb;
        __syncthreads();
        for (uint32_t k = 0; k < WARPS; k++) {
            const float4 q = part[k];
            bb = make_float4(fminf(bb.x, q.x), fminf(bb.y, q.y), fmaxf(bb.z, q.z), fmaxf(bb.w, q.w));
        }
        // This thread's elements: one a stretch of 32, the stretches of a warp consecutive (list order by warp, then
        // stretch, then lane). 'per' stretches a warp cover the segment.
        const uint32_t per = (n + THREADS - 1) / THREADS, base = warp * per * 32u + lane;
        uint32_t key[E], pos[E], rank[E];
#pragma unroll
        for (uint32_t k = 0; k < E; k++) {
            const uint32_t i = base + k * 32u;
            pos[k] = i;
            key[k] = 0u;
            if (k < per && i < n) key[k] = morton_key(t.caabb[__ldg(list + i)], bb.x, bb.y, bb.z, bb.w);
        }
        for (uint32_t shift = 0; shift < 32; shift += 8) {
            for (uint32_t i = threadIdx.x; i < WARPS * 256; i += THREADS) hist[i] = 0u;
            __syncthreads();
            uint32_t* const mine = hist + warp * 256;
#pragma unroll
            for (uint32_t k = 0; k < E; k++) {
                if (k >= per) break;
                const bool valid = base + k * 32u < n;
                const uint32_t d = (key[k] >> shift) & 255u;
                const uint32_t peers = digit_peers(d, valid);
                const uint32_t before = __popc(peers & ltMask);
                uint32_t first = 0;
                if (valid) first = mine[d];
                __syncwarp();
                if (valid && before == 0) mine[d] = first + __popc(peers);
                __syncwarp();
                rank[k] = first + before;
            }
            __syncthreads();
            for (uint32_t d = threadIdx.x; d < 256; d += THREADS) {
                uint32_t run = 0;
#pragma unroll 8
                for (uint32_t wi = 0; wi < WARPS; wi++) {
                    const uint32_t c = hist[wi * 256 + d];
                    hist[wi * 256 + d] = run;
                    run += c;
                }
                digit[d] = run;
            }
            __syncthreads();
            if (warp == 0) {   // exclusive scan of the digit counts, eight a lane
                uint32_t local[8], sum = 0;
#pragma unroll
                for (uint32_t j = 0; j < 8; j++) { local[j] = digit[lane * 8 + j]; sum += local[j]; }
                uint32_t incl = sum;
                for (uint32_t o = 1; o < 32; o <<= 1) {
                    const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += v;
                }
                uint32_t excl = incl - sum;
#pragma unroll
                for (uint32_t j = 0; j < 8; j++) { digit[lane * 8 + j] = excl; excl += local[j]; }
            }
            __syncthreads();
#pragma unroll
            for (uint32_t k = 0; k < E; k++) {
                if (k < per && base + k * 32u < n) {
                    const uint32_t d = (key[k] >> shift) & 255u;
                    const uint32_t at = digit[d] + mine[d] + rank[k];
                    sortKey[at] = key[k];
                    sortPos[at] = uint16_t(pos[k]);
                }
            }
            __syncthreads();
            if (shift < 24) {
#pragma unroll
                for (uint32_t k = 0; k < E; k++) {
                    const uint32_t i = base + k * 32u;
                    if (k < per && i < n) { key[k] = sortKey[i]; pos[k] = sortPos[i]; }
                }
            }
        }
        // Leaves in sorted order; thread i % THREADS takes leaf i from here on.
        for (uint32_t i = threadIdx.x; i < n; i += THREADS) {
            const uint32_t k = sortKey[i], c = __ldg(list + sortPos[i]);
            t.vals[lo + i] = c;
            t.keys[lo + i] = k;
            if (t.sortedWorld) t.sortedWorld[lo + i] = w;
            t.leafAabb[lo + i] = t.caabb[c];
            if (i + 1 < n) {
                const uint32_t x = k ^ sortKey[i + 1];
                shared[i] = uint8_t(x ? __clz(x) : 32 + __clz(i ^ (i + 1)));
                met[i] = 0u;
            }
        }
        __syncthreads();
        if (n > 1) {
            float4* const meet = MEET_SHARED ? treeTile : t.meet + 2 * size_t(lo);
            // Bits shared across the ends of a leaf's stretch, one more than they are; 0 beyond the segment. The subtree
            // over [l, r] is the left child of its parent (side 0, split after r) when it shares more on its right.
            auto bits_left = [&](uint32_t l) { return l > 0 ? uint32_t(shared[l - 1]) + 1u : 0u; };
            auto bits_right = [&](uint32_t r) { return r + 1 < n ? uint32_t(shared[r]) + 1u : 0u; };
            for (uint32_t i = threadIdx.x; i < n; i += THREADS)
                meet[bits_right(i) > bits_left(i) ? 2 * i : 2 * i - 1] = t.leafAabb[lo + i];   // written by this thread
            __syncthreads();
            // One loop over this thread's leaves and their way up: a lane whose sibling carries on takes its next leaf
            // while the others of its warp climb. A subtree leaves its outer bound and the bits shared there in the
            // meeting word, so that its sibling knows the node's place from the exchange alone.
            uint32_t i = threadIdx.x, l = i, r = i, bl = 0, br = 0;
            float4 box;
            auto leaf = [&] {
                l = r = i;
                bl = bits_left(i);
                br = bits_right(i);
                box = meet[br > bl ? 2 * i : 2 * i - 1];
            };
            if (i < n) leaf();
            while (i < n) {
                const bool right = br <= bl;             // this subtree's side
                const uint32_t g = right ? l - 1 : r;
                const uint32_t word = right ? (r + 1u) | br << 24 : (l + 1u) | bl << 24;
                const uint32_t other = atomicExch(met + g, word);
                bool up = other != 0u;                   // second here
                if (up) {
                    fence_cta();
                    const float4 o = meet[right ? 2 * g : 2 * g + 1];
                    if (right) { l = (other & 0xFFFFFFu) - 1u; bl = other >> 24; }
                    else { r = (other & 0xFFFFFFu) - 1u; br = other >> 24; }
                    met[g] = l | r << 16;                // the word now holds the node's range
                    const float4 a = right ? o : box, b = right ? box : o;
                    box = make_float4(fminf(a.x, b.x), fminf(a.y, b.y), fmaxf(a.z, b.z), fmaxf(a.w, b.w));
                    up = (bl | br) != 0u;                // not the root
                    if (up) {
                        meet[br > bl ? 2 * r : 2 * l - 1] = box;
                        fence_cta();
                    }
                }
                if (!up) {
                    i += THREADS;
                    if (i < n) leaf();
                }
            }
            __syncthreads();
            for (uint32_t g = threadIdx.x; g + 1 < n; g += THREADS) {
                const uint32_t l = met[g] & 0xFFFFu, r = met[g] >> 16;
                const bool root = l == 0 && r + 1 == n;
                const uint32_t node = lo + (root ? 0u : (bits_right(r) > bits_left(l) ? r : l));
                const int left = l == g ? ~int(lo + g) : int(lo + g);
                const int right = r == g + 1 ? ~int(lo + g + 1) : int(lo + g + 1);
                const float4 a = meet[2 * g], b = meet[2 * g + 1];
                NodeRec* const rec = t.rec + node;
                rec->box[0] = a;
                rec->box[1] = b;
                rec->child = make_int2(left, right);
                rec->last = make_int2(int(lo + g), int(lo + r));
                if (t.child) t.child[node] = make_int2(left, right);
                if (t.nodeAabb)
                    t.nodeAabb[node] = make_float4(fminf(a.x, b.x), fminf(a.y, b.y), fmaxf(a.z, b.z), fmaxf(a.w, b.w));
            }
        }
        __syncthreads();   // the tile is reused by the next segment
    }
    // This launch is done only when the class before it is: what follows waits for both.
    if (threadIdx.x == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <uint32_t THREADS, uint32_t E, bool MEET_SHARED>
static cudaError_t launch_tree_class(const TreeBuild& t, uint32_t minSize, uint32_t maxSize, uint32_t sms,
                                     cudaStream_t stream, uint32_t* launches)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(std::min(t.worlds, sms * std::max(1u, 2048u / THREADS)));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = TreeSmem<THREADS, E, MEET_SHARED>::bytes(maxSize);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = *launches > 0 || t.chained ? 1 : 0;   // beside the class launched before it, or chained
    ++*launches;
    return cudaLaunchKernelEx(&cfg, k_tree_segments<THREADS, E, MEET_SHARED>, t, minSize, maxSize);
}

template <uint32_t THREADS, uint32_t E, bool MEET_SHARED>
static cudaError_t tree_class_init(uint32_t maxSize)
{
    return cudaFuncSetAttribute(k_tree_segments<THREADS, E, MEET_SHARED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                int(TreeSmem<THREADS, E, MEET_SHARED>::bytes(maxSize)));
}

cudaError_t tree_segments_init()
{
    cudaError_t e = tree_class_init<512, 4, true>(2048);
    if (e == cudaSuccess) e = tree_class_init<1024, 4, true>(4096);
    if (e == cudaSuccess) e = tree_class_init<1024, 8, false>(8192);
    if (e == cudaSuccess) e = tree_class_init<1024, 16, false>(TREE_SEGMENT_MAX);
    return e;
}

cudaError_t launch_tree_segments(const TreeBuild& t, uint32_t largest, uint32_t sms, cudaStream_t stream,
                                 uint32_t* launches)
{
    // Size classes, each with the CTA that its largest segment keeps busy: segments of a ragged batch differ by a
    // factor of a hundred, and a small one in a wide CTA waits at barriers with most warps idle. The longest run first
    // and the classes overlap. Those up to 4,096 leaves keep the meeting boxes in shared memory (32 B a leaf), the two
    // above in global memory.
    const bool one = t.segStart == nullptr;   // one segment of 'largest' leaves: its class alone
    cudaError_t e = cudaSuccess;
    *launches = 0;
    auto takes = [&](uint32_t from, uint32_t to) { return e == cudaSuccess && largest > from && (!one || largest <= to); };
    auto top = [&](uint32_t to) { return std::min(largest, to); };
    if (takes(8192, TREE_SEGMENT_MAX)) e = launch_tree_class<1024, 16, false>(t, 8192, largest, sms, stream, launches);
    if (takes(4096, 8192)) e = launch_tree_class<1024, 8, false>(t, 4096, top(8192), sms, stream, launches);
    if (takes(2048, 4096)) e = launch_tree_class<1024, 4, true>(t, 2048, top(4096), sms, stream, launches);
    if (takes(1024, 2048)) e = launch_tree_class<512, 4, true>(t, 1024, top(2048), sms, stream, launches);
    if (takes(256, 1024)) e = launch_tree_class<256, 4, true>(t, 256, top(1024), sms, stream, launches);
    if (takes(0, 256)) e = launch_tree_class<128, 2, true>(t, 0, top(256), sms, stream, launches);
    return e;
}

// Bottom-up AABB refit (BvhTree::fitNodes equivalent). The two subtrees of a node meet in its slot: each swaps its
// bounds in with one 16-byte atomic exchange; the first finds the empty marker and stops, the second receives its
// sibling's bounds in the same operation (no flag, fence or second load on the chain), writes the node's record
// and bounds and carries on upwards.
__global__ void k_lbvh_refit(int n, const int2* child, const int* parent,
                             const int* leafParent, const float4* leafAabb,
                             float4* nodeAabb, float4* meet, NodeRec* rec)
{
    chain_begin();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int node = leafParent[i];   // -1 for the leaf of a one-collider segment
        int self = ~i;              // child encoding of the subtree this thread carries up
        float4 box = leafAabb[i];   // its bounds
        while (node >= 0) {
            // The tree links do not depend on the arrival: fetch them before the atomic.
            const int2 c = child[node];
            const int up = parent[node];
            const float4 o = exchange_box(meet + node, box);
            if (__float_as_uint(o.x) == MEET_EMPTY) break;   // first arrival: the sibling carries on
            const int side = c.x == self ? 0 : 1;
            const float4 a = side == 0 ? box : o;
            const float4 b = side == 0 ? o : box;
            __stcg(&rec[node].box[0], a);
            __stcg(&rec[node].box[1], b);
            box = make_float4(fminf(a.x, b.x), fminf(a.y, b.y), fmaxf(a.z, b.z), fmaxf(a.w, b.w));
            __stcg(nodeAabb + node, box);
            self = node;
            node = up;
        }
    }
}

// ---------------------------------------------------------------------------------------------------------------
// Pair query. For dynamic collider of sorted rank i: every dynamic collider of rank > i whose AABB strictly
// overlaps (BvhNode::overlaps, BvhNode.h:33-38) and has another owner body (LeafPairTesting.h:71-134), then every
// static/sleeping collider that overlaps (cross pairs, ordered (dynamic, other)). One traversal counts each query's
// pairs and keeps the first few; after a scan of the counts they land at their offsets: a deterministic pair list
// ordered by query rank and traversal order.
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ bool strict_overlap(const float4& a, const float4& b)
{
    return a.x < b.z && a.z > b.x && a.y < b.w && a.w > b.y;
}

// All pair partners of dynamic collider rank i, in traversal order; emit(k, collider) receives the k-th. Returns the
// count.
template <class Emit>
__device__ __forceinline__ uint32_t query_one(const TreeView& dyn, const TreeView& other,
                                              const uint32_t* __restrict__ cbody, int i, uint32_t me, Emit emit,
                                              uint32_t* __restrict__ status)
{
    const int n = dyn.n;
    const float4 q = dyn.leafAabb[i];
    const uint32_t myBody = cbody[me];
    // This collider's world: the segments of both trees it is tested against.
    int dlo = 0, dhi = n, olo = 0, ohi = other.n;
    if (dyn.sortedWorld) {
        const uint32_t wd = dyn.sortedWorld[i];
        dlo = int(dyn.segStart[wd]);
        dhi = int(dyn.segStart[wd + 1]);
        if (other.n > 0) {
            olo = int(other.segStart[wd]);
            ohi = int(other.segStart[wd + 1]);
        } else {
            ohi = 0;
        }
    }
    uint32_t count = 0;
    int stack[QUERY_STACK];
    // Self pairs within the dynamic tree.
    if (dhi - dlo > 1) {
        int sp = 0;
        stack[sp++] = dlo;
        while (sp > 0) {
            const int node = stack[--sp];
            const NodeRec r = dyn.rec[node];
#pragma unroll
            for (int side = 0; side < 2; side++) {
                const int ch = side == 0 ? r.child.x : r.child.y;
                const int last = side == 0 ? r.last.x : r.last.y;
                if (last <= i || !strict_overlap(q, r.box[side])) continue;   // every leaf below ranks <= i
                if (ch < 0) {
                    const uint32_t c = dyn.vals[~ch];
                    if (cbody[c] != myBody) emit(count++, c);
                } else if (sp < QUERY_STACK) {
                    stack[sp++] = ch;
                } else {
                    atomicOr(status, STATUS_STACK_OVERFLOW);
                }
            }
        }
    }
    // Cross pairs against the static + sleeping tree.
    if (ohi - olo == 1) {
        if (strict_overlap(q, other.leafAabb[olo])) emit(count++, other.vals[olo]);
    } else if (ohi - olo > 1 && strict_overlap(q, other.nodeAabb[olo])) {
        int sp = 0;
        stack[sp++] = olo;
        while (sp > 0) {
            const int node = stack[--sp];
            const NodeRec r = other.rec[node];
#pragma unroll
            for (int side = 0; side < 2; side++) {
                const int ch = side == 0 ? r.child.x : r.child.y;
                if (!strict_overlap(q, r.box[side])) continue;
                if (ch < 0) emit(count++, other.vals[~ch]);
                else if (sp < QUERY_STACK) stack[sp++] = ch;
                else atomicOr(status, STATUS_STACK_OVERFLOW);
            }
        }
    }
    return count;
}

// The pair query in one kernel: blocks take tiles of blockDim.x queries (dynamic colliders in sorted rank order) in
// ticket order (tileState and the ticket counter zeroed before the launch; at most QUERY_MAX_THREADS threads). Each
// thread traverses once, counting its query's pairs and keeping the first QUERY_STASH in shared memory; the tile
// scans the counts, takes its output offset from the decoupled look-back over the preceding tiles and writes the
// kept pairs in place. A query with more pairs than the stash holds traverses again for the rest, after its tile
// has published its prefix. The pairs come out ordered by query rank, then traversal order; the last tile writes
// the pair count.
__global__ void __launch_bounds__(QUERY_MAX_THREADS) k_query(TreeView dyn, TreeView other,
                                                             const uint32_t* cbody,
                                                             uint2* pairs, uint32_t pairCap,
                                                             uint32_t* total,
                                                             uint32_t* status,
                                                             uint32_t* tileState,
                                                             uint32_t* tileCounter)
{
    chain_begin();
    __shared__ uint32_t kept[QUERY_STASH * QUERY_MAX_THREADS];   // [k][thread]
    __shared__ uint32_t warpBase[QUERY_MAX_THREADS / 32];
    __shared__ uint32_t tileSlot, tileBase;
    const uint32_t n = uint32_t(dyn.n);
    const uint32_t tiles = (n + blockDim.x - 1) / blockDim.x;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nWarps = blockDim.x >> 5;
    while (true) {
        if (threadIdx.x == 0) tileSlot = atomicAdd(tileCounter, 1u);
        __syncthreads();
        const uint32_t tile = tileSlot;
        if (tile >= tiles) return;
        const uint32_t i = tile * blockDim.x + threadIdx.x;
        uint32_t count = 0;
        const uint32_t me = i < n ? dyn.vals[i] : 0u;
        if (i < n)
            count = query_one(dyn, other, cbody, int(i), me, [&](uint32_t k, uint32_t c) {
                if (k < QUERY_STASH) kept[k * blockDim.x + threadIdx.x] = c;
            }, status);
        // Block scan of the counts: lane prefix within the warp, then the warps' totals.
        uint32_t incl = count;
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) warpBase[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            const uint32_t c = lane < nWarps ? warpBase[lane] : 0u;
            uint32_t wi = c;
            for (uint32_t o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(0xffffffffu, wi, o);
                if (lane >= o) wi += t;
            }
            const uint32_t aggregate = __shfl_sync(0xffffffffu, wi, 31);
            if (lane < nWarps) warpBase[lane] = wi - c;
            volatile uint32_t* state = tileState;
            uint32_t prefix = 0;
            if (tile == 0) {
                if (lane == 0) state[0] = (2u << 30) | aggregate;
            } else {
                if (lane == 0) state[tile] = (1u << 30) | aggregate;
                prefix = scan_lookback(tile, tileState, status);
                if (lane == 0) state[tile] = (2u << 30) | (prefix + aggregate);
            }
            if (lane == 0) {
                tileBase = prefix;
                if (tile == tiles - 1) {
                    *total = prefix + aggregate;
                    if (prefix + aggregate > pairCap) atomicOr(status, STATUS_PAIR_OVERFLOW);
                }
            }
        }
        __syncthreads();
        const uint32_t out = tileBase + warpBase[warp] + incl - count;
        const uint32_t keptCount = min(count, QUERY_STASH);
        for (uint32_t k = 0; k < keptCount; k++)
            if (out + k < pairCap) pairs[out + k] = make_uint2(me, kept[k * blockDim.x + threadIdx.x]);
        if (count > QUERY_STASH)
            query_one(dyn, other, cbody, int(i), me, [&](uint32_t k, uint32_t c) {
                if (k >= QUERY_STASH && out + k < pairCap) pairs[out + k] = make_uint2(me, c);
            }, status);
        __syncthreads();   // tileSlot, tileBase, warpBase and the stash are reused by the next tile
    }
}

// ---------------------------------------------------------------------------------------------------------------
// Continuous collision (ContinuousCollisionDetector::processShapeRange / resolve, ContinuousCollisionDetector.cpp:
// 303-531). Per dynamic collider: skip unless both the body and the collider moved more than fastFactor x min
// extent this step; sweep the core circle's AABB through the static colliders of its world's static + sleeping
// tree (sleeping ones are skipped: the reference sweeps the static tree only); keep the earliest time of impact per
// body. 'prevPos' holds each body's (x, y) and 'prevPose' each collider's world pose from before integration.
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ float ccd_cast_core(const DeviceWorld& w, uint32_t c, V2 start, V2 d, float dd,
                                               float coreRadius, float best)
{
    const float4 pose = w.cpose[c];
    const float cs = pose.z, sn = pose.w;
    const float rx = start.x - pose.x, ry = start.y - pose.y;
    const V2 q0 = v2(cs * rx + sn * ry, cs * ry - sn * rx);
    const V2 dl = v2(cs * d.x + sn * d.y, cs * d.y - sn * d.x);
    const uint32_t packed = w.cshape[c];
    const uint32_t si = shape_index(packed);
    switch (shape_type(packed)) {
    case SHAPE_CIRCLE: return ccd_cast_circle(q0.x, q0.y, dl.x, dl.y, dd, w.circleRadius[si] + coreRadius, best);
    case SHAPE_BOX: {
        const float2 h = w.boxHalf[si];
        return ccd_cast_box(q0, dl, dd, h.x, h.y, coreRadius, best);
    }
    case SHAPE_CAPSULE: {
        const float2 h = w.boxHalf[si];
        return ccd_cast_capsule(q0, dl, dd, h.x, h.y, coreRadius, best);
    }
    default: {
        const uint32_t off = w.polyOffset[si];
        return ccd_cast_polygon(q0, dl, dd, w.polyVerts + off, w.polyNormals + off, w.polyCount[si], coreRadius, best);
    }
    }
}

__global__ void k_ccd_sweep(DeviceWorld w, const uint32_t* __restrict__ dynCol, uint32_t n, TreeView other,
                            const float4* __restrict__ prevPos, const float4* __restrict__ prevPose,
                            const float* __restrict__ minExtent, uint32_t* __restrict__ hitTime,
                            uint32_t* __restrict__ status)
{
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const uint32_t c = dynCol[k];
        const uint32_t body = w.cbody[c];
        const float4 com = w.bpos[body], pcom = prevPos[body];
        const float bodyDx = com.x - pcom.x, bodyDy = com.y - pcom.y;
        const float bodyDeltaSq = bodyDx * bodyDx + bodyDy * bodyDy;
        if (bodyDeltaSq <= CCD_MIN_DISPLACEMENT_SQ) continue;
        const float me = minExtent[c];
        if (me <= 0.0f) continue;
        const float threshold = CCD_FAST_FACTOR * me;
        const float thresholdSq = threshold * threshold;
        if (bodyDeltaSq <= thresholdSq) continue;
        const float4 pp = prevPose[c], cp = w.cpose[c];
        const V2 start = v2(pp.x, pp.y), end = v2(cp.x, cp.y);
        const V2 d = end - start;
        const float dd = dot(d, d);
        if (dd <= thresholdSq) continue;
        const float coreRadius = CCD_CORE_FRACTION * me;
        const float4 sweep = make_float4(rfminf(start.x, end.x) - coreRadius, rfminf(start.y, end.y) - coreRadius,
                                         rfmaxf(start.x, end.x) + coreRadius, rfmaxf(start.y, end.y) + coreRadius);
        // This collider's world segment of the static + sleeping tree.
        int lo = 0, hi = other.n;
        if (other.segStart) {
            const uint32_t wd = w.colWorld[c];
            lo = int(other.segStart[wd]);
            hi = int(other.segStart[wd + 1]);
        }
        float best = 1.0f;
        auto leaf = [&](int j) {
            const float4 b = other.leafAabb[j];
            if (!(sweep.x < b.z && sweep.z > b.x && sweep.y < b.w && sweep.w > b.y)) return;
            const uint32_t sc = other.vals[j];
            if (w.bstate[w.cbody[sc]] != STATE_STATIC) return;
            best = rfminf(best, ccd_cast_core(w, sc, start, d, dd, coreRadius, best));
        };
        if (hi - lo == 1) {
            leaf(lo);
        } else if (hi - lo > 1) {
            int stack[QUERY_STACK];
            int sp = 0;
            stack[sp++] = lo;
            while (sp > 0) {
                const int node = stack[--sp];
                const float4 nb = other.nodeAabb[node];
                if (nb.z < sweep.x || nb.x > sweep.z || nb.w < sweep.y || nb.y > sweep.w) continue;
                const int2 ch = other.child[node];
#pragma unroll
                for (int side = 0; side < 2; side++) {
                    const int x = side == 0 ? ch.x : ch.y;
                    if (x < 0) leaf(~x);
                    else if (sp < QUERY_STACK) stack[sp++] = x;
                    else atomicOr(status, STATUS_STACK_OVERFLOW);
                }
            }
        }
        if (best < 1.0f) atomicMin(hitTime + body, float_to_ordered(best));
    }
}

// Colliders of hit bodies move back with their body (worldPos += shift) and get their AABB rebuilt from the moved
// pose (resolve, ContinuousCollisionDetector.cpp:495-512, then buildColliderAABBs). Runs before the bodies move.
__global__ void k_ccd_shift_colliders(DeviceWorld w, const uint32_t* __restrict__ dynCol, uint32_t n,
                                      const float4* __restrict__ prevPos, const uint32_t* __restrict__ hitTime)
{
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const uint32_t c = dynCol[k];
        const uint32_t body = w.cbody[c];
        const float t = ordered_to_float(hitTime[body]);
        if (!(t < 1.0f)) continue;
        const float back = t - 1.0f;
        const float4 com = w.bpos[body], pcom = prevPos[body];
        const float shiftX = (com.x - pcom.x) * back, shiftY = (com.y - pcom.y) * back;
        float4 p = w.cpose[c];
        p.x += shiftX;
        p.y += shiftY;
        w.cpose[c] = p;
        w.caabb[c] = collider_aabb(w, c, p.x, p.y, p.z, p.w);
    }
}

// Hit bodies move back along their displacement to the time of impact; the hit time returns to 1.
__global__ void k_ccd_shift_bodies(DeviceWorld w, const uint32_t* __restrict__ dynBody, uint32_t n,
                                   const float4* __restrict__ prevPos, uint32_t* __restrict__ hitTime,
                                   StepCounters* counters)
{
    uint32_t moved = 0;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const uint32_t body = dynBody[k];
        const float t = ordered_to_float(hitTime[body]);
        if (!(t < 1.0f)) continue;
        const float back = t - 1.0f;
        float4 com = w.bpos[body];
        const float4 pcom = prevPos[body];
        const float shiftX = (com.x - pcom.x) * back, shiftY = (com.y - pcom.y) * back;
        com.x += shiftX;
        com.y += shiftY;
        w.bpos[body] = com;
        hitTime[body] = float_to_ordered(1.0f);
        moved++;
    }
    for (int o = 16; o > 0; o >>= 1) moved += __shfl_xor_sync(0xffffffffu, moved, o);
    if ((threadIdx.x & 31) == 0 && moved) atomicAdd(&counters->ccdHits, moved);
}

// ---------------------------------------------------------------------------------------------------------------
// Exclusive scan of uint32 (reduce-then-scan, 2048 elements per block); used for pair offsets, compaction and
// work lists.
// ---------------------------------------------------------------------------------------------------------------
// ---------------------------------------------------------------------------------------------------------------
// Single-pass exclusive scan (decoupled look-back, scan_lookback). Tiles of SCAN_TILE elements are taken in ticket
// order by a grid of persistent blocks. tileState and the ticket counter are zeroed before the launch.
// ---------------------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(SCAN_THREADS) k_scan(const uint32_t* __restrict__ in, uint32_t* __restrict__ out,
                                                       uint32_t n, const uint32_t* __restrict__ nDev,
                                                       uint32_t* __restrict__ total, uint32_t* __restrict__ tileState,
                                                       uint32_t* __restrict__ tileCounter, uint32_t* __restrict__ status)
{
    __shared__ uint32_t warpSums[SCAN_THREADS / 32];
    __shared__ uint32_t tileSlot, tilePrefix;
    if (nDev) n = min(n, *nDev);
    const uint32_t tiles = (n + SCAN_TILE - 1) / SCAN_TILE;
    if (n == 0) {
        if (blockIdx.x == 0 && threadIdx.x == 0 && total) *total = 0u;
        return;
    }
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    while (true) {
        if (threadIdx.x == 0) tileSlot = atomicAdd(tileCounter, 1u);
        __syncthreads();
        const uint32_t tile = tileSlot;
        if (tile >= tiles) return;
        const uint32_t base = tile * SCAN_TILE + threadIdx.x * SCAN_ITEMS;
        uint32_t v[SCAN_ITEMS];
        uint32_t sum = 0;
#pragma unroll
        for (uint32_t j = 0; j < SCAN_ITEMS; j++) { v[j] = base + j < n ? in[base + j] : 0u; sum += v[j]; }
        uint32_t incl = sum;
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) warpSums[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            const uint32_t ws = lane < SCAN_THREADS / 32 ? warpSums[lane] : 0u;
            uint32_t wi = ws;
            for (uint32_t o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(0xffffffffu, wi, o);
                if (lane >= o) wi += t;
            }
            const uint32_t aggregate = __shfl_sync(0xffffffffu, wi, SCAN_THREADS / 32 - 1);
            if (lane < SCAN_THREADS / 32) warpSums[lane] = wi - ws;
            volatile uint32_t* state = tileState;
            uint32_t prefix = 0;
            if (tile == 0) {
                if (lane == 0) state[0] = (2u << 30) | aggregate;
            } else {
                if (lane == 0) state[tile] = (1u << 30) | aggregate;
                prefix = scan_lookback(tile, tileState, status);
                if (lane == 0) state[tile] = (2u << 30) | (prefix + aggregate);
            }
            if (lane == 0) {
                tilePrefix = prefix;
                if (total && tile == tiles - 1) *total = prefix + aggregate;
            }
        }
        __syncthreads();
        uint32_t run = tilePrefix + warpSums[warp] + incl - sum;
#pragma unroll
        for (uint32_t j = 0; j < SCAN_ITEMS; j++) {
            if (base + j < n) out[base + j] = run;
            run += v[j];
        }
        __syncthreads();   // tileSlot and warpSums are reused by the next tile
    }
}

}  // namespace ag2d
