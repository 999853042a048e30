// Graph colouring + sequential-impulse solver as one device routine over a "team" of threads that share a barrier:
// one CTA (batched small worlds, single worlds of a few thousand bodies) or a cooperative grid (larger single worlds,
// whose passes then run as a dataflow without barriers). The per-constraint arithmetic (prep/warm/velocity/position)
// below is shared by every variant.
#pragma once

#include "ag2d_kernels.cuh"

namespace ag2d {

// ---------------------------------------------------------------------------------------------------------------
// Sequential-impulse solver (Solving/BodyCollisionSolver.cpp): computeConstraintData (:229-390), applyWarmStarting
// (:416-490), solveVelocityConstraints (:492-928; one-contact path, two-contact 2x2 block LCP with iterative
// fallback, iterative friction), solvePositionConstraints (:930-980), scatterImpulses (:392-414). A team runs every
// pass colour by colour with its barrier between colours.
// ---------------------------------------------------------------------------------------------------------------
// Body state seen by the solver, with the colouring words of each body (the round's highest priority and the mask of
// colours taken around the body): global memory indexed by body, or a team's contiguous body range staged in shared
// memory.
struct GlobalBodies {
    float4* vel;
    float4* pos;
    unsigned long long* maxW;    // [bodies], zeroed before the call
    unsigned long long* maskW;   // [bodies], zeroed before the call
    __device__ __forceinline__ float4 v(uint32_t b) const { return vel[b]; }
    __device__ __forceinline__ float4 p(uint32_t b) const { return pos[b]; }
    __device__ __forceinline__ void setV(uint32_t b, const float4& x) const { vel[b] = x; }
    __device__ __forceinline__ void setP(uint32_t b, const float4& x) const { pos[b] = x; }
    __device__ __forceinline__ float invMass(uint32_t b) const { return __ldcg(&vel[b].w); }
    __device__ __forceinline__ unsigned long long* maxWord(uint32_t b) const { return maxW + b; }
    __device__ __forceinline__ unsigned long long* maskWord(uint32_t b) const { return maskW + b; }
    static __device__ __forceinline__ unsigned long long ldWord(const unsigned long long* p) { return __ldcg(p); }
    __device__ __forceinline__ bool stage(uint32_t, uint32_t) const { return false; }
};
// Bodies [base, base + count) in shared memory. With 'lazy' set the colouring words occupy the front of the body
// cache while the team colours (inverse masses then come from global memory), and stage() loads the velocities and
// poses over them once the colours are known: 32 bytes of shared memory a body instead of 48, so more teams fit on
// an SM. Otherwise the team loaded the bodies before colouring and the words have a region of their own.
struct SharedBodies {
    float4* vel;                 // shared: bodies [base, base + count)
    float4* pos;
    unsigned long long* maxW;    // shared, zeroed by the team before colouring
    unsigned long long* maskW;
    uint32_t base;
    uint32_t count = 0;
    const float4* gvel = nullptr;   // lazy: the global velocities (inverse masses while colouring)
    const float4* gpos = nullptr;
    __device__ __forceinline__ float4 v(uint32_t b) const { return vel[b - base]; }
    __device__ __forceinline__ float4 p(uint32_t b) const { return pos[b - base]; }
    __device__ __forceinline__ void setV(uint32_t b, const float4& x) const { vel[b - base] = x; }
    __device__ __forceinline__ void setP(uint32_t b, const float4& x) const { pos[b - base] = x; }
    __device__ __forceinline__ float invMass(uint32_t b) const
    {
        return gvel ? gvel[b].w : vel[b - base].w;
    }
    // Loads the body cache over the colouring words (lazy only); the caller synchronises the team after it.
    __device__ __forceinline__ bool stage(uint32_t rank, uint32_t size) const
    {
        if (!gvel) return false;
        for (uint32_t i = rank; i < count; i += size) {
            vel[i] = gvel[base + i];
            pos[i] = gpos[base + i];
        }
        return true;
    }
    __device__ __forceinline__ unsigned long long* maxWord(uint32_t b) const { return maxW + (b - base); }
    __device__ __forceinline__ unsigned long long* maskWord(uint32_t b) const { return maskW + (b - base); }
    static __device__ __forceinline__ unsigned long long ldWord(const unsigned long long* p)
    {
        return *static_cast<const volatile unsigned long long*>(p);
    }
};

template <class Bodies>
__device__ __forceinline__ void prep_constraint(const DeviceWorld& w, const Bodies& B, const Manifold& m, uint32_t mi,
                                                Constraint& k)
{
    const uint32_t bA = w.cbody[m.a], bB = w.cbody[m.b];
    const float4 vA = B.v(bA), vB = B.v(bB), pA = B.p(bA), pB = B.p(bB);
    k.bodyA = bA; k.bodyB = bB; k.count = m.count; k.manifold = mi;
    k.nx = m.nx; k.ny = m.ny;
    k.imA = vA.w; k.imB = vB.w; k.iIA = pA.w; k.iIB = pB.w;
    k.jn0 = m.jn0; k.jt0 = m.jt0; k.jn1 = m.jn1; k.jt1 = m.jt1;
    k.penBase = m.depth + ((pB.x - pA.x) * m.nx + (pB.y - pA.y) * m.ny) - 0.001f;
    const float4 matA = w.materials[w.cmat[m.a]], matB = w.materials[w.cmat[m.b]];
    const float e = (matA.x + matB.x) * 0.5f;
    k.sf = sqrtf(rfmaxf(0.0f, matA.y * matB.y));
    k.df = sqrtf(rfmaxf(0.0f, matA.z * matB.z));
    const float effMass = k.imA + k.imB;
    const float tx = -m.ny, ty = m.nx;
    float rAn[2] = {0, 0}, rBn[2] = {0, 0}, rAt[2] = {0, 0}, rBt[2] = {0, 0}, nm[2] = {0, 0}, tm[2] = {0, 0}, bias[2] = {0, 0};
#pragma unroll
    for (uint32_t i = 0; i < 2; i++) {
        if (i >= m.count) break;
        const float px = i == 0 ? m.px0 : m.px1, py = i == 0 ? m.py0 : m.py1;
        const float rAx = px - pA.x, rAy = py - pA.y, rBx = px - pB.x, rBy = py - pB.y;
        rAn[i] = (-rAy) * m.nx + rAx * m.ny;
        rBn[i] = (-rBy) * m.nx + rBx * m.ny;
        rAt[i] = (-rAy) * tx + rAx * ty;
        rBt[i] = (-rBy) * tx + rBx * ty;
        const float nd = effMass + rAn[i] * rAn[i] * k.iIA + rBn[i] * rBn[i] * k.iIB;
        nm[i] = nd > 0.0f ? 1.0f / nd : 0.0f;
        const float td = effMass + rAt[i] * rAt[i] * k.iIA + rBt[i] * rBt[i] * k.iIB;
        tm[i] = td > 0.0f ? 1.0f / td : 0.0f;
        const float negVn = -(((vB.x - vA.x) * m.nx + (vB.y - vA.y) * m.ny) + rBn[i] * vB.z - rAn[i] * vA.z);
        bias[i] = (negVn > 0.0f) ? e * negVn : 0.0f;
    }
    k.rAn0 = rAn[0]; k.rBn0 = rBn[0]; k.rAt0 = rAt[0]; k.rBt0 = rBt[0]; k.nm0 = nm[0]; k.tm0 = tm[0]; k.bias0 = bias[0];
    k.rAn1 = rAn[1]; k.rBn1 = rBn[1]; k.rAt1 = rAt[1]; k.rBt1 = rBt[1]; k.nm1 = nm[1]; k.tm1 = tm[1]; k.bias1 = bias[1];
    k.pad = 0.0f;
}

// Impact impulse of a manifold for collision events (BodyCollisionSolver.cpp:320-350): the largest over its points
// of the approach speed along the normal times the normal effective mass, from the velocities the constraint data
// is built from. The arithmetic is prep_constraint's (rAn, rBn, the normal mass and negVn, in the same order), so
// the value is the one the reference computes beside its constraint data.
__device__ __forceinline__ float impact_impulse(const Manifold& m, float4 vA, float4 vB, float4 pA, float4 pB)
{
    const float effMass = vA.w + vB.w;
    float impact = 0.0f;
#pragma unroll
    for (uint32_t i = 0; i < 2; i++) {
        if (i >= m.count) break;
        const float px = i == 0 ? m.px0 : m.px1, py = i == 0 ? m.py0 : m.py1;
        const float rAx = px - pA.x, rAy = py - pA.y, rBx = px - pB.x, rBy = py - pB.y;
        const float rAn = (-rAy) * m.nx + rAx * m.ny;
        const float rBn = (-rBy) * m.nx + rBx * m.ny;
        const float nd = effMass + rAn * rAn * pA.w + rBn * rBn * pB.w;
        const float nm = nd > 0.0f ? 1.0f / nd : 0.0f;
        const float negVn = -(((vB.x - vA.x) * m.nx + (vB.y - vA.y) * m.ny) + rBn * vB.z - rAn * vA.z);
        impact = rfmaxf(impact, negVn * nm);   // std::fmax: a NaN product leaves the running value
    }
    return impact;
}

// The warm start of one constraint on its two bodies' velocities held in registers.
__device__ __forceinline__ void warm_solve(const Constraint& k, float4& vA, float4& vB)
{
    const float tx = -k.ny, ty = k.nx;
    const float jn0 = k.count > 0 ? k.jn0 : 0.0f, jt0 = k.count > 0 ? k.jt0 : 0.0f;
    const float jn1 = k.count > 1 ? k.jn1 : 0.0f, jt1 = k.count > 1 ? k.jt1 : 0.0f;
    const float sn = jn0 + jn1, st = jt0 + jt1;
    const float ix = sn * k.nx + st * tx, iy = sn * k.ny + st * ty;
    vA.x = vA.x - ix * k.imA; vA.y = vA.y - iy * k.imA;
    vB.x = vB.x + ix * k.imB; vB.y = vB.y + iy * k.imB;
    vA.z = vA.z - (jn0 * k.rAn0 + jt0 * k.rAt0 + jn1 * k.rAn1 + jt1 * k.rAt1) * k.iIA;
    vB.z = vB.z + (jn0 * k.rBn0 + jt0 * k.rBt0 + jn1 * k.rBn1 + jt1 * k.rBt1) * k.iIB;
}

template <class Bodies>
__device__ __forceinline__ void warm_constraint(const Bodies& B, const Constraint& k)
{
    float4 vA = B.v(k.bodyA), vB = B.v(k.bodyB);
    warm_solve(k, vA, vB);
    if (k.imA > 0.0f) B.setV(k.bodyA, vA);
    if (k.imB > 0.0f) B.setV(k.bodyB, vB);
}

// What the block solve of a two-point contact takes from its record alone, the same in every iteration: the 2x2
// matrix and the reciprocal of its determinant, negative where the matrix is too ill-conditioned to use it.
struct BlockMatrix {
    float K00, K01, K11, invDet;
};
__device__ __forceinline__ BlockMatrix block_matrix(const Constraint& k)
{
    BlockMatrix b;
    const float effMass = k.imA + k.imB;
    b.K00 = effMass + k.rAn0 * k.rAn0 * k.iIA + k.rBn0 * k.rBn0 * k.iIB;
    b.K11 = effMass + k.rAn1 * k.rAn1 * k.iIA + k.rBn1 * k.rBn1 * k.iIB;
    b.K01 = effMass + k.rAn0 * k.rAn1 * k.iIA + k.rBn0 * k.rBn1 * k.iIB;
    const float det = b.K00 * b.K11 - b.K01 * b.K01;
    const float maxK = rfmaxf(b.K00, b.K11);
    b.invDet = maxK * maxK < 1000.0f * det ? 1.0f / det : -1.0f;
    return b;
}

// One velocity iteration of one constraint on its two bodies' velocities held in registers.
__device__ __forceinline__ void velocity_solve(Constraint& k, const BlockMatrix& bm, float4& vA, float4& vB)
{
    const float imA = k.imA, imB = k.imB, iIA = k.iIA, iIB = k.iIB;
    const float nx = k.nx, ny = k.ny, tx = -ny, ty = nx;
    if (k.count == 1) {
        float jnSingle = 0.0f;
        {
            const float vn = ((vB.x - vA.x) * nx + (vB.y - vA.y) * ny) + k.rBn0 * vB.z - k.rAn0 * vA.z;
            if (!(vn > 0.0f && k.jn0 == 0.0f)) {
                const float jn = (k.bias0 - vn) * k.nm0;
                const float old = k.jn0;
                k.jn0 = rfmaxf(0.0f, old + jn);
                const float dj = k.jn0 - old;
                jnSingle = k.jn0;
                const float ix = dj * nx, iy = dj * ny;
                vA.x = vA.x - ix * imA; vA.y = vA.y - iy * imA;
                vA.z = vA.z - dj * k.rAn0 * iIA;
                vB.x = vB.x + ix * imB; vB.y = vB.y + iy * imB;
                vB.z = vB.z + dj * k.rBn0 * iIB;
            }
        }
        {
            const float slip = ((vB.x - vA.x) * tx + (vB.y - vA.y) * ty) + k.rBt0 * vB.z - k.rAt0 * vA.z;
            const float jt = -slip * k.tm0;
            const float old = k.jt0;
            const float target = old + jt;
            if (fabsf(target) <= jnSingle * k.sf) k.jt0 = target;
            else { const float maxD = jnSingle * k.df; k.jt0 = glm_clamp(target, -maxD, maxD); }
            const float dj = k.jt0 - old;
            const float ix = dj * tx, iy = dj * ty;
            vA.x = vA.x - ix * imA; vA.y = vA.y - iy * imA;
            vA.z = vA.z - dj * k.rAt0 * iIA;
            vB.x = vB.x + ix * imB; vB.y = vB.y + iy * imB;
            vB.z = vB.z + dj * k.rBt0 * iIB;
        }
    } else {
        float jnArr0 = 0.0f, jnArr1 = 0.0f;
        bool ok = false;
        {
            const float dvn = (vB.x - vA.x) * nx + (vB.y - vA.y) * ny;
            const float vn0 = dvn + k.rBn0 * vB.z - k.rAn0 * vA.z;
            const float vn1 = dvn + k.rBn1 * vB.z - k.rAn1 * vA.z;
            const float a0 = k.jn0, a1 = k.jn1;
            const float K00 = bm.K00, K11 = bm.K11, K01 = bm.K01;
            const float b0 = k.bias0 - vn0 + K00 * a0 + K01 * a1;
            const float b1 = k.bias1 - vn1 + K01 * a0 + K11 * a1;
            const float EPS = 1e-6f;
            float x0 = 0.0f, x1 = 0.0f;
            if (bm.invDet >= 0.0f) {
                const float invDet = bm.invDet;
                const float s0 = (K11 * b0 - K01 * b1) * invDet;
                const float s1 = (K00 * b1 - K01 * b0) * invDet;
                if (s0 >= -EPS && s1 >= -EPS) { x0 = rfmaxf(s0, 0.0f); x1 = rfmaxf(s1, 0.0f); ok = true; }
            }
            if (!ok && K11 > 0.0f) {
                const float s1 = b1 / K11;
                if (s1 >= -EPS && (K01 * s1 - b0) >= -EPS) { x0 = 0.0f; x1 = rfmaxf(s1, 0.0f); ok = true; }
            }
            if (!ok && K00 > 0.0f) {
                const float s0 = b0 / K00;
                if (s0 >= -EPS && (K01 * s0 - b1) >= -EPS) { x0 = rfmaxf(s0, 0.0f); x1 = 0.0f; ok = true; }
            }
            if (!ok && b0 <= EPS && b1 <= EPS) { x0 = 0.0f; x1 = 0.0f; ok = true; }
            if (ok) {
                const float d0 = x0 - a0, d1 = x1 - a1;
                k.jn0 = x0; k.jn1 = x1;
                jnArr0 = x0; jnArr1 = x1;
                const float sum = d0 + d1;
                const float sA = sum * imA, sB = sum * imB;
                vA.x = vA.x - nx * sA; vA.y = vA.y - ny * sA;
                vB.x = vB.x + nx * sB; vB.y = vB.y + ny * sB;
                vA.z = vA.z - (d0 * k.rAn0 + d1 * k.rAn1) * iIA;
                vB.z = vB.z + (d0 * k.rBn0 + d1 * k.rBn1) * iIB;
            }
        }
        if (!ok) {
#pragma unroll
            for (uint32_t i = 0; i < 2; i++) {
                const float rAn = i == 0 ? k.rAn0 : k.rAn1, rBn = i == 0 ? k.rBn0 : k.rBn1;
                const float bias = i == 0 ? k.bias0 : k.bias1, nmass = i == 0 ? k.nm0 : k.nm1;
                const float vn = ((vB.x - vA.x) * nx + (vB.y - vA.y) * ny) + rBn * vB.z - rAn * vA.z;
                const float jn = (bias - vn) * nmass;
                const float old = i == 0 ? k.jn0 : k.jn1;
                const float acc = rfmaxf(0.0f, old + jn);
                if (i == 0) { k.jn0 = acc; jnArr0 = acc; } else { k.jn1 = acc; jnArr1 = acc; }
                const float dj = acc - old;
                const float ix = dj * nx, iy = dj * ny;
                vA.x = vA.x - ix * imA; vA.y = vA.y - iy * imA;
                vA.z = vA.z - dj * rAn * iIA;
                vB.x = vB.x + ix * imB; vB.y = vB.y + iy * imB;
                vB.z = vB.z + dj * rBn * iIB;
            }
        }
#pragma unroll
        for (uint32_t i = 0; i < 2; i++) {
            const float rAt = i == 0 ? k.rAt0 : k.rAt1, rBt = i == 0 ? k.rBt0 : k.rBt1;
            const float tmass = i == 0 ? k.tm0 : k.tm1;
            const float slip = ((vB.x - vA.x) * tx + (vB.y - vA.y) * ty) + rBt * vB.z - rAt * vA.z;
            const float jt = -slip * tmass;
            const float old = i == 0 ? k.jt0 : k.jt1;
            const float target = old + jt;
            const float jn = i == 0 ? jnArr0 : jnArr1;
            float acc;
            if (fabsf(target) <= jn * k.sf) acc = target;
            else { const float maxD = jn * k.df; acc = glm_clamp(target, -maxD, maxD); }
            if (i == 0) k.jt0 = acc; else k.jt1 = acc;
            const float dj = acc - old;
            const float ix = dj * tx, iy = dj * ty;
            vA.x = vA.x - ix * imA; vA.y = vA.y - iy * imA;
            vA.z = vA.z - dj * rAt * iIA;
            vB.x = vB.x + ix * imB; vB.y = vB.y + iy * imB;
            vB.z = vB.z + dj * rBt * iIB;
        }
    }
}

template <class Bodies>
__device__ __forceinline__ void velocity_constraint(const Bodies& B, Constraint& k, const BlockMatrix& bm)
{
    float4 vA = B.v(k.bodyA), vB = B.v(k.bodyB);
    velocity_solve(k, bm, vA, vB);
    if (k.imA > 0.0f) B.setV(k.bodyA, vA);
    if (k.imB > 0.0f) B.setV(k.bodyB, vB);
}

// One position step of one constraint on its two bodies' poses held in registers; false when it moves nothing.
__device__ __forceinline__ bool position_solve(const Constraint& k, float4& pA, float4& pB)
{
    const float pen = k.penBase - ((pB.x - pA.x) * k.nx + (pB.y - pA.y) * k.ny);
    if (pen <= 0.0f) return false;
    const float imA = k.imA, imB = k.imB;
    const float total = pen / (imA + imB) * 0.5f;
    const float cA = imA * total, cB = imB * total;
    const float cAx = k.nx * cA, cAy = k.ny * cA, cBx = k.nx * cB, cBy = k.ny * cB;
    if (imA > 0.0f) { pA.x = pA.x - cAx; pA.y = pA.y - cAy; }
    if (imB > 0.0f) { pB.x = pB.x + cBx; pB.y = pB.y + cBy; }
    return true;
}

template <class Bodies>
__device__ __forceinline__ void position_constraint(const Bodies& B, const Constraint& k)
{
    float4 pA = B.p(k.bodyA), pB = B.p(k.bodyB);
    if (!position_solve(k, pA, pB)) return;
    if (k.imA > 0.0f) B.setP(k.bodyA, pA);
    if (k.imB > 0.0f) B.setP(k.bodyB, pB);
}

__device__ __forceinline__ uint32_t priority_hash(uint32_t x)
{
    x ^= x >> 16; x *= 0x85ebca6bu; x ^= x >> 13; x *= 0xc2b2ae35u; x ^= x >> 16;   // murmur3 finalizer (bijective)
    return x;
}

// Colour word of a manifold: colour in the low bits, steps it has kept that colour in the high byte.
constexpr uint32_t COLOR_AGE_SHIFT = 24;
constexpr uint32_t COLOR_MASK = (1u << COLOR_AGE_SHIFT) - 1u;
constexpr uint32_t COLOR_KEEP_STEPS = 16;

// Colour counters: one per colour, then whether kept colours clash, the lengths of the two uncoloured lists and the
// colour count, then a second counter per colour (one-point contacts placed from the colour's end).
constexpr uint32_t COLOR_SLOTS = 2 * MAX_COLORS + 4;
// Colours 0..63 are chosen first-fit from a body's 64-bit mask of neighbouring colours; a manifold whose bodies see
// all 64 taken gets colour 64 + its round (unique to the round, so still conflict-free). What is left after the last
// round (a body with more contacts than that, a ground that was given a mass) is the tail, the last colour: its manifolds
// may share bodies and are solved one after the other in list order.
constexpr uint32_t TAIL_COLOR = MAX_COLORS - 1;
constexpr uint32_t MAX_ROUNDS = TAIL_COLOR - 64;
constexpr uint32_t TAIL_MAX = 16384;   // manifolds of a tail; more: STATUS_COLOR_OVERFLOW
constexpr uint32_t ONE_BLOCK_ROUND = 4096;   // uncoloured manifolds that one block of a grid finishes

// Solver records in global memory, structure of arrays: field f of record c at q[f * stride + c], so that a warp that
// takes 32 consecutive records reads every field as four full lines. (As 128-byte structures a lane apart, each
// 16-byte load of a warp touched 32 lines, and the load unit, not latency or bandwidth, bounded every pass: one CTA on
// 3,265 manifolds took 4.5 us a colour.) A record with one contact point leaves out fields 5 to 7.
struct ConsRecords {
    float4* q;
    float* pen;        // penetration base
    uint32_t stride;
    static constexpr uint32_t FIELDS = 8;
    __device__ __forceinline__ ConsRecords from(uint32_t c) const { return ConsRecords{q + c, pen + c, stride}; }
    __device__ __forceinline__ void store(uint32_t c, const Constraint& k) const
    {
        float4* r = q + c;
        const size_t st = stride;
        r[0] = make_float4(__uint_as_float(k.bodyA | min(k.count, 3u) << 30), __uint_as_float(k.bodyB), k.nx, k.ny);
        r[st] = make_float4(k.imA, k.imB, k.iIA, k.iIB);
        r[2 * st] = make_float4(k.jn0, k.jt0, k.sf, k.df);
        r[3 * st] = make_float4(k.rAn0, k.rBn0, k.rAt0, k.rBt0);
        r[4 * st] = make_float4(k.nm0, k.tm0, k.bias0, k.bias1);
        if (k.count != 1u) {
            r[5 * st] = make_float4(k.jn1, k.jt1, k.nm1, k.tm1);
            r[6 * st] = make_float4(k.rAn1, k.rBn1, k.rAt1, k.rBt1);
            const BlockMatrix b = block_matrix(k);
            r[7 * st] = make_float4(b.K00, b.K01, b.K11, b.invDet);
        }
        pen[c] = k.penBase;
    }
    // The fields a position step reads: bodies, count, normal, masses, penetration base.
    __device__ __forceinline__ void loadHead(uint32_t c, Constraint& k) const
    {
        const float4 h = q[c], ms = q[size_t(stride) + c];
        k.bodyA = __float_as_uint(h.x) & 0x3FFFFFFFu;
        k.count = __float_as_uint(h.x) >> 30;
        k.bodyB = __float_as_uint(h.y);
        k.nx = h.z; k.ny = h.w;
        k.imA = ms.x; k.imB = ms.y; k.iIA = ms.z; k.iIB = ms.w;
    }
    __device__ __forceinline__ void load(uint32_t c, uint32_t kind, Constraint& k, BlockMatrix& bm) const;
    __device__ __forceinline__ void storeImpulses(uint32_t c, const Constraint& k) const
    {
        *reinterpret_cast<float2*>(q + 2 * size_t(stride) + c) = make_float2(k.jn0, k.jt0);
        if (k.count != 1u) *reinterpret_cast<float2*>(q + 5 * size_t(stride) + c) = make_float2(k.jn1, k.jt1);
    }
    // The impulses (jn0, jt0, jn1, jt1); 'second' the ones a record with one point left out.
    __device__ __forceinline__ float4 impulses(uint32_t c, float2 second) const
    {
        const float2 a = *reinterpret_cast<const float2*>(q + 2 * size_t(stride) + c);
        float2 b = second;
        if (__float_as_uint(q[c].x) >> 30 != 1u) b = *reinterpret_cast<const float2*>(q + 5 * size_t(stride) + c);
        return make_float4(a.x, a.y, b.x, b.y);
    }
    // Pulls a warp's 32 records [c0, c0 + 32) into L1 ahead of the pass that reads them: a line a lane.
    __device__ __forceinline__ void prefetch(uint32_t c0) const
    {
        const uint32_t lane = threadIdx.x & 31u;
        asm volatile("prefetch.global.L1 [%0];" ::"l"(q + size_t(lane >> 2) * stride + c0 + (lane & 3u) * 8u));
    }
};

// Scratch of one world's (or one team of worlds') colouring and solve.
struct SolveScratch {
    uint32_t* color;                  // [manifolds]
    uint32_t* order;                  // [manifolds] colour-major solving order
    unsigned long long* bodyMax;      // [bodies] global colouring words (GlobalBodies), zeroed before the call
    unsigned long long* bodyMask;     // [bodies] colours taken around each body, zeroed before the call
    uint32_t* colorCount;             // [COLOR_SLOTS], zeroed by the routine
    uint32_t* colorStart;             // [MAX_COLORS + 1]
    ConsRecords cons;                 // [manifolds]
    const uint32_t* prio;             // [manifolds] colouring priorities, or null: priority_hash(index)
    uint4* listA;                     // [manifolds] uncoloured manifold records, ping
    uint4* listB;                     // [manifolds] uncoloured manifold records, pong
    uint2* pairBodies;                // [manifolds] the two bodies, bit 31 set when the body is dynamic
    const uint32_t* hint;             // [manifolds] colour of the same contact pair last step (NO_COLOR: none), or null
};

// Team barriers. ld() reads a colour counter written by other team members before the last barrier: global memory
// through L2 for the grid, shared memory for one CTA.
struct BlockSync {
    static constexpr bool GRID = false;
    __device__ __forceinline__ bool operator()() const { __syncthreads(); return true; }
    static __device__ __forceinline__ uint32_t ld(const uint32_t* p) { return *static_cast<const volatile uint32_t*>(p); }
};
struct GridSync {
    static constexpr bool GRID = true;
    uint32_t* bar;
    uint32_t* status;
    __device__ __forceinline__ bool operator()() const { return grid_barrier(bar, status); }
    static __device__ __forceinline__ uint32_t ld(const uint32_t* p) { return __ldcg(p); }
};

// Constraint records of a team kept in shared memory for the warm, velocity and position passes: seven float4
// fields per constraint, structure of arrays (q[f * cap + c]), so a warp's 16-byte accesses are contiguous. Body
// indices are stored relative to the team's first body (12 bits each, MAX_TEAM_BODY_CAP <= 4096). cap == 0: the
// records stay in global memory (SolveScratch::cons). The arithmetic on a record is the same either way.
struct ConsSmem {
    float4* q = nullptr;
    uint32_t cap = 0;
    uint32_t base = 0;
    static constexpr uint32_t FIELDS = 7;
    __device__ __forceinline__ void store(uint32_t c, const Constraint& k) const
    {
        const uint32_t packed = (k.bodyA - base) | (k.bodyB - base) << 12 | k.count << 24;
        q[c] = make_float4(__uint_as_float(packed), k.penBase, k.nx, k.ny);
        q[cap + c] = make_float4(k.jn0, k.jt0, k.jn1, k.jt1);
        q[2 * cap + c] = make_float4(k.rAn0, k.rBn0, k.rAt0, k.rBt0);
        q[3 * cap + c] = make_float4(k.rAn1, k.rBn1, k.rAt1, k.rBt1);
        q[4 * cap + c] = make_float4(k.nm0, k.tm0, k.bias0, k.nm1);
        q[5 * cap + c] = make_float4(k.tm1, k.bias1, k.sf, k.df);
        q[6 * cap + c] = make_float4(k.imA, k.imB, k.iIA, k.iIB);
    }
    __device__ __forceinline__ void loadHead(uint32_t c, Constraint& k) const
    {
        const float4 a = q[c];
        const uint32_t packed = __float_as_uint(a.x);
        k.bodyA = base + (packed & 0xFFFu);
        k.bodyB = base + ((packed >> 12) & 0xFFFu);
        k.count = packed >> 24;
        k.penBase = a.y; k.nx = a.z; k.ny = a.w;
    }
    __device__ __forceinline__ void load(uint32_t c, Constraint& k) const
    {
        loadHead(c, k);
        const float4 j = q[cap + c], r0 = q[2 * cap + c], r1 = q[3 * cap + c], m0 = q[4 * cap + c],
                     m1 = q[5 * cap + c], ms = q[6 * cap + c];
        k.jn0 = j.x; k.jt0 = j.y; k.jn1 = j.z; k.jt1 = j.w;
        k.rAn0 = r0.x; k.rBn0 = r0.y; k.rAt0 = r0.z; k.rBt0 = r0.w;
        k.rAn1 = r1.x; k.rBn1 = r1.y; k.rAt1 = r1.z; k.rBt1 = r1.w;
        k.nm0 = m0.x; k.tm0 = m0.y; k.bias0 = m0.z; k.nm1 = m0.w;
        k.tm1 = m1.x; k.bias1 = m1.y; k.sf = m1.z; k.df = m1.w;
        k.imA = ms.x; k.imB = ms.y; k.iIA = ms.z; k.iIB = ms.w;
    }
    __device__ __forceinline__ void loadMasses(uint32_t c, Constraint& k) const
    {
        const float4 ms = q[6 * cap + c];
        k.imA = ms.x; k.imB = ms.y;
    }
    __device__ __forceinline__ void storeImpulses(uint32_t c, const Constraint& k) const
    {
        q[cap + c] = make_float4(k.jn0, k.jt0, k.jn1, k.jt1);
    }
    __device__ __forceinline__ float4 impulses(uint32_t c) const { return q[cap + c]; }
};
constexpr uint32_t CONS_SMEM_BYTES = ConsSmem::FIELDS * sizeof(float4);

// Phases of the solve: what a phase does with its records.
constexpr uint32_t PHASE_WARM = 0, PHASE_VELOCITY = 1, PHASE_POSITION = 2;

__device__ __forceinline__ void ConsRecords::load(uint32_t c, uint32_t kind, Constraint& k, BlockMatrix& bm) const
{
    loadHead(c, k);
    if (kind == PHASE_POSITION) {
        k.penBase = pen[c];
        return;
    }
    const float4* r = q + c;
    const size_t st = stride;
    const float4 j = r[2 * st], r0 = r[3 * st], m0 = r[4 * st];
    k.jn0 = j.x; k.jt0 = j.y; k.sf = j.z; k.df = j.w;
    k.rAn0 = r0.x; k.rBn0 = r0.y; k.rAt0 = r0.z; k.rBt0 = r0.w;
    k.nm0 = m0.x; k.tm0 = m0.y; k.bias0 = m0.z; k.bias1 = m0.w;
    if (k.count != 1u) {
        const float4 m1 = r[5 * st], r1 = r[6 * st];
        k.jn1 = m1.x; k.jt1 = m1.y; k.nm1 = m1.z; k.tm1 = m1.w;
        k.rAn1 = r1.x; k.rBn1 = r1.y; k.rAt1 = r1.z; k.rBt1 = r1.w;
        if (kind == PHASE_VELOCITY) {
            const float4 b = r[7 * st];
            bm.K00 = b.x; bm.K01 = b.y; bm.K11 = b.z; bm.invDet = b.w;
        }
    } else {
        k.jn1 = 0.0f; k.jt1 = 0.0f; k.nm1 = 0.0f; k.tm1 = 0.0f;
        k.rAn1 = 0.0f; k.rBn1 = 0.0f; k.rAt1 = 0.0f; k.rBt1 = 0.0f;
    }
}

// The records this thread's warp handles first in colour 'col' (or nothing), prefetched before the barrier that
// precedes that colour's pass.
template <class Sync>
__device__ __forceinline__ void prefetch_colour(const SolveScratch& s, uint32_t col, uint32_t ncol, uint32_t rank)
{
    if (col >= ncol) return;
    const uint32_t c0 = Sync::ld(s.colorStart + col) + (rank & ~31u);
    if (c0 < Sync::ld(s.colorStart + col + 1)) s.cons.prefetch(c0);
}

// One phase's step on a record held in registers; a velocity step writes the record's impulses back.
template <class Bodies>
__device__ __forceinline__ void solve_record(const Bodies& B, const ConsRecords& cons, uint32_t c, uint32_t kind,
                                             Constraint& k, const BlockMatrix& bm)
{
    if (kind == PHASE_WARM) {
        warm_constraint(B, k);
    } else if (kind == PHASE_VELOCITY) {
        velocity_constraint(B, k, bm);
        cons.storeImpulses(c, k);
    } else {
        position_constraint(B, k);
    }
}

// The warm, velocity and position passes with global records, pipelined: the passes are one sequence of phases
// (colour-major within each pass, the barrier between phases); in a phase this thread handles the records
// start + rank, + size, ... of the phase's colour, and the first of them is loaded one phase ahead. A record is
// written only by the thread that handles it (its impulses), so its load may cross the barrier, which orders the
// body state alone: the load is in flight while this phase computes and waits. Same arithmetic, same order as the
// unpipelined passes; more registers (two records live).
template <class Sync, class Bodies>
__device__ bool solve_passes_pipelined(const Bodies& B, const SolveScratch& s, uint32_t ncol, uint32_t velIters,
                                       uint32_t posIters, uint32_t rank, uint32_t size, Sync sync)
{
    const uint32_t nPhase = ncol * (1 + velIters + posIters);
    auto kindOf = [&](uint32_t ph) {
        const uint32_t p = ph / ncol;
        return p == 0 ? PHASE_WARM : (p <= velIters ? PHASE_VELOCITY : PHASE_POSITION);
    };
    constexpr uint32_t NO_REC = 0xFFFFFFFFu;
    // This thread's first record of a colour, or NO_REC; the tail is the first thread's alone, one after the other.
    auto first = [&](uint32_t col) {
        const uint32_t c = Sync::ld(s.colorStart + col) + rank;
        return c < Sync::ld(s.colorStart + col + 1) && (col != TAIL_COLOR || rank == 0) ? c : NO_REC;
    };
    Constraint nxt;
    BlockMatrix nxtBm;
    uint32_t cNext = NO_REC;
    if (nPhase) {
        cNext = first(0);
        if (cNext != NO_REC) s.cons.load(cNext, kindOf(0), nxt, nxtBm);
    }
    for (uint32_t ph = 0; ph < nPhase; ph++) {
        const uint32_t col = ph % ncol, kind = kindOf(ph);
        const uint32_t end = Sync::ld(s.colorStart + col + 1);
        Constraint k = nxt;
        BlockMatrix bm = nxtBm;
        uint32_t c = cNext;   // NO_REC (above every end) when this thread has no record in the phase
        cNext = NO_REC;
        if (ph + 1 < nPhase) {
            const uint32_t col2 = (ph + 1) % ncol;
            cNext = first(col2);
            if (cNext != NO_REC) s.cons.load(cNext, kindOf(ph + 1), nxt, nxtBm);
        }
        while (c < end) {
            solve_record(B, s.cons, c, kind, k, bm);
            // One colour: the next phase's record is this one, loaded before this phase's impulses.
            if (cNext == c) { nxt.jn0 = k.jn0; nxt.jt0 = k.jt0; nxt.jn1 = k.jn1; nxt.jt1 = k.jt1; }
            c += col == TAIL_COLOR ? 1u : size;   // a colour larger than the team
            if (c < end) s.cons.load(c, kind, k, bm);
        }
        if (!sync()) return false;
    }
    return true;
}

// Colouring followed by the colour-major solve. Colouring runs Jones-Plassmann rounds: in round r every uncoloured
// manifold whose priority is the largest on each of its dynamic bodies takes the smallest colour not yet taken
// around its dynamic bodies (first fit); winners of one round share no dynamic body, so the colours stay
// conflict-free and depend only on the manifold list and priorities. Each round visits only the manifolds still
// uncoloured (compacted into a list whose order does not affect the result). rank/size: this thread's index in the
// team. Returns false if the colouring ran out of colours or a barrier gave up.
// Colouring with carried colours: a manifold whose collider pair was solved last step (its hint) keeps that
// step's colour when it was a first-fit one (< 64) and has been kept for fewer than COLOR_KEEP_STEPS steps in a
// row (so each contact's place in the solving order is revisited regularly). Two kept manifolds of one colour
// cannot share a dynamic body (of finite mass): their predecessors were coloured together last step, and a body that
// turned dynamic since has no coloured manifolds (the host drops their colours when a command gives it a mass). The
// other manifolds run the Jones-Plassmann rounds around the kept colours. With no hints every manifold runs the
// rounds. Hints that two manifolds on one dynamic body share (from a checkpoint that was not saved so) end the routine
// with STATUS_COLOR_CLASH before anything moves. s.color holds colour | age << COLOR_AGE_SHIFT.
// s.pairBodies words: body index | PAIR_DYNAMIC (finite mass) | PAIR_KEPT (first word: colour carried over) or
// PAIR_TWO (second word: not a one-point contact).
constexpr uint32_t PAIR_DYNAMIC = 0x80000000u, PAIR_KEPT = 0x40000000u, PAIR_TWO = 0x40000000u, PAIR_BODY = 0x3FFFFFFFu;

template <class Sync, class Bodies>
__device__ bool color_manifolds(const DeviceWorld& w, const Bodies& B, const Manifold* m, uint32_t n,
                                const SolveScratch& s, uint32_t rank, uint32_t size, Sync sync,
                                uint32_t* outColors, uint32_t* status, uint32_t& ncolOut)
{
    for (uint32_t c = rank; c < COLOR_SLOTS; c += size) s.colorCount[c] = 0;
    // A grid counts per block in shared memory first: one atomic a manifold on the fourteen counters of a pile's colours
    // took 30 us of its colouring and again 35 us of its ordering (128,000 manifolds).
    __shared__ uint32_t blockCount[Sync::GRID ? 2 * MAX_COLORS : 1];
    auto clear_block_counts = [&] {
        if constexpr (Sync::GRID) {
            for (uint32_t c = threadIdx.x; c < 2 * MAX_COLORS; c += blockDim.x) blockCount[c] = 0u;
            __syncthreads();
        }
    };
    clear_block_counts();
    uint32_t* const nColors = s.colorCount + MAX_COLORS + 3;
    // Each manifold's two bodies and whether they are dynamic, looked up once for all colouring rounds; kept
    // colours are counted and marked around their bodies here.
    constexpr uint32_t DYN = PAIR_DYNAMIC, KEPT = PAIR_KEPT;
    if (s.hint && !sync()) return false;   // the counters are zeroed before kept colours are counted
    uint32_t keptTop = 0;
    bool clash = false;
    for (uint32_t i = rank; i < n; i += size) {
        const uint32_t bA = w.cbody[m[i].a], bB = w.cbody[m[i].b];
        const bool dA = B.invMass(bA) > 0.0f, dB = B.invMass(bB) > 0.0f;
        const uint32_t hw = s.hint ? s.hint[i] : NO_COLOR;
        const uint32_t h = hw & COLOR_MASK, age = hw >> COLOR_AGE_SHIFT;
        const bool kept = hw != NO_COLOR && h < 64 && age + 1 < COLOR_KEEP_STEPS;
        if (kept) {
            s.color[i] = h | (age + 1) << COLOR_AGE_SHIFT;
            atomicAdd(Sync::GRID ? blockCount + h : s.colorCount + h, 1u);
            keptTop = max(keptTop, h + 1);
            const unsigned long long bit = 1ull << h;
            const unsigned long long taken = (dA ? atomicOr(B.maskWord(bA), bit) : 0ull) |
                                             (dB ? atomicOr(B.maskWord(bB), bit) : 0ull);
            clash |= (taken & bit) != 0;
        }
        s.pairBodies[i] = make_uint2(bA | (dA ? DYN : 0u) | (kept ? KEPT : 0u), bB | (dB ? DYN : 0u) | (m[i].count != 1u ? PAIR_TWO : 0u));
    }
    if constexpr (Sync::GRID) {
        if (s.hint) {
            __syncthreads();
            for (uint32_t c = threadIdx.x; c < 64; c += blockDim.x)
                if (blockCount[c]) {
                    atomicAdd(s.colorCount + c, blockCount[c]);
                    atomicMax(nColors, c + 1);
                }
        }
    } else if (s.hint) {
        for (int o = 16; o > 0; o >>= 1) keptTop = max(keptTop, __shfl_xor_sync(0xffffffffu, keptTop, o));
        if ((threadIdx.x & 31) == 0 && keptTop) atomicMax(nColors, keptTop);
    }
    uint32_t* const clashes = s.colorCount + MAX_COLORS;   // the team's own word: every thread reads the same
    if (clash) {
        atomicExch(clashes, 1u);
        atomicOr(status, STATUS_COLOR_CLASH);
    }
    if (!sync()) return false;
    if (s.hint && Sync::ld(clashes)) return false;
    uint32_t len = n;
    const uint4* in = nullptr;   // round 0 visits every manifold; later rounds the uncoloured records
    // Record j of this round: {manifold, priority, body A | dynamic bit, body B | dynamic bit}. In round 0 a kept
    // manifold's record carries the KEPT bit and takes no part.
    auto rec = [&](uint32_t j) -> uint4 {
        if (in) return in[j];
        const uint2 pb = s.pairBodies[j];
        return make_uint4(j, s.prio ? s.prio[j] : priority_hash(j), pb.x, pb.y);
    };
    constexpr uint32_t BATCH = 4;   // records loaded together per thread (independent loads in flight)
    // Round r, by 'sz' threads of which this is number rk; false when the barrier gave up.
    auto round = [&](uint32_t r, uint32_t rk, uint32_t sz, auto barrier) {
        uint4* out = (r & 1) ? s.listB : s.listA;
        uint32_t* outLen = s.colorCount + MAX_COLORS + 1 + (r & 1);
        // This counter was last read before the barrier that ended the previous round.
        if (rk == 0) *outLen = 0;
        const unsigned long long tag = static_cast<unsigned long long>(r + 1) << 32;
        for (uint32_t j0 = rk; j0 < len; j0 += BATCH * sz) {
            uint4 e[BATCH];
#pragma unroll
            for (uint32_t u = 0; u < BATCH; u++) e[u] = j0 + u * sz < len ? rec(j0 + u * sz) : make_uint4(0, 0, 0, 0);
#pragma unroll
            for (uint32_t u = 0; u < BATCH; u++) {
                if (j0 + u * sz >= len) break;
                if (e[u].z & KEPT) continue;
                const unsigned long long key = tag | e[u].y;
                if (e[u].z & DYN) atomicMax(B.maxWord(e[u].z & PAIR_BODY), key);
                if (e[u].w & DYN) atomicMax(B.maxWord(e[u].w & PAIR_BODY), key);
            }
        }
        if (!barrier()) return false;
        uint32_t top = 0;
        for (uint32_t j0 = rk; j0 < len; j0 += BATCH * sz) {
            uint4 e[BATCH];
#pragma unroll
            for (uint32_t u = 0; u < BATCH; u++) e[u] = j0 + u * sz < len ? rec(j0 + u * sz) : make_uint4(0, 0, 0, 0);
#pragma unroll
            for (uint32_t u = 0; u < BATCH; u++) {
                if (j0 + u * sz >= len) break;
                if (e[u].z & KEPT) continue;
                const uint32_t i = e[u].x;
                const unsigned long long key = tag | e[u].y;
                const uint32_t bA = e[u].z & PAIR_BODY, bB = e[u].w & PAIR_BODY;
                const bool dA = (e[u].z & DYN) != 0, dB = (e[u].w & DYN) != 0;
                if ((!dA || B.ldWord(B.maxWord(bA)) == key) && (!dB || B.ldWord(B.maxWord(bB)) == key)) {
                    const unsigned long long used = (dA ? B.ldWord(B.maskWord(bA)) : 0ull) |
                                                    (dB ? B.ldWord(B.maskWord(bB)) : 0ull);
                    const uint32_t c = used == ~0ull ? 64u + r : uint32_t(__ffsll(static_cast<long long>(~used)) - 1);
                    s.color[i] = c;
                    atomicAdd(s.colorCount + c, 1u);
                    top = max(top, c + 1);
                    if (c < 64) {
                        if (dA) atomicOr(B.maskWord(bA), 1ull << c);
                        if (dB) atomicOr(B.maskWord(bB), 1ull << c);
                    }
                } else {
                    out[atomicAdd(outLen, 1u)] = e[u];
                }
            }
        }
        for (int o = 16; o > 0; o >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
        if ((threadIdx.x & 31) == 0 && top) atomicMax(nColors, top);
        if (!barrier()) return false;
        len = Sync::ld(outLen);
        in = out;
        return true;
    };
    uint32_t r = 0;
    for (; r < MAX_ROUNDS && len > 0 && !(Sync::GRID && r > 0 && len <= ONE_BLOCK_ROUND); r++)
        if (!round(r, rank, size, sync)) return false;
    if constexpr (Sync::GRID) {
        // The few manifolds that are left after the first rounds are finished by one block: a round is then two block
        // barriers, not two of the grid (10 us a round on 148 blocks).
        if (len > 0) {
            if (blockIdx.x == 0) {
                auto block = [] { __threadfence(); __syncthreads(); return true; };
                for (; r < MAX_ROUNDS && len > 0; r++) round(r, threadIdx.x, blockDim.x, block);
                if (rank == 0) s.colorCount[MAX_COLORS + 1] = len;
            }
            if (!sync()) return false;
            len = Sync::ld(s.colorCount + MAX_COLORS + 1);
        }
    }
    if (len > TAIL_MAX) { if (rank == 0) atomicOr(status, STATUS_COLOR_OVERFLOW); return false; }
    if (rank == 0 && len > 0) {
        s.colorCount[TAIL_COLOR] = len;
        atomicMax(nColors, MAX_COLORS);
    }
    if (len > 0 && !sync()) return false;
    const uint32_t ncol = ncolOut = Sync::ld(nColors);
    if (rank == 0) {
        uint32_t run = 0;
        for (uint32_t c = 0; c < ncol; c++) { s.colorStart[c] = run; run += s.colorCount[c]; s.colorCount[c] = 0; }
        s.colorStart[ncol] = run;
        atomicMax(outColors, ncol);
    }
    if (!sync()) return false;
    if (len > 0) {   // the tail in list order: a manifold's place is the number of the tail's below it
        const uint4* const tail = (MAX_ROUNDS - 1u) & 1u ? s.listB : s.listA;
        for (uint32_t j = rank; j < len; j += size) {
            const uint32_t i = tail[j].x;
            uint32_t below = 0;
            for (uint32_t k = 0; k < len; k++) below += tail[k].x < i;
            s.color[i] = TAIL_COLOR;
            s.order[Sync::ld(s.colorStart + TAIL_COLOR) + below] = i;
        }
        if (!sync()) return false;
    }
    // Within a colour (independent contacts, any order) two-point contacts come first and one-point contacts last, so
    // that few warps run both solves.
    if constexpr (Sync::GRID) {
        // Places within the block, then the blocks' ranges (front counter c, back counter MAX_COLORS + c).
        uint32_t* const place = reinterpret_cast<uint32_t*>(s.listA);   // the uncoloured lists are done with
        clear_block_counts();
        for (uint32_t i = rank; i < n; i += size)
            if ((s.color[i] & COLOR_MASK) != TAIL_COLOR) place[i] = atomicAdd(blockCount + (s.color[i] & COLOR_MASK) + (s.pairBodies[i].y & PAIR_TWO ? 0u : MAX_COLORS),
                                 1u);
        __syncthreads();
        for (uint32_t c = threadIdx.x; c < 2 * MAX_COLORS; c += blockDim.x)
            if (blockCount[c])
                blockCount[c] = atomicAdd(s.colorCount + (c < MAX_COLORS ? c : c + 4), blockCount[c]);
        __syncthreads();
        for (uint32_t i = rank; i < n; i += size) {
            const uint32_t c = s.color[i] & COLOR_MASK;
            if (c == TAIL_COLOR) continue;
            const uint32_t at = s.pairBodies[i].y & PAIR_TWO
                                    ? __ldcg(s.colorStart + c) + blockCount[c] + place[i]
                                    : __ldcg(s.colorStart + c + 1) - 1u - blockCount[MAX_COLORS + c] - place[i];
            s.order[at] = i;
        }
        return sync();
    }
    for (uint32_t i = rank; i < n; i += size) {
        const uint32_t c = s.color[i] & COLOR_MASK;
        if (c == TAIL_COLOR) continue;
        const uint32_t at = s.pairBodies[i].y & PAIR_TWO
                                ? Sync::ld(s.colorStart + c) + atomicAdd(s.colorCount + c, 1u)
                                : Sync::ld(s.colorStart + c + 1) - 1u - atomicAdd(s.colorCount + MAX_COLORS + 4 + c, 1u);
        s.order[at] = i;
    }
    return sync();
}

// The colour-major solve of coloured manifolds (s.order, s.colorStart), with the team's barrier between colours.
template <class Sync, class Bodies, bool PIPELINED = false>
__device__ bool solve_colored(const DeviceWorld& w, const Bodies& B, Manifold* m, uint32_t n,
                              const SolveScratch& s, uint32_t ncol, uint32_t velIters, uint32_t posIters,
                              uint32_t rank, uint32_t size, Sync sync, ConsSmem cs = ConsSmem{})
{
    // The colouring words are no longer needed: a lazily staged body cache is loaded over them now.
    if (B.stage(rank, size) && !sync()) return false;
    // Constraint build for every manifold before any velocity changes (computeConstraintData). The records go to
    // shared memory when the team's fit there (the colouring words they overwrite are no longer needed).
    const bool onChip = cs.cap >= n && cs.q != nullptr;
    for (uint32_t c = rank; c < n; c += size) {
        const uint32_t mi = __ldcg(s.order + c);
        Constraint k;
        prep_constraint(w, B, m[mi], mi, k);
        if (onChip) cs.store(c, k);
        else s.cons.store(c, k);
    }
    if (!sync()) return false;
    bool passesDone = false;
    if constexpr (PIPELINED) {
        if (!onChip) {
            if (!solve_passes_pipelined(B, s, ncol, velIters, posIters, rank, size, sync)) return false;
            passesDone = true;
        }
    }
    // The tail is the first thread's alone, one after the other.
    auto takes = [&](uint32_t col) { return col != TAIL_COLOR || rank == 0; };
    auto step = [&](uint32_t col) { return col == TAIL_COLOR ? 1u : size; };
    if (!passesDone) {
        for (uint32_t col = 0; col < ncol; col++) {
            const uint32_t end = Sync::ld(s.colorStart + col + 1);
            const uint32_t begin = Sync::ld(s.colorStart + col);
            for (uint32_t c = begin + rank; takes(col) && c < end; c += step(col)) {
                Constraint k;
                BlockMatrix bm;
                if (onChip) cs.load(c, k);
                else s.cons.load(c, PHASE_WARM, k, bm);
                warm_constraint(B, k);
            }
            if (!sync()) return false;
        }
        // Position iteration 'it' runs beside velocity iteration 'it': the two touch different body state (poses and
        // velocities), so a colour's position steps share the barrier interval of its velocity steps, on the threads
        // that have no velocity step: 8 + 1 passes of barriers instead of 8 + 3 + 1 at the default counts.
        const uint32_t iters = velIters > posIters ? velIters : posIters;
        for (uint32_t it = 0; it < iters; it++) {
            const bool vel = it < velIters, pos = it < posIters;
            for (uint32_t col = 0; col < ncol; col++) {
                const uint32_t begin = Sync::ld(s.colorStart + col), count = Sync::ld(s.colorStart + col + 1) - begin;
                const uint32_t posBase = vel ? (count + 31u) & ~31u : 0u;   // a warp does one kind of step
                const uint32_t total = pos ? posBase + count : count;
                for (uint32_t j = rank; takes(col) && j < total; j += step(col)) {
                    Constraint k;
                    BlockMatrix bm;
                    if (vel && j < count) {
                        const uint32_t c = begin + j;
                        if (onChip) {
                            cs.load(c, k);
                            bm = block_matrix(k);
                        } else {
                            s.cons.load(c, PHASE_VELOCITY, k, bm);
                        }
                        velocity_constraint(B, k, bm);
                        if (onChip) cs.storeImpulses(c, k);
                        else s.cons.storeImpulses(c, k);
                    } else if (j >= posBase) {
                        const uint32_t c = begin + j - posBase;
                        if (onChip) {
                            cs.loadHead(c, k);
                            cs.loadMasses(c, k);
                        } else {
                            s.cons.load(c, PHASE_POSITION, k, bm);
                        }
                        position_constraint(B, k);
                    }
                }
                // The next interval's constraint: from the next colour, or colour 0 of the next iteration.
                if (!onChip) prefetch_colour<Sync>(s, col + 1 < ncol ? col + 1 : 0, ncol, rank);
                if (!sync()) return false;
            }
        }
    }
    for (uint32_t c = rank; c < n; c += size) {
        Manifold& d = m[__ldcg(s.order + c)];
        const float4 j = onChip ? cs.impulses(c) : s.cons.impulses(c, make_float2(d.jn1, d.jt1));
        d.jn0 = j.x; d.jt0 = j.y; d.jn1 = j.z; d.jt1 = j.w;
    }
    return true;
}

template <class Sync, class Bodies, bool PIPELINED = false>
__device__ __forceinline__ bool color_and_solve(const DeviceWorld& w, const Bodies& B, Manifold* m,
                                                uint32_t n, const SolveScratch& s, uint32_t velIters,
                                                uint32_t posIters, uint32_t rank, uint32_t size, Sync sync,
                                                uint32_t* outColors, uint32_t* status,
                                                ConsSmem cs = ConsSmem{})
{
    uint32_t ncol = 0;
    return color_manifolds(w, B, m, n, s, rank, size, sync, outColors, status, ncol) &&
           solve_colored<Sync, Bodies, PIPELINED>(w, B, m, n, s, ncol, velIters, posIters, rank, size, sync, cs);
}

// Single worlds whose bodies fit one CTA's shared memory (32 B each, up to BLOCK_SOLVE_BODIES): one CTA colours,
// solves and links the islands, __syncthreads between colours. With more than BLOCK_SOLVE_MANIFOLDS contacts, and more
// than BLOCK_SOLVE_PER_COLOR of them a colour, the grid solves them all the same: one CTA pays per manifold, the grid per
// colour. A step's solve, one CTA against the grid: piles of 2,609 manifolds 167 and 183 us, 3,503: 208 and 191, 4,727: 237
// and 189, 9,269: 431 and 207; compound bodies of 9 and 16 boxes with 5,110 manifolds in 20 colours 348 and 358, 8,346 in
// 61: 927 and 1,086, 16,909 in 87: 1,282 and 1,259, 35,542 in 103: 2,219 and 1,670.
constexpr uint32_t BLOCK_SOLVE_BODIES = 6912;
constexpr uint32_t BLOCK_SOLVE_MANIFOLDS = 4096;
constexpr uint32_t BLOCK_SOLVE_PER_COLOR = 192;
struct BlockSolve {
    DeviceWorld w;
    Manifold* m;
    const uint32_t* nM;
    SolveScratch s;            // colour counters in global memory, copied out for the readers of colour starts
    uint32_t bodyCap;          // bodies of the shared-memory cache, >= w.nBodies
    uint32_t velIters, posIters;
    uint32_t* ufParent;        // [bodies] island roots out (smallest body index of the island)
    uint32_t* ufFlag;          // [bodies] set to 1
    StepCounters* counters;
};
// Host side: launches the one-CTA solver for about 'perColor' manifolds a colour.
cudaError_t launch_color_solve_block(uint32_t perColor, cudaStream_t stream, const BlockSolve& a);
// Host side: raises the one-CTA solver's dynamic shared-memory limit (once per device).
cudaError_t block_solver_init();

// Other single worlds: a cooperative grid colours the manifolds, then solves them as a dataflow over per-body
// versions instead of barriers (k_color_solve_flow).
constexpr uint32_t FLOW_VEL_WARPS = 16, FLOW_POS_WARPS = 4;   // warps of a CTA: velocity passes, position passes
constexpr uint32_t FLOW_THREADS = 32 * (FLOW_VEL_WARPS + FLOW_POS_WARPS);
constexpr uint32_t FLOW_HIGH = MAX_COLORS / 64 - 1;
struct FlowScratch {
    float4* vel;       // [bodies] vx, vy, w, version
    float4* pos;       // [bodies] x, y, -, version
    Constraint* cons;  // [manifolds] records, 'pad' the rank of a and its degree less one, those of b: one byte each
    float4 *posA, *posB;   // [manifolds] position records: normal, penetration base, ranks; masses, bodies. They may lie
                           // over the lists of uncoloured manifolds, which are done with by then
    unsigned long long* high;   // [FLOW_HIGH x bodies] colours above the first-fit 64 around each body, written on use
    uint32_t* parent;  // [bodies] islands to link beside the solve, every body its own; or null
};
__global__ void __launch_bounds__(FLOW_THREADS, 1)
k_color_solve_flow(DeviceWorld w, Manifold* m, const uint32_t* nM, SolveScratch s, FlowScratch f, uint32_t velIters,
                   uint32_t posIters, uint32_t* bar, StepCounters* counters);

// Batched worlds: teams of consecutive worlds (team k owns worlds [teamWorld[k], teamWorld[k + 1])), each coloured
// and solved by one CTA with __syncthreads between colours. Teams are taken from the work counter *nextTeam (zeroed
// before the launch) in 'teamOrder' order, largest first. Colouring priorities are world-local manifold indices, so
// the colours of a world do not depend on its team. The CTA size (64 to 512 threads) is a launch parameter;
// a team whose bodies fit 'bodyCap' keeps their state and colouring words in dynamic shared memory, and, when its
// manifolds fit 'consCap', its constraint records too (team_smem_bytes).
constexpr uint32_t MAX_TEAM_BODY_CAP = 4096;   // largest body range a team stages in shared memory
constexpr uint32_t TEAM_SMEM_MAX = 220 * 1024; // dynamic shared memory of a team CTA (sm_100 allows 227 KB in
                                               // all, the kernel's static arrays included)
// Dynamic shared memory of a team CTA: body velocities and poses, then one region holding first the colouring words
// (16 B a body) and then the constraint records (CONS_SMEM_BYTES each, consCap of them).
// With no records on chip (consCap 0) the colouring words share the body cache (SharedBodies, lazy): 32 B a body.
__host__ __device__ constexpr size_t team_smem_bytes(uint32_t bodyCap, uint32_t consCap)
{
    return consCap == 0 ? size_t(bodyCap) * 2 * sizeof(float4)
                        : size_t(bodyCap) * 2 * sizeof(float4) +
                              (size_t(bodyCap) * 16 > size_t(consCap) * CONS_SMEM_BYTES
                                   ? size_t(bodyCap) * 16
                                   : size_t(consCap) * CONS_SMEM_BYTES);
}
// Launch shapes of the CTAs that solve a world larger than the team size (one world each): threads per CTA and
// whether the global-record passes are pipelined (solve_passes_pipelined).
constexpr uint32_t BIG_TEAM_THREADS = 512;
struct TeamLaunch {
    DeviceWorld w;
    Manifold* m;
    const uint32_t* manSeg;
    const uint32_t* teamWorld;
    const uint32_t* teamOrder;
    uint32_t teams;
    uint32_t bodyCap;
    uint32_t consCap;   // constraint records a team keeps in shared memory (0: global memory)
    SolveScratch s;
    uint32_t velIters, posIters;
    uint32_t* nextTeam;
    StepCounters* counters;
    uint32_t* ufParent;   // non-null: each team also links its islands (union-find over its manifolds, roots the
                          // smallest body index) into this array, initialised to parent[b] = b before the launch
};
// Host side: launches the team solver with 'threads' per CTA; returns the launch error.
cudaError_t launch_color_solve_teams(bool chained, uint32_t threads, bool pipelined, uint32_t grid, cudaStream_t stream,
                                     const TeamLaunch& a);
// Host side: co-resident CTAs per SM of the team solver at this CTA size and shared-memory capacities. Also raises
// the kernel's dynamic shared-memory limit to TEAM_SMEM_MAX (the limit is per kernel, shared by every engine in the
// process, so it is never lowered).
cudaError_t team_solver_blocks_per_sm(uint32_t threads, bool pipelined, uint32_t bodyCap, uint32_t consCap, int* out);

}  // namespace ag2d
