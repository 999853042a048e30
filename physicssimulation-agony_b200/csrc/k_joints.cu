// Body constraints: springs, revolute, prismatic and slider joints, motors (Solving/SpringSolver.cpp,
// RevoluteJointSolver.cpp, PrismaticJointSolver.cpp, SliderJointSolver.cpp, MotorSolver.cpp), scheduled as
// ConstraintScheduler::solve does (Solving/ConstraintScheduler.cpp:9-80), between the two integration phases
// (Simulation.cpp:392-407). Paths are relative to PhysicsSimulation-Agony/PS_AGONY2D/.
//
// The reference solves each constraint type's active constraints one after another in dense order (Gauss-Seidel;
// below its threading threshold, one wave in identity order). Here each type's constraints come grouped by level:
// a constraint's level is one more than the highest level of the earlier constraints (in dense order) that write
// one of its bodies. Constraints of one level touch disjoint movable bodies and read only what earlier levels
// wrote, so solving a level in parallel, with a barrier between levels, gives the dense-order results bit for bit.
// One CTA runs the whole schedule: the compute tick over every type, the motors' warm start, then the interleaved
// velocity iterations (type t is active at iteration k when floor((k+1) n_t / max) > floor(k n_t / max)).
//
// Solver data (JointData::s) per kind. Spring: s0, s1 direction, s2 inverse effective mass (0: skip), s3 bias.
// Revolute joint: s0, s1 bias, s4 k11, s5 k12, s6 k22 of the inverse effective mass (all 0: skip). Prismatic and
// slider joints: s0, s1 axis, s2, s3 perpendicular, s4 s1, s5 s2 (perpendicular moment arms), s6 a1, s7 a2 (axis
// moment arms), s8 k11 (slider: the scalar inverse mass, 0: inactive), s9 k12, s10 k22, s11 block valid
// (prismatic), s12 bias1 (slider: bias), s13 bias2, s14 axis inverse effective mass, s15 axis bias, s16 limit
// direction (0: no limit this step), s17 accumulated axis impulse. Motor: s0 inverse inertia (0: skip), s1 inertia,
// s2 target speed, s3 max impulse, s4 impulse.
#include "ag2d_kernels.cuh"

#include <type_traits>

namespace ag2d {

namespace {

constexpr uint32_t K_SPRING = 0, K_REVOLUTE = 1, K_PRISMATIC = 2, K_SLIDER = 3, K_MOTOR = 4;

// glm::clamp for scalars: min(max(x, lo), hi) with max(x, y) = (x < y) ? y : x and min(x, y) = (y < x) ? y : x.
__device__ __forceinline__ float glm_clamp(float x, float lo, float hi)
{
    const float t = (x < lo) ? lo : x;
    return (hi < t) ? hi : t;
}

// Soft-constraint parameters from stiffness and damping (SpringSolver.cpp:92-101 and the same in every joint).
__device__ __forceinline__ void soft_params(float dt, float k, float c, float& gamma, float& beta)
{
    gamma = 0.0f;
    beta = 0.0f;
    const float denom = dt * (c + dt * k);
    if (denom > 1e-12f) {
        gamma = 1.0f / denom;
        beta = dt * k * gamma;
    }
}

// Wraps an angle into (-pi, pi] (PrismaticJointSolver.cpp:12-17).
__device__ __forceinline__ float wrap_to_pi(float angle)
{
    const float pi = 3.14159265358979323846f, twoPi = 2.0f * pi;
    return angle - twoPi * floorf((angle + pi) / twoPi);
}

struct Frame {   // the anchors of a pair constraint in world orientation
    float4 pA, pB;
    float imA, imB;
    float2 cA, cB;
    float rAx, rAy, rBx, rBy;
};
__device__ __forceinline__ Frame frame(const DeviceWorld& w, const JointRec& r)
{
    Frame f;
    f.pA = w.bpos[r.bodyA];
    f.pB = w.bpos[r.bodyB];
    f.imA = w.bvel[r.bodyA].w;
    f.imB = w.bvel[r.bodyB].w;
    f.cA = w.brot[r.bodyA];
    f.cB = w.brot[r.bodyB];
    f.rAx = r.ax * f.cA.x - r.ay * f.cA.y;
    f.rAy = r.ax * f.cA.y + r.ay * f.cA.x;
    f.rBx = r.bx * f.cB.x - r.by * f.cB.y;
    f.rBy = r.bx * f.cB.y + r.by * f.cB.x;
    return f;
}

// computeConstraintData of one spring (SpringSolver.cpp:7-108).
__device__ void spring_data(const DeviceWorld& w, const JointRec& r, float dt, JointData& d)
{
    d.s[2] = 0.0f;
    if (w.bvel[r.bodyA].w == 0.0f && w.bvel[r.bodyB].w == 0.0f) return;
    const Frame f = frame(w, r);
    const float dx = (f.pB.x + f.rBx) - (f.pA.x + f.rAx), dy = (f.pB.y + f.rBy) - (f.pA.y + f.rAy);
    const float lenSq = dx * dx + dy * dy;
    if (lenSq < 1e-12f) return;
    const float len = sqrtf(lenSq);
    const float nx = dx / len, ny = dy / len;
    const float C = len - r.p[0];
    const float raCn = (f.rAx * ny) - (f.rAy * nx);
    const float rbCn = (f.rBx * ny) - (f.rBy * nx);
    const float eff = f.imA + f.imB + f.pA.w * raCn * raCn + f.pB.w * rbCn * rbCn;
    if (eff <= 0.0f) return;
    float gamma, beta;
    soft_params(dt, r.p[1], r.p[2], gamma, beta);
    d.rAx = f.rAx; d.rAy = f.rAy; d.rBx = f.rBx; d.rBy = f.rBy;
    d.s[0] = nx; d.s[1] = ny;
    d.s[2] = 1.0f / (eff + gamma);
    d.s[3] = beta * C;
}

// computeConstraintData of one revolute joint (RevoluteJointSolver.cpp:7-115).
__device__ void revolute_data(const DeviceWorld& w, const JointRec& r, float dt, JointData& d)
{
    d.s[4] = d.s[5] = d.s[6] = 0.0f;
    if (w.bvel[r.bodyA].w == 0.0f && w.bvel[r.bodyB].w == 0.0f) return;
    const Frame f = frame(w, r);
    const float iIA = f.pA.w, iIB = f.pB.w;
    const float ex = (f.pB.x + f.rBx) - (f.pA.x + f.rAx), ey = (f.pB.y + f.rBy) - (f.pA.y + f.rAy);
    const float k11 = f.imA + f.imB + iIA * f.rAy * f.rAy + iIB * f.rBy * f.rBy;
    const float k22 = f.imA + f.imB + iIA * f.rAx * f.rAx + iIB * f.rBx * f.rBx;
    const float k12 = -iIA * f.rAx * f.rAy - iIB * f.rBx * f.rBy;
    float gamma, beta;
    soft_params(dt, r.p[1], r.p[2], gamma, beta);
    const float k11s = k11 + gamma, k22s = k22 + gamma;
    const float det = k11s * k22s - k12 * k12;
    if (det <= 1e-12f) return;
    const float invDet = 1.0f / det;
    d.rAx = f.rAx; d.rAy = f.rAy; d.rBx = f.rBx; d.rBy = f.rBy;
    d.s[0] = beta * ex; d.s[1] = beta * ey;
    d.s[4] = k22s * invDet;
    d.s[6] = k11s * invDet;
    d.s[5] = -k12 * invDet;
}

// computeConstraintData of one prismatic (slider == false; PrismaticJointSolver.cpp:20-158) or slider joint
// (SliderJointSolver.cpp:8-130): the perpendicular (and, prismatic, relative-angle) soft block and the hard
// one-sided axis limit.
__device__ void axis_joint_data(const DeviceWorld& w, const JointRec& r, float dt, bool slider, JointData& d)
{
    d.s[11] = 0.0f;   // block valid (prismatic)
    d.s[8] = 0.0f;    // scalar inverse mass (slider)
    d.s[16] = 0.0f;   // limit direction
    d.s[14] = 0.0f;
    d.s[17] = 0.0f;
    const float invDt = dt > 1e-12f ? 1.0f / dt : 0.0f;
    if (w.bvel[r.bodyA].w == 0.0f && w.bvel[r.bodyB].w == 0.0f) return;
    const Frame f = frame(w, r);
    const float iIA = f.pA.w, iIB = f.pB.w;
    const float dx = (f.pB.x + f.rBx) - (f.pA.x + f.rAx), dy = (f.pB.y + f.rBy) - (f.pA.y + f.rAy);
    const float axX = r.p[0] * f.cA.x - r.p[1] * f.cA.y, axY = r.p[0] * f.cA.y + r.p[1] * f.cA.x;
    const float pX = -axY, pY = axX;
    d.s[0] = axX; d.s[1] = axY; d.s[2] = pX; d.s[3] = pY;
    const float qx = dx + f.rAx, qy = dy + f.rAy;   // d + rotatedAnchorA
    const float s1 = qx * pY - qy * pX, s2 = f.rBx * pY - f.rBy * pX;
    d.s[4] = s1; d.s[5] = s2;
    float gamma, beta;
    soft_params(dt, r.p[2], r.p[3], gamma, beta);
    if (!slider) {
        const float k11 = f.imA + f.imB + iIA * s1 * s1 + iIB * s2 * s2;
        const float k12 = iIA * s1 + iIB * s2;
        float k22 = iIA + iIB;
        if (k22 == 0.0f) k22 = 1.0f;
        const float k11s = k11 + gamma, k22s = k22 + gamma;
        const float det = k11s * k22s - k12 * k12;
        if (det > 1e-12f) {
            const float invDet = 1.0f / det;
            d.s[8] = k22s * invDet;
            d.s[10] = k11s * invDet;
            d.s[9] = -k12 * invDet;
            d.s[11] = 1.0f;
            const float C1 = pX * dx + pY * dy;
            const float rel = wrap_to_pi(f.pB.z - f.pA.z);
            const float C2 = wrap_to_pi(rel - r.p[6]);
            d.s[12] = beta * C1;
            d.s[13] = beta * C2;
        }
    } else {
        const float k = f.imA + f.imB + iIA * s1 * s1 + iIB * s2 * s2;
        const float kSoft = k + gamma;
        if (kSoft > 1e-12f) {
            d.s[8] = 1.0f / kSoft;
            d.s[12] = beta * (pX * dx + pY * dy);
        }
    }
    if (r.flags & 1u) {
        const float translation = axX * dx + axY * dy;
        const float lower = r.p[4], upper = r.p[5];
        float direction = 0.0f, C = 0.0f;
        if (translation <= lower + 0.005f) { direction = 1.0f; C = translation - lower; }
        else if (translation >= upper - 0.005f) { direction = -1.0f; C = translation - upper; }
        if (direction != 0.0f) {
            const float a1 = qx * axY - qy * axX, a2 = f.rBx * axY - f.rBy * axX;
            const float kAxis = f.imA + f.imB + iIA * a1 * a1 + iIB * a2 * a2;
            if (kAxis > 1e-12f) {
                d.s[6] = a1; d.s[7] = a2;
                d.s[14] = 1.0f / kAxis;
                d.s[16] = direction;
                d.s[15] = 0.2f * invDt * C;
            }
        }
    }
}

// computeConstraintData of one motor (MotorSolver.cpp:7-45); the clamped accumulated impulse is written back.
__device__ void motor_data(const DeviceWorld& w, const JointRec& r, float dt, float* impulses, JointData& d)
{
    const float iI = w.bpos[r.bodyA].w;
    d.s[0] = iI;
    if (iI == 0.0f) {
        impulses[r.index] = 0.0f;
        return;
    }
    const float maxImpulse = r.p[1] * dt;
    const float impulse = glm_clamp(impulses[r.index], -maxImpulse, maxImpulse);
    d.s[1] = 1.0f / iI;
    d.s[2] = r.p[0];
    d.s[3] = maxImpulse;
    d.s[4] = impulse;
    impulses[r.index] = impulse;
}

// Applies a point impulse to both bodies, as the spring and revolute solvers do (A gains, B loses).
__device__ __forceinline__ void apply_pair(float4& vA, float4& vB, float iIA, float iIB, const JointData& d, float ix,
                                           float iy)
{
    if (vA.w > 0.0f) {
        vA.x = vA.x + ix * vA.w;
        vA.y = vA.y + iy * vA.w;
        const float tA = d.rAx * iy - d.rAy * ix;
        vA.z = vA.z + tA * iIA;
    }
    if (vB.w > 0.0f) {
        vB.x = vB.x - ix * vB.w;
        vB.y = vB.y - iy * vB.w;
        const float tB = d.rBx * iy - d.rBy * ix;
        vB.z = vB.z - tB * iIB;
    }
}

// Relative velocity of the anchors, B's minus A's (SpringSolver.cpp:140-147).
__device__ __forceinline__ float2 anchor_relative_velocity(float4 vA, float4 vB, const JointData& d)
{
    const float aAx = (-d.rAy) * vA.z, aAy = d.rAx * vA.z;
    const float aBx = (-d.rBy) * vB.z, aBy = d.rBx * vB.z;
    return make_float2((vB.x + aBx) - (vA.x + aAx), (vB.y + aBy) - (vA.y + aAy));
}

// The solves work on the two bodies' velocities in registers (vx, vy, w, inverse mass) and leave a body of infinite mass
// as it is.
__device__ __forceinline__ void spring_solve(const JointData& d, float4& vA, float4& vB, float iIA, float iIB)
{
    if (d.s[2] == 0.0f) return;
    const float2 rv = anchor_relative_velocity(vA, vB, d);
    const float cdot = rv.x * d.s[0] + rv.y * d.s[1];
    const float mag = (cdot + d.s[3]) * d.s[2];
    apply_pair(vA, vB, iIA, iIB, d, d.s[0] * mag, d.s[1] * mag);
}

__device__ __forceinline__ void revolute_solve(const JointData& d, float4& vA, float4& vB, float iIA, float iIB)
{
    if (d.s[4] == 0.0f && d.s[5] == 0.0f && d.s[6] == 0.0f) return;
    const float2 rv = anchor_relative_velocity(vA, vB, d);
    const float hx = rv.x + d.s[0], hy = rv.y + d.s[1];
    const float ix = d.s[4] * hx + d.s[5] * hy;
    const float iy = d.s[5] * hx + d.s[6] * hy;
    apply_pair(vA, vB, iIA, iIB, d, ix, iy);
}

// One velocity iteration of a prismatic (PrismaticJointSolver.cpp:160-255) or slider joint (SliderJointSolver.cpp:
// 132-220): the perpendicular block, then the axis limit with its accumulated, one-sided impulse.
__device__ __forceinline__ void axis_joint_solve(JointData& d, float4& vA0, float4& vB0, float iIA, float iIB,
                                                 bool slider)
{
    const bool block = slider ? d.s[8] > 0.0f : d.s[11] != 0.0f;
    if (!block && d.s[16] == 0.0f) return;
    float4 vA = vA0, vB = vB0;
    const float imA = vA.w, imB = vB.w;
    if (block) {
        const float pX = d.s[2], pY = d.s[3], s1 = d.s[4], s2 = d.s[5];
        const float cdot1 = (pX * (vB.x - vA.x) + pY * (vB.y - vA.y)) + s2 * vB.z - s1 * vA.z;
        float l1, LA, LB;
        if (slider) {
            l1 = -d.s[8] * (cdot1 + d.s[12]);
            LA = l1 * s1;
            LB = l1 * s2;
        } else {
            const float cdot2 = vB.z - vA.z;
            const float rhs1 = cdot1 + d.s[12], rhs2 = cdot2 + d.s[13];
            l1 = -(d.s[8] * rhs1 + d.s[9] * rhs2);
            const float l2 = -(d.s[9] * rhs1 + d.s[10] * rhs2);
            LA = l1 * s1 + l2;
            LB = l1 * s2 + l2;
        }
        const float Px = pX * l1, Py = pY * l1;
        vA.x = vA.x - Px * imA; vA.y = vA.y - Py * imA;
        vA.z = vA.z - LA * iIA;
        vB.x = vB.x + Px * imB; vB.y = vB.y + Py * imB;
        vB.z = vB.z + LB * iIB;
    }
    if (d.s[16] != 0.0f) {
        const float axX = d.s[0], axY = d.s[1], a1 = d.s[6], a2 = d.s[7];
        const float cdot = (axX * (vB.x - vA.x) + axY * (vB.y - vA.y)) + a2 * vB.z - a1 * vA.z;
        const float raw = -(cdot + d.s[15]) * d.s[14];
        const float oldImpulse = d.s[17];
        const float sum = oldImpulse + raw;
        const float newImpulse = d.s[16] > 0.0f ? (sum < 0.0f ? 0.0f : sum) : (0.0f < sum ? 0.0f : sum);
        const float applied = newImpulse - oldImpulse;
        d.s[17] = newImpulse;
        const float Px = axX * applied, Py = axY * applied;
        const float LA = applied * a1, LB = applied * a2;
        vA.x = vA.x - Px * imA; vA.y = vA.y - Py * imA;
        vA.z = vA.z - LA * iIA;
        vB.x = vB.x + Px * imB; vB.y = vB.y + Py * imB;
        vB.z = vB.z + LB * iIB;
    }
    if (imA > 0.0f) vA0 = vA;
    if (imB > 0.0f) vB0 = vB;
}

__device__ __forceinline__ void motor_warm(const JointData& d, float4& v)
{
    if (d.s[0] == 0.0f) return;
    v.z = v.z + d.s[4] * d.s[0];
}

__device__ __forceinline__ void motor_solve(uint32_t index, JointData& d, float4& v, float* impulses)
{
    if (d.s[0] == 0.0f) return;
    const float lambda = (d.s[2] - v.z) * d.s[1];
    const float oldImpulse = d.s[4];
    const float newImpulse = glm_clamp(oldImpulse + lambda, -d.s[3], d.s[3]);
    d.s[4] = newImpulse;
    impulses[index] = newImpulse;
    v.z = v.z + (newImpulse - oldImpulse) * d.s[0];
}

__device__ __forceinline__ void solve_one(uint32_t k, uint32_t index, JointData& d, float4& vA, float4& vB, float iIA,
                                          float iIB, float* impulses)
{
    switch (k) {
    case K_SPRING: spring_solve(d, vA, vB, iIA, iIB); break;
    case K_REVOLUTE: revolute_solve(d, vA, vB, iIA, iIB); break;
    case K_PRISMATIC: axis_joint_solve(d, vA, vB, iIA, iIB, false); break;
    case K_SLIDER: axis_joint_solve(d, vA, vB, iIA, iIB, true); break;
    default: motor_solve(index, d, vA, impulses); break;
    }
}

// Compute tick: every type's constraint data, read-only on the bodies.
__device__ __forceinline__ void compute_tick(const DeviceWorld& w, const JointLaunch& L)
{
    for (uint32_t k = 0; k < JOINT_KINDS_DEVICE; k++)
        for (uint32_t i = threadIdx.x; i < L.count[k]; i += blockDim.x) {
            JointData d;
            const JointRec r = L.rec[k][i];
            switch (k) {
            case K_SPRING: spring_data(w, r, L.dt, d); break;
            case K_REVOLUTE: revolute_data(w, r, L.dt, d); break;
            case K_PRISMATIC: axis_joint_data(w, r, L.dt, false, d); break;
            case K_SLIDER: axis_joint_data(w, r, L.dt, true, d); break;
            default: motor_data(w, r, L.dt, L.motorImpulse, d); break;
            }
            L.data[k][i] = d;
        }
}

// A body's velocity and version in one 16-byte word of shared memory, read and written whole.
__device__ __forceinline__ float4 word_load(const float4* p)
{
    unsigned long long lo, hi;
    const uint32_t a = uint32_t(__cvta_generic_to_shared(p));
    asm volatile("{\n\t.reg .b128 d;\n\tld.relaxed.cta.shared.b128 d, [%2];\n\tmov.b128 {%0, %1}, d;\n\t}"
                 : "=l"(lo), "=l"(hi) : "r"(a) : "memory");
    return make_float4(__uint_as_float(uint32_t(lo)), __uint_as_float(uint32_t(lo >> 32)),
                       __uint_as_float(uint32_t(hi)), __uint_as_float(uint32_t(hi >> 32)));
}
__device__ __forceinline__ void word_store(float4* p, float x, float y, float z, uint32_t version)
{
    const unsigned long long lo = uint64_t(__float_as_uint(x)) | uint64_t(__float_as_uint(y)) << 32;
    const unsigned long long hi = uint64_t(__float_as_uint(z)) | uint64_t(version) << 32;
    const uint32_t a = uint32_t(__cvta_generic_to_shared(p));
    asm volatile("{\n\t.reg .b128 s;\n\tmov.b128 s, {%1, %2};\n\tst.relaxed.cta.shared.b128 [%0], s;\n\t}"
                 :: "r"(a), "l"(lo), "l"(hi) : "memory");
}

}  // namespace

// The schedule as a dataflow over per-body versions, for constraint sets whose bodies fit shared memory. A body's
// constraints act on it in one order: iteration after iteration, type after type, dense order within a type. The body
// carries the number of updates made so far in the same word as its velocity; a constraint waits until each of its
// moving bodies has had all the updates before its own (whole types of the body's degree, then its rank among the
// type's constraints on it) and nothing else, so iterations follow one another down a chain like waves. Threads take
// constraints in that order and all are resident, so the oldest one can always go. The order of every body's updates
// is the dense order's, the results are the same bit for bit.
// Bound: the longest chain of updates, some 700 cycles each (a poll, the two words, the solve, two stores). Measured on
// 80 chains of 12 revolute joints with 240 motors and 316 springs between neighbouring chains, eight iterations (92
// levels an iteration), a step's constraints: 350 us with a block barrier after every level and the velocities in
// global memory; 222 us as a dataflow in level order, a warp's share of one type far from its share of the next, so
// that iterations followed one another end to end; 104 us in dense order and equal shares of each type. Sleeping in the
// polls gave nothing.
__global__ void __launch_bounds__(JOINT_THREADS) k_joints_flow(DeviceWorld w, JointLaunch L)
{
    chain_begin();
    extern __shared__ float4 jointSmem[];
    float4* const vel = jointSmem;                                            // [bodies] vx, vy, w, version
    JointBody* const body = reinterpret_cast<JointBody*>(vel + L.bodies);     // [bodies]
    float2* const mass = reinterpret_cast<float2*>(body + L.bodies);          // [bodies] inverse mass, inverse inertia
    compute_tick(w, L);   // the block's barrier below hands the data to the warps that solve with it
    for (uint32_t i = threadIdx.x; i < L.bodies; i += blockDim.x) {
        const JointBody b = L.body[i];
        const float4 v = w.bvel[b.body];
        body[i] = b;
        mass[i] = make_float2(v.w, w.bpos[b.body].w);
        vel[i] = make_float4(v.x, v.y, v.z, __uint_as_float(0u));
    }
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    uint32_t done[JOINT_KINDS_DEVICE] = {}, rest[JOINT_KINDS_DEVICE] = {};   // iterations made; interleaving's remainder
    bool gone = false;
    // One type's pass: this warp's share of the dense order. Every type is split in the same proportions, so that what
    // one warp waits for in one type is near what it waits for in the next, and a warp at the head of a long chain can
    // be iterations ahead of one at its tail.
    auto pass = [&](auto kind, bool warm) {
        constexpr uint32_t k = kind.value;
        const uint32_t end = uint32_t(uint64_t(L.count[k]) * (warp + 1u) / warps);
        for (uint32_t first = uint32_t(uint64_t(L.count[k]) * warp / warps); first < end && !gone; first += 32u) {
            const uint32_t i = first + lane;
            bool todo = i < end;
            JointFlow f{};
            JointData d;
            uint32_t index = 0, needA = 0, needB = 0;
            bool dynA = false, dynB = false;
            float2 mA = make_float2(0.0f, 0.0f), mB = mA;
            if (todo) {
                f = L.flow[k][i];
                d = L.data[k][i];
                if (k == K_MOTOR) index = L.rec[k][i].index;
                const JointBody bA = body[f.a], bB = body[f.b];
                mA = mass[f.a];
                mB = mass[f.b];
                dynA = bA.moves != 0;
                dynB = bB.moves != 0 && k != K_MOTOR;
                needA = f.rankA;
                needB = f.rankB;
#pragma unroll
                for (uint32_t t = 0; t < JOINT_KINDS_DEVICE; t++) {
                    needA += done[t] * bA.degree[t];
                    needB += done[t] * bB.degree[t];
                }
            }
            for (uint32_t spins = 0; __any_sync(0xffffffffu, todo); spins++) {
                if (todo) {
                    float4 vA = word_load(vel + f.a), vB = word_load(vel + f.b);
                    if ((!dynA || __float_as_uint(vA.w) == needA) && (!dynB || __float_as_uint(vB.w) == needB)) {
                        vA.w = mA.x;
                        vB.w = mB.x;
                        if (warm) motor_warm(d, vA);
                        else solve_one(k, index, d, vA, vB, mA.y, mB.y, L.motorImpulse);
                        if (dynA) word_store(vel + f.a, vA.x, vA.y, vA.z, needA + 1u);
                        if (dynB) word_store(vel + f.b, vB.x, vB.y, vB.z, needB + 1u);
                        if (!warm && k == K_MOTOR) L.data[k][i].s[4] = d.s[4];
                        if (k == K_PRISMATIC || k == K_SLIDER) L.data[k][i].s[17] = d.s[17];
                        todo = false;
                    }
                }
                if (spins > SPIN_LIMIT) {
                    atomicOr(L.status, STATUS_BARRIER_TIMEOUT);
                    gone = true;
                    break;
                }
            }
        }
    };
    // Warm start: the motors (the one type with a warm start); then the velocity iterations, the types interleaved in
    // ConstraintType order.
    pass(std::integral_constant<uint32_t, K_MOTOR>{}, true);
    done[K_MOTOR] = 1;
    auto turn = [&](auto kind) {
        constexpr uint32_t k = kind.value;
        rest[k] += L.iterations[k];
        if (L.count[k] == 0 || rest[k] < L.maxIterations) return;
        rest[k] -= L.maxIterations;
        pass(kind, false);
        done[k]++;
    };
    static_assert(K_SPRING == 0 && K_REVOLUTE == 1 && K_PRISMATIC == 2 && K_SLIDER == 3 && K_MOTOR == 4, "order");
    for (uint32_t it = 0; it < L.maxIterations && !gone; it++) {
        turn(std::integral_constant<uint32_t, K_SPRING>{});
        turn(std::integral_constant<uint32_t, K_REVOLUTE>{});
        turn(std::integral_constant<uint32_t, K_PRISMATIC>{});
        turn(std::integral_constant<uint32_t, K_SLIDER>{});
        turn(std::integral_constant<uint32_t, K_MOTOR>{});
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < L.bodies; i += blockDim.x)
        if (body[i].moves) w.bvel[body[i].body] = make_float4(vel[i].x, vel[i].y, vel[i].z, mass[i].x);
}

// Larger sets: a block barrier after every level, velocities in global memory.
__global__ void __launch_bounds__(JOINT_THREADS) k_joints(DeviceWorld w, JointLaunch L)
{
    const uint32_t tid = threadIdx.x, nt = blockDim.x;
    compute_tick(w, L);
    __syncthreads();
    // Warm start: the motors (the one type with a warm start), level by level.
    for (uint32_t l = 0; l < L.levels[K_MOTOR]; l++) {
        for (uint32_t i = L.levelStart[K_MOTOR][l] + tid; i < L.levelStart[K_MOTOR][l + 1]; i += nt) {
            const uint32_t b = L.rec[K_MOTOR][i].bodyA;
            float4 v = w.bvel[b];
            motor_warm(L.data[K_MOTOR][i], v);
            w.bvel[b] = v;
        }
        __syncthreads();
    }
    // Velocity iterations, the types interleaved in ConstraintType order.
    for (uint32_t it = 0; it < L.maxIterations; it++)
        for (uint32_t k = 0; k < JOINT_KINDS_DEVICE; k++) {
            const uint64_t n = L.iterations[k];
            if (L.count[k] == 0 || (uint64_t(it + 1) * n) / L.maxIterations == (uint64_t(it) * n) / L.maxIterations)
                continue;
            for (uint32_t l = 0; l < L.levels[k]; l++) {
                for (uint32_t i = L.levelStart[k][l] + tid; i < L.levelStart[k][l + 1]; i += nt) {
                    const uint32_t a = L.rec[k][i].bodyA, b = L.rec[k][i].bodyB;
                    float4 vA = w.bvel[a], vB = w.bvel[b];
                    solve_one(k, L.rec[k][i].index, L.data[k][i], vA, vB, w.bpos[a].w, w.bpos[b].w, L.motorImpulse);
                    if (k == K_MOTOR || vA.w > 0.0f) w.bvel[a] = vA;
                    if (k != K_MOTOR && vB.w > 0.0f) w.bvel[b] = vB;
                }
                __syncthreads();
            }
        }
}

cudaError_t joints_init()
{
    return cudaFuncSetAttribute(k_joints_flow, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                int(JOINT_FLOW_BODIES * JOINT_FLOW_BODY_BYTES));
}

}  // namespace ag2d
