// Device-side types and per-particle arithmetic shared by all kernels.
//
// All translation units of liblsp are compiled with -fmad=false -prec-div=true
// -prec-sqrt=true -ftz=false: every +, -, *, / and sqrtf below rounds once, IEEE
// round-to-nearest, in source order. The per-particle expressions restate the
// reference's CPU solver operation by operation (citations at each function), so
// each particle's result matches the reference's bits when the neighbour sums are
// taken in the same order, which the grid build guarantees.
#pragma once

#include <cstdint>
#include <cstring>
#include <cuda_runtime.h>

namespace lsp {

constexpr int kTableSize = 1001;        // SPHKernel m_subdivision = 1000 (SPHKernel.cpp:4-7)
// Kernel table block: 5 tables of kTableSize, the kTableSize + 1 slot thresholds on the
// distance, then the kTableSize + 1 thresholds on the squared distance.
constexpr int kThreshOffset = 5 * kTableSize;
constexpr int kThresh2Offset = kThreshOffset + kTableSize + 1;
constexpr int kTableFloats = kThresh2Offset + kTableSize + 1;
constexpr int kMaxColliders = 64;
constexpr int kMaxIterationsCap = 1024;

// Error bits of DevStatus::error_flags.
constexpr uint32_t kErrNaN = 1u;             // non-finite position or density
constexpr uint32_t kErrNeighborOverflow = 2u; // a neighbour list exceeded its capacity
constexpr uint32_t kErrTimeout = 4u;         // a bounded grid barrier gave up
constexpr uint32_t kErrScan = 8u;            // the cell scan saw inconsistent counts

struct Collider {
    int sphere;     // 0 box, 1 sphere
    int boundary;   // 0 obstacle (keep out), 1 boundary (keep in)
    float cx, cy, cz;
    float hx, hy, hz;   // box half extents
    float radius;       // sphere radius
    float pad;
};

struct DevStatus {
    uint32_t error_flags;
    uint32_t escaped;
    uint32_t max_neighbors;
    uint32_t max_err_bits;      // float bits of the current iteration's max |density error|
    int32_t iterations;
    int32_t converged;
    int32_t warm_used;
    uint32_t barrier_count;     // grid barrier arrivals (persistent loop)
    uint32_t barrier_gen;
    uint32_t timeout_site;
    float last_ratio;
    int32_t last_k;             // logical index of the loop's last iteration (persistent loop)
    uint32_t div_unsafe;        // a predicted position left exact_div_safe's range this step
    uint32_t np_unsafe;         // a start-of-step position, velocity or density left the range
                                // where the non-pressure pass divides with div_by
    uint32_t any_first;         // a particle is on its first step
    uint32_t gave_up;           // host copy only: a barrier of the one-launch step gave up (last word)
};

struct DevParams {
    float gx, gy, gz;
    float h;            // kernel radius = grid spacing
    float h2;           // h * h, the neighbour-test bound (SPHSpatialGrid.cpp:69)
    float cut2;         // smallest float s with sqrt(s) >= h: the table cutoff on d^2
    float step;         // table division step h / 1000 (SPHKernel.cpp:134-137)
    float inv_step;     // 1 / step, rounded (only a first guess of the table slot)
    float radius;       // particle radius (collisions)
    float mass;
    float rho0;
    float stiffness;
    float neg;          // negative pressure factor
    float viscosity;
    float sigma;
    float sigma_thr;
    float restitution;
    float friction;
    float delta;        // PCISPH pressure scaling of this step
    float eta;
    float dt;
    int n;
    int keep_initial_velocity;
    int ncoll;
    int ox, oy, oz;     // grid origin in cell coordinates
    int nx, ny, nz;     // grid dimensions
    uint32_t cells;
    int nbr_cap;        // neighbour list capacity per particle
    int64_t nbr_stride; // column stride of the neighbour list (>= n)
    int min_it, max_it;
    // Batches of scenes (all zero for a single scene): the scene's first particle slot,
    // its first cell in the batch's cell table and its first collider.
    int base;
    uint32_t cell_base;
    int coll_off;
    int scene;
    int exact_tables;   // HostKernels::exact_tables
    // Factors of the kernel formulas: poly6 W, gradient and Laplacian, spiky gradient,
    // viscosity Laplacian (HostKernels::build).
    float kw, kdw, kd2w, ksdw, kvd2w;
};

// ----------------------------------------------------------------- vector ops
// Vector3D semantics (LiquidPhysics/src/Math/Vector3D.cpp): component-wise, in order.
struct V3 {
    float x, y, z;
};
__device__ __forceinline__ V3 v3(float x, float y, float z) { return V3{x, y, z}; }
__device__ __forceinline__ V3 v3(const float4& a) { return V3{a.x, a.y, a.z}; }
__device__ __forceinline__ V3 operator+(V3 a, V3 b) { return V3{a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ V3 operator-(V3 a, V3 b) { return V3{a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ V3 operator*(V3 a, float s) { return V3{a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ V3 operator/(V3 a, float s) { return V3{a.x / s, a.y / s, a.z / s}; }
__device__ __forceinline__ void operator+=(V3& a, V3 b) { a.x = a.x + b.x; a.y = a.y + b.y; a.z = a.z + b.z; }
__device__ __forceinline__ void operator*=(V3& a, float s) { a.x = a.x * s; a.y = a.y * s; a.z = a.z * s; }
// Vector3D::operator*(Vector3D) is a dot product (Vector3D.cpp:133-136).
__device__ __forceinline__ float dot(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
// Vector3D::squareMagnitude / magnitude (Vector3D.cpp:55-63).
__device__ __forceinline__ float sqmag(V3 a) { return a.x * a.x + a.y * a.y + a.z * a.z; }
__device__ __forceinline__ float mag(V3 a) { return sqrtf(a.x * a.x + a.y * a.y + a.z * a.z); }
// Vector3D::normalize (Vector3D.cpp:66-71): scale by the rounded reciprocal.
__device__ __forceinline__ void normalize(V3& a)
{
    float m = mag(a);
    if (m > 0.f) a *= (1.f / m);
}
__device__ __forceinline__ float4 f4(V3 a, float w) { return make_float4(a.x, a.y, a.z, w); }

// Correctly rounded quotients a / d from one reciprocal per denominator, after Markstein's
// method (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000
// processor", IBM J. Res. Develop. 34(1), 1990; "IA-64 and Elementary Functions", 2000,
// ch. 8): one Newton-Raphson step with fused multiply-adds turns the hardware's approximate
// reciprocal (within one ulp) into RN(1 / d), and with y = RN(1 / d) and q0 = RN(a * y),
// within one ulp of a / d, the residual r = a - d * q0 is exact and RN(q0 + r * y) is
// RN(a / d). recip_rn is checked against the IEEE reciprocal for every positive normal
// float and div_by against IEEE division on billions of pairs
// (tests/cpp/exact_div_check.cu). The theorem needs every value normal: callers use them
// only where 2^-51 <= d <= 2^28 and a is 0 or 2^-51 <= |a| <= d (exact_div_safe). A zero
// numerator gives a zero of either sign, which adds to a sum started at +0 like the IEEE
// quotient's zero does.
__device__ __forceinline__ float recip_rn(float d)
{
    float y0;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(d));
    const float e = __fmaf_rn(-d, y0, 1.f);
    return __fmaf_rn(e, y0, y0);
}
__device__ __forceinline__ float div_by(float a, float d, float y)
{
    const float q0 = __fmul_rn(a, y);
    const float r = __fmaf_rn(-d, q0, a);
    return __fmaf_rn(r, y, q0);
}
// The IEEE square root of s in the same style: the approximate reciprocal square root, then
// one correction with the exact residual s - g^2 (Markstein's square-root step). Equal to
// the IEEE square root for every float s >= 2^-102 (checked for every one on the GPU,
// tests/cpp/exact_div_check.cu); below that the residual underflows and it is not exact.
// s = 0 gives NaN where IEEE gives 0: the force pass only takes it for pairs j != i, whose
// direction is 0 / 0 = NaN either way at zero distance.
__device__ __forceinline__ float sqrt_rn(float s)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(s));
    const float g = __fmul_rn(s, y);
    const float h = __fmul_rn(0.5f, y);
    const float r = __fmaf_rn(-g, g, s);
    return __fmaf_rn(r, h, g);
}
// A density the non-pressure pass may divide by with div_by: 2^-20 <= rho <= 2^20 (so that
// with numerators 0 or at least 2^-80 in magnitude every quotient and residual stays normal).
__device__ __forceinline__ bool exact_div_density(float r) { return r >= 0x1p-20f && r <= 0x1p20f; }
// A coordinate with which every pair difference, its squared length and its quotient by the
// pair distance stay where sqrt_rn and div_by are exact: 0, or 2^-28 <= |c| <= 2^26 (nonzero
// differences of such floats are at least 2^-51, squared lengths at least 2^-102 and at most
// 3 * 2^54, distances at most 2^28).
__device__ __forceinline__ bool exact_div_safe(float c)
{
    const float a = fabsf(c);
    return a == 0.f || (a >= 0x1p-28f && a <= 0x1p26f);
}
// A velocity component with which the non-pressure pass may divide by the density with div_by: 0,
// or 2^-57 <= |c| <= 2^26, so that a nonzero difference of two is at least 2^-80 (their last places).
// Holding velocities to the positions' 2^-28 sent whole steps of 991,440 particles in motion to IEEE
// division for one component below 4e-9 m/s (258 us against 119 for the pass).
__device__ __forceinline__ bool exact_div_velocity(float c)
{
    const float a = fabsf(c);
    return a == 0.f || (a >= 0x1p-57f && a <= 0x1p26f);
}

// SPHKernel::get*Weight (SPHKernel.cpp:13-44): zero at or beyond h, else the table
// entry at trunc(d / step), with d / step rounded as IEEE division rounds it.
//
// The slot is found without a division. thr[k] (kTableSize + 1 entries, built on the
// host by bisection over floats) is the smallest distance whose IEEE quotient d / step
// truncates to at least k, so the exact slot is the largest k with thr[k] <= d. An
// approximate quotient d * (1 / step), rounded to the nearest integer by the magic-number
// addition (1.5 * 2^23), lands on that slot or the one above it (its relative error is a
// few ulp and d / step < 1001), and one comparison with thr picks the right one. The
// clamp keeps any input inside the table (slots 0..1000; NaN takes slot 1000, +inf too,
// and the cutoff zeroes the latter).
__host__ __device__ __forceinline__ int slot_guess(float d, float inv_step)
{
    float r = d * inv_step + 12582912.f;
    int32_t bits;
    memcpy(&bits, &r, 4);
    int k = bits - 0x4B400000;
    return k < 1 ? 1 : (k > kTableSize - 1 ? kTableSize - 1 : k);
}
__host__ __device__ __forceinline__ int table_slot(float d, float inv_step, const float* thr)
{
    const int k = slot_guess(d, inv_step);
    return !(d < thr[k]) ? k : k - 1;
}

// The same slot from the squared distance s = |dx|^2 for passes that need the distance only
// for the table: the IEEE square root is monotone, so sqrt(s) >= thr[k] exactly when
// s >= thr2[k] (thr2[k]: the smallest float whose rounded square root reaches thr[k], built
// on the host by bisection). The first guess uses the approximate square root (relative
// error near 2^-23, far inside the half-slot margin of the rounding guess); the comparison
// is exact, so the slot is the one sqrt(s) would give, without the IEEE square root.
__host__ __device__ __forceinline__ int table_slot_sq_from(float s, float d_guess, float inv_step, const float* thr2)
{
    const int k = slot_guess(d_guess, inv_step);
    return !(s < thr2[k]) ? k : k - 1;
}

// The kernel weights by arithmetic. Table entry k is a formula in the table distance
// d_k = k * step (HostKernels::build), and the device evaluates the same operations in the same
// order on the slot number held as a float, so the value is the table's entry bit for bit (every
// operation rounds once on both sides; every entry of every table is checked against the
// host's, tests/test_pair_weights.py). What bounds the neighbour passes is the L1 data pipe (70 to 78 % of
// its wavefronts in every neighbour pass, against 52 % of the issue slots in the PCISPH loop): a
// read of a random slot in shared memory took 2.7 wavefronts of it and a pair needed two or more
// (31 % of the loop's wavefronts, 39 % of the non-pressure pass's), while the formula takes 4 to
// 10 multiplications and additions and no memory. With the two-pair forms below, at 991,440
// particles in motion (6 iterations a step): loop 1.130 -> 0.994 ms, non-pressure pass 0.206 ->
// 0.166 ms a step; 417,792 particles: loop 0.572 -> 0.495, non-pressure 0.091 -> 0.063 ms.
//
// The slot: t = d * inv_step - 1/2 rounded to the nearest integer is trunc(d / step) unless d / step lies
// within the error of the approximate quotient of an integer. For the squared-distance form
// the relative error is at most 2^-23 (sqrt.approx) + 5 * 2^-24 (inv_step, t, and the
// roundings of the square root and the quotient that define the slot) = 4.2e-7 < kSlotEps.
// Closer than that (one pair in about 1,500) the slot comes from the threshold tables in global
// memory, as does a NaN's. kSlotHalf = (1 - kSlotEps) / 2 shifts the rounding by half the margin
// so that one comparison covers both edges of the slot: with f = t - k, the quotient is at least
// k * kSlotEps above k and (k + 1) * kSlotEps below k + 1 exactly when |f| <= kSlotHalf - k * kSlotEps.
constexpr float kSlotEps = 4.8e-7f;
constexpr float kSlotHalf = 0.5f - 0.5f * kSlotEps;
constexpr float kSlotMagic = 12582912.f;   // 1.5 * 2^23: adding it rounds to an integer

// Slot of the distance (or its approximation) `guess` as a float; at or beyond h it may be any
// number, since every weight is 0 there. kNan: a NaN is unsure (the passes that divide by the
// distance leave it out: their terms are NaN whatever the weight, and the particle itself, at
// distance 0, is a NaN of sqrt_rn in every walk of the force pass).
template <bool kNan>
__device__ __forceinline__ float slot_from(float guess, float inv_step, bool& unsure)
{
    const float t = __fmaf_rn(guess, inv_step, -kSlotHalf);
    const float k = __fadd_rn(__fadd_rn(t, kSlotMagic), -kSlotMagic);
    const float f = fabsf(__fadd_rn(t, -k)), m = __fmaf_rn(k, -kSlotEps, kSlotHalf);
    unsure = kNan ? !(f <= m) : f > m;
    return k;
}
__device__ __forceinline__ float sqrt_guess(float s)
{
    float d;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(d) : "f"(s));
    return d;
}
// tables: the kernel table block (global memory), read only in the unsure case.
__device__ __forceinline__ float slot_sq(float s, const DevParams& P, const float* __restrict__ tables)
{
    const float d = sqrt_guess(s);
    bool unsure;
    float k = slot_from<true>(d, P.inv_step, unsure);
    if (unsure) k = (float)table_slot_sq_from(s, d, P.inv_step, tables + kThresh2Offset);
    return k;
}
__device__ __forceinline__ float slot_dist(float d, const DevParams& P, const float* __restrict__ tables)
{
    bool unsure;
    float k = slot_from<false>(d, P.inv_step, unsure);
    if (unsure) k = (float)table_slot(d, P.inv_step, tables + kThreshOffset);
    return k;
}

// Table entries at slot k (HostKernels::build's expressions).
__device__ __forceinline__ float entry_w(float k, const DevParams& P)
{
    const float d = k * P.step, t = P.h2 - d * d;
    return P.kw * t * t * t;
}
__device__ __forceinline__ float entry_sdw(float k, const DevParams& P)
{
    const float s = P.h - k * P.step;
    return P.ksdw * s * s;
}
// SPHKernel::get*Weight of a squared distance (poly6, d >= h exactly when s >= cut2) and of a
// distance (spiky gradient).
__device__ __forceinline__ float weight_w(float s, const DevParams& P, const float* __restrict__ tables)
{
    const float w = entry_w(slot_sq(s, P, tables), P);
    return !(s >= P.cut2) ? w : 0.f;
}
__device__ __forceinline__ float weight_sdw(float d, const DevParams& P, const float* __restrict__ tables)
{
    const float w = entry_sdw(slot_dist(d, P, tables), P);
    return !(d >= P.h) ? w : 0.f;
}
// The non-pressure pass's three weights at one squared distance.
struct NonpressureWeights {
    float dw, d2w, vd2w;
    __device__ __forceinline__ NonpressureWeights(float s, const DevParams& P, const float* __restrict__ tables)
    {
        const float k = slot_sq(s, P, tables);
        const float d = k * P.step, t = P.h2 - d * d;
        const bool inside = !(s >= P.cut2);
        dw = inside ? P.kdw * t * t : 0.f;
        d2w = inside ? P.kd2w * t * (3.f * P.h2 - 7.f * d * d) : 0.f;
        vd2w = inside ? P.kvd2w * (P.h - d) : 0.f;
    }
};

// Two pairs at a time: sm_100's packed float operations do two IEEE single operations in one
// instruction (each half rounds as the scalar operation does), which halves the issue slots of
// the pair arithmetic.
struct F2 {
    unsigned long long v;
};
__device__ __forceinline__ F2 f2(float a, float b)
{
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ F2 f2(float a) { return f2(a, a); }
__device__ __forceinline__ float lo(F2 a)
{
    float x, y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
    (void)y;
    return x;
}
__device__ __forceinline__ float hi(F2 a)
{
    float x, y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
    (void)x;
    return y;
}
__device__ __forceinline__ F2 operator+(F2 a, F2 b)
{
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 operator*(F2 a, F2 b)
{
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c)
{
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
// a - b for finite or infinite b: a + b * (-1), one rounding.
__device__ __forceinline__ F2 operator-(F2 a, F2 b) { return fma2(b, f2(-1.f), a); }
// -(x^2 + y^2 + z^2), each sum and product rounded once. ptxas contracts an add.rn.f32x2 of a
// mul.rn.f32x2 into one fma (with -fmad=false too: seen as one-ulp differences from the scalar
// form), also where the sum is written as an fma with 1; a product that enters an fma as the
// factor of -1 stays a product, so the sum is formed negated
// (tests/cpp/pair_weights_check.cu compares it and the operations below with the scalar ones).
__device__ __forceinline__ F2 neg_sqmag(F2 x, F2 y, F2 z)
{
    const F2 m = f2(-1.f);
    return fma2(z * z, m, fma2(y * y, m, (x * m) * x));
}

// sqrt_rn, recip_rn and div_by of two pairs on negated arguments: -sqrt(s) from ns = -s,
// 1 / d from nd = -d, a / d from nd and y = recip_rn(nd) (rounding to nearest is symmetric, so
// the bits are those of the scalar forms).
__device__ __forceinline__ F2 neg_sqrt_rn(F2 ns)
{
    float a, b;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(a) : "f"(-lo(ns)));
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(b) : "f"(-hi(ns)));
    const F2 y = f2(a, b);
    const F2 g = ns * y, h = y * f2(0.5f);
    return fma2(fma2(g, g, ns), h, g);
}
__device__ __forceinline__ F2 recip_rn(F2 nd)
{
    float a, b;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(a) : "f"(-lo(nd)));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(b) : "f"(-hi(nd)));
    const F2 y0 = f2(a, b);
    return fma2(fma2(nd, y0, f2(1.f)), y0, y0);
}
__device__ __forceinline__ F2 div_by(F2 a, F2 nd, F2 y)
{
    const F2 q0 = a * y;
    return fma2(fma2(nd, q0, a), y, q0);
}
// slot_from of two pairs, of the negated distances.
template <bool kNan>
__device__ __forceinline__ F2 slot_from(F2 nguess, float inv_step, bool& unsure0, bool& unsure1)
{
    const F2 t = fma2(nguess, f2(-inv_step), f2(-kSlotHalf));
    // The constants are shared where they can be (a packed constant takes two registers).
    const F2 k = (t + f2(kSlotMagic)) - f2(kSlotMagic);
    const F2 f = t - k;
    const F2 m = fma2(k, f2(kSlotEps), f2(-kSlotHalf));   // the margin, negated
    unsure0 = kNan ? !(fabsf(lo(f)) <= -lo(m)) : fabsf(lo(f)) > -lo(m);
    unsure1 = kNan ? !(fabsf(hi(f)) <= -hi(m)) : fabsf(hi(f)) > -hi(m);
    return k;
}
__device__ __forceinline__ F2 slot_sq(F2 ns, const DevParams& P, const float* __restrict__ tables)
{
    const float d0 = sqrt_guess(-lo(ns)), d1 = sqrt_guess(-hi(ns));
    bool u0, u1;
    F2 k = slot_from<true>(f2(-d0, -d1), P.inv_step, u0, u1);
    if (u0 || u1) {
        const float* th = tables + kThresh2Offset;
        k = f2((float)table_slot_sq_from(-lo(ns), d0, P.inv_step, th),
               (float)table_slot_sq_from(-hi(ns), d1, P.inv_step, th));
    }
    return k;
}
__device__ __forceinline__ F2 slot_dist(F2 nd, const DevParams& P, const float* __restrict__ tables)
{
    bool u0, u1;
    F2 k = slot_from<false>(nd, P.inv_step, u0, u1);
    if (u0 || u1) {
        const float* th = tables + kThreshOffset;
        k = f2((float)table_slot(-lo(nd), P.inv_step, th), (float)table_slot(-hi(nd), P.inv_step, th));
    }
    return k;
}
// weight_w of two negated squared distances, weight_sdw of two negated distances.
__device__ __forceinline__ F2 weight_w(F2 ns, const DevParams& P, const float* __restrict__ tables)
{
    const F2 d = slot_sq(ns, P, tables) * f2(P.step);
    const F2 t = f2(P.h2) - d * d;
    const F2 w = f2(P.kw) * t * t * t;
    return f2(!(-lo(ns) >= P.cut2) ? lo(w) : 0.f, !(-hi(ns) >= P.cut2) ? hi(w) : 0.f);
}
__device__ __forceinline__ F2 weight_sdw(F2 nd, const DevParams& P, const float* __restrict__ tables)
{
    const F2 s = f2(P.h) - slot_dist(nd, P, tables) * f2(P.step);
    const F2 w = f2(P.ksdw) * s * s;
    return f2(!(-lo(nd) >= P.h) ? lo(w) : 0.f, !(-hi(nd) >= P.h) ? hi(w) : 0.f);
}
// NonpressureWeights of two negated squared distances.
struct NonpressureWeights2 {
    F2 dw, d2w, vd2w;
    __device__ __forceinline__ NonpressureWeights2(F2 ns, const DevParams& P, const float* __restrict__ tables)
    {
        const F2 d = slot_sq(ns, P, tables) * f2(P.step);
        const F2 t = f2(P.h2) - d * d;
        const bool in0 = !(-lo(ns) >= P.cut2), in1 = !(-hi(ns) >= P.cut2);
        const F2 a = f2(P.kdw) * t * t;
        const F2 b = f2(P.kd2w) * t * (f2(3.f * P.h2) - f2(7.f) * d * d);
        const F2 c = f2(P.kvd2w) * (f2(P.h) - d);
        dw = f2(in0 ? lo(a) : 0.f, in1 ? hi(a) : 0.f);
        d2w = f2(in0 ? lo(b) : 0.f, in1 ? hi(b) : 0.f);
        vd2w = f2(in0 ? lo(c) : 0.f, in1 ? hi(c) : 0.f);
    }
};

// ----------------------------------------------------------------- collisions
// StaticCollisionObject::resolveCollisionWithParticle (StaticCollisionObject.cpp:21-38).
__device__ __forceinline__ void resolve(V3& pos, V3& vel, V3 n, V3 point, const DevParams& P)
{
    float sep = dot(vel, n);
    if (sep < 0.f) {
        V3 vn = n * sep;
        V3 vt = vel - vn;
        vn *= -P.restitution;
        vt *= P.friction;
        vel = vn + vt;
    }
    pos = point;
}

// StaticCollisionBox (StaticCollisionBox.cpp:10-118) and StaticCollisionSphere
// (StaticCollisionSphere.cpp:10-56) detection, then resolve on contact.
__device__ __forceinline__ void collide(const Collider& o, V3& pos, V3& vel, const DevParams& P)
{
    const float r = P.radius;
    V3 c = v3(o.cx, o.cy, o.cz);
    V3 n = v3(0.f, 0.f, 0.f);
    V3 point = pos;
    bool found = false;
    if (!o.sphere) {
        V3 half = v3(o.hx, o.hy, o.hz);
        V3 dv = c - pos;
        V3 dist = v3(fabsf(dv.x), fabsf(dv.y), fabsf(dv.z));
        if (!o.boundary) {
            V3 pen = half - dist;
            pen = v3(pen.x + r, pen.y + r, pen.z + r);
            if (pen.x > 0.f && pen.y > 0.f && pen.z > 0.f) {
                found = true;
                if (pen.x <= pen.y && pen.x <= pen.z) {
                    n.x = (pos.x - c.x >= 0.f) ? 1.f : -1.f;
                    point.x = c.x + n.x * (half.x + r);
                } else if (pen.y <= pen.x && pen.y <= pen.z) {
                    n.y = (pos.y - c.y >= 0.f) ? 1.f : -1.f;
                    point.y = c.y + n.y * (half.y + r);
                } else if (pen.z <= pen.y && pen.z <= pen.x) {
                    n.z = (pos.z - c.z >= 0.f) ? 1.f : -1.f;
                    point.z = c.z + n.z * (half.z + r);
                }
            }
        } else {
            V3 pen = dist - half;
            pen = v3(pen.x + r, pen.y + r, pen.z + r);
            if (pen.x > 0.f || pen.y > 0.f || pen.z > 0.f) {
                found = true;
                if (pen.x > 0.f) {
                    n.x = (pos.x - c.x <= 0.f) ? 1.f : -1.f;
                    point.x = c.x - n.x * (half.x - r);
                }
                if (pen.y > 0.f) {
                    n.y = (pos.y - c.y <= 0.f) ? 1.f : -1.f;
                    point.y = c.y - n.y * (half.y - r);
                }
                if (pen.z > 0.f) {
                    n.z = (pos.z - c.z <= 0.f) ? 1.f : -1.f;
                    point.z = c.z - n.z * (half.z - r);
                }
                normalize(n);
            }
        }
    } else {
        float R = o.radius;
        float dist = mag(c - pos);
        float pen = o.boundary ? dist - (R - r) : (R + r) - dist;
        if (pen > 0.f) {
            found = true;
            // Contact point from the un-normalised normal (StaticCollisionSphere.cpp:44-50).
            if (!o.boundary) {
                n = pos - c;
                point = c + n * (R + r);
            } else {
                n = c - pos;
                point = c - n * (R - r);
            }
            normalize(n);
        }
    }
    if (found) resolve(pos, vel, n, point, P);
}

__device__ __forceinline__ void collide_all(const Collider* cols, int ncoll, V3& pos, V3& vel, const DevParams& P)
{
    for (int c = 0; c < ncoll; c++) collide(cols[c], pos, vel, P);
}

// Neighbour-list layout: entry k of particle i is component k & 3 of the int4 at group k >> 2,
// and each group is column-major over the particles (group g of particle i at
// ((int4*)nbr)[g * stride + i]). A reader fetches four indices with one coalesced 16-byte
// load. The unused components of a list's last group hold the particle's own index.
__device__ __forceinline__ int list_entry(const int32_t* __restrict__ nbr, int64_t stride, int64_t i, int k)
{
    return nbr[(((int64_t)(k >> 2) * stride + i) << 2) + (k & 3)];
}

// Walks particle i's neighbour list in list order, two entries per call of f, software
// pipelined: while a group's records are fetched and its pairs computed (B records at a time,
// B = 2 or 4), the next group's four indices are already in flight, so the list's DRAM latency
// overlaps the arithmetic. f(j0, record0, j1, record1, two) runs in list order and must add
// entry j0's terms before j1's, so every sum accumulates in the reference's order; when `two`
// is false (an odd last entry) the second entry is the particle itself and adds nothing.
template <int B, typename Load, typename F>
__device__ __forceinline__ void for_each_neighbor(const int32_t* __restrict__ nbr, int i, int64_t stride, int cnt,
                                                  Load load, F f)
{
    static_assert(B == 2 || B == 4, "a walk batch divides the 4-entry group");
    const int4* g = reinterpret_cast<const int4*>(nbr) + i;
    int4 cur = make_int4(i, i, i, i);
    if (cnt > 0) cur = __ldg(g);
    for (int left = cnt; left > 0; left -= 4) {   // entries of this group and after
        g += stride;
        int4 nxt = cur;
        if (left > 4) nxt = __ldg(g);
        const auto r0 = load(cur.x);
        const auto r1 = load(cur.y);
        if (B == 4) {
            const auto r2 = load(cur.z);
            const auto r3 = load(cur.w);
            f(cur.x, r0, cur.y, r1, left > 1);
            if (left > 2) f(cur.z, r2, cur.w, r3, left > 3);
        } else {
            f(cur.x, r0, cur.y, r1, left > 1);
            if (left > 2) {
                const auto r2 = load(cur.z);
                const auto r3 = load(cur.w);
                f(cur.z, r2, cur.w, r3, left > 3);
            }
        }
        cur = nxt;
    }
}

// Cell coordinate of the reference's CPU grid (SPHSpatialGrid.cpp:80-82).
__device__ __forceinline__ int cell_coord(float x, float h) { return (int)(x / h); }

__device__ __forceinline__ int id_of(const float4& p) { return __float_as_int(p.w); }

}  // namespace lsp
