// Per-particle operations of the step, shared by the single-scene kernels (sph.cu,
// pcisph.cu) and the batched kernels (batch.cu): each function computes one particle's
// result exactly as the reference CPU solver does (citations at each function), so both
// kernel families produce the same bits.
#pragma once

#include "lsp_device.cuh"
#include "lsp_kernels.h"

namespace lsp {

// Cell key of a position inside the scene's grid box: the CPU grid's cell (int)(x / h)
// per axis (SPHSpatialGrid.cpp:80-82), clamped into the box, ordered x slowest and z
// fastest, plus the scene's first cell in a batch.
__device__ __forceinline__ uint32_t cell_key(const DevParams& P, const float4& p, bool& escaped, bool& bad)
{
    bad = !(isfinite(p.x) && isfinite(p.y) && isfinite(p.z));
    int c[3] = {cell_coord(p.x, P.h), cell_coord(p.y, P.h), cell_coord(p.z, P.h)};
    const int o[3] = {P.ox, P.oy, P.oz};
    const int d[3] = {P.nx, P.ny, P.nz};
    escaped = false;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        int v = c[a];
        if (v < o[a]) { v = o[a]; escaped = true; }
        if (v > o[a] + d[a] - 1) { v = o[a] + d[a] - 1; escaped = true; }
        c[a] = v - o[a];
    }
    return P.cell_base + (uint32_t)(((uint32_t)c[0] * (uint32_t)P.ny + (uint32_t)c[1]) * (uint32_t)P.nz + (uint32_t)c[2]);
}

// Cells the neighbour search of a particle at x visits, relative to the grid box
// (SPHSpatialGrid.cpp:44-50).
__device__ __forceinline__ void search_box(const DevParams& P, V3 x, int (&lo_)[3], int (&hi_)[3])
{
    const float h = P.h;
    const int a0[3] = {(int)((x.x - h) / h), (int)((x.y - h) / h), (int)((x.z - h) / h)};
    const int a1[3] = {(int)((x.x + h) / h), (int)((x.y + h) / h), (int)((x.z + h) / h)};
    const int o[3] = {P.ox, P.oy, P.oz};
    const int d[3] = {P.nx, P.ny, P.nz};
#pragma unroll
    for (int a = 0; a < 3; a++) {
        // Both ends clamped into the box: a particle outside it searches the edge cell
        // that holds every clamped particle.
        lo_[a] = min(max(a0[a], o[a]), o[a] + d[a] - 1) - o[a];
        hi_[a] = min(max(a1[a], o[a]), o[a] + d[a] - 1) - o[a];
    }
}

// Tests candidates [beg, beg + len), len <= 32, of a particle at xi: bit b of the result is
// candidate last - b (`above`: the float after h^2). Reads U at a time, up to U - 1 past the end.
template <int U>
__device__ __forceinline__ uint32_t scan_row(const float4* pos, V3 xi, float above, int beg, int len, int& last)
{
    const float4* p = pos + beg;
    uint32_t bits = 0;
    for (int k = 0; k < len; k += U, p += U) {
#pragma unroll
        for (int u = 0; u < U; u++) {
            const float s = sqmag(xi - v3(p[u]));
            bits = __funnelshift_l(__float_as_uint(s - above), bits, 1);
        }
    }
    const int over = -len & (U - 1);   // candidates tested past the end
    last = beg + len + over - 1;
    return bits & (0xffffffffu << over);
}

// scan_row over candidates staged as x[], y[], z[] (kStagePitch apart): those in [o, o + len), two at
// a time from the even place at or below o, len <= 32 - (o & 1). Reads up to 3 past the end. `last`
// is the staged index of the mask's bit 0. above - s is formed negated, s - above, for its sign.
__device__ __forceinline__ uint32_t scan_staged(const float* st, F2 nx, F2 ny, F2 nz, F2 nabove, int o, int len, int& last)
{
    const int c = o & ~1, n = len + (o & 1);
    const float* p = st + c;
    uint32_t bits = 0;
    for (int k = 0; k < n; k += 4, p += 4) {
#pragma unroll
        for (int u = 0; u < 4; u += 2) {
            const float2 x = *reinterpret_cast<const float2*>(p + u);
            const float2 y = *reinterpret_cast<const float2*>(p + u + kStagePitch);
            const float2 z = *reinterpret_cast<const float2*>(p + u + 2 * kStagePitch);
            const F2 s = fma2(neg_sqmag(f2(x.x, x.y) + nx, f2(y.x, y.y) + ny, f2(z.x, z.y) + nz), f2(-1.f), nabove);
            bits = __funnelshift_l(__float_as_uint(lo(s)), bits, 1);
            bits = __funnelshift_l(__float_as_uint(hi(s)), bits, 1);
        }
    }
    const int over = -n & 3;
    last = c + n + over - 1;
    if (o & 1) bits &= ~(1u << (last - c));
    return bits & (0xffffffffu << over);
}

// Start-of-step neighbour list and density sum of particle i: every j with
// |x_i - x_j|^2 <= h^2, including i, in the reference's order (SPHSpatialGrid::findNeighborParticles,
// SPHSpatialGrid.cpp:39-76): cell ranges from (x -+ h) / h per axis, x then y rows, each row a
// contiguous z-run of the sorted array. Stores at most nbr_cap entries in list_entry's layout
// (the last group filled up with i itself) and returns the true count; *wsum is the sum of W
// over the accepted pairs in list order, from their squared distances (|x_i - x_j|^2 equals
// |x_j - x_i|^2 bit for bit).
//
// Two phases. The scan tests the rows' candidates, 32 at a time, into bit masks without a
// branch: s - next_up(h^2) is negative exactly when s <= h^2 (a NaN's sign is clear), and a
// funnel shift appends that sign to the mask, first candidate highest. The masks wait in a
// column of shared memory per thread (col, entries `pitch` apart). Then the accepted entries are taken from the masks four
// at a time, by all lanes in step: their positions are fetched again, W is evaluated for two
// pairs at a time and the group of four goes out as one 16-byte store that coalesces over the
// lanes. A scan that handles each accepted candidate at once runs that branch for 10 of 32 lanes
// on average and scatters its 4-byte stores over as many lines, and its lists had to be regrouped
// by the next pass. Build 0.254 -> 0.229 ms, non-pressure pass without the regrouping and loop
// with the filled-up groups 1.16 -> 1.11 ms a step at 991,440 particles; 12,000 particles: build
// 39 -> 21 us.
//
// The scan is bound by the L1 data pipe: a candidate's 16-byte load by lanes in four or five cells
// takes four to eight wavefronts (84 % of the pipe's rate). kWarp (every lane calls, `valid` or not;
// stage: kStageFloats of the warp): a warp whose particles all search the same rows, as four of five
// do, first copies the candidates of a row, all lanes' ranges together, to shared memory as x[], y[],
// z[]; the lanes then read two candidates' coordinate by an 8-byte load, which is half the
// wavefronts, and test them with packed arithmetic; a row of more than kStage candidates goes through
// in pieces. Build 229 -> 182 us at 991,440 particles, 80 -> 58 at 250,000, 31 -> 29 at 102,400;
// 174, 57 and 29 in blocks of 128 instead of 256 threads. Slower: a warp's two row groups one after
// the other (216, 81, 31), a row's table entries fetched a row ahead (179, 58, 31). 64 or 128 staged
// candidates make no difference.
//
// Rows of more than 32 particles (kernels wider than about 4 radii, compressed fluid) need more masks
// than a column holds. A full column is emptied in the same groups of four, by a whole warp at once
// where it scans together: `room` counts the free masks that every lane has at least, so that rows
// of usual length cost one vote in six. Emptied one entry at a time, 64,000 particles with 117
// neighbours took 426 us and with 207 neighbours 795, now 119 and 248; 250,047 with 458 neighbours
// 5.42 -> 1.16 ms. A check per lane instead of the warp's took 264 us at 117 neighbours; scanning
// that can be left and resumed, so that the groups are taken in one place, 92 us there, but 193 us
// instead of 180 at 991,440 particles with 29.
template <bool kWarp = false>
__device__ __forceinline__ int neighbors_one(const DevParams& P, const float4* __restrict__ pos,
                                             const uint32_t* __restrict__ cell_start, int32_t* __restrict__ nbr,
                                             int i, const float* __restrict__ tables, uint2* col, int pitch,
                                             float* wsum, float* stage = nullptr, bool valid = true)
{
    const V3 xi = v3(pos[i]);
    int lo_[3], hi_[3];
    search_box(P, xi, lo_, hi_);
    const float above = __uint_as_float(__float_as_uint(P.h2) + 1u);   // the next float above h^2
    int4* out = reinterpret_cast<int4*>(nbr) + i;
    const int64_t stride = P.nbr_stride;
    float sum = 0.f;
    int stored = 0, pending = 0, chunks = 0;   // entries taken from the masks, entries still in them
    uint32_t m = 0;
    int last = 0;   // candidate of the mask's bit 0
    int next = 0;   // next chunk to take
    auto take = [&]() {
        if (m == 0u) {
            const uint2 e = col[next * pitch];
            next++;
            last = (int)e.x;
            m = e.y;
        }
        const int b = 31 - __clz((int)m);
        m ^= 1u << b;
        return last - b;
    };
    auto keep = [&](uint32_t bits, int last_q) {
        if (!bits) return;
        col[chunks * pitch] = make_uint2((uint32_t)last_q, bits);
        chunks++;
        pending += __popc(bits);
    };
    // Takes the waiting entries, four at a time, while at least `least` of them wait (1: all of them,
    // the last group filled up).
    auto emit = [&](int least) {
        for (; pending >= least; out += stride) {
            const int left = pending;
            int4 q = make_int4(i, i, i, i);
            q.x = take();
            if (left > 1) q.y = take();
            if (left > 2) q.z = take();
            if (left > 3) q.w = take();
            const float4 a = pos[q.x], b = pos[q.y], c = pos[q.z], e = pos[q.w];
            if (stored < P.nbr_cap) *out = q;
            const F2 w0 = weight_w(neg_sqmag(f2(a.x - xi.x, b.x - xi.x), f2(a.y - xi.y, b.y - xi.y), f2(a.z - xi.z, b.z - xi.z)),
                                   P, tables);
            const F2 w1 = weight_w(neg_sqmag(f2(c.x - xi.x, e.x - xi.x), f2(c.y - xi.y, e.y - xi.y), f2(c.z - xi.z, e.z - xi.z)),
                                   P, tables);
            sum += lo(w0);
            if (left > 1) sum += hi(w0);
            if (left > 2) sum += lo(w1);
            if (left > 3) sum += hi(w1);
            stored += min(left, 4);
            pending -= min(left, 4);
        }
    };
    // Makes room in the column: takes the whole groups of the waiting entries; the masks of the up to
    // three that are left move to its front.
    auto drain = [&]() {
        emit(4);
        int kept = 0;
        if (m) col[kept++ * pitch] = make_uint2((uint32_t)last, m);
        for (; next < chunks; next++) col[kept++ * pitch] = col[next * pitch];
        m = 0u;
        next = 0;
        chunks = kept;
    };
    valid = valid && lo_[2] <= hi_[2];
    bool together = false;
    if (kWarp) {
        const uint32_t all = 0xffffffffu;
        const uint32_t active = __ballot_sync(all, valid);
        const int lead = active ? __ffs((int)active) - 1 : 0;   // the others compare their rows with its
        const int x0 = __shfl_sync(all, lo_[0], lead), x1 = __shfl_sync(all, hi_[0], lead);
        const int y0 = __shfl_sync(all, lo_[1], lead), y1 = __shfl_sync(all, hi_[1], lead);
        together = __all_sync(all, !valid || (lo_[0] == x0 && hi_[0] == x1 && lo_[1] == y0 && hi_[1] == y1)) && active;
        if (together) {
            const int lane = threadIdx.x & 31;
            const F2 nx = f2(-xi.x), ny = f2(-xi.y), nz = f2(-xi.z), nabove = f2(-above);
            int room = kScanChunks;   // masks that every lane's column still holds, at least
            for (int cx = x0; cx <= x1; cx++) {
                for (int cy = y0; cy <= y1; cy++) {
                    const uint32_t row = P.cell_base + ((uint32_t)cx * (uint32_t)P.ny + (uint32_t)cy) * (uint32_t)P.nz;
                    int beg = 0, end = 0;
                    if (valid) {
                        beg = (int)cell_start[row + lo_[2]];
                        end = (int)cell_start[row + hi_[2] + 1];
                    }
                    const int ub = __reduce_min_sync(all, valid ? beg : 0x7fffffff), ue = __reduce_max_sync(all, end);
                    for (int from = ub; from < ue; from += kStage) {
                        const int staged = min(ue - from, kStage);
                        const int to = min(end - from, staged);   // this lane's candidates: [o, to)
                        int o = max(beg - from, 0);
                        const int masks = (staged + 32) >> 5;   // most that a lane adds
                        if (room < masks) {
                            room = kScanChunks - __reduce_max_sync(all, chunks);
                            if (room < masks) {
                                drain();
                                room = kScanChunks - 3;
                            }
                        }
                        room -= masks;
                        for (int k = lane; k < staged; k += 32) {
                            const float4 p = pos[from + k];
                            stage[k] = p.x;
                            stage[k + kStagePitch] = p.y;
                            stage[k + 2 * kStagePitch] = p.z;
                        }
                        __syncwarp();
                        while (o < to) {
                            const int len = min(to - o, 32 - (o & 1));
                            int last_o;
                            const uint32_t bits = scan_staged(stage, nx, ny, nz, nabove, o, len, last_o);
                            keep(bits, from + last_o);
                            o += len;
                        }
                        __syncwarp();
                    }
                }
            }
        }
    }
    if (!together && valid) {
        for (int cx = lo_[0]; cx <= hi_[0]; cx++) {
            for (int cy = lo_[1]; cy <= hi_[1]; cy++) {
                const uint32_t row = P.cell_base + ((uint32_t)cx * (uint32_t)P.ny + (uint32_t)cy) * (uint32_t)P.nz;
                const int end = (int)cell_start[row + hi_[2] + 1];
                for (int beg = (int)cell_start[row + lo_[2]]; beg < end; beg += 32) {
                    if (chunks == kScanChunks) drain();
                    int last_q;
                    const uint32_t bits = scan_row<4>(pos, xi, above, beg, min(end - beg, 32), last_q);
                    keep(bits, last_q);
                }
            }
        }
    }
    emit(1);
    *wsum = sum;
    return stored;
}

__device__ __forceinline__ uint32_t lanemask_lt()
{
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Warp-aggregated histogram of cell keys: one atomic per distinct key in the warp; lanes
// with the same key take consecutive slots in lane order. All 32 lanes must call it.
__device__ __forceinline__ uint32_t hist_slot(uint32_t k, bool valid, uint32_t* hist)
{
    const int lane = threadIdx.x & 31;
    uint32_t peers = __match_any_sync(0xffffffffu, k);
    uint32_t leader = __ffs(peers) - 1;
    uint32_t rank = __popc(peers & lanemask_lt());
    uint32_t base = 0;
    if (valid && lane == (int)leader) base = atomicAdd(&hist[k], (uint32_t)__popc(peers));
    base = __shfl_sync(0xffffffffu, base, leader);
    return base + rank;
}

// Escaped and non-finite positions of the warp, one atomic each. All 32 lanes call it.
__device__ __forceinline__ void record_key_flags(bool valid, bool escaped, bool bad, DevStatus* st)
{
    uint32_t esc = __ballot_sync(0xffffffffu, valid && escaped);
    uint32_t nan = __ballot_sync(0xffffffffu, valid && bad);
    if ((threadIdx.x & 31) == 0) {
        if (esc) atomicAdd(&st->escaped, (uint32_t)__popc(esc));
        if (nan) atomicOr(&st->error_flags, kErrNaN);
    }
}

// The stored neighbour count never exceeds the list capacity, so later passes stay inside
// the list even in an overflowed step; the true count only feeds the step's maximum and the
// overflow flag (one atomic per warp). All 32 lanes call it.
__device__ __forceinline__ void record_neighbor_count(const DevParams& P, int c, bool valid, DevStatus* st)
{
    uint32_t m = valid ? (uint32_t)c : 0u;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, off));
    if ((threadIdx.x & 31) == 0 && m > 0) {
        atomicMax(&st->max_neighbors, m);
        if (m > (uint32_t)P.nbr_cap) atomicOr(&st->error_flags, kErrNeighborOverflow);
    }
}

// Density, pressure and {v, rho} record of particle i from its neighbour count and sum of W
// (SPHSolver::calcParticleDensityPressure, CPU branch, SPHSolver.cpp:442-463).
// xpf (SPH, else null) gets {x, p / rho^2}, what the pressure force needs of a neighbour.
__device__ __forceinline__ void store_density(const DevParams& P, int i, int c, float sum, const float4* pos,
                                              const float4* vel, int32_t* count, float* rho, float* pres, float4* vrho,
                                              float4* xpf, DevStatus* st)
{
    count[i] = min(c, P.nbr_cap);
    const float r = P.mass * sum;
    float pr = P.stiffness * (r - P.rho0);
    if (pr < 0.f) pr *= P.neg;
    rho[i] = r;
    pres[i] = pr;
    const float4 v = vel[i];
    vrho[i] = make_float4(v.x, v.y, v.z, r);
    if (xpf) xpf[i] = f4(v3(pos[i]), pr / (r * r));
    if (!exact_div_density(r)) atomicOr(&st->np_unsafe, 1u);
}

// Stores a particle's persistent state (x|id, v|first, v_half|p1, v_half_old|p2) at its sorted slot.
__device__ __forceinline__ void store_sorted(const GridBuildArgs& g, uint32_t dest, int id, uint32_t key, float4 x, float4 v,
                                             float4 half, float4 old)
{
    g.pos_out[dest] = x;
    g.vel_out[dest] = v;
    // The non-pressure pass divides pair terms by densities with div_by while every position
    // and velocity of the step is in range.
    if (!(exact_div_safe(x.x) && exact_div_safe(x.y) && exact_div_safe(x.z) && exact_div_velocity(v.x) &&
          exact_div_velocity(v.y) && exact_div_velocity(v.z)))
        atomicOr(&g.status->np_unsafe, 1u);
    if (v.w != 0.f) atomicOr(&g.status->any_first, 1u);
    g.half_out[dest] = half;
    g.old_out[dest] = old;
    g.slot_of_id[id] = (int32_t)dest;
    g.sorted_key[dest] = key;
}

// Final slot of the particle scattered to p = cell start + number of particles of the same cell
// with a smaller caller id. Then moves the particle's persistent state.
constexpr int kMaxCellOccupancy = 4096;
__device__ __forceinline__ void rank_gather_one(const GridBuildArgs& g, int p)
{
    auto ld = [](const auto* q) { return __ldg(q); };
    const int2 e = ld(g.tmp + p);
    const uint32_t k = ld(g.key + e.x);
    const uint32_t beg = ld(g.cell_start + k), end = ld(g.cell_start + k + 1);
    uint32_t rank = 0;
    if (end - beg <= (uint32_t)kMaxCellOccupancy) {
        for (uint32_t q = beg; q < end; q++) rank += ld(g.tmp + q).y < e.y ? 1u : 0u;
    } else {
        rank = (uint32_t)p - beg;   // order inside an overfull cell is not the reference's
        atomicOr(&g.status->error_flags, kErrScan);
    }
    const uint32_t dest = beg + rank;
    store_sorted(g, dest, e.y, k, __ldg(g.pos_in + e.x), __ldg(g.vel_in + e.x), __ldg(g.half_in + e.x),
                 __ldg(g.old_in + e.x));
    if (g.hist_out) g.hist_out[dest] = __ldg(g.hist_in + e.x);
}

// SPHSolver::accumulateNonPressureForces, CPU branch (SPHSolver.cpp:201-248). The
// reference walks the list up to three times (normal, colour Laplacian when the normal
// exceeds the threshold, viscosity); each sum is independent, so one walk computes all
// three with the same per-sum rounding. kGrad adds |grad rho|, a warm-start feature. The
// distance serves only the weights (the normal sums the unnormalised difference), so the
// slot comes from the squared distance.
//
// With kExactDiv its seven quotients by the neighbour density per pair come from one
// reciprocal of rho_j (recip_rn, div_by), two pairs at a time: the same bits while the step's
// positions, velocities and densities are in range (DevStatus::np_unsafe clear) and the tables'
// entries are (DevParams::exact_tables), since every numerator is then 0 or at least 2^-80 in
// magnitude (nonpressure_one chooses). The particle itself then adds a zero to the viscosity
// sum, which starts at +0 and is left unchanged, so it needs no test.
__device__ __forceinline__ V3 nonpressure_force(const DevParams& P, float rhoi, V3 normal, float lap, V3 visc)
{
    V3 F = v3(0.f, 0.f, 0.f);
    F += v3(P.gx, P.gy, P.gz) * rhoi;
    normal *= P.mass;
    float len = mag(normal);
    if (len > P.sigma_thr) F += (normal / len) * (-P.sigma * lap * P.mass);
    visc *= P.viscosity * P.mass;
    F += visc;
    return F;
}
struct NonpressureRec {
    float4 x, vr;   // position; velocity and density ({v, rho}, StepBuffers::vrho)
};
// The terms of one pair with IEEE division, and of two pairs with div_by (the halves of the F2).
// grad: the warm-start feature's (rho_j - rho_i) / rho_j grad W_ij.
struct NonpressureTerms {
    V3 normal, visc, grad;
    float lap;
};
template <bool kGrad>
__device__ __forceinline__ NonpressureTerms nonpressure_term(const DevParams& P, const float* __restrict__ tables, V3 xi,
                                                             V3 vi, float rhoi, const NonpressureRec& r)
{
    NonpressureTerms t;
    const V3 dir = xi - v3(r.x);
    // |x_i - x_j|^2 equals |x_j - x_i|^2 bit for bit
    const NonpressureWeights at(sqmag(dir), P, tables);
    t.normal = dir * at.dw / r.vr.w;
    t.lap = at.d2w / r.vr.w;
    t.visc = ((v3(r.vr) - vi) / r.vr.w) * at.vd2w;
    if (kGrad) t.grad = dir * (at.dw * ((r.vr.w - rhoi) / r.vr.w));
    return t;
}
struct NonpressureTerms2 {
    F2 nx, ny, nz, lap, vx, vy, vz, gx, gy, gz;
};
template <bool kGrad>
__device__ __forceinline__ NonpressureTerms2 nonpressure_pair(const DevParams& P, const float* __restrict__ tables, V3 xi,
                                                              V3 vi, float rhoi, const NonpressureRec& r0,
                                                              const NonpressureRec& r1)
{
    NonpressureTerms2 t;
    const F2 dx = f2(xi.x - r0.x.x, xi.x - r1.x.x), dy = f2(xi.y - r0.x.y, xi.y - r1.x.y),
             dz = f2(xi.z - r0.x.z, xi.z - r1.x.z);
    const NonpressureWeights2 at(neg_sqmag(dx, dy, dz), P, tables);
    const F2 nrho = f2(-r0.vr.w, -r1.vr.w);
    const F2 y = recip_rn(nrho);
    auto q = [&](F2 a) { return div_by(a, nrho, y); };
    t.nx = q(dx * at.dw);
    t.ny = q(dy * at.dw);
    t.nz = q(dz * at.dw);
    t.lap = q(at.d2w);
    t.vx = q(f2(r0.vr.x - vi.x, r1.vr.x - vi.x)) * at.vd2w;
    t.vy = q(f2(r0.vr.y - vi.y, r1.vr.y - vi.y)) * at.vd2w;
    t.vz = q(f2(r0.vr.z - vi.z, r1.vr.z - vi.z)) * at.vd2w;
    if (kGrad) {
        const F2 g = at.dw * q(f2(r0.vr.w - rhoi, r1.vr.w - rhoi));
        t.gx = dx * g;
        t.gy = dy * g;
        t.gz = dz * g;
    }
    return t;
}
template <bool kGrad, bool kExactDiv>
__device__ __forceinline__ void nonpressure_walk(const DevParams& P, const StepBuffers& b, int i)
{
    const V3 xi = v3(b.pos[i]);
    const V3 vi = v3(b.vel[i]);
    const float rhoi = b.rho[i];
    V3 normal = v3(0.f, 0.f, 0.f);
    V3 visc = v3(0.f, 0.f, 0.f);
    V3 grad = v3(0.f, 0.f, 0.f);
    float lap = 0.f;
    auto one = [&](int j, const NonpressureRec& r) {
        const NonpressureTerms t = nonpressure_term<kGrad>(P, b.tables, xi, vi, rhoi, r);
        normal += t.normal;
        lap += t.lap;
        if (j != i) visc += t.visc;
        if (kGrad) grad += t.grad;
    };
    auto pair = [&](int j0, const NonpressureRec& r0, int j1, const NonpressureRec& r1, bool two) {
        if (!kExactDiv) {
            one(j0, r0);
            if (two) one(j1, r1);
            return;
        }
        const NonpressureTerms2 t = nonpressure_pair<kGrad>(P, b.tables, xi, vi, rhoi, r0, r1);
        normal += v3(lo(t.nx), lo(t.ny), lo(t.nz));
        lap += lo(t.lap);
        visc += v3(lo(t.vx), lo(t.vy), lo(t.vz));
        if (kGrad) grad += v3(lo(t.gx), lo(t.gy), lo(t.gz));
        if (two) {
            normal += v3(hi(t.nx), hi(t.ny), hi(t.nz));
            lap += hi(t.lap);
            visc += v3(hi(t.vx), hi(t.vy), hi(t.vz));
            if (kGrad) grad += v3(hi(t.gx), hi(t.gy), hi(t.gz));
        }
    };
    for_each_neighbor<2>(b.nbr, i, P.nbr_stride, __ldg(b.nbr_count + i),
                         [&](int j) { return NonpressureRec{b.pos[j], b.vrho[j]}; }, pair);
    if (kGrad) b.gradrho[i] = P.mass * mag(grad);
    b.force[i] = f4(nonpressure_force(P, rhoi, normal, lap, visc), rhoi);
}
template <bool kGrad>
__device__ __forceinline__ void nonpressure_one(const DevParams& P, const StepBuffers& b, int i)
{
    if (P.exact_tables && *(const volatile uint32_t*)&b.status->np_unsafe == 0u)
        nonpressure_walk<kGrad, true>(P, b, i);
    else
        nonpressure_walk<kGrad, false>(P, b, i);
}

// SPHParticle::integrate (SPHParticle.cpp:30-44) then SPHSolver::handleCollisions
// (SPHSolver.cpp:337-355) for one particle with total force F: x and half are moved on, v and old
// set; first is the first-step flag.
__device__ __forceinline__ void integrate_motion(const DevParams& P, const Collider* cols, V3 F, float rho, V3& x, V3& v,
                                                 float& first, V3& half, V3& old)
{
    V3 acc = F / rho;
    if (first != 0.f) {
        half = v - acc * P.dt / 2.f;
        first = 0.f;
    }
    old = half;
    half = v3(half.x + acc.x * P.dt, half.y + acc.y * P.dt, half.z + acc.z * P.dt);
    x = v3(x.x + half.x * P.dt, x.y + half.y * P.dt, x.z + half.z * P.dt);
    collide_all(cols, P.ncoll, x, half, P);
    v = (old + half) / 2.f;
}
// integrate_motion on the stored state. With add_pforce the PCISPH pressure force is added first
// (PCISPHSolver.cpp:166-169).
__device__ __forceinline__ void integrate_one(const DevParams& P, const StepBuffers& b, int i, int add_pforce)
{
    float4 p4 = b.pos[i], v4 = b.vel[i], h4 = b.half[i], o4 = b.old[i];
    V3 F = v3(b.force[i]);
    if (add_pforce) F += v3(b.pforce[i]);
    V3 x = v3(p4), v = v3(v4), half = v3(h4), old;
    float first = v4.w;
    integrate_motion(P, b.colliders + P.coll_off, F, b.rho[i], x, v, first, half, old);
    b.pos[i] = f4(x, p4.w);
    b.vel[i] = f4(v, first);
    b.half[i] = f4(half, h4.w);
    b.old[i] = f4(old, o4.w);
    if (b.hist) {
        // Warm-start pressure history: (p_n, p_{n-1}, p_{n-2}) for the next step's features.
        float4 hs = b.hist[i];
        b.hist[i] = make_float4(b.pres[i], hs.x, hs.y, 0.f);
    }
}

// PCISPHSolver.cpp:67-95 for one particle: predicted half velocity and position under F + Fp. The
// force pass divides by pair distances with div_by while every prediction of the step stays in its
// exact range; one position outside switches it to IEEE division (DevStatus::div_unsafe).
__device__ __forceinline__ void predict_motion(const DevParams& P, const Collider* cols, DevStatus* st, V3 F, V3 Fp,
                                               float rho, V3 x, V3 v, float first, V3 half, V3& px, V3& ph)
{
    V3 acc = (F + Fp) / rho;
    if (first != 0.f) half = v - acc * P.dt / 2.f;
    ph = half + acc * P.dt;
    px = x + ph * P.dt;
    collide_all(cols, P.ncoll, px, ph, P);
    if (!(exact_div_safe(px.x) && exact_div_safe(px.y) && exact_div_safe(px.z))) atomicOr(&st->div_unsafe, 1u);
}
// predict_motion on the stored state. Iteration 0 starts from p = 0, F_p = 0 (:58-62).
// aproximateVelocity (:96, SPHParticle.cpp:46-49) sets v = (v_half_old + v_half)/2; within a step
// it is idempotent, so it is applied in iteration 0 only, after the prediction has read v.
__device__ __forceinline__ void pci_predict_one(const DevParams& P, const StepBuffers& b, int i, int iteration,
                                                float4* ppos)
{
    float4 v4 = b.vel[i];
    const V3 half = v3(b.half[i]);
    const V3 Fp = iteration == 0 ? v3(0.f, 0.f, 0.f) : v3(b.pforce[i]);
    V3 px, ph;
    predict_motion(P, b.colliders + P.coll_off, b.status, v3(b.force[i]), Fp, b.rho[i], v3(b.pos[i]), v3(v4), v4.w, half,
                   px, ph);
    ppos[i] = f4(px, 0.f);
    b.phalf[i] = f4(ph, 0.f);
    if (iteration == 0 && !P.keep_initial_velocity) {
        V3 v = (v3(b.old[i]) + half) / 2.f;
        b.vel[i] = f4(v, v4.w);
    }
}

// W of the pairs of a particle at xi with particles at p and q.
__device__ __forceinline__ F2 density_pair(const DevParams& P, const float* __restrict__ tables, V3 xi, float4 p, float4 q)
{
    return weight_w(neg_sqmag(f2(p.x - xi.x, q.x - xi.x), f2(p.y - xi.y, q.y - xi.y), f2(p.z - xi.z, q.z - xi.z)), P,
                    tables);
}
// Sum of W over particle i's list at the positions x (a W of exactly 0 or more each: adding the
// +0 of a masked second entry changes no bit).
__device__ __forceinline__ float density_sum(const DevParams& P, const StepBuffers& b, const float4* x, int i)
{
    const V3 xi = v3(x[i]);
    float sum = 0.f;
    for_each_neighbor<4>(b.nbr, i, P.nbr_stride, __ldg(b.nbr_count + i), [&](int j) { return x[j]; },
                         [&](int, float4 p, int, float4 q, bool two) {
                             const F2 w = density_pair(P, b.tables, xi, p, q);
                             sum += lo(w);
                             if (two) sum += hi(w);
                         });
    return sum;
}

// PCISPHSolver.cpp:100-126 for one particle from its sum of W: predicted density, error and the
// pressure p moved on.
__device__ __forceinline__ void pressure_update(const DevParams& P, float sum, float& pd, float& er, float& p)
{
    pd = P.mass * sum;
    er = pd - P.rho0;
    float pp = P.delta * er;
    if (pp < 0.f) {
        er *= P.neg;
        pp *= P.neg;
    }
    p += pp;
}
// |error| for the maximum: 0 for NaN, which the reference's std::max ignores.
__device__ __forceinline__ float error_magnitude(float er)
{
    const float a = fabsf(er);
    return a == a ? a : 0.f;
}
// pressure_update on the stored state; returns the error's magnitude.
__device__ __forceinline__ float pci_density_finish(const DevParams& P, const StepBuffers& b, int i, int iteration,
                                                    float4* ppos, float sum)
{
    float pd, er, p = iteration == 0 ? 0.f : b.pres[i];
    pressure_update(P, sum, pd, er, p);
    b.prho[i] = pd;
    b.err[i] = er;
    b.pres[i] = p;
    // p / rho*^2, the per-particle factor of the pressure force, rides in x*.w so the force
    // pass fetches a neighbour's position and factor in one 16-byte load. Other threads
    // read only x*.xyz of this element during this pass.
    reinterpret_cast<float*>(ppos + i)[3] = p / (pd * pd);
    return error_magnitude(er);
}
__device__ __forceinline__ float pci_density_one(const DevParams& P, const StepBuffers& b, int i, int iteration,
                                                 float4* ppos)
{
    return pci_density_finish(P, b, i, iteration, ppos, density_sum(P, b, ppos, i));
}

// PCISPHSolver.cpp:129-150 for one particle. s = p / rho*^2 is the per-particle factor the
// reference recomputes per pair; the prefactor uses the current density rho_i. The pair
// distance is an IEEE square root and the direction (x_i - x_j) / d three IEEE quotients;
// with kExactDiv they come from sqrt_rn and one reciprocal of d (recip_rn, div_by), the same
// bits for the predicted positions the step's predict passes found safe
// (DevStatus::div_unsafe clear).
// F_p from the sum over the pairs; a NaN sum counts as no force (PCISPHSolver.cpp:144-149).
__device__ __forceinline__ V3 pci_pressure_force(const DevParams& P, float rho, V3 pf)
{
    pf *= -(P.mass * rho);
    if (isnan(pf.x)) pf = v3(0.f, 0.f, 0.f);
    return pf;
}
// The terms of one pair with IEEE operations, and of two pairs with the exact forms. A particle's
// own entry gives NaN (0 / 0) and is left out by the caller.
__device__ __forceinline__ V3 pci_force_term(const DevParams& P, const float* __restrict__ tables, V3 xi, float tf,
                                             float4 p)
{
    // |x_i - x_j| rounds exactly like the reference's |x_j - x_i| (the squares are equal), so one
    // difference serves both.
    const V3 dq = xi - v3(p);
    const float d = mag(dq);
    const V3 dir = dq / d;
    return dir * weight_sdw(d, P, tables) * (tf + p.w);
}
struct V3x2 {
    F2 x, y, z;
};
__device__ __forceinline__ V3x2 pci_force_pair(const DevParams& P, const float* __restrict__ tables, V3 xi, float tf,
                                               float4 p, float4 q)
{
    const F2 dx = f2(xi.x - p.x, xi.x - q.x), dy = f2(xi.y - p.y, xi.y - q.y), dz = f2(xi.z - p.z, xi.z - q.z);
    const F2 nd = neg_sqrt_rn(neg_sqmag(dx, dy, dz)), y = recip_rn(nd);
    const F2 w = weight_sdw(nd, P, tables), s = f2(tf + p.w, tf + q.w);
    return V3x2{div_by(dx, nd, y) * w * s, div_by(dy, nd, y) * w * s, div_by(dz, nd, y) * w * s};
}
// The sum over the pairs.
template <bool kExactDiv>
__device__ __forceinline__ V3 pci_force_walk(const DevParams& P, const StepBuffers& b, int i, const float4* ppos)
{
    const float4 pi4 = ppos[i];
    const V3 xi = v3(pi4);
    const float tf = pi4.w;
    V3 pf = v3(0.f, 0.f, 0.f);
    auto pair = [&](int j0, float4 p, int j1, float4 q, bool two) {
        if (!kExactDiv) {
            if (j0 != i) pf += pci_force_term(P, b.tables, xi, tf, p);
            if (two && j1 != i) pf += pci_force_term(P, b.tables, xi, tf, q);
            return;
        }
        const V3x2 f = pci_force_pair(P, b.tables, xi, tf, p, q);
        if (j0 != i) pf += v3(lo(f.x), lo(f.y), lo(f.z));
        if (two && j1 != i) pf += v3(hi(f.x), hi(f.y), hi(f.z));
    };
    for_each_neighbor<2>(b.nbr, i, P.nbr_stride, __ldg(b.nbr_count + i), [&](int j) { return ppos[j]; }, pair);
    return pf;
}
__device__ __forceinline__ V3 pci_force_sum(const DevParams& P, const StepBuffers& b, int i, const float4* ppos)
{
    return *(const volatile uint32_t*)&b.status->div_unsafe == 0u ? pci_force_walk<true>(P, b, i, ppos)
                                                                   : pci_force_walk<false>(P, b, i, ppos);
}
__device__ __forceinline__ void pci_force_one(const DevParams& P, const StepBuffers& b, int i, const float4* ppos)
{
    b.pforce[i] = f4(pci_pressure_force(P, b.rho[i], pci_force_sum(P, b, i, ppos)), 0.f);
}

// All forces of SPH in one walk of the list: nonpressure_walk's sums and, beside them, the pressure
// force's (SPHSolver::accumulatePressureForces, CPU branch, SPHSolver.cpp:268-290), which is the PCISPH
// force's sum over the positions and factors p / rho^2 (StepBuffers::xpf; the factor is the quotient the
// reference takes per pair), without its test for NaN. Where the step's positions are in range, the
// distance and direction come from the exact forms, two pairs at a time. Two walks, each fetching the
// list and the neighbours' positions, took 37 + 25 us at 250,047 particles; this one 45.5 in blocks
// of 128 threads with the 94 registers it asks for (47.5 with 80, 60 with 64 and spills, 50 in blocks
// of 256).
template <bool kExactDiv>
__device__ __forceinline__ void sph_forces_walk(const DevParams& P, const StepBuffers& b, int i)
{
    const float4 xi4 = b.xpf[i];
    const V3 xi = v3(xi4);
    const float tf = xi4.w;
    const V3 vi = v3(b.vel[i]);
    const float rhoi = b.rho[i];
    V3 normal = v3(0.f, 0.f, 0.f), visc = v3(0.f, 0.f, 0.f), pf = v3(0.f, 0.f, 0.f);
    float lap = 0.f;
    auto one = [&](int j, const NonpressureRec& r) {
        const NonpressureTerms t = nonpressure_term<false>(P, b.tables, xi, vi, rhoi, r);
        normal += t.normal;
        lap += t.lap;
        if (j == i) return;
        visc += t.visc;
        pf += pci_force_term(P, b.tables, xi, tf, r.x);
    };
    auto pair = [&](int j0, const NonpressureRec& r0, int j1, const NonpressureRec& r1, bool two) {
        if (!kExactDiv) {
            one(j0, r0);
            if (two) one(j1, r1);
            return;
        }
        const NonpressureTerms2 t = nonpressure_pair<false>(P, b.tables, xi, vi, rhoi, r0, r1);
        const V3x2 f = pci_force_pair(P, b.tables, xi, tf, r0.x, r1.x);
        normal += v3(lo(t.nx), lo(t.ny), lo(t.nz));
        lap += lo(t.lap);
        visc += v3(lo(t.vx), lo(t.vy), lo(t.vz));
        if (j0 != i) pf += v3(lo(f.x), lo(f.y), lo(f.z));
        if (two) {
            normal += v3(hi(t.nx), hi(t.ny), hi(t.nz));
            lap += hi(t.lap);
            visc += v3(hi(t.vx), hi(t.vy), hi(t.vz));
            if (j1 != i) pf += v3(hi(f.x), hi(f.y), hi(f.z));
        }
    };
    for_each_neighbor<2>(b.nbr, i, P.nbr_stride, __ldg(b.nbr_count + i),
                         [&](int j) { return NonpressureRec{b.xpf[j], b.vrho[j]}; }, pair);
    V3 F = nonpressure_force(P, rhoi, normal, lap, visc);
    pf *= -(P.mass * rhoi);
    F += pf;
    b.force[i] = f4(F, rhoi);
}
__device__ __forceinline__ void sph_forces_one(const DevParams& P, const StepBuffers& b, int i)
{
    if (P.exact_tables && *(const volatile uint32_t*)&b.status->np_unsafe == 0u)
        sph_forces_walk<true>(P, b, i);
    else
        sph_forces_walk<false>(P, b, i);
}

// The persistent loops' fused pass: the pressure force of iteration k - 1 at positions `from`, then
// the prediction of iteration k into `to`, or (last) the integration. The force goes from one to the
// other in registers and is stored in the last pass only; the particle's density rides in the
// non-pressure force's w (nonpressure_walk); first: some particle is on its first step
// (DevStatus::any_first), else its velocity is not read. 40 of about 150 bytes a particle and iteration
// less: 8 iterations of 991,440 particles 1.230 -> 1.188 ms, with the slot's shared constants.
__device__ __forceinline__ void pci_force_and_move(const DevParams& P, const StepBuffers& b, int i, const float4* from,
                                                   float4* to, bool last, bool first)
{
    const V3 sum = pci_force_sum(P, b, i, from);
    const float4 f4r = b.force[i], p4 = b.pos[i], h4 = b.half[i];
    const float4 v4 = first ? b.vel[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    V3 F = v3(f4r);
    const float rho = f4r.w;
    const V3 Fp = pci_pressure_force(P, rho, sum);
    if (!last) {
        V3 px, ph;
        predict_motion(P, b.colliders + P.coll_off, b.status, F, Fp, rho, v3(p4), v3(v4), v4.w, v3(h4), px, ph);
        to[i] = f4(px, 0.f);
        b.phalf[i] = f4(ph, 0.f);
        return;
    }
    b.pforce[i] = f4(Fp, 0.f);
    F += Fp;
    V3 x = v3(p4), v = v3(v4), half = v3(h4), old;
    float flag = v4.w;
    integrate_motion(P, b.colliders + P.coll_off, F, rho, x, v, flag, half, old);
    b.pos[i] = f4(x, p4.w);
    b.vel[i] = f4(v, flag);
    b.half[i] = f4(half, h4.w);
    b.old[i] = f4(old, 0.f);
    if (b.hist) {
        // Warm-start pressure history: (p_n, p_{n-1}, p_{n-2}) for the next step's features.
        const float4 hs = b.hist[i];
        b.hist[i] = make_float4(b.pres[i], hs.x, hs.y, 0.f);
    }
}

}  // namespace lsp
