// Per-particle operations by a group of L consecutive lanes, for scenes too small to fill the
// chip with one thread per particle (small_step.cu). Each lane takes the four entries of one
// group of the list and evaluates their terms, two at a time; the terms go through shared memory and are then
// added in list order, each component by one lane, so every sum carries the bits of the
// one-thread walk (particle_ops.cuh): a missing entry adds +0 to a sum that started at +0, which
// changes no bit. What bounds a small scene is the serial walk's latency (nine dependent list and
// position fetches for 36 neighbours), which becomes one or two. Adding the terms from shuffles
// (seven components times 36 entries in the non-pressure pass) took two to three times as long.
//
// Every lane of a warp calls these together (a group without a particle with an empty list). All
// data that the same kernel has written is read with plain loads (no read-only path).
#pragma once

#include "particle_ops.cuh"

namespace lsp {

constexpr uint32_t kFullWarp = 0xffffffffu;
constexpr int kGroupSums = 10;   // most components of a walk (SPH forces)
// Floats of a group's row of terms: 4 per lane, padded so that 16-byte accesses of eight rows
// fall in different banks.
__host__ __device__ constexpr int group_pitch(int lanes) { return 4 * lanes + 4; }
// Shared memory of a block of the group walks.
constexpr size_t group_smem(int threads, int lanes)
{
    return (size_t)(threads / lanes) * kGroupSums * group_pitch(lanes) * sizeof(float);
}

template <int L>
struct Group {
    static_assert(L >= 2 && L <= 16 && (L & (L - 1)) == 0, "part of a warp");
    int lane;     // this thread's lane in its group
    float* row;   // the group's rows of terms in shared memory
    __device__ __forceinline__ Group(float* smem)
    {
        lane = threadIdx.x & (L - 1);
        row = smem + (threadIdx.x / L) * kGroupSums * group_pitch(L);
    }
};

// Component c of a walk's sums, in every lane of the group.
template <int L, int N>
__device__ __forceinline__ float group_sum(const float (&sum)[N], int c)
{
    return __shfl_sync(kFullWarp, sum[c / L], c % L, L);
}

// Sums of the C components that terms(j0, r0, j1, r1, t) writes to t[c][0] and t[c][1] for two
// entries, over a list of cnt entries in order (most: the largest count of the warp's groups);
// index(s): this lane's int4 of the list's s-th segment of 4 L entries, whose unused components may
// be any particle. Lane l ends with components l, l + L, ...
template <int L, int C, typename Index, typename Load, typename Terms>
__device__ __forceinline__ void group_walk(const Group<L>& g, int cnt, int most, Index index, Load load, Terms terms,
                                           float (&sum)[(C + L - 1) / L])
{
    constexpr int N = (C + L - 1) / L;
#pragma unroll
    for (int s = 0; s < N; s++) sum[s] = 0.f;
    for (int seg = 0; 4 * L * seg < most; seg++) {
        const int k = 4 * (seg * L + g.lane);   // this lane's first entry
        if (k < cnt) {
            const int4 q = index(seg);
#pragma unroll
            for (int h = 0; h < 4; h += 2) {
                const int j0 = h ? q.z : q.x, j1 = h ? q.w : q.y;
                const int left = cnt - k - h;
                float t[C][2];
                terms(j0, load(j0), j1, load(j1), t);
#pragma unroll
                for (int c = 0; c < C; c++)
                    *reinterpret_cast<float2*>(g.row + c * group_pitch(L) + 4 * g.lane + h) =
                        make_float2(left > 0 ? t[c][0] : 0.f, left > 1 ? t[c][1] : 0.f);
            }
        }
        __syncwarp();
        const int end = min(cnt - 4 * L * seg, 4 * L);
#pragma unroll
        for (int s = 0; s < N; s++) {
            const int c = g.lane + s * L;
            if (c < C) {
                const float4* from = reinterpret_cast<const float4*>(g.row + c * group_pitch(L));
#pragma unroll 4
                for (int u = 0; u < end; u += 4, from++) {
                    const float4 v = *from;
                    sum[s] += v.x;
                    sum[s] += v.y;
                    sum[s] += v.z;
                    sum[s] += v.w;
                }
            }
        }
        __syncwarp();
    }
}

// A group's particle and its list, held in registers for the whole step: the lane's index groups
// of the first 64 entries, the rest read from the stored list.
template <int L>
struct HeldList {
    static constexpr int kHeld = 16 / L;
    int4 q[kHeld];
    int cnt, most;   // entries (0 for a group without a particle), and the most of the warp's groups
    const int4* first;
    int64_t stride;
    __device__ __forceinline__ HeldList(const Group<L>& g, const DevParams& P, const StepBuffers& b, int i, bool valid)
    {
        cnt = valid ? b.nbr_count[i] : 0;
        stride = P.nbr_stride;
        first = reinterpret_cast<const int4*>(b.nbr) + i + g.lane * stride;
#pragma unroll
        for (int s = 0; s < kHeld; s++) {
            q[s] = make_int4(i, i, i, i);
            if (4 * (s * L + g.lane) < cnt) q[s] = first[s * L * stride];
        }
        most = __reduce_max_sync(kFullWarp, cnt);
    }
    __device__ __forceinline__ int4 operator()(int seg) const
    {
        if (seg >= kHeld) return first[seg * L * stride];
        int4 v = q[0];
#pragma unroll
        for (int s = 1; s < kHeld; s++)
            if (seg == s) v = q[s];
        return v;
    }
};

// Sum of W of a particle at xi over its list at the positions x (density_sum), in every lane.
template <int L, typename Index>
__device__ __forceinline__ float group_density_sum(const Group<L>& g, const DevParams& P, const float* __restrict__ tables,
                                                   const float4* x, V3 xi, int cnt, int most, Index index)
{
    float sum[1];
    group_walk<L, 1>(
        g, cnt, most, index, [&](int j) { return x[j]; },
        [&](int, float4 p, int, float4 q, float (&t)[1][2]) {
            const F2 w = density_pair(P, tables, xi, p, q);
            t[0][0] = lo(w);
            t[0][1] = hi(w);
        },
        sum);
    return group_sum<L>(sum, 0);
}

// neighbors_one by a group: each lane scans whole rows (row r by lane r mod L), the entries' places
// follow from the rows' counts, and the list goes out four entries a lane from shared memory
// (list: kGroupList entries of the group). Returns the true count; *wsum as in neighbors_one. More
// than 16 rows, a row of more than 32 particles or a longer list: the group's first lane takes
// neighbors_one with the list's memory as its mask column.
constexpr int kGroupList = 128;
static_assert(kGroupList * sizeof(int) >= kScanChunks * sizeof(uint2), "the list's memory holds a mask column");
template <int L>
__device__ __forceinline__ int group_neighbors(const Group<L>& g, const DevParams& P, const float4* pos,
                                               const float* __restrict__ tables, const uint32_t* cell_start, int32_t* nbr,
                                               int i, bool valid, int* list, float* wsum)
{
    constexpr int S = 16 / L;   // rows per lane
    const V3 xi = v3(pos[i]);
    const float above = __uint_as_float(__float_as_uint(P.h2) + 1u);   // the next float above h^2
    int lo_[3], hi_[3];
    search_box(P, xi, lo_, hi_);
    const int ry = hi_[1] - lo_[1] + 1;
    const int rows = valid && lo_[2] <= hi_[2] && lo_[0] <= hi_[0] && ry > 0 ? (hi_[0] - lo_[0] + 1) * ry : 0;
    bool plain = rows <= 16;
    int beg[S], len[S];
#pragma unroll
    for (int s = 0; s < S; s++) {
        const int r = g.lane + s * L;
        beg[s] = len[s] = 0;
        if (r < rows) {
            const int cx = lo_[0] + r / ry, cy = lo_[1] + r % ry;
            const uint32_t row = P.cell_base + ((uint32_t)cx * (uint32_t)P.ny + (uint32_t)cy) * (uint32_t)P.nz;
            beg[s] = (int)cell_start[row + lo_[2]];
            len[s] = (int)cell_start[row + hi_[2] + 1] - beg[s];
        }
        plain = plain && len[s] <= 32;
    }
    uint32_t bits[S];
    int last[S], place[S], cnt = 0;
#pragma unroll
    for (int s = 0; s < S; s++) {
        bits[s] = scan_row<8>(pos, xi, above, beg[s], min(len[s], 32), last[s]);
        const int own = __popc(bits[s]);
        int upto = own;   // entries of this lane's row and the rows of the lanes before it
#pragma unroll
        for (int o = 1; o < L; o <<= 1) {
            const int y = __shfl_up_sync(kFullWarp, upto, o, L);
            if (g.lane >= o) upto += y;
        }
        place[s] = cnt + upto - own;
        cnt += __shfl_sync(kFullWarp, upto, L - 1, L);
    }
    plain = plain && cnt <= kGroupList;
    const uint32_t lanes = ((1u << L) - 1u) << ((threadIdx.x & 31) & ~(L - 1));
    const bool fast = (__ballot_sync(kFullWarp, !plain) & lanes) == 0u;
    if (fast) {
#pragma unroll
        for (int s = 0; s < S; s++) {
            uint32_t m = bits[s];
            for (int k = place[s]; m; k++) {
                const int bit = 31 - __clz((int)m);
                m ^= 1u << bit;
                list[k] = last[s] - bit;
            }
        }
        // The unused components of the last group.
        for (int k = cnt + g.lane; k < ((cnt + 3) & ~3); k += L) list[k] = i;
    }
    __syncwarp();
    int4* out = reinterpret_cast<int4*>(nbr) + i;
    const int4* in = reinterpret_cast<const int4*>(list);
    // A list longer than its capacity is cut; the step is redone with longer lists.
    const int stored = fast ? min(cnt, P.nbr_cap) : 0;
    for (int k = 4 * g.lane; k < stored; k += 4 * L) out[(int64_t)(k >> 2) * P.nbr_stride] = in[k >> 2];
    *wsum = group_density_sum(g, P, tables, pos, xi, stored, (int)__reduce_max_sync(kFullWarp, stored),
                              [&](int seg) { return in[seg * L + g.lane]; });
    if (!fast) {
        float sum = 0.f;
        if (g.lane == 0) cnt = neighbors_one(P, pos, cell_start, nbr, i, tables, reinterpret_cast<uint2*>(list), 1, &sum);
        *wsum = sum;
    }
    __syncwarp();
    return cnt;   // of the first lane where neighbors_one ran
}

// Whether the word is set, the same in every lane: the walks' two instances are full of warp-wide
// operations, so a warp has to take one of them as a whole, and another block may be setting the
// word (div_unsafe: predict_motion of a block that is a pass ahead). Both give the same bits then.
__device__ __forceinline__ bool any_lane_sees(const uint32_t* word)
{
    return __any_sync(kFullWarp, *(const volatile uint32_t*)word != 0u);
}

// The non-pressure force of particle i (nonpressure_one without the warm-start feature), in every lane.
template <int L, bool kExactDiv>
__device__ __forceinline__ V3 group_nonpressure_walk(const Group<L>& g, const DevParams& P, const StepBuffers& b, int i,
                                                     V3 xi, V3 vi, float rhoi, const HeldList<L>& list)
{
    float sum[(7 + L - 1) / L];
    group_walk<L, 7>(
        g, list.cnt, list.most, list, [&](int j) { return NonpressureRec{b.pos[j], b.vrho[j]}; },
        [&](int j0, const NonpressureRec& r0, int j1, const NonpressureRec& r1, float (&t)[7][2]) {
            if (kExactDiv) {
                const NonpressureTerms2 n = nonpressure_pair<false>(P, b.tables, xi, vi, rhoi, r0, r1);
                const F2 c[7] = {n.nx, n.ny, n.nz, n.lap, n.vx, n.vy, n.vz};
#pragma unroll
                for (int k = 0; k < 7; k++) t[k][0] = lo(c[k]), t[k][1] = hi(c[k]);
            } else {
                auto one = [&](int j, const NonpressureRec& r, int e) {
                    const NonpressureTerms n = nonpressure_term<false>(P, b.tables, xi, vi, rhoi, r);
                    t[0][e] = n.normal.x, t[1][e] = n.normal.y, t[2][e] = n.normal.z, t[3][e] = n.lap;
                    t[4][e] = j != i ? n.visc.x : 0.f, t[5][e] = j != i ? n.visc.y : 0.f, t[6][e] = j != i ? n.visc.z : 0.f;
                };
                one(j0, r0, 0);
                one(j1, r1, 1);
            }
        },
        sum);
    float s[7];
#pragma unroll
    for (int c = 0; c < 7; c++) s[c] = group_sum<L>(sum, c);
    return nonpressure_force(P, rhoi, v3(s[0], s[1], s[2]), s[3], v3(s[4], s[5], s[6]));
}
template <int L>
__device__ __forceinline__ V3 group_nonpressure(const Group<L>& g, const DevParams& P, const StepBuffers& b, int i, V3 xi,
                                                V3 vi, float rhoi, const HeldList<L>& list)
{
    return P.exact_tables && !any_lane_sees(&b.status->np_unsafe)
               ? group_nonpressure_walk<L, true>(g, P, b, i, xi, vi, rhoi, list)
               : group_nonpressure_walk<L, false>(g, P, b, i, xi, vi, rhoi, list);
}

// The pressure force's sum over the pairs of particle i at predicted position xi with factor tf
// (pci_force_walk), in every lane.
template <int L, bool kExactDiv>
__device__ __forceinline__ V3 group_pci_force_walk(const Group<L>& g, const DevParams& P, const StepBuffers& b, int i,
                                                   const float4* ppos, V3 xi, float tf, const HeldList<L>& list)
{
    float sum[(3 + L - 1) / L];
    group_walk<L, 3>(
        g, list.cnt, list.most, list, [&](int j) { return ppos[j]; },
        [&](int j0, float4 p, int j1, float4 q, float (&t)[3][2]) {
            V3 f0, f1;
            if (kExactDiv) {
                const V3x2 f = pci_force_pair(P, b.tables, xi, tf, p, q);
                f0 = v3(lo(f.x), lo(f.y), lo(f.z));
                f1 = v3(hi(f.x), hi(f.y), hi(f.z));
            } else {
                f0 = pci_force_term(P, b.tables, xi, tf, p);
                f1 = pci_force_term(P, b.tables, xi, tf, q);
            }
            t[0][0] = j0 != i ? f0.x : 0.f, t[1][0] = j0 != i ? f0.y : 0.f, t[2][0] = j0 != i ? f0.z : 0.f;
            t[0][1] = j1 != i ? f1.x : 0.f, t[1][1] = j1 != i ? f1.y : 0.f, t[2][1] = j1 != i ? f1.z : 0.f;
        },
        sum);
    return v3(group_sum<L>(sum, 0), group_sum<L>(sum, 1), group_sum<L>(sum, 2));
}
template <int L>
__device__ __forceinline__ V3 group_pci_force(const Group<L>& g, const DevParams& P, const StepBuffers& b, int i,
                                              const float4* ppos, V3 xi, float tf, float rhoi, const HeldList<L>& list)
{
    return pci_pressure_force(P, rhoi,
                              any_lane_sees(&b.status->div_unsafe)
                                  ? group_pci_force_walk<L, false>(g, P, b, i, ppos, xi, tf, list)
                                  : group_pci_force_walk<L, true>(g, P, b, i, ppos, xi, tf, list));
}
// All forces of SPH of particle i (sph_forces_walk), in every lane. In one walk instead of two, each with
// its fetches and block of ordered sums, a step of 12,000 particles takes 1.6 us less.
template <int L, bool kExactDiv>
__device__ __forceinline__ V3 group_sph_walk(const Group<L>& g, const DevParams& P, const StepBuffers& b, int i, V3 xi, V3 vi,
                                             float rhoi, const HeldList<L>& list)
{
    const float tf = b.xpf[i].w;
    float sum[(10 + L - 1) / L];
    group_walk<L, 10>(
        g, list.cnt, list.most, list, [&](int j) { return NonpressureRec{b.xpf[j], b.vrho[j]}; },
        [&](int j0, const NonpressureRec& r0, int j1, const NonpressureRec& r1, float (&t)[10][2]) {
            if (kExactDiv) {
                const NonpressureTerms2 n = nonpressure_pair<false>(P, b.tables, xi, vi, rhoi, r0, r1);
                const V3x2 f = pci_force_pair(P, b.tables, xi, tf, r0.x, r1.x);
                const F2 c[10] = {n.nx, n.ny, n.nz, n.lap, n.vx, n.vy, n.vz, f.x, f.y, f.z};
#pragma unroll
                for (int k = 0; k < 10; k++) {
                    t[k][0] = k < 7 || j0 != i ? lo(c[k]) : 0.f;
                    t[k][1] = k < 7 || j1 != i ? hi(c[k]) : 0.f;
                }
            } else {
                auto one = [&](int j, const NonpressureRec& r, int e) {
                    const NonpressureTerms n = nonpressure_term<false>(P, b.tables, xi, vi, rhoi, r);
                    const V3 f = pci_force_term(P, b.tables, xi, tf, r.x);
                    t[0][e] = n.normal.x, t[1][e] = n.normal.y, t[2][e] = n.normal.z, t[3][e] = n.lap;
                    t[4][e] = j != i ? n.visc.x : 0.f, t[5][e] = j != i ? n.visc.y : 0.f, t[6][e] = j != i ? n.visc.z : 0.f;
                    t[7][e] = j != i ? f.x : 0.f, t[8][e] = j != i ? f.y : 0.f, t[9][e] = j != i ? f.z : 0.f;
                };
                one(j0, r0, 0);
                one(j1, r1, 1);
            }
        },
        sum);
    float s[10];
#pragma unroll
    for (int c = 0; c < 10; c++) s[c] = group_sum<L>(sum, c);
    V3 F = nonpressure_force(P, rhoi, v3(s[0], s[1], s[2]), s[3], v3(s[4], s[5], s[6]));
    V3 pf = v3(s[7], s[8], s[9]);
    pf *= -(P.mass * rhoi);
    F += pf;
    return F;
}
template <int L>
__device__ __forceinline__ V3 group_sph_forces(const Group<L>& g, const DevParams& P, const StepBuffers& b, int i, V3 xi,
                                               V3 vi, float rhoi, const HeldList<L>& list)
{
    return P.exact_tables && !any_lane_sees(&b.status->np_unsafe)
               ? group_sph_walk<L, true>(g, P, b, i, xi, vi, rhoi, list)
               : group_sph_walk<L, false>(g, P, b, i, xi, vi, rhoi, list);
}

}  // namespace lsp
